// Fused decode path: ONE persistent cooperative kernel per token (one CTA per SM; a prompt fed token by token: per up to 32 positions) instead of ~9 launches per layer.
// Replaces the launch sequence of run_llama_network (llama2_q4.cu:430-538), on one GPU or on every rank of a
// tensor-parallel group (hybrid split, llama2_q4.cu:45-50).
//
// What bounds it: a 7B layer is 105 MB of weights = 16 us of HBM time, and five dependent steps whose hand-overs through L2
// cost about as much. Weight addresses never depend on activations, so every warp keeps a private shared-memory ring full
// with cp.async.bulk (TMA, 1-D, no multicast), running ahead across the steps; what is left on the critical path is kept
// short: each warp waits only for the 256 inputs it multiplies, and the products run on the integer tensor pipe.
//
// Stream layout (built once per model on the device from the file layout, bytes per weight unchanged):
//   tile  = 8 output columns (gate/up: 4 columns of each, alternating); pair = 2 groups of 128 inputs
//   item  = tile x pair = [h = 0, 1: lane] uint4, [h = 2, 3: lane] uint4, then 16 words (fp16 scale | zero point << 16); lane 4c + t
//           holds words 4h + t of column c, groups A and B in turn: the registers of the product's row operand
//   Each CTA has a run of consecutive tiles; which CTAs have one more goes round from phase to phase, so that none always has the
//   extra tile. A CTA's items are ordered by pair, then tile, and cut into kW equal contiguous runs, one per warp: a warp
//   stages a pair's inputs once for all its tiles. Two items make a chunk, one bulk copy; chunk c of all warps of all CTAs
//   lie side by side, so that the chip streams one contiguous region at any moment.
//
// The W4 dot product runs on the integer tensor pipe (q4_w4dot.cuh). Per token of four 7B layers 179.5 us with DP4A, slots staged
// for the whole CTA and outputs in plain order, 152 now (position 1800: 220 and 187; two 70B layers: 229 and 192); the stream
// alone runs at 5.8 (7B) to 6.5 TB/s (70B). What is left per 7B layer (about 33 us): the items' instructions (about 14 us; two
// items take a warp as long to wait for and to replace as to multiply), hand-overs (1.3 us each and the CTAs' skew), staging 4 us,
// attention 4.6 us. Measured and not kept: one ring for the CTA with a 17th warp that fills it (96 registers, spills: 184 us) or
// with the warps taking turns (174 to 182 us: whoever refills holds the others up).
//
// Every wait is bounded (mbarrier polls, tag polls and barrier spins are limited by the global timer); on expiry the
// kernel records Q4_ERR_TIMEOUT in a status word, all later waits fall through, and the kernel returns.
#include <math_constants.h>
#include <stdio.h>
#include <stdlib.h>

#include "q4_bulk.cuh"
#include "q4_comm_internal.h"
#include "q4_model.h"
#include "q4_w4dot.cuh"

namespace {

constexpr int kW = 16;                  // warps per CTA, all alike: 4 per SM sub-partition, one per pair of a 4096-long input
constexpr int kThreads = 32 * kW;
constexpr int kItemBytes = 1088;        // 8 columns x 256 inputs: 1024 B of nibbles, 64 B of scales and zero points
constexpr int kChunkBytes = 2 * kItemBytes;
constexpr int kMaxDepth = 6, kMinDepth = 2;   // ring chunks per warp; the host picks as many as fit
constexpr int kClsChunk = 1024;         // halfs of one classifier row per ring chunk
constexpr int kTileStride = kW * 8 + 8; // floats between tiles of the partial sums (padded: the summing threads hit distinct banks)
constexpr int kMaxDim = 11264;          // largest model dimension this path takes
constexpr int kMaxGroups = 256;         // most groups of an input vector
constexpr int kSplitLen = 128;          // positions per attention split before a head is split further
constexpr int kMaxSplit = 4;            // attention splits per head (merged in registers by the next phase)
constexpr int kAttnPart = 128 + 4;      // tagged words per attention partial: 128 outputs as fp16 (normalised by the split's own sum),
                                        // then max and sum as two 16-bit pieces each
constexpr int kAttnPartStride = 160;    // whole 128-byte lines
constexpr int kTraceCols = 8;           // timestamps per phase: 0 start, 1 first inputs staged, 2 items done, 3 outputs written, 4-6 staging detail
constexpr unsigned kPollLimit = 1u << 26;                        // polls, and
constexpr unsigned long long kDefaultWaitNs = 2000ULL * 1000 * 1000;  // default limit of a device-side wait: two seconds on the global timer (FParams::wait_ns)

// Measurement and test switches of the kernel (skip the math, keep the exchange local) exist only in the test build of the
// library; in the product build the expression is the constant 0 and the branches are compiled out.
#ifdef Q4_TEST_BUILD
#define Q4_DBG(p) ((p).debug)
#else
#define Q4_DBG(p) 0
#endif

enum Kind { K_QKV = 0, K_O = 1, K_GU = 2, K_DOWN = 3, K_KINDS = 4 };
// trace codes of the phases (q4_model_trace)
enum PhaseType { PH_EMBED = 0, PH_GEMV = 1, PH_ATTN = 2, PH_CLS = 3, PH_ARGMAX = 4 };
constexpr int kLayerPhases = 5;         // QKV, attention, O, gate/up, down
enum LayerPhase { LP_QKV = 0, LP_ATTN = 1, LP_O = 2, LP_GU = 3, LP_DOWN = 4 };

// One kind of matrix step; the same in every layer.
struct FKind {
    int K, P;               // inputs, pairs of groups
    int NT, nt_div, nt_mod; // tiles; tiles per CTA and remainder: run c (of CTA (c + rotation) % grid) has nt_div + (c < nt_mod)
    float inv_long, inv_short;   // 1 / (nt_div + 1), 1 / nt_div
    int xtile, xstride;     // exchange layout of the outputs: words per tile, and per run (whole 128-byte lines)
    int barrier_after;      // fewer tiles than CTAs: a grid barrier keeps the CTAs without one in step
};

struct FParams {
    FKind kind[K_KINDS];
    int n_layers, nphases;
    const uint8_t* const* stream[K_KINDS];  // [n_layers] stream-layout weights of each step
    const __half* const* norms[2];          // [n_layers] RMSNorm weights before QKV and before gate/up
    const void* const* table;               // far form only: [n_layers][K_KINDS] of the first, then [n_layers][2] of the second
    const __half* rms_final;
    int dim, kv_n, q_n, kv_mul, n_heads, nsplit, v_n;
    long long layer_stride;        // halfs of one layer's K (or V) cache
    float gpu_count;
    // Tagged activations: every element is a 32-bit word, fp16 value in the low half and the low 16 bits of
    // (tag_base + producing phase + 1) in the high half. A reader polls the words themselves until all carry the expected
    // tag, so op boundaries need no grid barrier: one L2 round trip instead of fence + arrive + poll. A buffer is rewritten
    // only after every CTA has provably read it: a CTA writes a phase's outputs only after a CTA-wide barrier that all its
    // warps reach having read their inputs, every CTA has a tile of every phase, and a writer of a buffer has polled, as a CTA,
    // outputs that all CTAs produced after their last read of it. (Phases with fewer tiles than CTAs end with a grid barrier,
    // because a CTA without tiles writes nothing that anyone waits for and could otherwise fall behind unnoticed.)
    //
    // Every vector is laid out by who writes it: a CTA's outputs in 128-byte lines of their own (exchange_at). 148 CTAs that write their
    // shares of a 16 KB vector and poll all of it need 4.2 us per exchange when a 32-byte sector has two writers, 1.5 with one
    // writer per sector and 1.3 with one per line.
    //
    // The residual stream is the one vector that all ranks of a tensor-parallel group share. It lives in the exchange
    // area of the communicator as g partial vectors ("slots", one per source rank) in two alternating buffers:
    // buffer 1 is written by the embedding and by every down projection, buffer 0 by every o projection. A rank's
    // epilogue stores half(own partial sum + old x / g) into its slot on EVERY rank (plain peer stores, tagged), and
    // a reader sums the g slots in rank order in fp32: that is the all-reduce of cuda_comm.h:203-300 without a
    // separate step, and every rank computes bit-identical sums. A rank that writes buffer b has, for every other rank, consumed
    // data which that rank produced after its last read of b (o projection: the peer's down-projection partials of the
    // previous layer, read while staging QKV; down projection: the peer's o-projection partials, read while staging gate/up).
    uint32_t* xb[2][Q4_MAX_GPUS];      // [buffer][rank p]: buffer base (g slots of kLLMaxDim words) in rank p's exchange area
    unsigned long long* cand[Q4_MAX_GPUS];  // rank p's candidate mailbox [2][Q4_MAX_GPUS][2]
    uint16_t* ll_logits[Q4_MAX_GPUS];  // rank p's gathered logits
    int g, rank, vocab_off, vocab_size;
    unsigned launch_parity;
    uint32_t *hb, *qkv;      // tagged, in exchange layout: SiLU output; q | k | v
    unsigned tag_base;       // of the first position
    int n_tokens;            // positions of this launch, one after the other; the hand-off is the last one's
    __half *logits, *kc, *vc;
    const __half *emb, *wcls;
    const float* rope;       // [seq_len][64] (cos, sin)
    uint32_t* attn_part;     // [heads*nsplit][kAttnPartStride], tagged with the attention phase
    float* cand_val;         // [grid]
    int* cand_idx;           // [grid]
    int* pos_dev;
    int* tokens_pinned;
    volatile int* pos_pinned;
    unsigned long long* bar_counter;
    unsigned long long bar_base;  // barriers completed by earlier launches
    int* status;
    int write_token;
    int no_handoff;              // 1: leave the token mailbox and the last position's step alone (a sampling kernel follows on the stream)
    int debug;                   // test build only (Q4_TEST_BUILD; always 0 and compiled out of the product library):
                                 // 1 = consumers skip the waits and the math (pure streaming), 2 = the positions behind a launch's first embed
                                 // nothing, so that their readers' waits run out, 16 = tensor-parallel exchange kept local (no NVLink dependency)
    unsigned long long wait_ns;  // limit of every device-side wait on the global timer; on expiry the kernel records Q4_ERR_TIMEOUT
    int depth;                   // ring chunks per warp
    int split_len;               // positions per attention split (a head is split in ceil(T / split_len) parts, at most nsplit)
    unsigned long long* trace;   // optional: [2 CTAs][nphases][8] device timestamps (ns), or null
    // shared memory carve-up (bytes): ring | digit scratch | x | partial sums A (QKV, gate/up; attention scratch) | B (o, down) | tables
    int scr_off, x_off, part_a_off, part_b_off, table_off;
};

// ------------------------------------------------------------------------------------------------------------
// device helpers
// ------------------------------------------------------------------------------------------------------------
// Bounded wait of a whole warp. Returns false (and records the error) when the limit is hit, or at once when another wait has run out.
__device__ __noinline__ bool mbar_wait_slow(uint64_t* b, uint32_t parity, int* status, unsigned long long limit_ns) {
    unsigned long long t0 = 0;
    for (unsigned i = 0; i < kPollLimit; i++) {
        if (mbar_try(b, parity)) return true;
        if ((i & 63u) == 63u) {
            if (*(volatile int*)status != 0) return false;
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit_ns) break;
        }
    }
    if (atomicCAS(status, 0, Q4_ERR_TIMEOUT) == 0) status[1] = 0x40000 + (int)(smem_u32(b) & 0xFFFF);
    return false;
}
__device__ __forceinline__ float fma_mixed(__half a, __half b, float c) {
    float d;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"(__half_as_ushort(a)), "h"(__half_as_ushort(b)), "f"(c));
    return d;
}

// Grid-wide barrier among all CTAs.
__device__ __forceinline__ void grid_barrier(const FParams& p, unsigned& nbar) {
    __syncthreads();  // orders every thread's stores before thread 0's release below (cumulativity)
    if (threadIdx.x == 0) {
        nbar++;
        const unsigned long long target = (p.bar_base + nbar) * (unsigned long long)gridDim.x;
        unsigned long long v;
        asm volatile("atom.add.release.gpu.global.u64 %0, [%1], 1;" : "=l"(v) : "l"(p.bar_counter) : "memory");
        unsigned spins = 0;
        unsigned long long t0 = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p.bar_counter) : "memory");
            if (v >= target) break;
            if ((++spins & 63u) == 0) {
                if (*(volatile int*)p.status != 0) break;
                const unsigned long long now = global_ns();
                if (t0 == 0) t0 = now;
                else if (now - t0 > 2 * p.wait_ns) {   // longer than any single data wait, so that the root cause is what gets recorded
                    if (atomicCAS(p.status, 0, Q4_ERR_TIMEOUT) == 0) { p.status[1] = 0x50000 + (int)nbar; p.status[2] = (int)v; p.status[3] = (int)target; }
                    break;
                }
            }
        }
    }
    __syncthreads();
}

// Timestamps of CTA 0 and of the last CTA (thread 0), see kTraceCols
#define TRACE(pi, k)                                                                                          \
    do {                                                                                                      \
        if (p.trace && tid == 0 && (cta == 0 || cta == grid - 1))                                             \
            p.trace[((size_t)(cta == 0 ? 0 : 1) * p.nphases + (pi)) * kTraceCols + (k)] = global_ns();        \
    } while (0)

__device__ __forceinline__ float silu_mul(float g, float u) {
    float val = g;
    val *= 1.0f / (1.0f + expf(-val));
    val *= u;
    return val;
}

// ---- tagged activations -----------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tag_of(unsigned base, int phase) { return ((base + (unsigned)phase + 1u) & 0xFFFFu) << 16; }   // base: the position's first
__device__ __forceinline__ uint32_t tagged(__half v, uint32_t tag_hi) { return tag_hi | (uint32_t)__half_as_ushort(v); }
// Tagged words are exchanged between CTAs without a barrier, so both sides use strong (volatile) accesses: a weak load
// may be served from a stale copy for as long as it likes (observed: polling with ld.global.cg never saw the update),
// and the compiler may hoist it out of the wait loop.
__device__ __forceinline__ uint4 ld_poll(const uint4* p) {
    uint4 r;
    asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ void st_tagged(uint32_t* p, uint32_t v) { asm volatile("st.volatile.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void st_tagged4(uint32_t* p, uint4 v) {
    asm volatile("st.volatile.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// 8 consecutive tagged elements, as two 128-bit loads
struct Tagged8 { uint4 a, b; };
__device__ __forceinline__ Tagged8 ld_tagged8(const uint32_t* src) {
    Tagged8 t;
    t.a = ld_poll(reinterpret_cast<const uint4*>(src));
    t.b = ld_poll(reinterpret_cast<const uint4*>(src) + 1);
    return t;
}
__device__ __forceinline__ uint32_t tag_mismatch(const Tagged8& t, uint32_t tag_hi) {
    return ((t.a.x ^ tag_hi) | (t.a.y ^ tag_hi) | (t.a.z ^ tag_hi) | (t.a.w ^ tag_hi) | (t.b.x ^ tag_hi) | (t.b.y ^ tag_hi) | (t.b.z ^ tag_hi) | (t.b.w ^ tag_hi)) >> 16;
}
__device__ __forceinline__ uint4 tagged_values(const Tagged8& t) {
    return make_uint4(prmt(t.a.x, t.a.y, 0x5410), prmt(t.a.z, t.a.w, 0x5410), prmt(t.b.x, t.b.y, 0x5410), prmt(t.b.z, t.b.w, 0x5410));
}
// The 8 fp16 values as a uint4; ORs every tag mismatch into `bad`.
__device__ __forceinline__ uint4 load_tagged8(const uint32_t* src, uint32_t tag_hi, uint32_t& bad) {
    const Tagged8 t = ld_tagged8(src);
    bad |= tag_mismatch(t, tag_hi);
    return tagged_values(t);
}
// Bounded retry bookkeeping for the tag polls: returns false when the wait must be given up.
__device__ __forceinline__ bool keep_polling(unsigned& polls, unsigned long long& t0, int* status, unsigned long long limit_ns, int where = 0) {
    if ((++polls & 15u) == 0) {
        if (*(volatile int*)status != 0) return false;
        const unsigned long long now = global_ns();
        if (t0 == 0) t0 = now;
        else if (now - t0 > limit_ns) {
            if (atomicCAS(status, 0, Q4_ERR_TIMEOUT) == 0) status[1] = where;  // where the first wait ran out (diagnostics)
            return false;
        }
    }
    return true;
}

// Words (8 elements each) at at[b] of the residual stream: waits for the g partial vectors (one per source rank) and sums
// them in rank order in fp32, rounded to fp16 once - the arithmetic of a fixed-order all-reduce. Up to four slots of a
// word are in flight per round trip (on one GPU: the NB words).
template <int NB>
__device__ __forceinline__ void load_x_batch(uint4 (&xv)[NB], const bool (&valid)[NB], const int (&at)[NB], const uint32_t* base, int g,
                                             uint32_t want, int* status, unsigned long long limit_ns, int where) {
    unsigned polls = 0;
    unsigned long long t0 = 0;
    if (g == 1) {
        for (;;) {
            uint32_t bad = 0;
#pragma unroll
            for (int b = 0; b < NB; b++) {
                xv[b] = make_uint4(0, 0, 0, 0);
                if (valid[b]) xv[b] = load_tagged8(base + at[b], want, bad);
            }
            if (bad == 0 || !keep_polling(polls, t0, status, limit_ns, where)) break;
        }
        return;
    }
    constexpr int SB = 1;   // words per sub-batch (two would make the kernel spill, and there is next to no L1 behind a spill)
#pragma unroll
    for (int b0 = 0; b0 < NB; b0 += SB) {
        float acc[SB][8];
#pragma unroll
        for (int b = 0; b < SB; b++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[b][j] = 0.f;
        bool any = false;
#pragma unroll
        for (int b = 0; b < SB; b++) any |= valid[b0 + b];
        for (int r0 = 0; r0 < g && any; r0 += 4) {
            uint4 a[SB][4];
            for (;;) {
                uint32_t bad = 0;
#pragma unroll
                for (int b = 0; b < SB; b++)
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        a[b][c] = make_uint4(0, 0, 0, 0);
                        if (valid[b0 + b] && r0 + c < g) a[b][c] = load_tagged8(base + (size_t)(r0 + c) * kLLMaxDim + at[b0 + b], want, bad);
                    }
                if (bad == 0 || !keep_polling(polls, t0, status, limit_ns, where)) break;
            }
#pragma unroll
            for (int b = 0; b < SB; b++)
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (r0 + c < g) {
                        const __half2* ha = reinterpret_cast<const __half2*>(&a[b][c]);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const float2 fa = __half22float2(ha[j]);
                            acc[b][2 * j] += fa.x;
                            acc[b][2 * j + 1] += fa.y;
                        }
                    }
                }
        }
#pragma unroll
        for (int b = 0; b < SB; b++) {
            __half2* oh = reinterpret_cast<__half2*>(&xv[b0 + b]);
#pragma unroll
            for (int j = 0; j < 4; j++) oh[j] = __floats2half2_rn(acc[b][2 * j], acc[b][2 * j + 1]);
        }
    }
}

// Where tile t's outputs lie in the exchange layout of step k.
__device__ __forceinline__ int exchange_at(const FKind& k, int t) {
    const int longs = k.nt_mod * (k.nt_div + 1);     // tiles in the runs with one more
    const int c = t < longs ? (int)(((float)t + 0.5f) * k.inv_long) : k.nt_mod + (int)(((float)(t - longs) + 0.5f) * k.inv_short);
    return c * k.xstride + (t - (c * k.nt_div + min(c, k.nt_mod))) * k.xtile;
}
// This warp's share of a matrix step: its CTA has run `run`, tiles t0, t0 + 1, ...; its items [i0, i1) of tiles x pairs, pair-major.
struct Share { int run, t0, tiles, i0, i1; };
__device__ __forceinline__ Share share_of(const FKind& k, int rot, int cta, int grid, int w) {
    Share s;
    s.run = cta - rot;
    if (s.run < 0) s.run += grid;
    s.t0 = s.run * k.nt_div + min(s.run, k.nt_mod);
    s.tiles = k.nt_div + (s.run < k.nt_mod ? 1 : 0);
    const int n = s.tiles * k.P;
    s.i0 = (w * n) / kW;
    s.i1 = ((w + 1) * n) / kW;
    return s;
}
__device__ __forceinline__ int next_rot(const FKind& k, int rot, int grid) {
    rot += k.nt_mod;
    return rot >= grid ? rot - grid : rot;
}

// A warp's private ring of weight chunks. The warp that has read a chunk requests the one that takes its place, so there is no
// producer, no "empty" barrier, and a slot's parity cannot be mistaken for another round's: nobody else waits for it.
// What only the requesting lane 0 needs lies in shared memory: with 512 threads every register counts, and next to this much
// shared memory the L1 that would hold a spill is 4 KB.
struct Requests {           // the segment being requested: this warp's chunks of a matrix step, or one classifier row
    const uint8_t* src;
    uint32_t left, chunk;   // bytes left in it, bytes per chunk
    uint32_t step;          // distance between chunks
    int seg, rot, row;
};
struct Ring {
    uint8_t* base;
    uint64_t* bar;
    Requests* rq;
    int* more;              // kMany: positions behind the one whose segment is being requested
    int slot;
    uint32_t parity;        // of the round the next wait is for
    bool dead;              // a wait ran out: nothing more is requested or read
};
template <bool kMany>
__device__ __forceinline__ void next_segment(Requests& r, int* more, const FParams& p, const uint8_t* const* streams) {
    const int cta = blockIdx.x, grid = gridDim.x, w = threadIdx.x >> 5;
    int seg = r.seg, rot = r.rot;
    r.left = 0;
    for (;;) {
        if (seg == K_KINDS * p.n_layers) {
            if (!kMany || r.row < p.v_n || *more == 0) break;
            --*more;
            r.row = cta * kW + w;
            seg = rot = 0;
        }
        const FKind& k = p.kind[seg & (K_KINDS - 1)];
        const Share s = share_of(k, rot, cta, grid, w);
        rot = next_rot(k, rot, grid);
        const uint8_t* b = streams[seg++];
        if (s.i1 > s.i0) {
            r.left = (uint32_t)(s.i1 - s.i0) * kItemBytes;
            r.chunk = kChunkBytes;
            r.step = (uint32_t)grid * kW * kChunkBytes;
            r.src = b + (size_t)(cta * kW + w) * kChunkBytes;
            r.seg = seg;
            r.rot = rot;
            return;
        }
    }
    r.seg = seg;
    if (r.row >= p.v_n) return;
    r.left = (uint32_t)p.dim * 2;
    r.chunk = r.step = kClsChunk * 2;
    r.src = reinterpret_cast<const uint8_t*>(p.wcls + (size_t)r.row * p.dim);
    r.row += grid * kW;
}
// Requests the next chunk into `slot` (free: released just now, or never used). Lane 0.
template <bool kMany>
__device__ __forceinline__ void ring_request(const Ring& ring, int slot, const FParams& p, const uint8_t* const* streams) {
    Requests& r = *ring.rq;
    const uint32_t left = r.left, bytes = min(left, r.chunk);
    if (left == 0) return;
    const uint8_t* src = r.src;
    mbar_expect_tx(&ring.bar[slot], bytes);
    bulk_g2s(ring.base + slot * kChunkBytes, src, bytes, &ring.bar[slot]);
    r.left = left - bytes;
    r.src = src + r.step;
    if (left == bytes) next_segment<kMany>(r, ring.more, p, streams);
}
__device__ __forceinline__ const uint8_t* ring_wait(Ring& r, const FParams& p) {
    if (!r.dead && !__all_sync(0xffffffffu, mbar_try(&r.bar[r.slot], r.parity))) {
        const bool ok = mbar_wait_slow(&r.bar[r.slot], r.parity, p.status, p.wait_ns);
        if (!__all_sync(0xffffffffu, ok)) r.dead = true;
    }
    return r.base + r.slot * kChunkBytes;
}
// The warp has read the chunk: a shuffle or vote of values made from all that each lane read of it is behind the caller (a barrier alone
// does not wait for loads in flight).
template <bool kMany>
__device__ __forceinline__ void ring_release(Ring& r, const FParams& p, const uint8_t* const* streams) {
    __syncwarp();
    if (r.dead) return;
    if ((threadIdx.x & 31) == 0) ring_request<kMany>(r, r.slot, p, streams);
    if (++r.slot == p.depth) { r.slot = 0; r.parity ^= 1u; }
}

// ------------------------------------------------------------------------------------------------------------
// Staging of activations
// ------------------------------------------------------------------------------------------------------------
// One word (8 consecutive elements) of the attention output from the per-split partials (max, sum, un-normalised V sum):
// all splits' loads are issued together, merged in fixed split order, normalised and rounded to fp16 like the
// reference's attention output (gpu_kernels.h:335-336).
struct AttnWord {
    uint4 a[kMaxSplit];      // 8 fp16 values of the split's normalised output
    float2 ml[kMaxSplit];
};
// The partials arrive tagged (no grid barrier after the attention phase): every tag mismatch is ORed into `bad`.
__device__ __forceinline__ void attn_word_load(AttnWord& w, const FParams& p, int ns, int wd, bool valid, uint32_t want, uint32_t& bad) {
    const int h = (wd * 8) / 128, d = (wd * 8) % 128;
#pragma unroll
    for (int s = 0; s < kMaxSplit; s++) {
        w.ml[s] = make_float2(-CUDART_INF_F, 0.f);
        w.a[s] = make_uint4(0, 0, 0, 0);
        if (valid && s < ns) {
            const uint32_t* base = p.attn_part + ((size_t)h * p.nsplit + s) * kAttnPartStride;
            w.a[s] = load_tagged8(base + d, want, bad);
            const uint4 t = ld_poll(reinterpret_cast<const uint4*>(base + 128));
            bad |= ((t.x ^ want) | (t.y ^ want) | (t.z ^ want) | (t.w ^ want)) >> 16;
            w.ml[s] = make_float2(__uint_as_float((t.x & 0xFFFFu) | (t.y << 16)), __uint_as_float((t.z & 0xFFFFu) | (t.w << 16)));
        }
    }
}
__device__ __forceinline__ uint4 attn_word_merge(const AttnWord& w) {
    float M = -CUDART_INF_F;
#pragma unroll
    for (int s = 0; s < kMaxSplit; s++) M = fmaxf(M, w.ml[s].x);
    float L = 0.f, a[8];
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] = 0.f;
#pragma unroll
    for (int s = 0; s < kMaxSplit; s++) {
        if (w.ml[s].x != -CUDART_INF_F) {
            const float e = w.ml[s].y * __expf(w.ml[s].x - M);  // weight of the split = its sum, rescaled to the common max
            // (merge weights: the fast exponential's error is far below the fp16 outputs; the scores themselves use expf)
            L += e;
            const __half2* hh = reinterpret_cast<const __half2*>(&w.a[s]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __half22float2(hh[j]);
                a[2 * j] += f.x * e;
                a[2 * j + 1] += f.y * e;
            }
        }
    }
    uint4 out;
    __half2* oh = reinterpret_cast<__half2*>(&out);
    const float rl = L > 0.f ? 1.0f / L : 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) oh[j] = __floats2half2_rn(a[2 * j] * rl, a[2 * j + 1] * rl);
    return out;
}

// Splits per head at sequence length T: short contexts are not split at all (one CTA per head, no partial traffic).
__device__ __forceinline__ int attn_splits_for(const FParams& p, int T) { return min(p.nsplit, max(1, (T + p.split_len - 1) / p.split_len)); }

// An item's registers. The scales come first: shared-memory loads of a warp return in order, so that the product's start says that
// all of the item has been read.
struct Item { uint32_t meta; uint4 a, b; };
__device__ __forceinline__ void item_load(Item& it, const uint8_t* ib, int lane) {
    it.meta = *reinterpret_cast<const uint32_t*>(ib + 1024 + (lane >> 1) * 4);   // column lane >> 2, group (lane >> 1) & 1
    it.a = *reinterpret_cast<const uint4*>(ib + lane * 16);
    it.b = *reinterpret_cast<const uint4*>(ib + 512 + lane * 16);
}

// Waits for the residual stream, files it in xs (fp16, summed over the ranks) and returns 1 / rms. The sum of squares is taken per
// pair of groups once the pair has arrived and over the pairs in a fixed order: never in arrival order, which would make the last
// bit differ from run to run and from rank to rank. One CTA-wide barrier.
__device__ __forceinline__ float stage_residual(const FParams& p, int xbuf, uint32_t want, uint4* xs, float* ssq, int w, int lane, int where) {
    const int nwords = p.dim >> 3, npairs = (p.dim + 255) >> 8;
    for (int pr = w; pr < npairs; pr += 2 * kW) {
        const int wd[2] = {pr * 32 + lane, (pr + kW) * 32 + lane};
        const bool valid[2] = {wd[0] < nwords, wd[1] < nwords};
        uint4 xv[2];
        const int at[2] = {exchange_at(p.kind[K_DOWN], wd[0]), exchange_at(p.kind[K_DOWN], wd[1])};   // (a tile is a word)
        load_x_batch<2>(xv, valid, at, p.xb[xbuf][p.rank], p.g, want, p.status, p.wait_ns, where);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            if (pr + b * kW >= npairs) break;
            if (valid[b]) xs[wd[b]] = xv[b];
            float ss = 0.f;
            const __half2* h = reinterpret_cast<const __half2*>(&xv[b]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __half22float2(h[j]);
                ss = fmaf(f.x, f.x, ss);
                ss = fmaf(f.y, f.y, ss);
            }
            ss = warp_sum(ss);
            if (lane == 0) ssq[pr + b * kW] = ss;
        }
    }
    __syncthreads();
    float ss = lane < npairs ? ssq[lane] : 0.f;      // (at most 44 pairs)
    if (lane + 32 < npairs) ss += ssq[lane + 32];
    ss = warp_sum(ss);
    ss /= p.dim;
    ss += 1e-5f;
    return 1.0f / sqrtf(ss);
}
// x * (inv_rms * w) of 8 elements, rounded to fp16 once (gpu_kernels.h:100-102)
__device__ __forceinline__ uint4 norm_word(const uint4& xv, const uint4& wv, float inv_rms) {
    uint4 out;
    const __half2 *xh = reinterpret_cast<const __half2*>(&xv), *wh = reinterpret_cast<const __half2*>(&wv);
    __half2* oh = reinterpret_cast<__half2*>(&out);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 xf = __half22float2(xh[j]), wf = __half22float2(wh[j]);
        oh[j] = __floats2half2_rn(xf.x * (inv_rms * wf.x), xf.y * (inv_rms * wf.y));
    }
    return out;
}

// Dot product of 16 dims in a lane, fp16 operands, fp32 sum
__device__ __forceinline__ float dot16(const uint4 (&k)[2], const uint4 (&q)[2]) {
    const __half *kh = reinterpret_cast<const __half*>(k), *qh = reinterpret_cast<const __half*>(q);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 16; j++) s = fma_mixed(kh[j], qh[j], s);
    return s;
}
// Rotates one head's 128 values at this position: lane l holds dims 2l, 2l + 1 and their partners 64 above (gpu_kernels.h:340-363,
// angles tabulated at load time). first_tile: the head's first tile in the QKV step.
__device__ __forceinline__ void rotate_head(const FParams& p, int first_tile, uint32_t want, int pos, __half* dst, int lane, int where) {
    const uint32_t* src = p.qkv + exchange_at(p.kind[K_QKV], first_tile + (lane >> 2)) + 2 * (lane & 3);
    const uint32_t* src_hi = p.qkv + exchange_at(p.kind[K_QKV], first_tile + 8 + (lane >> 2)) + 2 * (lane & 3);
    const float4 cs = __ldg(reinterpret_cast<const float4*>(p.rope + (size_t)pos * 128) + lane);
    uint32_t lo0, lo1, hi0, hi1;
    unsigned polls = 0;
    unsigned long long t0 = 0;
    for (;;) {
        asm volatile("ld.volatile.global.v2.u32 {%0,%1}, [%2];" : "=r"(lo0), "=r"(lo1) : "l"(src) : "memory");
        asm volatile("ld.volatile.global.v2.u32 {%0,%1}, [%2];" : "=r"(hi0), "=r"(hi1) : "l"(src_hi) : "memory");
        if ((((lo0 ^ want) | (lo1 ^ want) | (hi0 ^ want) | (hi1 ^ want)) >> 16) == 0 || !keep_polling(polls, t0, p.status, p.wait_ns, where)) break;
    }
    auto f = [](uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v & 0xFFFFu))); };
    const float a0 = f(lo0), a1 = f(lo1), b0 = f(hi0), b1 = f(hi1);
    reinterpret_cast<__half2*>(dst)[lane] = __floats2half2_rn(a0 * cs.x - b0 * cs.y, a1 * cs.z - b1 * cs.w);
    reinterpret_cast<__half2*>(dst + 64)[lane] = __floats2half2_rn(a0 * cs.y + b0 * cs.x, a1 * cs.w + b1 * cs.z);
}

// ------------------------------------------------------------------------------------------------------------
// The kernel
// ------------------------------------------------------------------------------------------------------------
// kFar: the table of addresses stays in global memory (so many layers that it would leave the rings too little).
// kMany: several positions in one launch (a form of its own: with the loop around it a single position took 1 us longer).
template <bool kFar, bool kMany>
__global__ void __launch_bounds__(kThreads, 1) fused_token_kernel(const __grid_constant__ FParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full_bar[kW * kMaxDepth];
    __shared__ Requests requests[kW];
    __shared__ int behind[kMany ? kW : 1];
    __shared__ float ssq[(kMaxDim + 255) / 256];
    __shared__ __align__(16) __half new_row[3][128];   // this position's rotated query, rotated key and value of the head at hand
    __shared__ float sm_m[kW], sm_l[kW];
    __shared__ int next_id[2];         // kMany: tokens of the positions with an even and an odd number behind them (CTAs that embed)
    __shared__ int sm_i[kW];

    uint4* const xs = reinterpret_cast<uint4*>(smem + p.x_off);               // residual stream (fp16); the classifier's input
    float* const part_a = reinterpret_cast<float*>(smem + p.part_a_off);
    float* const part_b = reinterpret_cast<float*>(smem + p.part_b_off);
    const void* const* const table = kFar ? p.table : reinterpret_cast<const void* const*>(smem + p.table_off);
    const uint8_t* const* const streams = reinterpret_cast<const uint8_t* const*>(table);
    const __half* const* const norms = reinterpret_cast<const __half* const*>(table + K_KINDS * p.n_layers);

    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int cta = blockIdx.x, grid = gridDim.x;

    if (tid < kW * kMaxDepth) mbar_init(&full_bar[tid], 1);
    if (!kFar) {
        const void** const to = reinterpret_cast<const void**>(smem + p.table_off);
        for (int i = tid; i < K_KINDS * p.n_layers; i += kThreads) to[i] = p.stream[i % K_KINDS][i / K_KINDS];
        for (int i = tid; i < 2 * p.n_layers; i += kThreads) to[K_KINDS * p.n_layers + i] = p.norms[i & 1][i >> 1];
    }
    mbar_init_fence();
    __syncthreads();

    Ring ring;
    ring.base = smem + (size_t)w * p.depth * kChunkBytes;
    ring.bar = full_bar + w * kMaxDepth;
    ring.rq = requests + w;
    ring.more = behind + (kMany ? w : 0);
    ring.slot = 0;
    ring.parity = 0;
    ring.dead = false;
    if (lane == 0) {
        Requests& r = requests[w];
        r.seg = r.rot = 0;
        r.row = cta * kW + w;
        if (kMany) *ring.more = p.n_tokens - 1;
        next_segment<kMany>(r, ring.more, p, streams);
        for (int i = 0; i < p.depth; i++) ring_request<kMany>(ring, i, p, streams);
    }
    __syncwarp();

    uint8_t* const scr = smem + p.scr_off + w * kPairScratch;
    int pos = *p.pos_dev;
    unsigned nbar = 0, tag0 = p.tag_base;
    int token_pos = 0;
    const bool embeds = cta * kThreads < p.dim / 8;      // (the grid has more threads than the longest x has words)

    const int n_tokens = kMany ? p.n_tokens : 1;
    for (int more = n_tokens - 1;; more--) {
    // ---- embedding: copy_embedding_kernel (gpu_kernels.h:61-69); the token id comes from the pinned host mailbox ----
    TRACE(0, 0);
    int rot = 0;
    const int word = cta * kThreads + tid;
    if (word < p.dim / 8 && !(kMany && (Q4_DBG(p) & 2) && more < n_tokens - 1)) {
        const int token = more == n_tokens - 1 ? p.tokens_pinned[pos] : next_id[more & 1];
        const uint4 v = reinterpret_cast<const uint4*>(p.emb + (size_t)token * p.dim)[word];
        const uint32_t tg = tag_of(tag0, 0);
        // every rank files the row as slot 0 of its own buffer 1 and zeros as the other ranks' partials
        uint32_t* dst = p.xb[1][p.rank] + exchange_at(p.kind[K_DOWN], word);
        st_tagged4(dst, make_uint4(tg | (v.x & 0xFFFFu), tg | (v.x >> 16), tg | (v.y & 0xFFFFu), tg | (v.y >> 16)));
        st_tagged4(dst + 4, make_uint4(tg | (v.z & 0xFFFFu), tg | (v.z >> 16), tg | (v.w & 0xFFFFu), tg | (v.w >> 16)));
        for (int r = 1; r < p.g; r++) {
            st_tagged4(dst + (size_t)r * kLLMaxDim, make_uint4(tg, tg, tg, tg));
            st_tagged4(dst + (size_t)r * kLLMaxDim + 4, make_uint4(tg, tg, tg, tg));
        }
    }

    for (int seg = 0; seg < K_KINDS * p.n_layers; seg++) {
        const int layer = seg / K_KINDS, f = seg % K_KINDS;
        const int pi0 = 1 + layer * kLayerPhases;
        const long long loff = layer * p.layer_stride;
        // The next position's token, from host memory, while nobody waits for it. (The word is not the one the embedding above reads: with one
        // layer there is no barrier between the two.)
        if (kMany && more > 0 && seg == K_KINDS * (p.n_layers - 1) && embeds && tid == 0)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&next_id[~more & 1])), "l"(p.tokens_pinned + pos + 1) : "memory");

        if (f == K_O && !(Q4_DBG(p) & 1)) {
            // ---- attention of one query per head over positions 0..pos, split over CTAs (llama2_q4.cu:410-427) ----
            // 8 lanes per position, 16 dims each, eight of either half of the head: a load of the lane group is 128 bytes in a row (16
            // consecutive dims per lane are every second 16 bytes twice, twice the sectors from L2: 9.3 us of a layer at position 1800,
            // 6.4 so); two positions per lane group and step, the next step's keys and values each requested as soon as this step's
            // have been used.
            const int pi = pi0 + LP_ATTN;
            TRACE(pi, 0);
            float* sm_acc = part_a;                              // [kW][128]; the QKV sums in it are done with after the barrier below
            const int d0 = (tid & 7) * 8, d1 = d0 + 64, grp = tid >> 3;
            const int T = pos + 1;
            const float alpha = (float)(1.0 / sqrt(128.0));
            const int ns = attn_splits_for(p, T);
            const int nitems = p.n_heads * ns;
            const uint32_t want = tag_of(tag0, pi0 + LP_QKV), out_tag = tag_of(tag0, pi);
            const __half* kc = p.kc + loff;
            const __half* vc = p.vc + loff;
            for (int id = cta; id < nitems; id += grid) {
                const int h = id / ns, split = id % ns;
                const int kvh = h / p.kv_mul;
                const int units = (T + 31) / 32;
                const int t0 = (int)((long long)units * split / ns) * 32, t1 = min((int)((long long)units * (split + 1) / ns) * 32, T);
                const size_t col = (size_t)kvh * 128 + d0;
                constexpr int kStep = 2 * (kThreads / 8);
                uint4 k[2][2], v[2][2];
                // rows past the split's end read its first row, and are not counted; the new position's rows come from new_row
                auto row_of = [&](int t) { return t < t1 ? t : t0; };
                auto fetch = [&](uint4 (&r)[2][2], const __half* cache, int tb) {
                    if (tb >= t1) return;
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int t = row_of(tb + grp + u * (kThreads / 8));
                        if (t != pos) {
                            const uint4* src = reinterpret_cast<const uint4*>(cache + (size_t)t * p.kv_n + col);
                            r[u][0] = __ldcg(src); r[u][1] = __ldcg(src + 8);
                        }
                    }
                };
                fetch(k, kc, t0);   // requested before the wait for the query
                fetch(v, vc, t0);
                if (w == 0) {
                    rotate_head(p, h * 16, want, pos, new_row[0], lane, 0x20000 + pi);
                } else if (split == ns - 1 && w == 1) {
                    rotate_head(p, p.q_n / 8 + kvh * 16, want, pos, new_row[1], lane, 0x30000 + pi);
                    __syncwarp();
                    if (h % p.kv_mul == 0)   // the head group's first query head files the rotated key for later tokens
                        reinterpret_cast<uint2*>(p.kc + loff + (size_t)pos * p.kv_n + (size_t)kvh * 128)[lane] = reinterpret_cast<const uint2*>(new_row[1])[lane];
                } else if (split == ns - 1 && w == 2) {
                    const uint4* src = reinterpret_cast<const uint4*>(p.qkv + exchange_at(p.kind[K_QKV], (p.q_n + p.kv_n) / 8 + kvh * 16 + (lane >> 1)) + 4 * (lane & 1));
                    uint4 v;
                    unsigned polls = 0;
                    unsigned long long tw = 0;
                    for (;;) {
                        v = ld_poll(src);
                        if ((((v.x ^ want) | (v.y ^ want) | (v.z ^ want) | (v.w ^ want)) >> 16) == 0 || !keep_polling(polls, tw, p.status, p.wait_ns, 0x38000 + pi)) break;
                    }
                    reinterpret_cast<uint2*>(new_row[2])[lane] = make_uint2(prmt(v.x, v.y, 0x5410), prmt(v.z, v.w, 0x5410));
                }
                __syncthreads();
                TRACE(pi, 1);
                uint4 qh[2];
                qh[0] = *reinterpret_cast<const uint4*>(&new_row[0][d0]);
                qh[1] = *reinterpret_cast<const uint4*>(&new_row[0][d1]);
                float m = -CUDART_INF_F, l = 0.f, acc[16];
#pragma unroll
                for (int j = 0; j < 16; j++) acc[j] = 0.f;
                for (int tb = t0; tb < t1; tb += kStep) {
                    const int ta = tb + grp, tz = ta + kThreads / 8;
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        if (row_of(u ? tz : ta) == pos) {
                            k[u][0] = *reinterpret_cast<const uint4*>(&new_row[1][d0]); k[u][1] = *reinterpret_cast<const uint4*>(&new_row[1][d1]);
                            v[u][0] = *reinterpret_cast<const uint4*>(&new_row[2][d0]); v[u][1] = *reinterpret_cast<const uint4*>(&new_row[2][d1]);
                        }
                    }
                    float s0 = dot16(k[0], qh), s1 = dot16(k[1], qh);
                    fetch(k, kc, tb + kStep);   // each into the registers just read
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) {
                        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
                    }
                    if (ta < t1) {   // (then the second position may still be past the end)
                        s0 = __half2float(__float2half(s0 * alpha));  // scores are fp16 in the reference (gpu_kernels.h:171-175)
                        s1 = __half2float(__float2half(s1 * alpha));
                        const bool two = tz < t1;
                        const float mn = fmaxf(m, two ? fmaxf(s0, s1) : s0);
                        const float corr = expf(m - mn), p0 = expf(s0 - mn), p1 = two ? expf(s1 - mn) : 0.f;
                        l = l * corr + p0;
                        l += p1;
                        const __half2 *v0 = reinterpret_cast<const __half2*>(v[0]), *v1 = reinterpret_cast<const __half2*>(v[1]);
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const float2 a = __half22float2(v0[j]);
                            acc[2 * j] = fmaf(p0, a.x, acc[2 * j] * corr);
                            acc[2 * j + 1] = fmaf(p0, a.y, acc[2 * j + 1] * corr);
                        }
                        if (two) {
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                const float2 a = __half22float2(v1[j]);
                                acc[2 * j] = fmaf(p1, a.x, acc[2 * j]);
                                acc[2 * j + 1] = fmaf(p1, a.y, acc[2 * j + 1]);
                            }
                        }
                        m = mn;
                    }
                    fetch(v, vc, tb + kStep);
                }
                // merge the lane groups of this CTA: the four of each warp (lanes 8 and 16 apart) in registers, then the warps through
                // shared memory; the splits of a head are merged by the o projection while it stages its input
#pragma unroll
                for (int o = 8; o <= 16; o <<= 1) {
                    const float mo = __shfl_xor_sync(0xffffffffu, m, o), lo2 = __shfl_xor_sync(0xffffffffu, l, o);
                    const float mn = fmaxf(m, mo);
                    const float ca = m == -CUDART_INF_F ? 0.f : __expf(m - mn), cb = mo == -CUDART_INF_F ? 0.f : __expf(mo - mn);
                    l = l * ca + lo2 * cb;
#pragma unroll
                    for (int j = 0; j < 16; j++) acc[j] = acc[j] * ca + __shfl_xor_sync(0xffffffffu, acc[j], o) * cb;
                    m = mn;
                }
                if (lane == 0) { sm_m[w] = m; sm_l[w] = l; }
                if (lane < 8) {
#pragma unroll
                    for (int j = 0; j < 4; j++) *reinterpret_cast<float4*>(sm_acc + w * 128 + (j < 2 ? d0 : d1) + 4 * (j & 1)) = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
                }
                __syncthreads();
                // Slot (h, split) of a fixed [heads][nsplit] layout. The CTA that writes a head's last split in use also stamps
                // the head's unused slots with this launch's tag: every slot is rewritten by every launch, so a slot that
                // comes into use when the context grows never holds a tag from thousands of launches ago that could equal
                // (modulo 2^16) the tag its first reader waits for.
                uint32_t* outp = p.attn_part + ((size_t)h * p.nsplit + split) * kAttnPartStride;
                if (tid < 128) {
                    float M = -CUDART_INF_F;
#pragma unroll
                    for (int i = 0; i < kW; i++) M = fmaxf(M, sm_m[i]);
                    float a = 0.f, L = 0.f;
#pragma unroll
                    for (int i = 0; i < kW; i++) {
                        if (sm_m[i] != -CUDART_INF_F) {
                            const float e = __expf(sm_m[i] - M);
                            a += sm_acc[i * 128 + tid] * e;
                            L += sm_l[i] * e;
                        }
                    }
                    // the split's own softmax-weighted V average (|.| <= max |V|, safe in fp16) plus its (max, sum)
                    st_tagged(outp + tid, tagged(__float2half(L > 0.f ? a / L : 0.f), out_tag));
                    if (tid == 0) {
                        const uint32_t mb = __float_as_uint(M), lb = __float_as_uint(L);
                        st_tagged4(outp + 128, make_uint4(out_tag | (mb & 0xFFFFu), out_tag | (mb >> 16), out_tag | (lb & 0xFFFFu), out_tag | (lb >> 16)));
                    }
                }
                if (split == ns - 1 && tid >= 128 && tid < 128 + kAttnPart)
                    for (int s2 = ns; s2 < p.nsplit; s2++) st_tagged(p.attn_part + ((size_t)h * p.nsplit + s2) * kAttnPartStride + tid - 128, out_tag);
                if (id + grid < nitems) __syncthreads();   // the merge buffers are reused by this CTA's next item
            }
            TRACE(pi, 3);
        }

        // ---- one matrix step: QKV (+ RMSNorm), O (+ residual), gate/up (+ RMSNorm, SiLU) or down (+ residual) ----
        const int pi = pi0 + (f == K_QKV ? LP_QKV : f == K_O ? LP_O : f == K_GU ? LP_GU : LP_DOWN);
        TRACE(pi, 0);
        const FKind& kd = p.kind[f];
        const Share s = share_of(kd, rot, cta, grid, w);
        rot = next_rot(kd, rot, grid);
        float* const part = (f == K_QKV || f == K_GU) ? part_a : part_b;   // alternate: a warp that is ahead never writes what others still sum
        const bool norm = f == K_QKV || f == K_GU;
        int pair = s.tiles ? s.i0 / s.tiles : 0, tile = s.i0 - pair * s.tiles, left = s.i1 - s.i0;
        float* const col = part + w * 8 + (lane >> 2);         // this warp's sums of the lane's column: [tile]
        if (left < s.tiles || tile > 0) {   // the first pair does not reach every tile
            for (int i = lane; i < s.tiles * 8; i += 32) part[(i >> 3) * kTileStride + w * 8 + (i & 7)] = 0.f;
            __syncwarp();
        }
        float inv_rms = 0.f;
        const __half* nw = nullptr;
        uint4 nwv = make_uint4(0, 0, 0, 0);    // norm weights of the next pair to be staged
        if (norm) {
            nw = norms[2 * layer + (f == K_GU)];
            if (left > 0 && (pair * 32 + lane) * 8 < kd.K) nwv = __ldg(reinterpret_cast<const uint4*>(nw) + pair * 32 + lane);
            if (!(Q4_DBG(p) & 1)) inv_rms = stage_residual(p, f == K_QKV ? 1 : 0, tag_of(tag0, f == K_QKV ? pi - 1 : pi0 + LP_O), xs, ssq, w, lane, 0x60000 + pi);
        }
        TRACE(pi, 4);
        Tagged8 ahead;           // down: the next pair's words, requested while this one is worked on
        ahead.a = ahead.b = make_uint4(0, 0, 0, 0);
        bool first = true;
        int sub = 0;
        const uint8_t* chunk = nullptr;
        while (left > 0) {
            // ---- one pair: its activations into registers ----
            int n = min(left, s.tiles - tile);
            PairX px;
            if (!(Q4_DBG(p) & 1)) {
                const int wd = pair * 32 + lane;
                const bool valid = wd * 8 < kd.K, more = left > n && (wd + 32) * 8 < kd.K;
                uint4 hv = make_uint4(0, 0, 0, 0);
                unsigned polls = 0;
                unsigned long long t0 = 0;
                if (norm) {
                    if (valid) hv = norm_word(xs[wd], nwv, inv_rms);
                    if (more) nwv = __ldg(reinterpret_cast<const uint4*>(nw) + wd + 32);
                } else if (f == K_O) {
                    const int ns = attn_splits_for(p, pos + 1);
                    AttnWord aw;
                    for (;;) {   // this poll is the op boundary between the attention phase and the o projection
                        uint32_t bad = 0;
                        attn_word_load(aw, p, ns, wd, valid, tag_of(tag0, pi - 1), bad);
                        if (bad == 0 || !keep_polling(polls, t0, p.status, p.wait_ns, 0x80000 + pi)) break;
                    }
                    if (valid) hv = attn_word_merge(aw);
                } else {
                    const uint32_t want = tag_of(tag0, pi - 1);
                    auto load = [&](int word) {   // 8 elements: two tiles of the gate/up step
                        ahead.a = ld_poll(reinterpret_cast<const uint4*>(p.hb + exchange_at(p.kind[K_GU], 2 * word)));
                        ahead.b = ld_poll(reinterpret_cast<const uint4*>(p.hb + exchange_at(p.kind[K_GU], 2 * word + 1)));
                    };
                    if (valid) {
                        if (first) load(wd);
                        while (tag_mismatch(ahead, want) && keep_polling(polls, t0, p.status, p.wait_ns, 0x100 + pi)) load(wd);
                        hv = tagged_values(ahead);
                    }
                    if (more) load(wd + 32);
                }
                __syncwarp();
                if (first) TRACE(pi, 5);
                quant_pair(hv, scr, lane, px);
                if (first) TRACE(pi, 1);
            }
            // ---- its n items, two at a time; a tile's later pairs add to the first one's ----
            left -= n;
            float* dst = col + tile * kTileStride;
            auto one = [&]() {
                if (sub == 0) chunk = ring_wait(ring, p);
                float y = 0.f;
                if (!(Q4_DBG(p) & 1)) {
                    Item it;
                    int c[4];
                    item_load(it, chunk + sub * kItemBytes, lane);
                    pair_mma(c, it.a, it.b, px);
                    y = quad_sum(pair_share(c, it.meta, px, lane));
                }
                if ((lane & 3) == 0) *dst = first ? y : *dst + y;
                dst += kTileStride;
                sub ^= 1;
                if (sub == 0 || left + n == 1) ring_release<kMany>(ring, p, streams);
                n--;
            };
            if (sub) one();
            if (n > 1) {
                float* dst2 = dst + (lane & 1) * kTileStride;
                const int chunks = n >> 1;
                for (int i = 0; i < chunks; i++) {
                    chunk = ring_wait(ring, p);
                    if (!(Q4_DBG(p) & 1)) {
                        Item i0, i1;
                        int c0[4], c1[4];
                        item_load(i0, chunk, lane);
                        item_load(i1, chunk + kItemBytes, lane);
                        pair_mma(c0, i0.a, i0.b, px);
                        pair_mma(c1, i1.a, i1.b, px);
                        const float y = quad_sum2(pair_share(c0, i0.meta, px, lane), pair_share(c1, i1.meta, px, lane), lane);
                        if ((lane & 2) == 0) *dst2 = first ? y : *dst2 + y;
                        dst2 += 2 * kTileStride;
                    }
                    ring_release<kMany>(ring, p, streams);
                }
                dst += 2 * chunks * kTileStride;
                n -= 2 * chunks;
            }
            if (n) one();
            tile = 0;
            pair++;
            first = false;
        }
        __syncthreads();
        TRACE(pi, 2);
        // ---- sums over the warps (in warp order) and outputs: thread 8 * tile + row ----
        const uint32_t out_tag = tag_of(tag0, pi);
        const int out_at = s.run * kd.xstride;     // this CTA's lines of the output vector
        for (int e0 = w * 32; e0 < s.tiles * 8; e0 += kThreads) {
            const int e = e0 + lane, r = e & 7, t = s.t0 + (e >> 3);
            const bool on = e < s.tiles * 8;
            float sum = 0.f;
            if (on) {
                const float* q = part + (e >> 3) * kTileStride + r;
                float a[4];
#pragma unroll
                for (int i = 0; i < 4; i++) a[i] = ((q[i * 32] + q[i * 32 + 8]) + q[i * 32 + 16]) + q[i * 32 + 24];
                sum = ((a[0] + a[1]) + a[2]) + a[3];
            }
            if (f == K_GU) {
                const float up = __shfl_xor_sync(0xffffffffu, sum, 1);
                if (on && !(r & 1)) st_tagged(p.hb + out_at + (e >> 1), tagged(__float2half(silu_mul(sum, up)), out_tag));
            } else if (on && f == K_QKV) {
                const int n = t * 8 + r;
                const __half hv = __float2half(sum);
                st_tagged(p.qkv + out_at + e, tagged(hv, out_tag));
                const int nv = n - p.q_n - p.kv_n;
                if (nv >= 0) p.vc[loff + (long long)pos * p.kv_n + nv] = hv;   // V row into the cache for later tokens
            } else if (on) {
                // Residual: old x is what this CTA staged for the norm before (xs). A word of xs is replaced only when all of its pair's
                // new values have arrived, this one among them, so it cannot be overtaken by a warp that is a phase ahead.
                const int n = t * 8 + r;
                const float old = __half2float(reinterpret_cast<const __half*>(xs)[n]);
                sum += p.g == 1 ? old : old / p.gpu_count;   // each rank adds x / g (gpu_kernels.h:237-238)
                const uint32_t word = tagged(__float2half(sum), out_tag);
                const int xb = f == K_DOWN ? 1 : 0;
                if (Q4_DBG(p) & 16) {
                    // measurement only: the same stores, but all into this rank's own area (zeros as the peers'
                    // partials), so that no step waits on NVLink: step time minus this = exposed exchange time
                    for (int r2 = 0; r2 < p.g; r2++) st_tagged(p.xb[xb][p.rank] + (size_t)r2 * kLLMaxDim + out_at + e, r2 == p.rank ? word : out_tag);
                } else {
                    for (int peer = 0; peer < p.g; peer++) st_tagged(p.xb[xb][peer] + (size_t)p.rank * kLLMaxDim + out_at + e, word);
                }
            }
        }
        TRACE(pi, 3);
        if (kd.barrier_after) grid_barrier(p, nbar);
    }

    // ---- classifier: fp16 rows streamed through the same rings, one warp per row; per-CTA argmax candidate ----
    {
        const int pi = p.nphases - 2;
        TRACE(pi, 0);
        const int nwords = p.dim >> 3;
        // Host memory: read at the hand-off it was two to three microseconds of every token (four 7B layers 149 -> 146 us per position).
        if (cta == 0 && tid == 0) token_pos = *p.pos_pinned;
        if (!(Q4_DBG(p) & 1)) {
            const float inv_rms = stage_residual(p, 1, tag_of(tag0, pi - 1), xs, ssq, w, lane, 0x60000 + pi);
            for (int i = tid; i < nwords; i += kThreads) xs[i] = norm_word(xs[i], __ldg(reinterpret_cast<const uint4*>(p.rms_final) + i), inv_rms);
        }
        if (kMany) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (kMany && more > 0 && word < p.dim / 8) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint4*>(p.emb + (size_t)next_id[~more & 1] * p.dim) + word));
        TRACE(pi, 1);
        float best = -CUDART_INF_F;
        int bi = 0x7fffffff;
        for (int row = cta * kW + w; row < p.v_n; row += grid * kW) {
            float a[8];
#pragma unroll
            for (int j = 0; j < 8; j++) a[j] = 0.f;
            for (int w0 = 0; w0 < nwords && !ring.dead; w0 += kClsChunk / 8) {
                const uint4* wv = reinterpret_cast<const uint4*>(ring_wait(ring, p));
                if (ring.dead) break;
#pragma unroll
                for (int u = 0; u < kClsChunk / 256; u++) {
                    const int i = u * 32 + lane;
                    if (w0 + i < nwords) {
                        const uint4 wr = wv[i], xr = xs[w0 + i];
                        const __half *wh = reinterpret_cast<const __half*>(&wr), *xh = reinterpret_cast<const __half*>(&xr);
#pragma unroll
                        for (int j = 0; j < 8; j++) a[j] = fma_mixed(wh[j], xh[j], a[j]);
                    }
                }
                // The vote needs every lane's a[0], and that every one of its loads of the chunk; no product leaves this NaN's bits.
                if (!__all_sync(0xffffffffu, __float_as_uint(a[0]) != 0x7F800001u)) break;
                ring_release<kMany>(ring, p, streams);
            }
            const float sum = warp_sum(((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7])));
            const int n = p.vocab_off + row;   // global vocabulary index
            const __half hv = __float2half(sum);
            if (lane == 0) {
                if (p.g == 1) p.logits[n] = hv;
                else   // the all-gather of the logits: this rank's slice goes to every rank (plain peer stores)
                    for (int peer = 0; peer < p.g; peer++) p.ll_logits[(Q4_DBG(p) & 16) ? p.rank : peer][n] = __half_as_ushort(hv);
            }
            const float v = __half2float(hv);
            if (v > best || (v == best && n < bi)) { best = v; bi = n; }
        }
        if (lane == 0) { sm_m[w] = best; sm_i[w] = bi; }
        __syncthreads();
        if (tid == 0) {
            for (int i = 1; i < kW; i++)
                if (sm_m[i] > best || (sm_m[i] == best && sm_i[i] < bi)) { best = sm_m[i]; bi = sm_i[i]; }
            p.cand_val[cta] = best;
            p.cand_idx[cta] = bi;
        }
        TRACE(pi, 2);
        // (A further position's embedding and its attention's reads of the cache are behind this barrier, as they are behind the launch else.)
        grid_barrier(p, nbar);
        TRACE(pi, 3);
    }
    if (!kMany || more == 0) break;
    pos++;
    tag0 += (unsigned)p.nphases;
    }
    if (ring.dead) {   // before the CTA's shared memory goes: every requested copy must have landed (bounded; the last slots may hold none)
        for (int n = p.depth; n > 0; n--) {
            const unsigned long long t0 = global_ns();
            while (!mbar_try(&ring.bar[ring.slot], ring.parity))
                if (global_ns() - t0 > 20ULL * 1000 * 1000) break;   // 20 ms: far beyond any copy's flight time
            if (++ring.slot == p.depth) { ring.slot = 0; ring.parity ^= 1u; }
        }
    }

    // ---- greedy hand-off (gpu_kernels.h:456-501): lowest index among equal maxima ----
    {
        const int pi = p.nphases - 1;
        TRACE(pi, 0);
        if (cta == 0 && w == 0) {
            float best = -CUDART_INF_F;
            int bi = 0x7fffffff;
            for (int c = lane; c < grid; c += 32) {
                const float ov = __ldcg(p.cand_val + c);
                const int oi = __ldcg(p.cand_idx + c);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            if (p.g > 1) {
                // Exchange of the ranks' candidates: two tagged 64-bit words per rank, stored into every rank's
                // mailbox. The system-scope fence orders this rank's logits slice (stored by all its CTAs before
                // the grid barrier above) before the candidate, so a rank that holds all candidates also holds all
                // logits. Every rank picks the same winner (highest value, lowest index).
                const unsigned long long tg = (unsigned long long)(tag_of(tag0, pi) >> 16) << 32;
                const size_t slot = ((size_t)p.launch_parity * Q4_MAX_GPUS + p.rank) * 2;
                if (lane == 0) {
                    __threadfence_system();
                    for (int peer = 0; peer < p.g; peer++) {
                        // (debug 16: into this rank's own mailbox, once per rank slot)
                        unsigned long long* dst = (Q4_DBG(p) & 16) ? p.cand[p.rank] + ((size_t)p.launch_parity * Q4_MAX_GPUS + peer) * 2 : p.cand[peer] + slot;
                        asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(dst), "l"(tg | __float_as_uint(best)) : "memory");
                        asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(dst + 1), "l"(tg | (unsigned)bi) : "memory");
                    }
                }
                best = -CUDART_INF_F;
                bi = 0x7fffffff;
                if (lane < p.g) {
                    const unsigned long long* src = p.cand[p.rank] + ((size_t)p.launch_parity * Q4_MAX_GPUS + lane) * 2;
                    unsigned long long w0, w1;
                    unsigned polls = 0;
                    unsigned long long t0 = 0;
                    for (;;) {
                        asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(w0) : "l"(src) : "memory");
                        asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(w1) : "l"(src + 1) : "memory");
                        if (((w0 ^ tg) >> 32) == 0 && ((w1 ^ tg) >> 32) == 0) { best = __uint_as_float((unsigned)w0); bi = (int)(unsigned)w1; break; }
                        if (!keep_polling(polls, t0, p.status, p.wait_ns, 0x70000 + lane)) break;
                    }
                }
                __threadfence_system();
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
                }
            }
            if (lane == 0 && (!p.no_handoff || kMany)) {
                token_pos += n_tokens - (p.no_handoff ? 1 : 0);     // (a sampling kernel steps past the last position itself)
                if (p.write_token && !p.no_handoff) p.tokens_pinned[token_pos] = (bi == 0x7fffffff) ? 0 : bi;
                *p.pos_pinned = token_pos;
                *p.pos_dev = token_pos;
            }
        }
        if (cta == 0 && p.g > 1) {
            // all candidates are in, hence all logits slices: copy the gathered vector where the host reads it
            __syncthreads();
            const uint4* src = reinterpret_cast<const uint4*>(p.ll_logits[p.rank]);
            uint4* dst = reinterpret_cast<uint4*>(p.logits);
            for (int i = tid; i < p.vocab_size / 8; i += kThreads) dst[i] = __ldcg(src + i);
            for (int i = (p.vocab_size / 8) * 8 + tid; i < p.vocab_size; i += kThreads)
                p.logits[i] = __ushort_as_half(__ldcg(p.ll_logits[p.rank] + i));
        }
    }
}

// ------------------------------------------------------------------------------------------------------------
// Stream-layout builder (device): one block of 64 threads per (tile, pair) item.
// ------------------------------------------------------------------------------------------------------------
struct RepackMat { const uint32_t* w; const uint32_t* z; const __half* s; int tile0; };   // tile0: first tile of the matrix in the step
struct RepackArgs {
    RepackMat m[3];
    int nmat, alternate;    // alternate: rows of a tile belong to matrices 0 and 1 in turn (gate, up)
    int PW, PZ, G, rot, grid;
    FKind kind;
};
__global__ void repack_kernel(uint8_t* dst, const RepackArgs a) {
    const int pr = blockIdx.x, t = blockIdx.y, th = threadIdx.x;
    const int longs = a.kind.nt_mod * (a.kind.nt_div + 1);
    const int run = t < longs ? t / (a.kind.nt_div + 1) : a.kind.nt_mod + (t - longs) / a.kind.nt_div;
    const int cta = (run + a.rot) % a.grid;
    const Share s = share_of(a.kind, a.rot, cta, a.grid, 0);
    const int n = s.tiles * a.kind.P, idx = pr * s.tiles + t - s.t0;
    const int w = (kW * (idx + 1) - 1) / n;           // the warp whose run [w n / kW, (w + 1) n / kW) holds idx
    const int j = idx - (w * n) / kW;
    uint8_t* item = dst + ((size_t)(j >> 1) * a.grid * kW + (size_t)cta * kW + w) * kChunkBytes + (j & 1) * kItemBytes;
    auto row = [&](int c, int& mi) {
        mi = 0;
        if (a.alternate) { mi = c & 1; return t * 4 + (c >> 1); }
        for (int i = 1; i < a.nmat; i++)
            if (t >= a.m[i].tile0) mi = i;
        return (t - a.m[mi].tile0) * 8 + c;
    };
    // a row of the item is 128 contiguous bytes: in by 16 bytes a thread, out in operand order
    __shared__ uint32_t sw[8][33];
    {
        const int c = th >> 3, word = pr * 32 + (th & 7) * 4;
        int mi;
        const size_t r = row(c, mi);
        const uint4 v = word < a.PW ? *reinterpret_cast<const uint4*>(a.m[mi].w + r * a.PW + word) : make_uint4(0, 0, 0, 0);
        uint32_t* d = &sw[c][(th & 7) * 4];
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    }
    __syncthreads();
    {   // (group A, h), (group B, h), (group A, h + 1), (group B, h + 1)
        const uint32_t* d = &sw[(th & 31) >> 2][8 * (th >> 5) + (th & 3)];
        reinterpret_cast<uint4*>(item)[th] = make_uint4(d[0], d[16], d[4], d[20]);
    }
    if (th < 16) {
        const int c = th >> 1, g = 2 * pr + (th & 1);
        int mi;
        const size_t r = row(c, mi);
        uint32_t v = 0;
        if (g < a.G) v = (uint32_t)__half_as_ushort(a.m[mi].s[r * a.G + g]) | (((a.m[mi].z[r * a.PZ + (g >> 3)] >> (4 * (g & 7))) & 0xFu) << 16);
        reinterpret_cast<uint32_t*>(item + 1024)[th] = v;
    }
}

// (cos, sin) of every position and frequency, with the reference's expressions (gpu_kernels.h:346-350).
__global__ void rope_table_kernel(float2* out, int seq_len, int head_size, float theta) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int half_hs = head_size / 2;
    if (i >= seq_len * half_hs) return;
    const int pos = i / half_hs, d = i % half_hs;
    const int head_dim = (d * 2) % head_size;
    const float freq = 1.0f / powf(theta, head_dim / (float)head_size);
    const float val = pos * freq;
    out[i] = make_float2(cosf(val), sinf(val));
}

FKind make_kind(int K, int tiles, int grid, int xtile = 8) {
    FKind k;
    k.K = K;
    k.P = q4_div_up(q4_groups(K), 2);
    k.NT = tiles;
    k.nt_div = tiles / grid;
    k.nt_mod = tiles % grid;
    k.inv_long = 1.0f / (k.nt_div + 1);
    k.inv_short = k.nt_div ? 1.0f / k.nt_div : 0.f;
    k.xtile = xtile;
    k.xstride = (int)align_up((size_t)(k.nt_div + (k.nt_mod ? 1 : 0)) * xtile, 32);
    k.barrier_after = tiles < grid;
    return k;
}
int max_tiles(const FKind& k) { return k.nt_div + (k.nt_mod ? 1 : 0); }
// chunks of the warp with the longest run, over all CTAs and rotations
int max_chunks(const FKind& k) { return (q4_div_up(max_tiles(k) * k.P, kW) + 1) / 2; }
size_t stream_bytes(const FKind& k, int grid) { return (size_t)max_chunks(k) * grid * kW * kChunkBytes; }

}  // namespace

struct q4_fused {
    std::vector<void*> allocs;
    int nphases = 0;
    FParams params;
    size_t smem_bytes = 0;
    int grid = 0;
    int barriers_per_launch = 0;
    unsigned long long launches = 0;   // positions, whatever the number of launches
    bool unsupported = false;
    bool far = false;               // the table of addresses does not fit beside the rings
    void (*kernel)(FParams) = nullptr, (*kernel_many)(FParams) = nullptr;   // one position, several
    unsigned long long* trace = nullptr;
    Q4LLArea* ll_local = nullptr;   // this rank's exchange area (inside the communicator's inbox, or own allocation at g = 1)
    size_t attn_part_bytes = 0, hb_bytes = 0, qkv_bytes = 0;
    bool armed = false;             // buffers and counters are in their initial state or in step with the launches so far
    unsigned long long wait_ns = kDefaultWaitNs;
};

#ifdef Q4_TEST_BUILD
// Switches of the test build (see Q4_DBG): set through exported functions, never through the environment.
static int g_test_debug = 0, g_test_split_len = 0, g_test_depth = 0;
static bool g_test_far_table = false;
static int g_test_fail_alloc = -1;   // >= 0: the allocation with this running index fails once (host-side fault injection)
static int g_test_alloc_index = 0;
extern "C" void q4_test_set_fused_debug(int bits) { g_test_debug = bits; }
extern "C" void q4_test_set_split_len(int positions) { g_test_split_len = positions; }
extern "C" void q4_test_set_ring_depth(int chunks) { g_test_depth = chunks; }
extern "C" void q4_test_set_far_table(int on) { g_test_far_table = on != 0; }
extern "C" void q4_test_fail_fused_alloc(int index) { g_test_fail_alloc = index; g_test_alloc_index = 0; }
#endif

static int fused_alloc(q4_fused* f, void** p, size_t bytes) {
#ifdef Q4_TEST_BUILD
    if (g_test_fail_alloc >= 0 && g_test_alloc_index++ == g_test_fail_alloc) { g_test_fail_alloc = -1; return Q4_ERR_CUDA; }
#endif
    Q4_CUDA_TRY(cudaMalloc(p, bytes));
    f->allocs.push_back(*p);
    return Q4_OK;
}

// Stream-layout weights of one matrix step (see the layout at the top), `rot` as the kernel's walk has it there.
static int make_stream(q4_fused* f, const FKind& kind, int rot, const DevQW* const (&mats)[3], bool alternate, const uint8_t** out) {
    uint8_t* d = nullptr;
    if (int e = fused_alloc(f, (void**)&d, stream_bytes(kind, f->grid))) return e;
    RepackArgs a;
    memset(&a, 0, sizeof(a));
    int tile0 = 0;
    for (int i = 0; i < 3 && mats[i]; i++) {
        a.m[i] = RepackMat{mats[i]->w.weight, mats[i]->w.zeros, (const __half*)mats[i]->w.scales, tile0};
        tile0 += mats[i]->N / 8;
        a.nmat = i + 1;
    }
    a.alternate = alternate;
    a.PW = q4_pw(kind.K);
    a.PZ = q4_pz(kind.K);
    a.G = q4_groups(kind.K);
    a.rot = rot;
    a.grid = f->grid;
    a.kind = kind;
    repack_kernel<<<dim3(kind.P, kind.NT), 64>>>(d, a);
    Q4_CUDA_TRY(cudaGetLastError());
    *out = d;
    return Q4_OK;
}

void q4_fused_free(q4_model* m) {
    if (!m->fused) return;
    for (void* p : m->fused->allocs) cudaFree(p);
    delete m->fused;
    m->fused = nullptr;
}

// Called by q4_model_reset. Launch and barrier counters (and with them the activation tags) simply keep counting
// across generations; only after a recorded error is everything re-armed from zero. In a tensor-parallel group the
// ranks' tags must stay in step and a rank's exchange area is written by its peers, so after an error (as after
// q4_model_prepare) every rank has to finish its reset before any rank launches again: the callers put a host
// barrier there.
void q4_fused_reset(q4_model* m, bool clean) {
    if (!m->fused || m->fused->unsupported) return;
    q4_fused* f = m->fused;
    if (f->armed && clean) return;
    int st = 0;
    cudaDeviceSynchronize();
    if (f->armed && cudaMemcpy(&st, f->params.status, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess && st == 0) return;
    f->armed = false;
    bool ok = true;
    ok &= cudaMemset(f->params.bar_counter, 0, sizeof(unsigned long long)) == cudaSuccess;
    ok &= cudaMemset(f->params.status, 0, 4 * sizeof(int)) == cudaSuccess;
    ok &= cudaMemset(f->ll_local->x, 0, sizeof(f->ll_local->x)) == cudaSuccess;
    ok &= cudaMemset(f->ll_local->cand, 0, sizeof(f->ll_local->cand)) == cudaSuccess;
    ok &= cudaMemset(f->params.hb, 0, f->hb_bytes) == cudaSuccess;
    ok &= cudaMemset(f->params.qkv, 0, f->qkv_bytes) == cudaSuccess;
    ok &= cudaMemset(f->params.attn_part, 0, f->attn_part_bytes) == cudaSuccess;
    ok &= cudaDeviceSynchronize() == cudaSuccess;  // the memsets run on the default stream; forward calls use the caller's stream
    f->launches = 0;
    f->armed = ok;
}

const int* q4_fused_status_word(const q4_model* m) { return m->fused && !m->fused->unsupported ? m->fused->params.status : nullptr; }

// Limit of every device-side wait of the fused kernel (default two seconds); takes effect with the next launch.
void q4_fused_set_wait_limit(q4_model* m, unsigned long long ns) {
    if (m->fused && !m->fused->unsupported) m->fused->wait_ns = ns ? ns : kDefaultWaitNs;
}

int q4_fused_status(q4_model* m) {
    if (!m->fused || m->fused->unsupported) return Q4_OK;
    int st[4] = {0, 0, 0, 0};
    Q4_CUDA_TRY(cudaMemcpy(st, m->fused->params.status, sizeof(st), cudaMemcpyDeviceToHost));
    if (st[0] != 0) {
        fprintf(stderr, "q4 fused path: a bounded device-side wait ran out (status %d, location 0x%x)\n", st[0], st[1]);
    }
    return st[0];
}

static int fused_build(q4_model* m, q4_fused* f);

// Builds the fused path's state into a private object and publishes it in the model only when every step has
// succeeded. A model that the path cannot serve is remembered as such (an empty object with `unsupported` set); any
// other failure (out of memory, a CUDA error) frees what was allocated and leaves the model as it was, so that a later
// call starts from scratch instead of launching a half-built state.
int q4_fused_prepare(q4_model* m) {
    if (m->fused) return m->fused->unsupported ? Q4_ERR_UNSUPPORTED_SIZE : Q4_OK;
    q4_fused* f = new q4_fused();
    int e = fused_build(m, f);
    if (e == Q4_OK) {
        m->fused = f;
        q4_fused_reset(m);
        if (cudaDeviceSynchronize() != cudaSuccess || !f->armed) e = Q4_ERR_CUDA;
        if (e == Q4_OK) return Q4_OK;
        m->fused = nullptr;
    }
    for (void* p : f->allocs) cudaFree(p);
    f->allocs.clear();
    if (e == Q4_ERR_UNSUPPORTED_SIZE && f->unsupported) {
        m->fused = f;
        return e;
    }
    delete f;
    return e;
}

static int fused_build(q4_model* m, q4_fused* f) {
    const q4_config& c = m->cfg;
    const int g = m->g;
    if (m->column || m->head_size != 128 || (c.dim % 128) || (m->h_kc % 8) || c.dim > kMaxDim || c.dim > kLLMaxDim || c.vocab_size > kLLMaxVocab || (m->v_n % 2) || (m->kv_n % 128) || (m->q_n % 128) ||
        (g > 1 && (!m->comm || q4_comm_world(m->comm) != g || q4_comm_rank(m->comm) != m->rank))) {
        f->unsupported = true;
        return Q4_ERR_UNSUPPORTED_SIZE;
    }
    int dev = 0, sms = 0, coop = 0;
    Q4_CUDA_TRY(cudaGetDevice(&dev));
    Q4_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    Q4_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) { f->unsupported = true; return Q4_ERR_UNSUPPORTED_SIZE; }
    f->grid = sms;

    FParams& p = f->params;
    memset(&p, 0, sizeof(p));
    p.dim = c.dim;
    p.n_layers = c.n_layers;
    p.vocab_size = c.vocab_size;
    p.q_n = m->q_n;
    p.kv_n = m->kv_n;
    p.v_n = m->v_n;
    p.layer_stride = (long long)c.seq_len * m->kv_n;
    p.rms_final = (const __half*)m->rms_final;
    p.kv_mul = m->kv_mul;
    p.n_heads = c.n_heads / g;    // this rank's query heads
    p.nsplit = std::min(kMaxSplit, std::max(1, sms / p.n_heads));
    p.gpu_count = (float)g;
    p.g = g;
    p.rank = m->rank;
    p.vocab_off = m->rank * m->v_n;
    p.logits = (__half*)m->logits;
    p.kc = (__half*)m->kc; p.vc = (__half*)m->vc;
    p.emb = (const __half*)m->emb; p.wcls = (const __half*)m->wcls;
    p.pos_dev = m->pos;
    p.tokens_pinned = (int*)m->shared->tokens;
    p.pos_pinned = &m->shared->pos;
    p.kind[K_QKV] = make_kind(c.dim, (m->q_n + 2 * m->kv_n) / 8, sms);
    p.kind[K_O] = make_kind(m->o_kc, c.dim / 8, sms);
    p.kind[K_GU] = make_kind(c.dim, m->h_kc / 4, sms, 4);   // 4 gate and the same 4 up columns per tile
    p.kind[K_DOWN] = make_kind(m->h_kc, c.dim / 8, sms);
    for (const FKind& k : p.kind)
        if (q4_groups(k.K) > kMaxGroups || sms * p.kind[K_DOWN].xstride > kLLMaxDim) { f->unsupported = true; return Q4_ERR_UNSUPPORTED_SIZE; }

    int e;
#define FTRY(expr) do { e = (expr); if (e != Q4_OK) return e; } while (0)
    if (g > 1) {
        for (int r = 0; r < g; r++) {
            Q4LLArea* a = q4_comm_ll_area(m->comm, r);
            if (!a) { f->unsupported = true; return Q4_ERR_UNSUPPORTED_SIZE; }
            int peer_sms = 0;
            Q4_CUDA_TRY(cudaMemcpy(&peer_sms, &a->sms, sizeof(peer_sms), cudaMemcpyDefault));
            if (peer_sms != sms) {   // every rank finds the same difference and takes the per-op path
                fprintf(stderr, "q4 fused path: rank %d has %d SMs, rank %d has %d\n", r, peer_sms, m->rank, sms);
                f->unsupported = true;
                return Q4_ERR_UNSUPPORTED_SIZE;
            }
            p.xb[0][r] = &a->x[0][0][0];
            p.xb[1][r] = &a->x[1][0][0];
            p.cand[r] = &a->cand[0][0][0];
            p.ll_logits[r] = a->logits;
        }
        f->ll_local = q4_comm_ll_area(m->comm, m->rank);
    } else {
        FTRY(fused_alloc(f, (void**)&f->ll_local, sizeof(Q4LLArea)));
        p.xb[0][0] = &f->ll_local->x[0][0][0];
        p.xb[1][0] = &f->ll_local->x[1][0][0];
        p.cand[0] = &f->ll_local->cand[0][0][0];
        p.ll_logits[0] = f->ll_local->logits;
    }
    f->hb_bytes = 4 * (size_t)sms * p.kind[K_GU].xstride;
    f->qkv_bytes = 4 * (size_t)sms * p.kind[K_QKV].xstride;
    FTRY(fused_alloc(f, (void**)&p.hb, f->hb_bytes));
    FTRY(fused_alloc(f, (void**)&p.qkv, f->qkv_bytes));
    Q4_CUDA_TRY(cudaMemset(p.hb, 0, f->hb_bytes));
    Q4_CUDA_TRY(cudaMemset(p.qkv, 0, f->qkv_bytes));
    f->attn_part_bytes = sizeof(uint32_t) * (size_t)p.n_heads * p.nsplit * kAttnPartStride;
    FTRY(fused_alloc(f, (void**)&p.attn_part, f->attn_part_bytes));
    Q4_CUDA_TRY(cudaMemset(p.attn_part, 0, f->attn_part_bytes));
    {
        float2* rope = nullptr;
        const int n = c.seq_len * (m->head_size / 2);
        FTRY(fused_alloc(f, (void**)&rope, sizeof(float2) * (size_t)n));
        rope_table_kernel<<<q4_div_up(n, 256), 256>>>(rope, c.seq_len, m->head_size, c.rope_theta);
        Q4_CUDA_TRY(cudaGetLastError());
        p.rope = reinterpret_cast<const float*>(rope);
    }
    FTRY(fused_alloc(f, (void**)&p.cand_val, sizeof(float) * sms));
    FTRY(fused_alloc(f, (void**)&p.cand_idx, sizeof(int) * sms));
    FTRY(fused_alloc(f, (void**)&p.bar_counter, sizeof(unsigned long long)));
    FTRY(fused_alloc(f, (void**)&p.status, 4 * sizeof(int)));

    // shared memory: ring | digit scratch | x | partial sums A (or the attention's) | B | tables. The ring gets what the rest leaves.
    const int part_a = std::max(kTileStride * std::max(max_tiles(p.kind[K_QKV]), max_tiles(p.kind[K_GU])), kW * 128) * (int)sizeof(float);
    const int part_b = kTileStride * std::max(max_tiles(p.kind[K_O]), max_tiles(p.kind[K_DOWN])) * (int)sizeof(float);
    const int x_bytes = (int)align_up(2 * (size_t)c.dim, 128);
    size_t tables = align_up((size_t)(K_KINDS + 2) * c.n_layers * 8, 16);
    const size_t budget = 224 * 1024;   // + about 2 KB of static shared memory, of 227 KB per CTA
    const size_t other = (size_t)kW * kPairScratch + x_bytes + align_up(part_a, 128) + align_up(part_b, 128);
    f->far = other + tables + (size_t)kMinDepth * kW * kChunkBytes > budget;
#ifdef Q4_TEST_BUILD
    f->far |= g_test_far_table;
#endif
    if (f->far) tables = 0;
    int depth = other + tables < budget ? (int)((budget - other - tables) / (kW * kChunkBytes)) : 0;
    depth = std::min(depth, kMaxDepth);
    if (depth < kMinDepth) { f->unsupported = true; return Q4_ERR_UNSUPPORTED_SIZE; }
#ifdef Q4_TEST_BUILD
    if (g_test_depth > 0) depth = std::max(kMinDepth, std::min(depth, g_test_depth));
#endif
    p.depth = depth;
    p.scr_off = kW * depth * kChunkBytes;
    p.x_off = p.scr_off + kW * kPairScratch;
    p.part_a_off = p.x_off + x_bytes;
    p.part_b_off = p.part_a_off + (int)align_up(part_a, 128);
    p.table_off = p.part_b_off + (int)align_up(part_b, 128);
    f->smem_bytes = (size_t)p.table_off + tables;

    f->nphases = p.nphases = 1 + kLayerPhases * c.n_layers + 2;
    f->barriers_per_launch = 1;
    std::vector<const void*> streams[K_KINDS], norms[2];
    int rot = 0;
    for (int l = 0; l < c.n_layers; l++) {
        const DevLayer& L = m->layers[l];
        const DevQW* const mats[K_KINDS][3] = {{&L.q, &L.k, &L.v}, {&L.o, nullptr, nullptr}, {&L.gate, &L.up, nullptr}, {&L.down, nullptr, nullptr}};
        for (int k = 0; k < K_KINDS; k++) {
            const uint8_t* d = nullptr;
            FTRY(make_stream(f, p.kind[k], rot, mats[k], k == K_GU, &d));
            streams[k].push_back(d);
            rot = (rot + p.kind[k].nt_mod) % sms;
            f->barriers_per_launch += p.kind[k].barrier_after;
        }
        norms[0].push_back(L.rms_att);
        norms[1].push_back(L.rms_ffn);
    }
    Q4_CUDA_TRY(cudaDeviceSynchronize());  // repacks done
    auto table = [&](const void** to, const std::vector<const void*>& v) {
        void* d = nullptr;
        if (int err = fused_alloc(f, &d, v.size() * sizeof(void*))) return err;
        Q4_CUDA_TRY(cudaMemcpy(d, v.data(), v.size() * sizeof(void*), cudaMemcpyHostToDevice));
        *to = d;
        return (int)Q4_OK;
    };
    for (int k = 0; k < K_KINDS; k++) FTRY(table((const void**)&p.stream[k], streams[k]));
    for (int k = 0; k < 2; k++) FTRY(table((const void**)&p.norms[k], norms[k]));
    if (f->far) {
        std::vector<const void*> all;
        for (int l = 0; l < c.n_layers; l++)
            for (int k = 0; k < K_KINDS; k++) all.push_back(streams[k][l]);
        for (int l = 0; l < c.n_layers; l++)
            for (int k = 0; k < 2; k++) all.push_back(norms[k][l]);
        FTRY(table((const void**)&p.table, all));
    }
    f->kernel = f->far ? fused_token_kernel<true, false> : fused_token_kernel<false, false>;
    f->kernel_many = f->far ? fused_token_kernel<true, true> : fused_token_kernel<false, true>;
    // (the limit belongs to the function, not to this model: always the largest any model may need, so that a smaller one prepared
    // later does not lower it)
    Q4_CUDA_TRY(cudaFuncSetAttribute(f->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
    Q4_CUDA_TRY(cudaFuncSetAttribute(f->kernel_many, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
    int per_sm = 0, many_per_sm = 0;
    Q4_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f->kernel, kThreads, f->smem_bytes));
    Q4_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&many_per_sm, f->kernel_many, kThreads, f->smem_bytes));
    if (per_sm < 1 || many_per_sm < 1) {
        fprintf(stderr, "q4 fused path: kernel does not fit one SM (%zu B shared memory, %d threads)\n", f->smem_bytes, kThreads);
        f->unsupported = true;
        return Q4_ERR_UNSUPPORTED_SIZE;
    }
#undef FTRY
    return Q4_OK;
}

// Positions of one launch: 32 at most, and no more than about 4 ms of them, as a launch keeps every SM and another stream's kernels wait for its end. (A
// position takes about 8 us per layer beside its bytes at 5 TB/s: four 7B layers 123 us, measured 130; 7B 0.98 ms, 1.05; two 70B layers 0.20, 0.20. So four
// positions of 7B, two of 13B, one of 70B; what a launch saves, some 8 us per position, is next to nothing there.) Tags have 16 bits.
static int positions_at_once(double bytes, int n_layers) {
    const double us = bytes / 5e6 + 8.0 * n_layers;
    return std::max(1, std::min(std::min(32, (int)(4000.0 / us)), 32768 / (1 + kLayerPhases * n_layers + 2)));
}
int q4_fused_positions_at_once(const q4_model* m, int pos) { return positions_at_once(q4_model_token_bytes(m, pos), m->cfg.n_layers); }

int q4_fused_forward(q4_model* m, cudaStream_t s, int gen_token, int no_handoff, int n_tokens) {
    q4_fused* f = m->fused;
    if (!f || f->unsupported) return Q4_ERR_UNSUPPORTED_SIZE;
    if (!f->armed) return Q4_ERR_CUDA;   // the last re-arm did not complete
    FParams p = f->params;
    p.write_token = gen_token;
    p.no_handoff = no_handoff;
    p.trace = f->trace;
    p.debug = 0;
    p.split_len = kSplitLen;
    p.wait_ns = f->wait_ns;
#ifdef Q4_TEST_BUILD
    p.debug = g_test_debug & 31;
    if (g_test_split_len > 0) p.split_len = g_test_split_len;
#endif
    if (n_tokens < 1 || (n_tokens > 1 && m->g > 1)) return Q4_ERR_INVALID;
    p.n_tokens = n_tokens;
    p.bar_base = f->launches * (unsigned long long)f->barriers_per_launch;
    p.tag_base = (unsigned)((f->launches * (unsigned long long)f->nphases) & 0xFFFFu);
    p.launch_parity = (unsigned)(f->launches & 1);
    f->launches += n_tokens;
    void* args[] = {&p};
    Q4_CUDA_TRY(cudaLaunchCooperativeKernel((void*)(n_tokens > 1 ? f->kernel_many : f->kernel), dim3(f->grid), dim3(kThreads), args, f->smem_bytes, s));
    return Q4_OK;
}

#ifdef Q4_TEST_BUILD
extern "C" int q4_test_positions_at_once(double bytes, int n_layers) { return positions_at_once(bytes, n_layers); }
// Test build only: the fused path's W4 dot product (staging to block fixed point, product) on a caller's activation
// vector, outside the token kernel, so that tests can feed it vectors the model never produces on its own (outliers, empty
// groups, subnormals, the largest fp16 values). One CTA per 8-column tile; plain loads, not tuned.
namespace {
__global__ void __launch_bounds__(kThreads) test_gemv_kernel(const uint8_t* stream, const __half* x, __half* y, const FKind kind) {
    __shared__ __align__(16) uint8_t scr[kW][kPairScratch], items[kW][kItemBytes];
    __shared__ float part[kTileStride];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, grid = gridDim.x, cta = blockIdx.x;
    const Share s = share_of(kind, 0, cta, grid, w);   // one tile: items = pairs
    float acc = 0.f;
    for (int it = s.i0; it < s.i1; it++) {
        uint4 hv = make_uint4(0, 0, 0, 0);
        __half* h = reinterpret_cast<__half*>(&hv);
        for (int j = 0; j < 8; j++)
            if (it * 256 + lane * 8 + j < kind.K) h[j] = x[it * 256 + lane * 8 + j];
        PairX px;
        quant_pair(hv, scr[w], lane, px);
        const int c = it - s.i0;
        const uint4* src = reinterpret_cast<const uint4*>(stream + ((size_t)(c >> 1) * grid * kW + (size_t)cta * kW + w) * kChunkBytes + (c & 1) * kItemBytes);
        for (int i = lane; i < kItemBytes / 16; i += 32) reinterpret_cast<uint4*>(items[w])[i] = src[i];
        __syncwarp();
        Item item;
        int d[4];
        item_load(item, items[w], lane);
        pair_mma(d, item.a, item.b, px);
        acc += quad_sum(pair_share(d, item.meta, px, lane));
        __syncwarp();
    }
    if ((lane & 3) == 0) part[w * 8 + (lane >> 2)] = acc;
    __syncthreads();
    if (threadIdx.x < 8) {
        float sum = 0.f;
        for (int i = 0; i < kW; i++) sum += part[i * 8 + threadIdx.x];
        y[cta * 8 + threadIdx.x] = __float2half(sum);
    }
}
}  // namespace

extern "C" int q4_test_fused_gemv(void* stream, uint16_t* y, const uint16_t* x, const q4_qweight* w, int K, int N) {
    if (!y || !x || !w || K <= 0 || N <= 0 || (N & 7) || (K & 7)) return Q4_ERR_INVALID;
    if (q4_groups(K) > kMaxGroups) return Q4_ERR_UNSUPPORTED_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    q4_fused f;
    f.grid = N / 8;
    DevQW q;
    q.w = *w;
    q.K = K;
    q.N = N;
    const FKind kind = make_kind(K, N / 8, f.grid);
    const DevQW* const mats[3] = {&q, nullptr, nullptr};
    const uint8_t* d = nullptr;
    int e = make_stream(&f, kind, 0, mats, false, &d);
    cudaError_t ce = cudaDeviceSynchronize();   // the layout is built on the default stream
    if (e == Q4_OK && ce == cudaSuccess) {
        test_gemv_kernel<<<f.grid, kThreads, 0, s>>>(d, (const __half*)x, (__half*)y, kind);
        ce = cudaGetLastError();
        if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    }
    for (void* p : f.allocs) cudaFree(p);
    Q4_CUDA_TRY(ce);
    return e;
}
#endif  // Q4_TEST_BUILD

// Profiling hook: arms per-phase timestamps (CTA 0 and the last CTA) for the following fused launches and, when
// `out` is given, copies the last launch's stamps out. Layout [2][nphases][8] of nanoseconds (kTraceCols); also returns the
// phase types so that the caller can group them.
extern "C" int q4_model_trace(q4_model* m, unsigned long long* out, int* phase_types, int max_phases) {
    if (!m) return Q4_ERR_INVALID;
    if (int e = q4_fused_prepare(m)) return e;
    q4_fused* f = m->fused;
    const size_t n = (size_t)2 * f->nphases * kTraceCols;
    if (!f->trace) {
        if (int e = fused_alloc(f, (void**)&f->trace, n * sizeof(unsigned long long))) return e;
        Q4_CUDA_TRY(cudaMemset(f->trace, 0, n * sizeof(unsigned long long)));
    }
    Q4_CUDA_TRY(cudaDeviceSynchronize());
    if (out && phase_types && max_phases >= f->nphases) {
        Q4_CUDA_TRY(cudaMemcpy(out, f->trace, n * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
        for (int i = 0; i < f->nphases; i++) {
            const int lp = (i - 1) % kLayerPhases;
            phase_types[i] = i == 0 ? PH_EMBED * 16 : i == f->nphases - 2 ? PH_CLS * 16 : i == f->nphases - 1 ? PH_ARGMAX * 16
                           : lp == LP_ATTN ? PH_ATTN * 16 : PH_GEMV * 16 + (lp == LP_QKV ? 1 : lp == LP_GU ? 9 : 4);
        }
    }
    return f->nphases;
}
