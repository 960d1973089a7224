// AWQ W4 g128 dequantize-and-multiply for a handful of rows (1 <= M <= 16): the projections of batched decode.
//
// The reference has one sequence per process (RunState, common.h:62-78) and its mat_vec_kernel_int4 family
// (gpu_kernels.h:179-283) reads every weight once per token; with several sequences decoded together the weights are
// still read once per STEP, so the op stays bound by HBM as long as the per-weight work is small. That is what this
// kernel is built for; the tcgen05 GEMM (q4_gemm.cu) takes over from M > 16, where the contraction starts to matter.
//
// Two forms of the kernel; streamed() has the line between them and both sides' figures.
//
// Sliced: a unit is 16 * MT output features of one launch over the whole K axis; one persistent CTA (12 warps; 8 for
// 9-16 rows) per SM walks the units; a warp takes one share of a unit's 128-input groups, its own or, going round, share
// (w + u) % warps of unit u, and the shares' partial tiles are summed in the order of the shares through shared memory (fixed order:
// results are bit-reproducible, and the same either way). Inside a warp the product runs on mma.sync m16n8k16 (fp16 in, fp32 out) with
// the weights as the 16-row operand and the batch as the 8-column one. The k index of an MMA is only a summation
// label, so the packed words are used as they lie in the file: thread (g, t) of the warp loads 16 bytes = 32 inputs of
// feature rows g and g + 8 at input offset 32 t of the group, unpacks a word into the half2 pairs (q0,q4) (q1,q5)
// (q2,q6) (q3,q7) with the zero point subtracted exactly (magic-number trick, no int -> float conversion), and feeds
// them as the A fragment; the B fragment is the same eight inputs of batch row g in the same pairing. Per group the
// fp32 tile is scaled by the group's fp16 scale in fp32, as the reference does (gpu_kernels.h:222-228), so weights
// are never rounded to fp16 after scaling.
//
// Stream: a CTA of 16 warps per SM has consecutive tiles of 16 features. Each warp keeps the x fragments of its own groups (two with up to
// eight rows, one with more) in registers for all of them, and the items of the groups that are left are dealt out over the warps tile by
// tile; an item (16 features over a group, 1 KB) comes through the warp's private ring of four (cp.async; a lane reads what it has copied
// itself, so that no barrier is needed), the first ones ahead of griddepcontrol.wait. Scales and zero points of a pass of tiles lie in shared
// memory, one word for both. The warps' partial tiles wait there for one sum at the end of the pass. What bounds it: the unpack and the products
// (150 clocks of a scheduler per item where nothing else runs, about 220 here; HBM's rate is 200) and, with few tiles, the start: x of all rows goes
// to every SM, 64 KB with 8 rows of 4096. Back to back from HBM, 8 rows: gate/up of 7B 13.0 us = 3.6 TB/s (16.4 sliced), 8192 -> 10240 15.2 = 2.9 (22.0),
// 70B gate/up 64.3 = 3.8 (77.9).
//
// Epilogues: plain, residual (y = product + residual * scale: matmul(QWeight)'s accum form, gpu_kernels.h:237-238),
// and SiLU (ffn_matvec_silu_kernel, gpu_kernels.h:251-283: the CTA holds 16 gate and the same 16 up features and writes
// silu(gate) * up without rounding gate or up to fp16 first).
#include "q4_bulk.cuh"
#include "q4_model.h"

namespace {

struct SkMat {
    const uint32_t* w;
    const uint32_t* z;
    const __half* s;
    __half* y;
    int ldy;     // halfs between rows of y
    int tile0;   // first 16-feature tile of this matrix in the launch
};

struct SkParams {
    const __half* x;   // [M][K]
    int M, K, PW, PZ, G;
    int nmat;
    SkMat m[3];
    int total_tiles;
    const __half* residual;   // [M][ldy of m[0]] or null
    float rscale;
    bool late;                // dependents are signalled at the end (q4_qkv_rows_launch)
};

__device__ __forceinline__ void mma_f16(float c[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One packed word minus the zero point as four half2: (q0,q4) (q1,q5) (q2,q6) (q3,q7), exact.
// (w & 0x000F000F) | 0x6400 is the half 1024 + q; (w & 0x00F000F0) | 0x5400 is the half 64 + q (one unit of q is 16 ulps there).
__device__ __forceinline__ void unpack8(uint32_t w, uint32_t zlo, uint32_t zhi, uint32_t d[4]) {
    d[0] = h22u(__hsub2(u2h2(lop3_and_or(w, 0x000F000Fu, 0x64006400u)), u2h2(zlo)));
    d[1] = h22u(__hsub2(u2h2(lop3_and_or(w, 0x00F000F0u, 0x54005400u)), u2h2(zhi)));
    w >>= 8;
    d[2] = h22u(__hsub2(u2h2(lop3_and_or(w, 0x000F000Fu, 0x64006400u)), u2h2(zlo)));
    d[3] = h22u(__hsub2(u2h2(lop3_and_or(w, 0x00F000F0u, 0x54005400u)), u2h2(zhi)));
}

#ifndef SK_WARPS
#define SK_WARPS 12
#endif
#ifndef SK_D1
#define SK_D1 3
#endif
#ifndef SK_D2
#define SK_D2 2
#endif
#ifndef SK_D22
#define SK_D22 3
#endif
// warps of a CTA = K slices of a unit
__host__ __device__ constexpr int warps_of(int MT, int NT) { return NT == 2 ? 8 : SK_WARPS; }   // (16 batch rows need the registers of 8-warp CTAs)
// How the groups of a CTA's units are dealt to the warps, and when the partial tiles are summed:
//   FIXED      a warp keeps its share; every unit is summed behind a barrier of its own, while the other warps go on
//   ROTATING   shares go round; units are summed several at a time
// fixed_shares() tells which. Units that wait in shared memory for one sum: as many as 72 KB hold, so that L1 keeps enough for x.
enum Deal { FIXED, ROTATING };
// units whose partial tiles have a place in shared memory
__host__ __device__ constexpr int slots_of(int NT, Deal deal) { return deal == FIXED ? 2 : NT == 2 ? 4 : 6; }
// units that are summed together
__host__ __device__ constexpr int units_at_once(int NT, Deal deal) { return deal == ROTATING ? slots_of(NT, deal) : 1; }

// MT: 16-feature tiles per unit (1 or 2); NT: 8-row batch tiles (1: M <= 8, 2: M <= 16); SILU: tile 0 = gate, tile 1 = up.
// Persistent: one CTA per SM walks units blockIdx.x, blockIdx.x + gridDim.x, ...; a warp's weight loads run D groups ahead
// of its math ACROSS unit boundaries and its x fragments one group ahead (a unit gives a warp only G / kWarps groups - four
// at K = 4096 - so a pipeline that restarted per unit would spend its time on load latency, and one-unit CTAs would
// quantise the work badly over the SMs). Measured on the four 7B ops with 8 rows (us): 8 warps with 4 groups ahead
// 4.4 / 10.4 / 11.9 / 19.9; 12 warps with 2-3 ahead 4.5 / 9.4 / 10.6 / 16.6; 16 warps with 2 ahead 4.8 / 9.6 / 11.6 / 19.2.
template <int MT, int NT, bool SILU, Deal DEAL>
__global__ void __launch_bounds__(warps_of(MT, NT) * 32, 1) q4_skinny_kernel(const SkParams p) {
    constexpr int kWarps = warps_of(MT, NT);
    extern __shared__ float red_raw[];
    constexpr int kSlots = slots_of(NT, DEAL), kSum = units_at_once(NT, DEAL);
    float (*red)[kWarps][MT][NT][4][32] = reinterpret_cast<float (*)[kWarps][MT][NT][4][32]>(red_raw);   // [unit % kSlots][share]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int units = SILU ? p.total_tiles : p.total_tiles / MT;
    const int my_units = blockIdx.x < units ? (units - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    // This warp's steps (unit, group), unit by unit. The shares of a unit differ by one group (32 groups over 12 warps are 2 or 3): with a
    // fixed share per warp and a barrier per unit all wait for those with three, so there they go round.
    struct Cursor {
        int u, share, g, g_end;
        __device__ __forceinline__ void settle(int G, int n) {   // to the first unit from u on in which the share has a group
            g = G * share / kWarps;
            g_end = G * (share + 1) / kWarps;
            while (g == g_end && u < n) {
                u++;
                if (DEAL != ROTATING) continue;
                share = share + 1 == kWarps ? 0 : share + 1;
                g = G * share / kWarps;
                g_end = G * (share + 1) / kWarps;
            }
        }
        __device__ __forceinline__ void next(int G, int n) {
            if (++g < g_end) return;
            u++;
            if (DEAL != ROTATING) {
                g = G * share / kWarps;
                return;
            }
            share = share + 1 == kWarps ? 0 : share + 1;
            settle(G, n);
        }
    };
    Cursor cur = {0, warp, 0, 0};
    cur.settle(p.G, my_units);

    // rows of unit u: tile mt holds features f0 .. f0 + 15 of matrix mi
    auto unit_tile = [&](int u, int mt, int& mi, int& f0) {
        const int unit = blockIdx.x + u * gridDim.x;
        int tile;
        if (SILU) {
            mi = mt;
            tile = unit;
        } else {
            tile = unit * MT + mt;
            mi = 0;
            if (p.nmat > 1 && tile >= p.m[1].tile0) mi = 1;
            if (p.nmat > 2 && tile >= p.m[2].tile0) mi = 2;
            tile -= p.m[mi].tile0;
        }
        f0 = tile * 16;
    };

    // A step's operands per thread: 16 bytes of packed weights, the zeros word and the scale for each of its 2 MT rows.
    constexpr int D = MT == 1 ? SK_D1 : (NT == 1 ? SK_D2 : SK_D22);
    struct Stage {
        uint4 w[MT][2];
        uint32_t zw[MT][2];
        __half sc[MT][2];
    };
    Stage st[D];
    // prefetch cursor, and its unit's row pointers (row g of each tile; row g + 8 lies 8 rows further)
    Cursor pf = cur;
    const uint4* pw[MT];
    const uint32_t* pz[MT];
    const __half* ps[MT];
    auto set_rows = [&](int u) {
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            int mi, f0;
            unit_tile(u, mt, mi, f0);
            const size_t row = (size_t)f0 + g;
            pw[mt] = reinterpret_cast<const uint4*>(p.m[mi].w + row * p.PW) + t;
            pz[mt] = p.m[mi].z + row * p.PZ;
            ps[mt] = p.m[mi].s + row * p.G;
        }
    };
    auto prefetch = [&](Stage& d) {
        if (pf.u < my_units) {
            const int grp = pf.g, u = pf.u;
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    d.w[mt][hh] = ldg_stream(pw[mt] + hh * 2 * p.PW + 4 * grp);
                    d.zw[mt][hh] = __ldg(pz[mt] + hh * 8 * p.PZ + (grp >> 3));
                    d.sc[mt][hh] = __ldg(ps[mt] + hh * 8 * p.G + grp);
                }
            pf.next(p.G, my_units);
            if (pf.u != u && pf.u < my_units) set_rows(pf.u);
        }
    };
    if (pf.u < my_units) set_rows(pf.u);
#pragma unroll
    for (int d = 0; d < D; d++) prefetch(st[d]);
    griddep_wait();
    if (!p.late) griddep_launch_dependents();

    // x: the batch rows' 32 inputs of this thread's quarter of a group, fetched one step ahead
    const __half* xrow[NT];
    bool xok[NT];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        xok[nt] = g + 8 * nt < p.M;
        xrow[nt] = p.x + (size_t)(xok[nt] ? g + 8 * nt : 0) * p.K + 32 * t;
    }
    uint4 xn[NT][4];
    auto load_x = [&](int grp) {
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                xn[nt][j] = make_uint4(0, 0, 0, 0);
                if (xok[nt]) xn[nt][j] = *reinterpret_cast<const uint4*>(xrow[nt] + 128 * grp + 8 * j);
            }
    };

    float acc[MT][NT][4];
    auto clear_acc = [&]() {
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++) acc[mt][nt][0] = acc[mt][nt][1] = acc[mt][nt][2] = acc[mt][nt][3] = 0.f;
    };
    clear_acc();

    // End of unit u for this warp: its share's partial tile goes to shared memory. ROTATING sums up to kSum units together, without a
    // barrier on the way (with one per unit, eight rows of 70B gate/up 84.1 us, 77.5 so; 13B 25.6, 23.4).
    auto unit_end = [&](int u) {
        const int share = DEAL == ROTATING ? (warp + u) % kWarps : warp, slot = u % kSlots, last = u % kSum;
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) red[slot][share][mt][nt][e][lane] = acc[mt][nt][e];
        clear_acc();
        if (last + 1 < kSum && u + 1 < my_units) return;
        __syncthreads();
        // thread = (nt, e, lane): element (feature f0 + g + 8 (e >> 1), batch row 8 nt + 2 t + (e & 1)) of every tile
        for (int i = threadIdx.x; i < (last + 1) * NT * 4 * 32; i += kWarps * 32) {
            const int l = i & 31, e = (i >> 5) & 3, nt = (i >> 7) % NT, par = (i >> 7) / NT, u0 = u - last + par;
            const int row = 8 * nt + 2 * (l & 3) + (e & 1);
            float v[MT];
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                float sum = 0.f;
#pragma unroll
                for (int w = 0; w < kWarps; w++) sum += red[slot - last + par][w][mt][nt][e][l];
                v[mt] = sum;
            }
            if (row >= p.M) continue;
            if (SILU) {
                int mi, f0;
                unit_tile(u0, 0, mi, f0);
                float val = v[0];
                val *= 1.0f / (1.0f + expf(-val));
                val *= v[MT - 1];
                p.m[0].y[(size_t)row * p.m[0].ldy + f0 + (l >> 2) + 8 * (e >> 1)] = __float2half(val);
            } else {
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    int mi, f0;
                    unit_tile(u0, mt, mi, f0);
                    const SkMat& mm = p.m[mi];
                    const size_t at = (size_t)row * mm.ldy + f0 + (l >> 2) + 8 * (e >> 1);
                    float val = v[mt];
                    if (p.residual) val += __half2float(p.residual[at]) * p.rscale;
                    mm.y[at] = __float2half(val);
                }
            }
        }
        if (DEAL == ROTATING && u + 1 < my_units) __syncthreads();   // the buffers are written again (FIXED: behind the next unit's barrier only)
    };

    for (int u = 0; u < cur.u; u++) unit_end(u);   // (fewer groups than warps: units in which this one has none)
    if (cur.u < my_units) load_x(cur.g);
    while (cur.u < my_units) {
#pragma unroll
        for (int d = 0; d < D; d++) {
            if (cur.u >= my_units) break;
            const int grp = cur.g, u = cur.u;
            cur.next(p.G, my_units);
            // this step's x pairs in the unpack's order; the next step's x leaves now
            uint32_t xp[NT][4][4];
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int j = 0; j < 4; j++) permute_x8(xn[nt][j], xp[nt][j]);
            if (cur.u < my_units) load_x(cur.g);
            const Stage& now = st[d];
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                uint32_t zlo[2], zhi[2];
                float sc[2];
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    const uint32_t z = (now.zw[mt][hh] >> (4 * (grp & 7))) & 0xFu;
                    zlo[hh] = (0x6400u | z) * 0x00010001u;          // 1024 + z
                    zhi[hh] = (0x5400u | (z << 4)) * 0x00010001u;   // 64 + z
                    sc[hh] = __half2float(now.sc[mt][hh]);
                }
                float c[NT][4];
#pragma unroll
                for (int nt = 0; nt < NT; nt++) c[nt][0] = c[nt][1] = c[nt][2] = c[nt][3] = 0.f;
                const uint32_t wa[4] = {now.w[mt][0].x, now.w[mt][0].y, now.w[mt][0].z, now.w[mt][0].w};
                const uint32_t wb[4] = {now.w[mt][1].x, now.w[mt][1].y, now.w[mt][1].z, now.w[mt][1].w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint32_t da[4], db[4];
                    unpack8(wa[j], zlo[0], zhi[0], da);
                    unpack8(wb[j], zlo[1], zhi[1], db);
#pragma unroll
                    for (int nt = 0; nt < NT; nt++) {
                        mma_f16(c[nt], da[0], db[0], da[1], db[1], xp[nt][j][0], xp[nt][j][1]);
                        mma_f16(c[nt], da[2], db[2], da[3], db[3], xp[nt][j][2], xp[nt][j][3]);
                    }
                }
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    acc[mt][nt][0] = fmaf(sc[0], c[nt][0], acc[mt][nt][0]);
                    acc[mt][nt][1] = fmaf(sc[0], c[nt][1], acc[mt][nt][1]);
                    acc[mt][nt][2] = fmaf(sc[1], c[nt][2], acc[mt][nt][2]);
                    acc[mt][nt][3] = fmaf(sc[1], c[nt][3], acc[mt][nt][3]);
                }
            }
            prefetch(st[d]);   // the stage is spent: its next occupant, D steps ahead, leaves now
            for (int e = u; e < cur.u; e++) unit_end(e);
        }
    }
    if (p.late) griddep_launch_dependents();
}

// ------------------------------------------------------------------------------------------------------------
// Stream form
// ------------------------------------------------------------------------------------------------------------
namespace stream {
constexpr int kWarps = 16;
constexpr int kThreads = 32 * kWarps;
constexpr int kItemBytes = 1024;     // a tile's 16 rows over a group
constexpr int kDepth = 4;            // items in a warp's ring, a multiple of those that are kept (12: 70B gate/up 83 us, 64: fewer tiles fit into a pass)
constexpr int kSmemBytes = 226 * 1024;
constexpr int kRingBytes = kWarps * kDepth * kItemBytes;
__host__ __device__ constexpr int part_bytes(int NT) { return NT * kWarps * 512; }      // partial sums of a tile
// Words of a row of scales and zero points (scale | zero point << 16): an odd number, so that the rows of a tile lie in different banks.
__host__ __device__ constexpr int meta_row(int G) { return G | 1; }
constexpr int tiles_in_pass(int G, int NT) { return (kSmemBytes - kRingBytes) / (part_bytes(NT) + 64 * meta_row(G)); }
}  // namespace stream

struct StreamParams {
    SkParams s;
    int tiles, nt_div, nt_mod;       // of 16 rows (SILU: eight gate and the same eight up features); CTA c has nt_div + (c < nt_mod) consecutive ones
    int pass_tiles;
    float inv_mrow;                  // 1 / meta_row(G)
};

// NT: batch columns of eight; GP: groups that every warp keeps; the items of the groups that are left are dealt out over the warps.
template <int NT, int GP, bool SILU>
__global__ void __launch_bounds__(stream::kThreads, 1) q4_rows_stream_kernel(const __grid_constant__ StreamParams r) {
    using namespace stream;
    extern __shared__ __align__(128) uint8_t smem[];
    const SkParams& p = r.s;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, cta = blockIdx.x;
    const int cta_tile0 = cta * r.nt_div + min(cta, r.nt_mod), cta_tiles = r.nt_div + (cta < r.nt_mod);
    const int g0 = w * GP, rest = p.G - GP * kWarps, mrow = meta_row(p.G);
    uint8_t* const mine = smem + w * kDepth * kItemBytes + lane * 16;
    float* const part = reinterpret_cast<float*>(smem + kRingBytes);
    uint32_t* const meta = reinterpret_cast<uint32_t*>(smem + kRingBytes + r.pass_tiles * part_bytes(NT));
    // matrix and row of row i (0-15) of a tile; the rows 0-7 and 8-15 are the product's
    auto row_of = [&](int tile, int i, int& row) -> const SkMat& {
        if (SILU) {
            row = tile * 8 + (i & 7);
            return p.m[i >> 3];
        }
        const int mi = p.nmat > 2 && tile >= p.m[2].tile0 ? 2 : p.nmat > 1 && tile >= p.m[1].tile0 ? 1 : 0;
        row = (tile - p.m[mi].tile0) * 16 + i;
        return p.m[mi];
    };

    // Walks this warp's items: in a pass its own groups tile by tile, then its share of the items of the groups that are left, group by group. A lane
    // copies the 16 bytes of rows g and 8 + g that it reads.
    const uint32_t dst0 = smem_u32(mine);
    const int step = (SILU ? 8 : 16) * p.PW;
    struct {
        const uint32_t *src, *src8;  // rows g and 8 + g of the tile: its first own group, or the item (rest)
        int tile, k, grp, left, b0, tiles;     // k < GP: own groups; GP: rest, `left` items of it to come, `grp` the group
        int end;                     // the tiles of this pass and matrix end here
    } q;
    auto seek = [&](int grp) {
        int row;
        const SkMat& m = row_of(cta_tile0 + q.tile, g, row);
        q.src = m.w + (size_t)row * p.PW + grp * 16 + t * 4;
        q.src8 = SILU ? p.m[1].w + (size_t)row * p.PW + grp * 16 + t * 4 : q.src + 8 * p.PW;
        q.end = q.b0 + q.tiles;
        if (!SILU && p.nmat > 1) {
            const int last = cta_tile0 + q.tile >= p.m[2].tile0 ? r.tiles : cta_tile0 + q.tile >= p.m[1].tile0 ? p.m[2].tile0 : p.m[1].tile0;
            q.end = min(q.end, last - cta_tile0);
        }
    };
    auto open_pass = [&]() {
        q.tiles = min(r.pass_tiles, cta_tiles - q.b0);
        q.tile = q.b0;
        q.k = 0;
        if (q.tiles > 0) seek(g0);
    };
    auto open_rest = [&]() {
        const int r0 = w * rest * q.tiles / kWarps, r1 = (w + 1) * rest * q.tiles / kWarps;
        q.k = GP;
        q.left = r1 - r0;
        q.grp = GP * kWarps + r0 / q.tiles;
        q.tile = q.b0 + r0 % q.tiles;
        if (q.left > 0) seek(q.grp);
    };
    auto settle = [&]() {      // past rests that are empty
        while (q.tiles > 0 && q.k == GP && q.left == 0) {
            q.b0 += q.tiles;
            open_pass();
        }
    };
    auto next = [&]() {
        if (q.k < GP) {
            if (++q.k < GP) return;
            q.k = 0;
            q.src += step;
            q.src8 += step;
            if (++q.tile < q.end) return;
            if (q.tile < q.b0 + q.tiles) {
                seek(g0);
                return;
            }
            open_rest();
        } else {
            q.left--;
            q.src += step;
            q.src8 += step;
            if (++q.tile == q.b0 + q.tiles) {
                q.tile = q.b0;
                q.grp++;
                if (q.left > 0) seek(q.grp);
            } else if (q.tile == q.end && q.left > 0) {
                seek(q.grp);
            }
        }
        settle();
    };
    auto request = [&](uint32_t slot) {      // (slot: its first byte)
        if (q.k == GP && q.left > 1 && q.tile + 1 < q.end) {     // (the next item is the next tile's)
            copy16(dst0 + slot, q.src);
            copy16(dst0 + slot + 512, q.src8);
            q.src += step;
            q.src8 += step;
            q.tile++;
            q.left--;
        } else if (q.tiles > 0) {
            const int k = q.k < GP ? q.k * 16 : 0;
            copy16(dst0 + slot, q.src + k);
            copy16(dst0 + slot + 512, q.src8 + k);
            next();
        }
        copies_commit();
    };
    q.b0 = q.left = q.end = q.tile = 0;
    open_pass();
    for (int i = 0; i < kDepth; i++) request(i * kItemBytes);
    // A pass's scales and zero points into shared memory, several of a thread in flight.
    constexpr int kFlight = NT == 2 ? 4 : 8;     // (registers: the form for more than eight rows spills three to five of them once)
    struct Meta {
        __half s[kFlight];
        uint32_t z[kFlight];
    };
    auto fetch_meta = [&](Meta& v, int e0, int b0, int n) {
#pragma unroll
        for (int u = 0; u < kFlight; u++) {
            const int e = e0 + u * kThreads, i = (int)(((float)e + 0.5f) * r.inv_mrow), grp = e - i * mrow;
            v.s[u] = __float2half(0.f);
            v.z[u] = 0;
            if (e < n && grp < p.G) {
                int row;
                const SkMat& m = row_of(cta_tile0 + b0 + (i >> 4), i & 15, row);
                v.s[u] = __ldg(m.s + (size_t)row * p.G + grp);
                v.z[u] = __ldg(m.z + (size_t)row * p.PZ + (grp >> 3));
            }
        }
    };
    auto file_meta = [&](const Meta& v, int e0, int n) {
#pragma unroll
        for (int u = 0; u < kFlight; u++) {
            const int e = e0 + u * kThreads, grp = e - (int)(((float)e + 0.5f) * r.inv_mrow) * mrow;
            if (e < n) meta[e] = (uint32_t)__half_as_ushort(v.s[u]) | (((v.z[u] >> (4 * (grp & 7))) & 0xFu) << 16);
        }
    };
    auto load_meta = [&](int e0, int b0, int n) {
        for (; e0 < n; e0 += kFlight * kThreads) {
            Meta v;
            fetch_meta(v, e0, b0, n);
            file_meta(v, e0, n);
        }
    };
    Meta first;
    const int first_n = min(r.pass_tiles, cta_tiles) * 16 * mrow;
    fetch_meta(first, tid, 0, first_n);
    griddep_wait();
    if (!p.late) griddep_launch_dependents();

    // The rows' inputs of a group, in the order of the unpacked pairs. 32 bytes in one access: with 16 every sector would come from L2 twice (next to
    // this much shared memory there is little L1).
    const bool whole = ((uintptr_t)p.x & 31) == 0;
    auto load_x = [&](int grp, uint4 (&v)[NT][4]) {
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                uint4 &a = v[nt][j], &b = v[nt][j + 1];
                a = b = make_uint4(0, 0, 0, 0);
                if (g + 8 * nt >= p.M) continue;
                const __half* src = p.x + (size_t)(g + 8 * nt) * p.K + 128 * grp + 32 * t + 8 * j;
                if (whole) {
                    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "l"(src));
                } else {
                    a = reinterpret_cast<const uint4*>(src)[0];
                    b = reinterpret_cast<const uint4*>(src)[1];
                }
            }
    };
    struct X { uint32_t v[NT][4][4]; };
    X xp[GP + 1];        // (the last one: a group that is left, for the tiles it is this warp's)
    auto permute = [&](const uint4 (&v)[NT][4], X& x) {
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int j = 0; j < 4; j++) permute_x8(v[nt][j], x.v[nt][j]);
    };
    {
        uint4 xv[GP][NT][4];
#pragma unroll
        for (int k = 0; k < GP; k++) load_x(g0 + k, xv[k]);
        file_meta(first, tid, first_n);
        load_meta(tid + kFlight * kThreads, 0, first_n);
#pragma unroll
        for (int k = 0; k < GP; k++) permute(xv[k], xp[k]);
    }

    uint32_t slot = 0;           // the next item's, its first byte
    // acc += one item's product; the copies that take its place are `more`'s
    auto item = [&](float (&acc)[NT][4], const X& x, const uint32_t* me, auto&& more) {
        copies_wait<kDepth - 1>();
        const uint4 va = *reinterpret_cast<const uint4*>(mine + slot), vb = *reinterpret_cast<const uint4*>(mine + slot + 512);
        const uint32_t ma = me[0], mb = me[8 * mrow];
        const uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
        const uint32_t zla = 0x64006400u + (ma >> 16) * 0x00010001u, zha = 0x54005400u + (ma >> 16) * 0x00100010u;      // 1024 + z, 64 + z
        const uint32_t zlb = 0x64006400u + (mb >> 16) * 0x00010001u, zhb = 0x54005400u + (mb >> 16) * 0x00100010u;
        float c[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) c[nt][0] = c[nt][1] = c[nt][2] = c[nt][3] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint32_t da[4], db[4];
            unpack8(wa[j], zla, zha, da);
            unpack8(wb[j], zlb, zhb, db);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                mma_f16(c[nt], da[0], db[0], da[1], db[1], x.v[nt][j][0], x.v[nt][j][1]);
                mma_f16(c[nt], da[2], db[2], da[3], db[3], x.v[nt][j][2], x.v[nt][j][3]);
            }
        }
        more(slot);
        slot += kItemBytes;
        if (slot == kDepth * kItemBytes) slot = 0;
        const float sa = __half2float(__ushort_as_half((unsigned short)(ma & 0xFFFFu))), sb = __half2float(__ushort_as_half((unsigned short)(mb & 0xFFFFu)));
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            acc[nt][0] = fmaf(sa, c[nt][0], acc[nt][0]);
            acc[nt][1] = fmaf(sa, c[nt][1], acc[nt][1]);
            acc[nt][2] = fmaf(sb, c[nt][2], acc[nt][2]);
            acc[nt][3] = fmaf(sb, c[nt][3], acc[nt][3]);
        }
    };
    for (int b0 = 0; b0 < cta_tiles; b0 += r.pass_tiles) {
        const int tiles = min(r.pass_tiles, cta_tiles - b0);
        float4* const col = reinterpret_cast<float4*>(part + w * 128) + lane;      // this lane's sums: [tile][NT][warp][lane]
        __syncthreads();         // the pass's scales and zero points are in place, and the sums of the one before are done with
        const uint32_t* me = meta + g * mrow + g0;
        for (int i = 0; i < tiles; i++) {
            float acc[NT][4];
#pragma unroll
            for (int nt = 0; nt < NT; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
            // Within the own groups of a pass and of a matrix the next requests are those of one tile.
            if (q.tiles > 0 && q.k == 0 && q.tile + 1 < q.end) {
#pragma unroll
                for (int k = 0; k < GP; k++)
                    item(acc, xp[k], me + k, [&](uint32_t at) {
                        copy16(dst0 + at, q.src + k * 16);
                        copy16(dst0 + at + 512, q.src8 + k * 16);
                        copies_commit();
                    });
                q.src += step;
                q.src8 += step;
                q.tile++;
            } else {
#pragma unroll
                for (int k = 0; k < GP; k++) item(acc, xp[k], me + k, request);
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++) col[(i * NT + nt) * kWarps * 32] = make_float4(acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3]);
            me += 16 * mrow;
        }
        // this warp's share of the items of the groups that are left
        const int r0 = w * rest * tiles / kWarps, r1 = (w + 1) * rest * tiles / kWarps;
        int grp = GP * kWarps + r0 / tiles, tile = r0 % tiles, left = r1 - r0;
        while (left > 0) {
            const int count = min(left, tiles - tile);
            uint4 xv[NT][4];
            load_x(grp, xv);
            permute(xv, xp[GP]);
            left -= count;
            me = meta + (tile * 16 + g) * mrow + grp;
            for (int i = tile; i < tile + count; i++) {
                float acc[NT][4];
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    const float4 v = col[(i * NT + nt) * kWarps * 32];
                    acc[nt][0] = v.x; acc[nt][1] = v.y; acc[nt][2] = v.z; acc[nt][3] = v.w;
                }
                item(acc, xp[GP], me, request);
#pragma unroll
                for (int nt = 0; nt < NT; nt++) col[(i * NT + nt) * kWarps * 32] = make_float4(acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3]);
                me += 16 * mrow;
            }
            grp++;
            tile = 0;
        }
        __syncthreads();
        // the warps' sums in warp order; lane 4g + t has rows g and 8 + g of the tile for batch rows 2t and 2t + 1
        for (int i = w; i < tiles * NT; i += kWarps) {
            const float4* src = reinterpret_cast<const float4*>(part) + (size_t)i * kWarps * 32 + lane;
            float4 v = src[0];
#pragma unroll
            for (int u = 1; u < kWarps; u++) {
                const float4 a = src[u * 32];
                v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
            }
            int f;
            const SkMat& m = row_of(cta_tile0 + b0 + i / NT, g, f);
            const int row = 8 * (i % NT) + 2 * t;
            const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < (SILU ? 2 : 4); e++) {
                if (row + (e & 1) >= p.M) continue;
                const size_t to = (size_t)(row + (e & 1)) * m.ldy + f + (e >> 1) * 8;
                float y = o[e];
                if (SILU) {
                    y *= 1.0f / (1.0f + expf(-y));
                    y *= o[e + 2];
                } else if (p.residual) {
                    y += __half2float(p.residual[to]) * p.rscale;
                }
                m.y[to] = __float2half(y);
            }
        }
        if (b0 + tiles < cta_tiles) load_meta(tid, b0 + tiles, min(r.pass_tiles, cta_tiles - b0 - tiles) * 16 * mrow);
    }
    if (p.late) griddep_launch_dependents();
}


constexpr int kSms = 148;   // B200: one persistent CTA per SM (a smaller part would only leave CTAs queued behind the first wave)
constexpr size_t unit_bytes(int MT, int NT) { return (size_t)warps_of(MT, NT) * MT * NT * 4 * 32 * sizeof(float); }

int fill(SkParams& p, const uint16_t* x, int M, int K) {
    if (!x || M < 1 || M > 16) return Q4_ERR_INVALID;
    if (K <= 0 || (K % 128)) return Q4_ERR_UNSUPPORTED_SIZE;
    p.x = reinterpret_cast<const __half*>(x);
    p.M = M;
    p.K = K;
    p.PW = q4_pw(K);
    p.PZ = q4_pz(K);
    p.G = q4_groups(K);
    return Q4_OK;
}

SkMat sk_mat(const q4_qweight* w, uint16_t* y, int ldy, int tile0) {
    SkMat m;
    m.w = w->weight;
    m.z = w->zeros;
    m.s = reinterpret_cast<const __half*>(w->scales);
    m.y = reinterpret_cast<__half*>(y);
    m.ldy = ldy;
    m.tile0 = tile0;
    return m;
}

template <int MT, int NT, bool SILU, Deal DEAL>
int launch_deal(const SkParams& p, int units, cudaStream_t s) {
    constexpr int kSlots = slots_of(NT, DEAL);
    const int per_cta = q4_div_up(units, kSms);
    // (the limit belongs to the function: always the largest any launch needs)
    if (kSlots * unit_bytes(MT, NT) > 48 * 1024)
        Q4_CUDA_TRY(cudaFuncSetAttribute(q4_skinny_kernel<MT, NT, SILU, DEAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSlots * unit_bytes(MT, NT))));
    // x comes out of L1 again and again: behind a kernel that takes all of the SM's memory as shared (the stream form) the split would stay as it is
    // (eight sequences, 32 steps of four 7B layers 7600 us, 6860 so).
    static std::atomic<unsigned long long> preferred{0};
    Q4_CUDA_TRY(q4_prefer_carveout(q4_skinny_kernel<MT, NT, SILU, DEAL>, 50, preferred));
    const size_t smem = (per_cta < kSlots ? per_cta : kSlots) * unit_bytes(MT, NT);
    Q4Launch L(dim3(units < kSms ? units : kSms), dim3(warps_of(MT, NT) * 32), smem, s);
    Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, q4_skinny_kernel<MT, NT, SILU, DEAL>, p));
    return Q4_OK;
}

// Whether a warp keeps its share of every unit: where shares that go round make no warp's load lighter, a barrier per unit and one unit's
// sum at a time are cheaper than cursors that move and a sum of several units at the end (us from HBM, fixed against going round, on shapes that
// streamed() leaves to this form).
//   9 to 16 rows, equal shares of one group or an even number: 4096 -> 8192 9.5, 10.1 (9 rows), 10.0, 10.2 (16); 6144 -> 8192 13.6, 14.3 and 14.2, 14.6;
//   4096 -> 2 x 4096 9.4, 10.1 and 10.0, 10.5; 1024 -> 2 x 20000 11.9, 13.1 and 13.0, 13.9. With shares of three or five groups the two are close, and
//   going round wins with 16 rows of long launches (3072 -> 12288 11.4, 11.5 and 12.2, 11.7); with unequal ones it wins clearly (2560 -> 3 x 2560 7.3,
//   6.7 and 7.9, 6.9).
//   9 to 16 rows, one unit per CTA: 7B o 5.3, 5.6 and 5.6, 5.8; the step of nine sequences (32 steps of four 7B layers) 8985 us, 9055 going round. With up to
//   8 rows 4.4, 4.6 alone, but there the step, whose launches take turns with the stream form's, says the opposite: eight sequences 7015 us, 6835 going
//   round; one 6530, 6330.
//   Gate/up with two units per CTA whose heaviest pair of neighbouring shares is two heaviest ones: 8 rows, 4096 -> 2 x 4096 7.2, 7.6; 7168 -> 2 x 4096
//   11.3, 11.6 (and 5120 -> 2 x 4096, where it is not, 9.0, 8.6). With very long shares the barrier costs more (28672 -> 8192 in two units 42.0, 41.6).
bool fixed_shares(int G, int warps, int NT, bool silu, int per_cta) {
    if (NT == 2 && per_cta == 1) return true;
    if (NT == 2 && G % warps == 0) return G == warps || G / warps % 2 == 0;
    if (!silu || per_cta != 2 || G > 12 * warps) return false;
    auto share = [&](int i) { return G * (i % warps + 1) / warps - G * (i % warps) / warps; };
    int most = 0, pair = 0;
    for (int i = 0; i < warps; i++) {
        most = share(i) > most ? share(i) : most;
        pair = share(i) + share(i + 1) > pair ? share(i) + share(i + 1) : pair;
    }
    return pair == 2 * most;
}

template <int MT, int NT, bool SILU>
int launch_variant(const SkParams& p, cudaStream_t s) {
    const int units = SILU ? p.total_tiles : p.total_tiles / MT;
    if (fixed_shares(p.G, warps_of(MT, NT), NT, SILU, q4_div_up(units, kSms))) return launch_deal<MT, NT, SILU, FIXED>(p, units, s);
    return launch_deal<MT, NT, SILU, ROTATING>(p, units, s);
}

template <int NT, int GP, bool SILU>
int launch_stream(const SkParams& p, cudaStream_t s) {
    StreamParams r;
    r.s = p;
    r.tiles = SILU ? 2 * p.total_tiles : p.total_tiles;
    const int grid = r.tiles < kSms ? r.tiles : kSms;
    r.nt_div = r.tiles / grid;
    r.nt_mod = r.tiles % grid;
    const int most = r.nt_div + (r.nt_mod > 0);
    r.pass_tiles = q4_div_up(most, q4_div_up(most, stream::tiles_in_pass(p.G, NT)));
    r.inv_mrow = 1.0f / stream::meta_row(p.G);
    // (the limit belongs to the function: always the largest any launch needs)
    Q4_CUDA_TRY(cudaFuncSetAttribute(q4_rows_stream_kernel<NT, GP, SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, stream::kSmemBytes));
    Q4Launch L(dim3(grid), dim3(stream::kThreads), (size_t)stream::kSmemBytes, s);
    Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, q4_rows_stream_kernel<NT, GP, SILU>, r));
    return Q4_OK;
}

// The stream form where an SM has three or more of the tiles of 16 rows (gate/up: eight of each) and rows are 4096 inputs or longer; from
// seven tiles also from 2048 inputs. us back to back from HBM, sliced and stream, 8 rows and 16: 7B gate/up 16.4, 13.0 and 23.1, 22.3; q|k|v 10.1, 9.3 and
// 14.3, 13.4; 13B q|k|v 20.2, 13.3 and 31.5, 18.7; gate/up 23.2, 18.9 and 36.1, 30.8; 13824 -> 5120 21.6, 17.4 and 35.3, 23.0; 70B gate/up 77.9, 64.3 and
// 120, 94; 8192 -> 10240 22.0, 15.2 and 36.6, 20.6; 2048 -> 16384 9.8, 7.6 and 14.7, 9.3 (16640, whose pairs of tiles divide better 7.6, 7.7 and 10.4, 9.5).
// Below, the sliced form's shorter start wins: two tiles 7B o 4.7, 5.5 and 5.6, 7.6; 11008 -> 4096 9.5, 11.5 and 12.7, 15.8; 2048 -> 3 x 4096 5.9, 6.7 and
// 8.1, 8.1. Four tiles (445 to 592 in all) are two even rounds of the sliced form's pairs, which keeps up then: 4096 -> 3 x 3072 7.9, 8.3 and 10.3, 10.9;
// 8192 x 8192 13.1, 13.0 and 19.4, 17.4 (8 rows on words in L2 12.0, 12.3).
bool streamed(int G, int tiles) {
    const int most = q4_div_up(tiles, kSms);
    if (stream::tiles_in_pass(G, 2) == 0) return false;
    if (G < 32) return G >= 16 && most >= 7;
    return most >= 3 && (most != 4 || G >= 64);
}

template <bool SILU>
int launch(const SkParams& p, cudaStream_t s) {
    if (streamed(p.G, SILU ? 2 * p.total_tiles : p.total_tiles)) {
        if (p.M > 8) return launch_stream<2, 1, SILU>(p, s);
        return p.G >= 2 * stream::kWarps ? launch_stream<1, 2, SILU>(p, s) : launch_stream<1, 1, SILU>(p, s);
    }
    const bool two = p.M > 8;
    if (SILU) return two ? launch_variant<2, 2, true>(p, s) : launch_variant<2, 1, true>(p, s);
    // Two tiles per unit halve the reads of x but double the grain the work is dealt in: take pairs when the most loaded
    // SM then carries no more features than with single tiles.
    const int t = p.total_tiles;
    const bool pair = (t % 2 == 0) && 2 * q4_div_up(t / 2, kSms) <= q4_div_up(t, kSms);
    if (pair) return two ? launch_variant<2, 2, false>(p, s) : launch_variant<2, 1, false>(p, s);
    return two ? launch_variant<1, 2, false>(p, s) : launch_variant<1, 1, false>(p, s);
}

}  // namespace

extern "C" int q4_matmul_q4_rows(void* stream, uint16_t* y, const uint16_t* x, const q4_qweight* w, int M, int inpSize, int opSize,
                                 const uint16_t* residual, float residual_scale) {
    SkParams p = {};
    if (int e = fill(p, x, M, inpSize)) return e;
    if (!y || !w) return Q4_ERR_INVALID;
    if (opSize <= 0 || (opSize % 16)) return Q4_ERR_UNSUPPORTED_SIZE;
    p.nmat = 1;
    p.m[0] = sk_mat(w, y, opSize, 0);
    p.total_tiles = opSize / 16;
    p.residual = reinterpret_cast<const __half*>(residual);
    p.rscale = residual_scale;
    return launch<false>(p, (cudaStream_t)stream);
}

extern "C" int q4_qkv_matmul_rows(void* stream, uint16_t* q, uint16_t* k, uint16_t* v, const uint16_t* x, const q4_qweight* qw,
                                  const q4_qweight* kw, const q4_qweight* vw, int M, int inpSize, int opSize, int kvSize) {
    return q4_qkv_rows_launch(stream, q, k, v, x, qw, kw, vw, M, inpSize, opSize, kvSize, false);
}

// late: the successor is the attention of batched decode, whose few CTAs would be dealt out as this kernel's CTAs (one per SM, most
// of its registers) leave: three or four to each of the first SMs, where they walk their keys while the other SMs idle. Signalled
// at the end they spread (one sequence at position 1900, step of two 7B layers: 275 us against 173). Not for a successor that
// streams weights, which loses its head start (the 7B product back to back, 8 rows: 10.6 us, 11.7 signalled at the end).
int q4_qkv_rows_launch(void* stream, uint16_t* q, uint16_t* k, uint16_t* v, const uint16_t* x, const q4_qweight* qw, const q4_qweight* kw, const q4_qweight* vw,
                       int M, int inpSize, int opSize, int kvSize, bool late) {
    SkParams p = {};
    p.late = late;
    if (int e = fill(p, x, M, inpSize)) return e;
    if (!q || !k || !v || !qw || !kw || !vw) return Q4_ERR_INVALID;
    if (opSize <= 0 || kvSize <= 0 || (opSize % 32) || (kvSize % 32)) return Q4_ERR_UNSUPPORTED_SIZE;   // a CTA's two tiles lie in one matrix
    p.nmat = 3;
    const int tq = opSize / 16, tkv = kvSize / 16;
    p.m[0] = sk_mat(qw, q, opSize, 0);
    p.m[1] = sk_mat(kw, k, kvSize, tq);
    p.m[2] = sk_mat(vw, v, kvSize, tq + tkv);
    p.total_tiles = tq + 2 * tkv;
    return launch<false>(p, (cudaStream_t)stream);
}

extern "C" int q4_ffn_silu_rows(void* stream, uint16_t* h, const uint16_t* x, const q4_qweight* gate_w, const q4_qweight* up_w, int M,
                                int inpSize, int opSize) {
    SkParams p = {};
    if (int e = fill(p, x, M, inpSize)) return e;
    if (!h || !gate_w || !up_w) return Q4_ERR_INVALID;
    if (opSize <= 0 || (opSize % 16)) return Q4_ERR_UNSUPPORTED_SIZE;
    p.nmat = 2;
    p.m[0] = sk_mat(gate_w, h, opSize, 0);
    p.m[1] = sk_mat(up_w, h, opSize, 0);
    p.total_tiles = opSize / 16;
    return launch<true>(p, (cudaStream_t)stream);
}
