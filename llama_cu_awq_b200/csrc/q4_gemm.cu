// Batched / prefill W4 g128 dequant-GEMM on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a only:
//   Y[M][N] = X[M][K] * deq(W)[K][N],  deq(W)(k, n) = (q(n, k) - z(n, k / 128)) * s(n, k / 128)
// fp16 in, fp32 accumulation in tensor memory, fp16 out. The reference has no batched path: it pushes a prompt through
// the batch-1 GEMV token by token (llama2_q4.cu:710-735, mat_vec_kernel_int4 gpu_kernels.h:179-248); M rows here are M
// applications of that GEMV, and that is what the tests compare against.
//
// Swap-AB: the weights are the MMA's 256-row operand, the batch its N side (a multiple of 32 up to 256 rows of X per tile).
// A pair of SMs (cluster of two, cta_group::2) works on one tile of 256 features x MT rows: each CTA dequantises its own 128
// features and fetches half of the X tile, so X crosses the L2-to-SM path once per 256 features. The dequantised weights
// never touch shared memory: the converters store them straight into tensor memory, from where the MMA reads them as
// its A operand. Both follow from what bounded the kernel before (one CTA per tile, A staged in shared memory, 845
// TFLOP/s at 2000 rows): 72 B per clock and SM of L2 reads for a 64 B port, and 200 B per clock of shared-memory traffic
// (MMA operands, conversion stores, TMA writes) for 128 B. Now: 40 and 80.
//
// Persistent pairs; a pair takes an equal, contiguous share of all (tile, 256-input chunk) steps, so no wave is ever partly
// empty (96 tiles of a 512-row QKV projection over 74 pairs would take two waves, 65 % busy). A tile cut by a share boundary
// is summed through fp32 partial tiles in the workspace, always in K order, by whichever CTA arrives last.
// Roles (512 threads; registers are moved from the first warpgroup to the epilogue):
//   warp 0      TMA of packed weight chunks (128 features x 256 inputs = 128 B per row, 128-byte swizzle) into a staging ring
//   warp 1      TMA of X slabs (MT / 2 rows x 64 inputs, 128-byte swizzle); both CTAs' copies report to the leader's barrier
//   warp 2      leader CTA: one thread issues tcgen05.mma.cta_group::2.kind::f16 and commits the stages back to both CTAs
//   warps 4-11  converters, two warpgroups on alternate 128-input blocks (= quantisation groups): a thread owns a feature
//               row, reads 64 B of nibbles (conflict free thanks to the swizzle), dequantises in registers (LOP3 magic-number
//               unpack, one exact subtract, one rounding multiply) and writes 64 tensor-memory columns (tcgen05.st)
//   warps 12-15 epilogue: drain the accumulator into registers, release it, then scale / add / store while the next
//               tile's MMAs run
// Tensor memory: columns 0 .. MT - 1 accumulator, behind it as many A stages of 64 columns as fit (four at 256 rows, seven at
// 64). A stage and the X slabs of the same 128 inputs form one ring entry: one wait and one commit per eight MMAs, because at
// small MT the issuing warp's waits and commits are what bounds the kernel.
//
// Every wait is bounded by the global timer; on expiry the kernel records Q4_ERR_TIMEOUT in the workspace's status word,
// lets all later waits fall through (those of launches queued behind it too), waits (bounded) for its own copies in flight, frees
// its tensor memory and returns. Threads that meet at a barrier or run a warp-wide instruction behind a wait take its outcome
// together: a warp in the converters and the MMA issuer, all four warps in the epilogue. A role that gives up says so in s_gave_up.
#include <cuda.h>
#include <stdio.h>

#include <mutex>

#include "q4_model.h"

namespace {

constexpr int kBN = 128;        // output features per CTA
constexpr int kPairN = 256;     // per tile (two CTAs)
constexpr int kChunkK = 256;    // inputs per packed-weight copy: 32 words = 128 B per feature row
constexpr int kBlockK = 128;    // inputs per A stage: one quantisation group
constexpr int kSlabK = 64;      // inputs per X copy: one 128-byte swizzle row of fp16
constexpr int kMaxMT = 256;
constexpr int kMaxStages = 7, kAStageCols = kBlockK / 2, kTmemCols = 512;
constexpr int kConvWarp0 = 4, kConvWarps = 8, kEpiWarp0 = 12, kEpiWarps = 4;
constexpr int kGemmThreads = 512;
constexpr int kPStageBytes = kBN * (kChunkK / 8) * 4;            // 16 KB
constexpr int kRingBytes = 208 * 1024;                           // shared memory of the two rings
constexpr int kOutRows = 32;                                     // rows of Y per staged store
constexpr int kOutBytes = kOutRows * kBN * 2;                    // 8 KB, two buffers
constexpr int kMaxP = 12;
constexpr unsigned long long kGemmWaitNs = 300ULL * 1000 * 1000;   // limit of every device-side wait
enum GemmEpi { EPI_PLAIN = 0, EPI_RESIDUAL = 1, EPI_SILU = 2 };

struct GemmParams {
    const uint32_t* zeros;
    const __half* scales;
    const __half* residual;   // EPI_RESIDUAL: [M][N], y = product + residual * residual_scale, rounded once (may alias y)
    float residual_scale;
    __half* y;           // PLAIN_Y
    float* partials;     // [pair][2 slots][2 CTAs][MT / 4][128][4] fp32
    int* counters;       // [tile][2 CTAs]
    int* status;         // [0] error code, [1] where
    int M, K, N, G, PZ;
    int MT, m_tiles, n_chunks;
    long long total_chunks;   // tiles * n_chunks
    int settled;         // 1: no kernel in flight writes the packed words
    int stages, np, slab_bytes;   // operand stages (A in tensor memory, X in shared memory), weight copies in flight, bytes of an X slab
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// cluster address of the leader's copy of a barrier
__device__ __forceinline__ uint32_t leader_addr(const void* p) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_addr(p)));
    return r;
}
__device__ __forceinline__ void mb_init(uint64_t* b, int count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count)); }
__device__ __forceinline__ void mb_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mb_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory"); }
__device__ __forceinline__ void mb_arrive_cluster(uint32_t addr) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory"); }
__device__ __forceinline__ bool mb_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0,1,0,p; }"
                 : "=r"(ok) : "r"(smem_addr(b)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: false when the limit is hit (the error is recorded) or an error is already on record.
__device__ __forceinline__ bool mb_wait(uint64_t* b, uint32_t parity, int* status, int where) {
    unsigned long long t0 = 0;
    for (unsigned i = 0;; i++) {
        if (mb_try(b, parity)) return true;
        if ((i & 63u) == 63u) {
            if (*(volatile int*)status != 0) return false;
            const unsigned long long now = gtimer();
            if (t0 == 0) t0 = now;
            else if (now - t0 > kGemmWaitNs) break;
        }
    }
    if (atomicCAS(status, 0, Q4_ERR_TIMEOUT) == 0) status[1] = where;
    return false;
}
// the same for a whole warp; the result is warp-uniform
__device__ __forceinline__ bool warp_wait(uint64_t* b, uint32_t parity, int* status, int where) { return __all_sync(0xffffffffu, mb_wait(b, parity, status, where)); }
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0,1,0,p; }" : "=r"(e));
    return e != 0;
}
// after an error: gives a copy in flight up to 50 ms to land
__device__ __forceinline__ void mb_drain(uint64_t* b, uint32_t parity) {
    const unsigned long long t0 = gtimer();
    while (!mb_try(b, parity) && gtimer() - t0 < 50ULL * 1000 * 1000) {}
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_addr(dst)),
                 "l"(map), "r"(smem_addr(bar)), "r"(x), "r"(y)
                 : "memory");
}
// the same box into L2 only
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
// into this CTA's shared memory, reporting to a barrier of either CTA of the pair (no multicast)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_addr(dst)),
                 "l"(map), "r"(bar), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// arrives on this barrier in both CTAs of the pair when the MMAs issued so far have completed
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr(bar)), "h"((uint16_t)3) : "memory");
}
// D[256 x N] (+)= A[256 x 16] (tensor memory, each CTA its 128 rows) * B[N x 16]^T (shared memory, each CTA half of the rows)
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
#define Q4_R8(v, i) "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]), "r"(v[i + 4]), "r"(v[i + 5]), "r"(v[i + 6]), "r"(v[i + 7])
#define Q4_W8(v, i) "=r"(v[i]), "=r"(v[i + 1]), "=r"(v[i + 2]), "=r"(v[i + 3]), "=r"(v[i + 4]), "=r"(v[i + 5]), "=r"(v[i + 6]), "=r"(v[i + 7])
#define Q4_RW8(v, i) "+r"(v[i]), "+r"(v[i + 1]), "+r"(v[i + 2]), "+r"(v[i + 3]), "+r"(v[i + 4]), "+r"(v[i + 5]), "+r"(v[i + 6]), "+r"(v[i + 7])
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), Q4_R8(v, 0), Q4_R8(v, 8), Q4_R8(v, 16), Q4_R8(v, 24) : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : Q4_W8(v, 0), Q4_W8(v, 8), Q4_W8(v, 16), Q4_W8(v, 24) : "r"(taddr));
    // the registers are listed as operands of the wait, so that no use of them can be scheduled ahead of it
    asm volatile("tcgen05.wait::ld.sync.aligned;" : Q4_RW8(v, 0), Q4_RW8(v, 8), Q4_RW8(v, 16), Q4_RW8(v, 24) : : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile [rows][64 halfs] stored with the 128-byte swizzle: rows of
// 128 B, groups of 8 rows 1024 B apart (stride byte offset), leading byte offset unused (1), descriptor version 1,
// layout type 2 (SWIZZLE_128B). The tile base is 1024-byte aligned (base offset 0). Advancing 16 inputs along K inside
// the swizzled row = + 32 bytes on the start address.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ULL << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ULL << 46) | (2ULL << 61);
}
// Instruction descriptor, kind::f16: D fp32 (bits 4-5 = 1), A and B fp16 (0), both K-major (0), N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t umma_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kPairN >> 4) << 24); }

// One packed word (8 nibbles) -> 8 fp16 weights in input order. INTERLEAVED: the word's nibbles hold inputs 0,2,4,6,1,3,5,7
// (prepared by q4_gemm_interleave_weights), so the two mask patterns yield the pairs (0,1) (2,3) (4,5) (6,7) directly; the file
// layout yields (0,4) (1,5) (2,6) (3,7) and needs four byte permutes. (q - z) is exact in fp16 (|q - z| <= 15; (w & 0x00F0) | 0x5400
// is the half 64 + q), the multiplication by the fp16 scale rounds once.
template <bool INTERLEAVED>
__device__ __forceinline__ void dequant8(uint32_t w, __half2 zlo, __half2 zhi, __half2 s2, uint32_t* o) {
    const __half2 a = __hmul2(__hsub2(u2h2(lop3_and_or(w, 0x000F000Fu, 0x64006400u)), zlo), s2);
    const __half2 b = __hmul2(__hsub2(u2h2(lop3_and_or(w, 0x00F000F0u, 0x54005400u)), zhi), s2);
    w >>= 8;
    const __half2 c = __hmul2(__hsub2(u2h2(lop3_and_or(w, 0x000F000Fu, 0x64006400u)), zlo), s2);
    const __half2 d = __hmul2(__hsub2(u2h2(lop3_and_or(w, 0x00F000F0u, 0x54005400u)), zhi), s2);
    if (INTERLEAVED) {
        o[0] = h22u(a); o[1] = h22u(b); o[2] = h22u(c); o[3] = h22u(d);
    } else {   // a = (0,4) b = (1,5) c = (2,6) d = (3,7)
        o[0] = prmt(h22u(a), h22u(b), 0x5410); o[1] = prmt(h22u(c), h22u(d), 0x5410);
        o[2] = prmt(h22u(a), h22u(b), 0x7632); o[3] = prmt(h22u(c), h22u(d), 0x7632);
    }
}

// A pair's share of the work, segment by segment: consecutive chunks of one tile.
struct Segments {
    long long c, end;
    int n_chunks;
    int tile, c0, c1;
    __device__ __forceinline__ Segments(const GemmParams& p, int pair, int pairs) {
        c = p.total_chunks * pair / pairs;
        end = p.total_chunks * (pair + 1) / pairs;
        n_chunks = p.n_chunks;
    }
    __device__ __forceinline__ bool next() {
        if (c >= end) return false;
        tile = (int)(c / n_chunks);
        c0 = (int)(c - (long long)tile * n_chunks);
        const long long left = end - c;
        c1 = left < n_chunks - c0 ? c0 + (int)left : n_chunks;
        c += c1 - c0;
        return true;
    }
};
// the pair whose share holds global chunk c
__device__ __forceinline__ int pair_of(long long c, long long total, int pairs) { return (int)(((c + 1) * pairs - 1) / total); }

// silu(g) * u in the arithmetic of ffn_matvec_silu_kernel (gpu_kernels.h:278-281): g *= 1 / (1 + expf(-g)), times u, in fp32. The
// reciprocal is the hardware's with one Newton step: compared over all 65536 fp16 gates, g / (1 + e) has the bits of the IEEE division
// but for the 22 gates between -88.75 and -87.3, whose reciprocal is a denormal and whose result is zero in fp16 either way. The
// division's own branch kept the compiler from interleaving evaluations (512 x 4096 x 22016: 12 us longer).
__device__ __forceinline__ float silu_mul(float g, float u) {
    const float d = 1.0f + expf(-g);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    r = d < 0x1p126f ? fmaf(r, fmaf(-d, r, 1.0f), r) : r;
    return g * r * u;
}

// ---- epilogue pieces: 32 accumulator columns (= batch rows c0 .. c0 + 31 of the tile) of one feature, as 16 packed words ----
template <int EPI>
__device__ __forceinline__ void epi_pack(const float (&v)[32], const uint32_t* res, float rscale, uint32_t* out) {
#pragma unroll
    for (int j = 0; j < 16; j++) {
        float a = v[2 * j], b = v[2 * j + 1];
        if (EPI == EPI_RESIDUAL) {
            const float2 f = __half22float2(u2h2(res[j]));
            a += f.x * rscale;
            b += f.y * rscale;
        }
        out[j] = h22u(__floats2half2_rn(a, b));
    }
}
// The 32 rows of the chunk into a staging buffer [row][128 features] (two bytes per lane, 64 B per warp store).
__device__ __forceinline__ void epi_stage(const uint32_t* out, uint8_t* buf, int r) {
    unsigned short* p = reinterpret_cast<unsigned short*>(buf) + r;
#pragma unroll
    for (int j = 0; j < 16; j++) {
        p[(2 * j) * kBN] = (unsigned short)(out[j] & 0xFFFFu);
        p[(2 * j + 1) * kBN] = (unsigned short)(out[j] >> 16);
    }
}
// EPI_SILU: features 2j and 2j + 1 are gate j and up j (rounded to fp16 like every GEMM result), one word of the staged rows; silu
// and product in fp32 go to the store buffer [row][64]. Rolled over the staged words: evaluated on the registers before they are
// staged, fully unrolled, the same arithmetic cost 27 us more for 512 x 4096 x 22016 (16 evaluations in each of nine places of the code).
__device__ __forceinline__ void epi_silu(const uint8_t* staged, uint8_t* buf, int etid) {
    const __half2* src = reinterpret_cast<const __half2*>(staged);
    __half* dst = reinterpret_cast<__half*>(buf);
    constexpr int U = 8;   // in flight per thread
#pragma unroll 1
    for (int i = etid; i < kOutRows * kBN / 2; i += U * kEpiWarps * 32) {
        float2 gu[U];
#pragma unroll
        for (int k = 0; k < U; k++) gu[k] = __half22float2(src[i + k * kEpiWarps * 32]);
#pragma unroll
        for (int k = 0; k < U; k++) dst[i + k * kEpiWarps * 32] = __float2half(silu_mul(gu[k].x, gu[k].y));
    }
}
__device__ __forceinline__ void epi_load_residual(uint32_t* res, const __half* x, int c0, int rows, size_t ld) {
    const unsigned short* p = reinterpret_cast<const unsigned short*>(x) + (size_t)c0 * ld;
#pragma unroll
    for (int j = 0; j < 16; j++) {
        uint32_t a = 0, b = 0;
        if (c0 + 2 * j < rows) a = *p;
        p += ld;
        if (c0 + 2 * j + 1 < rows) b = *p;
        p += ld;
        res[j] = a | (b << 16);
    }
}

// PLAIN_Y: y does not start on 16 bytes, which a tensor copy cannot write (a template argument: as a branch it took 0.3 us of the
// 25 of 64 x 4096 x 22016).
template <bool INTERLEAVED, int EPI, bool PLAIN_Y>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
q4_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
               const GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sB = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sP = sB + (size_t)p.stages * 2 * p.slab_bytes;
    __shared__ uint64_t full_p[kMaxP], empty_p[kMaxP], full[kMaxStages], empty[kMaxStages], tmem_full, tmem_empty, drained;
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_flag, s_gave_up;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    if (tid == 0) {
        for (int s = 0; s < kMaxP; s++) { mb_init(&full_p[s], 1); mb_init(&empty_p[s], kConvWarps); }
        for (int s = 0; s < kMaxStages; s++) { mb_init(&full[s], 9); mb_init(&empty[s], 1); }   // (four converter warps of each CTA, X copies)
        mb_init(&tmem_full, 1);
        mb_init(&tmem_empty, 2 * kEpiWarps);
        mb_init(&drained, 1);
        s_gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {   // all of the tensor memory, in both CTAs (one CTA per SM: nobody else holds any)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem_base)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // both CTAs' barriers and tensor memory are ready before either is touched from the other side
    tc_fence_after();
    const uint32_t tmem_base = *(volatile uint32_t*)&s_tmem_base;
    // everything above overlaps the tail of the previous kernel on the stream (programmatic dependent launch) where both fit an SM,
    // that is, not behind another of these, whose shared memory fills it; from here on this kernel reads what that kernel wrote. The warp of the
    // packed words starts before: a model's words are nobody's result by then, a caller's may be that kernel's (q4_gemm_interleave_weights)
    // and come as far as L2 only. us, both behind the wait, the caller's and the model's form: 64 x 4096 x 22016 back to back 25.6, 24.7, 24.9;
    // 78 tokens of two 13B layers 309.5, 308.9, 307.2
    // The kernel behind is let in by warps that have waited (the first signal of a CTA counts for all of it): its words are read ahead of its own wait,
    // and may be the result of the kernel in front of this one.
    if (warp != 0) {
        griddep_wait();
        griddep_launch_dependents();
    }
    Segments seg(p, pair, pairs);

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0 && lane == 0) {
            // ===================== packed weights =====================
            int ps = 0;
            uint32_t ph = 1;
            unsigned issued = 0;
            bool ok = true, more = seg.next();
            if (!p.settled) {
                for (int c = seg.c0; more && c < seg.c1 && c < seg.c0 + p.np; c++) tma_prefetch_2d(&map_w, c * (kChunkK / 8), (seg.tile / p.m_tiles) * kPairN + rank * kBN);
                griddep_wait();
            }
            for (; ok && more; more = seg.next()) {
                const int row = (seg.tile / p.m_tiles) * kPairN + rank * kBN;
                for (int c = seg.c0; c < seg.c1; c++) {
                    if (!mb_wait(&empty_p[ps], ph, p.status, 0x100)) { ok = false; break; }
                    mb_expect_tx(&full_p[ps], kPStageBytes);
                    tma_load_2d(sP + (size_t)ps * kPStageBytes, &map_w, c * (kChunkK / 8), row, &full_p[ps]);
                    issued++;
                    if (++ps == p.np) { ps = 0; ph ^= 1; }
                }
            }
            if (!ok) s_gave_up = 1;
            if (!ok)   // the newest copy of every ring position may still be in flight
                for (unsigned i = issued > (unsigned)p.np ? issued - p.np : 0; i < issued; i++) mb_drain(&full_p[i % p.np], (i / p.np) & 1);
        } else if (warp == 1 && lane == 0) {
            // ===================== X slabs =====================
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            const int half_rows = p.MT / 2;
            while (ok && seg.next()) {
                const int row = (seg.tile % p.m_tiles) * p.MT + rank * half_rows;
                for (int b = seg.c0 * 2; b < seg.c1 * 2; b++) {   // 128-input blocks
                    if (!mb_wait(&empty[s], ph, p.status, 0x200)) { ok = false; break; }
                    if (rank == 0) mb_expect_tx(&full[s], 4 * p.slab_bytes);   // (the peer's bytes may be counted before: same phase)
                    uint8_t* dst = sB + (size_t)s * 2 * p.slab_bytes;
                    const uint32_t bar = leader_addr(&full[s]);
                    tma_load_2d_pair(dst, &map_x, b * kBlockK, row, bar);
                    tma_load_2d_pair(dst + p.slab_bytes, &map_x, b * kBlockK + kSlabK, row, bar);
                    if (++s == p.stages) { s = 0; ph ^= 1; }
                }
            }
            if (!ok) s_gave_up = 1;   // (its copies report to the leader, whose barriers may never complete: waited out below)
        } else if (warp == 2 && rank == 0) {
            // ===================== MMA issuer =====================
            // The whole warp walks the loop with warp-uniform values (descriptors and addresses then live in uniform registers) and
            // one elected lane issues.
            const uint32_t idesc = umma_idesc(p.MT);
            const uint64_t bdesc0 = umma_desc(smem_addr(sB));
            const bool issuer = elect_one();
            int st = 0;
            uint32_t ph = 0, pe = 1;
            bool ok = true;
            while (ok && seg.next()) {
                if (!warp_wait(&tmem_empty, pe, p.status, 0x300)) { ok = false; break; }   // both epilogues have drained the accumulator
                pe ^= 1;
                uint32_t accumulate = 0;
                const int blocks = (seg.c1 - seg.c0) * (kChunkK / kBlockK);
                for (int b = 0; b < blocks; b++) {
                    if (!warp_wait(&full[st], ph, p.status, 0x400)) { ok = false; break; }
                    tc_fence_after();
                    if (issuer) {
                        const uint32_t at = tmem_base + p.MT + st * kAStageCols;
                        const uint64_t bd = bdesc0 + (uint64_t)((st * 2 * p.slab_bytes) >> 4);
#pragma unroll
                        for (int k16 = 0; k16 < kBlockK / 16; k16++)
                            tc_mma_f16_pair(tmem_base, at + k16 * 8, bd + (k16 >= 4 ? p.slab_bytes >> 4 : 0) + 2 * (k16 & 3), idesc, k16 == 0 ? accumulate : 1u);
                        tc_commit_pair(&empty[st]);   // arrives when these MMAs have read their operands
                        if (b == blocks - 1) tc_commit_pair(&tmem_full);
                    }
                    __syncwarp();
                    accumulate = 1;
                    if (++st == p.stages) { st = 0; ph ^= 1; }
                }
            }
            if (!ok && issuer) {   // MMAs in flight read shared memory and report to both CTAs: let them finish
                s_gave_up = 1;
                tc_commit_pair(&drained);
                mb_drain(&drained, 0);
            }
            __syncwarp();
        }
    } else if (warp < kEpiWarp0) {
        // ===================== converters =====================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
        const int wg = (warp - kConvWarp0) >> 2;              // this warpgroup takes block wg of every chunk
        const int r = (warp & 3) * 32 + lane;                 // feature row of this CTA's half = tensor-memory lane
        const uint32_t a_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + p.MT;
        const int sw = r & 7;
        int ps = 0;
        uint32_t pp = 0, pe = 1;
        int sa = wg;   // its blocks go to every second stage of the ring
        bool ok = true;
        while (ok && seg.next()) {
            const int n = (seg.tile / p.m_tiles) * kPairN + rank * kBN + r;
            const uint32_t* zrow = p.zeros + (size_t)n * p.PZ;
            const __half* srow = p.scales + (size_t)n * p.G;
            // Zero points and scales: one zeros word covers four chunks, and their four scales of this warpgroup's blocks are
            // requested with it, one span of four chunks ahead (a load consumed in the block it is issued for would stall
            // the warp for a memory latency per block). Beyond the matrix both are 0, and so are the weights.
            uint32_t z_next = 0, z_cur = 0;
            __half s_next[4], s_cur[4];
            auto fetch_meta = [&](int span) {
                const int g0 = span * 8;
                z_next = 0;
#pragma unroll
                for (int i = 0; i < 4; i++) s_next[i] = __float2half(0.f);
                if (n < p.N && g0 < p.G) {
                    z_next = __ldg(zrow + span);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (g0 + 2 * i + wg < p.G) s_next[i] = __ldg(srow + g0 + 2 * i + wg);
                }
            };
            const int span_end = (seg.c1 - 1) >> 2;
            fetch_meta(seg.c0 >> 2);
            for (int span = seg.c0 >> 2; span <= span_end && ok; span++) {
                z_cur = z_next;
#pragma unroll
                for (int i = 0; i < 4; i++) s_cur[i] = s_next[i];
                if (span < span_end) fetch_meta(span + 1);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                const int c = span * 4 + i;
                if (c < seg.c0 || c >= seg.c1) continue;
                const uint32_t z = (z_cur >> (8 * i + 4 * wg)) & 0xFu;
                const __half2 s2 = __half2half2(s_cur[i]);
                const __half2 zlo = u2h2((0x6400u | z) * 0x00010001u), zhi = u2h2((0x5400u | (z << 4)) * 0x00010001u);
                // Both the words and the stage, one vote for the two: usually neither has to be waited for (a vote at each costs
                // 2.5 % at 64 rows, where this loop sets the pace).
                if (!__all_sync(0xffffffffu, mb_try(&full_p[ps], pp) & mb_try(&empty[sa], pe))) {
                    ok = warp_wait(&full_p[ps], pp, p.status, 0x600) && warp_wait(&empty[sa], pe, p.status, 0x700);
                    if (!ok) break;
                }
                const uint8_t* src = sP + (size_t)ps * kPStageBytes + r * 128;
                uint4 pk[4];
#pragma unroll
                for (int j = 0; j < 4; j++) pk[j] = *reinterpret_cast<const uint4*>(src + (((wg * 4 + j) ^ sw) << 4));
                uint32_t o[32];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    dequant8<INTERLEAVED>(pk[j].x, zlo, zhi, s2, o + 16 * j);
                    dequant8<INTERLEAVED>(pk[j].y, zlo, zhi, s2, o + 16 * j + 4);
                    dequant8<INTERLEAVED>(pk[j].z, zlo, zhi, s2, o + 16 * j + 8);
                    dequant8<INTERLEAVED>(pk[j].w, zlo, zhi, s2, o + 16 * j + 12);
                }
                tc_fence_after();
                tc_st32(a_lane + sa * kAStageCols, o);
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    dequant8<INTERLEAVED>(pk[2 + j].x, zlo, zhi, s2, o + 16 * j);
                    dequant8<INTERLEAVED>(pk[2 + j].y, zlo, zhi, s2, o + 16 * j + 4);
                    dequant8<INTERLEAVED>(pk[2 + j].z, zlo, zhi, s2, o + 16 * j + 8);
                    dequant8<INTERLEAVED>(pk[2 + j].w, zlo, zhi, s2, o + 16 * j + 12);
                }
                tc_st32(a_lane + sa * kAStageCols + 32, o);
                tc_st_wait();
                tc_fence_before();
                __syncwarp();
                // The staging slot is given back only here, behind the tensor-memory stores that consumed its words: with the arrive
                // right behind the loads a few feature rows were wrong in one launch out of hundreds (the slot's next copy had
                // landed before all of its reads were done).
                if (lane == 0) {
                    mb_arrive_cluster(leader_addr(&full[sa]));
                    mb_arrive(&empty_p[ps]);
                }
                if (++ps == p.np) { ps = 0; pp ^= 1; }
                sa += 2;
                if (sa >= p.stages) { sa -= p.stages; pe ^= 1; }
                }
            }
        }
        if (!ok) s_gave_up = 1;
    } else {
        // ===================== epilogue =====================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        const int qtr = warp & 3;              // the tensor-memory lane quarter this warp may read
        const int r = qtr * 32 + lane;
        const int etid = (warp - kEpiWarp0) * 32 + lane;
        const uint32_t t_lane = tmem_base + ((uint32_t)(qtr * 32) << 16);
        const uint32_t empty_addr = leader_addr(&tmem_empty);
        const size_t ld = p.N;
        const int MT = p.MT;
        auto release = [&]() {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive_cluster(empty_addr);
        };
        // the accumulator is complete; the four warps meet at named barriers from here on, so they go on or give up together
        auto tile_ready = [&](uint32_t parity) {
            const uint32_t mine = warp_wait(&tmem_full, parity, p.status, 0x800);
            uint32_t all;
            asm volatile("{ .reg .pred p, q; setp.ne.u32 q, %1, 0; bar.red.and.pred p, 2, %2, q; selp.u32 %0, 1, 0, p; }" : "=r"(all) : "r"(mine), "n"(kEpiWarps * 32) : "memory");
            if (!all) s_gave_up = 1;
            return all != 0;
        };
        auto partial_of = [&](int pr, bool head) { return reinterpret_cast<float4*>(p.partials) + ((size_t)((pr * 2 + (head ? 1 : 0)) * 2 + rank) * (MT / 4)) * kBN + r; };
        // Y leaves through shared memory: 32 rows are staged and written by one tensor copy (rows and columns beyond Y are
        // clipped there) while the next 32 are staged. Storing from the registers (a lane is a feature, so two bytes per lane and
        // row) took 34000 to 40000 clocks per 256-row tile, more than its 32 chunks of MMAs.
        uint8_t* sY = sB + kRingBytes;   // two store buffers; EPI_SILU: the staged gates and ups, and two store buffers of half the size
        int buf = 0;
        auto put = [&](const uint32_t* out, int nt, int row0, int rows_left) {   // all epilogue threads; rows_left > 0
            uint8_t* store = EPI == EPI_SILU ? sY + kOutBytes + buf * (kOutBytes / 2) : sY + buf * kOutBytes;
            if (etid == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");   // the copy that read this buffer last is done
            asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");
            if (EPI == EPI_SILU) {
                epi_stage(out, sY, r);
                asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");
                epi_silu(sY, store, etid);
            } else {
                epi_stage(out, store, r);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");
            if (PLAIN_Y) {   // (the next chunk is staged in the other buffer, behind a barrier that follows these reads)
                const int col = nt * kPairN + rank * kBN, cols = min(kBN, p.N - col);
                const __half* src = reinterpret_cast<const __half*>(store);
#pragma unroll 1
                for (int i = etid; i < kOutRows * kBN; i += kEpiWarps * 32)
                    if (i / kBN < rows_left && i % kBN < cols) p.y[(size_t)(row0 + i / kBN) * p.N + col + i % kBN] = src[i];
            } else if (etid == 0) {
                const int col = (nt * kPairN + rank * kBN) / (EPI == EPI_SILU ? 2 : 1);
                if (rows_left > 0 && nt * kPairN + rank * kBN < p.N)
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(&map_y), "r"(smem_addr(store)), "r"(col), "r"(row0)
                                 : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            buf ^= 1;
        };
        uint32_t pf = 0;
        while (seg.next()) {
            const int nt = seg.tile / p.m_tiles, mt = seg.tile - nt * p.m_tiles;
            const int n = nt * kPairN + rank * kBN + r;
            const int rows = min(MT, p.M - mt * MT), my_rows = n < p.N ? rows : 0;
            const __half* res = EPI == EPI_RESIDUAL ? p.residual + (size_t)mt * MT * ld + n : nullptr;
            const bool whole = seg.c0 == 0 && seg.c1 == p.n_chunks;
            if (whole) {
                // drain everything into registers (packed halfs), give the accumulator back, then store: the stores run
                // under the next tile's MMAs. The residual (which may be y itself) is in registers before the wait.
                constexpr int W = 16;
                uint32_t out[W * 8];
                if (EPI == EPI_RESIDUAL) {
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (32 * i < MT) epi_load_residual(out + W * i, res, 32 * i, my_rows, ld);
                }
                if (!tile_ready(pf)) break;
                pf ^= 1;
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    if (32 * i < MT) {
                        uint32_t v[32];
                        float f[32];
                        tc_ld32(t_lane + 32 * i, v);
#pragma unroll
                        for (int j = 0; j < 32; j++) f[j] = __uint_as_float(v[j]);
                        epi_pack<EPI>(f, out + W * i, p.residual_scale, out + W * i);
                    }
                }
                release();
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (32 * i < MT) put(out + W * i, nt, mt * MT + 32 * i, rows - 32 * i);
                continue;
            }
            // ---- a tile shared with other pairs: partial sums in K order, finished by the CTA that arrives last ----
            const long long t0 = (long long)seg.tile * p.n_chunks;
            const int first = pair_of(t0, p.total_chunks, pairs), last = pair_of(t0 + p.n_chunks - 1, p.total_chunks, pairs);
            int* counter = p.counters + seg.tile * 2 + rank;
            if (!tile_ready(pf)) break;
            pf ^= 1;
            tc_fence_after();
            if (etid == 0) {
                int seen;
                asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
                s_flag = seen == last - first;
            }
            asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");
            bool finish = s_flag != 0, own_in_tmem = finish;
            if (!finish) {
                float4* mine = partial_of(pair, pair == first);
#pragma unroll 1
                for (int c0 = 0; c0 < MT; c0 += 32) {
                    uint32_t v[32];
                    tc_ld32(t_lane + c0, v);
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        __stcg(mine + (size_t)(c0 / 4 + j) * kBN, make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])));
                }
                release();
                __threadfence();
                asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");   // (all have read s_flag and written their partials)
                if (etid == 0) s_flag = atomicAdd(counter, 1) == last - first;
                asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");
                finish = s_flag != 0;
            }
            if (finish) {
                __threadfence();
                // Pieces (32 columns of one stored part) in the order they are added, two requested ahead of the sum whichever part they belong
                // to. With the next columns of the first two parts ahead the third and fourth were a latency of L2 each: 77 x 13824 x
                // 5120 in three parts 25.5 us, 24.3 so. (Three or four ahead spill: no gain.)
                const int others = last - first + (own_in_tmem ? 0 : 1);
                constexpr int kAhead = 2;
                float4 ring[kAhead][8];
                float acc[32];
                uint32_t rs[16], out[16];
                int fetch_c = 0, fetch_j = 0, c0 = 0, j = 0;
                auto fetch_next = [&](float4 (&v)[8]) {
                    if (fetch_c >= MT) return;
                    const int pr = first + fetch_j + (own_in_tmem && first + fetch_j >= pair ? 1 : 0);
                    const float4* part = partial_of(pr, pr == first) + (size_t)(fetch_c / 4) * kBN;
#pragma unroll
                    for (int i = 0; i < 8; i++) v[i] = __ldcg(part + (size_t)i * kBN);
                    if (++fetch_j == others) { fetch_j = 0; fetch_c += 32; }
                };
                auto add_own = [&]() {
                    uint32_t v[32];
                    tc_ld32(t_lane + c0, v);
#pragma unroll
                    for (int i = 0; i < 32; i++) acc[i] += __uint_as_float(v[i]);
                };
#pragma unroll
                for (int u = 0; u < kAhead; u++) fetch_next(ring[u]);
#pragma unroll 1
                while (c0 < MT) {
#pragma unroll
                    for (int u = 0; u < kAhead; u++) {
                        if (c0 >= MT) break;
                        if (j == 0) {
                            if (EPI == EPI_RESIDUAL) epi_load_residual(rs, res, c0, my_rows, ld);
#pragma unroll
                            for (int i = 0; i < 32; i++) acc[i] = 0.f;
                            if (own_in_tmem && pair == first) add_own();
                        }
#pragma unroll
                        for (int i = 0; i < 8; i++) { acc[4 * i] += ring[u][i].x; acc[4 * i + 1] += ring[u][i].y; acc[4 * i + 2] += ring[u][i].z; acc[4 * i + 3] += ring[u][i].w; }
                        fetch_next(ring[u]);
                        j++;
                        if (own_in_tmem && first + j == pair) add_own();   // its place in K order
                        if (j == others) {
                            epi_pack<EPI>(acc, rs, p.residual_scale, out);
                            put(out, nt, mt * MT + c0, rows - c0);
                            c0 += 32;
                            j = 0;
                        }
                    }
                }
                if (own_in_tmem) release();
                if (etid == 0) *counter = 0;   // ready for the next launch
            }
            asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");   // s_flag is rewritten by the next segment
        }
        if (etid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // Y is written before this CTA leaves
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (s_gave_up) {
        // Copies or MMAs may be in flight in this CTA only when its epilogue has not seen all of its tiles, and then it gave up as
        // well: a millisecond is far beyond a copy's flight time or a tile's MMAs.
        const unsigned long long t0 = gtimer();
        while (gtimer() - t0 < 1000000ULL) {}
        __syncwarp();
    }
    cluster_sync_all();   // no CTA leaves while the other may still report to its barriers
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// dst word: nibble i holds input order[i] of the same 8 inputs, order = 0,2,4,6,1,3,5,7
__global__ void interleave_kernel(uint32_t* dst, const uint32_t* src, size_t nwords) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nwords; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t w = src[i];
        const uint32_t even = w & 0x0F0F0F0Fu, odd = (w >> 4) & 0x0F0F0F0Fu;   // bytes: inputs 0,2,4,6 / 1,3,5,7
        // pack the four bytes of each into four consecutive nibbles
        const uint32_t e = (even & 0xFu) | ((even >> 4) & 0xF0u) | ((even >> 8) & 0xF00u) | ((even >> 12) & 0xF000u);
        const uint32_t o = (odd & 0xFu) | ((odd >> 4) & 0xF0u) | ((odd >> 8) & 0xF00u) | ((odd >> 12) & 0xF000u);
        dst[i] = e | (o << 16);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
std::mutex g_encode_mu;
EncodeTiledFn g_encode = nullptr;

int get_encode(EncodeTiledFn* out) {
    std::lock_guard<std::mutex> lk(g_encode_mu);
    if (!g_encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        Q4_CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
        if (!fn || qres != cudaDriverEntryPointSuccess) return Q4_ERR_CUDA;
        g_encode = (EncodeTiledFn)fn;
    }
    *out = g_encode;
    return Q4_OK;
}

int make_map_2d(CUtensorMap* map, CUtensorMapDataType dt, int elem_bytes, const void* base, uint64_t inner, uint64_t outer, uint64_t row_bytes, uint32_t box_inner,
                uint32_t box_outer, bool swizzle = true) {
    EncodeTiledFn enc;
    if (int e = get_encode(&enc)) return e;
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t estr[2] = {1, 1};
    (void)elem_bytes;
    const CUresult r = enc(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { fprintf(stderr, "q4 gemm: cuTensorMapEncodeTiled failed (%d)\n", (int)r); return Q4_ERR_CUDA; }
    return Q4_OK;
}

// Workspace layout, the same for every shape, so that calls of different shapes can share one workspace (the tile counters
// must read zero at the start of every call): status words | tile counters | fp32 partial sums.
constexpr size_t kWsHeader = 256;
constexpr int kWsMaxTiles = 16384;   // (two counters per tile of 256 features: 8192 tiles of 256 x 256 outputs)
constexpr size_t kWsPartials = kWsHeader + sizeof(int) * kWsMaxTiles;

struct GemmPlan { int MT, m_tiles, n_tiles, n_chunks, pairs, stages, np, slab; long long total; };

// Batch tile and number of pairs, by an estimate of the slowest pair's time over all of them, in us. The lines were fitted to 70 shapes
// (K and N of the 7B, 13B and 70B projections, 24 to 512 rows) with all their tiles and 5 to 12 numbers of pairs each; the plan it
// picks is 0.4 % off the best of them on average, 5 % at most. (Where only shares of equal length counted as aligned it was 1.4 and
// 14 %: 64 x 11008 x 4096 on 68 pairs, five parts to a tile, 19.5 us, on 64 pairs with four 18.0; 77 x 5120 x 5120 16.7, 16.0.)
//   chunk    a 256-input chunk: 4.6 ns per batch row on the tensor pipe and 0.08 us whatever the rows, 0.72 us at least (issue of its 16
//            MMAs, conversion of its 128 x 256 weights). With 5 ns per row and nothing else, eight tiles of 160 rows were as good as five of
//            256: 1200 x 28672 x 8192 470 us, 443 so; 1200 x 8192 x 57344 851, 793; 900 x 28672 x 8192 353, 331
//   segment  each further tile that a share touches: its turn at the accumulator
//   drain    the last tile's output, which is not hidden by anything: 9 ns per row
//   split    a tile cut by a share boundary: a partial tile written, counted and, by the last CTA, one read per other contributor at
//            9 ns per row and 0.25 us, which is why 64 pairs with every tile in two or four parts often beat 74 (a multiple of the
//            number of tiles does that whatever the chunks: shares are dealt out balanced, pair_of); other shares meet at other times
// Rings: operand stages as tensor memory allows, the shared memory that their X slabs leave for packed weights (at few rows
// the kernel is a weight stream: ten 16 KB copies in flight per SM cover HBM's latency).
GemmPlan make_plan(int M, int K, int N, int sms) {
    GemmPlan g = {};
    g.n_tiles = q4_div_up(N, kPairN);
    g.n_chunks = q4_div_up(K, kChunkK);
    const int max_pairs = sms / 2 > 0 ? sms / 2 : 1;
    double best = 1e300;
    int last_mt = 0;
    for (int m_tiles = q4_div_up(M, kMaxMT); m_tiles <= q4_div_up(M, kMaxMT) * 8; m_tiles++) {
        const int mt = q4_div_up(q4_div_up(M, m_tiles), 32) * 32;
        if (mt == last_mt || (long long)g.n_tiles * q4_div_up(M, mt) * 2 > kWsMaxTiles) continue;
        last_mt = mt;
        const int mtl = q4_div_up(M, mt);
        const int tiles = g.n_tiles * mtl;
        const long long total = (long long)tiles * g.n_chunks;
        const double t_rows = 0.08 + 0.0046 * mt, t_chunk = t_rows > 0.72 ? t_rows : 0.72;
        for (int P = (int)(total < max_pairs ? total : max_pairs); P >= 1; P--) {
            const long long share = (total + P - 1) / P;
            if (share * t_chunk >= best) break;   // fewer pairs only take longer from here on
            const bool whole = tiles % P == 0, aligned = P % tiles == 0;   // no share, or every tile, starts where a tile does
            double cost = share * t_chunk + 0.009 * mt + 0.4 * (q4_div_up((int)share, g.n_chunks) - (whole || aligned ? 1 : 0));
            if (!whole) {   // contributors of a tile, at most
                const long long parts = aligned ? P / tiles : share >= g.n_chunks ? 2 : (g.n_chunks - 2) / share + 2;
                cost += 1.2 + 0.015 * mt + (parts - 1) * (0.25 + 0.009 * mt) + (aligned ? 0.0 : 0.8);
            }
            if (cost < best) { best = cost; g.pairs = P; g.MT = mt; g.m_tiles = mtl; g.total = total; }
        }
    }
    if (g.pairs == 0) return g;
    g.slab = g.MT / 2 * kSlabK * 2;
    g.stages = (kTmemCols - g.MT) / kAStageCols < kMaxStages ? (kTmemCols - g.MT) / kAStageCols : kMaxStages;
    g.np = (kRingBytes - g.stages * 2 * g.slab) / kPStageBytes < kMaxP ? (kRingBytes - g.stages * 2 * g.slab) / kPStageBytes : kMaxP;
    return g;
}

int sm_count(int* out) {
    int dev = 0;
    Q4_CUDA_TRY(cudaGetDevice(&dev));
    Q4_CUDA_TRY(cudaDeviceGetAttribute(out, cudaDevAttrMultiProcessorCount, dev));
    return Q4_OK;
}

template <bool IL, int EPI, bool PLAIN_Y = false>
int launch_gemm(cudaStream_t s, int pairs, const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& my, const GemmParams& p) {
    const size_t smem = kRingBytes + 2 * kOutBytes + 1024;
    Q4_CUDA_TRY(cudaFuncSetAttribute(q4_gemm_kernel<IL, EPI, PLAIN_Y>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    Q4Launch L(dim3(2 * pairs), dim3(kGemmThreads), smem, s);   // programmatic dependent launch: the prologue overlaps the previous kernel's tail
    Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, q4_gemm_kernel<IL, EPI, PLAIN_Y>, mw, mx, my, p));
    return Q4_OK;
}

}  // namespace

// Grows with M only (the largest batch tile of up to M rows), so that a workspace for M rows serves every smaller call.
extern "C" size_t q4_matmul_q4_batched_workspace_bytes(int M, int K, int N) {
    if (M <= 0 || K <= 0 || N <= 0) return 0;
    int sms = 148;
    sm_count(&sms);
    const int mt = M >= kMaxMT ? kMaxMT : q4_div_up(M, 32) * 32;
    return kWsPartials + (size_t)(sms / 2 > 0 ? sms / 2 : 1) * 4 * kBN * mt * sizeof(float);
}

extern "C" int q4_gemm_interleave_weights(void* stream, uint32_t* dst, const uint32_t* weight, int K, int N) {
    if (!dst || !weight || K <= 0 || N <= 0) return Q4_ERR_INVALID;
    const size_t nwords = (size_t)N * q4_pw(K);
    interleave_kernel<<<148 * 8, 256, 0, (cudaStream_t)stream>>>(dst, weight, nwords);
    Q4_CUDA_TRY(cudaGetLastError());
    return Q4_OK;
}

extern "C" int q4_matmul_q4_batched(void* stream, uint16_t* y, const uint16_t* x, const q4_qweight* w, const uint32_t* weight_interleaved, int M, int K,
                                    int N, void* workspace, size_t workspace_bytes) {
    return q4_matmul_q4_batched_residual(stream, y, x, w, weight_interleaved, M, K, N, nullptr, 0.f, workspace, workspace_bytes);
}

extern "C" int q4_matmul_q4_batched_residual(void* stream, uint16_t* y, const uint16_t* x, const q4_qweight* w, const uint32_t* weight_interleaved, int M,
                                             int K, int N, const uint16_t* residual, float residual_scale, void* workspace, size_t workspace_bytes) {
    return q4_gemm_launch(stream, y, x, w, weight_interleaved, M, K, N, residual, residual_scale, false, false, workspace, workspace_bytes);
}

int q4_gemm_launch(void* stream, uint16_t* y, const uint16_t* x, const q4_qweight* w, const uint32_t* weight_interleaved, int M, int K, int N,
                   const uint16_t* residual, float residual_scale, bool silu, bool settled, void* workspace, size_t workspace_bytes) {
    if (!y || !x || !w || !w->zeros || !w->scales || !workspace || M <= 0 || K <= 0 || N <= 0) return Q4_ERR_INVALID;
    if (!w->weight && !weight_interleaved) return Q4_ERR_INVALID;
    if ((K % 128) || (N % 8)) return Q4_ERR_UNSUPPORTED_SIZE;
    if (silu && (N % 16)) return Q4_ERR_UNSUPPORTED_SIZE;
    if (((uintptr_t)x & 15) || ((uintptr_t)y & 1) || ((uintptr_t)w->weight & 15) || ((uintptr_t)weight_interleaved & 15) || ((uintptr_t)workspace & 15)) return Q4_ERR_INVALID;
    if (workspace_bytes < q4_matmul_q4_batched_workspace_bytes(M, K, N)) return Q4_ERR_LIMIT;
    cudaStream_t s = (cudaStream_t)stream;
    int sms = 0;
    if (int e = sm_count(&sms)) return e;
    const GemmPlan g = make_plan(M, K, N, sms);
    GemmParams p;
    p.zeros = w->zeros;
    p.scales = (const __half*)w->scales;
    p.residual = (const __half*)residual;
    p.residual_scale = residual_scale;
    p.status = (int*)workspace;
    p.counters = (int*)((char*)workspace + kWsHeader);
    p.partials = (float*)((char*)workspace + kWsPartials);
    if (g.pairs == 0) return Q4_ERR_UNSUPPORTED_SIZE;   // more tiles than counters
    p.M = M; p.K = K; p.N = N;
    p.G = q4_groups(K);
    p.PZ = q4_pz(K);
    p.MT = g.MT; p.m_tiles = g.m_tiles; p.n_chunks = g.n_chunks; p.total_chunks = g.total;
    p.settled = settled;
    p.stages = g.stages; p.np = g.np; p.slab_bytes = g.slab;
    // (status word and tile counters start at zero: the caller zeroes the workspace once, the kernel leaves the counters at
    // zero; after a recorded time-out the caller zeroes it again)
    CUtensorMap mw, mx, my;
    const uint32_t* wsrc = weight_interleaved ? weight_interleaved : w->weight;
    if (int e = make_map_2d(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, wsrc, (uint64_t)q4_pw(K), (uint64_t)N, (uint64_t)q4_pw(K) * 4, kChunkK / 8, kBN)) return e;
    if (int e = make_map_2d(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, kSlabK, (uint32_t)(g.MT / 2))) return e;
    const int n_out = silu ? N / 2 : N;
    p.y = (__half*)y;
    const bool il = weight_interleaved != nullptr;
    if ((uintptr_t)y & 15) {
        if (silu) return Q4_ERR_INVALID;   // (row buffers of this library only)
        if (residual) return il ? launch_gemm<true, EPI_RESIDUAL, true>(s, g.pairs, mw, mx, mx, p) : launch_gemm<false, EPI_RESIDUAL, true>(s, g.pairs, mw, mx, mx, p);
        return il ? launch_gemm<true, EPI_PLAIN, true>(s, g.pairs, mw, mx, mx, p) : launch_gemm<false, EPI_PLAIN, true>(s, g.pairs, mw, mx, mx, p);
    }
    if (int e = make_map_2d(&my, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, y, (uint64_t)n_out, (uint64_t)M, (uint64_t)n_out * 2, silu ? kBN / 2 : kBN, kOutRows, false)) return e;
    if (silu) return il ? launch_gemm<true, EPI_SILU>(s, g.pairs, mw, mx, my, p) : Q4_ERR_INVALID;
    if (residual) return il ? launch_gemm<true, EPI_RESIDUAL>(s, g.pairs, mw, mx, my, p) : launch_gemm<false, EPI_RESIDUAL>(s, g.pairs, mw, mx, my, p);
    return il ? launch_gemm<true, EPI_PLAIN>(s, g.pairs, mw, mx, my, p) : launch_gemm<false, EPI_PLAIN>(s, g.pairs, mw, mx, my, p);
}

extern "C" int q4_matmul_q4_batched_status(void* stream, const void* workspace) {
    if (!workspace) return Q4_ERR_INVALID;
    int st[2] = {0, 0};
    Q4_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    Q4_CUDA_TRY(cudaMemcpy(st, workspace, sizeof(st), cudaMemcpyDeviceToHost));
    if (st[0]) fprintf(stderr, "q4 gemm: a bounded device-side wait ran out (status %d, location 0x%x)\n", st[0], st[1]);
    return st[0];
}

// Measurement hook: q4_matmul_q4_batched over `nmat` distinct weight matrices of one shape, captured as one CUDA graph
// and replayed `reps` times between two events on `stream` (weights from HBM rather than L2, no launch gaps timed).
extern "C" int q4_time_matmul_q4_batched(void* stream, uint16_t* y, const uint16_t* x, const q4_qweight* mats, const uint32_t* const* interleaved, int nmat,
                                         int M, int K, int N, void* workspace, size_t workspace_bytes, int reps, double* us_per_launch) {
    if (!mats || nmat < 1 || reps < 1 || !us_per_launch) return Q4_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    Q4_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    int e = Q4_OK;
    for (int i = 0; i < nmat && e == Q4_OK; i++)
        e = q4_matmul_q4_batched(s, y, x, &mats[i], interleaved ? interleaved[i] : nullptr, M, K, N, workspace, workspace_bytes);
    cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (e != Q4_OK) { if (graph) cudaGraphDestroy(graph); return e; }
    Q4_CUDA_TRY(ce);
    Q4_CUDA_TRY(cudaGraphInstantiate(&exec, graph, 0));
    cudaEvent_t e0, e1;
    Q4_CUDA_TRY(cudaEventCreate(&e0));
    Q4_CUDA_TRY(cudaEventCreate(&e1));
    for (int r = 0; r < 3; r++) Q4_CUDA_TRY(cudaGraphLaunch(exec, s));
    Q4_CUDA_TRY(cudaEventRecord(e0, s));
    for (int r = 0; r < reps; r++) Q4_CUDA_TRY(cudaGraphLaunch(exec, s));
    Q4_CUDA_TRY(cudaEventRecord(e1, s));
    Q4_CUDA_TRY(cudaEventSynchronize(e1));
    float ms = 0.f;
    Q4_CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaGraphExecDestroy(exec);
    cudaGraphDestroy(graph);
    *us_per_launch = 1e3 * ms / ((double)reps * nmat);
    return Q4_OK;
}

#ifdef Q4_TEST_BUILD
// The gate / up form by itself (the product reaches it through prompts only). `weight` is in file layout, rows 2j and 2j + 1 gate j and
// up j; `interleaved` as from q4_gemm_interleave_weights; y is [M][N / 2].
extern "C" int q4_test_gemm_silu(void* stream, uint16_t* y, const uint16_t* x, const q4_qweight* w, const uint32_t* interleaved, int M, int K, int N,
                                 void* workspace, size_t workspace_bytes) {
    return q4_gemm_launch(stream, y, x, w, interleaved, M, K, N, nullptr, 0.f, true, false, workspace, workspace_bytes);
}
// A writer that lets the next kernel in at once and writes late: src to dst, `ns` nanoseconds after it has started (bounded by a number of turns too).
// Few blocks, without shared memory, so that the kernel behind it finds room beside them.
static __global__ void __launch_bounds__(256) test_write_late_kernel(uint32_t* dst, const uint32_t* src, size_t n, unsigned long long ns) {
    griddep_launch_dependents();
    const unsigned long long t0 = gtimer();
    for (int i = 0; i < 1000000 && gtimer() - t0 < ns; i++) {}
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) dst[i] = src[i];
}
extern "C" int q4_test_write_late(void* stream, uint32_t* dst, const uint32_t* src, size_t n, unsigned long long ns) {
    test_write_late_kernel<<<8, 256, 0, (cudaStream_t)stream>>>(dst, src, n, ns);
    Q4_CUDA_TRY(cudaGetLastError());
    return Q4_OK;
}
// What make_plan picks on a GPU with `sms` SMs (host only): batch tile and number of pairs.
extern "C" int q4_test_gemm_plan(int M, int K, int N, int sms, int* mt, int* pairs) {
    const GemmPlan g = make_plan(M, K, N, sms);
    *mt = g.MT;
    *pairs = g.pairs;
    return g.pairs ? Q4_OK : Q4_ERR_UNSUPPORTED_SIZE;
}
#endif  // Q4_TEST_BUILD
