// fp16 attention of one query per head over the KV cache, split along the sequence so that every SM has work
// at any context length (the reference's three kernels give one head's AV product to 4 blocks only).
// Replaces MultiHeadAttention (llama2_q4.cu:410-427; mat_vec_kernel_simple, softmax_kernel, vec_mat_kernel at
// gpu_kernels.h:150-176,365-454,287-337).
//
// A block takes positions [t0, t1) of one head. Eight lanes share a position (8 dims of every 64: a load of theirs is 128 bytes in a row), a block of
// eight warps has 64 positions in hand per step and the next 64 requested. Scores are rounded to fp16 like the reference's; the
// softmax runs online in fp32 (running max, sum and un-normalised V accumulator per lane group), merged across the block in registers
// and shared memory. A head's blocks are a thread-block cluster and read one another's (max, sum, acc) from shared memory: one launch, no
// scratch. What bounds it is latency: 32 heads at position 600 are 10 MB. Before (16 positions in hand per block, none requested
// ahead, up to 32 blocks per head and a second launch that merged them through global memory), back to back at positions 60, 600, 1900
// and 3800: 4 heads 8.2, 12.2, 13.6, 15.5 us, now 3.5, 4.2, 5.5, 7.7; 32 heads 8.0, 10.1, 24.3, 40.5, now 4.2, 5.3, 9.9, 15.2; 64 heads in
// groups of 8 6.8, 11.0, 19.6, 61.6, now 4.2, 6.1, 10.4, 18.7. Two 7B layers call by call at position 600 133 -> 120 us.
// The sequence length comes from *pPos on the device; the grid does not depend on it.
#include <math_constants.h>

#include <stdio.h>

#include "q4_common.cuh"
#include "q4_model.h"

namespace {

constexpr int kAttnThreads = 256, kAttnWarps = kAttnThreads / 32;
constexpr int kGroups = kAttnThreads / 8;  // lane groups of a block; each has two positions in hand
constexpr int kMaxHeadSize = 256;

// Blocks of a head's cluster: the most that leaves two blocks per SM over all heads, which is what fits at once (positions 60, 600, 1900
// and 3800: 32 heads 4.2, 5.3, 9.9, 15.2 us with eight and 3.7, 5.2, 12.2, 19.9 with four; 40 heads 7.2, 9.4, 16.7, 26.1 with eight and
// 4.1, 6.4, 13.5, 21.8 with four; 96 heads 7.1, 14.1, 26.4, 44.3 with four and 4.3, 10.1, 22.3, 40.2 with two).
int attn_cluster(int num_heads) {
    int blocks = 8;
    while (blocks > 1 && blocks * num_heads > 2 * 148) blocks /= 2;
    return blocks;
}
// what a host's scratch was sized by when the blocks of a head exchanged their parts through it
int attn_splits(int num_heads) {
    int s = q4_div_up(2 * 148, num_heads);
    if (s < 1) s = 1;
    if (s > 32) s = 32;
    return s;
}

template <int HS>
struct AttnShared {
    float m[kAttnWarps], l[kAttnWarps], acc[kAttnWarps][HS];
    float M, L, out[HS];   // the block's: maximum, sum, un-normalised V sum
};

// This block's share of head h, into sm.M, sm.L and sm.out (behind a barrier).
template <int HS>
__device__ __forceinline__ void attn_share(AttnShared<HS>& sm, const __half* q, const __half* kc, const __half* vc, int kv_mul, int kv_stride, const int* pPos, int h,
                                           int split, int nsplit) {
    constexpr int PER = HS / 8;      // head dims per lane
    constexpr int VEC = PER / 8;     // uint4 per lane per row
    const int lane8 = threadIdx.x & 7, grp = threadIdx.x >> 3, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint4 qv[VEC];
#pragma unroll
    for (int v = 0; v < VEC; v++) qv[v] = *reinterpret_cast<const uint4*>(q + (size_t)h * HS + v * 64 + lane8 * 8);
    const int T = *pPos + 1;
    // split boundaries in units of kGroups positions
    const int units = (T + kGroups - 1) / kGroups;
    const int t0 = (int)((long long)units * split / nsplit) * kGroups, t1 = min((int)((long long)units * (split + 1) / nsplit) * kGroups, T);
    float qf[PER];
#pragma unroll
    for (int v = 0; v < VEC; v++) {
        const __half2* hh = reinterpret_cast<const __half2*>(&qv[v]);
#pragma unroll
        for (int j = 0; j < 4; j++) { const float2 f = __half22float2(hh[j]); qf[v * 8 + 2 * j] = f.x; qf[v * 8 + 2 * j + 1] = f.y; }
    }
    const float alpha = (float)(1.0 / sqrt((double)HS));
    const size_t head_off = (size_t)(h / kv_mul) * HS + lane8 * 8;

    float m = -CUDART_INF_F, l = 0.f;
    float acc[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) acc[i] = 0.f;

    constexpr int kStep = 2 * kGroups;
    uint4 k4[2][VEC], v4[2][VEC];
    // rows past the share's end read its first row and are not counted
    auto fetch = [&](uint4 (&r)[2][VEC], const __half* cache, int tb) {
        if (tb >= t1) return;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int t = tb + grp + u * kGroups;
            const uint4* src = reinterpret_cast<const uint4*>(cache + (size_t)(t < t1 ? t : t0) * kv_stride + head_off);
#pragma unroll
            for (int v = 0; v < VEC; v++) r[u][v] = src[8 * v];
        }
    };
    fetch(k4, kc, t0);
    fetch(v4, vc, t0);
    // the trip count is the same for every lane of the block (shuffles below use the full mask)
    for (int tb = t0; tb < t1; tb += kStep) {
        float s[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            s[u] = 0.f;
#pragma unroll
            for (int v = 0; v < VEC; v++) {
                const __half2* hh = reinterpret_cast<const __half2*>(&k4[u][v]);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 f = __half22float2(hh[j]);
                    s[u] = fmaf(f.x, qf[v * 8 + 2 * j], s[u]);
                    s[u] = fmaf(f.y, qf[v * 8 + 2 * j + 1], s[u]);
                }
            }
        }
        fetch(k4, kc, tb + kStep);   // into the registers just read
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int u = 0; u < 2; u++) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (tb + grp + u * kGroups < t1) {
                const float sc = __half2float(__float2half(s[u] * alpha));  // the reference stores scores as fp16 (gpu_kernels.h:171-175)
                const float mn = fmaxf(m, sc);
                const float base = mn == -CUDART_INF_F ? 0.f : mn;          // scores of -infinity only: their weights are 0, a NaN's is NaN
                const float corr = expf(m - base), p = expf(sc - base);     // (corr is 0 on the first position)
                l = l * corr + p;
#pragma unroll
                for (int v = 0; v < VEC; v++) {
                    const __half2* hh = reinterpret_cast<const __half2*>(&v4[u][v]);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float2 f = __half22float2(hh[j]);
                        acc[v * 8 + 2 * j] = fmaf(p, f.x, acc[v * 8 + 2 * j] * corr);
                        acc[v * 8 + 2 * j + 1] = fmaf(p, f.y, acc[v * 8 + 2 * j + 1] * corr);
                    }
                }
                m = mn;
            }
        }
        fetch(v4, vc, tb + kStep);
    }
    // weight of a part whose maximum and sum are (pm, pl) in a whole with maximum M: nothing where nothing was added up
    auto weight = [](float pm, float pl, float M) { return pl == 0.f ? 0.f : expf(pm - (M == -CUDART_INF_F ? 0.f : M)); };
    // the four lane groups of a warp, then the warps
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) {
        const float mo = __shfl_xor_sync(0xffffffffu, m, o), lo = __shfl_xor_sync(0xffffffffu, l, o);
        const float mn = fmaxf(m, mo), ca = weight(m, l, mn), cb = weight(mo, lo, mn);
        l = l * ca + lo * cb;
#pragma unroll
        for (int i = 0; i < PER; i++) acc[i] = acc[i] * ca + __shfl_xor_sync(0xffffffffu, acc[i], o) * cb;
        m = mn;
    }
    if (lane == 0) { sm.m[warp] = m; sm.l[warp] = l; }
    if (lane < 8) {
#pragma unroll
        for (int i = 0; i < PER; i += 4) *reinterpret_cast<float4*>(&sm.acc[warp][(i >> 3) * 64 + lane8 * 8 + (i & 7)]) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
    }
    __syncthreads();
    if (threadIdx.x < HS) {
        float M = -CUDART_INF_F, L = 0.f, a = 0.f;
#pragma unroll
        for (int w = 0; w < kAttnWarps; w++) M = fmaxf(M, sm.m[w]);
#pragma unroll
        for (int w = 0; w < kAttnWarps; w++) {
            const float e = weight(sm.m[w], sm.l[w], M);
            L += sm.l[w] * e;
            a += sm.acc[w][threadIdx.x] * e;
        }
        sm.out[threadIdx.x] = a;
        if (threadIdx.x == 0) { sm.M = M; sm.L = L; }
    }
}

// grid (cluster, heads), the blocks of a head one cluster: each merges its part of the head's dims.
template <int HS>
__global__ void __launch_bounds__(kAttnThreads) attn_cluster_kernel(__half* output, const __half* q, const __half* kc, const __half* vc, int kv_mul, int kv_stride,
                                                                    const int* pPos) {
    __shared__ __align__(16) AttnShared<HS> sm;
    const int h = blockIdx.y, rank = blockIdx.x, nblocks = gridDim.x;
    griddep_wait();
    griddep_launch_dependents();
    attn_share<HS>(sm, q, kc, vc, kv_mul, kv_stride, pPos, h, rank, nblocks);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int dims = HS / nblocks;
    if (threadIdx.x < dims) {
        const int d = rank * dims + threadIdx.x;
        auto remote = [](const float* p, int r) {
            uint32_t addr;
            float v;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(r));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
            return v;
        };
        float pm[8], pl[8], pa[8], M = -CUDART_INF_F, L = 0.f, a = 0.f;
#pragma unroll
        for (int r = 0; r < 8; r++) {
            pm[r] = -CUDART_INF_F;
            pl[r] = pa[r] = 0.f;
            if (r < nblocks) { pm[r] = remote(&sm.M, r); pl[r] = remote(&sm.L, r); pa[r] = remote(&sm.out[d], r); }
        }
#pragma unroll
        for (int r = 0; r < 8; r++) M = fmaxf(M, pm[r]);
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const float e = pl[r] == 0.f ? 0.f : expf(pm[r] - (M == -CUDART_INF_F ? 0.f : M));
            L += pl[r] * e;
            a += pa[r] * e;
        }
        output[(size_t)h * HS + d] = __float2half(a / L);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // no block leaves while another reads its shared memory
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace

extern "C" size_t q4_attention_scratch_bytes(int num_heads, int head_size) {
    if (num_heads <= 0 || head_size <= 0) return 0;
    return (size_t)num_heads * attn_splits(num_heads) * (head_size + 2) * sizeof(float);
}

template <int HS>
static int attention_launch(cudaStream_t s, __half* output, const __half* q, const __half* kc, const __half* vc, int num_heads, int kv_mul, const int* pPos) {
    const int blocks = attn_cluster(num_heads);
    Q4Launch L(dim3(blocks, num_heads), dim3(kAttnThreads), 0, s);
    cudaLaunchAttribute attr[2] = {L.attr[0], {}};
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = blocks;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    L.cfg.attrs = attr;
    L.cfg.numAttrs = 2;
    Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, attn_cluster_kernel<HS>, output, q, kc, vc, kv_mul, num_heads * HS / kv_mul, pPos));
    return Q4_OK;
}

// What both entry points and the model launch.
int q4_attention_launch(cudaStream_t s, uint16_t* output, const uint16_t* q, const uint16_t* key_cache, const uint16_t* value_cache, int num_heads,
                               int head_size, int kv_mul, const int* pPos) {
    __half* out = (__half*)output;
    const __half *qh = (const __half*)q, *kc = (const __half*)key_cache, *vc = (const __half*)value_cache;
    switch (head_size) {
        case 64: return attention_launch<64>(s, out, qh, kc, vc, num_heads, kv_mul, pPos);
        case 128: return attention_launch<128>(s, out, qh, kc, vc, num_heads, kv_mul, pPos);
        case 256: return attention_launch<256>(s, out, qh, kc, vc, num_heads, kv_mul, pPos);
        default: return Q4_ERR_UNSUPPORTED_SIZE;
    }
}

extern "C" int q4_attention(void* stream, uint16_t* output, const uint16_t* q, const uint16_t* key_cache, const uint16_t* value_cache,
                            void* scratch, int num_heads, int head_size, int kv_mul, int max_seq_len, const int* pPos) {
    (void)max_seq_len;  // the reference sizes its grid with it (llama2_q4.cu:415); this grid is length-independent
    if (!output || !q || !key_cache || !value_cache || !scratch || !pPos || num_heads <= 0 || kv_mul <= 0 || num_heads % kv_mul)
        return Q4_ERR_INVALID;
    if (head_size > kMaxHeadSize) return Q4_ERR_UNSUPPORTED_SIZE;
    return q4_attention_launch((cudaStream_t)stream, output, q, key_cache, value_cache, num_heads, head_size, kv_mul, pPos);
}

// The same for hosts that hand this library nothing but the reference's own buffers and may not allocate device memory themselves (a
// serving process whose device memory is fully committed at start-up, a plugin that only receives raw pointers). The kernel has no such
// limit: it is what this call has always refused, by the size of a scratch nobody writes any more, and stays part of its contract.
extern "C" int q4_attention_static(void* stream, uint16_t* output, const uint16_t* q, const uint16_t* key_cache,
                                   const uint16_t* value_cache, int num_heads, int head_size, int kv_mul, int max_seq_len, const int* pPos) {
    (void)max_seq_len;
    if (!output || !q || !key_cache || !value_cache || !pPos || num_heads <= 0 || kv_mul <= 0 || num_heads % kv_mul) return Q4_ERR_INVALID;
    if (head_size > kMaxHeadSize) return Q4_ERR_UNSUPPORTED_SIZE;
    if (q4_attention_scratch_bytes(num_heads, head_size) > (size_t)Q4_ATTENTION_STATIC_MAX_BYTES) {
        fprintf(stderr, "q4_attention_static: %d heads of size %d are beyond this call's limit (q4_attention_scratch_bytes %zu, at most %d); q4_attention takes them\n", num_heads,
                head_size, q4_attention_scratch_bytes(num_heads, head_size), Q4_ATTENTION_STATIC_MAX_BYTES);
        return Q4_ERR_LIMIT;
    }
    return q4_attention_launch((cudaStream_t)stream, output, q, key_cache, value_cache, num_heads, head_size, kv_mul, pPos);
}
