// Temperature / top-p sampling of the next token: the non-greedy branch of sample() (sampler.h:85-115) with its kernels
// softmax_logits_kernel and sample_top_p_kernel (gpu_kernels.h:507-592) and the radix sort / prefix sum between them.
//
// One launch of one cluster of eight CTAs instead of four launches. Semantics kept from the reference:
//   val = fp16(logit / temperature); e = fp16(exp(val - max)); p = fp16(e / sum(exp, unrounded fp32)); (written back in place)
//   0 < topp < 1: order = p descending (equal p: lower index first, the radix sort is stable), threshold = coin * topp
//   otherwise   : order = index order, threshold = coin
//   token = first element in that order whose inclusive prefix sum of p reaches the threshold; the last one if none does.
// The reference accumulates the prefix sum in fp16 in whatever order the device-wide scan takes. Here the sum is EXACT:
// every fp16 probability is an integer multiple of 2^-24, so prefix sums are integers (below 2^25) and the result does not
// depend on any summation order. The sorted order is never materialised: two histogram passes over the fp16 bit pattern
// (high byte, then low byte) find the probability value at which the prefix crosses the threshold, and a count over the
// ties in index order finds the element.
//
// The op is latency: 64 KB of logits for 32000 words, a chain of five reductions over all of them. One CTA of 1024 threads took
// 121 us (32 elements per thread and pass, 64-bit shared-memory atomics that all fall on the few exponents a softmax
// produces, bin scans by one thread, contiguous 32-element walks per thread); eight CTAs with the elements kept in shared
// memory and the partial results exchanged through distributed shared memory bring a sampled token's tail (classifier of
// 32000 x 4096 and this kernel, launched together) from 197 to 65 us. Eight is the largest portable cluster.
#include <cooperative_groups.h>
#include <math_constants.h>

#include <type_traits>

#include "q4_common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kT = 1024;                 // virtual threads of the sum's fixed order; also the threads of a CTA
constexpr int kCtas = 8;                 // one cluster
constexpr int kCols = kT / kCtas;        // virtual threads per CTA: CTA r owns elements i with i % 1024 in [128 r, 128 r + 128)
constexpr int kRowsAtOnce = kT / kCols;  // rows (i / 1024) a CTA works on at a time
constexpr int kMaxRows = (1 << 18) / kT;
constexpr size_t kRowBytes = (sizeof(float) + sizeof(unsigned short)) * kCols;   // of dynamic shared memory per row

__device__ __forceinline__ unsigned prob_units(unsigned short h) {   // fp16 in [0, 1] -> multiples of 2^-24
    const unsigned e = (h >> 10) & 31u, mnt = h & 1023u;
    return e == 0 ? mnt : (1024u + mnt) << (e - 1);
}

// Inclusive scan over a warp.
__device__ __forceinline__ unsigned warp_scan(unsigned v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// Probabilities sum to 1 up to roundings (2^24 units, below 2^25 with n <= 2^18), so every prefix fits 32 bits. The one input
// that breaks this is a NaN or +inf among the logits: then the sum and all probabilities are NaN, and the first element of
// either order already carries the prefix past any threshold, which is what the kernel answers without looking further.
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kT)
sample_topp_kernel(__half* __restrict__ logits, int n, float temperature, float topp, float coin, int* result, volatile int* pPos, int* pPosGpu) {
    extern __shared__ __align__(16) unsigned char dyn[];
    const int rows = (n + kT - 1) / kT;
    float* s_v = reinterpret_cast<float*>(dyn);                                           // [rows][kCols] exp values
    unsigned short* s_key = reinterpret_cast<unsigned short*>(dyn + sizeof(float) * (size_t)rows * kCols);   // [rows][kCols] fp16 bits
    __shared__ float s_red[32];
    __shared__ float s_max[kCtas], s_wsum[32];
    __shared__ unsigned s_part[kRowsAtOnce][64];            // high-byte histogram, one copy per group of 128 threads
    __shared__ __align__(16) unsigned s_hist[64], s_hist2[256];   // this CTA's histograms, read by the whole cluster
    __shared__ unsigned s_cnt[kMaxRows];                    // per row: matches (or units) among this CTA's 128 columns
    __shared__ unsigned s_all[kMaxRows * kCtas];            // CTA 0: the same of all CTAs, in index order
    __shared__ __align__(16) unsigned s_hists[kCtas * 256]; // all CTAs' histograms
    __shared__ unsigned s_last[kCtas];
    __shared__ int s_bin;
    __shared__ unsigned s_before, s_seg, s_seg_before;
    cg::cluster_group cluster = cg::this_cluster();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, rank = (int)cluster.block_rank();
    const int col = t & (kCols - 1), row0 = t / kCols;
    const int i_col = rank * kCols + col;
    cluster.sync();   // every CTA of the cluster has started: its shared memory may be written from here on
    griddep_wait();
    griddep_launch_dependents();

    int token_pos = 0;
    if (rank == 0 && t == 0) token_pos = *pPos;   // (host memory: read at the hand-off the kernel ended two microseconds later)

    // ---- softmax with temperature (softmax_logits_kernel) ----
    float mx = -CUDART_INF_F;
    constexpr int U = 4;   // elements of a thread in flight
    for (int j0 = row0; j0 < rows; j0 += U * kRowsAtOnce) {
        __half in[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = (j0 + u * kRowsAtOnce) * kT + i_col;
            in[u] = i < n ? logits[i] : __half();
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = j0 + u * kRowsAtOnce;
            if (j * kT + i_col < n) {
                float val = __half2float(in[u]);
                val /= temperature;
                const __half hv = __float2half(val);
                s_key[j * kCols + col] = __half_as_ushort(hv);
                mx = fmaxf(mx, __half2float(hv));
            }
        }
    }
    for (int i = t; i < 256; i += kT) s_hist2[i] = 0;
    if (t < kRowsAtOnce * 64) (&s_part[0][0])[t] = 0;
    for (int j = t; j < rows; j += kT) s_cnt[j] = 0;
    mx = warp_max(mx);
    if (lane == 0) s_red[warp] = mx;
    __syncthreads();
    if (warp == 0) {
        mx = warp_max(s_red[lane]);
        if (lane < kCtas) cluster.map_shared_rank(s_max, lane)[rank] = mx;
    }
    cluster.sync();
    mx = s_max[0];
#pragma unroll
    for (int r = 1; r < kCtas; r++) mx = fmaxf(mx, s_max[r]);
    for (int j = row0; j < rows; j += kRowsAtOnce) {
        if (j * kT + i_col < n) {
            const float v = expf(__half2float(__ushort_as_half(s_key[j * kCols + col])) - mx);
            s_key[j * kCols + col] = __half_as_ushort(__float2half(v));
            s_v[j * kCols + col] = v;
        }
    }
    __syncthreads();
    // The sum in a fixed order that does not depend on the cluster: virtual thread i % 1024 adds its elements in index order,
    // then an xor tree 16..1 inside each warp of virtual threads and the same tree over the 32 warps. The CPU oracle repeats
    // exactly this order.
    if (t < kCols) {
        float sum = 0.f;
        int j = 0;
        for (; j + 4 <= rows - 1; j += 4) {   // (all but the last row are full)
            const float a = s_v[j * kCols + t], b = s_v[(j + 1) * kCols + t], c = s_v[(j + 2) * kCols + t], d = s_v[(j + 3) * kCols + t];
            sum += a; sum += b; sum += c; sum += d;
        }
        for (; j < rows; j++)
            if (j * kT + i_col < n) sum += s_v[j * kCols + t];
        sum = warp_sum(sum);
        if (lane < kCtas) cluster.map_shared_rank(s_wsum, lane)[rank * (kCols / 32) + warp] = sum;
    }
    cluster.sync();
    const float sum = warp_sum(s_wsum[lane]);
    const bool sorted = topp > 0.f && topp < 1.f;
    for (int j = row0; j < rows; j += kRowsAtOnce) {
        const int i = j * kT + i_col;
        if (i < n) {
            const __half p = __float2half(__half2float(__ushort_as_half(s_key[j * kCols + col])) / sum);
            const unsigned short k = __half_as_ushort(p);
            logits[i] = p;
            s_key[j * kCols + col] = k;
            if (sorted && k != 0 && k <= 0x3C00) atomicAdd(&s_part[row0][k >> 8], prob_units(k));
        }
    }

    const float threshold = sorted ? coin * topp : coin;
    // prefix >= threshold  <=>  integer prefix >= ceil(threshold * 2^24). A threshold <= 0 selects the first element of
    // the order whatever its probability (`prefix >= 0` holds at once): index 0 in index order; in sorted order the
    // largest probability, which is what need = 1 finds.
    const double td = ceil((double)threshold * 16777216.0);
    const unsigned need = td <= 1.0 ? 1u : (td >= 4.0e9 ? 0xFFFFFFFFu : (unsigned)td);
    int token = -1;          // known to every thread, or searched for as the target-th unit of the rows below
    unsigned target = need;  // matches or units up to and including the token
    int key = -1;
    if (!(sum == sum) || (!sorted && !(threshold > 0.f))) {
        token = 0;
    } else if (sorted) {
        // ---- descending probability: the fp16 value at which the prefix crosses, high byte then low byte ----
        __syncthreads();
        if (t < 64) {
            unsigned h = 0;
#pragma unroll
            for (int c = 0; c < kRowsAtOnce; c++) h += s_part[c][t];
            s_hist[t] = h;
        }
        cluster.sync();
        // The cluster's histograms into this CTA's memory, a warp to each, whole lines at a time (all read by warp 0, bin by bin, the second one took
        // 5300 clocks, now 1900)
        auto gather = [&](const unsigned* hist, auto bins) {
            constexpr int per_lane = decltype(bins)::value, kV = per_lane < 4 ? per_lane : 4;
            struct alignas(4 * kV) Words { unsigned w[kV]; };
            if (warp < kCtas) {
                const Words* from = reinterpret_cast<const Words*>(cluster.map_shared_rank(hist, warp));
                Words* to = reinterpret_cast<Words*>(s_hists + warp * 32 * per_lane);
#pragma unroll
                for (int u = 0; u < per_lane / kV; u++) to[u * 32 + lane] = from[u * 32 + lane];
            }
            __syncthreads();
        };
        auto find_bin = [&](auto bins, unsigned before) {   // warp 0; lane's bins, highest first
            constexpr int per_lane = decltype(bins)::value;
            unsigned v[per_lane], tot = 0;
            const int top = per_lane * (32 - lane) - 1;
#pragma unroll
            for (int b = 0; b < per_lane; b++) {
                v[b] = 0;
#pragma unroll
                for (int r = 0; r < kCtas; r++) v[b] += s_hists[r * 32 * per_lane + top - b];
            }
#pragma unroll
            for (int b = 0; b < per_lane; b++) tot += v[b];
            const unsigned incl = warp_scan(tot, lane);
            unsigned c = before + incl - tot;
            const unsigned hit = __ballot_sync(0xffffffffu, before + incl >= need);
            if (hit == 0) { if (lane == 0) s_bin = -1; return; }
            if (lane == __ffs(hit) - 1) {
                int at = top;
                bool on = true;
#pragma unroll
                for (int b = 0; b < per_lane; b++) {
                    on = on && c + v[b] < need;
                    if (on) { c += v[b]; at--; }
                }
                s_bin = at;
                s_before = c;
            }
        };
        gather(s_hist, std::integral_constant<int, 2>());
        if (warp == 0) find_bin(std::integral_constant<int, 2>(), 0u);
        __syncthreads();
        if (s_bin < 0) {
            // the threshold is never reached: the last element of the order = lowest probability, highest index among equals
            unsigned best = 0xFFFFFFFFu;   // (key << 18 | ~index) minimised: lowest key (< 2^14), then highest index (n <= 2^18)
            for (int j = row0; j < rows; j += kRowsAtOnce) {
                const int i = j * kT + i_col;
                if (i < n) best = min(best, ((unsigned)s_key[j * kCols + col] << 18) | (unsigned)(0x3FFFF - i));
            }
            best = __reduce_min_sync(0xffffffffu, best);
            if (lane == 0) s_red[warp] = __uint_as_float(best);
            __syncthreads();
            if (warp == 0) {
                best = __reduce_min_sync(0xffffffffu, __float_as_uint(s_red[lane]));
                if (lane < kCtas) cluster.map_shared_rank(s_last, lane)[rank] = best;
            }
            cluster.sync();
            best = s_last[0];
#pragma unroll
            for (int r = 1; r < kCtas; r++) best = min(best, s_last[r]);
            token = 0x3FFFF - (int)(best & 0x3FFFFu);
        } else {
            key = s_bin;
            const unsigned before = s_before;
            for (int j = row0; j < rows; j += kRowsAtOnce) {
                if (j * kT + i_col < n) {
                    const unsigned short k = s_key[j * kCols + col];
                    if ((k >> 8) == key) atomicAdd(&s_hist2[k & 255], prob_units(k));
                }
            }
            cluster.sync();
            gather(s_hist2, std::integral_constant<int, 8>());
            if (warp == 0) find_bin(std::integral_constant<int, 8>(), before);
            __syncthreads();
            key = (key << 8) | s_bin;
            // the k-th element (index order) among those whose probability has exactly this bit pattern
            const unsigned pv = prob_units((unsigned short)key);
            target = (need - s_before + pv - 1) / pv;   // 1-based, >= 1
        }
    }

    if (token < 0) {
        // ---- the element at which the prefix in index order reaches `target`: matches of `key`, or probability units ----
        for (int j = row0; j < rows; j += kRowsAtOnce) {
            const bool in = j * kT + i_col < n;
            const unsigned short k = in ? s_key[j * kCols + col] : (unsigned short)0;
            const unsigned v = sorted ? (unsigned)__popc(__ballot_sync(0xffffffffu, in && k == (unsigned short)key))
                                      : __reduce_add_sync(0xffffffffu, in ? prob_units(k) : 0u);
            if (lane == 0) atomicAdd(&s_cnt[j], v);
        }
        __syncthreads();
        for (int j = t; j < rows; j += kT) cluster.map_shared_rank(s_all, 0)[j * kCtas + rank] = s_cnt[j];   // row-major: index order
        cluster.sync();
        if (rank == 0) {
            // scan over the (row, CTA) segments, two per thread
            const int nseg = rows * kCtas;
            const unsigned a = 2 * t < nseg ? s_all[2 * t] : 0u, b = 2 * t + 1 < nseg ? s_all[2 * t + 1] : 0u;
            unsigned incl = warp_scan(a + b, lane);
            if (lane == 31) s_red[warp] = __uint_as_float(incl);
            if (t == 0) s_seg = 0xFFFFFFFFu;
            __syncthreads();
            const unsigned w = __float_as_uint(s_red[lane]);
            const unsigned wincl = warp_scan(w, lane);
            incl += __shfl_sync(0xffffffffu, wincl - w, warp);
            const unsigned excl = incl - (a + b);
            if (excl < target && incl >= target) {   // exactly one thread, when the target is reached at all
                const bool second = excl + a < target;
                s_seg = 2 * t + (second ? 1 : 0);
                s_seg_before = second ? excl + a : excl;
            }
            __syncthreads();
            if (warp == 0) {
                token = n - 1;
                if (s_seg != 0xFFFFFFFFu) {
                    const int j = (int)(s_seg / kCtas), r = (int)(s_seg % kCtas);
                    const unsigned short* keys = cluster.map_shared_rank(s_key, r) + j * kCols;
                    unsigned c = s_seg_before;
                    unsigned short mine[kCols / 32];       // (all requested at once)
#pragma unroll
                    for (int u = 0; u < kCols / 32; u++) mine[u] = j * kT + r * kCols + 32 * u + lane < n ? keys[32 * u + lane] : (unsigned short)0;
#pragma unroll
                    for (int u = 0; u < kCols / 32; u++) {
                        const int c0 = 32 * u, i = j * kT + r * kCols + c0 + lane;
                        const unsigned short k = mine[u];
                        const unsigned v = i >= n ? 0u : sorted ? (unsigned)(k == (unsigned short)key) : prob_units(k);
                        const unsigned here = c + warp_scan(v, lane);
                        const unsigned hit = __ballot_sync(0xffffffffu, here >= target);
                        if (hit) { token = j * kT + r * kCols + c0 + __ffs(hit) - 1; break; }
                        c = __shfl_sync(0xffffffffu, here, 31);
                    }
                }
            }
        }
        cluster.sync();   // CTA 0 reads the others' shared memory until here
    }
    if (rank == 0 && t == 0) {   // hand-off as in sample_top_p_kernel (gpu_kernels.h:583-591)
        token_pos++;
        result[token_pos] = token;
        *pPos = token_pos;
        *pPosGpu = token_pos;
    }
}

}  // namespace

// xorshift* of the reference (sampler.h:66-75): the host draws one coin per forward call.
extern "C" unsigned int q4_random_u32(unsigned long long* state) {
    *state ^= *state >> 12;
    *state ^= *state << 25;
    *state ^= *state >> 27;
    return (unsigned int)((*state * 0x2545F4914F6CDD1Dull) >> 32);
}
extern "C" float q4_random_f32(unsigned long long* state) { return (q4_random_u32(state) >> 8) / 16777216.0f; }

extern "C" int q4_sample_topp(void* stream, uint16_t* logits, int n, float temperature, float topp, float coin, int* tokens_pinned,
                              volatile int* pos_pinned, int* pos_dev) {
    if (!logits || !tokens_pinned || !pos_pinned || !pos_dev || n <= 0 || n > (1 << 18) || !(temperature > 0.f)) return Q4_ERR_INVALID;
    const size_t smem = kRowBytes * q4_div_up(n, kT);
    // The static arrays take 21 KB of the 48 KB that need no opt-in. The limit belongs to the function on the device and not to this
    // call: it is always set to the largest size, so that calls of other threads between here and the launch cannot lower it.
    if (smem > 24 * 1024) Q4_CUDA_TRY(cudaFuncSetAttribute(sample_topp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kRowBytes * kMaxRows)));
    Q4Launch L(dim3(kCtas), dim3(kT), smem, (cudaStream_t)stream);
    Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, sample_topp_kernel, (__half*)logits, n, temperature, topp, coin, tokens_pinned, pos_pinned, pos_dev));
    return Q4_OK;
}
