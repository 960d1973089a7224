// Many rows through the network at once: prompt prefill (the rows are consecutive positions of one sequence) and batched
// decode (the rows are the current positions of several sequences). The reference has neither: it pushes a prompt
// through the batch-1 schedule token by token (llama2_q4.cu:710-735) and holds one sequence (RunState, common.h:62-78).
// The schedule per layer is run_llama_network's (llama2_q4.cu:444-524) with every op widened to rows:
//   RMSNorm -> Q, K, V (W4 dequant-GEMM on tcgen05, q4_gemm.cu) -> RoPE, K/V rows into the cache -> causal attention
//   -> O projection + residual [-> all-reduce] -> RMSNorm -> gate, up (GEMM) -> SiLU * up -> down + residual [-> all-reduce]
// with the rounding points of the batch-1 path (fp16 activations between ops, fp32 inside). A row is (sequence, position):
// the K/V cache row it writes and the range of cached positions it attends to follow from that pair, so one set of
// kernels serves both uses. The small row-wise kernels here are bandwidth-trivial next to the GEMMs and are kept simple.
#include <math_constants.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>

#include "q4_model.h"

namespace {

constexpr int kRowThreads = 256;

// Every kernel of this file starts with griddepcontrol.wait + launch_dependents and is launched with programmatic
// stream serialisation: its successor (often a weight-streaming kernel whose first loads do not depend on it) then begins
// its prologue while this one runs, and waits for this one's completion before it touches anything produced here.
template <typename... KArgs, typename... Args>
cudaError_t launch_rows(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    Q4Launch L(grid, block, smem, s);
    return cudaLaunchKernelEx(&L.cfg, kernel, KArgs(args)...);
}

// Where the rows come from: row m is the token at tok_base[seq * tok_stride + pos] of sequence row_seq[m] and position row_pos[m]; pos0 >= 0: of sequence 0 and
// position pos0 + m, and the two are written.
struct Embed {
    const __half* table;
    const int* tok_base;
    long long tok_stride;
    int *row_seq, *row_pos;
    int vocab, pos0;
};

// rmsnorm_kernel (gpu_kernels.h:72-105) per row: o = x * (rsqrt(mean(x^2) + 1e-5) * w), fp32 inside, fp16 out.
// size % 8 == 0; a thread keeps up to four 8-element pieces of the row in registers between the two passes.
__device__ __forceinline__ float sumsq8(const uint4& v) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 f = __half22float2(h[j]);
        s += f.x * f.x + f.y * f.y;
    }
    return s;
}
__device__ __forceinline__ uint4 scale8(const uint4& v, const uint4& w, float r) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
    const __half2* wh = reinterpret_cast<const __half2*>(&w);
    uint4 o;
    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 f = __half22float2(h[j]), g = __half22float2(wh[j]);
        oh[j] = __floats2half2_rn(f.x * (r * g.x), f.y * (r * g.y));
    }
    return o;
}
// x = half(y + x): the residual of matmul(QWeight)'s accum form (gpu_kernels.h:237-238) on a GEMM result that was written without it
__device__ __forceinline__ uint4 add8(const uint4& x, const uint4& y) {
    const __half2* xh = reinterpret_cast<const __half2*>(&x);
    const __half2* yh = reinterpret_cast<const __half2*>(&y);
    uint4 o;
    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 a = __half22float2(xh[j]), b = __half22float2(yh[j]);
        oh[j] = __floats2half2_rn(b.x + a.x, b.y + a.y);
    }
    return o;
}
// ROW_ADD: the row is x + y first, and goes back to x (a prompt's projections on one GPU: the GEMM's own residual epilogue reads two
// bytes per lane and row, 20 us per 512 x 4096 tile row, where this pass has the row in registers anyway). ROW_EMBED: it is its token's row of the
// table, and goes to x (as kernels of their own the rows' positions and embedding were two launches in front of the first product: 78 tokens of two 13B
// layers 316.5 us, 308.8 so; 333 behind 700 of a 70B layer 180.4, 176).
enum RowSource { ROW_X, ROW_ADD, ROW_EMBED };
template <RowSource SRC>
__global__ void __launch_bounds__(kRowThreads) rmsnorm_rows_kernel(__half* o, __half* x, const __half* y, const __half* w, int size, Embed em) {
    griddep_wait();   // launched with programmatic stream serialisation: wait for the producer, then let the consumer's prologue start
    griddep_launch_dependents();
    __shared__ float red[kRowThreads / 32];
    const uint4* token_row = nullptr;
    if (SRC == ROW_EMBED) {
        const int m = blockIdx.x, seq = em.pos0 >= 0 ? 0 : em.row_seq[m], pos = em.pos0 >= 0 ? em.pos0 + m : em.row_pos[m];
        int token = em.tok_base[(long long)seq * em.tok_stride + pos];
        if (token < 0 || token >= em.vocab) token = 0;   // (ids are validated on the host; a generated id is always in range)
        token_row = reinterpret_cast<const uint4*>(em.table + (size_t)token * size);
        if (em.pos0 >= 0 && threadIdx.x == 0) {
            em.row_seq[m] = 0;
            em.row_pos[m] = pos;
        }
    }
    uint4* xr = reinterpret_cast<uint4*>(x + (size_t)blockIdx.x * size);
    const uint4* yr = reinterpret_cast<const uint4*>(y + (size_t)blockIdx.x * size);
    uint4* orow = reinterpret_cast<uint4*>(o + (size_t)blockIdx.x * size);
    const uint4* wv = reinterpret_cast<const uint4*>(w);
    const int nvec = size / 8;
    constexpr int kKeep = 4;
    uint4 v[kKeep], wk[kKeep];   // (the weights are requested with the row: behind the sum they were a memory latency of their own)
    float ss = 0.f;
    auto row = [&](int i) {
        uint4 r = SRC == ROW_EMBED ? token_row[i] : xr[i];
        if (SRC == ROW_ADD) r = add8(r, yr[i]);
        if (SRC != ROW_X) xr[i] = r;
        return r;
    };
#pragma unroll
    for (int c = 0; c < kKeep; c++) {
        const int i = threadIdx.x + c * kRowThreads;
        if (i < nvec) { v[c] = row(i); wk[c] = __ldg(wv + i); }
    }
#pragma unroll
    for (int c = 0; c < kKeep; c++)
        if (threadIdx.x + c * kRowThreads < nvec) ss += sumsq8(v[c]);
    for (int i = threadIdx.x + kKeep * kRowThreads; i < nvec; i += kRowThreads) ss += sumsq8(row(i));
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < kRowThreads / 32; i++) tot += red[i];
    tot /= size;
    tot += 1e-5f;
    tot = 1.0f / sqrtf(tot);
#pragma unroll
    for (int c = 0; c < kKeep; c++) {
        const int i = threadIdx.x + c * kRowThreads;
        if (i < nvec) orow[i] = scale8(v[c], wk[c], tot);
    }
    for (int i = threadIdx.x + kKeep * kRowThreads; i < nvec; i += kRowThreads) orow[i] = scale8(xr[i], wv[i], tot);
}

// RoPERotation_kernel (gpu_kernels.h:340-363) per row, and the row's K and V into the cache: query heads are rotated in place,
// the key heads are rotated on their way into cache row `pos` of the row's sequence, the value heads are copied there.
// head_size 128. A thread takes eight rotation pairs of one head (16 bytes of each half of the head); the angles come from a
// table [position][pair] built once with the reference's arithmetic (evaluating powf, cosf and sinf per block of four heads,
// two bytes per access, took 21.6 us for 512 rows of 32 + 32 heads). grid (rows, parts), block 256. Rows below q_row0 have no query.
__global__ void __launch_bounds__(256) rope_store_rows_kernel(__half* q, const __half* k, const __half* v, int ldq, int ldkv, __half* kc, __half* vc, int n_heads,
                                                              int n_kv_heads, const float2* table, const int* row_seq, const int* row_pos, long long seq_stride,
                                                              long long loff, int q_row0) {
    griddep_wait();   // launched with programmatic stream serialisation: wait for the producer, then let the consumer's prologue start
    griddep_launch_dependents();
    constexpr int HS = 128, kPer = 8;   // threads per head
    const int m = blockIdx.x;
    const int pos = row_pos[m];
    const size_t dst0 = (size_t)row_seq[m] * seq_stride + loff + (size_t)pos * n_kv_heads * HS;
    for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < (n_heads + 2 * n_kv_heads) * kPer; e += gridDim.y * blockDim.x) {
        const int hh = e / kPer, i = (e % kPer) * 8;
        if (hh >= n_heads + n_kv_heads) {
            const int h = hh - n_heads - n_kv_heads;
            const uint4* src = reinterpret_cast<const uint4*>(v + (size_t)m * ldkv + (size_t)h * HS + 2 * i);
            uint4* dst = reinterpret_cast<uint4*>(vc + dst0 + (size_t)h * HS + 2 * i);
            dst[0] = src[0];
            dst[1] = src[1];
            continue;
        }
        const bool is_q = hh < n_heads;
        if (is_q && m < q_row0) continue;
        const __half* src = is_q ? q + (size_t)m * ldq + (size_t)hh * HS : k + (size_t)m * ldkv + (size_t)(hh - n_heads) * HS;
        __half* dst = is_q ? q + (size_t)m * ldq + (size_t)hh * HS : kc + dst0 + (size_t)(hh - n_heads) * HS;
        uint4 lo = *reinterpret_cast<const uint4*>(src + i), hi = *reinterpret_cast<const uint4*>(src + i + HS / 2);
        const float4* tp = reinterpret_cast<const float4*>(table + (size_t)pos * (HS / 2) + i);
        __half* l = reinterpret_cast<__half*>(&lo);
        __half* g = reinterpret_cast<__half*>(&hi);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 cs = __ldg(tp + j);
            rope_rotate(l + 2 * j, g + 2 * j, l + 2 * j, g + 2 * j, make_float2(cs.x, cs.y));
            rope_rotate(l + 2 * j + 1, g + 2 * j + 1, l + 2 * j + 1, g + 2 * j + 1, make_float2(cs.z, cs.w));
        }
        *reinterpret_cast<uint4*>(dst + i) = lo;
        *reinterpret_cast<uint4*>(dst + i + HS / 2) = hi;
    }
}
__global__ void rope_rows_table_kernel(float2* table, int positions, int head_size, float theta) {
    const int half_hs = head_size / 2;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < positions * half_hs; i += gridDim.x * blockDim.x)
        table[i] = rope_cos_sin(i / half_hs, i % half_hs, head_size, theta);
}

// MultiHeadAttention (llama2_q4.cu:410-427) for one (row, head): the query attends to positions 0 .. pos of its own sequence.
// Scores are rounded to fp16 as the reference stores them (gpu_kernels.h:171-175); the softmax runs online in fp32 over the keys
// a warp visits, the warps are merged at the end. A warp takes four keys per round (keys 4 (warp + 8 i) .. + 3) and issues
// their eight K/V loads together, so a round costs one memory latency, not eight. head_size 128: a lane holds four dims.
// grid (heads, rows), block 256.
// FUSED (batched decode: no two rows of a launch share a sequence): q, k and v come as the projections left them. Every warp
// rotates its query (rope_store_rows_kernel's table and rounding), the warp whose turn position pos is rotates the new key
// and takes it and the new value from registers, and the first query head of a key/value head files both in the cache: one
// launch less per layer (batch-8 step of four 7B layers: 247 -> 231 us). Otherwise the row's K and V are in the cache already and q is rotated.
constexpr int kAttWarps = 8, kAttKeys = 4;
template <bool FUSED>
__global__ void __launch_bounds__(kAttWarps * 32) attention_rows_kernel(__half* out, const __half* q, int ldq, __half* kc, __half* vc, int n_heads, int kv_mul,
                                                                       const int* row_seq, const int* row_pos, long long seq_stride, long long loff, int kv_n,
                                                                       const __half* knew, const __half* vnew, const float2* table) {
    griddep_wait();   // launched with programmatic stream serialisation: wait for the producer, then let the consumer's prologue start
    griddep_launch_dependents();
    constexpr int HS = 128;
    const int h = blockIdx.x, m = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = row_pos[m];
    const int T = FUSED ? pos : pos + 1;   // positions read from the cache
    const size_t head_at = (size_t)row_seq[m] * seq_stride + loff + (size_t)(h / kv_mul) * HS + lane * 4;
    const __half* kb = kc + head_at;
    const __half* vb = vc + head_at;
    float4 cs01 = {}, cs23 = {};   // (cos, sin) of this lane's four pairs
    if (FUSED) {
        const float4* tp = reinterpret_cast<const float4*>(table + (size_t)pos * (HS / 2) + (lane & 15) * 4);
        cs01 = __ldg(tp);
        cs23 = __ldg(tp + 1);
    }
    // four elements of a head whose other halves of the pairs lie 16 lanes away, rotated and rounded to fp16
    auto rotate = [&](uint2 v) {
        uint2 o;
        o.x = __shfl_xor_sync(0xffffffffu, v.x, 16);
        o.y = __shfl_xor_sync(0xffffffffu, v.y, 16);
        const uint2 l = lane < 16 ? v : o, g = lane < 16 ? o : v;
        __half lo[4], hi[4];
        *reinterpret_cast<uint2*>(lo) = l;
        *reinterpret_cast<uint2*>(hi) = g;
        rope_rotate(lo, hi, lo, hi, make_float2(cs01.x, cs01.y));
        rope_rotate(lo + 1, hi + 1, lo + 1, hi + 1, make_float2(cs01.z, cs01.w));
        rope_rotate(lo + 2, hi + 2, lo + 2, hi + 2, make_float2(cs23.x, cs23.y));
        rope_rotate(lo + 3, hi + 3, lo + 3, hi + 3, make_float2(cs23.z, cs23.w));
        return lane < 16 ? *reinterpret_cast<uint2*>(lo) : *reinterpret_cast<uint2*>(hi);
    };
    float qf[4];
    {
        uint2 qv = *reinterpret_cast<const uint2*>(q + (size_t)m * ldq + (size_t)h * HS + lane * 4);
        if (FUSED) qv = rotate(qv);
        const __half2* qh = reinterpret_cast<const __half2*>(&qv);
        qf[0] = __low2float(qh[0]); qf[1] = __high2float(qh[0]); qf[2] = __low2float(qh[1]); qf[3] = __high2float(qh[1]);
    }
    const float alpha = (float)(1.0 / sqrt((double)HS));
    float mx = -CUDART_INF_F, l = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
    // keys kv[u], values vv[u]; those with u >= live do not count (the first always does)
    auto round4 = [&](const uint2 (&kv)[kAttKeys], const uint2 (&vv)[kAttKeys], int live) {
        float sc[kAttKeys];
#pragma unroll
        for (int u = 0; u < kAttKeys; u++) {
            const __half2* kh = reinterpret_cast<const __half2*>(&kv[u]);
            sc[u] = qf[0] * __low2float(kh[0]) + qf[1] * __high2float(kh[0]) + qf[2] * __low2float(kh[1]) + qf[3] * __high2float(kh[1]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < kAttKeys; u++) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o);
        float mn = mx;
#pragma unroll
        for (int u = 0; u < kAttKeys; u++) {
            sc[u] = u < live ? __half2float(__float2half(sc[u] * alpha)) : -CUDART_INF_F;
            mn = fmaxf(mn, sc[u]);
        }
        const float corr = expf(mx - mn);   // the round's first key is always valid, so mn is finite
        l *= corr;
#pragma unroll
        for (int j = 0; j < 4; j++) acc[j] *= corr;
#pragma unroll
        for (int u = 0; u < kAttKeys; u++) {
            const float pr = expf(sc[u] - mn);
            const __half2* vh = reinterpret_cast<const __half2*>(&vv[u]);
            l += pr;
            acc[0] += pr * __low2float(vh[0]);
            acc[1] += pr * __high2float(vh[0]);
            acc[2] += pr * __low2float(vh[1]);
            acc[3] += pr * __high2float(vh[1]);
        }
        mx = mn;
    };
    auto load4 = [&](uint2 (&kv)[kAttKeys], uint2 (&vv)[kAttKeys], int t0) {
#pragma unroll
        for (int u = 0; u < kAttKeys; u++) {
            const int t = max(min(t0 + u, T - 1), 0);   // a round's tail reads some earlier row instead (row 0 where there is none)
            kv[u] = *reinterpret_cast<const uint2*>(kb + (size_t)t * kv_n);
            vv[u] = *reinterpret_cast<const uint2*>(vb + (size_t)t * kv_n);
        }
    };
    int t0 = warp * kAttKeys;
    for (; FUSED ? t0 + kAttKeys <= pos : t0 <= pos; t0 += kAttWarps * kAttKeys) {
        uint2 kv[kAttKeys], vv[kAttKeys];
        load4(kv, vv, t0);
        round4(kv, vv, pos + 1 - t0);
    }
    // The round that holds position pos is a warp's last, behind a loop that knows nothing of it (64 registers instead of 71: 16
    // sequences at position 1900, step of two 7B layers, 415 -> 335 us).
    if (FUSED && t0 <= pos) {
        uint2 kv[kAttKeys], vv[kAttKeys];
        load4(kv, vv, t0);
        const size_t at = (size_t)m * kv_n + (size_t)(h / kv_mul) * HS + lane * 4;
        const uint2 k = rotate(*reinterpret_cast<const uint2*>(knew + at)), v = *reinterpret_cast<const uint2*>(vnew + at);
#pragma unroll
        for (int u = 0; u < kAttKeys; u++)
            if (t0 + u >= pos) { kv[u] = k; vv[u] = v; }   // (those behind it do not count, but must not bring in a NaN)
        if (h % kv_mul == 0) {
            *reinterpret_cast<uint2*>(kc + head_at + (size_t)pos * kv_n) = k;
            *reinterpret_cast<uint2*>(vc + head_at + (size_t)pos * kv_n) = v;
        }
        round4(kv, vv, pos + 1 - t0);
    }
    __shared__ float s_m[kAttWarps], s_l[kAttWarps], s_acc[kAttWarps][HS];
    if (lane == 0) { s_m[warp] = mx; s_l[warp] = l; }
#pragma unroll
    for (int j = 0; j < 4; j++) s_acc[warp][lane * 4 + j] = acc[j];
    __syncthreads();
    if (threadIdx.x < HS) {
        float M = -CUDART_INF_F;
        for (int w = 0; w < kAttWarps; w++) M = fmaxf(M, s_m[w]);
        float a = 0.f, L = 0.f;
        for (int w = 0; w < kAttWarps; w++) {
            if (s_m[w] != -CUDART_INF_F) {
                const float e = expf(s_m[w] - M);
                a += s_acc[w][threadIdx.x] * e;
                L += s_l[w] * e;
            }
        }
        out[((size_t)m * n_heads + h) * HS + threadIdx.x] = __float2half(L > 0.f ? a / L : 0.f);
    }
}

// ---- causal attention of a prompt (rows = consecutive positions of one sequence) on the tensor cores ----
// The (row, head) kernel above re-reads the whole K/V history once per row; for a prompt that is rows^2 / 2 cache rows per
// head. Here a CTA takes 64 consecutive rows of one head (a warp: 16 of them) and walks the keys in chunks of 64, so a cache
// row is read once per 64 query rows. S = Q K^T and O += P V run as mma.sync m16n8k16 (fp16 in, fp32 out); the scores are
// scaled and rounded to fp16 exactly where MultiHeadAttention stores them (gpu_kernels.h:171-175), the softmax is the online
// form in fp32, P is rounded to fp16 for the second product (the reference's att buffer is fp16 too) and its row sums come
// from the same product with a column of ones. head_size 128. Keys beyond the last row's position are zero-filled and masked.
//
// It runs at 0.43 of the rate mma.sync reaches here (1024 clocks per 64 x 64 block and SM at that rate; 2000 rows); the rest is the
// softmax between the two products and, below a thousand rows, CTAs of unequal length that do not fill the SMs. Chunks are copied
// with cp.async one ahead of the math; both operands come through ldmatrix (K as it lies, V transposed); only the chunks a
// warp's diagonal crosses are masked; the running output is scaled only when a maximum moved; the CTAs with the most keys
// start first; three CTAs of four warps per SM cover each other's softmax. 2000 rows of 32 heads: 231 -> 143 us, 512 rows:
// 42 -> 22 us (before: single-buffered chunks, 4-byte fragment loads of K, every chunk masked).
constexpr int kAtRows = 64, kAtKeys = 64, kAtLd = 136;   // 136 halfs = 272 B between rows: conflict-free fragment loads
constexpr int kAtChunk = kAtKeys * kAtLd;                // halfs of a chunk of K or V
constexpr size_t kAtSmem = 2 * 2 * (size_t)kAtChunk * sizeof(__half);   // two buffers of K and V

__device__ __forceinline__ void mma_f16(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// 16 bytes to shared memory, zeros where !valid (src is readable either way)
__device__ __forceinline__ void cp_async16_or_zero(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// grid (heads, ceil(n / 64)), block 128. kc / vc point at this layer's cache rows of the sequence (position 0).
__global__ void __launch_bounds__(128, 3) attention_prefill_kernel(__half* out, const __half* q, int ldq, const __half* kc, const __half* vc, int n_heads, int kv_mul,
                                                                   int n, int pos0, int kv_n) {
    griddep_wait();   // launched with programmatic stream serialisation: wait for the producer, then let the consumer's prologue start
    griddep_launch_dependents();
    constexpr int HS = 128;
    extern __shared__ __align__(16) __half at_smem[];   // [2 buffers][K, V][kAtKeys][kAtLd]
    const uint32_t smem = (uint32_t)__cvta_generic_to_shared(at_smem);
    const int h = blockIdx.x, m0 = (int)(gridDim.y - 1 - blockIdx.y) * kAtRows;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int row_a = m0 + warp * 16 + g, row_b = row_a + 8;          // this thread's two query rows
    const int last_pos = pos0 + n - 1;                                // newest cache row that is valid
    const int pos_a = min(pos0 + row_a, last_pos), pos_b = min(pos0 + row_b, last_pos);
    const int warp_first = min(pos0 + m0 + warp * 16, last_pos);      // newest key that every row of this warp attends to
    const int warp_last = min(pos0 + m0 + warp * 16 + 15, last_pos);  // newest key any row of this warp attends to
    const int cta_last = min(pos0 + m0 + kAtRows - 1, last_pos);
    const size_t head_off = (size_t)(h / kv_mul) * HS;

    const int piece = (threadIdx.x & 15) * 8, row0 = threadIdx.x >> 4;   // this thread copies rows row0, row0 + 8, ... of a chunk
    auto load_chunk = [&](int t0, int buf) {
        const uint32_t dst = smem + (uint32_t)(2 * buf * kAtChunk + row0 * kAtLd + piece) * 2;
#pragma unroll
        for (int i = 0; i < kAtKeys / 8; i++) {
            const int key = t0 + row0 + 8 * i;
            const bool valid = key <= cta_last;
            const size_t off = (size_t)(valid ? key : 0) * kv_n + head_off + piece;
            cp_async16_or_zero(dst + i * 8 * kAtLd * 2, kc + off, valid);
            cp_async16_or_zero(dst + (kAtChunk + i * 8 * kAtLd) * 2, vc + off, valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_chunk(0, 0);

    // Q fragments: 8 k-steps of 16 dims; rows past the prompt read as zero
    uint32_t qa[8][4];
    {
        const __half* qa_p = q + (size_t)row_a * ldq + (size_t)h * HS;
        const __half* qb_p = q + (size_t)row_b * ldq + (size_t)h * HS;
#pragma unroll
        for (int s = 0; s < 8; s++) {
            qa[s][0] = row_a < n ? *reinterpret_cast<const uint32_t*>(qa_p + 16 * s + 2 * t) : 0u;
            qa[s][1] = row_b < n ? *reinterpret_cast<const uint32_t*>(qb_p + 16 * s + 2 * t) : 0u;
            qa[s][2] = row_a < n ? *reinterpret_cast<const uint32_t*>(qa_p + 16 * s + 2 * t + 8) : 0u;
            qa[s][3] = row_b < n ? *reinterpret_cast<const uint32_t*>(qb_p + 16 * s + 2 * t + 8) : 0u;
        }
    }
    const float alpha = (float)(1.0 / sqrt((double)HS));
    float o[16][4], l[4] = {0.f, 0.f, 0.f, 0.f};   // l: row sums of P (rows a: elements 0, 1; rows b: 2, 3)
#pragma unroll
    for (int d = 0; d < 16; d++) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
    float mx_a = -CUDART_INF_F, mx_b = -CUDART_INF_F;

    for (int t0 = 0, buf = 0; t0 <= cta_last; t0 += kAtKeys, buf ^= 1) {
        if (t0 + kAtKeys <= cta_last) {
            load_chunk(t0 + kAtKeys, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();           // the chunk has landed for every thread
        if (t0 <= warp_last) {     // (warp-uniform; else nothing of this chunk is visible to the warp's rows)
            const uint32_t sk = smem + (uint32_t)(2 * buf * kAtChunk) * 2, sv = sk + kAtChunk * 2;
            // S = Q K^T for 16 rows x 64 keys, scaled and rounded to fp16 as the reference stores the scores
            __half2 sc[8][2];
#pragma unroll
            for (int jj = 0; jj < 8; jj += 4) {
                float c[4][4];
#pragma unroll
                for (int j = 0; j < 4; j++) c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
#pragma unroll
                for (int s = 0; s < 8; s += 2) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        uint32_t b0, b1, b2, b3;
                        const uint32_t addr = sk + (uint32_t)((8 * (jj + j) + (lane & 7)) * kAtLd + 16 * s + 8 * (lane >> 3)) * 2;
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3) : "r"(addr) : "memory");
                        mma_f16(c[j], qa[s], b0, b1);
                        mma_f16(c[j], qa[s + 1], b2, b3);
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    sc[jj + j][0] = __floats2half2_rn(c[j][0] * alpha, c[j][1] * alpha);
                    sc[jj + j][1] = __floats2half2_rn(c[j][2] * alpha, c[j][3] * alpha);
                }
            }
            if (t0 + kAtKeys - 1 > warp_first) {   // the diagonal, or the end of the keys
                const __half ninf = __ushort_as_half((unsigned short)0xFC00u);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int key = t0 + 8 * j + 2 * t;
                    sc[j][0] = __halves2half2(key <= pos_a ? __low2half(sc[j][0]) : ninf, key + 1 <= pos_a ? __high2half(sc[j][0]) : ninf);
                    sc[j][1] = __halves2half2(key <= pos_b ? __low2half(sc[j][1]) : ninf, key + 1 <= pos_b ? __high2half(sc[j][1]) : ninf);
                }
            }
            __half2 cm_a = sc[0][0], cm_b = sc[0][1];
#pragma unroll
            for (int j = 1; j < 8; j++) {
                cm_a = __hmax2(cm_a, sc[j][0]);
                cm_b = __hmax2(cm_b, sc[j][1]);
            }
            float ca = fmaxf(__low2float(cm_a), __high2float(cm_a)), cb = fmaxf(__low2float(cm_b), __high2float(cm_b));
            ca = fmaxf(ca, __shfl_xor_sync(0xffffffffu, ca, 1));
            ca = fmaxf(ca, __shfl_xor_sync(0xffffffffu, ca, 2));
            cb = fmaxf(cb, __shfl_xor_sync(0xffffffffu, cb, 1));
            cb = fmaxf(cb, __shfl_xor_sync(0xffffffffu, cb, 2));
            // key 0 is visible to every row, so after the first chunk the running maxima are finite
            const float nm_a = fmaxf(mx_a, ca), nm_b = fmaxf(mx_b, cb);
            if (__any_sync(0xffffffffu, nm_a != mx_a || nm_b != mx_b)) {
                const float corr_a = __expf(mx_a - nm_a), corr_b = __expf(mx_b - nm_b);
#pragma unroll
                for (int d = 0; d < 16; d++) { o[d][0] *= corr_a; o[d][1] *= corr_a; o[d][2] *= corr_b; o[d][3] *= corr_b; }
                l[0] *= corr_a; l[1] *= corr_a; l[2] *= corr_b; l[3] *= corr_b;
                mx_a = nm_a; mx_b = nm_b;
            }
            // P = exp(S - max), rounded to fp16, as A fragments (k-step jj covers keys 16 jj .. 16 jj + 15); O += P V with the V
            // fragments through ldmatrix.trans (V is [key][dim]; the product wants keys along k)
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                uint32_t pa[4];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const float2 fa = __half22float2(sc[2 * jj + u][0]), fb = __half22float2(sc[2 * jj + u][1]);
                    pa[2 * u] = pack_h2(__expf(fa.x - nm_a), __expf(fa.y - nm_a));
                    pa[2 * u + 1] = pack_h2(__expf(fb.x - nm_b), __expf(fb.y - nm_b));
                }
                mma_f16(l, pa, 0x3C003C00u, 0x3C003C00u);
#pragma unroll
                for (int d = 0; d < 16; d += 2) {
                    uint32_t v0, v1, v2, v3;
                    const uint32_t addr = sv + (uint32_t)((16 * jj + (lane & 15)) * kAtLd + 8 * d + 8 * (lane >> 4)) * 2;
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(v0), "=r"(v1), "=r"(v2), "=r"(v3) : "r"(addr) : "memory");
                    mma_f16(o[d], pa, v0, v1);
                    mma_f16(o[d + 1], pa, v2, v3);
                }
            }
        }
        __syncthreads();   // the chunk is consumed: its buffer is filled again in the next round
    }
    const float inv_a = l[0] > 0.f ? 1.0f / l[0] : 0.f, inv_b = l[2] > 0.f ? 1.0f / l[2] : 0.f;
#pragma unroll
    for (int d = 0; d < 16; d++) {
        if (row_a < n) *reinterpret_cast<uint32_t*>(out + ((size_t)row_a * n_heads + h) * HS + 8 * d + 2 * t) = pack_h2(o[d][0] * inv_a, o[d][1] * inv_a);
        if (row_b < n) *reinterpret_cast<uint32_t*>(out + ((size_t)row_b * n_heads + h) * HS + 8 * d + 2 * t) = pack_h2(o[d][2] * inv_b, o[d][3] * inv_b);
    }
}

// Rows of `len` elements to every step-th row of dst (set-up only: q|k|v behind one another, gate and up in turn). A block
// takes whole rows, 16 bytes per access where the rows are a multiple of that (the packed words always are). One 16-bit
// element per thread with a division for its row made the set-up of four 7B layers 50 ms longer than the copies it replaced.
template <typename T>
__global__ void place_rows_kernel(T* dst, const T* src, int len, int step, int rows) {
    for (int row = blockIdx.x; row < rows; row += gridDim.x)
        for (int i = threadIdx.x; i < len; i += blockDim.x) dst[(size_t)row * step * len + i] = src[(size_t)row * len + i];
}

// both position words (device, pinned host) to `pos`, in stream order
__global__ void set_pos_kernel(int* pos_dev, volatile int* pos_pinned, int pos) {
    griddep_wait();   // launched with programmatic stream serialisation: wait for the producer, then let the consumer's prologue start
    griddep_launch_dependents();
    *pos_dev = pos;
    *pos_pinned = pos;
}

// mat_vec_kernel (gpu_kernels.h:117-147) for B rows of x at once: a warp takes one classifier row and B dot products, so the
// classifier is read once per step, not once per sequence. x rows sit in shared memory. B <= 16.
__global__ void __launch_bounds__(256) matvec_f16_rows_kernel(__half* y, const __half* x, const __half* w, int n, int d, int B, int y_stride) {
    griddep_wait();   // launched with programmatic stream serialisation: wait for the producer, then let the consumer's prologue start
    griddep_launch_dependents();
    extern __shared__ __align__(16) __half sx[];
    for (int i = threadIdx.x; i < B * n / 8; i += blockDim.x) reinterpret_cast<uint4*>(sx)[i] = reinterpret_cast<const uint4*>(x)[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int row = blockIdx.x * 8 + warp; row < d; row += gridDim.x * 8) {
        float acc[16];
#pragma unroll
        for (int b = 0; b < 16; b++) acc[b] = 0.f;
        const uint4* wr = reinterpret_cast<const uint4*>(w + (size_t)row * n);
        for (int i = lane; i < n / 8; i += 32) {
            const uint4 wv = ldg_stream(wr + i);
            const __half2* wh = reinterpret_cast<const __half2*>(&wv);
#pragma unroll
            for (int b = 0; b < 16; b++) {
                if (b < B) {
                    const uint4 xv = reinterpret_cast<const uint4*>(sx + (size_t)b * n)[i];
                    const __half2* xh = reinterpret_cast<const __half2*>(&xv);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float2 a = __half22float2(wh[j]), c = __half22float2(xh[j]);
                        acc[b] = fmaf(a.x, c.x, acc[b]);
                        acc[b] = fmaf(a.y, c.y, acc[b]);
                    }
                }
            }
        }
#pragma unroll
        for (int b = 0; b < 16; b++) {
            if (b < B) {
                const float v = warp_sum(acc[b]);
                if (lane == 0) y[(size_t)b * y_stride + row] = __float2half(v);
            }
        }
    }
}

// The same product on mma.sync m16n8k16 when the shapes allow (n % 32 == 0, d % 16 == 0): a CTA takes 16 classifier rows, its
// eight warps an eighth of n each, and the warps' partial tiles are added in warp order (bit-reproducible). The k index of
// an MMA is only a summation label, so thread (g, t) feeds the eight consecutive weights it loaded with one 16-byte load
// (rows g and g + 8, inputs 32 c + 8 t ..) as A and the same eight inputs of batch row g as B; fp32 accumulation as in
// mat_vec_kernel. HBM-bound when all SMs stream: with a warp over the whole of n and 128 rows per CTA, a rank's or a small
// model's few thousand rows left most SMs idle (4000 x 4096, 8 rows: 70 us; one 16-row tile per CTA: 18 us).
constexpr int kClsWarps = 8;
template <int NT>
__global__ void __launch_bounds__(kClsWarps * 32) classifier_rows_kernel(__half* y, const __half* x, const __half* w, int n, int d, int B, int y_stride) {
    __shared__ float part[kClsWarps][NT][4][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int chunks = n / 32, c_begin = chunks * warp / kClsWarps, c_end = chunks * (warp + 1) / kClsWarps;
    const int tile = blockIdx.x;
    const uint4* wa = reinterpret_cast<const uint4*>(w + (size_t)(tile * 16 + g) * n) + t;
    const uint4* wb = reinterpret_cast<const uint4*>(w + (size_t)(tile * 16 + g + 8) * n) + t;
    constexpr int U = 4;
    uint4 a[U], b[U];
    auto fetch = [&](int c0) {
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c0 + u < c_end) { a[u] = ldg_stream(wa + 4 * (c0 + u)); b[u] = ldg_stream(wb + 4 * (c0 + u)); }
    };
    fetch(c_begin);   // the weights do not depend on the previous kernel: the first loads run while it finishes
    griddep_wait();
    griddep_launch_dependents();
    const uint4* xr[NT];
    bool ok[NT];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        ok[nt] = g + 8 * nt < B;
        xr[nt] = reinterpret_cast<const uint4*>(x + (size_t)(ok[nt] ? g + 8 * nt : 0) * n) + t;
    }
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    for (int c0 = c_begin; c0 < c_end; c0 += U) {
        uint4 ca[U], cb[U];
#pragma unroll
        for (int u = 0; u < U; u++) { ca[u] = a[u]; cb[u] = b[u]; }
        fetch(c0 + U);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (c0 + u < c_end) {
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    uint4 xv = make_uint4(0, 0, 0, 0);
                    if (ok[nt]) xv = xr[nt][4 * (c0 + u)];
                    const uint32_t A0[4] = {ca[u].x, cb[u].x, ca[u].y, cb[u].y}, A1[4] = {ca[u].z, cb[u].z, ca[u].w, cb[u].w};
                    mma_f16(acc[nt], A0, xv.x, xv.y);
                    mma_f16(acc[nt], A1, xv.z, xv.w);
                }
            }
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) part[warp][nt][e][lane] = acc[nt][e];
    __syncthreads();
    for (int i = threadIdx.x; i < NT * 128; i += kClsWarps * 32) {
        const int l = i & 31, e = (i >> 5) & 3, nt = i >> 7;
        const int row = 8 * nt + 2 * (l & 3) + (e & 1);
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < kClsWarps; k++) v += part[k][nt][e][l];
        if (row < B) y[(size_t)row * y_stride + tile * 16 + (l >> 2) + 8 * (e >> 1)] = __float2half(v);
    }
}

// argmax per row (lowest index among equal maxima, like q4_argmax) and the hand-off of batched decode: the id becomes
// the sequence's next token when that position is past its prompt, and the sequence moves on by one position.
__global__ void __launch_bounds__(1024) argmax_rows_kernel(const __half* logits, int vocab, int* tokens, long long tok_stride, int* pos, int n_prompt) {
    griddep_wait();   // launched with programmatic stream serialisation: wait for the producer, then let the consumer's prologue start
    griddep_launch_dependents();
    __shared__ float sval[32];
    __shared__ int sidx[32];
    const int s = blockIdx.x;
    const __half* x = logits + (size_t)s * vocab;
    float best = -CUDART_INF_F;
    int bi = 0x7fffffff;
    const int nvec = (vocab % 8 == 0) ? vocab / 8 : 0;   // rows of a multiple of 8 halfs start 16-byte aligned
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
        const uint4 v = reinterpret_cast<const uint4*>(x)[i];
        const __half* h = reinterpret_cast<const __half*>(&v);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float f = __half2float(h[j]);
            if (f > best) { best = f; bi = i * 8 + j; }
        }
    }
    for (int i = nvec * 8 + threadIdx.x; i < vocab; i += blockDim.x) {
        const float v = __half2float(x[i]);
        if (v > best) { best = v; bi = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if ((threadIdx.x & 31) == 0) { sval[threadIdx.x >> 5] = best; sidx[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++)
            if (sval[w] > best || (sval[w] == best && sidx[w] < bi)) { best = sval[w]; bi = sidx[w]; }
        const int p = pos[s];
        if (p + 1 >= n_prompt) tokens[(long long)s * tok_stride + p + 1] = bi == 0x7fffffff ? 0 : bi;
        pos[s] = p + 1;
    }
}

}  // namespace

// ------------------------------------------------------------------------------------------------------------
// row buffers and the interleaved weight copies the GEMM prefers (built on first use)
// ------------------------------------------------------------------------------------------------------------
struct q4_rows {
    int cap = 0;   // rows the buffers hold
    __half *X = nullptr, *XB = nullptr, *Q = nullptr, *K = nullptr, *V = nullptr, *ATT = nullptr, *G = nullptr;
    __half *QKV = nullptr, *Y = nullptr;   // GEMM path: [rows][q_n + 2 kv_n], written by one GEMM; [rows][dim], a projection's result
    int *row_seq = nullptr, *row_pos = nullptr;
    float2* rope = nullptr;   // [seq_len][head_size / 2] (cos, sin)
    void* ws = nullptr;
    size_t ws_bytes = 0;
    // GEMM path, per layer four matrices: q|k|v stacked along the output axis, gate and up row by row in turn (row 2j = gate j,
    // 2j + 1 = up j: the GEMM's epilogue finds both in neighbouring lanes and writes silu(gate) * up), o, down; one launch each.
    // Interleaved copy of the packed words, and for the joined ones a copy of zeros and scales in the same order.
    struct GemmMat { uint32_t* wi; q4_qweight w; int K, N; };
    std::vector<GemmMat> gm;     // [layer * 4 + {0 qkv, 1 o, 2 gate|up, 3 down}]
    std::vector<void*> allocs;
};

#ifdef Q4_TEST_BUILD
static int g_fail_alloc = -1;   // host-side fault injection: the allocation after this many more fails, once
extern "C" void q4_test_fail_rows_alloc(int n) { g_fail_alloc = n; }
static bool g_fail_set_pos = false;   // the next launch of a prompt's position words fails, once
extern "C" void q4_test_fail_set_pos() { g_fail_set_pos = true; }
#endif

static int rows_alloc(q4_rows* r, void** p, size_t bytes) {
#ifdef Q4_TEST_BUILD
    if (g_fail_alloc >= 0 && g_fail_alloc-- == 0) return Q4_ERR_CUDA;
#endif
    Q4_CUDA_TRY(cudaMalloc(p, bytes));
    r->allocs.push_back(*p);
    return Q4_OK;
}

void q4_rows_free(q4_model* m) {
    if (!m->rows) return;
    for (void* p : m->rows->allocs) cudaFree(p);
    delete m->rows;
    m->rows = nullptr;
}

// Status word of the GEMM workspace (Q4_ERR_TIMEOUT after a bounded device-side wait ran out); the device is idle.
int q4_rows_status(q4_model* m) {
    if (!m->rows || !m->rows->ws) return Q4_OK;
    int st[2] = {0, 0};
    Q4_CUDA_TRY(cudaMemcpy(st, m->rows->ws, sizeof(st), cudaMemcpyDeviceToHost));
    if (st[0]) fprintf(stderr, "q4 prefill / batch path: a bounded device-side wait of the GEMM ran out (status %d, location 0x%x)\n", st[0], st[1]);
    return st[0];
}

// More than this many rows go through the tcgen05 GEMM, fewer through the mma.sync kernels that stream the packed weights.
constexpr int kSkinnyRows = 16;

static int rows_grow(q4_model* m, q4_rows* r, int rows) {
    const q4_config& c = m->cfg;
    int e;
#define RTRY(expr) do { e = (expr); if (e != Q4_OK) return e; } while (0)
    if (r->gm.empty() && rows > kSkinnyRows) {
        r->gm.assign((size_t)c.n_layers * 4, q4_rows::GemmMat{});
        for (int l = 0; l < c.n_layers; l++) {
            const DevLayer& L = m->layers[l];
            const DevQW* groups[4][3] = {{&L.q, &L.k, &L.v}, {&L.o, nullptr, nullptr}, {&L.gate, &L.up, nullptr}, {&L.down, nullptr, nullptr}};
            for (int i = 0; i < 4; i++) {
                q4_rows::GemmMat& gmat = r->gm[(size_t)l * 4 + i];
                const int K = groups[i][0]->K;
                int N = 0, parts = 0;
                for (int j = 0; j < 3 && groups[i][j]; j++) { N += groups[i][j]->N; parts++; }
                gmat.K = K;
                gmat.N = N;
                RTRY(rows_alloc(r, (void**)&gmat.wi, (size_t)N * q4_pw(K) * 4));
                uint32_t* zeros = nullptr;
                uint16_t* scales = nullptr;
                if (parts > 1) {
                    RTRY(rows_alloc(r, (void**)&zeros, (size_t)N * q4_pz(K) * 4));
                    RTRY(rows_alloc(r, (void**)&scales, (size_t)N * q4_groups(K) * 2));
                }
                // part j's rows go to rows row0, row0 + step, ... of the joined matrix
                const int step = i == 2 ? 2 : 1;
                size_t row0 = 0;
                auto place = [&](void* dst, const void* src, size_t row_bytes, int n) {   // row_bytes is a multiple of 2; both ends are 16-byte aligned where it is one of 16
                    char* to = (char*)dst + row0 * row_bytes;
                    if (row_bytes % 16 == 0) place_rows_kernel<<<148 * 8, 256>>>((uint4*)to, (const uint4*)src, (int)(row_bytes / 16), step, n);
                    else place_rows_kernel<<<148 * 8, 256>>>((uint16_t*)to, (const uint16_t*)src, (int)(row_bytes / 2), step, n);
                };
                for (int j = 0; j < parts; j++) {
                    const DevQW* q = groups[i][j];
                    place(gmat.wi, q->w.weight, (size_t)q4_pw(K) * 4, q->N);
                    if (parts > 1) {
                        place(zeros, q->w.zeros, (size_t)q4_pz(K) * 4, q->N);
                        place(scales, q->w.scales, (size_t)q4_groups(K) * 2, q->N);
                    }
                    row0 += i == 2 ? 1 : q->N;
                }
                Q4_CUDA_TRY(cudaGetLastError());
                RTRY(q4_gemm_interleave_weights(nullptr, gmat.wi, gmat.wi, K, N));   // (word by word: in place)
                gmat.w.weight = gmat.wi;   // (the GEMM reads the interleaved words; this field only has to be non-null)
                gmat.w.zeros = parts > 1 ? zeros : groups[i][0]->w.zeros;
                gmat.w.scales = parts > 1 ? scales : groups[i][0]->w.scales;
            }
        }
        Q4_CUDA_TRY(cudaDeviceSynchronize());
    }
    if (!r->rope) {
        RTRY(rows_alloc(r, (void**)&r->rope, sizeof(float2) * (size_t)c.seq_len * (m->head_size / 2)));
        rope_rows_table_kernel<<<148 * 2, 256>>>(r->rope, c.seq_len, m->head_size, c.rope_theta);
        Q4_CUDA_TRY(cudaGetLastError());
        Q4_CUDA_TRY(cudaDeviceSynchronize());
    }
    if (rows > r->cap) {
        const int cap = (rows + 63) / 64 * 64;
        const size_t dim = c.dim, hk = m->h_kc;
        RTRY(rows_alloc(r, (void**)&r->X, 2 * cap * dim));
        RTRY(rows_alloc(r, (void**)&r->XB, 2 * cap * dim));
        RTRY(rows_alloc(r, (void**)&r->Q, 2 * (size_t)cap * m->q_n));
        RTRY(rows_alloc(r, (void**)&r->K, 2 * (size_t)cap * m->kv_n));
        RTRY(rows_alloc(r, (void**)&r->V, 2 * (size_t)cap * m->kv_n));
        RTRY(rows_alloc(r, (void**)&r->ATT, 2 * (size_t)cap * m->q_n));
        RTRY(rows_alloc(r, (void**)&r->G, 2 * cap * hk));
        RTRY(rows_alloc(r, (void**)&r->QKV, 2 * (size_t)cap * (m->q_n + 2 * m->kv_n)));
        RTRY(rows_alloc(r, (void**)&r->Y, 2 * cap * dim));
        RTRY(rows_alloc(r, (void**)&r->row_seq, sizeof(int) * cap));
        RTRY(rows_alloc(r, (void**)&r->row_pos, sizeof(int) * cap));
        size_t ws = 0;
        const int shapes[4][2] = {{c.dim, m->q_n + 2 * m->kv_n}, {m->o_kc, c.dim}, {c.dim, 2 * m->h_kc}, {m->h_kc, c.dim}};
        for (auto& s : shapes)
            for (int mm : {1, 16, 17, 64, 65, cap}) ws = std::max(ws, q4_matmul_q4_batched_workspace_bytes(std::min(mm, cap), s[0], s[1]));
        RTRY(rows_alloc(r, &r->ws, ws));
        Q4_CUDA_TRY(cudaMemset(r->ws, 0, ws));
        Q4_CUDA_TRY(cudaDeviceSynchronize());   // the fill runs on the default stream; the caller's need not wait for that one, and the GEMM counts from zero
        r->ws_bytes = ws;
        r->cap = cap;
    }
#undef RTRY
    return Q4_OK;
}

// Buffers for up to `rows` rows (grown on demand) and, once and only when the GEMM will be used, the interleaved weight copies.
// Complete or nothing: when an allocation or a copy fails part-way, what this call made is released and the next call starts over.
static int rows_prepare(q4_model* m, int rows) {
    if (m->column || m->head_size != 128 || (m->cfg.dim % 128) || (m->o_kc % 128) || (m->h_kc % 128)) return Q4_ERR_UNSUPPORTED_SIZE;
    if (!m->rows) m->rows = new q4_rows();
    q4_rows* r = m->rows;
    if (rows <= r->cap && r->rope && (rows <= kSkinnyRows || !r->gm.empty())) return Q4_OK;
    const q4_rows before = *r;   // (buffers that were outgrown stay allocated: a captured batch step may hold their addresses)
    const int e = rows_grow(m, r, rows);
    if (e != Q4_OK) {
        for (size_t i = before.allocs.size(); i < r->allocs.size(); i++) cudaFree(r->allocs[i]);
        *r = before;
        cudaGetLastError();   // (reported; a later call's launch check must not find it)
    }
    return e;
}

// Sum of the ranks' partial [count] vectors: NCCL when it is attached, the communicator's choice says so (large messages)
// and the caller allows it (a prompt's rows); else the one-shot peer push in pieces its inbox holds (always for the
// batched-decode step, which is replayed from a CUDA graph and keeps to kernels of this library).
static int rows_all_reduce(q4_model* m, cudaStream_t s, __half* buf, size_t count, bool allow_nccl) {
    if (m->g == 1) return Q4_OK;
    for (size_t at = 0; at < count;) {
        const bool nccl = allow_nccl && q4_comm_prefers_nccl(m->comm, (int)std::min<size_t>(count - at, (size_t)1 << 30));
        const size_t n = nccl ? count - at : std::min<size_t>(count - at, (size_t)Q4_COMM_MAX_HALFS);
        if (int e = nccl ? q4_all_reduce(m->comm, s, (uint16_t*)(buf + at), (int)n) : q4_all_reduce_peer_push(m->comm, s, (uint16_t*)(buf + at), (int)n)) return e;
        at += n;
    }
    return Q4_OK;
}

// What the caller needs behind the last layer: every row (batched decode), the last row (a prompt: only its logits are asked for)
// or nothing but the K/V rows (a prompt whose last position follows through another path).
enum RowsWanted { WANT_ALL, WANT_LAST, WANT_CACHE };

// All layers for `n` rows, from their tokens' embeddings on; K/V rows go to (kc, vc) with `seq_stride` halfs between sequences.
// embed.pos0 >= 0: the rows are positions pos0 .. pos0 + n - 1 of one sequence (prompt); -1: one row per sequence (batched decode).
// In the last layer the rows that nobody asks for end at their K/V row: no later layer reads them.
// embed.row_seq, embed.row_pos: the rows' sequences and positions, on the device.
static int rows_layers(q4_model* m, cudaStream_t s, int n, const Embed& embed, __half* kc, __half* vc, long long seq_stride, RowsWanted want) {
    q4_rows* r = m->rows;
    const int *row_seq = embed.row_seq, *row_pos = embed.row_pos, pos0 = embed.pos0;
    const q4_config& c = m->cfg;
    const int g = m->g, dim = c.dim;
    const int heads = c.n_heads / g, kv_heads = c.n_kv_heads / g;
    int e;
#define OP(expr) do { e = (expr); if (e != Q4_OK) return e; } while (0)
    // mat: 0 q|k|v, 1 o, 2 gate / up with silu(gate) * up, 3 down; residual: y = product + y / g
    auto gemm = [&](__half* y, const __half* x, int l, int mat, bool residual) {
        const q4_rows::GemmMat& gmat = r->gm[(size_t)l * 4 + mat];
        return q4_gemm_launch(s, (uint16_t*)y, (const uint16_t*)x, &gmat.w, gmat.wi, n, gmat.K, gmat.N, residual ? (const uint16_t*)y : nullptr, 1.0f / g, mat == 2, true, r->ws,
                              r->ws_bytes);
    };
    // k and v alone: the rows of q|k|v behind q's
    auto gemm_kv = [&](__half* y, const __half* x, int l) {
        q4_rows::GemmMat part = r->gm[(size_t)l * 4];
        part.wi += (size_t)m->q_n * q4_pw(part.K);
        part.w.weight = part.wi;
        part.w.zeros += (size_t)m->q_n * q4_pz(part.K);
        part.w.scales += (size_t)m->q_n * q4_groups(part.K);
        return q4_gemm_launch(s, (uint16_t*)y, (const uint16_t*)x, &part.w, part.wi, n, part.K, 2 * m->kv_n, nullptr, 1.0f / g, false, true, r->ws, r->ws_bytes);
    };
    // q, k, v of the rows: three buffers (few-rows kernels) or three slices of the fused GEMM's output (two in a prompt's last layer)
    const int nqkv = m->q_n + 2 * m->kv_n;
    const bool skinny = n <= kSkinnyRows;
    // (the attention of batched decode takes k and v as the few-rows kernels leave them, and behind the GEMMs the last layer's down
    // projection would still have to be added)
    if (!skinny && (pos0 < 0 || want == WANT_ALL)) return Q4_ERR_INVALID;
    // A prompt's rows on one GPU: the o and down projections leave their result in Y and the next RMSNorm adds it to x
    // (with more ranks the partial sums have to be exchanged as x first: the GEMM adds the residual itself).
    const bool fused_add = !skinny && g == 1;
    if (pos0 >= 0 && !skinny) Q4_CUDA_TRY(cudaFuncSetAttribute(attention_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAtSmem));
    auto norm = [&](const __half* w, const __half* y) {
        if (y) launch_rows(rmsnorm_rows_kernel<ROW_ADD>, dim3(n), dim3(kRowThreads), 0, s, r->XB, r->X, y, w, dim, Embed{});
        else launch_rows(rmsnorm_rows_kernel<ROW_X>, dim3(n), dim3(kRowThreads), 0, s, r->XB, r->X, (const __half*)nullptr, w, dim, Embed{});
    };
    for (int l = 0; l < c.n_layers; l++) {
        const DevLayer& L = m->layers[l];
        const long long loff = (long long)l * c.seq_len * m->kv_n;
        if (l == 0) launch_rows(rmsnorm_rows_kernel<ROW_EMBED>, dim3(n), dim3(kRowThreads), 0, s, r->XB, r->X, (const __half*)nullptr, (const __half*)L.rms_att, dim, embed);
        else norm((const __half*)L.rms_att, fused_add ? r->Y : nullptr);
        // The last layer of a prompt: nobody reads the other rows' queries (of 70B's q|k|v four fifths; 333 rows behind 700 of one 70B layer
        // 222 us, 203 so; 2000 rows of two 7B layers 1113, 1064), so k and v alone go through the GEMM and the last row's query, if asked
        // for, through the batch-1 product.
        const bool kv_only = !skinny && l == c.n_layers - 1 && want != WANT_ALL;
        if (kv_only) {
            if (want == WANT_LAST) OP(q4_matmul_q4(s, (uint16_t*)r->Q, (const uint16_t*)(r->XB + (size_t)(n - 1) * dim), &L.q.w, dim, m->q_n, 0, 1, -1, nullptr));
            OP(gemm_kv(r->QKV, r->XB, l));
        } else if (skinny) {
            OP(q4_qkv_rows_launch(s, (uint16_t*)r->Q, (uint16_t*)r->K, (uint16_t*)r->V, (const uint16_t*)r->XB, &L.q.w, &L.k.w, &L.v.w, n, dim, m->q_n, m->kv_n, pos0 < 0));
        } else {
            OP(gemm(r->QKV, r->XB, l, 0, false));
        }
        __half* qp = skinny || kv_only ? r->Q : r->QKV;
        const __half* kp = skinny ? r->K : kv_only ? r->QKV : r->QKV + m->q_n;
        const __half* vp = skinny ? r->V : kp + m->kv_n;
        const int ldq = kv_only ? 0 : skinny ? m->q_n : nqkv, ldkv = kv_only ? 2 * m->kv_n : skinny ? m->kv_n : nqkv;   // (kv_only: one query, the last row's)
        if (pos0 >= 0) {   // (batched decode: the attention kernel rotates and files)
            const int queries = kv_only && want == WANT_CACHE ? 0 : heads;
            launch_rows(rope_store_rows_kernel, dim3(n, q4_div_up((queries + 2 * kv_heads) * 8, 256)), dim3(256), 0, s, qp, kp, vp, ldq, ldkv, kc, vc, queries, kv_heads,
                        r->rope, row_seq, row_pos, seq_stride, loff, kv_only ? n - 1 : 0);
        }
        if (l == c.n_layers - 1 && want != WANT_ALL) {
            if (want == WANT_CACHE) break;
            // one row: the split attention and the products of the batch-1 path (70B: o, gate / up and down 147 us with the few-rows kernels,
            // about 105 so, and less error)
            const size_t last = (size_t)(n - 1);
            uint16_t* x = (uint16_t*)(r->X + last * dim);
            OP(q4_attention_launch(s, (uint16_t*)r->ATT, (const uint16_t*)qp + last * ldq, (const uint16_t*)(kc + loff), (const uint16_t*)(vc + loff), heads, m->head_size, m->kv_mul,
                                   row_pos + last));
            OP(q4_matmul_q4(s, x, (const uint16_t*)r->ATT, &L.o.w, m->o_kc, dim, 1, g, -1, nullptr));
            OP(rows_all_reduce(m, s, (__half*)x, dim, true));
            launch_rows(rmsnorm_rows_kernel<ROW_X>, dim3(1), dim3(kRowThreads), 0, s, r->XB, (__half*)x, (const __half*)nullptr, (const __half*)L.rms_ffn, dim, Embed{});
            OP(q4_ffn_matvec_silu(s, (uint16_t*)r->G, (const uint16_t*)r->XB, &L.gate.w, &L.up.w, dim, m->h_kc));
            OP(q4_matmul_q4(s, x, (const uint16_t*)r->G, &L.down.w, m->h_kc, dim, 1, g, -1, nullptr));
            OP(rows_all_reduce(m, s, (__half*)x, dim, true));
            break;
        }
        if (pos0 >= 0 && !skinny)
            launch_rows(attention_prefill_kernel, dim3(heads, q4_div_up(n, kAtRows)), dim3(128), kAtSmem, s, r->ATT, (const __half*)qp, ldq, kc + loff, vc + loff, heads,
                        m->kv_mul, n, pos0, m->kv_n);
        else if (pos0 >= 0)
            launch_rows(attention_rows_kernel<false>, dim3(heads, n), dim3(kAttWarps * 32), 0, s, r->ATT, (const __half*)qp, ldq, kc, vc, heads, m->kv_mul, row_seq,
                        row_pos, seq_stride, loff, m->kv_n, (const __half*)nullptr, (const __half*)nullptr, (const float2*)nullptr);
        else
            launch_rows(attention_rows_kernel<true>, dim3(heads, n), dim3(kAttWarps * 32), 0, s, r->ATT, (const __half*)qp, ldq, kc, vc, heads, m->kv_mul, row_seq,
                        row_pos, seq_stride, loff, m->kv_n, kp, vp, r->rope);
        // x = o_proj(att) + x / g, summed over the ranks (gpu_kernels.h:237-238, llama2_q4.cu:472-476)
        if (skinny) OP(q4_matmul_q4_rows(s, (uint16_t*)r->X, (const uint16_t*)r->ATT, &L.o.w, n, m->o_kc, dim, (const uint16_t*)r->X, 1.0f / g));
        else OP(gemm(fused_add ? r->Y : r->X, r->ATT, l, 1, !fused_add));
        OP(rows_all_reduce(m, s, r->X, (size_t)n * dim, pos0 >= 0));
        norm((const __half*)L.rms_ffn, fused_add ? r->Y : nullptr);
        if (skinny) {
            // gate and up stay in fp32 until silu(gate) * up, as in ffn_matvec_silu_kernel (gpu_kernels.h:278-281)
            OP(q4_ffn_silu_rows(s, (uint16_t*)r->G, (const uint16_t*)r->XB, &L.gate.w, &L.up.w, n, dim, m->h_kc));
            OP(q4_matmul_q4_rows(s, (uint16_t*)r->X, (const uint16_t*)r->G, &L.down.w, n, m->h_kc, dim, (const uint16_t*)r->X, 1.0f / g));
        } else {
            OP(gemm(r->G, r->XB, l, 2, false));
            OP(gemm(fused_add ? r->Y : r->X, r->G, l, 3, !fused_add));
        }
        OP(rows_all_reduce(m, s, r->X, (size_t)n * dim, pos0 >= 0));
    }
    Q4_CUDA_TRY(cudaGetLastError());
#undef OP
    return Q4_OK;
}

// ------------------------------------------------------------------------------------------------------------
// prefill
// ------------------------------------------------------------------------------------------------------------
// Both position words to `pos`, in stream order.
static int move_pos(q4_model* m, cudaStream_t s, int pos) {
#ifdef Q4_TEST_BUILD
    if (g_fail_set_pos) { g_fail_set_pos = false; return Q4_ERR_CUDA; }
#endif
    Q4_CUDA_TRY(launch_rows(set_pos_kernel, dim3(1), dim3(1), 0, s, m->pos, &m->shared->pos, pos));
    return Q4_OK;
}

static int prefill(q4_model* m, cudaStream_t s, int n, int gen_token, bool logits) {
    if (!m || n < 1) return Q4_ERR_INVALID;
    const q4_config& c = m->cfg;
    const int pos0 = m->host_pos;
    if (pos0 + n > c.seq_len || pos0 + n >= Q4_MAX_SEQ_LEN) return Q4_ERR_LIMIT;
    int e;
    if ((e = rows_prepare(m, n)) != Q4_OK) return e;
    q4_rows* r = m->rows;
    const Embed embed = {(const __half*)m->emb, (const int*)m->shared->tokens, 0, r->row_seq, r->row_pos, c.vocab_size, pos0};
    if ((e = rows_layers(m, s, n, embed, (__half*)m->kc, (__half*)m->vc, 0, logits ? WANT_LAST : WANT_CACHE)) != Q4_OK) return e;
    if ((e = move_pos(m, s, logits ? pos0 + n - 1 : pos0 + n)) != Q4_OK) return e;
    if (logits) {
        // the last row goes on through the batch-1 tail (llama2_q4.cu:528-537, sampler.h:77-84): final norm, classifier,
        // [all-gather], hand-off; the position words were moved to that row, the hand-off steps them past it
        if ((e = q4_rmsnorm(s, m->x, (const uint16_t*)(r->X + (size_t)(n - 1) * c.dim), m->rms_final, c.dim)) != Q4_OK) return e;
        if ((e = q4_matmul_f16(s, m->logits + (size_t)m->rank * m->v_n, m->x, m->wcls, c.dim, m->v_n, 1.0f)) != Q4_OK) return e;
        if (m->g > 1 && (e = q4_all_gather(m->comm, s, m->logits + (size_t)m->rank * m->v_n, m->logits, m->v_n)) != Q4_OK) return e;
        if ((e = q4_argmax(s, m->logits, c.vocab_size, (int*)m->shared->tokens, &m->shared->pos, m->pos, gen_token != 0)) != Q4_OK) return e;
    }
    // sample() draws one coin per position, used or not (sampler.h:79): keep the generator where n token steps leave it
    for (int i = 0; i < n; i++) (void)q4_random_f32(&m->rng_state);
    m->host_pos = pos0 + n;
    return Q4_OK;
}

extern "C" int q4_model_prefill(q4_model* m, void* stream, int n_tokens, int gen_token) { return prefill(m, (cudaStream_t)stream, n_tokens, gen_token, true); }
// The prompt positions into the cache and nothing else: what follows takes its own logits (q4_generate).
int q4_prefill_cache(q4_model* m, cudaStream_t s, int n_tokens) { return prefill(m, s, n_tokens, 0, false); }

// ------------------------------------------------------------------------------------------------------------
// batched decode: several sequences, one position each per step
// ------------------------------------------------------------------------------------------------------------
struct q4_batch {
    q4_model* m;
    int n_seq, n_prompt, max_len;
    __half *kc = nullptr, *vc = nullptr, *logits = nullptr, *xf = nullptr, *part = nullptr;
    int *tokens = nullptr, *pos = nullptr, *seq = nullptr;   // seq: 0, 1, 2, ...
    long long seq_stride;
    int steps = 0;
    // A step is the same work every time (positions and ids live in device memory), so it is captured once as a CUDA
    // graph and replayed: ~260 launches per step on a 32-layer model would otherwise be issued one by one.
    cudaGraphExec_t step_graph = nullptr;
    bool use_graph = true;
};

extern "C" int q4_batch_free(q4_batch* b) {
    if (!b) return Q4_OK;
    if (b->step_graph) cudaGraphExecDestroy(b->step_graph);
    cudaFree(b->kc); cudaFree(b->vc); cudaFree(b->logits); cudaFree(b->xf); cudaFree(b->part); cudaFree(b->tokens); cudaFree(b->pos); cudaFree(b->seq);
    delete b;
    return Q4_OK;
}

extern "C" int q4_batch_create(q4_batch** out, q4_model* m, int n_seq) {
    if (!out || !m || n_seq < 1 || n_seq > 16) return Q4_ERR_INVALID;
    if (int e = rows_prepare(m, n_seq)) return e;
    const q4_config& c = m->cfg;
    constexpr int kMaxSmem = 200 * 1024;   // the plain classifier keeps the rows in shared memory (one limit for all batches: it belongs to the function)
    if (2 * (size_t)n_seq * c.dim > kMaxSmem && !(c.dim % 32 == 0 && m->v_n % 16 == 0)) return Q4_ERR_UNSUPPORTED_SIZE;
    Q4_CUDA_TRY(cudaFuncSetAttribute(matvec_f16_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    q4_batch* b = new q4_batch();
    b->m = m;
    b->n_seq = n_seq;
    b->n_prompt = 0;
    b->max_len = c.seq_len;
    b->seq_stride = (long long)c.n_layers * c.seq_len * m->kv_n;
    const size_t kv_bytes = 2 * (size_t)n_seq * b->seq_stride;
    cudaError_t e = cudaMalloc((void**)&b->kc, kv_bytes);
    if (e == cudaSuccess) e = cudaMalloc((void**)&b->vc, kv_bytes);
    if (e == cudaSuccess) e = cudaMalloc((void**)&b->logits, 2 * (size_t)n_seq * c.vocab_size);
    if (e == cudaSuccess) e = cudaMalloc((void**)&b->xf, 2 * (size_t)n_seq * c.dim);
    if (e == cudaSuccess) e = cudaMalloc((void**)&b->part, 2 * (size_t)n_seq * m->v_n);
    if (e == cudaSuccess) e = cudaMalloc((void**)&b->tokens, sizeof(int) * (size_t)n_seq * (c.seq_len + 1));
    if (e == cudaSuccess) e = cudaMalloc((void**)&b->pos, sizeof(int) * n_seq);
    if (e == cudaSuccess) e = cudaMalloc((void**)&b->seq, sizeof(int) * n_seq);
    int order[16];
    for (int i = 0; i < n_seq; i++) order[i] = i;
    if (e == cudaSuccess) e = cudaMemcpy(b->seq, order, sizeof(int) * n_seq, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(b->kc, 0, kv_bytes);
    if (e == cudaSuccess) e = cudaMemset(b->vc, 0, kv_bytes);
    if (e != cudaSuccess) { q4_note_cuda_error(e, __FILE__, __LINE__); q4_batch_free(b); return Q4_ERR_CUDA; }
    *out = b;
    return Q4_OK;
}

// prompts: [n_seq][n_prompt] token ids; all sequences start at position 0
extern "C" int q4_batch_reset(q4_batch* b, const int* prompts, int n_prompt) {
    if (!b || !prompts || n_prompt < 1 || n_prompt > b->max_len) return Q4_ERR_INVALID;
    for (int i = 0; i < b->n_seq * n_prompt; i++)
        if (prompts[i] < 0 || prompts[i] >= b->m->cfg.vocab_size) return Q4_ERR_INVALID;
    Q4_CUDA_TRY(cudaDeviceSynchronize());
    Q4_CUDA_TRY(cudaMemset(b->tokens, 0, sizeof(int) * (size_t)b->n_seq * (b->max_len + 1)));
    Q4_CUDA_TRY(cudaMemcpy2D(b->tokens, sizeof(int) * (b->max_len + 1), prompts, sizeof(int) * n_prompt, sizeof(int) * n_prompt, b->n_seq, cudaMemcpyHostToDevice));
    Q4_CUDA_TRY(cudaMemset(b->pos, 0, sizeof(int) * b->n_seq));
    // The copies and fills run on the default stream, which a caller's non-blocking stream does not wait for: a step queued right away
    // read the positions of the run before.
    Q4_CUDA_TRY(cudaDeviceSynchronize());
    if (b->step_graph && n_prompt != b->n_prompt) {   // the prompt length is an argument of the captured hand-off kernel
        cudaGraphExecDestroy(b->step_graph);
        b->step_graph = nullptr;
    }
    b->n_prompt = n_prompt;
    b->steps = 0;
    return Q4_OK;
}

static int batch_step(q4_batch* b, cudaStream_t s);

// One position of every sequence: embedding .. logits .. greedy hand-off per sequence. Asynchronous on `stream`.
extern "C" int q4_batch_forward(q4_batch* b, void* stream) {
    if (!b || b->n_prompt < 1) return Q4_ERR_INVALID;
    if (b->steps >= b->max_len) return Q4_ERR_LIMIT;
    cudaStream_t s = (cudaStream_t)stream;
    if (!b->use_graph) {
        if (int e = batch_step(b, s)) return e;
    } else {
        if (!b->step_graph) {
            cudaGraph_t graph = nullptr;
            Q4_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            const int e = batch_step(b, s);
            const cudaError_t ce = cudaStreamEndCapture(s, &graph);
            if (e != Q4_OK) { if (graph) cudaGraphDestroy(graph); return e; }
            Q4_CUDA_TRY(ce);
            Q4_CUDA_TRY(cudaGraphInstantiate(&b->step_graph, graph, 0));
            Q4_CUDA_TRY(cudaGraphDestroy(graph));
        }
        Q4_CUDA_TRY(cudaGraphLaunch(b->step_graph, s));
    }
    b->steps++;
    return Q4_OK;
}

static int batch_step(q4_batch* b, cudaStream_t s) {
    q4_model* m = b->m;
    q4_rows* r = m->rows;
    const q4_config& c = m->cfg;
    const int n = b->n_seq;
    // row i is sequence i, and the hand-off moves the positions only when every kernel of the step has read them: no copies of either
    const Embed embed = {(const __half*)m->emb, b->tokens, b->max_len + 1, b->seq, b->pos, c.vocab_size, -1};
    if (int e = rows_layers(m, s, n, embed, b->kc, b->vc, b->seq_stride, WANT_ALL)) return e;
    launch_rows(rmsnorm_rows_kernel<ROW_X>, dim3(n), dim3(kRowThreads), 0, s, b->xf, r->X, (const __half*)nullptr, (const __half*)m->rms_final, c.dim, Embed{});
    const size_t smem = 2 * (size_t)n * c.dim;
    __half* cls_out = m->g == 1 ? b->logits : b->part;   // TP: every rank computes its vocabulary slice of every row; the slices are gathered row by row
    const int cls_stride = m->g == 1 ? c.vocab_size : m->v_n;
    if (c.dim % 32 == 0 && m->v_n % 16 == 0) {
        if (n <= 8) launch_rows(classifier_rows_kernel<1>, dim3(m->v_n / 16), dim3(kClsWarps * 32), 0, s, cls_out, b->xf, (const __half*)m->wcls, c.dim, m->v_n, n, cls_stride);
        else launch_rows(classifier_rows_kernel<2>, dim3(m->v_n / 16), dim3(kClsWarps * 32), 0, s, cls_out, b->xf, (const __half*)m->wcls, c.dim, m->v_n, n, cls_stride);
    } else {
        launch_rows(matvec_f16_rows_kernel, dim3(148 * 2), dim3(256), smem, s, cls_out, b->xf, (const __half*)m->wcls, c.dim, m->v_n, n, cls_stride);
    }
    if (m->g > 1) {
        for (int i = 0; i < n; i++)
            if (int e = q4_all_gather(m->comm, s, (const uint16_t*)(b->part + (size_t)i * m->v_n), (uint16_t*)(b->logits + (size_t)i * c.vocab_size), m->v_n)) return e;
    }
    launch_rows(argmax_rows_kernel, dim3(n), dim3(1024), 0, s, b->logits, c.vocab_size, b->tokens, b->max_len + 1, b->pos, b->n_prompt);
    Q4_CUDA_TRY(cudaGetLastError());
    return Q4_OK;
}

extern "C" const uint16_t* q4_batch_logits(const q4_batch* b) { return b ? (const uint16_t*)b->logits : nullptr; }

// tokens[s][0 .. len) of every sequence (synchronises the device)
extern "C" int q4_batch_read_tokens(const q4_batch* b, int* out, int len) {
    if (!b || !out || len < 1 || len > b->max_len + 1) return Q4_ERR_INVALID;
    Q4_CUDA_TRY(cudaDeviceSynchronize());
    Q4_CUDA_TRY(cudaMemcpy2D(out, sizeof(int) * len, b->tokens, sizeof(int) * (b->max_len + 1), sizeof(int) * len, b->n_seq, cudaMemcpyDeviceToHost));
    return Q4_OK;
}
