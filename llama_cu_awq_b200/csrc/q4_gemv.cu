// AWQ W4 g128 dequantize-and-multiply GEMV kernel (batch 1) and its C-ABI launchers.
//
// Replaces mat_vec_kernel_int4 / qkv_matvec_kernel / ffn_matvec_silu_kernel of the reference
// (gpu_kernels.h:179-283) and their wrappers (llama2_q4.cu:367-404).
//
// Work split: a tile is 8 consecutive output columns of one matrix (gate/up: 4 columns of each). Two persistent CTAs per SM, each with
// every grid-th group of T tiles. A stage is a group's packed words over Pc pairs of 128-input groups: row copies of Pc * 128 bytes
// (cp.async.bulk, local memory, no multicast; adjacent in the file layout) by a producer warp into a ring of 4 stages. Pc * T <= 16
// (tile, pair) units make a stage; math warp w of 8 has units w and w + 8, so that it stages the activations of two pairs, straight
// from x, for all of the CTA's groups. make_split takes the Pc and T with the fewest stages: 16 pairs of one tile for long rows, more
// tiles for short ones. The product runs on the integer tensor pipe (q4_w4dot.cuh). The units' sums go to shared memory and are
// added in pair order.
//
// What bounds it: the launch's ramp (grid start, first copies, last sums) and, in between, a warp's serial chain per stage (wait, loads,
// products, sums: about 800 clocks), of which four per SM sub-partition run side by side. Under programmatic dependent launch the next
// product's ring fills as soon as a CTA of this one has left (weights never depend on activations).
// Back to back on weights from HBM, before (half2 FMA, one tile per warp) and now, us: 4096 x 4096 5.1, 4.6; 11008 -> 4096 9.75, 9.8; q|k|v
// 9.5, 8.5; 4096 -> 2 x 11008 13.6, 10.8 (4.3 TB/s); 28672 -> 8192 33.2, 30.4; error against 64 bits 3.8e-4, 2.1e-4 (an fp16 result's own
// rounding). A dedicated CTA per SM with 16 math warps: 4.1, 10.9, 7.8, 12.3, 46.
#include <algorithm>

#include "q4_bulk.cuh"
#include "q4_w4dot.cuh"

namespace {

constexpr int kRows = 8;             // output columns per tile
constexpr int kMathWarps = 8;
constexpr int kUnits = 2 * kMathWarps;
constexpr int kThreads = 32 * (kMathWarps + 1);
constexpr int kMaxT = 4;             // tiles per stage at most: one lane of the producer per row
constexpr int kPairBytes = 128;      // of one row
constexpr int kRowPad = 16;          // rows four banks apart (mod 32): a load of four words of each of eight rows does not collide
constexpr int kStageBytes = kUnits * kRows * kPairBytes + kMaxT * kRows * kRowPad;
constexpr int kStages = 4;
constexpr int kBlockTiles = 16;      // tiles per pass (their partial sums, scales and zero points are in shared memory)
constexpr int kTileStride = kUnits * kRows + 8;
constexpr int kMetaBytes = 2 * kBlockTiles * 64;   // per warp: 8 columns x 2 groups of its two units in every group of tiles, fp16 scale | zero point << 16
constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + kMathWarps * (2 * kPairScratch + kMetaBytes) + (size_t)kBlockTiles * kTileStride * 4;

struct GemvMat {
    const uint32_t* w;
    const uint32_t* z;
    const __half* s;
    __half* out;
    int n;       // output columns of this matrix
    int tile0;   // first tile index of this matrix in the launch
    int kv;      // 1: out += loff + *pos * n
};

struct GemvParams {
    const __half* x;
    int K, PW, PZ, G;
    int nmat;
    GemvMat m[3];
    int total_tiles;
    int accum;
    float gpu_count;
    long long loff;
    const int* pos;
    int Pc, T, nchunks;   // pairs and tiles per stage, chunks of Pc pairs
};

__device__ __forceinline__ float silu_mul(float g, float u) {
    float val = g;
    val *= 1.0f / (1.0f + expf(-val));
    val *= u;
    return val;
}

// Matrix of a tile's row r and the row's number in it (SILU: rows 0, 2, 4, 6 are gate columns, 1, 3, 5, 7 the same up columns)
template <bool SILU>
__device__ __forceinline__ const GemvMat& row_of(const GemvParams& p, int tile, int r, int& row) {
    if (SILU) {
        row = tile * 4 + (r >> 1);
        return p.m[r & 1];
    }
    const int mi = p.nmat > 2 && tile >= p.m[2].tile0 ? 2 : p.nmat > 1 && tile >= p.m[1].tile0 ? 1 : 0;
    row = (tile - p.m[mi].tile0) * kRows + r;
    return p.m[mi];
}

// MULTI: more than one chunk or pass, whose activations and scales are requested while the one before is worked on (the registers that
// takes cost a single pass 10 %).
template <bool SILU, bool MULTI>
__global__ void __launch_bounds__(kThreads, 2) q4_gemv_kernel(const __grid_constant__ GemvParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[kStages], empty[kStages];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cta = blockIdx.x, grid = gridDim.x;
    const int Pc = p.Pc, T = p.T, nchunks = p.nchunks, row_bytes = Pc * kPairBytes + kRowPad;
    const int groups = (p.total_tiles + T - 1) / T, my_groups = (groups - cta + grid - 1) / grid, per_pass = kBlockTiles / T;
    if (tid < kStages) {
        mbar_init(&full[tid], 1);
        mbar_init(&empty[tid], kMathWarps);
    }
    mbar_init_fence();
    __syncthreads();

    if (warp == kMathWarps) {
        // ---- producer: passes, chunks of Pc pairs, groups of tiles; lane r copies row r ----
        int stage = 0, issued = 0;
        uint32_t parity = 1;     // the first round finds every stage empty
        for (int b0 = 0; b0 < my_groups; b0 += per_pass)
            for (int c = 0; c < nchunks; c++)
                for (int lg = b0; lg < min(b0 + per_pass, my_groups); lg++) {
                    const int word0 = c * Pc * 32, tile0 = (cta + lg * grid) * T;
                    const uint32_t bytes = 4u * (uint32_t)min(Pc * 32, p.PW - word0);
                    const int rows = min(T, p.total_tiles - tile0) * kRows;
                    if (!mbar_wait_warp(&empty[stage], parity)) { b0 = my_groups; c = nchunks; break; }
                    issued++;
                    if (lane == 0) mbar_expect_tx(&full[stage], rows * bytes);
                    __syncwarp();
                    if (lane < rows) {
                        int row;
                        const GemvMat& m = row_of<SILU>(p, tile0 + (lane >> 3), lane & 7, row);
                        bulk_g2s(smem + stage * kStageBytes + lane * row_bytes, m.w + (size_t)row * p.PW + word0, bytes, &full[stage]);
                    }
                    __syncwarp();
                    if (++stage == kStages) { stage = 0; parity ^= 1u; }
                }
        // the CTA's shared memory stays until every copy has landed (bounded; the math warps have waited for all of them unless a wait ran out)
        for (int i = max(0, issued - kStages); i < issued; i++) mbar_wait_warp(&full[i % kStages], (i / kStages) & 1);
        return;
    }

    uint8_t* const scr = smem + kStages * kStageBytes + warp * 2 * kPairScratch;
    uint32_t* const meta = reinterpret_cast<uint32_t*>(smem + kStages * kStageBytes + kMathWarps * 2 * kPairScratch + warp * kMetaBytes);
    float* const part = reinterpret_cast<float*>(smem + kStages * kStageBytes + kMathWarps * (2 * kPairScratch + kMetaBytes));
    const int r = lane >> 2, t = lane & 3;
    int ts[2], pi[2];            // this warp's units: tile in the group, pair in the chunk
#pragma unroll
    for (int j = 0; j < 2; j++) {
        ts[j] = (warp + j * kMathWarps) / Pc;
        pi[j] = warp + j * kMathWarps - ts[j] * Pc;
    }
    int stage = 0;
    uint32_t parity = 0;
    bool ok = true;
    // This warp's scales and zero points for the groups of a pass in a chunk: entry [group][unit][2 * column + group of the pair]. The first
    // kAhead groups' are requested a chunk ahead.
    constexpr int kAhead = MULTI ? 4 : 0;
    uint32_t zn[kAhead + 1];
    __half sn[kAhead + 1];
    const int en = lane & 15, tj = (lane >> 4) ? ts[1] : ts[0], pj = (lane >> 4) ? pi[1] : pi[0];
    auto load_one = [&](int lg, int c, uint32_t& z, __half& sc) {
        const int tile = (cta + lg * grid) * T + tj, grp = 2 * (c * Pc + pj) + (en & 1);
        z = 0;
        sc = __float2half(0.f);
        if (tj < T && tile < p.total_tiles && grp < p.G) {
            int row;
            const GemvMat& m = row_of<SILU>(p, tile, en >> 1, row);
            z = __ldg(m.z + (size_t)row * p.PZ + (grp >> 3)) >> (4 * (grp & 7));
            sc = __ldg(m.s + (size_t)row * p.G + grp);
        }
    };
    auto ahead = [&](int b0, int bn, int c) {
#pragma unroll
        for (int i = 0; i < kAhead; i++)
            if (i < bn) load_one(b0 + i, c, zn[i], sn[i]);
    };
    auto file_meta = [&](int b0, int bn, int c) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kAhead; i++)
            if (i < bn) meta[i * 32 + lane] = (uint32_t)__half_as_ushort(sn[i]) | ((zn[i] & 0xFu) << 16);
#pragma unroll 4
        for (int lg = kAhead; lg < bn; lg++) {
            uint32_t z;
            __half sc;
            load_one(b0 + lg, c, z, sc);
            meta[lg * 32 + lane] = (uint32_t)__half_as_ushort(sc) | ((z & 0xFu) << 16);
        }
        __syncwarp();
    };
    ahead(0, min(per_pass, my_groups), 0);
    file_meta(0, min(per_pass, my_groups), 0);   // as the weights, before the predecessor's results are waited for
    if (nchunks > 1)                             // the later chunks' on their way into L2
        for (int i = tid; i < my_groups * T * kRows; i += 32 * kMathWarps) {
            int row;
            const int tile = (cta + i / (T * kRows) * grid) * T + (i / kRows) % T;
            if (tile < p.total_tiles) {
                const GemvMat& m = row_of<SILU>(p, tile, i & 7, row);
                for (int g = 2 * Pc; g < p.G; g += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(m.s + (size_t)row * p.G + g));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(m.z + (size_t)row * p.PZ));
            }
        }
    griddep_wait();
    griddep_launch_dependents();
    uint4 hv[2];                 // a chunk's activations, requested a chunk ahead (zero beyond K: padded weight words contribute nothing)
    auto load_x = [&](int c) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int k0 = (c * Pc + pi[j]) * 256 + lane * 8;
            hv[j] = make_uint4(0, 0, 0, 0);
            if (ts[j] < T && k0 < p.K) hv[j] = *reinterpret_cast<const uint4*>(p.x + k0);
        }
    };
    load_x(0);
    for (int b0 = 0; b0 < my_groups; b0 += per_pass) {
        const int bn = min(per_pass, my_groups - b0);
        for (int c = 0; c < nchunks; c++) {
            PairX px[2];
            bool active[2];
#pragma unroll
            for (int j = 0; j < 2; j++) active[j] = ts[j] < T && 2 * (c * Pc + pi[j]) < p.G;
            if (b0 + c > 0) file_meta(b0, bn, c);
#pragma unroll
            for (int j = 0; j < 2; j++) quant_pair(hv[j], scr + j * kPairScratch, lane, px[j]);
            const bool last = c + 1 == nchunks;
            if (MULTI && (!last || b0 + per_pass < my_groups)) {
                load_x(last ? 0 : c + 1);
                ahead(last ? b0 + per_pass : b0, last ? min(per_pass, my_groups - b0 - per_pass) : bn, last ? 0 : c + 1);
            }
            for (int lg = 0; lg < bn; lg++) {
                if (ok) ok = mbar_wait_warp(&full[stage], parity);
                // words t, 4 + t, 8 + t, 12 + t of column r, groups A and B in turn: single loads, straight into operand order. (Units that
                // are not there multiply whatever lies in the stage; their sums are not kept.)
                uint32_t me[2];
                int c4[2][4];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const uint32_t* src = reinterpret_cast<const uint32_t*>(smem + stage * kStageBytes + ((active[j] ? ts[j] * kRows : 0) + r) * row_bytes + (active[j] ? pi[j] : 0) * kPairBytes) + t;
                    me[j] = meta[lg * 32 + j * 16 + (lane >> 1)];
                    pair_mma(c4[j], make_uint4(src[0], src[16], src[4], src[20]), make_uint4(src[8], src[24], src[12], src[28]), px[j]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[stage]);
                if (++stage == kStages) { stage = 0; parity ^= 1u; }
                float y = quad_sum2(pair_share(c4[0], me[0], px[0], lane), pair_share(c4[1], me[1], px[1], lane), lane);
                if (!ok) y = CUDART_NAN_F;   // a copy that never came must not pass for a result
                const bool odd = t & 1;
                if (t < 2 && (odd ? active[1] : active[0])) {
                    float* const d = part + (lg * T + (odd ? ts[1] : ts[0])) * kTileStride + (odd ? pi[1] : pi[0]) * kRows + r;
                    *d = c == 0 ? y : *d + y;
                }
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kMathWarps) : "memory");
        for (int e0 = warp * 32; e0 < bn * T * kRows; e0 += 32 * kMathWarps) {   // thread 8 * tile + column
            const int e = e0 + lane, lt = e >> 3, tile = (cta + (b0 + lt / T) * grid) * T + lt % T;
            const bool on = e < bn * T * kRows && tile < p.total_tiles;
            float sum = 0.f;
            if (on)
                for (int i = 0; i < Pc; i += 4) {
                    const float* q = part + lt * kTileStride + i * kRows + (e & 7);
                    float v[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) v[u] = i + u < Pc ? q[u * kRows] : 0.f;
                    sum += ((v[0] + v[1]) + v[2]) + v[3];
                }
            int row;
            const GemvMat& m = row_of<SILU>(p, on ? tile : 0, e & 7, row);
            if (SILU) {
                const float up = __shfl_xor_sync(0xffffffffu, sum, 1);
                if (on && !(e & 1)) p.m[0].out[row] = __float2half(silu_mul(sum, up));
            } else if (on) {
                __half* out = m.out;
                if (m.kv) out += p.loff + (long long)(*p.pos) * m.n;
                if (p.accum) sum += __half2float(out[row]) / p.gpu_count;
                out[row] = __float2half(sum);
            }
        }
        if (b0 + per_pass < my_groups) asm volatile("bar.sync 1, %0;" ::"n"(32 * kMathWarps) : "memory");
    }
}

int check_sizes(int K, int N) { return ((K & 7) || (N & 7) || K <= 0 || N <= 0) ? Q4_ERR_UNSUPPORTED_SIZE : Q4_OK; }

void fill_dims(GemvParams& p, int K) {
    p.K = K;
    p.PW = q4_pw(K);
    p.PZ = q4_pz(K);
    p.G = q4_groups(K);
}

constexpr int kCtas = 2 * 148;   // B200: two persistent CTAs per SM

// Pairs and tiles per stage: the split that takes the CTA with the most work the least time, a chunk's start (activations, scales) counted
// as 1.2 stages (13824 -> 5120: 16 pairs of one tile 4 chunks x 3 stages; 5 pairs of 3 tiles 11 x 1, 21 us).
void make_split(GemvParams& p) {
    const int P = q4_div_up(p.G, 2);
    int best = 0;
    for (int Pc = std::min(P, kUnits); Pc >= 1; Pc--)
        for (int T = 1; T <= std::min(kUnits / Pc, kMaxT); T++) {
            const int cost = q4_div_up(P, Pc) * (10 * q4_div_up(q4_div_up(p.total_tiles, T), kCtas) + 12);
            if (best && cost >= best) continue;
            best = cost;
            p.Pc = Pc;
            p.T = T;
        }
    p.nchunks = q4_div_up(P, p.Pc);
}

template <bool SILU>
int launch(GemvParams& p, cudaStream_t s) {
    static_assert(2 * (kSmemBytes + 1024 + 256) <= 228 * 1024, "two CTAs per SM");
    make_split(p);
    const int groups = q4_div_up(p.total_tiles, p.T);
    // (an opt-in of the function on the device, always to the same value)
    auto* kernel = p.nchunks > 1 || groups > kCtas * (kBlockTiles / p.T) ? q4_gemv_kernel<SILU, true> : q4_gemv_kernel<SILU, false>;
    Q4_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    Q4Launch L(dim3(std::min(groups, kCtas)), dim3(kThreads), kSmemBytes, s);
    Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, kernel, p));
    return Q4_OK;
}

GemvMat mat(const q4_qweight* w, uint16_t* out, int n, int tile0, int kv) {
    GemvMat m;
    m.w = w->weight;
    m.z = w->zeros;
    m.s = reinterpret_cast<const __half*>(w->scales);
    m.out = reinterpret_cast<__half*>(out);
    m.n = n;
    m.tile0 = tile0;
    m.kv = kv;
    return m;
}

}  // namespace

extern "C" int q4_matmul_q4(void* stream, uint16_t* xout, const uint16_t* x, const q4_qweight* w, int inpSize,
                            int opSize, int accum, int gpu_count, int loff, const int* pPos) {
    if (int e = check_sizes(inpSize, opSize)) return e;
    if (!xout || !x || !w || gpu_count < 1 || (loff != -1 && !pPos)) return Q4_ERR_INVALID;
    GemvParams p = {};
    fill_dims(p, inpSize);
    p.x = reinterpret_cast<const __half*>(x);
    p.nmat = 1;
    p.m[0] = mat(w, xout, opSize, 0, loff != -1);
    p.total_tiles = opSize / kRows;
    p.accum = accum != 0;
    p.gpu_count = (float)gpu_count;
    p.loff = loff == -1 ? 0 : loff;
    p.pos = pPos;
    return launch<false>(p, (cudaStream_t)stream);
}

extern "C" int q4_qkv_matvec(void* stream, uint16_t* q, uint16_t* key_cache, uint16_t* value_cache, const uint16_t* x,
                             const q4_qweight* qw, const q4_qweight* kw, const q4_qweight* vw, int inpSize, int opSize,
                             int kvSize, int loff, const int* pPos) {
    if (int e = check_sizes(inpSize, opSize)) return e;
    if (int e = check_sizes(inpSize, kvSize)) return e;
    if (!q || !key_cache || !value_cache || !x || !qw || !kw || !vw || !pPos || loff < 0) return Q4_ERR_INVALID;
    GemvParams p = {};
    fill_dims(p, inpSize);
    p.x = reinterpret_cast<const __half*>(x);
    p.nmat = 3;
    const int tq = opSize / kRows, tkv = kvSize / kRows;
    p.m[0] = mat(qw, q, opSize, 0, 0);
    p.m[1] = mat(kw, key_cache, kvSize, tq, 1);
    p.m[2] = mat(vw, value_cache, kvSize, tq + tkv, 1);
    p.total_tiles = tq + 2 * tkv;
    p.accum = 0;
    p.gpu_count = 1.f;
    p.loff = loff;
    p.pos = pPos;
    return launch<false>(p, (cudaStream_t)stream);
}

extern "C" int q4_ffn_matvec_silu(void* stream, uint16_t* xout, const uint16_t* x, const q4_qweight* gate_w,
                                  const q4_qweight* up_w, int inpSize, int opSize) {
    if (int e = check_sizes(inpSize, opSize)) return e;
    if (!xout || !x || !gate_w || !up_w) return Q4_ERR_INVALID;
    GemvParams p = {};
    fill_dims(p, inpSize);
    p.x = reinterpret_cast<const __half*>(x);
    p.nmat = 2;
    p.m[0] = mat(gate_w, xout, opSize, 0, 0);
    p.m[1] = mat(up_w, xout, opSize, 0, 0);
    p.total_tiles = opSize / 4;
    p.gpu_count = 1.f;
    return launch<true>(p, (cudaStream_t)stream);
}
