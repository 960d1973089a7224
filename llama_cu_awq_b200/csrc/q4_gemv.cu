// AWQ W4 g128 dequantize-and-multiply GEMV kernel (batch 1) and its C-ABI launchers.
//
// Replaces mat_vec_kernel_int4 / qkv_matvec_kernel / ffn_matvec_silu_kernel of the reference
// (gpu_kernels.h:179-283) and their wrappers (llama2_q4.cu:367-404).
//
// A tile is 8 consecutive output columns of one matrix (gate/up: 4 columns of each); a pair is two groups of 128 inputs; an item is a
// tile's packed words over a pair, 1 KB. The product runs on the integer tensor pipe with x as it is (PairExact, q4_w4dot.cuh): one warp,
// one item. Two forms of the kernel (launch() has the line between them and both sides' figures):
//
// Direct: one CTA of 16 warps per SM with consecutive tiles. Words go from memory into registers in the order in which the product takes
// them, three items ahead; no shared memory, barrier or wait on the way. A warp stages the activations of a pair once for all the CTA's
// tiles. What bounds it: the launch's ramp, and for long rows the staging (a pair per warp and 16 pairs); from HBM it reads 3.1 TB/s.
//
// Ring: two CTAs per SM, each with every grid-th group of T tiles. A stage is a group's packed words over Pc pairs: row copies of Pc * 128
// bytes (cp.async.bulk, local memory, no multicast; adjacent in the file layout) by a producer warp into a ring of 4 stages. Pc * T <= 16
// (tile, pair) units make a stage; math warp w of 8 has units w and w + 8, so that it stages the activations of two pairs for all of
// the CTA's groups. make_split takes the Pc and T with the fewest stages. What bounds it: the ramp, and a warp's serial chain per stage
// (wait, loads, products, sums).
//
// Under programmatic dependent launch the next product's packed words are requested while this one drains (weights never depend on
// activations). Back to back on weights from HBM, with half2 FMA, with x as 16-bit fixed point in the ring form alone, and now, us:
// 4096 x 4096 5.1, 4.4, 4.2; q|k|v 9.9, 9.2, 9.2; 4096 -> 2 x 11008 13.9, 11.0, 11.4; 11008 -> 4096 9.9, 9.6, 10.4; 28672 -> 8192 34.1, 31.3,
// 33.5; 11008 -> 512 5.3, 5.6, 4.0; 5120 -> 1280 4.4, 4.8, 3.7; 13520 -> 544 6.8, 7.0, 5.4; 512 x 512 1.8, 2.3, 1.7. Error against 64 bits 3.8e-4,
// 2.1e-4, 2.1e-4 (an fp16 result's own rounding).
#include <algorithm>

#include "q4_bulk.cuh"
#include "q4_w4dot.cuh"

namespace {

constexpr int kRows = 8;             // output columns per tile
constexpr int kWarps = 16;
constexpr int kThreads = 32 * kWarps;
constexpr int kAhead = 3;            // items a warp has requested ahead of the one it multiplies
constexpr int kBlockTiles = 32;      // tiles per pass (their partial sums are in shared memory)
constexpr int kTileStride = kWarps * kRows + 8;   // floats (padded: the summing threads hit distinct banks)
constexpr int kSms = 148;            // B200

namespace ring {
constexpr int kMathWarps = 8;
constexpr int kUnits = 2 * kMathWarps;
constexpr int kThreads = 32 * (kMathWarps + 1);
constexpr int kCtas = 2 * kSms;      // two persistent CTAs per SM
constexpr int kMaxT = 4;             // tiles per stage at most: one lane of the producer per row
constexpr int kPairBytes = 128;      // of one row
constexpr int kRowPad = 64;          // two rows' 64-byte pieces of a load lie in different banks
constexpr int kStageBytes = kUnits * kRows * kPairBytes + kMaxT * kRows * kRowPad;
constexpr int kStages = 4;
constexpr int kBlockTiles = 13;      // tiles per pass (their partial sums, scales and zero points are in shared memory)
constexpr int kTileStride = kUnits * kRows + 8;
constexpr int kMetaBytes = 2 * kBlockTiles * 64;   // per warp: 8 columns x 2 groups of its two units in every group of tiles, fp16 scale | zero point << 16
constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + kMathWarps * (2 * kExactScratch + kMetaBytes) + (size_t)kBlockTiles * kTileStride * 4;
}  // namespace ring

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
    int K, PW, PZ, G, P;
    int nmat;
    GemvMat m[3];
    int total_tiles;
    int accum;
    float gpu_count;
    long long loff;
    const int* pos;
    int nt_div, nt_mod;   // direct form: CTA c has nt_div + (c < nt_mod) consecutive tiles
    int Pc, T, nchunks;   // ring form: pairs and tiles per stage, chunks of Pc pairs
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

// One item (a tile's 8 columns over a pair of groups) in lane 4c + t: words 4t..4t + 3 of column c in groups A and B, and the column's zero
// word and scale in group (t >> 1).
struct Item {
    uint4 a, b;
    uint32_t z;
    __half s;
};
// The order of a warp's items in a pass: pairs w, w + 16, ... below `full` (a multiple of 16), each over all tiles, so that the warps read
// 16 neighbouring pieces of a row at a time; then the warp's share of the tiles of the pairs that are left, from (rest_pair, rest_tile) on.
struct Order {
    int tiles, full, rest_pair, rest_tile;
    __device__ __forceinline__ void next_pair(int& pair, int& tile) const {
        tile = 0;
        if (pair >= full) pair++;
        else if (pair + kWarps < full) pair += kWarps;
        else {
            pair = rest_pair;
            tile = rest_tile;
        }
    }
};
// Walks a warp's items; the addresses of the item it is at. A step to the next tile of the same matrix is three additions.
template <bool SILU>
struct Cursor {
    const uint32_t* w;
    const uint32_t* z;
    const __half* s;
    int tile, pair, end;     // end: the tiles from here to it have their rows in the same matrix
    __device__ __forceinline__ void seek(const GemvParams& p, int tile0, const Order& o, int lane) {
        int row;
        const GemvMat& m = row_of<SILU>(p, tile0 + tile, lane >> 2, row);
        end = o.tiles;
        if (!SILU && p.nmat > 1) end = min(end, m.tile0 + m.n / kRows - tile0);
        w = m.w + (size_t)row * p.PW + pair * 32 + (lane & 3) * 4;
        const int g = 2 * pair + ((lane >> 1) & 1);
        z = m.z + (size_t)row * p.PZ + (g >> 3);
        s = m.s + (size_t)row * p.G + g;
    }
    __device__ __forceinline__ void next(const GemvParams& p, int tile0, const Order& o, int lane) {
        constexpr int kStep = SILU ? kRows / 2 : kRows;
        if (++tile < end) {
            w += kStep * p.PW;
            z += kStep * p.PZ;
            s += kStep * p.G;
            return;
        }
        if (tile == o.tiles) o.next_pair(pair, tile);
        seek(p, tile0, o, lane);
    }
    // (words past a row's end and a group that is not there keep what the registers hold: it meets digits that are zero)
    __device__ __forceinline__ void words(const GemvParams& p, Item& it, int lane) const {
        const int at = pair * 32 + (lane & 3) * 4;
        if (at < p.PW) it.a = ldg_stream(reinterpret_cast<const uint4*>(w));
        if (at + 16 < p.PW) it.b = ldg_stream(reinterpret_cast<const uint4*>(w + 16));
    }
    __device__ __forceinline__ void meta(const GemvParams& p, Item& it, int lane) const {
        it.s = __float2half(0.f);
        if (2 * pair + ((lane >> 1) & 1) < p.G) {
            it.z = __ldg(z);
            it.s = __ldg(s);
        }
    }
};

// What quant_pair_exact left out of pair `pair`, added in fp32 to the pair's sums (at part, part_step apart) of `tiles` tiles, every
// tile_step-th from `tile`. Seldom: the words come from memory once more, so that the loop that is always there carries nothing for it.
// One warp.
template <bool SILU>
__device__ __noinline__ void add_small(const GemvParams& p, float* part, int part_step, uint32_t small, int tile, int tile_step, int tiles, int pair) {
    const int lane = threadIdx.x & 31, t = lane & 3;
    __syncwarp();
    for (int i = 0; i < tiles && tile < p.total_tiles; i++, tile += tile_step) {
        int row;
        const GemvMat& m = row_of<SILU>(p, tile, lane >> 2, row);
        float y = 0.f;
        for (int g = 2 * pair; g < min(2 * pair + 2, p.G); g++) {
            const uint32_t lim = g & 1 ? small >> 16 : small & 0xFFFFu;
            if (lim == 0) continue;
            const int zero = (int)(__ldg(m.z + (size_t)row * p.PZ + (g >> 3)) >> (4 * (g & 7))) & 0xF;
            float sum = 0.f;
            for (int w = g * 16 + t; w < min(g * 16 + 16, p.PW) && w * 8 < p.K; w += 4)
                sum = small_dot(__ldg(m.w + (size_t)row * p.PW + w), *reinterpret_cast<const uint4*>(p.x + w * 8), lim, zero, sum);
            y = fmaf(__half2float(__ldg(m.s + (size_t)row * p.G + g)), sum, y);
        }
        y = quad_sum(y);
        if (t == 0) part[i * part_step + (lane >> 2)] += y;
    }
}

template <bool SILU>
__global__ void __launch_bounds__(kThreads, 1) q4_gemv_kernel(const __grid_constant__ GemvParams p) {
    __shared__ __align__(16) uint8_t scratch[kWarps][kExactScratch];
    __shared__ float part[kBlockTiles * kTileStride];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, cta = blockIdx.x;
    const int cta_tile0 = cta * p.nt_div + min(cta, p.nt_mod), cta_tiles = p.nt_div + (cta < p.nt_mod);
    uint8_t* const scr = scratch[w];

    for (int b0 = 0; b0 < cta_tiles; b0 += kBlockTiles) {
        const int tiles = min(kBlockTiles, cta_tiles - b0), tile0 = cta_tile0 + b0;
        Order order;
        order.tiles = tiles;
        order.full = p.P / kWarps * kWarps;
        const int rest = (p.P - order.full) * tiles, r0 = w * rest / kWarps, r1 = (w + 1) * rest / kWarps;
        order.rest_pair = order.full + r0 / tiles;
        order.rest_tile = r0 - r0 / tiles * tiles;
        int pair = order.full ? w : order.rest_pair, tile = order.full ? 0 : order.rest_tile;
        int left = order.full / kWarps * tiles + r1 - r0;
        float* const col = part + w * kRows + (lane >> 2);
        if (left < tiles || tile > 0)      // the first pair does not reach every tile
            for (int i = lane; i < tiles * kRows; i += 32) part[(i >> 3) * kTileStride + w * kRows + (i & 7)] = 0.f;
        __syncwarp();
        Item items[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; u++) {
            items[u].a = items[u].b = make_uint4(0, 0, 0, 0);
            items[u].z = 0;
        }
        const Cursor<SILU> start = [&] {
            Cursor<SILU> c;
            c.tile = tile;
            c.pair = pair;
            if (left > 0) c.seek(p, tile0, order, lane);
            return c;
        }();
        Cursor<SILU> cur = start;
#pragma unroll
        for (int u = 0; u < kAhead; u++)
            if (u < left) {
                cur.words(p, items[u], lane);
                if (u + 1 < left) cur.next(p, tile0, order, lane);
            }
        if (b0 == 0) {
            griddep_wait();
            griddep_launch_dependents();
        }
        auto load_x = [&](int pr) {
            const int k = pr * 256 + lane * 8;
            return k < p.K ? *reinterpret_cast<const uint4*>(p.x + k) : make_uint4(0, 0, 0, 0);
        };
        uint4 hv = left > 0 ? load_x(pair) : make_uint4(0, 0, 0, 0);
        cur = start;
#pragma unroll
        for (int u = 0; u < kAhead; u++)
            if (u < left) {
                cur.meta(p, items[u], lane);
                if (u + 1 < left) cur.next(p, tile0, order, lane);
            }
        bool first = true;
        int slot = 0;              // of items: the next one's
        while (left > 0) {
            PairExact px;
            const bool wide = quant_pair_exact(hv, scr, lane, px);
            zero_step(px);
            const int count = min(left, tiles - tile), shift = 4 * ((2 * pair + ((lane >> 1) & 1)) & 7);
            int pair2 = pair, tile2 = tile;
            order.next_pair(pair2, tile2);
            if (left > count) hv = load_x(pair2);
            float* d = col + tile * kTileStride;
            for (int n = count; n > 0;) {
#pragma unroll
                for (int u = 0; u < kAhead; u++) {   // (registers cannot be indexed: a copy of the step for each slot)
                    if (slot != u) continue;
                    slot = u + 1 == kAhead ? 0 : u + 1;
                    Item& it = items[u];
                    int c[4];
                    pair_mma_exact(c, it.a, it.b, px);
                    const uint32_t meta = (uint32_t)__half_as_ushort(it.s) | (((it.z >> shift) & 0xFu) << 16);
                    if (left > kAhead) {
                        cur.words(p, it, lane);
                        cur.meta(p, it, lane);
                        if (left > kAhead + 1) cur.next(p, tile0, order, lane);
                    }
                    left--;
                    const float y = quad_sum(pair_share(c, meta, px, lane));
                    if ((lane & 3) == 0) *d = first ? y : *d + y;
                    d += kTileStride;
                    if (--n == 0) break;
                }
            }
            if (wide)
                add_small<SILU>(p, part + tile * kTileStride + w * kRows, kTileStride, *reinterpret_cast<const uint32_t*>(scr), tile0 + tile, 1, count, pair);
            pair = pair2;
            tile = tile2;
            first = false;
        }
        __syncthreads();
        for (int e0 = w * 32; e0 < tiles * kRows; e0 += kThreads) {   // thread 8 * tile + column: the warps' sums in warp order
            const int e = e0 + lane;
            const bool on = e < tiles * kRows;
            float sum = 0.f;
            if (on) {
                const float* q = part + (e >> 3) * kTileStride + (e & 7);
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = ((q[i * 32] + q[i * 32 + 8]) + q[i * 32 + 16]) + q[i * 32 + 24];
                sum = ((v[0] + v[1]) + v[2]) + v[3];
            }
            int row;
            const GemvMat& m = row_of<SILU>(p, tile0 + (on ? e >> 3 : 0), e & 7, row);
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
        if (b0 + kBlockTiles < cta_tiles) __syncthreads();
    }
}

// Q4_ERR_TIMEOUT once a wait of the ring form has run out (q4_ops_status)
__device__ int g_status;

// MULTI: more than one chunk or pass, whose activations and scales are requested while the one before is worked on (the registers that
// takes cost a single pass 10 %).
template <bool SILU, bool MULTI>
__global__ void __launch_bounds__(ring::kThreads, 2) q4_gemv_ring_kernel(const __grid_constant__ GemvParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[ring::kStages], empty[ring::kStages];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cta = blockIdx.x, grid = gridDim.x;
    const int Pc = p.Pc, T = p.T, nchunks = p.nchunks, row_bytes = Pc * ring::kPairBytes + ring::kRowPad;
    const int groups = (p.total_tiles + T - 1) / T, my_groups = (groups - cta + grid - 1) / grid, per_pass = ring::kBlockTiles / T;
    if (tid < ring::kStages) {
        mbar_init(&full[tid], 1);
        mbar_init(&empty[tid], ring::kMathWarps);
    }
    mbar_init_fence();
    __syncthreads();

    if (warp == ring::kMathWarps) {
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
                        bulk_g2s(smem + stage * ring::kStageBytes + lane * row_bytes, m.w + (size_t)row * p.PW + word0, bytes, &full[stage]);
                    }
                    __syncwarp();
                    if (++stage == ring::kStages) { stage = 0; parity ^= 1u; }
                }
        // the CTA's shared memory stays until every copy has landed (bounded; the math warps have waited for all of them unless a wait ran out).
        for (int i = max(0, issued - ring::kStages); i < issued; i++) mbar_wait_warp(&full[i % ring::kStages], (i / ring::kStages) & 1);
        return;
    }

    uint8_t* const scr = smem + ring::kStages * ring::kStageBytes + warp * 2 * kExactScratch;
    uint32_t* const meta = reinterpret_cast<uint32_t*>(smem + ring::kStages * ring::kStageBytes + ring::kMathWarps * 2 * kExactScratch + warp * ring::kMetaBytes);
    float* const part = reinterpret_cast<float*>(smem + ring::kStages * ring::kStageBytes + ring::kMathWarps * (2 * kExactScratch + ring::kMetaBytes));
    const int r = lane >> 2, t = lane & 3;
    int ts[2], pi[2];            // this warp's units: tile in the group, pair in the chunk
#pragma unroll
    for (int j = 0; j < 2; j++) {
        ts[j] = (warp + j * ring::kMathWarps) / Pc;
        pi[j] = warp + j * ring::kMathWarps - ts[j] * Pc;
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
    for (int i = tid; i < my_groups * T * kRows; i += 32 * ring::kMathWarps) {   // scales and zero points on their way into L2
        int row;
        const int tile = (cta + i / (T * kRows) * grid) * T + (i / kRows) % T;
        if (tile < p.total_tiles) {
            const GemvMat& m = row_of<SILU>(p, tile, i & 7, row);
            for (int g = 0; g < p.G; g += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(m.s + (size_t)row * p.G + g));
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
    ahead(0, min(per_pass, my_groups), 0);
    file_meta(0, min(per_pass, my_groups), 0);
    for (int b0 = 0; b0 < my_groups; b0 += per_pass) {
        const int bn = min(per_pass, my_groups - b0);
        for (int c = 0; c < nchunks; c++) {
            PairExact px[2];
            bool active[2];
            int wide = 0;
#pragma unroll
            for (int j = 0; j < 2; j++) active[j] = ts[j] < T && 2 * (c * Pc + pi[j]) < p.G;
            if (b0 + c > 0) file_meta(b0, bn, c);
#pragma unroll
            for (int j = 0; j < 2; j++) wide |= (int)quant_pair_exact(hv[j], scr + j * kExactScratch, lane, px[j]) << j;
#pragma unroll
            for (int j = 0; j < 2; j++) zero_step(px[j]);
            const bool last = c + 1 == nchunks;
            if (MULTI && (!last || b0 + per_pass < my_groups)) {
                load_x(last ? 0 : c + 1);
                ahead(last ? b0 + per_pass : b0, last ? min(per_pass, my_groups - b0 - per_pass) : bn, last ? 0 : c + 1);
            }
            for (int lg = 0; lg < bn; lg++) {
                if (ok) {
                    ok = mbar_wait_warp(&full[stage], parity);
                    if (!ok) atomicExch(&g_status, Q4_ERR_TIMEOUT);
                }
                // words 4t..4t + 3 of column r in groups A and B. (Units that are not there multiply whatever lies in the stage; their sums are
                // not kept.)
                uint32_t me[2];
                int c4[2][4];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const uint4* src = reinterpret_cast<const uint4*>(smem + stage * ring::kStageBytes + ((active[j] ? ts[j] * kRows : 0) + r) * row_bytes + (active[j] ? pi[j] : 0) * ring::kPairBytes) + t;
                    const uint4 a = src[0], b = src[4];
                    me[j] = meta[lg * 32 + j * 16 + (lane >> 1)];
                    pair_mma_exact(c4[j], a, b, px[j]);
                }
                __syncwarp();
                if (lane == 0 && ok) mbar_arrive(&empty[stage]);   // (a stage whose copy has not come is not filled again: the producer gives up too)
                if (++stage == ring::kStages) { stage = 0; parity ^= 1u; }
                float y = quad_sum2(pair_share(c4[0], me[0], px[0], lane), pair_share(c4[1], me[1], px[1], lane), lane);
                if (!ok) y = CUDART_NAN_F;   // a copy that never came must not pass for a result
                const bool odd = t & 1;
                if (t < 2 && (odd ? active[1] : active[0])) {
                    float* const d = part + (lg * T + (odd ? ts[1] : ts[0])) * ring::kTileStride + (odd ? pi[1] : pi[0]) * kRows + r;
                    *d = c == 0 ? y : *d + y;
                }
            }
#pragma unroll
            for (int j = 0; j < 2; j++)
                if ((wide >> j) & 1)
                    add_small<SILU>(p, part + ts[j] * ring::kTileStride + pi[j] * kRows, T * ring::kTileStride, *reinterpret_cast<const uint32_t*>(scr + j * kExactScratch), (cta + b0 * grid) * T + ts[j], grid * T, bn, c * Pc + pi[j]);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * ring::kMathWarps) : "memory");
        for (int e0 = warp * 32; e0 < bn * T * kRows; e0 += 32 * ring::kMathWarps) {   // thread 8 * tile + column
            const int e = e0 + lane, lt = e >> 3, tile = (cta + (b0 + lt / T) * grid) * T + lt % T;
            const bool on = e < bn * T * kRows && tile < p.total_tiles;
            float sum = 0.f;
            if (on)
                for (int i = 0; i < Pc; i += 4) {
                    const float* q = part + lt * ring::kTileStride + i * kRows + (e & 7);
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
        if (b0 + per_pass < my_groups) asm volatile("bar.sync 1, %0;" ::"n"(32 * ring::kMathWarps) : "memory");
    }
}

int check_sizes(int K, int N) { return ((K & 7) || (N & 7) || K <= 0 || N <= 0) ? Q4_ERR_UNSUPPORTED_SIZE : Q4_OK; }

void fill_dims(GemvParams& p, int K) {
    p.K = K;
    p.PW = q4_pw(K);
    p.PZ = q4_pz(K);
    p.G = q4_groups(K);
    p.P = q4_div_up(p.G, 2);
}

// Pairs and tiles per stage: the split that takes the CTA with the most work the least time, a chunk's start (activations, scales) counted
// as 1.2 stages (13824 -> 5120: 16 pairs of one tile 4 chunks x 3 stages; 5 pairs of 3 tiles 11 x 1, 21 us).
void make_split(GemvParams& p) {
    const int P = q4_div_up(p.G, 2);
    int best = 0;
    for (int Pc = std::min(P, ring::kUnits); Pc >= 1; Pc--)
        for (int T = 1; T <= std::min(ring::kUnits / Pc, ring::kMaxT); T++) {
            const int cost = q4_div_up(P, Pc) * (10 * q4_div_up(q4_div_up(p.total_tiles, T), ring::kCtas) + 12);
            if (best && cost >= best) continue;
            best = cost;
            p.Pc = Pc;
            p.T = T;
        }
    p.nchunks = q4_div_up(P, p.Pc);
}

// The ring form from 22 MB of packed words and three tiles per SM up: it streams long rows from HBM faster (us, direct and ring: 4096 ->
// 2 x 11008 16.2, 11.3; 28672 -> 8192 42, 33; 8192 x 8192 12.8, 11.3; 11008 -> 4096 10.7, 10.3), the direct one wins below (4096 x 4096 4.2,
// 4.7; 13824 -> 2560 10.8, 11.6) and where tiles are few, whatever the size (28672 -> 2048 15.5, 16.3; 26712 -> 2904 19.9, 20.5).
template <bool SILU>
int launch(GemvParams& p, cudaStream_t s) {
    if (4LL * p.total_tiles * kRows * p.PW > 22000000 && p.total_tiles > 3 * kSms) {
        static_assert(2 * (ring::kSmemBytes + 1024 + 256) <= 228 * 1024, "two CTAs per SM");
        make_split(p);
        const int groups = q4_div_up(p.total_tiles, p.T);
        // (an opt-in of the function on the device, always to the same value)
        auto* kernel = p.nchunks > 1 || groups > ring::kCtas * (ring::kBlockTiles / p.T) ? q4_gemv_ring_kernel<SILU, true> : q4_gemv_ring_kernel<SILU, false>;
        Q4_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ring::kSmemBytes));
        Q4Launch L(dim3(std::min(groups, ring::kCtas)), dim3(ring::kThreads), ring::kSmemBytes, s);
        Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, kernel, p));
        return Q4_OK;
    }
    const int grid = std::min(p.total_tiles, kSms);
    p.nt_div = p.total_tiles / grid;
    p.nt_mod = p.total_tiles % grid;
    Q4Launch L(dim3(grid), dim3(kThreads), 0, s);
    Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, q4_gemv_kernel<SILU>, p));
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

extern "C" int q4_ops_status(void) {
    int st = 0;
    const int none = 0;
    Q4_CUDA_TRY(cudaDeviceSynchronize());
    Q4_CUDA_TRY(cudaMemcpyFromSymbol(&st, g_status, sizeof(st)));
    if (st) Q4_CUDA_TRY(cudaMemcpyToSymbol(g_status, &none, sizeof(none)));
    return st;
}

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
