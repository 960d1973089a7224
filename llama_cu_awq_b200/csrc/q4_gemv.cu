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
// Stream: the same CTAs and tiles. Every warp keeps the digits of up to four pairs in registers for all tiles, so that an item costs its words' way
// through a private ring in shared memory (cp.async by the lanes that read it: no barrier between warps) and about 50 instructions; pairs that
// do not divide by 16 warps are dealt out by items (20 pairs of a 5120-long row: 1.25 a warp; whole ones would be two for some). Scales and
// zero points of a pass of tiles lie in shared memory as the product takes them, brought once for all warps: as copies of their own in the ring they
// were half as many requests again as the words (8192 x 8192 10.1 us; 8.2 without). What bounds it: 2.5 us of start and end (x, scales and the staging behind
// the wait; the sums) and the stream, 5.4 to 5.9 TB/s (2 x 23.4, 2 x 122 MB beyond 23 and 47); 60 % of the issue slots.
//
// Under programmatic dependent launch the next product's packed words are requested while this one drains (weights never depend on
// activations). Back to back on weights from HBM, bulk copies into a ring shared by a CTA's warps (before) and now, us: 4096 x 4096 4.2 (direct, both);
// q|k|v of 7B 9.1, 7.3, of 13B 14.4, 10.7; 4096 -> 2 x 11008 11.3, 10.5; 5120 -> 2 x 13824 22.2, 15.7; 8192 -> 2 x 28672 54, 46.9; 11008 -> 4096 10.4, 8.2;
// 28672 -> 8192 34.8, 27.2; 8192 x 8192 11.3, 8.2; 512 x 512 1.6 (direct, both). Error against 64 bits 2.1e-4 (an fp16 result's own rounding).
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
    int nt_div, nt_mod;   // direct and stream forms: CTA c has nt_div + (c < nt_mod) consecutive tiles
    int pass_tiles;       // stream form: tiles per pass
    float inv_mrow;       // 1 / meta_row(G)
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

// The warps' sums in warp order and the outputs of `tiles` tiles; 16 warps. Thread 8 * tile + column.
template <bool SILU>
__device__ __forceinline__ void write_out(const GemvParams& p, const float* part, int tile0, int tiles, int w, int lane) {
    for (int e0 = w * 32; e0 < tiles * kRows; e0 += kThreads) {
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
        write_out<SILU>(p, part, tile0, tiles, w, lane);
        if (b0 + kBlockTiles < cta_tiles) __syncthreads();
    }
}

namespace stream {
// Pairs that a warp keeps: its digits take ten registers each (5 instead of 4: 28672 -> 8192 30.8 us, 29.8; 7 spill dozens, 33.5; gate/up with 4 spills one, once).
constexpr int kMaxOwn = 4;
constexpr int kItemBytes = 1024;
constexpr int kPassTiles = 28;       // tiles per pass at most (their partial sums are in shared memory)
constexpr int kSmemBytes = 226 * 1024;
// Items in a warp's ring: a multiple of the pairs it keeps, so that the requests beside a tile's items are those of one tile. (Ten instead of six:
// q|k|v of 7B 7.9 us, 7.3; 13824 -> 5120 11.6, 10.7; four: 8.5 for 8192 x 8192, 8.2.)
__host__ __device__ constexpr int depth(int PP) { return PP == 4 ? 8 : 6; }
constexpr int kEarly = 4;            // of them, requested before the kernel in front has ended (six: q|k|v 7.5, 7.3; two: 4096 x 11008 6.9, 6.7)
__host__ __device__ constexpr int ring_bytes(int PP) { return kWarps * (depth(PP) * kItemBytes + kExactScratch); }
__host__ __device__ constexpr int meta_bytes(int PP) { return kSmemBytes - ring_bytes(PP) - kPassTiles * kTileStride * 4; }   // scales and zero points of a pass
// Words of a row of them (scale | zero point << 16, and zero for the group that a last pair may lack): an odd number, so that the rows of a tile
// lie in different banks.
__host__ __device__ constexpr int meta_row(int G) { return (G + 1) | 1; }
constexpr int tiles_in_pass(int G, int PP) { return std::min(meta_bytes(PP) / (4 * kRows * meta_row(G)), kPassTiles); }
}  // namespace stream

// PP: pairs that every warp keeps; the items of the pairs that are left are dealt out over the warps.
template <bool SILU, int PP>
__global__ void __launch_bounds__(kThreads, 1) q4_gemv_stream_kernel(const __grid_constant__ GemvParams p) {
    using namespace stream;
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int kDepth = depth(PP);
    __shared__ uint32_t small_of[kWarps][PP + 1];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, cta = blockIdx.x;
    const int cta_tile0 = cta * p.nt_div + min(cta, p.nt_mod), cta_tiles = p.nt_div + (cta < p.nt_mod);
    const int p0 = w * PP, rest = p.P - PP * kWarps;
    uint8_t* const ring = smem + w * kDepth * kItemBytes;
    uint8_t* const scr = smem + kWarps * kDepth * kItemBytes + w * kExactScratch;
    uint32_t* const meta = reinterpret_cast<uint32_t*>(smem + ring_bytes(PP));
    float* const part = reinterpret_cast<float*>(smem + ring_bytes(PP) + meta_bytes(PP));
    const int mrow = meta_row(p.G);

    // Walks this warp's items with the lane's addresses: in a pass its own pairs tile by tile, then its share of the items of the pairs that are
    // left, pair by pair. The lane copies 16 bytes (lane & 7) of rows lane >> 3 and 4 + (lane >> 3); in odd rows the pair's groups change places,
    // so that two rows' pieces of a load lie in different banks.
    const uint32_t dst0 = smem_u32(ring) + (lane >> 3) * 128 + (((lane & 7) ^ ((lane >> 1) & 4)) * 16);
    const int step = (SILU ? kRows / 2 : kRows) * p.PW, half = (SILU ? 2 : 4) * p.PW;
    struct {
        const uint32_t* src;     // of the tile's first own pair, or of the item (rest)
        int tile, k, pair, left, b0, tiles, end;     // k < PP: own pairs; PP: rest, `left` items of it to come, `pair` the pair
    } q;
    auto seek = [&](int pair) {
        int row;
        const GemvMat& m = row_of<SILU>(p, cta_tile0 + q.tile, lane >> 3, row);
        q.src = m.w + (size_t)row * p.PW + pair * 32 + (lane & 7) * 4;
        q.end = cta_tiles;
        if (!SILU && p.nmat > 1) q.end = min(q.end, m.tile0 + m.n / kRows - cta_tile0);
    };
    // to the rest of the pass that starts at q.b0, or, if the warp has none, to the next pass
    auto open_pass = [&]() {
        q.tiles = min(p.pass_tiles, cta_tiles - q.b0);
        q.tile = q.b0;
        q.k = 0;
        q.pair = p0;
        if (q.tiles > 0) seek(p0);
    };
    auto open_rest = [&]() {
        const int r0 = w * rest * q.tiles / kWarps, r1 = (w + 1) * rest * q.tiles / kWarps;
        q.k = PP;
        q.left = r1 - r0;
        q.pair = PP * kWarps + r0 / q.tiles;
        q.tile = q.b0 + r0 % q.tiles;
        if (q.left > 0) seek(q.pair);
    };
    auto settle = [&]() {      // past rests that are empty
        while (q.tiles > 0 && q.k == PP && q.left == 0) {
            q.b0 += q.tiles;
            open_pass();
            if (PP == 0 && q.tiles > 0) open_rest();
        }
    };
    auto next = [&]() {
        if (q.k < PP) {
            if (++q.k < PP) return;
            q.k = 0;
            q.src += step;
            if (++q.tile < q.b0 + q.tiles) {
                if (!SILU && p.nmat > 1 && q.tile == q.end) seek(p0);
                return;
            }
            open_rest();
        } else {
            q.left--;
            q.src += step;
            if (++q.tile == q.b0 + q.tiles) {
                q.tile = q.b0;
                q.pair++;
                if (q.left > 0) seek(q.pair);
            } else if (!SILU && p.nmat > 1 && q.tile == q.end && q.left > 0) {
                seek(q.pair);
            }
        }
        settle();
    };
    auto request = [&](uint32_t slot) {      // (slot: its first byte)
        if (q.tiles > 0) {
            const int at = (q.k < PP ? p0 + q.k : q.pair) * 32 + (lane & 7) * 4;
            if (at < p.PW) {
                const uint32_t* src = q.src + (q.k < PP ? q.k * 32 : 0);
                copy16(dst0 + slot, src);
                copy16(dst0 + slot + 512, src + half);
            }
            next();
        }
        copies_commit();
    };
    q.b0 = q.left = 0;
    open_pass();
    if (PP == 0) {
        open_rest();
        settle();
    }
    for (int i = 0; i < kEarly; i++) request(i * kItemBytes);
    // scales and zero points on their way into L2
    for (int i = tid; i < cta_tiles * kRows; i += kThreads) {
        int row;
        const GemvMat& m = row_of<SILU>(p, cta_tile0 + i / kRows, i % kRows, row);
        for (int g = 0; g < p.G; g += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(m.s + (size_t)row * p.G + g));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(m.z + (size_t)row * p.PZ));
    }
    griddep_wait();
    griddep_launch_dependents();
    auto load_x = [&](int pair) {
        const int at = pair * 256 + lane * 8;
        return at < p.K ? *reinterpret_cast<const uint4*>(p.x + at) : make_uint4(0, 0, 0, 0);
    };
    uint4 hv[PP + 1];
#pragma unroll
    for (int k = 0; k < PP; k++) hv[k] = load_x(p0 + k);
    // A pass's scales and zero points into shared memory; eight a thread in flight.
    constexpr int kFlight = 8;
    auto load_meta = [&](int b0, int tiles) {
        const int ns = tiles * kRows * mrow;
        for (int e0 = tid; e0 < ns; e0 += kFlight * kThreads) {
            __half v[kFlight];
            uint32_t z[kFlight];
#pragma unroll
            for (int u = 0; u < kFlight; u++) {
                const int e = e0 + u * kThreads, i = (int)(((float)e + 0.5f) * p.inv_mrow), g = e - i * mrow;
                v[u] = __float2half(0.f);
                z[u] = 0;
                if (e < ns && g < p.G) {
                    int row;
                    const GemvMat& m = row_of<SILU>(p, cta_tile0 + b0 + i / kRows, i % kRows, row);
                    v[u] = __ldg(m.s + (size_t)row * p.G + g);
                    z[u] = __ldg(m.z + (size_t)row * p.PZ + (g >> 3));
                }
            }
#pragma unroll
            for (int u = 0; u < kFlight; u++) {
                const int e = e0 + u * kThreads, g = e - (int)(((float)e + 0.5f) * p.inv_mrow) * mrow;
                if (e < ns) meta[e] = (uint32_t)__half_as_ushort(v[u]) | (((z[u] >> (4 * (g & 7))) & 0xFu) << 16);
            }
        }
    };
    // this warp's share of a pass's items of the pairs that are left
    int pair, tile, left;
    uint4 hr = make_uint4(0, 0, 0, 0);
    auto open_share = [&](int tiles) {
        const int r0 = w * rest * tiles / kWarps, r1 = (w + 1) * rest * tiles / kWarps;
        pair = PP * kWarps + r0 / tiles;
        tile = r0 % tiles;
        left = r1 - r0;
        if (left > 0) hr = load_x(pair);
    };
    open_share(min(p.pass_tiles, cta_tiles));
    load_meta(0, min(p.pass_tiles, cta_tiles));
    for (int i = kEarly; i < kDepth; i++) request(i * kItemBytes);
    PairExact px[PP + 1];        // (the last one: a pair that is left, for the tiles it is this warp's)
    int wide = 0;
#pragma unroll
    for (int k = 0; k < PP; k++) {
        if (quant_pair_exact(hv[k], scr, lane, px[k])) {
            wide |= 1 << k;
            if (lane == 0) small_of[w][k] = *reinterpret_cast<const uint32_t*>(scr);
            __syncwarp();
        }
        zero_step(px[k]);
    }

    const int c = lane >> 2, t = lane & 3;
    const uint8_t* const words = ring + c * 128 + t * 16 + (c & 1) * 64;
    const int other = c & 1 ? -64 : 64;
    uint32_t slot = 0;           // the next item's, its first byte
    // One item's share of the lane; the copies that take its place are `more`'s.
    auto item = [&](const PairExact& x, uint32_t me, auto&& more) {
        copies_wait<kDepth - 1>();
        __syncwarp();
        const uint4 a = *reinterpret_cast<const uint4*>(words + slot), b = *reinterpret_cast<const uint4*>(words + slot + other);
        int d[4];
        pair_mma_exact(d, a, b, x);
        const float y = pair_share(d, me, x, lane);
        __syncwarp();
        more(slot);
        slot += kItemBytes;
        if (slot == kDepth * kItemBytes) slot = 0;
        return y;
    };
    for (int b0 = 0; b0 < cta_tiles; b0 += p.pass_tiles) {
        const int tiles = min(p.pass_tiles, cta_tiles - b0);
        float* const col = part + w * kRows + c;
        if (PP == 0)
            for (int i = lane; i < tiles * kRows; i += 32) part[(i >> 3) * kTileStride + w * kRows + (i & 7)] = 0.f;
        __syncthreads();         // the pass's scales and zero points are in place
        const uint32_t* me = meta + c * mrow + ((lane >> 1) & 1) + 2 * p0;
        if (PP > 0) {
            const int lane_at = p0 * 32 + (lane & 7) * 4;
            for (int i = 0; i < tiles; i++) {
                float y = 0.f;
                // Within the own pairs of a pass and of a matrix the next requests are those of one tile.
                if (q.tiles > 0 && q.k == 0 && q.tile + 1 < min(q.end, q.b0 + q.tiles)) {
#pragma unroll
                    for (int k = 0; k < PP; k++)
                        y += item(px[k], me[2 * k], [&](uint32_t at) {
                            if (lane_at + k * 32 < p.PW) {
                                copy16(dst0 + at, q.src + k * 32);
                                copy16(dst0 + at + 512, q.src + k * 32 + half);
                            }
                            copies_commit();
                        });
                    q.src += step;
                    q.tile++;
                } else {
#pragma unroll
                    for (int k = 0; k < PP; k++) y += item(px[k], me[2 * k], request);
                }
                y = quad_sum(y);
                if (t == 0) col[i * kTileStride] = y;
                me += kRows * mrow;
            }
            for (int k = 0; wide >> k; k++)
                if ((wide >> k) & 1) add_small<SILU>(p, part + w * kRows, kTileStride, small_of[w][k], cta_tile0 + b0, 1, tiles, p0 + k);
        }
        while (left > 0) {
            const int count = min(left, tiles - tile);
            const bool more = quant_pair_exact(hr, scr, lane, px[PP]);
            zero_step(px[PP]);
            left -= count;
            if (left > 0) hr = load_x(pair + 1);
            me = meta + (tile * kRows + c) * mrow + ((lane >> 1) & 1) + 2 * pair;
            for (int i = 0; i < count; i++) {
                const float y = quad_sum(item(px[PP], *me, request));
                if (t == 0) col[(tile + i) * kTileStride] += y;
                me += kRows * mrow;
            }
            if (more)
                add_small<SILU>(p, part + tile * kTileStride + w * kRows, kTileStride, *reinterpret_cast<const uint32_t*>(scr), cta_tile0 + b0 + tile, 1, count, pair);
            pair++;
            tile = 0;
        }
        __syncthreads();
        write_out<SILU>(p, part, cta_tile0 + b0, tiles, w, lane);
        if (b0 + tiles < cta_tiles) {
            open_share(min(p.pass_tiles, cta_tiles - b0 - tiles));
            load_meta(b0 + tiles, min(p.pass_tiles, cta_tiles - b0 - tiles));
            __syncthreads();     // (the partial sums are written again)
        }
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

template <bool SILU, int PP>
int launch_stream(GemvParams& p, cudaStream_t s) {
    const int grid = std::min(p.total_tiles, kSms);
    p.nt_div = p.total_tiles / grid;
    p.nt_mod = p.total_tiles % grid;
    const int most = p.nt_div + (p.nt_mod > 0);
    p.pass_tiles = q4_div_up(most, q4_div_up(most, stream::tiles_in_pass(p.G, PP)));
    p.inv_mrow = 1.0f / stream::meta_row(p.G);
    // (an opt-in of the function on the device, always to the same value)
    Q4_CUDA_TRY(cudaFuncSetAttribute(q4_gemv_stream_kernel<SILU, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, stream::kSmemBytes));
    Q4Launch L(dim3(grid), dim3(kThreads), (size_t)stream::kSmemBytes, s);
    Q4_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, q4_gemv_stream_kernel<SILU, PP>, p));
    return Q4_OK;
}

// The stream form from 20 MB of packed words up, and from rows of 32 pairs on below that (bytes * pairs of a row >= 180 MB). The direct form starts about
// a microsecond earlier, which a call on words that are in L2 already (one matrix again and again) shows most; a model's come from HBM. The line lies where
// what one side loses is what the other gains (two layers of 13B call by call, whose o is 13 MB: 129.4 us, 128.3 in the stream form). us, direct and stream, from HBM; from L2: 1024 x 24000 5.4, 5.5; 4.2, 5.3. 2048 x 9216 4.6, 4.9; 3.8, 4.8.
// 4096 x 4608 4.5, 4.5; 3.6, 4.4. 5120 x 5120 6.6, 6.1; 4.9, 6.0. 4096 x 8192 6.9, 6.1; 4.7, 5.8. 4096 x 10240 (21 MB) 8.1, 6.6; 5.5, 6.3.
// 8192 x 2048 4.9, 4.5; 4.3, 4.5. 8192 x 4096 7.6, 6.1; 5.6, 5.8. 12288 x 1024 4.9, 4.5; 4.7, 4.5. 13824 x 640 5.4, 4.9; 5.1, 4.9. 28672 x 512 9.6, 7.8;
// 8.3, 8.0. Ratio over the range (3 to 28 MB), L2 and HBM: 4 to 12 pairs 1.2, 1.1 at 9 MB, 1.2, 0.9 at 18, 1.14, 0.85 at 22; 16 to 28 pairs 1.2, 0.9 at 16, 1.1,
// 0.8 at 22; 32 to 43 pairs 1.0 to 1.1, 0.75 to 0.9 from 6 MB; 48 and 64 pairs 0.9 to 1.0, 0.65 to 0.9. Rows of less than four pairs stay with the direct form whatever the
// size (512 x 60000 7.6, 8.5 from HBM), and rows whose scales for a tile do not fit into shared memory (more than 266496 inputs).
template <bool SILU>
int launch(GemvParams& p, cudaStream_t s) {
    const long long bytes = 4LL * p.total_tiles * kRows * p.PW;
    if (p.P >= 4 && (bytes >= 20000000 || (p.P >= 32 && bytes * p.P >= 180000000)) && stream::tiles_in_pass(p.G, stream::kMaxOwn) > 0) {
        switch (std::min(p.P / kWarps, stream::kMaxOwn)) {
            case 0: return launch_stream<SILU, 0>(p, s);
            case 1: return launch_stream<SILU, 1>(p, s);
            case 2: return launch_stream<SILU, 2>(p, s);
            case 3: return launch_stream<SILU, 3>(p, s);
            default: return launch_stream<SILU, 4>(p, s);
        }
    }
    const int grid = std::min(p.total_tiles, kSms);
    p.nt_div = p.total_tiles / grid;
    p.nt_mod = p.total_tiles % grid;
    Q4Launch L(dim3(grid), dim3(kThreads), 0, s);
    // (scales and zero words are read from L1 again and again: behind a kernel that has taken the SM's memory as shared, as the stream form does, the
    // split would stay as it is. Two layers call by call 99.7 us, 97.9 so)
    static std::atomic<unsigned long long> preferred{0};
    Q4_CUDA_TRY(q4_prefer_carveout(q4_gemv_kernel<SILU>, 20, preferred));
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
    Q4_CUDA_TRY(cudaDeviceSynchronize());
    return Q4_OK;     // (no product has a wait that could run out)
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
