// The W4 dot product of one activation row on the integer tensor pipe, shared by the fused decode kernel (q4_fused.cu) and the
// per-op GEMV (q4_gemv.cu).
//
// Activations are re-expressed per group of 128 as 16-bit block fixed point X = rint(x / sx), sx = max|x| / 32512. A packed
// byte b = 16*qo + ql (odd and even input) is multiplied as it lies and once more with its low nibble:
//     sum b*Xo + sum ql*(16*Xe - Xo) = 16 * sum q*X,
// one AND per packed word. Both multipliers are split into signed bytes (weights 65536, 256, 1), which are columns of
// mma.sync.m16n8k32 (u8 x s8, int32): exact integer arithmetic. Rows 0-7 of the product are 8 output columns over group A of a
// pair of groups, rows 8-15 the same columns over group B; columns 0-3 are group A's bytes, 4-7 group B's, and the two crosswise
// quarters are not used. Per (column, group): y += scale * sx * sum (q - zero) * X, fp32. An element is off by max|x| / 65024 at most,
// below fp16's own rounding of the largest elements; nibbles, zero points and scales are used exactly. The fused kernel multiplies so
// what it has computed itself; a caller's x goes through the exact form below (PairExact).
// Per 16 columns x 128 inputs: 8 half-rate ANDs per lane and 4 products at 8 clocks, where DP4A took 48 half-rate operations and
// half2 FMA 72.
#pragma once
#include <math_constants.h>

#include "q4_common.cuh"

constexpr int kPairScratch = 1024;   // bytes of shared memory per warp: one pair's digits on their way into operand order

__device__ __forceinline__ void mma_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_u8s8_first(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {   // c = a b
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
// One pair's activations (2 groups = 256 inputs) in operand order, in registers.
struct PairX {
    uint4 raw, lo;      // digits that meet the packed bytes as they lie, and the low nibbles
    float sx;           // scale of X, divided by 16
    int s16;            // 16 * sum of X over the lane's group (lanes that hold the high digits), else 0
};

// Quantises one pair (lane l holds elements 8l..8l+7 as fp16). X comes out of an FMA with a magic constant (the integer sits in the
// low mantissa bits) that also adds 0x8080: the bytes of X + 0x8080, each with its top bit flipped, are X's signed digits, and
// likewise those of 16*Xe - Xo + 0x808080. The digits are gathered by four with byte permutes and go through the warp's scratch
// into the product's column operand. Lane 4n + t of it is column n and holds four of the group's 16 words: t, 4 + t, 8 + t, 12 + t.
// A NaN makes its group's scale NaN, an infinity makes it infinite (the group's finite elements count as nothing beside it).
__device__ __forceinline__ void quant_pair(const uint4& hv, uint8_t* scr, int lane, PairX& px) {
    constexpr float kMagic = 12582912.0f + 32896.0f;   // 1.5 * 2^23 + 0x8080
    constexpr uint32_t kBits = 0x4B408080u;
    const __half2* h = reinterpret_cast<const __half2*>(&hv);
    const bool high = lane & 16;                    // 16 lanes = 1 group
    // |x| as integers: fp16 bits without the sign are in the order of the values, NaN above infinity
    const uint32_t m4 = __vmaxu2(__vmaxu2(hv.x & 0x7FFF7FFFu, hv.y & 0x7FFF7FFFu), __vmaxu2(hv.z & 0x7FFF7FFFu, hv.w & 0x7FFF7FFFu));
    const uint32_t mine = max(m4 & 0xFFFFu, m4 >> 16);
    const uint32_t ma = __reduce_max_sync(0xffffffffu, high ? 0u : mine), mb = __reduce_max_sync(0xffffffffu, high ? mine : 0u);
    const float amax = __half2float(__ushort_as_half((unsigned short)(high ? mb : ma)));
    float inv = amax > 0.f ? 32512.0f / amax : 0.f;
    float2 f[4];
#pragma unroll
    for (int j = 0; j < 4; j++) f[j] = __half22float2(h[j]);
    if (amax == CUDART_INF_F) {
        inv = 32512.0f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            f[j].x = isinf(f[j].x) ? copysignf(1.f, f[j].x) : 0.f;
            f[j].y = isinf(f[j].y) ? copysignf(1.f, f[j].y) : 0.f;
        }
    }
    uint32_t e[4], o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        e[j] = __float_as_uint(fmaf(f[j].x, inv, kMagic));
        o[j] = __float_as_uint(fmaf(f[j].y, inv, kMagic));
    }
    const int part = (int)(((e[0] + o[0]) + (e[1] + o[1])) + ((e[2] + o[2]) + (e[3] + o[3])) - 8u * kBits);
    const int sum_a = __reduce_add_sync(0xffffffffu, high ? 0 : part), sum_b = __reduce_add_sync(0xffffffffu, high ? part : 0);
    const uint32_t o01 = prmt(o[0], o[1], 0x5140), o23 = prmt(o[2], o[3], 0x5140);
    const uint32_t r0 = prmt(o01, o23, 0x5410) ^ 0x80808080u, r1 = prmt(o01, o23, 0x7632) ^ 0x80808080u;
    uint32_t z[4];
#pragma unroll
    for (int j = 0; j < 4; j++) z[j] = 16u * e[j] - o[j] + (0x808080u - 15u * kBits);
    const uint32_t z01 = prmt(z[0], z[1], 0x5140), z23 = prmt(z[2], z[3], 0x5140);
    const uint32_t l0 = prmt(z01, z23, 0x5410) ^ 0x80808080u, l1 = prmt(z01, z23, 0x7632) ^ 0x80808080u;
    const uint32_t l2 = prmt(prmt(z[0], z[1], 0x0062), prmt(z[2], z[3], 0x0062), 0x5410) ^ 0x80808080u;
    // word j = lane & 15 of group lane >> 4 -> [column 4 * group + digit][t][position in t's four words]
    const int j = lane & 15, at = (j & 3) * 4 + (j >> 2);
    uint32_t* d = reinterpret_cast<uint32_t*>(scr) + (lane >> 4) * 64 + at;
    __syncwarp();       // the previous pair's digits have been read
    d[0] = 0;       d[16] = r1;       d[32] = r0;       d[48] = 0;
    d[128] = l2;    d[128 + 16] = l1; d[128 + 32] = l0; d[128 + 48] = 0;
    __syncwarp();
    px.raw = *reinterpret_cast<const uint4*>(scr + lane * 16);
    px.lo = *reinterpret_cast<const uint4*>(scr + 512 + lane * 16);
    px.sx = __half2float(__ushort_as_half((unsigned short)((lane & 2) ? mb : ma))) * (1.0f / (32512.0f * 16.0f));
    if (px.sx == CUDART_INF_F && (lane & 1)) px.sx = 0.f;   // (the low digits are zero then, and must not turn the sum into 0 * inf)
    px.s16 = (lane & 1) ? 0 : 16 * ((lane & 2) ? sum_b : sum_a);
}

// One pair's product with 8 columns. Lane 4c + t: wa = words h = 0, 1 and wb = words h = 2, 3 of its four packed words of column c,
// each as (group A, h), (group B, h), (group A, h + 1), (group B, h + 1): the product's row operand as it lies in registers.
__device__ __forceinline__ void pair_mma(int (&c)[4], const uint4& wa, const uint4& wb, const PairX& px) {
    constexpr uint32_t kLow = 0x0F0F0F0Fu;
    mma_u8s8_first(c, wa.x, wa.y, wa.z, wa.w, px.raw.x, px.raw.y);
    mma_u8s8(c, wa.x & kLow, wa.y & kLow, wa.z & kLow, wa.w & kLow, px.lo.x, px.lo.y);
    mma_u8s8(c, wb.x, wb.y, wb.z, wb.w, px.raw.z, px.raw.w);
    mma_u8s8(c, wb.x & kLow, wb.y & kLow, wb.z & kLow, wb.w & kLow, px.lo.z, px.lo.w);
}
// This lane's share of column lane >> 2, to be added over the quad. meta: fp16 scale | zero point << 16 of the column in group
// (lane >> 1) & 1. Lanes t = 0, 1 hold rows 0-7, columns 0, 1 (weights 65536, 256) and 2, 3 (1, unused) of group A, t = 2, 3 rows 8-15
// of group B.
__device__ __forceinline__ float pair_share(const int (&c)[4], uint32_t meta, const PairX& px, int lane) {
    const bool upper = lane & 2;
    const int w0 = (lane & 1) ? 1 : 65536, w1 = (lane & 1) ? 0 : 256;
    const int v = (upper ? c[2] : c[0]) * w0 + (upper ? c[3] : c[1]) * w1 - (int)(meta >> 16) * px.s16;
    return (float)v * (__half2float(__ushort_as_half((unsigned short)(meta & 0xFFFFu))) * px.sx);
}
// ---- the same product with x as it is (the per-op GEMV, whose x is the caller's) ----
// X = x / sx with a power of two for sx, so that the group's largest element has 26 bits: every element down to 2^-15 of it is held
// exactly, all four columns of a group carry digits (weights 2^24, 65536, 256, 1), and the zero point is taken off column by column, so
// that an element whose weight is zero leaves nothing behind. Smaller elements are rounded to 2^-27 of the largest (2^-15 of what that
// one's own fp16 rounding is; an output of SiLU has many such), unless fewer than kManyHeld elements are held exactly: then, and in a
// group with a NaN or an infinity, the elements that X does not hold are left out of it and multiplied in fp32 (small_dot).
constexpr int kManyHeld = 32;
constexpr int kExactScratch = 1152;  // bytes of shared memory per warp
struct PairExact {
    uint4 raw, lo;
    float sx;           // scale of the lane's columns of digits, divided by 16
    int zero;           // what one step of the zero point adds to them
};

// Returns true (to the whole warp) when some elements are left to small_dot: those of group A (B) whose magnitude is below the fp16 bits
// in the lower (upper) half of the scratch's first word.
__device__ __forceinline__ bool quant_pair_exact(const uint4& hv, uint8_t* scr, int lane, PairExact& px) {
    const __half2* h = reinterpret_cast<const __half2*>(&hv);
    const bool high = lane & 16;
    const uint32_t mag[4] = {hv.x & 0x7FFF7FFFu, hv.y & 0x7FFF7FFFu, hv.z & 0x7FFF7FFFu, hv.w & 0x7FFF7FFFu};
    const uint32_t m4 = __vmaxu2(__vmaxu2(mag[0], mag[1]), __vmaxu2(mag[2], mag[3]));
    const uint32_t mine = max(m4 & 0xFFFFu, m4 >> 16);
    const uint32_t ma = __reduce_max_sync(0xffffffffu, high ? 0u : mine), mb = __reduce_max_sync(0xffffffffu, high ? mine : 0u);
    // 2^(40 - E) for the largest element's exponent field E (fp16): X = x * that, up to 2^26
    const float mul = __uint_as_float((167u - ((high ? mb : ma) >> 10)) << 23);
    float2 f[4];
#pragma unroll
    for (int j = 0; j < 4; j++) f[j] = __half22float2(h[j]);
    uint32_t small = 0;
    if (max(ma, mb) >= (17u << 10)) {   // 4 and more: below, every fp16 has all its bits in X
        // the fp16 bits below which an element has bits that X does not hold; everything in a group with a NaN or an infinity
        auto below = [](uint32_t m) { return m >= 0x7C00u ? 0x8000u : m >= (17u << 10) ? ((m >> 10) - 15u) << 10 : 0u; };
        uint32_t lim = below(high ? mb : ma);
        int held = 0;       // elements that are not zero and have all their bits in X
#pragma unroll
        for (int j = 0; j < 4; j++) held += ((mag[j] & 0xFFFFu) >= max(lim, 1u)) + ((mag[j] >> 16) >= max(lim, 1u));
        const int na = __reduce_add_sync(0xffffffffu, high ? 0 : held), nb = __reduce_add_sync(0xffffffffu, high ? held : 0);
        const uint32_t la = ma < 0x7C00u && na >= kManyHeld ? 0u : below(ma), lb = mb < 0x7C00u && nb >= kManyHeld ? 0u : below(mb);
        small = la | (lb << 16);
        lim = high ? lb : la;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if ((mag[j] & 0xFFFFu) < lim) f[j].x = 0.f;
            if ((mag[j] >> 16) < lim) f[j].y = 0.f;
        }
    }
    // The bytes of X + 0x80808080, each with its top bit flipped, are X's signed digits, and likewise those of 16 Xe - Xo + 0x80808080.
    // (Conversions have a pipe of their own; splitting X by magic constants instead costs twice as many issue slots.)
    uint32_t o[4], z[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        o[j] = (uint32_t)__float2int_rn(f[j].y * mul) + 0x80808080u;
        z[j] = 16u * (uint32_t)__float2int_rn(f[j].x * mul) + (0x01010100u - o[j]);
    }
    // word j = lane & 15 of group lane >> 4 -> [column 4 * group + digit][j], the groups 16 banks apart
    uint32_t* d = reinterpret_cast<uint32_t*>(scr) + (lane >> 4) * 80 + (lane & 15);
    __syncwarp();       // the previous pair's digits have been read
    auto file = [](uint32_t* to, const uint32_t (&w)[4]) {
        const uint32_t l01 = prmt(w[0], w[1], 0x5140), l23 = prmt(w[2], w[3], 0x5140), h01 = prmt(w[0], w[1], 0x7362), h23 = prmt(w[2], w[3], 0x7362);
        to[0] = prmt(h01, h23, 0x7632) ^ 0x80808080u;
        to[16] = prmt(h01, h23, 0x5410) ^ 0x80808080u;
        to[32] = prmt(l01, l23, 0x7632) ^ 0x80808080u;
        to[48] = prmt(l01, l23, 0x5410) ^ 0x80808080u;
    };
    file(d, o);
    file(d + 144, z);
    __syncwarp();
    const uint8_t* mine4 = scr + lane * 16 + (lane >> 4) * 64;
    px.raw = *reinterpret_cast<const uint4*>(mine4);
    px.lo = *reinterpret_cast<const uint4*>(mine4 + 576);
    // sx / 16 = 2^(E - 44), and for the upper two digits' columns 65536 times that
    px.sx = __uint_as_float((((lane & 2) ? mb : ma) >> 10) + ((lane & 1) ? 83u : 99u) << 23);
    px.zero = 0;        // (zero_step)
    if (small) {
        __syncwarp();
        if (lane == 0) *reinterpret_cast<uint32_t*>(scr) = small;
        __syncwarp();
    }
    return small != 0;
}
// The product with weights of one everywhere (17 as a byte, 1 as a low nibble): what one step of the zero point adds to each column. Apart
// from quant_pair_exact, so that a warp with two pairs does not wait for the first one's digits before it starts on the second's.
__device__ __forceinline__ void zero_step(PairExact& px) {
    int a[4], b[4];
    mma_u8s8_first(a, 0x11111111u, 0x11111111u, 0x11111111u, 0x11111111u, px.raw.x, px.raw.y);
    mma_u8s8_first(b, 0x11111111u, 0x11111111u, 0x11111111u, 0x11111111u, px.raw.z, px.raw.w);
    mma_u8s8(a, 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u, px.lo.x, px.lo.y);
    mma_u8s8(b, 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u, px.lo.z, px.lo.w);
    px.zero = 256 * (a[0] + b[0]) + a[1] + b[1];
}
// pair_mma of lane 4c + t with words 4t..4t + 3 of column c in groups A and B, as two chains: a chain's next product waits for the one before
__device__ __forceinline__ void pair_mma_exact(int (&c)[4], const uint4& a, const uint4& b, const PairExact& px) {
    constexpr uint32_t kLow = 0x0F0F0F0Fu;
    int d[4];
    mma_u8s8_first(c, a.x, b.x, a.y, b.y, px.raw.x, px.raw.y);
    mma_u8s8_first(d, a.z, b.z, a.w, b.w, px.raw.z, px.raw.w);
    mma_u8s8(c, a.x & kLow, b.x & kLow, a.y & kLow, b.y & kLow, px.lo.x, px.lo.y);
    mma_u8s8(d, a.z & kLow, b.z & kLow, a.w & kLow, b.w & kLow, px.lo.z, px.lo.w);
#pragma unroll
    for (int i = 0; i < 4; i++) c[i] += d[i];
}
// As pair_share: lanes t = 0, 2 hold the upper two digits' columns of their group, t = 1, 3 the lower two.
__device__ __forceinline__ float pair_share(const int (&c)[4], uint32_t meta, const PairExact& px, int lane) {
    const bool upper = lane & 2;
    const uint32_t v = (uint32_t)(upper ? c[2] : c[0]) * 256u + (uint32_t)(upper ? c[3] : c[1]) - (meta >> 16) * (uint32_t)px.zero;
    return (float)(int)v * (__half2float(__ushort_as_half((unsigned short)(meta & 0xFFFFu))) * px.sx);
}
// sum + the products of a packed word's nibbles, less the zero point, with those of its 8 inputs whose magnitude is below lim (fp16 bits)
__device__ __forceinline__ float small_dot(uint32_t w, const uint4& xv, uint32_t lim, int zero, float sum) {
    const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const uint32_t bits = (j & 1) ? xw[j >> 1] >> 16 : xw[j >> 1] & 0xFFFFu;
        if ((bits & 0x7FFFu) < lim) sum = fmaf((float)((int)((w >> (4 * j)) & 0xFu) - zero), __half2float(__ushort_as_half((unsigned short)bits)), sum);
    }
    return sum;
}

__device__ __forceinline__ float quad_sum(float y) {
    y += __shfl_xor_sync(0xffffffffu, y, 1);
    return y + __shfl_xor_sync(0xffffffffu, y, 2);
}
// Both sums over the quad: y0's in its even lanes, y1's in its odd ones
__device__ __forceinline__ float quad_sum2(float y0, float y1, int lane) {
    const bool odd = lane & 1;
    const float other = __shfl_xor_sync(0xffffffffu, odd ? y0 : y1, 1);
    const float y = (odd ? y1 : y0) + other;
    return y + __shfl_xor_sync(0xffffffffu, y, 2);
}
