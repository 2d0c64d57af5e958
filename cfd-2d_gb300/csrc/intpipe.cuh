// IEEE binary64 arithmetic on the integer pipes.
//
// GB300's FP64 unit takes two lanes per clock and SM: a warp's FP64 instruction holds it for
// 16 clocks, in which the SM can issue 64 instructions to its other pipes. Kernels that form
// everything on that unit held it 83-88% and the integer pipes under 5%; an operation formed
// from about thirty integer instructions then costs less than the FP64 instruction, and the two
// run side by side (the flux kernel now: 72% and 53%). Every function here returns the correctly
// rounded (to nearest, ties to even) result, the very bits of the FP64 instruction or of the
// IEEE quotient and square root, so a kernel may form any of its operations on either side
// (x^a: within 0.54 units in the last place).
//
// Measured on one SM with all warps resident (clocks per warp operation): product or sum 20
// native (17 as a multiply-add of three registers; an operand from the constant bank or an
// immediate costs the 20), product 10.9 here, 8.3 per product with two native to three here;
// reciprocal 24 (90 native), quotient 34 (144), square root 34 (170). An integer sum took 22.6
// and lost in every kernel it was tried in (two steps at 2.1M triangles 6.48 -> 7.17 ms); it was
// not kept, sums are native. Kernels: k_flux at 2.1M triangles 1.42 -> 0.62 ms, with a lane per
// Gauss point; the same arithmetic in one thread per edge gained nothing there (200-255
// registers). With a warp or less per scheduler an operation's latency counts, and the native
// product is the shorter one (adj_native in adj_inst.cuh).
//
// The common path takes operands with 2^-510 <= |x| < 2^510, whose products and quotients
// stay normal; zeros, and anything else, leave it by a branch.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

namespace cfd2d {
namespace ip {

typedef unsigned int u32;
typedef unsigned long long u64;

#if defined(__CUDA_ARCH__)
#define IP_FN __device__ __forceinline__
__device__ __forceinline__ u32 hi(double x) { return (u32)__double2hiint(x); }
__device__ __forceinline__ u32 lo(double x) { return (u32)__double2loint(x); }
__device__ __forceinline__ double make(u32 h, u32 l) { return __hiloint2double((int)h, (int)l); }
// low word of (h:l) >> s, 0 <= s < 32
__device__ __forceinline__ u32 shr2(u32 l, u32 h, u32 s) { return __funnelshift_r(l, h, s); }
__device__ __forceinline__ u32 shl2(u32 l, u32 h, u32 s) { return __funnelshift_l(l, h, s); }
// approximations of 1/x and 1/sqrt(x), within a few units of the 23rd fraction bit
__device__ __forceinline__ float rcp_seed(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rsqrt_seed(float x) { float y; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ u32 f2u(float x) { return __float2uint_rz(x); }
__device__ __forceinline__ float u2f_bits(u32 b) { return __uint_as_float(b); }
// (qh:ql) + (E << 32), plus one when z > 0x80000000 (z: the bits below the last place with the
// parity and sticky bit merged into bit 0)
__device__ __forceinline__ double round_pack(u32 qh, u32 ql, u32 z, u32 E) {
    u32 h, l;
    asm("{\n\t.reg .u32 d;\n\tadd.cc.u32 d, %4, 0x7fffffff;\n\taddc.cc.u32 %1, %2, 0;\n\taddc.u32 %0, %3, %5;\n\t}"
        : "=r"(h), "=r"(l) : "r"(ql), "r"(qh), "r"(z), "r"(E));
    return make(h, l);
}
// the same with the bits below z in `low`: plus one when z:low > 0x80000000:0 (z's bit 0: the parity)
__device__ __forceinline__ double round_pack2(u32 qh, u32 ql, u32 z, u32 low, u32 E) {
    u32 h, l;
    asm("{\n\t.reg .u32 d;\n\tadd.cc.u32 d, %6, 0xffffffff;\n\taddc.cc.u32 d, %4, 0x7fffffff;\n\t"
        "addc.cc.u32 %1, %2, 0;\n\taddc.u32 %0, %3, %5;\n\t}"
        : "=r"(h), "=r"(l) : "r"(ql), "r"(qh), "r"(z), "r"(E), "r"(low));
    return make(h, l);
}
#else
#define IP_FN inline
inline u64 bits(double x) { u64 b; std::memcpy(&b, &x, 8); return b; }
inline u32 hi(double x) { return (u32)(bits(x) >> 32); }
inline u32 lo(double x) { return (u32)bits(x); }
inline double make(u32 h, u32 l) { const u64 b = ((u64)h << 32) | l; double x; std::memcpy(&x, &b, 8); return x; }
inline u32 shr2(u32 l, u32 h, u32 s) { return (u32)((((u64)h << 32) | l) >> (s & 31)); }
inline u32 shl2(u32 l, u32 h, u32 s) { return (u32)(((((u64)h << 32) | l) << (s & 31)) >> 32); }
inline u32 f2u(float x) { return (u32)x; }
inline float u2f_bits(u32 b) { float x; std::memcpy(&x, &b, 4); return x; }
// off by seed_ulps units in the last place: the results must not depend on the seed
inline int& seed_ulps() { static int d = 0; return d; }
inline float nudge(float x) { u32 b; std::memcpy(&b, &x, 4); return u2f_bits(b + (u32)seed_ulps()); }
inline float rcp_seed(float x) { return nudge(1.0f / x); }
inline float rsqrt_seed(float x) { return nudge((float)(1.0 / __builtin_sqrt((double)x))); }
inline double round_pack(u32 qh, u32 ql, u32 z, u32 E) {
    const u64 q = (((u64)qh << 32) | ql) + (z > 0x80000000u ? 1 : 0) + ((u64)E << 32);
    return make((u32)(q >> 32), (u32)q);
}
inline double round_pack2(u32 qh, u32 ql, u32 z, u32 low, u32 E) { return round_pack(qh, ql, z + (low != 0 ? 1 : 0), E); }
#endif

IP_FN u64 wide(u32 a, u32 b) { return (u64)a * b; }
// 2^-510 <= |x| < 2^510
IP_FN bool in_range(double x) { return (hi(x) << 1) - 0x40200000u < 0x7f800000u; }
IP_FN u32 mant_hi(double x) { return (hi(x) & 0xfffffu) | 0x100000u; }

// a b for operands in range: the 106-bit product of the significands in four wide
// multiplications, shifted to 53 bits and rounded.
IP_FN double mul_core(double a, double b) {
    const u32 ma = mant_hi(a), mb = mant_hi(b), al = lo(a), bl = lo(b);
    const u64 p0 = wide(al, bl);
    u64 t = wide(ma, bl) + (u32)(p0 >> 32);
    t += wide(al, mb);
    const u64 p1 = wide(ma, mb) + (u32)(t >> 32);  // 41 or 42 bits
    const u32 mid = (u32)t, p1l = (u32)p1, p1h = (u32)(p1 >> 32), low = (u32)p0;
    const u32 s = p1h >> 9, sh = s + 20;
    const u32 ql = shr2(mid, p1l, sh), qh = shr2(p1l, p1h, sh), rm = shr2(0u, mid, sh);
    // the sign bits add to their exclusive or, the exponents to the product's
    const u32 E = (hi(a) & 0xfff00000u) + (hi(b) & 0xfff00000u) + (s << 20) - (1024u << 20);
    return round_pack2(qh, ql, rm | (ql & 1u), low, E);
}

// ---- any operands: what the branches above leave to

#if defined(__CUDA_ARCH__)
#define IP_RARE static __device__ __noinline__
#else
#define IP_RARE static inline
#endif

IP_RARE double mul_rare(double a, double b) {
    if (in_range(a) && in_range(b)) return mul_core(a, b);
    return a * b;
}
// a zero times a finite number is the signed zero
IP_FN bool zero_product(double a, double b) {
    const u32 xa = hi(a) << 1, xb = hi(b) << 1;
    return ((xa | lo(a)) == 0 && xb < 0xffe00000u) || ((xb | lo(b)) == 0 && xa < 0xffe00000u);
}
IP_FN double mul_any(double a, double b) {
    if (zero_product(a, b)) return make((hi(a) ^ hi(b)) & 0x80000000u, 0u);
    return mul_rare(a, b);
}
// a b for any operands
IP_FN double mul(double a, double b) {
    if (__builtin_expect(in_range(a) && in_range(b), 1)) return mul_core(a, b);
    return mul_any(a, b);
}
IP_FN double neg(double x) { return make(hi(x) ^ 0x80000000u, lo(x)); }

// N products behind one branch: the compiler interleaves them
template <int N>
IP_FN void muln(double* r, const double* a, const double* b) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < N; k++) ok = ok && in_range(a[k]) && in_range(b[k]);
    if (__builtin_expect(ok, 1)) {
#pragma unroll
        for (int k = 0; k < N; k++) r[k] = mul_core(a[k], b[k]);
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) r[k] = mul_any(a[k], b[k]);
    }
}

// ---- reciprocal, quotient, square root

// 1/m for the significand m of b (1 <= m < 2), Q63, at most 1 unit too small and 2 too large
// (measured over 1.8e8 operands with seeds two units off: -1.002 to 1.996): a binary32 seed and
// two Newton steps in fixed point, the first with a 64-bit significand and a 32-bit reciprocal
// (error 2^-22 -> 2^-43), the second with both in 64 bits, where the error left (2^-86) is far
// below a unit. What counts is the rounding of that second step: the remainder's product without
// its lowest part Bl yl (below 2^-62) makes y up to 2 units too large, the last shift, rounding
// down, up to 1 too small; the remainder's own shift (2^-72) and yh for y (2^-74) add 2^-9 units.
// The last bit of a quotient is decided by the guard bits below it unless these lie within the
// approximation's error of one half; then the exact remainder decides (a quotient of two
// 53-bit significands is never a tie).
struct Recip { u32 yh, yl; };
IP_FN Recip recip_of(double b) {
    const u32 Bh = shl2(lo(b), mant_hi(b), 11), Bl = lo(b) << 11;  // Q63
    // seed: 1/(m 2^-31) in [2^30, 2^31)
    u32 y0 = f2u(rcp_seed(u2f_bits(((Bh >> 8) & 0x7fffffu) | (96u << 23))));
    y0 = y0 < 0x7fffffffu ? y0 : 0x7fffffffu;
    const u64 p = wide(Bh, y0) + (u32)(wide(Bl, y0) >> 32);                   // Q62, about 2^62
    const int e0 = (int)((long long)((1ull << 62) - p) >> 10);                // Q52
    const u64 y1 = ((u64)y0 << 32) + (u64)(((long long)(int)y0 * e0) >> 20);  // Q63
    const u32 yh = (u32)(y1 >> 32), yl = (u32)y1;
    // 1 - m y1 in Q94, modulo 2^64 (the product's lowest 32 bits left out)
    const u64 q = wide(Bh, yl) + wide(Bl, yh) + ((u64)(Bh * yh) << 32);
    const int e1 = (int)((long long)(0ull - q) >> 22);                        // Q72
    const u64 y2 = y1 + (u64)(((long long)(int)yh * e1) >> 40);
    return Recip{(u32)(y2 >> 32), (u32)y2};
}

// whether twice the remainder n 2^k - q mb exceeds mb (modulo 2^64; nl: the low 64 bits of n 2^k)
IP_RARE u32 round_by_remainder(u64 nl, u32 qh, u32 ql, u32 mbh, u32 mbl) {
    const u64 pr = wide(ql, mbl) + ((u64)(ql * mbh + qh * mbl) << 32);
    return 2 * (nl - pr) > (((u64)mbh << 32) | mbl) ? 0xffffffffu : 0u;
}

// 1/b, b in range, y = recip_of(b)
IP_FN double rcp_core(double b, const Recip& y) {
    const u32 ql = shr2(y.yl, y.yh, 10), qh = y.yh >> 10;
    u32 z = y.yl << 22;  // ten guard bits, y's error as recip_of says
    if (__builtin_expect(z - (0x80000000u - (2u << 22)) <= (5u << 22), 0))
        z = round_by_remainder(0ull, qh, ql, mant_hi(b), lo(b));
    return round_pack(qh, ql, z, ((2044u << 20) - (hi(b) & 0x7ff00000u)) + (hi(b) & 0x80000000u));
}

// a/b, both in range, y = recip_of(b)
IP_FN double quot_core(double a, double b, const Recip& y) {
    const u32 Ah = shl2(lo(a), mant_hi(a), 11), Al = lo(a) << 11;  // Q63
    const u64 T = wide(Ah, y.yh) + (u32)(wide(Ah, y.yl) >> 32) + (u32)(wide(Al, y.yh) >> 32);  // Q62, in (2^61, 2^63)
    const u32 Th = (u32)(T >> 32), Tl = (u32)T;
    const u32 s = Th >> 30, sh = 9 + s;
    const u32 ql = shr2(Tl, Th, sh), qh = Th >> sh;
    u32 z = shr2(0u, Tl, sh);  // nine or ten guard bits; T within 5 units: y's 2, three products rounded down
    if (__builtin_expect(z - (0x80000000u - (5u << 23)) <= (10u << 23), 0))
        z = round_by_remainder((((u64)mant_hi(a) << 32) | lo(a)) << (53 - s), qh, ql, mant_hi(b), lo(b));
    const u32 E = (hi(a) & 0x7ff00000u) - (hi(b) & 0x7ff00000u) + ((1021u + s) << 20);
    return round_pack(qh, ql, z, E + ((hi(a) ^ hi(b)) & 0x80000000u));
}

IP_RARE double quot_rare(double a, double b) {
    const u32 xa = hi(a) & 0x7fffffffu, xb = hi(b) & 0x7fffffffu;
    if ((xa | lo(a)) == 0 && xb < 0x7ff00000u && (xb | lo(b)) != 0)  // 0 / b
        return make((hi(a) ^ hi(b)) & 0x80000000u, 0u);
    return a / b;
}
IP_RARE double rcp_rare(double b) { return 1.0 / b; }

IP_FN double rcp(double b) {
    if (__builtin_expect(in_range(b), 1)) return rcp_core(b, recip_of(b));
    return rcp_rare(b);
}
IP_FN double quot(double a, double b) {
    if (__builtin_expect(in_range(a) && in_range(b), 1)) return quot_core(a, b, recip_of(b));
    return quot_rare(a, b);
}
// N quotients by one divisor
template <int N>
IP_FN void quotn(double* r, const double* a, double b) {
    bool ok = in_range(b);
#pragma unroll
    for (int k = 0; k < N; k++) ok = ok && in_range(a[k]);
    if (__builtin_expect(ok, 1)) {
        const Recip y = recip_of(b);
#pragma unroll
        for (int k = 0; k < N; k++) r[k] = quot_core(a[k], b, y);
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) r[k] = quot(a[k], b);
    }
}

// square root of a positive x in range: m = x / 2^(2k) in [1, 4), a binary32 seed y of
// 1/sqrt(m), one Newton step (2^-44), s = m y, and s + (m - s^2) y / 2 from the exact
// remainder (2^-60); the last bit as for the quotient.
IP_RARE u32 round_by_square(u64 xl, u32 qh, u32 ql) {
    const u64 R = xl - (wide(ql, ql) + ((u64)(2 * ql * qh) << 32));  // x 2^j - q^2, below 2 q + 1
    return R > (((u64)qh << 32) | ql) ? 0xffffffffu : 0u;
}
IP_FN double sqrt_core(double x) {
    const u32 odd = (~hi(x) >> 20) & 1u;  // the exponent without its bias is odd
    const u32 mh = mant_hi(x), ml = lo(x);
    const u32 Mh = shl2(ml, mh, 10 + odd), Ml = ml << (10 + odd);  // Q62
    const u32 y0r = f2u(rsqrt_seed(u2f_bits(((mh << 3) & 0x7fffffu) | (ml >> 29) | ((65u + odd) << 23))));
    const u32 y0 = y0r < 0x7fffffffu ? y0r : 0x7fffffffu;          // Q31, in (2^30, 2^31)
    const u64 yy = wide(y0, y0);                                    // Q62
    const u32 yyh = (u32)(yy >> 32), yyl = (u32)yy;
    const u64 p = wide(Mh, yyh) + (u32)(wide(Mh, yyl) >> 32) + (u32)(wide(Ml, yyh) >> 32);  // Q60
    const int e0 = (int)((long long)((1ull << 60) - p) >> 9);      // Q51
    const u64 y1 = ((u64)y0 << 32) + (u64)(((long long)(int)y0 * e0) >> 20);  // Q63: y0 (1 + e0/2)
    const u32 yh = (u32)(y1 >> 32), yl = (u32)y1;
    const u64 s1 = wide(Mh, yh) + (u32)(wide(Mh, yl) >> 32) + (u32)(wide(Ml, yh) >> 32);    // Q61
    const u32 sh = (u32)(s1 >> 32), sl = (u32)s1;
    const u64 sq = ((u64)(sh * sh) << 32) + 2 * wide(sh, sl) + (u32)(wide(sl, sl) >> 32);   // Q90, modulo 2^64
    const u64 M28 = ((u64)shl2(Ml, Mh, 28) << 32) | (Ml << 28);
    const int r = (int)((long long)(M28 - sq) >> 20);              // Q70
    const u64 s2 = s1 + (u64)(((long long)(int)yh * r) >> 41);     // r y / 2
    const u32 Sh = (u32)(s2 >> 32), Sl = (u32)s2;
    const u32 ql = shr2(Sl, Sh, 9), qh = Sh >> 9;
    u32 z = Sl << 23;  // nine guard bits
    if (__builtin_expect(z - (0x80000000u - (4u << 23)) <= (8u << 23), 0))
        z = round_by_square((((u64)mh << 32) | ml) << (52 + odd), qh, ql);
    return round_pack(qh, ql, z, ((((hi(x) >> 20) + 1021u) >> 1) << 20));
}
IP_RARE double sqrt_rare(double x) { return ::sqrt(x); }
IP_FN double sqrt(double x) {
    // positive and in range: the sign bit would put hi(x) above the range
    if (__builtin_expect(hi(x) - 0x20100000u < 0x3fc00000u, 1)) return sqrt_core(x);
    return sqrt_rare(x);
}

// ---- x^a

// 64 intervals of the significand m: c = kLogC / 1024 >= 1/m at the interval's left end, so
// that r = m c - 1 is exact and 0 <= r < 2^-5; kLogT = -log2(c), Q62; kExpT = 2^(i/64), Q63.
#if defined(__CUDA_ARCH__)
#define IP_TABLE static __device__ const
#else
#define IP_TABLE static const
#endif
IP_TABLE unsigned short kLogC[64] = {
    1024, 1009, 993, 979, 964, 950, 937, 924, 911, 898, 886, 874, 863, 852, 841, 830,
    820, 810, 800, 790, 781, 772, 763, 754, 745, 737, 729, 721, 713, 705, 698, 690,
    683, 676, 669, 662, 656, 649, 643, 637, 631, 625, 619, 613, 607, 602, 596, 591,
    586, 580, 575, 570, 565, 561, 556, 551, 547, 542, 538, 533, 529, 525, 521, 517};
IP_TABLE u64 kLogT[64] = {
    0x0000000000000000ull, 0x015ccece78a4a9e2ull, 0x02d6a1c52f5f99c0ull, 0x0426417de5c11ef5ull,
    0x0593389b019c55adull, 0x06ed040be494e4f1ull, 0x0832b45fc2bb59adull, 0x097cf196adfee84dull,
    0x0acbdcb3bc4e88faull, 0x0c1f98266e2d535cull, 0x0d5d9654f63a3931ull, 0x0e9feaa1d256ae3dull,
    0x0fcb4bf9de86679dull, 0x10fa848044b35108ull, 0x122dadc2ab3496d2ull, 0x1364e2511cc820cfull,
    0x148365e695d796aaull, 0x15a56d7a370ded62ull, 0x16cb0f6865c8ea03ull, 0x17f462e58e168828ull,
    0x1903372e90bee3f2ull, 0x1a152f142981b3d7ull, 0x1b2a5d6f51ff82b2ull, 0x1c42d5c4c688b3cfull,
    0x1d5eac4d463d7de1ull, 0x1e5dddf7e46e0a54ull, 0x1f5fd8a9063e3490ull, 0x2064ac1d23cb3bc1ull,
    0x216c68978eb5cdfaull, 0x22771ee8884eb752ull, 0x2362fd0935b84c2cull, 0x2473772407798668ull,
    0x25647ca36738f606ull, 0x2657fdc6e1dcd0cbull, 0x274e07ca1f49be5aull, 0x2846a853ae553ba8ull,
    0x291dde3262f321a8ull, 0x2a1b72da09d5469aull, 0x2af6fd70071f5e6cull, 0x2bd496ee30ab9accull,
    0x2cb4494dab9de792ull, 0x2d961ed0cb91d406ull, 0x2e7a2205e5813045ull, 0x2f605dca45dfdfb6ull,
    0x3048dd4d4c00d553ull, 0x310c600e275bf88full, 0x31f92499135908dfull, 0x32c04702422a3142ull,
    0x33891a8be56a4a25ull, 0x347c5e95887ec06bull, 0x35490566b9539d52ull, 0x361775c932bace07ull,
    0x36e7b7cd16b43760ull, 0x378fa7d29bdb897aull, 0x386344fba0169378ull, 0x3938cb84d4664657ull,
    0x39e503e2be17ce3aull, 0x3abe11f27f31124aull, 0x3b6d29207b2970ddull, 0x3c49dd15d3e18a0eull,
    0x3cfbebfca715669dull, 0x3daf54df46b1e14eull, 0x3e641d088b6533daull, 0x3f1a49e2a175d53aull};
IP_TABLE u64 kExpT[64] = {
    0x8000000000000000ull, 0x8164d1f3bc030773ull, 0x82cd8698ac2ba1d7ull, 0x843a28c3acde4046ull,
    0x85aac367cc487b14ull, 0x871f61969e8d1010ull, 0x88980e8092da8527ull, 0x8a14d575496efd9aull,
    0x8b95c1e3ea8bd6e6ull, 0x8d1adf5b7e5ba9e5ull, 0x8ea4398b45cd53c0ull, 0x9031dc431466b1dcull,
    0x91c3d373ab11c336ull, 0x935a2b2f13e6e92bull, 0x94f4efa8fef70961ull, 0x96942d3720185a00ull,
    0x9837f0518db8a96full, 0x99e0459320b7fa64ull, 0x9b8d39b9d54e5538ull, 0x9d3ed9a72cffb750ull,
    0x9ef5326091a111adull, 0xa0b0510fb9714fc2ull, 0xa27043030c496818ull, 0xa43515ae09e6809eull,
    0xa5fed6a9b15138eaull, 0xa7cd93b4e9653569ull, 0xa9a15ab4ea7c0ef8ull, 0xab7a39b5a93ed337ull,
    0xad583eea42a14ac6ull, 0xaf3b78ad690a4374ull, 0xb123f581d2ac258full, 0xb311c412a9112489ull,
    0xb504f333f9de6484ull, 0xb6fd91e328d17791ull, 0xb8fbaf4762fb9ee9ull, 0xbaff5ab2133e45fbull,
    0xbd08a39f580c36beull, 0xbf1799b67a731082ull, 0xc12c4cca66709456ull, 0xc346ccda24976407ull,
    0xc5672a115506daddull, 0xc78d74c8abb9b15cull, 0xc9b9bd866e2f27a2ull, 0xcbec14fef2727c5cull,
    0xce248c151f8480e3ull, 0xd06333daef2b2594ull, 0xd2a81d91f12ae45aull, 0xd4f35aabcfedfa1full,
    0xd744fccad69d6af4ull, 0xd99d15c278afd7b5ull, 0xdbfbb797daf23755ull, 0xde60f4825e0e9123ull,
    0xe0ccdeec2a94e111ull, 0xe33f8972be8a5a51ull, 0xe5b906e77c8348a8ull, 0xe8396a503c4bdc68ull,
    0xeac0c6e7dd24392eull, 0xed4f301ed9942b84ull, 0xefe4b99bdcdaf5cbull, 0xf281773c59ffb139ull,
    0xf5257d152486cc2cull, 0xf7d0df730ad13bb8ull, 0xfa83b2db722a033aull, 0xfd3e0c0cf486c174ull};
#undef IP_TABLE

// high 64 bits of a b, at most 3 too small
IP_FN u64 mulhi(u64 a, u64 b) {
    const u32 ah = (u32)(a >> 32), al = (u32)a, bh = (u32)(b >> 32), bl = (u32)b;
    return wide(ah, bh) + (u32)(wide(ah, bl) >> 32) + (u32)(wide(al, bh) >> 32);
}
IP_FN u32 mulhi32(u32 a, u32 b) { return (u32)(wide(a, b) >> 32); }

// x^a for 2^-120 <= x < 2^120, 2^-9 <= a < 4 (in [2^-480, 2^480] as a result), within 0.54
// units in the last place (0.532 the largest of 3 million samples per binade of a): log2 and
// exp2 by tables of 64 entries and polynomials (the scheme of Tang, ACM TOMS 15 (1989) and 16
// (1990)) in fixed point, the products of the high terms in 32 bits. The coefficients are Taylor's.
IP_FN double pow_core(double x, double a) {
    // a in Q61, exactly: its significand's lowest bit is Q62's tenth
    const u32 ea = hi(a) >> 20;  // 1014 .. 1024
    const u64 am = ((u64)shl2(lo(a), mant_hi(a), 10) << 32) | (lo(a) << 10);  // Q62 of [1, 2)
    const u64 A = am >> (1024u - ea);                                           // Q61: a = am 2^(ea-1023-62)
    // log2(x) = e + F, F in Q62
    const u32 xh = hi(x), i = (xh >> 14) & 63u, c = kLogC[i];
    const u64 m0 = wide(lo(x), c);
    const u64 m1 = wide(mant_hi(x), c) + (u32)(m0 >> 32);
    const u64 R = ((m1 << 32) | (u32)m0) - (1ull << 62);  // r, Q62
    const u64 rs = R << 6;                                  // Q68
    const u32 rh = (u32)(rs >> 32);                         // Q36
    u32 p = 2626u;                                     // Q14
    p = 47274u - mulhi32(p, rh);                       // Q18
    p = 864443u - mulhi32(p, rh);
    p = 16136271u - mulhi32(p, rh);
    p = 309816401u - mulhi32(p, rh);                   // Q30
    u64 P = 0x000171547652b830ull - (wide(p, rh) >> 16);   // Q50
    P = 0x001ec709dc3a03fdull - mulhi(P, rs);
    P = 0x02e2a8eca5705fc3ull - mulhi(P, rs);
    P = 0x5c551d94ae0bf85eull - mulhi(P, rs);              // Q62
    const u64 F = kLogT[i] + (mulhi(P, rs) >> 4);
    // y = a (e + F), Q61: a (e + 512) - 512 a + a F over 96 bits
    const u32 eb = (xh >> 20) - 511u;
    const u64 y0 = wide((u32)A, eb), aF = mulhi(A, F) << 2;
    const u64 ylo = (u64)(u32)y0 + (u32)aF;                       // low word of a (e + 512) + a F
    u64 yh = wide((u32)(A >> 32), eb) + (u32)(y0 >> 32) + (u32)(aF >> 32) + (u32)(ylo >> 32);
    u64 yl = (u32)ylo;
    const u64 sub = A << 9;                                        // 512 a modulo 2^64; its top: A >> 55
    const u64 l2 = yl - (u32)sub;
    yh = yh - ((A >> 23) + ((l2 >> 32) & 1u));
    yl = (u32)l2;
    // 2^y: y = k + i/64 + s
    const int k = (int)((long long)yh >> 29);
    const u64 fr = ((yh << 35) | (yl << 3));                       // Q64
    const u32 j = (u32)(fr >> 58);
    const u64 s = fr << 6;                                          // Q70
    const u32 sh = (u32)(s >> 32);
    u32 q = 4094u;                                     // Q28
    q = 2646306u + mulhi32(q, sh);
    q = 1466040222u + mulhi32(q, sh);                   // Q40
    u64 Q = 0x0000009d955b7dd2ull + mulhi32(q, sh);        // Q46
    Q = 0x0000e35846b82506ull + mulhi(Q, s);
    Q = 0x00f5fdeffc162c75ull + mulhi(Q, s);
    Q = 0xb17217f7d1cf79acull + mulhi(Q, s);               // Q64
    const u64 T = kExpT[j];
    const u64 E = T + (mulhi(T, mulhi(Q, s)) >> 6);                // Q63
    const u32 Eh = (u32)(E >> 32), El = (u32)E;
    const u32 ql = shr2(El, Eh, 11);
    return round_pack(Eh >> 11, ql, (El << 21) | (ql & 1u), (u32)(k + 1022) << 20);
}
IP_RARE double pow_rare(double x, double a) { return ::exp(::log(x) * a); }
// x^a; what the fixed-point form does not take goes through exp and log. A smaller exponent (a gas
// with gamma < 1.004) would lose its last bits in Q61 (up to 0.80 units, exp and log 0.50 to 0.71);
// from 2^-9 on exp and log are the less exact (0.85 units, 30 at a = 1/4).
IP_FN double pow(double x, double a) {
    // 2^-120 <= x < 2^120, 2^-9 <= a < 4
    if (__builtin_expect(hi(x) - 0x38700000u < 0x0f000000u && hi(a) - 0x3f600000u < 0x00b00000u, 1)) return pow_core(x, a);
    return pow_rare(x, a);
}

// a < b and x >= 0 (false for NaN) without an FP64 comparison
#if defined(__CUDA_ARCH__)
static __device__ __noinline__ bool less_rare(double a, double b) { return a < b; }
#else
static inline bool less_rare(double a, double b) { return a < b; }
#endif
IP_FN bool less(double a, double b) {
    // the bits of a negative number inverted below its sign: ordered as integers
    const u32 na = (u32)((int)hi(a) >> 31), nb = (u32)((int)hi(b) >> 31);
    const int ah = (int)(hi(a) ^ (na >> 1)), bh = (int)(hi(b) ^ (nb >> 1));
    if (__builtin_expect(in_range(a) && in_range(b), 1)) return ah < bh || (ah == bh && (lo(a) ^ na) < (lo(b) ^ nb));
    return less_rare(a, b);
}
IP_FN bool positive(double x) {  // 0 < x
    const long long b = (long long)(((u64)hi(x) << 32) | lo(x));
    return b > 0 && b <= 0x7ff0000000000000ll;
}
IP_FN bool not_negative(double x) {  // 0 <= x, -0 too
    const u64 b = ((u64)hi(x) << 32) | lo(x);
    return b <= 0x7ff0000000000000ull || b == 0x8000000000000000ull;
}
IP_FN bool zero(double x) { return ((hi(x) << 1) | lo(x)) == 0; }
// x / 2: exact for normal results and zeros, by the exponent
IP_FN double half(double x) {
    const u32 xa = hi(x) & 0x7fffffffu;
    if (__builtin_expect(xa - 0x00200000u < 0x7fd00000u, 1)) return make(hi(x) - 0x00100000u, lo(x));
    return (xa | lo(x)) == 0 ? x : mul_rare(x, 0.5);
}
// 0 + x: x, with -0 turned into +0
IP_FN double plus_zero(double x) { return make((hi(x) == 0x80000000u && lo(x) == 0) ? 0u : hi(x), lo(x)); }
// a/b with y = recip_of(b)
IP_FN double quot_by(double a, double b, const Recip& y) {
    if (__builtin_expect(in_range(a) && in_range(b), 1)) return quot_core(a, b, y);
    return quot_rare(a, b);
}

#if defined(__CUDACC__)
// 1.0 in a register the compiler cannot see through. A fused multiply-add of three registers
// takes 17 clocks of the FP64 unit per warp, an addition, a product, or a multiply-add with an
// operand from the constant bank, a uniform register or an immediate 20 (measured, one SM, all
// warps resident). a + b is therefore formed as a * one + b: the same rounding of the same sum.
__device__ __forceinline__ double one() {
#if defined(__CUDA_ARCH__)
    u32 h;
    asm("{\n\t.reg .u32 m;\n\tmov.u32 m, %%lanemask_eq;\n\tpopc.b32 m, m;\n\tadd.u32 %0, m, 0x3fefffff;\n\t}" : "=r"(h));
    return make(h, 0u);
#else
    return 1.0;
#endif
}
// a constant in a register of its own, for the same reason
__device__ __forceinline__ double reg(double x) {
#if defined(__CUDA_ARCH__)
    u32 z;
    asm("{\n\t.reg .u32 m;\n\tmov.u32 m, %%lanemask_eq;\n\tpopc.b32 m, m;\n\tsub.u32 %0, m, 1;\n\t}" : "=r"(z));
    return make(hi(x) + z, lo(x) + z);
#else
    return x;
#endif
}
__device__ __forceinline__ double fadd(double a, double b) { return __fma_rn(a, one(), b); }
__device__ __forceinline__ double fsub(double a, double b) { return __fma_rn(a, one(), neg(b)); }

// A binary64 number whose products, quotients and square roots are formed on the integer
// pipes and whose sums run on the FP64 unit as multiply-adds: the two sides of a kernel then
// overlap. Bit for bit the arithmetic of double.
struct xd {
    double v;
    xd() = default;
    __device__ __forceinline__ explicit xd(double x) : v(x) {}
    __device__ __forceinline__ explicit operator double() const { return v; }
};
__device__ __forceinline__ xd operator+(xd a, xd b) { return xd(fadd(a.v, b.v)); }
__device__ __forceinline__ xd operator-(xd a, xd b) { return xd(fsub(a.v, b.v)); }
__device__ __forceinline__ xd operator-(xd a) { return xd(neg(a.v)); }
__device__ __forceinline__ xd operator*(xd a, xd b) { return xd(mul(a.v, b.v)); }
__device__ __forceinline__ xd operator/(xd a, xd b) { return xd(quot(a.v, b.v)); }
__device__ __forceinline__ xd& operator+=(xd& a, xd b) { a = a + b; return a; }
__device__ __forceinline__ xd& operator-=(xd& a, xd b) { a = a - b; return a; }
__device__ __forceinline__ bool operator>(xd a, xd b) { return a.v > b.v; }
__device__ __forceinline__ bool operator<(xd a, xd b) { return a.v < b.v; }
__device__ __forceinline__ bool operator>=(xd a, xd b) { return a.v >= b.v; }
__device__ __forceinline__ bool operator<=(xd a, xd b) { return a.v <= b.v; }
#endif

}  // namespace ip
}  // namespace cfd2d
