// exp2_fixed.cuh -- 2^-y of a fixed-point argument in integer arithmetic.
//
// FP64 runs at 1/64 of the FP32 rate on this part, and its exponential takes 16
// of its instructions: 305 SM cycles per warp. The integer pipe takes about 30:
// 2^-y = 2^-n T[j] p(v) with y = n + j / 256 + v / 256, n integer, 0 <= v < 1,
// T[j] = 2^(-j / 256) from a table and p the Taylor polynomial of degree 5
// of 2^(-v / 256) by Horner, each step in as many bits as its weight asks for.
// The result carries an error below 2^-59 of it before it is rounded to a
// double (worst of 20000 random arguments against 60 digits: 5.5 x 2^-62), so
// the double is within 0.52 ulp; CUDA's exp() is within 1 ulp.
#pragma once
#include <math.h>
#include <stdint.h>

// 2^63 2^(-i / 16) and 2^63 2^(-i / 256), i < 16, rounded to nearest
__device__ const unsigned long long EXP2_T1[16] = {
    0x8000000000000000ULL, 0x7a92be8a92436616ULL, 0x75606373ee921c97ULL, 0x70666f76154a7089ULL,
    0x6ba27e656b4eb57aULL, 0x6712460a8fc24072ULL, 0x62b39508aa836d6fULL, 0x5e8451cfac061b5fULL,
    0x5a827999fcef3242ULL, 0x56ac1f752150a563ULL, 0x52ff6b54d8a89c75ULL, 0x4f7a993048d088d7ULL,
    0x4c1bf828c6dc54b8ULL, 0x48e1e9b9d588e19bULL, 0x45cae0f1f545eb73ULL, 0x42d561b3e6243d8aULL};
__device__ const unsigned long long EXP2_T2[16] = {
    0x8000000000000000ULL, 0x7fa765aca88f6453ULL, 0x7f4f08ae3dc7c426ULL, 0x7ef6e8da4b544f9aULL,
    0x7e9f06067a4360baULL, 0x7e47600890f223deULL, 0x7deff6b672f84e24ULL, 0x7d98c9e62113e1faULL,
    0x7d41d96db915019dULL, 0x7ceb252375c9cf9bULL, 0x7c94acddaeea5d3aULL, 0x7c3e7072d904a6ceULL,
    0x7be86fb985689ddcULL, 0x7b92aa886214411cULL, 0x7b3d20b6399fc237ULL, 0x7ae7d219f329b948ULL};

// Entry j < 256 of the table: 2^63 2^(-j / 256).
__device__ __forceinline__ unsigned long long exp2_table_entry(int j) {
    return __umul64hi(EXP2_T1[j >> 4], EXP2_T2[j & 15]) << 1;
}

// The high half of a 64-bit product, at most 2 low (the low halves' product and
// the cross products' carries are left out).
__device__ __forceinline__ unsigned long long umul64hi_low2(unsigned long long a, unsigned long long b) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    return (unsigned long long)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

// 2^-y as a double, y in units of 2^-fb, |y| < 2^62; T: the table. FB = 56: fb
// is that (and 2^-y a normal number); FB = 0: 32 <= fb <= 56, results below
// 2^-1021 become 0 and those above 2^1020 infinite.
template <int FB>
__device__ __forceinline__ double exp2_fixed(long long y, int fb, const unsigned long long *T) {
    if (FB) fb = FB;
    const int n = (int)(y >> fb);
    const unsigned long long f = (unsigned long long)y << (64 - fb);
    const unsigned long long v = f << 8;
    const uint32_t vh = (uint32_t)(v >> 32);
    // c_k = (ln 2 / 256)^k / k! in units of 2^-70, 2^-70, 2^-60, 2^-80, 2^-72
    const uint32_t t4 = 2643811198u - __umulhi(vh, 1431680u);
    const uint32_t t3 = 3814213304u - (__umulhi(vh, t4) >> 10);
    const unsigned long long t2 = 0x3d7f7bff058b1d51ULL - (((unsigned long long)vh * t3) >> 12);
    const unsigned long long t1 = 0xb17217f7d1cf79acULL - (umul64hi_low2(v, t2) >> 8);
    const unsigned long long e = (1ULL << 63) - (umul64hi_low2(v, t1) >> 9);
    const unsigned long long m = umul64hi_low2(e, T[f >> 56]);  // in (2^61, 2^62]: units of 2^-62
    long long bits = ((long long)(1022 - n) << 52) + (long long)((m - (1ULL << 61) + 256) >> 9);
    if (!FB) {
        if (n > 1020) bits = 0;
        if (n < -1020) bits = 0x7ff0000000000000LL;
    }
    return __longlong_as_double(bits);
}

// log2(e) gamma q in units of 2^-fb: |q| = M 2^(E - 1075), times cg 2^-ec.
__device__ __forceinline__ long long fixed_scaled(double q, unsigned long long cg, int ec, int fb) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(q);
    const int E = (int)((b >> 52) & 0x7ff);
    long long v = 0;
    if (E != 0) {
        const unsigned long long M = ((b & ((1ULL << 52) - 1)) | (1ULL << 52)) << 11;  // q = M 2^(E - 1086)
        const unsigned long long h = __umul64hi(M, cg);                               // M cg 2^-64
        const int sh = -(E - 1086 + 64 - ec + fb);                                    // value = h 2^-sh
        if (sh <= 0) v = (long long)(h << min(-sh, 1));  // (bounded by the choice of fb: not reached)
        else if (sh < 64) v = (long long)((h >> (sh - 1)) + 1 >> 1);
        if (b >> 63) v = -v;
    }
    return v;
}

// gamma log2(e) = g 2^-e with g in [2^62, 2^63): the 53-bit mantissa of gamma
// times log2(e) 2^62, exactly.
inline void scaled_gamma(double gamma, unsigned long long *g, int *e) {
    int x;
    const double m = frexp(gamma, &x);  // gamma = m 2^x, m in [0.5, 1)
    unsigned __int128 p = (unsigned __int128)(unsigned long long)(m * 9007199254740992.0) * 0x5c551d94ae0bf85eULL;
    int s = 0;  // gamma log2(e) = p 2^(x - 53 - 62)
    while ((p >> s) >> 63) ++s;
    *g = (unsigned long long)(p >> s);
    *e = 115 - x - s;
}
