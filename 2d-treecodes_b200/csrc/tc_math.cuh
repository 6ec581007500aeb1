// tc_math.cuh -- binomial table and small complex helpers shared by the expansion kernels.
#pragma once

#include "tc_common.cuh"
#include "tc_log_table.cuh"
#include "tc_near_log_table.cuh"

namespace tc {

constexpr int BINOM_N = 2 * MAX_ORDER;

// Pascal's triangle in double, exact in every entry used: C(l+k-1, k-1) up to C(47,23) ~ 1.6e13 in
// translations of order 24, C(55,27) ~ 3.8e15 in those of order 28, and in a potential's common far
// fields C(l+k-1, k-1), l <= 31, k <= 28; those above 2^53 (up to C(58,27) ~ 2.6e16) have enough factors
// of two (tests/test_binomials.py).
// The reference bakes the same integers into its kernels through kernels/binomial.py:1-5.
struct BinomTable {
    double c[BINOM_N][BINOM_N];
};

constexpr BinomTable make_binom_table() {
    BinomTable t{};
    for (int n = 0; n < BINOM_N; ++n) {
        t.c[n][0] = 1.0;
        for (int k = 1; k <= n; ++k) t.c[n][k] = t.c[n - 1][k - 1] + (k < n ? t.c[n - 1][k] : 0.0);
    }
    return t;
}

// Natural logarithm of a positive normal double, for the potential kernels' log r^2 terms
// (arguments r^2 + 10 eps or |z|^2 of a far cell, never zero, subnormal or infinite).
// Table-driven, after Tang's method (P. T. P. Tang, ACM TOMS 16(4), 1990): x = 2^e m with m in
// [sqrt(1/2), sqrt(2)); c = the single-precision reciprocal of m (from its top 20 fraction bits)
// rounded to 10 significant bits, so that r = m c - 1 is exact in one fma (m c has at most 62
// significant bits and |r| <= 2^-10 (1 + 2^-7)); log x = e ln 2 - log c + log1p(r), log1p(r) =
// r + r^2 q(r) with q of degree 3.  -log c comes from a table of LOG_NTAB doubles indexed by the
// rounded float bits of c, which the caller keeps in shared memory (load_log_table); m is in
// [sqrt(1/2), sqrt(2)) by construction, which puts the index in [20, 532] for any x.  The last
// step, e ln 2 + (-log c + log1p r), rounds twice: for e = 0 only the sum, and for e != 0 the
// result is at least ln 2 / 2 in size, so ln 2's own rounding (2^-55) stays below half an ulp of
// it.  fit_log_table.py beside this file writes the table and q (tc_log_table.cuh).  8 FP64
// operations, one single-precision reciprocal, one conversion and one shared load, against the
// library log's ~100 instructions; within 2 ulp of the exact logarithm (tests/test_gpu_parity.py
// checks 4 ulp against the library log on 2^20 arguments).
__device__ __forceinline__ double log_pos(double x, const double *__restrict__ neg_log_c) {
    const int ix = __double2hiint(x) - 0x3fe6a09f;   // high word of sqrt(1/2), rounded up
    const int e = ix >> 20;
    const int mf = ix & 0x000fffff;                 // fraction bits of m, offset
    const double m = __hiloint2double(mf + 0x3fe6a09f, __double2loint(x));
    const float mfl = __int_as_float((mf << 3) + (0x07e6a09f << 3));   // m to 20 bits, as float
    float rc;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc) : "f"(mfl));
    // round the reciprocal to 10 significant bits: key = its float bits >> LOG_KEY_SHIFT
    const unsigned key = (__float_as_uint(rc) + (1u << (LOG_KEY_SHIFT - 1))) >> LOG_KEY_SHIFT;
    const double c = __hiloint2double((int)(key << (LOG_KEY_SHIFT - 3)) + (896 << 20), 0);
    const double r = fma(m, c, -1.0);
    double q = LOG_Q3;
    q = fma(q, r, LOG_Q2);
    q = fma(q, r, LOG_Q1);
    q = fma(q, r, LOG_Q0);
    const double p = fma(r * r, q, r);
    constexpr double LN2 = 0x1.62e42fefa39efp-1;
    return fma((double)e, LN2, neg_log_c[(int)key - LOG_IDX_BASE] + p);
}

// Copies log_pos's table into the block's shared memory; every thread of the block calls it.
__device__ __forceinline__ void load_log_table(double *s_neg_log_c) {
    for (int i = threadIdx.x; i < LOG_NTAB; i += blockDim.x) s_neg_log_c[i] = LOG_NEG_LOG_C[i];
    __syncthreads();
}

// The logarithm of the FP64 potential evaluation: as log_pos, with the reduction's reciprocal c
// read from the table beside -log c instead of formed by the approximate-reciprocal unit, and
// the polynomial nested onto the table value: 7 FP64 operations, one conversion, 6 integer ones
// and one 16-byte shared load, against log_pos's 8, one, 9, a reciprocal and an 8-byte load.  (An
// FP64 instruction takes two issue slots, so both kinds count.)  The table stands in shared
// memory NLOG_COPIES times, copy k of entry i at 8 i + k, and a lane reads copy lane % 8: the eight
// lanes that a 16-byte shared load serves at once then never meet in a bank.
// fit_near_log_table.py beside this file writes the table.  Any x from 2^-1022 up to 2^NLOG_TOP: c's
// exponent field (1022 or 1023) less x's exponent stays that of a normal number, and from 2^1022 on it
// would not.  Within 2 ulp of the exact logarithm (tests/test_near_log_table.py,
// tests/test_potential_reach.py).
constexpr int NLOG_COPIES = 8;
constexpr int NLOG_TOP = 1020;   // (2 NEAR_REACH^2 is below it)

// `tab`: the table's 32-bit shared-memory address; `copy`: the lane's copy, 16 (lane % 8).
__device__ __forceinline__ unsigned shared_address(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

// (in the constant bank: as literals they were moved into uniform registers again for every source)
static __constant__ double c_nlog[5] = {NLOG_Q0, NLOG_Q1, NLOG_Q2, NLOG_Q3, 0x1.62e42fefa39efp-1};

__device__ __forceinline__ double log_near(double x, unsigned tab, int copy) {
    const int ix = __double2hiint(x) - NLOG_BASE;
    const int e = ix >> 20;
    // entry (ix >> (20 - NLOG_BITS)) mod NLOG_NTAB, NLOG_COPIES * 16 bytes each
    constexpr int SHIFT = 20 - NLOG_BITS - 7;
    static_assert(NLOG_COPIES * sizeof(double2) == 128, "entry stride 2^7 bytes");
    const int off = ((ix >> SHIFT) & ((NLOG_NTAB - 1) << 7)) | copy;
    double c, t0;   // (not volatile: the table does not change while it is read)
    asm("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(c), "=d"(t0) : "r"(tab + off));
    // r = m c - 1 = x (c 2^-e) - 1: c's exponent takes the scaling (c is in [0.7, 1.42))
    c = __hiloint2double(__double2hiint(c) - (ix & (int)0xfff00000), __double2loint(c));
    const double r = fma(x, c, -1.0);
    double t = fma(c_nlog[3], r, c_nlog[2]);
    t = fma(t, r, c_nlog[1]);
    t = fma(t, r, c_nlog[0]);
    t = fma(t, r, 1.0);
    return fma((double)e, c_nlog[4], fma(t, r, t0));
}

// Fills the block's copies of log_near's table; every thread of the block calls it.
__device__ __forceinline__ void load_near_log_table(double2 *s_tab) {
    for (int i = threadIdx.x; i < NLOG_NTAB * NLOG_COPIES; i += blockDim.x)
        s_tab[i] = NLOG_TAB[i / NLOG_COPIES];
    __syncthreads();
}

struct cplx {
    double re, im;
};

__device__ __forceinline__ cplx cmul(cplx a, cplx b) {
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

// a * b + c
__device__ __forceinline__ cplx cfma(cplx a, cplx b, cplx c) {
    return {fma(a.re, b.re, fma(-a.im, b.im, c.re)), fma(a.re, b.im, fma(a.im, b.re, c.im))};
}

// z^e for 0 <= e < 32 by square-and-multiply
__device__ __forceinline__ cplx cpow_int(cplx z, int e) {
    cplx r = {1.0, 0.0};
    cplx b = z;
#pragma unroll
    for (int bit = 0; bit < 5; ++bit) {
        if (e & (1 << bit)) r = cmul(r, b);
        b = cmul(b, b);
    }
    return r;
}

}  // namespace tc
