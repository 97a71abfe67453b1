// fixed_recon.cuh -- the fast first pass's GP reconstruction in fixed point.
//
// A cell's face states (left/right/bottom/top faces at 2 or 3 Gauss points) are
// constant-weight sums over its 13-point (order 5) or 5-point (order 3) stencil.  On this part an SM issues
// an FP64 instruction every 16-19 cycles but two integer instructions per
// cycle beside it (measured: eight 32x32+64-bit multiply-adds next to every
// FP64 FMA cost nothing), and the first pass is bound by the FP64 pipe, so the
// sums run on the integer pipe and FP64 is left to the Riemann solves.  Radius 1
// (order 3, 5 points) uses the same form.
//
// Per variable and stencil the values are aligned to one exponent E by what
// they weigh: a group of mirror images (fix_group) whose weights are below 2^-k
// takes part in E, the largest biased exponent, with e - k, and its weights are
// stored times 2^k.  A double M * 2^(e-1075) becomes Q = M << 5 >> (E + k - e), a
// 58-bit integer.  The mirror-symmetry components (GpOrbit) are exact integer
// sums of up to four Q (60 bits).  A weight is w * 2^(58+k), at most 1, rounded to
// an integer.  Both factors are split as h * 2^30 + l, |l| <= 2^29, and a product
// keeps h*h (accumulated on its own) and h*l + l*h (accumulated together); l*l, at
// most one unit of Q, is dropped.  With sum |w| 2^k <= 15 over a state's cells
// (the host picks k so; sum |w| <= 4 is checked, FixOrbit::ok) neither
// accumulator passes 2^62 and no result 2^62.  The 64-bit results, in units of
// 2^(E-1080), are rounded to double once.  Error: a unit per cell for its
// alignment and its dropped product, and the final rounding, against one FP64
// rounding per multiply-add before: RMS 0.35 to 0.8 of FP64's wherever in the
// stencil one value stands out (tests/test_fixed_recon.py,
// tests/test_fixed_recon_groups.py).  With one exponent and no k a large value in
// an outer cell (weight ~0.05) left the states 3 to 20 times FP64's error.
//
// Not representable that way, and decided per variable and stencil: E below 58
// (values under 2^-965) gives zero states; 2040 and up (values over 2^1017, where
// k lowers E up to 2^1023; infinities, NaN) gives NaN states, hence a NaN flux as
// the FP64 sums' overflow in HLLC does.
#pragma once
#include <stdint.h>

#include "gpm_common.h"

#ifdef __CUDACC__
#define GPM_HD __host__ __device__ __forceinline__
#else
#define GPM_HD inline
#endif

// Biased exponent and signed mantissa (M << 5) of a double; subnormals are zero.
GPM_HD long long fix_decode(long long bits, int* e) {
    const int ex = (int)(bits >> 52) & 0x7ff;
    const long long m = ((bits & 0x000fffffffffffffLL) | 0x0010000000000000LL) << 5;
    *e = ex;
    const long long s = bits >> 63;  // 0 or -1
    return ex ? (m ^ s) - s : 0;
}

// v >> n for n >= 0; any n past 63 gives 0 or -1.
GPM_HD long long fix_shift(long long v, unsigned n) {
#ifdef __CUDA_ARCH__
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
#else
    return v >> (n > 63 ? 63 : n);
#endif
}

// The group of stencil value i (the order below): 0 the cell itself, 1 and 2 its
// neighbours along n and t, 3 and 4 the next ones, 5 the corners.
GPM_HD constexpr int fix_group(int i) { return i == 0 ? 0 : i < 9 ? (i + 1) / 2 : 5; }

// The stencil values q(i), decoded, aligned by their exponents e and their groups'
// k into v; returns E.
template <int NP, class Load>
GPM_HD int fix_align(const int* k, int* e, long long* v, Load q) {
    int E = 0;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 0; i < NP; i++) {
        if (i) e[i] -= k[fix_group(i)];
        E = e[i] > E ? e[i] : E;
    }
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 0; i < NP; i++) v[i] = fix_shift(q(i), (unsigned)(E - e[i]));
    return E;
}

GPM_HD long long fix_wide(int a, int b) { return (long long)a * b; }

// Mirror-symmetry components (the order of FixOrbit) of the aligned stencil
// values v, each split into signed halves.  Order 5: v at (n, t) = (0,0),
// (-1,0), (1,0), (0,-1), (0,1), (-2,0), (2,0), (0,-2), (0,2), (-1,-1), (1,-1),
// (-1,1), (1,1); order 3: the first five.
struct FixHalves {
    int h, l;
};
GPM_HD FixHalves fix_split(long long q) {
    FixHalves s;
    s.h = (int)((q + (1LL << 29)) >> 30);
    s.l = (int)((unsigned)q - ((unsigned)s.h << 30));
    return s;
}
template <int ORD>
GPM_HD void fix_components(const long long* v, FixHalves* c) {
    if (ORD == 3) {
        c[0] = fix_split(v[0]);
        c[1] = fix_split(v[1] + v[2]);
        c[2] = fix_split(v[3] + v[4]);
        c[3] = fix_split(v[1] - v[2]);
        c[4] = fix_split(v[3] - v[4]);
        return;
    }
    const long long s1 = v[9] + v[10], s2 = v[11] + v[12], d1 = v[9] - v[10], d2 = v[11] - v[12];
    c[0] = fix_split(v[0]);
    c[1] = fix_split(v[1] + v[2]);
    c[2] = fix_split(v[5] + v[6]);
    c[3] = fix_split(v[3] + v[4]);
    c[4] = fix_split(v[7] + v[8]);
    c[5] = fix_split(s1 + s2);
    c[6] = fix_split(v[1] - v[2]);
    c[7] = fix_split(v[5] - v[6]);
    c[8] = fix_split(d1 + d2);
    c[9] = fix_split(v[3] - v[4]);
    c[10] = fix_split(v[7] - v[8]);
    c[11] = fix_split(s1 - s2);
    c[12] = fix_split(d1 - d2);
}

// sum_i w[i] c[i] in Q's unit.
template <int N>
GPM_HD long long fix_dot(const FixWeight* w, const FixHalves* c) {
    long long hh = 0, hl = 0;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 0; i < N; i++) {
        hh += fix_wide(c[i].h, w[i].h);
        hl += fix_wide(c[i].h, w[i].l);
        hl += fix_wide(c[i].l, w[i].h);
    }
    return (long long)((unsigned long long)hh << 2) + (hl >> 28);
}

// The states of an axis's two faces (lo: left or bottom, hi: right or top) at
// its NGP Gauss points from the components in that axis's frame.
template <int ORD, int NGP>
GPM_HD void fix_family(const FixWeight* w0, const FixWeight* w1, const FixHalves* c, long long* lo, long long* hi) {
    constexpr int P = ORD == 5 ? 6 : 3, M = ORD == 5 ? 3 : 1;  // sizes of the first group, of the next two
    const long long pp = fix_dot<P>(w0, c), mp = fix_dot<M>(w0 + P, c + P), pm = fix_dot<M>(w0 + P + M, c + P + M);
    const long long mm = ORD == 5 ? fix_dot<1>(w0 + 12, c + 12) : 0;
    const long long A = pp + pm, B = mp + mm, C = pp - pm, D = mp - mm;
    lo[0] = A + B;
    hi[0] = A - B;
    lo[NGP - 1] = C + D;
    hi[NGP - 1] = C - D;
    if (NGP == 3) {
        const long long p1 = fix_dot<P>(w1, c), m1 = fix_dot<M>(w1 + P, c + P);
        lo[1] = p1 + m1;
        hi[1] = p1 - m1;
    }
}

// Whether exponent E has normal results (see the head of the file).
GPM_HD bool fix_exponent_ok(int E) { return (unsigned)(E - 58) < 2040u - 58u; }

// r * 2^(E-1080) for |r| < 2^62, E ok, rounded to nearest (halves away from
// zero), in integer instructions: cvt.f64.s64 runs on the FP64 pipe (measured
// 17 cycles beside FMAs, as an FMA).
GPM_HD double fix_value(long long r, int E) {
#ifdef __CUDA_ARCH__
    const long long s = r >> 63;
    const unsigned long long a = (unsigned long long)((r ^ s) - s);
    const int lz = __clzll((long long)a);  // 2..64
    const unsigned long long m = ((a << (lz - 1)) + 0x200) >> 10;  // leading one at bit 52
    const int hi = (int)(m >> 32) + ((E + 5 - lz) << 20);
    const int neg = (int)(s & 0x80000000LL);
    return a ? __hiloint2double(hi | neg, (int)m) : 0.0;
#else
    unsigned long long a = (unsigned long long)(r < 0 ? -r : r), bits = 0;
    if (a) {
        const int lz = __builtin_clzll(a);
        bits = (((a << (lz - 1)) + 0x200) >> 10) + ((unsigned long long)(E + 5 - lz) << 52);
        if (r < 0) bits |= 1ull << 63;
    }
    union {
        unsigned long long i;
        double f;
    } u;
    u.i = bits;
    return u.f;
#endif
}
// ... and every state of a stencil whose exponent is not: zero or NaN.
GPM_HD long long fix_special_bits(int E) { return E < 58 ? 0 : 0x7ff8000000000000LL; }
