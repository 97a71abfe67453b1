// fast_rcp.cuh -- reciprocal and square root for the fast floating-point mode.
//
// On this part an FP64 instruction costs an SM 16-19 cycles and a lone warp 64,
// an integer one half a cycle and ~5, so few FP64 instructions is what counts.
//
// 1/d in integers, no FP64 instruction: from y ~ 1/d (PTX rcp.approx.ftz.f64,
// whose low word is zero: a 21-bit mantissa Y, relative error at most 2^-19.9)
// the residual e = 1 - d*y is exact in the low 64 bits of the mantissas'
// product D*Y = 2^P (1 - e), and 1/d = y (1 + e + e^2) + O(2^-59.7), the cubic
// ("hyperpower") iteration of M. Altman, Pacific J. Math. 10(4):1107-1113,
// 1960, is evaluated on the mantissa with 8 to 10 guard bits and rounded once:
// within 1.01 half-ulps on 4e7 samples.  ~35 integer instructions; three FP64
// FMAs for the same series cost the 2048^2 first pass 12 of its 48 per Riemann
// solve.  From |d| = 2^1022 on, where reciprocals turn subnormal, the result is
// the seed: 2^-1022 to its 20 bits, then a zero of d's sign.  Zero, subnormal,
// infinite and NaN d give NaN.
//
// sqrt(x) in integers too: from y ~ 1/sqrt(x) (PTX rsqrt.approx.ftz.f64, low
// word zero) the residual e = 1 - x*y^2 is exact to 2^-60 in the middle bits of
// the mantissas' product X*Y^2 = 2^P (1 - e), and sqrt(x) = x*y (1 - e)^(-1/2) =
// x*y (1 + e/2 + 3/8 e^2) + O(e^3) (the binomial series).  Measured |e| <=
// 2^-19, so the remainder is under 2^-58.  ~60 integer instructions for five
// FP64 ones (2048^2 Sedov, 2 steps: 19.6 -> 17.4 ms), within 1.28 half-ulps on
// 2e7 samples with the largest residual; the FP64 form was within an ulp or so.  Zero, negative,
// subnormal and infinite x give NaN; the solver takes it only of a pressure over
// a density that it has already tested, or will test, for positivity.
#pragma once

__device__ __forceinline__ double gpm_fast_rcp(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const unsigned dh = (unsigned)__double2hiint(d), dl = (unsigned)__double2loint(d), yh = (unsigned)__double2hiint(y);
    const unsigned Y = (yh & 0xfffffu) | 0x100000u, Dh = (dh & 0xfffffu) | 0x100000u;
    const unsigned ey = (yh >> 20) & 0x7ffu;
    const int sh = 2054 - (int)((dh >> 20) & 0x7ffu) - (int)ey;  // P - 64: 8, 9 or 10
    const unsigned long long lo = (unsigned long long)dl * Y;
    // -e 2^P
    const long long f = (long long)(lo + ((unsigned long long)(Dh * Y) << 32));
    const int fh = (int)(f >> 24);
    const long long g = (((long long)fh * fh) >> (sh + 16)) - f;  // (e + e^2) 2^P
    // Y (1 + e + e^2) 2^(P - 32), the leading one near bit 60 + sh - 8
    const unsigned long long c = (unsigned long long)((long long)(int)(g >> 32) * (long long)Y) +
                                 (((unsigned long long)(unsigned)g * Y) >> 32);
    const unsigned long long W = ((unsigned long long)(Y << sh) << 32) + c;
    const int s2 = 11 - __clz((int)(W >> 32));
    const unsigned long long M = (W + (1ull << (s2 - 1))) >> s2;
    const unsigned hi = (yh & 0xfff00000u) + ((unsigned)(M >> 32) - 0x100000u) + ((unsigned)(s2 - sh) << 20);
    const unsigned mag = dh & 0x7fffffffu, other = mag - 0x7fd00000u < 0x200000u ? yh : 0x7ff80000u;
    return mag - 0x100000u < 0x7fc00000u ? __hiloint2double((int)hi, (int)M) : __hiloint2double((int)other, 0);
}

__device__ __forceinline__ double gpm_fast_sqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x), yh = (unsigned)__double2hiint(y);
    const unsigned Y = (yh & 0xfffffu) | 0x100000u, Xh = (xh & 0xfffffu) | 0x100000u;
    const int ex = (int)(xh >> 20), ey = (int)((yh >> 20) & 0x7ffu);
    const int q = 3129 - ex - 2 * ey;  // P - 32: 60 to 63
    const unsigned long long Y2 = (unsigned long long)Y * Y;
    const unsigned Yl = (unsigned)Y2, Yt = (unsigned)(Y2 >> 32);
    // -e 2^q
    const long long f = (long long)((((unsigned long long)xl * Yl) >> 32) + (unsigned long long)xl * Yt +
                                    (unsigned long long)Xh * Yl + ((unsigned long long)(Xh * Yt) << 32) - (1ull << q));
    const int fh = (int)(f >> 20);
    const long long C = (((long long)fh * (3 * fh)) >> (q - 37)) - (f >> 1);  // (e/2 + 3/8 e^2) 2^q
    // X Y 2^-11 (1 + C 2^-q), the leading one near bit 61 or 62
    const unsigned long long G = ((unsigned long long)Xh * Y << 21) + (((unsigned long long)xl * Y) >> 11);
    const unsigned gh = (unsigned)(G >> 32);
    const int gl = (int)((unsigned)G >> 1);
    const unsigned long long W = G + ((unsigned long long)((long long)(int)gh * (int)(C >> 32)) << (64 - q)) +
                                 (((unsigned long long)gh * (unsigned)C) >> (q - 32)) +
                                 (unsigned long long)(((long long)gl * (int)(C >> 13)) >> (q - 14));
    const int s2 = 11 - __clz((int)(W >> 32));
    const unsigned long long M = (W + (1ull << (s2 - 1))) >> s2;
    const unsigned hi = (unsigned)(M >> 32) + ((unsigned)(ex + ey + s2 - 1033) << 20);
    return (unsigned)(ex - 1) < 2046u ? __hiloint2double((int)hi, (int)M) : __longlong_as_double(0x7ff8000000000000LL);
}
