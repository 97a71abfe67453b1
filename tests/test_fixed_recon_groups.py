"""The fixed-point reconstruction of the fast first pass (csrc/fixed_recon.cuh,
csrc/gp_weights.cpp) on the CPU, aligned by the cells' weights: its RMS error,
relative to the size of a state's terms, against binary128 sums of the same
stencils and weights is no larger than that of the same sums in FP64, wherever
in the stencil one value stands out and however far."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gp-mood_gb300" / "csrc"

SOURCE = r"""
#include <math.h>
#include <stdio.h>
#include <string.h>
#include <random>
#include "fixed_recon.cuh"
typedef __float128 f128;
// stencil index of v's entries in the axis's (n, t) frame
static const int v_to_st[2][13] = {{0, 1, 3, 4, 2, 10, 12, 9, 11, 5, 8, 6, 7}, {0, 4, 2, 1, 3, 9, 11, 10, 12, 5, 6, 8, 7}};
template <int ORD>
static void fixed(const GpWeights& w, int axis, const double* q, double lo[3], double hi[3]) {
    constexpr int NP = ORD == 5 ? 13 : 5;
    long long m[13], v[13], l[3], h[3];
    int e[13];
    for (int i = 0; i < NP; i++) {
        long long b;
        memcpy(&b, &q[v_to_st[axis][i]], 8);
        m[i] = fix_decode(b, &e[i]);
    }
    const FixOrbit& o = w.orb[ORD / 2 - 1];
    const int E = fix_align<NP>(o.k[axis], e, v, [&](int i) { return m[i]; });
    FixHalves c[13];
    fix_components<ORD>(v, c);
    fix_family<ORD, 3>(o.g0[axis], o.g1[axis], c, l, h);
    for (int g = 0; g < 3; g++) {
        double sp;
        long long b = fix_special_bits(E);
        memcpy(&sp, &b, 8);
        lo[g] = fix_exponent_ok(E) ? fix_value(l[g], E) : sp;
        hi[g] = fix_exponent_ok(E) ? fix_value(h[g], E) : sp;
    }
}
// the same sums in T with the symmetrised double weights
template <class T, class Fma>
static void sums(const GpWeights& w, int o, int axis, const double* q, T lo[3], T hi[3], Fma fm) {
    const int* s = v_to_st[axis];
    const int np = o == 2 ? 13 : 5;
    auto Q = [&](int i) { return i < np ? (T)q[s[i]] : (T)0; };
    const T s1 = Q(9) + Q(10), s2 = Q(11) + Q(12), d1 = Q(9) - Q(10), d2 = Q(11) - Q(12);
    const T c[13] = {Q(0), Q(1) + Q(2), Q(5) + Q(6), Q(3) + Q(4), Q(7) + Q(8), s1 + s2, Q(1) - Q(2), Q(5) - Q(6),
                     d1 + d2, Q(3) - Q(4), Q(7) - Q(8), s1 - s2, d1 - d2};
    auto weights = [&](int g, double* c13) {
        const double* zt = w.zt[o][axis ? 3 : 0][g];
        double z[13];
        for (int i = 0; i < 13; i++) z[i] = i < np ? zt[s[i]] : 0.0;
        const double k[13] = {z[0], 0.5 * (z[1] + z[2]), 0.5 * (z[5] + z[6]), 0.5 * (z[3] + z[4]), 0.5 * (z[7] + z[8]),
                              0.25 * (z[9] + z[10] + z[11] + z[12]), 0.5 * (z[1] - z[2]), 0.5 * (z[5] - z[6]),
                              0.25 * (z[9] - z[10] + z[11] - z[12]), 0.5 * (z[3] - z[4]), 0.5 * (z[7] - z[8]),
                              0.25 * (z[9] + z[10] - z[11] - z[12]), 0.25 * (z[9] - z[10] - z[11] + z[12])};
        memcpy(c13, k, sizeof k);
    };
    double z[13], y[13];
    weights(0, z);
    weights(1, y);
    auto dot = [&](const double* a, const T* x, int n) {
        T r = (T)a[0] * x[0];
        for (int i = 1; i < n; i++) r = fm((T)a[i], x[i], r);
        return r;
    };
    const T pp = dot(z, c, 6), mp = dot(z + 6, c + 6, 3), pm = dot(z + 9, c + 9, 3), mm = (T)z[12] * c[12];
    const T A = pp + pm, B = mp + mm, C = pp - pm, D = mp - mm;
    const T p1 = dot(y, c, 6), m1 = dot(y + 6, c + 6, 3);
    lo[0] = A + B;
    hi[0] = A - B;
    lo[2] = C + D;
    hi[2] = C - D;
    lo[1] = p1 + m1;
    hi[1] = p1 - m1;
}
int main() {
    std::mt19937_64 r(1);
    std::uniform_real_distribution<double> U(-1, 1);
    // the cell itself, its neighbours along n and t, the next ones, the corners
    const int first[] = {0, 1, 3, 5, 7, 9}, count[] = {1, 2, 2, 2, 2, 4};
    GpWeights w;
    double ie[3], lo[3], hi[3], q[13];
    for (double ell : {1.0, 3.0, 12.0, 50.0})
        for (double aspect : {1.0, 0.25, 8.0}) {
            if (gpm_gp_presim(ell, 1.0, aspect, 64, 64, 5, 3, &w, ie) || !w.orb[0].ok || !w.orb[1].ok) return 2;
            for (int o = 1; o <= 2; o++)
                for (int axis = 0; axis < 2; axis++)
                    for (int group = 0; group < (o == 2 ? 6 : 3); group++)
                        for (double scale : {1.0, 10.0, 100.0, 1e4, 1e6, 1e10}) {
                            double ef = 0, ed = 0;
                            for (int it = 0; it < 1000; it++) {
                                for (int m = 0; m < 13; m++) q[m] = 1 + 0.1 * U(r);
                                q[v_to_st[axis][first[group] + it % count[group]]] *= scale;
                                double f[2][3], d[2][3];
                                f128 x[2][3];
                                o == 2 ? fixed<5>(w, axis, q, f[0], f[1]) : fixed<3>(w, axis, q, f[0], f[1]);
                                sums(w, o, axis, q, d[0], d[1], [](double a, double b, double c) { return fma(a, b, c); });
                                sums(w, o, axis, q, x[0], x[1], [](f128 a, f128 b, f128 c) { return a * b + c; });
                                for (int side = 0; side < 2; side++)
                                    for (int g = 0; g < 3; g++) {
                                        // the state's terms: its own size unless they cancel
                                        const double* z = w.zt[o][axis ? (side ? 1 : 3) : (side ? 2 : 0)][g];
                                        double size = 0;
                                        for (int m = 0; m < (o == 2 ? 13 : 5); m++) size += fabs(z[m] * q[m]);
                                        const f128 ex = x[side][g];
                                        const double a = (double)((f[side][g] - ex) / size), c = (double)((d[side][g] - ex) / size);
                                        ef += a * a;
                                        ed += c * c;
                                    }
                            }
                            printf("%g %g %d %d %d %g %.3e %.3e\n", ell, aspect, o, axis, group, scale, sqrt(ef), sqrt(ed));
                        }
        }
    // the range: values that overflow or vanish wherever they sit
    if (gpm_gp_presim(12, 1, 1, 64, 64, 5, 3, &w, ie)) return 2;
    for (int axis = 0; axis < 2; axis++)
        for (int at = 0; at < 13; at++)
            for (double bad : {(double)INFINITY, -(double)INFINITY, (double)NAN}) {
                for (int m = 0; m < 13; m++) q[m] = m == at ? bad : 0.7;
                fixed<5>(w, axis, q, lo, hi);
                for (int g = 0; g < 3; g++)
                    if (!isnan(lo[g]) || !isnan(hi[g])) return 4;
                // a huge value: its states to rounding, or NaN
                for (int m = 0; m < 13; m++) q[m] = m == at ? ldexp(1.5, 1000) : 0.7;
                fixed<5>(w, axis, q, lo, hi);
                double a[3], b[3];
                sums(w, 2, axis, q, a, b, [](double a, double b, double c) { return fma(a, b, c); });
                for (int g = 0; g < 3; g++)
                    if (!(fabs(lo[g] - a[g]) <= 1e-13 * fabs(a[g])) || !(fabs(hi[g] - b[g]) <= 1e-13 * fabs(b[g]))) return 6;
            }
    for (double small : {0.0, -0.0, 1e-300, 5e-324}) {
        for (int m = 0; m < 13; m++) q[m] = small;
        fixed<5>(w, 0, q, lo, hi);
        for (int g = 0; g < 3; g++)
            if (lo[g] != 0 || hi[g] != 0) return 5;
    }
    return 0;
}
"""


def test_error_of_the_state_is_no_larger_than_fp64(tmp_path):
    gxx = shutil.which("g++")
    cuda = Path("/usr/local/cuda/include")
    if not gxx or not cuda.exists():
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "fixed.cpp", tmp_path / "fixed"
    src.write_text(SOURCE)
    subprocess.run([gxx, "-O2", "-std=gnu++17", "-ffp-contract=off", f"-I{CSRC}", f"-I{cuda}", "-x", "c++", str(src),
                    str(CSRC / "gp_weights.cpp"), "-o", str(exe), "-lm"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, (out.returncode, out.stdout[-400:])
    rows = [[float(v) for v in line.split()] for line in out.stdout.splitlines()]
    assert len(rows) == 4 * 3 * 2 * (3 + 6) * 6
    for row in rows:
        assert row[-2] <= row[-1], row
