// adjoint.cu -- hand-written adjoint (vector-Jacobian product) of one GP-MOOD
// RK stage with its MOOD order mask frozen.
//
// With the orders fixed, a stage is the smooth-almost-everywhere map
//   Uout = Uin + qy*Fy(c-y) + qx*Fx(c-x) - qx*Fx(c) - qy*Fy(c)   (interior c)
//   F    = sum_g w_g HLLC(uL_g, uR_g),  uL_g/uR_g = GP dot products of BC(Uin)
// (mod_FE.f90:75-145, mod_GP_MOOD.f90:58-65, mod_HLLC.f90:11-169).  Its VJP:
//   mu_F        = q * (lam(high cell) - lam(low cell))            per face
//   mu_uL_g     = w_g * J_L(g)^T mu_F,  mu_uR_g = w_g * J_R(g)^T mu_F
//   mu_U(c)    += z_m * mu_u  over every face state whose stencil holds c
//   lam_in      = lam_out + BC^T(mu_U)
// J^T mu of HLLC is its hand-written reverse sweep (the branch is picked on the
// values, as in HLLC).
#define GPM_EXACT 1
#include "physics.cuh"
#include "adjoint.h"

#include <type_traits>

namespace {

// One side of a face in its normal frame, and the adjoints of these quantities.
struct ASide {
    double r, n, t, e, ir, v, w, p, c;
};
struct ABar {
    double r, n, t, e, v, w, p, c;
};

__device__ __forceinline__ ASide adj_side(double r, double n, double t, double e) {
    ASide s;
    s.r = r;
    s.n = n;
    s.t = t;
    s.e = e;
    s.ir = 1. / r;
    s.v = n * s.ir;
    s.w = t * s.ir;
    s.p = (GPM_GAMMA - 1.) * (e - 0.5 * (n * s.v + t * s.w));
    s.c = sqrt(GPM_GAMMA * s.p * s.ir);
    return s;
}

// From the adjoints of (v, w, p, c) and of the state's own uses to the state's:
// c^2 = gamma p / r, p = (gamma-1)(e - (n v + t w)/2), v = n/r, w = t/r.
__device__ __forceinline__ void adj_close(const ASide& s, ABar& b) {
    const double h = 0.5 * b.c / s.c * s.ir;  // c_bar / (2 c r)
    b.p += GPM_GAMMA * h;
    b.r -= h * s.c * s.c;
    const double gp = (GPM_GAMMA - 1.) * b.p;
    b.e += gp;
    b.n += b.v * s.ir - gp * s.v;
    b.t += b.w * s.ir - gp * s.w;
    b.r += 0.5 * gp * (s.v * s.v + s.w * s.w) - (b.v * s.v + b.w * s.w) * s.ir;
}

// Reverse sweep of HLLC for admissible states: the adjoints (br, bn, bt, be) of
// the flux (mass, normal and tangential momentum, energy) to those of the two
// states.  The star flux is taken at the contact speed (hllc_normal's form,
// equal to mod_HLLC.f90's by the Rankine-Hugoniot relations):
//   om = u* - v, q = 1/(S - u*), ps = p + a om, m = a q u*,
//   T = e (S - v) + om (p + a u*),  F = (m, m u* + ps, m w, u* (T q + ps)).
// ~170 FP64 instructions; forward-mode duals over the eight inputs took ~1000.
__device__ __forceinline__ void adj_hllc(const ASide& L, const ASide& R, double br, double bn, double bt, double be,
                                         ABar& bL, ABar& bR) {
    const double lo0 = L.v - L.c, lo1 = R.v - R.c, hi0 = L.v + L.c, hi1 = R.v + R.c;
    const double SL = lo1 < lo0 ? lo1 : lo0, SR = hi1 > hi0 ? hi1 : hi0;
    const double xL = SL - L.v, xR = SR - R.v, aL = L.r * xL, aR = R.r * xR;
    const double iD = 1. / (aL - aR);
    const double us = (R.p - L.p + aL * L.v - aR * R.v) * iD;
    bL = ABar{0., 0., 0., 0., 0., 0., 0., 0.};
    bR = bL;
    const bool left = SL >= 0. || us >= 0.;
    const ASide& K = left ? L : R;
    ABar bK = bL;
    if (SL >= 0. || (us < 0. && !(SR >= 0.))) {  // the side's physical flux
        bK.n = br + bn * K.v + bt * K.w;
        bK.v = bn * K.n + be * (K.e + K.p);
        bK.w = bt * K.n;
        bK.p = bn + be * K.v;
        bK.e = be * K.v;
        (left ? bL : bR) = bK;
    } else {
        const double S = left ? SL : SR, a = left ? aL : aR, x = left ? xL : xR;
        const double om = us - K.v, q = 1. / (S - us), ps = K.p + a * om, m = a * q * us;
        const double pu = K.p + a * us, T = K.e * x + om * pu;
        const double mb = br + bn * us + bt * K.w, psb = bn + be * us, Tb = be * us * q;
        const double qb = be * us * T + mb * a * us;
        double ab = mb * q * us + Tb * om * us + psb * om;
        double ub = bn * m + be * (T * q + ps) + mb * a * q + Tb * om * a;
        const double omb = Tb * pu + psb * a, xb = Tb * K.e, db = -qb * q * q;  // d = S - u*
        bK.w = bt * m;
        bK.e = Tb * x;
        bK.p = Tb * om + psb;
        bK.v = -omb - xb;
        double Sb = xb + db;
        ub += omb - db;
        (left ? bL : bR) = bK;
        // u* = N / D, N = pR - pL + aL vL - aR vR, D = aL - aR
        const double Nb = ub * iD, Db = -Nb * us;
        bR.p += Nb;
        bL.p -= Nb;
        bL.v += Nb * aL;
        bR.v -= Nb * aR;
        const double aLb = Nb * L.v + Db + (left ? ab : 0.), aRb = -Nb * R.v - Db + (left ? 0. : ab);
        // aK = rK (SK - vK)
        bL.r += aLb * xL;
        bL.v -= aLb * L.r;
        bR.r += aRb * xR;
        bR.v -= aRb * R.r;
        const double SLb = aLb * L.r + (left ? Sb : 0.), SRb = aRb * R.r + (left ? 0. : Sb);
        if (lo1 < lo0) {
            bR.v += SLb;
            bR.c -= SLb;
        } else {
            bL.v += SLb;
            bL.c -= SLb;
        }
        if (hi1 > hi0) {
            bR.v += SRb;
            bR.c += SRb;
        } else {
            bL.v += SRb;
            bL.c += SRb;
        }
    }
    adj_close(L, bL);
    adj_close(R, bR);
}

__device__ __forceinline__ size_t aidx(int nx, int l, int n) { return (size_t)(n + 3) * nx + (size_t)(l + 3); }

// Per face and Gauss point: the states at the frozen order and their adjoints
// mu_uL[g][4], mu_uR[g][4] (stored per face).  One lane per Gauss point, 32/NGP
// faces per warp, x faces first (a warp holds one direction), as the first
// pass (k_flux_gp).
template <int NGP>
__global__ void __launch_bounds__(128, 4) k_adj_faces(AdjArgs a, const __grid_constant__ GpWeights w) {
    constexpr int FPW = 32 / NGP;
    __shared__ double z[3][4][NGP][13];
    const GridGeom& g = a.g;
    for (int i = threadIdx.x; i < 12 * NGP * 13; i += 128) {
        const int o = i / (4 * NGP * 13), r = i - o * (4 * NGP * 13);
        z[o][r / (NGP * 13)][r / 13 % NGP][r % 13] = w.zt[o][r / (NGP * 13)][r / 13 % NGP][r % 13];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, fl = lane / NGP, gp = lane - fl * NGP;
    const long long nfx = (long long)(g.lf + 1) * g.nf, nfy = (long long)g.lf * (g.nf + 1);
    const long long nxw = (nfx + FPW - 1) / FPW, wi = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int dir = wi < nxw ? 0 : 1, len = dir == 0 ? g.lf + 1 : g.lf;
    const long long i = (dir == 0 ? wi : wi - nxw) * FPW + fl;
    if (fl >= FPW || i >= (dir == 0 ? nfx : nfy)) return;
    const int row = (int)(i / len), col = (int)(i - (long long)row * len);
    const int l = dir == 0 ? col : 1 + col, n = dir == 0 ? 1 + row : row;
    const size_t c0 = aidx(g.nx, l, n), c1 = dir == 0 ? c0 + 1 : c0 + g.nx;
    const int FL = dir == 0 ? 2 : 1, FH = dir == 0 ? 0 : 3;
    const bool lin = (l >= 1 && l <= g.lf && n >= 1 && n <= g.nf);
    const int lh = dir == 0 ? l + 1 : l, nh = dir == 0 ? n : n + 1;
    const bool hin = (lh >= 1 && lh <= g.lf && nh >= 1 && nh <= g.nf);
    const double q = (dir == 0 ? a.qx : a.qy) * w.gw[gp];
    double muF[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double lo = lin ? a.lam_out[4 * c0 + k] : 0.0, hi = hin ? a.lam_out[4 * c1 + k] : 0.0;
        muF[k] = q * (hi - lo);
    }
    double u[2][4];
    auto states = [&](auto np, int o) {
        constexpr int NP = decltype(np)::value;
        const ptrdiff_t r = g.nx;
#pragma unroll
        for (int side = 0; side < 2; side++) {
            const double* p = a.u_in + 4 * (side ? c1 : c0);
            Cell c[NP];
#pragma unroll
            for (int m = 0; m < NP; m++) c[m] = ld_cell(p + 4 * (st_ox(m) + r * st_oy(m)));
            gp_recon_at<NP>(&z[o][side ? FH : FL][gp][0], c, u[side]);
        }
    };
    const int o = min((int)a.order[c0], (int)a.order[c1]);
    if (o >= 5) states(std::integral_constant<int, 13>{}, 2);
    else if (o >= 3) states(std::integral_constant<int, 5>{}, 1);
    else states(std::integral_constant<int, 1>{}, 0);
    const bool y = dir != 0;
    const ASide L = adj_side(u[0][0], y ? u[0][2] : u[0][1], y ? u[0][1] : u[0][2], u[0][3]);
    const ASide R = adj_side(u[1][0], y ? u[1][2] : u[1][1], y ? u[1][1] : u[1][2], u[1][3]);
    ABar bL, bR;
    adj_hllc(L, R, muF[0], y ? muF[2] : muF[1], y ? muF[1] : muF[2], muF[3], bL, bR);
    double* out = a.face_adj + (dir == 0 ? 0 : (size_t)g.nx * g.ny * 8 * GPM_MAXGP) + c0 * 8 * GPM_MAXGP + gp * 8;
    st_cell(out, Cell{bL.r, y ? bL.t : bL.n, y ? bL.n : bL.t, bL.e});
    st_cell(out + 4, Cell{bR.r, y ? bR.t : bR.n, y ? bR.n : bR.t, bR.e});
}

// mu_U(c) for every padded cell within reach of a face: gather over the face
// states whose stencils hold c, one thread per variable (a quarter of the
// chain of a thread per cell, and four lanes read 32 bytes together: 48.6 us a
// stage of 128^2 before).
template <int NGP>
__global__ void __launch_bounds__(128) k_adj_gather(AdjArgs a, const __grid_constant__ GpWeights w) {
    const GridGeom& g = a.g;
    const long long ncell = (long long)g.nx * g.ny;
    const long long ck = (long long)blockIdx.x * blockDim.x + threadIdx.x, c = ck >> 2;
    const int k = (int)(ck & 3);
    if (c >= ncell) return;
    const int l = (int)(c % g.nx) - 3, n = (int)(c / g.nx) - 3;
    double mu = 0.;
    for (int m = 0; m < 13; m++) {
#pragma unroll
        for (int dir = 0; dir < 2; dir++) {
            // as the low cell's stencil point m: face with low cell (l - ox, n - oy)
            // as the high cell's stencil point m: face with high cell (l - ox, n - oy)
#pragma unroll
            for (int side = 0; side < 2; side++) {
                const int cl = l - st_ox(m) - (side == 1 && dir == 0 ? 1 : 0);
                const int cn = n - st_oy(m) - (side == 1 && dir == 1 ? 1 : 0);
                const bool ok = dir == 0 ? (cl >= 0 && cl <= g.lf && cn >= 1 && cn <= g.nf)
                                         : (cl >= 1 && cl <= g.lf && cn >= 0 && cn <= g.nf);
                if (!ok) continue;
                const size_t f0 = aidx(g.nx, cl, cn), f1 = dir == 0 ? f0 + 1 : f0 + g.nx;
                const int o = min((int)a.order[f0], (int)a.order[f1]);
                const int np = o >= 5 ? 13 : (o >= 3 ? 5 : 1);
                if (m >= np) continue;
                const int oi = o >= 5 ? 2 : (o >= 3 ? 1 : 0);
                const int face = dir == 0 ? (side == 0 ? 2 : 0) : (side == 0 ? 1 : 3);
                const double* fa = a.face_adj + (dir == 0 ? 0 : (size_t)g.nx * g.ny * 8 * GPM_MAXGP) + f0 * 8 * GPM_MAXGP;
#pragma unroll
                for (int gp = 0; gp < NGP; gp++) mu += w.zt[oi][face][gp][m] * __ldg(fa + gp * 8 + side * 4 + k);
            }
        }
    }
    a.mu_pad[4 * c + k] = mu;
}

// Transpose of Boundary_C (BC.f90:10-421: ghost columns, then ghost rows): first the
// ghost rows are folded into the interior rows they copy (every column), then
// the ghost columns into the interior columns.  Reflective ghosts carry the
// sign flip of the normal momentum.
__device__ __forceinline__ int ghost_source(int bc, int i, int nint, int* sign) {
    // source index of ghost i (i <= 0 or i > nint) along one axis; sign -1 on a mirror
    *sign = 1;
    if (bc == 17) return i <= 0 ? 1 : nint;
    if (bc == 18) return i <= 0 ? i + nint : i - nint;
    *sign = -1;  // 20
    return i <= 0 ? 1 - i : 2 * nint + 1 - i;
}

__global__ void k_adj_fold_y(GridGeom g, double* __restrict__ mu) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)g.nx * g.nf) return;
    const int l = (int)(idx % g.nx) - 3, n = 1 + (int)(idx / g.nx);
    double s[4];
    const size_t c = aidx(g.nx, l, n);
#pragma unroll
    for (int k = 0; k < 4; k++) s[k] = mu[4 * c + k];
    for (int j = 0; j < GPM_NGC; j++) {
        for (int top = 0; top < 2; top++) {
            const int ng = top ? g.nf + 1 + j : -j;
            int sg;
            if (ghost_source(g.bc_type, ng, g.nf, &sg) != n) continue;
            const size_t cg = aidx(g.nx, l, ng);
            s[0] += mu[4 * cg + 0];
            s[1] += mu[4 * cg + 1];
            s[2] += sg * mu[4 * cg + 2];
            s[3] += mu[4 * cg + 3];
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) mu[4 * c + k] = s[k];
}

__global__ void k_adj_fold_x(GridGeom g, const double* __restrict__ mu, const double* base, double* out) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)g.lf * g.nf) return;
    const int l = 1 + (int)(idx % g.lf), n = 1 + (int)(idx / g.lf);
    const size_t c = aidx(g.nx, l, n);
    double s[4];
#pragma unroll
    for (int k = 0; k < 4; k++) s[k] = base[4 * c + k] + mu[4 * c + k];
    for (int j = 0; j < GPM_NGC; j++) {
        for (int right = 0; right < 2; right++) {
            const int lg = right ? g.lf + 1 + j : -j;
            int sg;
            if (ghost_source(g.bc_type, lg, g.lf, &sg) != l) continue;
            const size_t cg = aidx(g.nx, lg, n);
            s[0] += mu[4 * cg + 0];
            s[1] += sg * mu[4 * cg + 1];
            s[2] += mu[4 * cg + 2];
            s[3] += mu[4 * cg + 3];
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) out[4 * c + k] = s[k];
}

void launch_fold(const GridGeom& g, double* mu, const double* base, double* out, cudaStream_t s) {
    const long long ny = (long long)g.nx * g.nf, nx = (long long)g.lf * g.nf;
    k_adj_fold_y<<<(int)((ny + 255) / 256), 256, 0, s>>>(g, mu);
    k_adj_fold_x<<<(int)((nx + 255) / 256), 256, 0, s>>>(g, mu, base, out);
}

template <int NGP>
void launch_adj_n(const AdjArgs& a, const GpWeights& w, cudaStream_t s) {
    constexpr int FPW = 32 / NGP;
    const long long nfx = (long long)(a.g.lf + 1) * a.g.nf, nfy = (long long)a.g.lf * (a.g.nf + 1);
    k_adj_faces<NGP><<<(unsigned)(((nfx + FPW - 1) / FPW + (nfy + FPW - 1) / FPW + 3) / 4), 128, 0, s>>>(a, w);
    const long long nc = 4 * (long long)a.g.nx * a.g.ny;  // (cell, variable)
    k_adj_gather<NGP><<<(unsigned)((nc + 127) / 128), 128, 0, s>>>(a, w);
    launch_fold(a.g, a.mu_pad, a.lam_out, a.lam_in, s);
}

}  // namespace

int gpm_adj_stage(const AdjArgs& a, const GpWeights& w, cudaStream_t s) {
    switch (a.g.ngp) {
    case 1: launch_adj_n<1>(a, w, s); break;
    case 2: launch_adj_n<2>(a, w, s); break;
    case 3: launch_adj_n<3>(a, w, s); break;
    case 4: launch_adj_n<4>(a, w, s); break;
    default: launch_adj_n<5>(a, w, s); break;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int gpm_adj_fold(const GridGeom& g, double* mu, const double* base, double* out, cudaStream_t s) {
    launch_fold(g, mu, base, out, s);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
