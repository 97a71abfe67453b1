// batch_fast.cuh -- the fast mode's arithmetic of the batched form: reciprocal,
// square root, HLLC, quadrature, Setdt's cell term and the two-direction cell
// tile, in FP64 throughout.  Included by stage_kernels.cu inside its namespace.
//
// An ensemble starts from piecewise constant states.  Upwind of a jump in
// supersonic flow a cell then keeps its density but for rounding, and
// DETECTION compares it with a bound that equals it: the last place decides
// whether a whole line of cells is lowered.  Measured on 768 four-quadrant
// problems (64..256 cells a side, 3 steps), another rounding of the same
// formulas moves such a decision in 1.3 % of them, and the state by 1e-7.  The
// batched form keeps its rounding, so that an ensemble's results stay what they
// were; the single-problem form went to the shorter HLLC of physics.cuh and the
// fixed-point sums of fixed_recon.cuh.  That is a choice (the same start as a
// single run moves in the same way), and its price is that in the fast mode a
// problem of a batch is not its own single run: of 512 such problems 1 after one
// step, 9 after 3 and 18 after 10 differ by more than 1e-13 (relative L1; at most
// 3e-4), the others by ~1e-16.  The exact mode's are equal bit for bit.
#pragma once

namespace ens {

// 1/d: two Newton steps from the hardware's approximation, y + y (1 - d y)
// (P. Markstein, IBM J. Res. Dev. 34(1):111-119, 1990).
__device__ __forceinline__ double rcp(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    double e = fma(-d, y, 1.0);
    y = fma(y, e, y);
    e = fma(-d, y, 1.0);
    return fma(y, e, y);
}


// sqrt(x): the coupled iteration of the same paper from the approximate
// reciprocal square root, and a last correction.
__device__ __forceinline__ double root(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
    const double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    const double e = fma(-g, g, x);
    return fma(h, e, g);
}

struct Prim {
    double vn, vt, p, c;
    bool adm;
    double vx;  // x-velocity, needed for the 1/(vx-vx) of an inadmissible state
    double ir;  // 1/rho
};

template <int DIR>
__device__ __forceinline__ Prim c2p(const double* u, double ir_in = 0.0) {
    Prim s;
    const double ir = ir_in;  // 1/rho, supplied by the caller
    const double vx = u[1] * ir;
    const double vy = u[2] * ir;
    s.p = (GPM_GAMMA - 1.) * (u[3] - 0.5 * (u[1] * vx + u[2] * vy));
    s.c = root(GPM_GAMMA * s.p * ir);  // NaN for p <= 0, which is inadmissible
    s.ir = ir;
    s.vx = vx;
    s.vn = DIR == 0 ? vx : vy;
    s.vt = DIR == 0 ? vy : vx;
    s.adm = !(le_zero_or_nan(u[0]) || le_zero_or_nan(s.p));
    return s;
}

template <int DIR>
__device__ __forceinline__ void phys_flux(const double* u, const Prim& s, double* r) {
    if (DIR == 0) {
        r[0] = u[1];
        r[1] = u[0] * (s.vn * s.vn) + s.p;
        r[2] = u[2] * s.vn;
        r[3] = s.vn * (u[3] + s.p);
    } else {
        r[0] = u[2];
        r[1] = u[1] * s.vn;
        r[2] = u[0] * (s.vn * s.vn) + s.p;
        r[3] = s.vn * (u[3] + s.p);
    }
}

// HLLC_Flux, mod_HLLC.f90:11-169, one reciprocal for both 1/rho and one for
// the star state; only the branch the reference selects is evaluated.
template <int DIR>
__device__ __forceinline__ void hllc(const double* ul, const double* ur, double* F) {
    const double rr = rcp(ul[0] * ur[0]);  // one reciprocal for both 1/rho
    const Prim L = c2p<DIR>(ul, ur[0] * rr);
    const Prim R = c2p<DIR>(ur, ul[0] * rr);
    const double SL = fmin(L.vn - L.c, R.vn - R.c);
    const double SR = fmax(L.vn + L.c, R.vn + R.c);
    if (!(L.adm && R.adm)) {  // :166
        const double bad = 1. / (R.vx - R.vx);
        F[0] = F[1] = F[2] = F[3] = bad;
        return;
    }
    if (SL >= 0.) {
        phys_flux<DIR>(ul, L, F);
        return;
    }
    const double numerL = SL - L.vn, numerR = SR - R.vn;
    double uStar = ul[0] * L.vn * numerL - ur[0] * R.vn * numerR;
    uStar = (R.p - L.p) + uStar;
    const double aL = ul[0] * numerL, aR = ur[0] * numerR;
    uStar = uStar * rcp(aL - aR);
    const bool left = (SL < 0.) && (uStar >= 0.);
    const bool right = (uStar < 0.) && (SR >= 0.);
    if (!left && !right) {
        phys_flux<DIR>(ur, R, F);
        return;
    }
    const double* u = left ? ul : ur;
    const Prim& s = left ? L : R;
    const double S = left ? SL : SR;
    const double a = left ? aL : aR;
    double Fk[4];
    phys_flux<DIR>(u, s, Fk);
    double st[4];
    st[0] = 1.;
    st[DIR == 0 ? 1 : 2] = uStar;
    st[DIR == 0 ? 2 : 1] = s.vt;
    const double den = S - uStar;
    const double inv = rcp(a * den);  // one reciprocal for a/den and p/a
    const double dStar = a * a * inv;
    st[3] = u[3] * s.ir + (uStar - s.vn) * (uStar + s.p * den * inv);
#pragma unroll
    for (int k = 0; k < 4; k++) F[k] = Fk[k] + S * (st[k] * dStar - u[k]);
}

// The same arithmetic with the branches turned into selects, and minima, maxima
// and signs taken from the bits (9 FP64 instructions of ~95, the same result);
// false, with F undefined, when either state is inadmissible.
template <int DIR>
__device__ __forceinline__ bool hllc_select(const double* ul, const double* ur, double* F) {
    const double rr = rcp(ul[0] * ur[0]);
    const Prim L = c2p<DIR>(ul, ur[0] * rr);
    const Prim R = c2p<DIR>(ur, ul[0] * rr);
    const double sl0 = L.vn - L.c, sl1 = R.vn - R.c, sr0 = L.vn + L.c, sr1 = R.vn + R.c;
    const double SL = key_min(sl0, sl1), SR = key_max(sr0, sr1);
    const double numerL = SL - L.vn, numerR = SR - R.vn;
    double uStar = ul[0] * L.vn * numerL - ur[0] * R.vn * numerR;
    uStar = (R.p - L.p) + uStar;
    const double aL = ul[0] * numerL, aR = ur[0] * numerR;
    uStar = uStar * rcp(aL - aR);
    const bool left = negative(SL) && nonnegative(uStar);
    const bool right = negative(uStar) && nonnegative(SR);
    const bool useL = nonnegative(SL) || left;  // whose physical flux hllc returns or corrects
    double u[4];
#pragma unroll
    for (int k = 0; k < 4; k++) u[k] = useL ? ul[k] : ur[k];
    Prim s;
    s.vn = useL ? L.vn : R.vn;
    s.vt = useL ? L.vt : R.vt;
    s.p = useL ? L.p : R.p;
    s.ir = useL ? L.ir : R.ir;
    const double S = left ? SL : SR;
    const double a = left ? aL : aR;
    double Fk[4];
    phys_flux<DIR>(u, s, Fk);
    double st[4];
    st[0] = 1.;
    st[DIR == 0 ? 1 : 2] = uStar;
    st[DIR == 0 ? 2 : 1] = s.vt;
    const double den = S - uStar;
    const double inv = rcp(a * den);
    const double dStar = a * a * inv;
    st[3] = u[3] * s.ir + (uStar - s.vn) * (uStar + s.p * den * inv);
    const bool star = left || right;
#pragma unroll
    for (int k = 0; k < 4; k++) F[k] = star ? Fk[k] + S * (st[k] * dStar - u[k]) : Fk[k];
    return L.adm && R.adm;
}
template <int DIR>
__device__ __forceinline__ void solve(int nflux, const double* ul, const double* ur, double* F) {
    if (nflux == 100) hllc<DIR>(ul, ur, F);
    else riemann<DIR>(nflux, ul, ur, F);
}

// Face flux with Gauss quadrature, mod_FE.f90:80-98: sum_g Fg*w_g from zero.
template <int DIR, int NGP>
__device__ __forceinline__ void quad_flux(const double (*uL)[4], const double (*uR)[4], const double* gw, double* F,
                                          int nflux = 100) {
    double acc[4];
    if (nflux == 100) {  // HLLC without branches; NaN flux at an inadmissible Gauss point
        bool adm = true;
#pragma unroll
        for (int g = 0; g < NGP; g++) {
            double Fg[4];
            adm = hllc_select<DIR>(uL[g], uR[g], Fg) && adm;
#pragma unroll
            for (int k = 0; k < 4; k++) acc[k] = (g == 0) ? Fg[k] * gw[0] : acc[k] + Fg[k] * gw[g];
        }
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
#pragma unroll
        for (int k = 0; k < 4; k++) F[k] = adm ? acc[k] : nan;
        return;
    }
#pragma unroll
    for (int g = 0; g < NGP; g++) {
        double Fg[4];
        solve<DIR>(nflux, uL[g], uR[g], Fg);
#pragma unroll
        for (int k = 0; k < 4; k++) acc[k] = (g == 0) ? Fg[k] * gw[0] : acc[k] + Fg[k] * gw[g];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) F[k] = acc[k];
}

// dx*dy / ((|u|+c)*dy + (|v|+c)*dx) (physics.f90:78-129 up to rounding).
__device__ __forceinline__ double cell_dt(const Cell& u, double dx, double dy) {
    const double ir = rcp(u.r);
    const double vx = u.mx * ir, vy = u.my * ir;
    const double c = root(GPM_GAMMA * pressure_ir(u, ir) * ir);
    return dx * dy * rcp((fabs(vx) + c) * dy + (fabs(vy) + c) * dx);
}

// The cell tile: every cell's 12 face states from the mirror-symmetry
// components of its 13-point stencil (GpOrbit; 80 FP64 operations per variable
// against 128 face by face), left and bottom states handed to the neighbours
// through shared memory.
constexpr int XS = 13;  // doubles per published state set (12 used, padded)

struct XyOut {
    double lo[3][4];  // left (x) or bottom (y) face states
    double hi[3][4];  // right (x) or top (y) face states
};

// Components of the stencil values of variable k around tile position (cx, cy).
struct Comp {
    double v[13];  // [Q0 Q1p Q2p Q3p Q4p Q5pp Q1m Q2m Q5mp Q3m Q4m Q5pm Q5mm]
};

__device__ __forceinline__ void components(const Cell (*tile)[XT + 5], int cx, int cy, int k, Comp& c) {
    auto q = [&](int ox, int oy) { return cell_var(tile[cy + oy][cx + ox], k); };
    const double qm1 = q(-1, 0), qp1 = q(1, 0), qm2 = q(-2, 0), qp2 = q(2, 0);
    const double qb1 = q(0, -1), qt1 = q(0, 1), qb2 = q(0, -2), qt2 = q(0, 2);
    const double a = q(-1, -1), b = q(1, -1), cc = q(-1, 1), d = q(1, 1);
    c.v[0] = q(0, 0);
    c.v[1] = qm1 + qp1;
    c.v[2] = qm2 + qp2;
    c.v[3] = qb1 + qt1;
    c.v[4] = qb2 + qt2;
    const double s1 = a + b, s2 = cc + d, d1 = a - b, d2 = cc - d;
    c.v[5] = s1 + s2;
    c.v[6] = qm1 - qp1;
    c.v[7] = qm2 - qp2;
    c.v[8] = d1 + d2;
    c.v[9] = qb1 - qt1;
    c.v[10] = qb2 - qt2;
    c.v[11] = s1 - s2;
    c.v[12] = d1 - d2;
}

// x family: left (lo) and right (hi) face states at Gauss points 0, 1, 2.
__device__ __forceinline__ void x_family(const GpOrbit& o, const Comp& c, int k, XyOut& r) {
    const double Ppp = o.x0[0] * c.v[0] + o.x0[1] * c.v[1] + o.x0[2] * c.v[2] + o.x0[3] * c.v[3] +
                       o.x0[4] * c.v[4] + o.x0[5] * c.v[5];
    const double Pmp = o.x0[6] * c.v[6] + o.x0[7] * c.v[7] + o.x0[8] * c.v[8];
    const double Ppm = o.x0[9] * c.v[9] + o.x0[10] * c.v[10] + o.x0[11] * c.v[11];
    const double Pmm = o.x0[12] * c.v[12];
    const double A = Ppp + Ppm, B = Pmp + Pmm, C = Ppp - Ppm, D = Pmp - Pmm;
    r.lo[0][k] = A + B;
    r.hi[0][k] = A - B;
    r.lo[2][k] = C + D;
    r.hi[2][k] = C - D;
    const double P1pp = o.x1[0] * c.v[0] + o.x1[1] * c.v[1] + o.x1[2] * c.v[2] + o.x1[3] * c.v[3] +
                        o.x1[4] * c.v[4] + o.x1[5] * c.v[5];
    const double P1mp = o.x1[6] * c.v[6] + o.x1[7] * c.v[7] + o.x1[8] * c.v[8];
    r.lo[1][k] = P1pp + P1mp;
    r.hi[1][k] = P1pp - P1mp;
}

// y family: bottom (lo) and top (hi) face states at Gauss points 0, 1, 2.
__device__ __forceinline__ void y_family(const GpOrbit& o, const Comp& c, int k, XyOut& r) {
    const double Ppp = o.y0[0] * c.v[0] + o.y0[1] * c.v[1] + o.y0[2] * c.v[2] + o.y0[3] * c.v[3] +
                       o.y0[4] * c.v[4] + o.y0[5] * c.v[5];
    const double Pmp = o.y0[6] * c.v[6] + o.y0[7] * c.v[7] + o.y0[8] * c.v[8];
    const double Ppm = o.y0[9] * c.v[9] + o.y0[10] * c.v[10] + o.y0[11] * c.v[11];
    const double Pmm = o.y0[12] * c.v[12];
    const double A = Ppp + Ppm, B = Pmp + Pmm, C = Ppp - Ppm, D = Pmp - Pmm;
    r.lo[0][k] = A + B;
    r.lo[2][k] = A - B;
    r.hi[0][k] = C + D;
    r.hi[2][k] = C - D;
    const double P1pp = o.y1[0] * c.v[0] + o.y1[1] * c.v[1] + o.y1[2] * c.v[2] + o.y1[3] * c.v[3] +
                        o.y1[4] * c.v[4] + o.y1[5] * c.v[5];
    const double P1pm = o.y1[6] * c.v[9] + o.y1[7] * c.v[10] + o.y1[8] * c.v[11];
    r.lo[1][k] = P1pp + P1pm;
    r.hi[1][k] = P1pp - P1pm;
}

__device__ __forceinline__ void publish(double* dst, const double (*st)[4]) {
#pragma unroll
    for (int g = 0; g < 3; g++)
#pragma unroll
        for (int k = 0; k < 4; k++) dst[4 * g + k] = st[g][k];
}

struct XySmem {
    Cell tile[XY + 5][XT + 5];
    double left[XY][XT][XS];    // left-face states of cells l0+1 .. l0+XT
    double bottom[XY][XT][XS];  // bottom-face states of rows n0+1 .. n0+XY
    double top[XY][XT][XS];     // each cell's own top-face states, parked during its x-face solve
};

// The faces of one cell tile (the first pass), halo tile loaded here.
__device__ __forceinline__ void xy_tile(const GridGeom& g, const GpWeights& w, const double* __restrict__ uin,
                                        double* __restrict__ fx, double* __restrict__ fy, int l0, int n0,
                                        XySmem& sm) {
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * XT + tx;
    for (int i = tid; i < (XT + 5) * (XY + 5); i += XT * XY) {
        const int cy = i / (XT + 5), cx = i - cy * (XT + 5);
        const int l = l0 - 2 + cx, n = n0 - 2 + cy;
        if (l >= -3 && l <= g.lf + 4 && n >= -3 && n <= g.nf + 4)
            sm.tile[cy][cx] = ld_cell(uin + 4 * cidx(g, l, n));
    }
    __syncthreads();
    const int l = l0 + tx, n = n0 + ty;
    // a cell up to (lf+1, nf+1) provides states: its stencil stays inside the padded grid
    const bool live = l <= g.lf + 1 && n <= g.nf + 1;
    XyOut xs, ys;
    if (live) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            Comp c;
            components(sm.tile, tx + 2, ty + 2, k, c);
            x_family(w.orbd, c, k, xs);
            y_family(w.orbd, c, k, ys);
        }
        if (tx > 0) publish(sm.left[ty][tx - 1], xs.lo);
        if (ty > 0) publish(sm.bottom[ty - 1][tx], ys.lo);
        publish(sm.top[ty][tx], ys.hi);
    }
    // the extra column (left states of cells l0+XT) and row (bottom states of n0+XY)
    if (ty == XY - 1 && l <= g.lf + 1 && n0 + XY <= g.nf + 1) {
        XyOut e;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            Comp c;
            components(sm.tile, tx + 2, XY + 2, k, c);
            y_family(w.orbd, c, k, e);
        }
        publish(sm.bottom[XY - 1][tx], e.lo);
    }
    if (ty == XY - 2 && tx < XY && l0 + XT <= g.lf + 1 && n0 + tx <= g.nf + 1) {
        XyOut e;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            Comp c;
            components(sm.tile, XT + 2, tx + 2, k, c);
            x_family(w.orbd, c, k, e);
        }
        publish(sm.left[tx][XT - 1], e.lo);
    }
    __syncthreads();
    if (l <= g.lf && n <= g.nf) {  // x face between (l,n) and (l+1,n)
        double uR[3][4], F[4];
        const double* src = sm.left[ty][tx];
#pragma unroll
        for (int gp = 0; gp < 3; gp++)
#pragma unroll
            for (int k = 0; k < 4; k++) uR[gp][k] = src[4 * gp + k];
        quad_flux<0, 3>(xs.hi, uR, w.gw, F);
        st_cell(fx + 4 * cidx(g, l, n), Cell{F[0], F[1], F[2], F[3]});
    }
    if (l <= g.lf && n <= g.nf) {  // y face between (l,n) and (l,n+1)
        double uL[3][4], uR[3][4], F[4];
        const double* src = sm.bottom[ty][tx];
        const double* own = sm.top[ty][tx];
#pragma unroll
        for (int gp = 0; gp < 3; gp++)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uL[gp][k] = own[4 * gp + k];
                uR[gp][k] = src[4 * gp + k];
            }
        quad_flux<1, 3>(uL, uR, w.gw, F);
        st_cell(fy + 4 * cidx(g, l, n), Cell{F[0], F[1], F[2], F[3]});
    }
}

}  // namespace ens
