// stage_kernels.cu -- the kernels of one GP-MOOD Runge-Kutta stage.
//
// Compiled twice into libgpmood.so:
//   -DGPM_EXACT=1 --fmad=false  -> namespace gpm_exact (bit-identical to the
//                                  reference's operation order)
//   -DGPM_EXACT=0 --fmad=true   -> namespace gpm_fast
//
// One stage (Forward_Euler, gp-mood-code/mod_FE.f90:20-190) runs as:
//   k_bc                  Boundary_C(Uin)                      BC.f90:10-421
//   k_flux_xy_tma         every face: GP recon + HLLC + quadrature, stored
//   (k_flux_gp)           (the first MOOD pass, mod_FE.f90:73-145); fast mode
//                         by tiles of cells, exact mode by Gauss points
//   k_update_detect       Uout = Uin + flux differences, DETECTION on every
//                         cell, troubled cells (order already lowered 5->3->1)
//                         compacted into a list
//   k_mood_loop           while the list is not empty (the MOOD loop,
//   k_mood_team           mod_FE.f90:69-174), long lists in a cooperative
//                         launch, short ones on one cluster: recompute the 4
//                         faces of each troubled cell, then Uout of its
//                         5-point cross with DETECTION there -> next list
//   k_bc                  Boundary_C(Uout)
//   k_combine_bc          SSP-RK3 combination (mod_SSP_RK3.f90:28,33) with
//                         Boundary_C(Uout) of the stage before it and, in the
//                         last, the next step's Setdt reduction
//
// Why the list-based loop equals the reference's full-grid loop: after a
// DETECTION pass the reference flags exactly the faces of troubled cells and
// the cells of their 5-point crosses (mod_subroutine_MOOD.f90:133-182), resets
// those cells to Uin, and in the next pass recomputes flagged faces and
// re-applies stored fluxes to flagged cells only.  Every other cell keeps its
// Uout.  A stored flux always equals the flux at the current orders (a face is
// recomputed whenever an adjacent order drops), so recomputing a flagged
// cell's Uout from Uin and its four current face fluxes, in the reference's
// accumulation order, reproduces the reference bit for bit.
#include "physics.cuh"
#include "fixed_recon.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <cooperative_groups.h>

#include <mutex>
#include <type_traits>

#if GPM_EXACT
#define GPM_NS gpm_exact
#else
#define GPM_NS gpm_fast
#endif

namespace GPM_NS {

__device__ __forceinline__ size_t cidx(const GridGeom& g, int l, int n) {
    return (size_t)(n + 3) * (size_t)g.nx + (size_t)(l + 3);
}

static int sm_count() {
    static std::atomic<int> sms[GPM_MAX_DEVICES];
    const int dev = gpm_device();
    int n = sms[dev].load(std::memory_order_relaxed);
    if (!n) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
        sms[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// ---------------------------------------------------------------------------
// Boundary_C, BC.f90:10-421.  Pass 1 fills the ghost columns of interior rows,
// pass 2 the ghost rows of every column (so corners come from pass 1 values,
// as in the reference's loop nest).  Each of the two passes as a launch cost
// ~3.4 us, twelve times a step.

__device__ __forceinline__ void p2c(double r, double u, double v, double p, double* out) {
    out[0] = r;
    out[1] = r * u;
    out[2] = r * v;
    out[3] = ((p / (GPM_GAMMA - 1.)) + 0.5 * r * (u * u + v * v));
}

__device__ __forceinline__ void f_dmr(double x, double y, double* r) {  // IC.f90:336-355
    const double xmin = 1. / 6;
    const double ymin = (x - xmin) * sqrt(3.);
    if (y > ymin) p2c(8., 7.1447096, -4.125, 116.5, r);
    else p2c(1.4, 0.0, 0.0, 1.0, r);
}

// The value that pass 1 gives the ghost column l <= 0 or l > lf of interior
// row n, from the interior of u.
__device__ __forceinline__ Cell bc_x_cell(const GridGeom& g, const double* __restrict__ u,
                                          const DevScalars* __restrict__ sc, int l, int n) {
    const bool right = l > g.lf;
    const int j = right ? l - g.lf - 1 : -l;  // 0..3
    auto at = [&](int ls) { return ld_cell_cg(u + 4 * cidx(g, ls, n)); };
    double w[4];
    switch (g.bc_type) {
    case 18:  // Periodic
    case 403:  // KH: periodic in x, BC.f90:394-400
        return at(right ? 1 + j : g.lf - j);
    case 20:     // Reflective: mirror, flip normal momentum
    case 402: {  // RT: reflective in x, BC.f90:344-362
        Cell c = at(right ? g.lf - j : 1 + j);
        c.mx = -c.mx;
        return c;
    }
    case 35:  // DMR: exact pre/post-shock states
        f_dmr(l * g.dx - g.dx / 2, n * g.dy - g.dy / 2, w);
        break;
    case 19:  // Dirichlet: the right states come from the host (sin), BC.f90:61-75
        if (right) return Cell{sc->bcd[j][0], sc->bcd[j][1], sc->bcd[j][2], sc->bcd[j][3]};
        p2c(3.857143, 2.629369, 0., 10.33333, w);
        break;
    case 401:  // RMI: inflow left, outflow right, BC.f90:243-256
        if (right) return at(g.lf);
        p2c(2.666666666666667, 2. * sqrt(1.4), 0., 4.5, w);
        break;
    default:  // 17 Neumann; 201, 301 Mach800 jets: outflow in x, BC.f90:137-152
        return at(right ? g.lf : 1);
    }
    return Cell{w[0], w[1], w[2], w[3]};
}

// Boundary_C's value of ghost cell (l, n): pass 1's in interior rows, else
// pass 2's, whose source columns outside the interior are pass 1's values.
// Only interior cells are read, so both passes are one kernel.
__device__ __forceinline__ Cell bc_cell(const GridGeom& g, const double* __restrict__ u,
                                        const DevScalars* __restrict__ sc, int stage, int l, int n) {
    if (n >= 1 && n <= g.nf) return bc_x_cell(g, u, sc, l, n);
    const bool top = n > g.nf;
    const int j = top ? n - g.nf - 1 : -n;
    const bool inner = l >= 1 && l <= g.lf;
    auto at = [&](int ns) { return inner ? ld_cell_cg(u + 4 * cidx(g, l, ns)) : bc_x_cell(g, u, sc, l, ns); };
    double w[4];
    switch (g.bc_type) {
    case 18:
        return at(top ? 1 + j : g.nf - j);
    case 20:
    case 401: {  // RMI: reflective in y, BC.f90:258-280
        Cell c = at(top ? g.nf - j : 1 + j);
        c.my = -c.my;
        return c;
    }
    case 35: {
        const double x = l * g.dx - g.dx / 2;
        if (top) {
            // t_rk of the stage (mod_SSP_RK3.f90:22,26,29)
            const double t_rk = stage == 0 ? sc->t : (stage == 1 ? sc->t + sc->dt : sc->t + 0.5 * sc->dt);
            const double xmin = 1. / 6 + 10. * t_rk / (0.5 * sqrt(3.)) + 1. / sqrt(3.);
            if (x < xmin) p2c(8., 7.1447096, -4.125, 116.5, w);
            else p2c(1.4, 0.0, 0.0, 1.0, w);
        } else if (x > 1. / 6) {
            Cell c = at(1 + j);
            c.my = -c.my;
            return c;
        } else {
            p2c(8., 7.1447096, -4.125, 116.5, w);
        }
        break;
    }
    case 201:
    case 301:  // outflow, then the jets (BC.f90:154-178, :199-236)
        if (fabs((l * g.dx - g.dx / 2) - 0.75) <= 0.05 && (!top || g.bc_type == 301)) {
            p2c(1.4, 0.0, top ? -800.0 : 800.0, 1.0, w);
            break;
        }
        return at(top ? g.nf : 1);
    case 402: {  // RT: hydrostatic ghosts, g = real(0.1, 4), BC.f90:364-389
        const Cell c = at(top ? g.nf - j : 1 + j);
        const double q[4] = {c.r, c.mx, c.my, c.e};
        const double grav = (double)0.1f;
        const double pr = (GPM_GAMMA - 1.) * (q[3] - (0.5 * (q[1] * q[1] + q[2] * q[2]) / q[0]));
        const double dp = 2 * j * g.dy * grav * q[0];
        p2c(q[0], q[1] / q[0], -(q[2] / q[0]), top ? pr - dp : pr + dp, w);
        break;
    }
    default:  // 17; 19, 403: Neumann in y (BC.f90:77-87, :402-413)
        return at(top ? g.nf : 1);
    }
    return Cell{w[0], w[1], w[2], w[3]};
}

// One thread per ghost cell: the 8 ghost columns of the interior rows, then
// the 8 ghost rows.
__global__ void __launch_bounds__(256) k_bc(GridGeom g, double* __restrict__ u, const DevScalars* __restrict__ sc,
                                            int stage) {
    int i = blockIdx.x * blockDim.x + threadIdx.x, l, n;
    if (i < 8 * g.nf) {
        const int k = i & 7;
        n = 1 + (i >> 3);
        l = k < 4 ? -k : g.lf + k - 3;
    } else {
        i -= 8 * g.nf;
        if (i >= 8 * g.nx) return;
        const int k = i / g.nx;
        l = i - k * g.nx - 3;
        n = k < 4 ? -k : g.nf + k - 3;
    }
    st_cell(u + 4 * cidx(g, l, n), bc_cell(g, u, sc, stage, l, n));
}

void launch_bc(const GridGeom& g, double* u, const DevScalars* sc, int stage, cudaStream_t s) {
    k_bc<<<(8 * (g.nf + g.nx) + 255) / 256, 256, 0, s>>>(g, u, sc, stage);
}

// ---------------------------------------------------------------------------
// First MOOD pass: every face of the stage (k_flux_gp; k_flux_xy in fast mode
// where it applies).

// Gauss-point states of face `face` of one cell at order index o: the fast
// kernels use the mirror-symmetric split for ngp = 3 above first order.
template <int DIR, int NP, int NGP>
__device__ __forceinline__ void recon_face(const GpWeights& w, int o, int face, const Cell* q, double (*u)[4]) {
#if !GPM_EXACT
    if constexpr (NGP == 3 && NP > 1) {
        gp_recon_sym3<DIR, NP>(w.sym[o][face], q, u);
        return;
    }
#endif
    gp_recon<NP, NGP>(&w.zt[o][face][0][0], q, u);
}

// NN_GP_MOOD_CC_ (mod_NN_GP_MOOD_CC.f90:63-70): with the reference network
// on, a face state of cell (l, n) at order 1 is the cell value itself and at
// order 3 the blend v1*U(l,n) + v2*Uh with (v1, v2) = values_NN(l, n) taken
// to double.  values_NN is (0, 1) except in column g.cc_col of rows 1..nf:
// the reference's network loop writes its outputs to values_NN(L, n, :)
// (mod_NN.f90:41,44; Fortran reads `l` there as the input count L), so the
// row's last cell leaves its softmax there.  A (0, 1) blend is applied like
// any other, as the reference does.
__device__ __forceinline__ void cc_weights(const GridGeom& g, const float* ccw, int l, int n, double* v1,
                                           double* v2) {
    *v1 = 0.0;
    *v2 = 1.0;
    if (l == g.cc_col && n >= 1 && n <= g.nf) {
        *v1 = (double)ccw[2 * n];
        *v2 = (double)ccw[2 * n + 1];
    }
}

template <int NP>
__device__ __forceinline__ void cc_blend(double v1, double v2, const Cell& c, double* u) {
    const double cv[4] = {c.r, c.mx, c.my, c.e};
#pragma unroll
    for (int k = 0; k < 4; k++) u[k] = NP == 1 ? cv[k] : v1 * cv[k] + v2 * u[k];
}

// One lane per Gauss point of a face, 32/NGP faces per warp, x faces first (a
// warp holds one direction): each lane reconstructs both sides at its point,
// solves its Riemann problem, and the face's lanes sum the quadrature by
// shuffles in Gauss-point order, quad_flux's expression, so the bits are those
// of a thread per face.  That form ran 1100 FP64 instructions in a row in the
// exact mode, 64 cycles each for a lone warp, in two launches (two directions)
// of few large CTAs: 88 us each from 48x40 up to 128^2, 393 us each at 400^2
// (71 % of the FP64 pipe: too few warps at 170 registers, and a tail per
// direction).  A third of the chain, both directions in one launch of
// 128-thread CTAs.  Stencils come through L1, whose lines a face's lanes share;
// the weights from shared memory, where lanes of different points read apart.
template <int NGP, int UORD>  // UORD: uniform order (1,3,5) or 0 = per-face from the order array
__global__ void __launch_bounds__(128, 4) k_flux_gp(StageArgs a, const __grid_constant__ GpWeights w) {
    constexpr int NO = UORD == 0 ? 3 : 1, FPW = 32 / NGP;
    __shared__ double z[NO][4][NGP][13];
    const GridGeom& g = a.g;
    for (int i = threadIdx.x; i < NO * 4 * NGP * 13; i += 128) {
        const int o = i / (4 * NGP * 13), r = i - o * (4 * NGP * 13);
        z[o][r / (NGP * 13)][r / 13 % NGP][r % 13] = w.zt[UORD == 0 ? o : UORD / 2][r / (NGP * 13)][r / 13 % NGP][r % 13];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, fl = lane / NGP, gp = lane - fl * NGP, lead = lane - gp;
    const long long nfx = (long long)(g.lf + 1) * g.nf, nfy = (long long)g.lf * (g.nf + 1);
    const long long nxw = (nfx + FPW - 1) / FPW, wi = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int dir = wi < nxw ? 0 : 1;
    const long long i = (dir == 0 ? wi : wi - nxw) * FPW + fl;
    const bool act = fl < FPW && gp < NGP && i < (dir == 0 ? nfx : nfy);
    const int len = dir == 0 ? g.lf + 1 : g.lf;
    const int row = act ? (int)(i / len) : 0;
    const int l = dir == 0 ? (act ? (int)(i - (long long)row * len) : 0) : 1 + (act ? (int)(i - (long long)row * len) : 0);
    const int n = dir == 0 ? 1 + row : row;
    const size_t c0 = cidx(g, l, n), c1 = dir == 0 ? c0 + 1 : c0 + g.nx;
    double F[4] = {0., 0., 0., 0.};
    if (act) {
        const int FL = dir == 0 ? 2 : 1, FH = dir == 0 ? 0 : 3;
        double uL[4], uR[4];
        auto states = [&](auto np, int o) {
            constexpr int NP = decltype(np)::value;
            const ptrdiff_t r = g.nx;
#pragma unroll
            for (int side = 0; side < 2; side++) {
                const double* u = a.uin + 4 * (side ? c1 : c0);
                const double* zz = &z[UORD == 0 ? o : 0][side ? FH : FL][gp][0];
                double* s = side ? uR : uL;
                Cell q[NP];
#pragma unroll
                for (int m = 0; m < NP; m++) q[m] = ld_cell(u + 4 * (st_ox(m) + r * st_oy(m)));
                gp_recon_at<NP>(zz, q, s);
                if (NP < 13 && UORD == 0 && a.ccw) {
                    double v1, v2;
                    cc_weights(g, a.ccw, l + (side && dir == 0), n + (side && dir == 1), &v1, &v2);
                    cc_blend<NP>(v1, v2, q[0], s);
                }
            }
        };
        if (UORD != 0) {
            states(std::integral_constant<int, np_of(UORD == 0 ? 1 : UORD)>{}, 0);
        } else {
            const int o = min((int)a.order[c0], (int)a.order[c1]);
            if (o >= 5) states(std::integral_constant<int, 13>{}, 2);
            else if (o >= 3) states(std::integral_constant<int, 5>{}, 1);
            else states(std::integral_constant<int, 1>{}, 0);
        }
        if (dir == 0) riemann<0>(g.num_flux, uL, uR, F);
        else riemann<1>(g.num_flux, uL, uR, F);
    }
    double acc[4];
#pragma unroll
    for (int j = 0; j < NGP; j++) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const double v = __shfl_sync(0xffffffffu, F[k], min(lead + j, 31));
            acc[k] = (j == 0) ? v * w.gw[0] : acc[k] + v * w.gw[j];
        }
    }
    if (act && gp == 0) {
#if GPM_EXACT
#pragma unroll
        for (int k = 0; k < 4; k++) acc[k] = plus_zero(acc[k]);
#endif
        st_cell((dir == 0 ? a.fx : a.fy) + 4 * c0, Cell{acc[0], acc[1], acc[2], acc[3]});
    }
}

// The Riemann solve and quadrature a face function uses; the batched form has
// its own in fast mode (batch_fast.cuh).
struct FaceMath {
#if GPM_EXACT
    template <int DIR, int NGP>
    static __device__ __forceinline__ void quad(const double (*uL)[4], const double (*uR)[4], const double* gw,
                                                double* F, int nflux) {
        quad_flux<DIR, NGP>(uL, uR, gw, F, nflux);
    }
#endif
    template <int DIR>
    static __device__ __forceinline__ void solve(int nflux, const double* uL, const double* uR, double* F) {
        riemann<DIR>(nflux, uL, uR, F);
    }
};

#if !GPM_EXACT
// ---------------------------------------------------------------------------
// Fast first pass at a uniform order 3 or 5 with 2 or 3 Gauss points: both
// face directions of a tile of cells in one CTA.  A cell's states on an axis's
// two faces come from the mirror-symmetry components of its stencil (FixOrbit)
// in fixed point, on the integer pipe (fixed_recon.cuh), so the FP64 pipe,
// which bounds this kernel, runs only the Riemann solves: at order 5 with 3
// points 126 FP64 instructions per face instead of 284 with FP64 sums.  After
// staging, a CTA turns its tile into signed mantissas (in place) and 16-bit
// exponents once.  Then, for x and for y: every cell's states go to shared
// memory, its far-face (right, top) states in its own slot and its near-face
// (left, bottom) states in the slot of the neighbour that shares the face, and
// every thread solves the face of which its cell is the low side.  Both axes
// and all four variables run the same code (an axis's frame is a pair of
// strides): unrolled, the kernel outgrew the instruction cache.  Tiles own the
// interior cells (l0..l0+XT-1, n0..n0+R-1), l0, n0 >= 1; the near-face states of
// the next column and row are computed by one warp in a second turn.  The
// faces whose low cell is a ghost (x faces (0,n), y faces (l,0)) have blocks of
// their own at the front of the grid, which stage the same tiles and solve only
// those faces (done by the low-edge tiles themselves, or by a launch of their
// own, they were 20 us of dependent FP64 at the end of a 256^2 first pass).
//
// Several small CTAs an SM keep some in the FP64 phase while others are in the
// integer phase, and hide its latency: 2048^2 Sedov, order 5, 2 steps: 20.3 ms
// with five of 4 rows, 24.5 with four, 19.6 with three of 8 rows (all with FP64 roots;
// 16.6 now).
constexpr int XT = 32, XY = 8;  // cells per tile of the batched form; XT is also the width here
constexpr int TW = XT + 6;      // tile width with halo: 3 cells below, 3 above

template <int NGP, int R>
struct XySmem {
    static constexpr int XS = 4 * NGP + 1;  // doubles per state set, padded to an odd stride
    Cell tile[R + 6][TW];                   // staged doubles, then their signed mantissas (fix_decode)
    ushort4 ex[R + 6][TW];                  // biased exponents of the four variables
    double far[R][XT][XS];                  // each cell's right (top) face states
    double near[R][XT][XS];                 // the left (bottom) face states of its right (upper) neighbour
};

// Variable k's states on the two faces of one axis of the cell at tile
// position `at`; sn, st: strides in cells along and across the axis.
template <int ORD, int NGP, class S>
__device__ __forceinline__ void recon_axis(const S& sm, const FixOrbit& o, int axis, int at, int sn, int st, int k,
                                           double* lo, double* hi) {
    constexpr int NP = np_of(ORD);
    const int off[13] = {0, -sn, sn, -st, st, -2 * sn, 2 * sn, -2 * st, 2 * st, -sn - st, sn - st, st - sn, sn + st};
    const unsigned short* ex = reinterpret_cast<const unsigned short*>(&sm.ex[0][0] + at) + k;
    const long long* q = reinterpret_cast<const long long*>(&sm.tile[0][0] + at) + k;
    int e[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) e[i] = ex[4 * off[i]];
    long long v[NP];
    const int E = fix_align<NP>(o.k[axis], e, v, [&](int i) { return q[4 * off[i]]; });
    FixHalves c[NP];
    fix_components<ORD>(v, c);
    long long l[NGP], h[NGP];
    fix_family<ORD, NGP>(o.g0[axis], o.g1[axis], c, l, h);
    const bool ok = fix_exponent_ok(E);
    const double special = __longlong_as_double(fix_special_bits(E));
#pragma unroll
    for (int g = 0; g < NGP; g++) {
        lo[g] = ok ? fix_value(l[g], E) : special;
        hi[g] = ok ? fix_value(h[g], E) : special;
    }
}

// staged: the halo tile is already in sm.tile (TMA); otherwise load it here.
// edge_axis: -1, or the axis whose low-edge faces this block solves.
template <int ORD, int NGP, int R>
__device__ __forceinline__ void xy_tile(const GridGeom& g, const FixOrbit& o, const double* gw,
                                        const double* __restrict__ uin, double* __restrict__ fx,
                                        double* __restrict__ fy, int l0, int n0, int edge_axis, XySmem<NGP, R>& sm,
                                        bool staged) {
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * XT + tx;
    if (!staged)
        for (int i = tid; i < TW * (R + 6); i += XT * R) {
            const int cy = i / TW, cx = i - cy * TW;
            const int l = l0 - 3 + cx, n = n0 - 3 + cy;
            if (l >= -3 && l <= g.lf + 4 && n >= -3 && n <= g.nf + 4)
                sm.tile[cy][cx] = ld_cell(uin + 4 * cidx(g, l, n));
        }
    __syncthreads();
    for (int i = tid; i < TW * (R + 6); i += XT * R) {
        long long* c = reinterpret_cast<long long*>(&sm.tile[0][0] + i);
        int e[4];
#pragma unroll
        for (int k = 0; k < 4; k++) c[k] = fix_decode(c[k], &e[k]);
        (&sm.ex[0][0])[i] = make_ushort4((unsigned short)e[0], (unsigned short)e[1], (unsigned short)e[2],
                                         (unsigned short)e[3]);
    }
#pragma unroll 1
    for (int axis = 0; axis < 2; axis++) {
        const int edge = edge_axis >= 0;  // an edge block: the faces below the tile's first column or row
        if (edge && axis != edge_axis) continue;
        __syncthreads();  // the tile is decoded; the states are free
        const int sn = axis == 0 ? 1 : TW, st = axis == 0 ? TW : 1;
        const int across = axis == 0 ? R : XT;  // cells of a tile's column (x) or row (y)
        // Turn 0: every cell of the tile; turn 1: the next column or row.  On the edge: the ghost column or row
        // (warp 0, far states) and the first one (warp 1, near states), face j in the slot of the tile's j-th cell.
        // A cell up to (lf+1, nf+1) provides states: its stencil stays inside the padded grid.
        int cx = tx, cy = ty;
        if (edge) {
            const int c = (tid >> 5) - 1;  // -1: ghost, 0: first
            cx = axis == 0 ? c : tx;
            cy = axis == 0 ? tx : c;
        }
#pragma unroll 1
        for (int turn = 0; turn < 2 - edge; turn++) {
            const bool mine = edge ? tid < 64 && tx < across : turn == 0 || tid < across;
            if (mine && l0 + cx <= g.lf + 1 && n0 + cy <= g.nf + 1) {
                const int px = edge ? (axis == 0 ? 0 : tx) : cx - (axis == 0);  // slot of the near states
                const int py = edge ? (axis == 0 ? tx : 0) : cy - (axis != 0);
                const bool give = edge ? tid >= 32 : px >= 0 && py >= 0, keep = edge ? tid < 32 : turn == 0;
                const int fx_ = edge ? px : cx, fy_ = edge ? py : cy;           // slot of the far states
#pragma unroll 1
                for (int k = 0; k < 4; k++) {
                    double lo[NGP], hi[NGP];
                    recon_axis<ORD, NGP>(sm, o, axis, (cy + 3) * TW + cx + 3, sn, st, k, lo, hi);
#pragma unroll
                    for (int gp = 0; gp < NGP; gp++) {
                        if (give) sm.near[py][px][4 * gp + k] = lo[gp];
                        if (keep) sm.far[fy_][fx_][4 * gp + k] = hi[gp];
                    }
                }
            }
            cx = axis == 0 ? XT : tid;
            cy = axis == 0 ? tid : R;
        }
        __syncthreads();
        // the face of low cell (l, n): the thread's own cell, or the ghost before the j-th cell of the edge
        const int sx = edge ? (axis == 0 ? 0 : tx) : tx, sy = edge ? (axis == 0 ? tx : 0) : ty;
        const int l = l0 + sx - (edge && axis == 0), n = n0 + sy - (edge && axis != 0);
        if ((!edge || tid < across) && l <= g.lf && n <= g.nf) {
            const double *uL = sm.far[sy][sx], *uR = sm.near[sy][sx];
            const int kn = 1 + axis, kt = 2 - axis;  // normal and tangential momentum
            NormalFlux acc{0., 0., 0., 0.};
            bool adm = true;
#pragma unroll
            for (int gp = 0; gp < NGP; gp++) {
                NormalFlux f;
                const double *a = uL + 4 * gp, *b = uR + 4 * gp;
                adm = hllc_normal(a[0], a[kn], a[kt], a[3], b[0], b[kn], b[kt], b[3], f) && adm;
                if (gp == 0) acc = NormalFlux{f.r * gw[0], f.n * gw[0], f.t * gw[0], f.e * gw[0]};
                else acc = NormalFlux{acc.r + f.r * gw[gp], acc.n + f.n * gw[gp], acc.t + f.t * gw[gp], acc.e + f.e * gw[gp]};
            }
            double F[4] = {acc.r, axis == 0 ? acc.n : acc.t, axis == 0 ? acc.t : acc.n, acc.e};
            nan_flux(!adm, F);
            st_cell((axis == 0 ? fx : fy) + 4 * cidx(g, l, n), Cell{F[0], F[1], F[2], F[3]});
        }
    }
}

// One face, with stencils read straight from global memory.
template <int DIR, int NP, int NGP, class M>
__device__ __forceinline__ void face_global(const GridGeom& g, const GpWeights& w, int o, const double* __restrict__ uin,
                                            size_t c0, double* F) {
    constexpr int FL = DIR == 0 ? 2 : 1;
    constexpr int FH = DIR == 0 ? 0 : 3;
    const ptrdiff_t row = g.nx;
    const size_t c1 = DIR == 0 ? c0 + 1 : c0 + g.nx;
    double uL[NGP][4], uR[NGP][4];
    {
        Cell q[NP];
#pragma unroll
        for (int m = 0; m < NP; m++) q[m] = ld_cell(uin + 4 * (c0 + st_ox(m) + row * st_oy(m)));
        recon_face<DIR, NP, NGP>(w, o, FL, q, uL);
    }
    {
        Cell q[NP];
#pragma unroll
        for (int m = 0; m < NP; m++) q[m] = ld_cell(uin + 4 * (c1 + st_ox(m) + row * st_oy(m)));
        recon_face<DIR, NP, NGP>(w, o, FH, q, uR);
    }
    M::template quad<DIR, NGP>(uL, uR, w.gw, F, g.num_flux);
}

// Edge item: faces k0 .. k0+EDGE_T-1 of the list [x faces (0,1..nf), y faces
// (1..lf,0)], one warp per item so that the few edge faces spread over many SMs.
constexpr int EDGE_T = 32;
template <class M>
__device__ __forceinline__ void edge_faces(const GridGeom& g, const GpWeights& w, const double* __restrict__ uin,
                                           double* __restrict__ fx, double* __restrict__ fy, int k0) {
    const int k = k0 + (int)threadIdx.x;
    double F[4];
    if (k < g.nf) {
        const size_t c0 = cidx(g, 0, k + 1);
        face_global<0, 13, 3, M>(g, w, 2, uin, c0, F);
        st_cell(fx + 4 * c0, Cell{F[0], F[1], F[2], F[3]});
    } else if (k < g.nf + g.lf) {
        const size_t c0 = cidx(g, k - g.nf + 1, 0);
        face_global<1, 13, 3, M>(g, w, 2, uin, c0, F);
        st_cell(fy + 4 * c0, Cell{F[0], F[1], F[2], F[3]});
    }
}

// CTAs an SM should hold: five of 4 rows (20 warps at 96 registers a thread),
// three of 8 (24 warps at 80).
constexpr int xy_ctas(int R) { return R == 8 ? 3 : 20 / R; }

// The tile of a block: the edge blocks come first (one per row of tiles for
// the x faces, one per column for the y faces), then one per tile, x fastest.
template <int R>
__device__ __forceinline__ void xy_block(int tiles_x, int tiles_y, int* l0, int* n0, int* edge) {
    const int b = (int)blockIdx.x, t = b - (tiles_x + tiles_y);
    const int by = t >= 0 ? t / tiles_x : b < tiles_y ? b : 0;
    const int bx = t >= 0 ? t - by * tiles_x : b < tiles_y ? 0 : b - tiles_y;
    *edge = t >= 0 ? -1 : b < tiles_y ? 0 : 1;
    *l0 = 1 + bx * XT;
    *n0 = 1 + by * R;
}

template <int ORD, int NGP, int R>
__global__ void __launch_bounds__(XT * R, xy_ctas(R)) k_flux_xy(StageArgs a, const __grid_constant__ GpWeights w,
                                                                int tiles_x, int tiles_y) {
    extern __shared__ __align__(16) unsigned char xy_raw[];
    XySmem<NGP, R>& sm = *reinterpret_cast<XySmem<NGP, R>*>(xy_raw);
    int l0, n0, edge;
    xy_block<R>(tiles_x, tiles_y, &l0, &n0, &edge);
    xy_tile<ORD, NGP, R>(a.g, w.orb[ORD / 2 - 1], w.gw, a.uin, a.fx, a.fy, l0, n0, edge, sm, false);
}

// ---- the same kernel with the halo tile staged by the Tensor Memory Accelerator
// The padded state is a 2-D tensor of ny rows by 4*nx doubles; one
// cp.async.bulk.tensor copies the tile's (R+6) rows of 4*(XT+6) doubles --
// exactly the row-major layout of XySmem::tile -- into this CTA's own shared
// memory and completes on an mbarrier.  The innermost start coordinate is
// 4*l0 doubles, a multiple of 32 bytes; boxes that reach past the padded
// grid on the right or top are zero-filled, and those cells feed no live
// cell's stencil.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bounded wait for phase `parity` of an mbarrier (~1 s at most).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity) {
    for (int it = 0; it < (1 << 20); it++) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

template <int ORD, int NGP, int R>
__global__ void __launch_bounds__(XT * R, xy_ctas(R)) k_flux_xy_tma(StageArgs a, const __grid_constant__ GpWeights w,
                                                                    const __grid_constant__ CUtensorMap tm,
                                                                    int tiles_x, int tiles_y) {
    extern __shared__ __align__(1024) unsigned char xy_raw[];
    using Smem = XySmem<NGP, R>;
    static_assert(sizeof(Smem) % 8 == 0, "mbarrier after the tile data");
    Smem& sm = *reinterpret_cast<Smem*>(xy_raw);
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(xy_raw + sizeof(Smem));
    int l0, n0, edge;
    xy_block<R>(tiles_x, tiles_y, &l0, &n0, &edge);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                     "r"((unsigned)sizeof(Smem::tile))
                     : "memory");
        // padded cell (l0-3, n0-3) is column l0, row n0 of the padded grid
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
            "[%4];" ::"r"(smem_addr(&sm.tile[0][0])),
            "l"(reinterpret_cast<uint64_t>(&tm)), "r"(4 * l0), "r"(n0), "r"(smem_addr(bar))
            : "memory");
    }
    __syncthreads();  // the barrier is initialised before anyone waits on it
    const bool ok = mbar_wait(bar, 0);
    if (!__syncthreads_and(ok)) {
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            atomicOr(&a.sc->status, GPM_STATUS_TMA);
            mbar_wait(bar, 0);  // once more, bounded, for the copy in flight before the CTA leaves
        }
        return;
    }
    xy_tile<ORD, NGP, R>(a.g, w.orb[ORD / 2 - 1], w.gw, a.uin, a.fx, a.fy, l0, n0, edge, sm, true);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no -lcuda).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    });
    return fn;
}

// The tile map of a padded state: ny rows of 4*nx doubles, boxes of R+6 rows
// by 4*(XT+6) doubles.  False if the CUDA driver refuses it or the state is not
// 16-byte aligned (TMA's rule for the global address).
static bool encode_tile_map(CUtensorMap* m, const double* u, const GridGeom& g, int R) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc || (reinterpret_cast<uintptr_t>(u) & 15)) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)4 * g.nx, (cuuint64_t)g.ny};
    const cuuint64_t strides[1] = {(cuuint64_t)4 * g.nx * sizeof(double)};
    const cuuint32_t box[2] = {4 * TW, (cuuint32_t)R + 6};
    const cuuint32_t estr[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double*>(u), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int ORD, int NGP, int R>
static void launch_flux_xy_t(const StageArgs& a, const GpWeights& w, cudaStream_t s) {
    static std::atomic<bool> attr[GPM_MAX_DEVICES];
    const int dev = gpm_device();
    constexpr int smem = (int)sizeof(XySmem<NGP, R>), tma_smem = smem + 8;  // + the mbarrier
    if (!attr[dev].load(std::memory_order_relaxed)) {
        cudaFuncSetAttribute(k_flux_xy<ORD, NGP, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(k_flux_xy_tma<ORD, NGP, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, tma_smem);
        attr[dev].store(true, std::memory_order_relaxed);
    }
    const int tx = (a.g.lf + XT - 1) / XT, ty = (a.g.nf + R - 1) / R;
    CUtensorMap tm;
    if (a.g.flux_tma && encode_tile_map(&tm, a.uin, a.g, R))
        k_flux_xy_tma<ORD, NGP, R><<<tx * ty + tx + ty, dim3(XT, R), tma_smem, s>>>(a, w, tm, tx, ty);
    else
        k_flux_xy<ORD, NGP, R><<<tx * ty + tx + ty, dim3(XT, R), smem, s>>>(a, w, tx, ty);
}

template <int ORD, int NGP>
static void launch_flux_xy(const StageArgs& a, const GpWeights& w, cudaStream_t s) {
    // 8-row tiles do less work twice and run 24 warps an SM for 20, but in coarser pieces: 2048^2 (36 waves of
    // them) 20.3 -> 19.6 ms per 2 steps, 701x499 (3 waves) 1.23 -> 1.25, 397x203 radius 1 1.08 -> 1.21.
    const long long tiles8 = (long long)((a.g.lf + XT - 1) / XT) * ((a.g.nf + 7) / 8);
    if (tiles8 >= 8LL * xy_ctas(8) * sm_count()) launch_flux_xy_t<ORD, NGP, 8>(a, w, s);
    else launch_flux_xy_t<ORD, NGP, 4>(a, w, s);
}
#endif

template <int NGP>
void launch_flux_ngp(const StageArgs& a, const GpWeights& w, cudaStream_t s) {
    constexpr int FPW = 32 / NGP;
    const long long nfx = (long long)(a.g.lf + 1) * a.g.nf, nfy = (long long)a.g.lf * (a.g.nf + 1);
    const unsigned grid = (unsigned)(((nfx + FPW - 1) / FPW + (nfy + FPW - 1) / FPW + 3) / 4);
    if (!a.uniform_order) k_flux_gp<NGP, 0><<<grid, 128, 0, s>>>(a, w);
    else if (a.g.mord == 5) k_flux_gp<NGP, 5><<<grid, 128, 0, s>>>(a, w);
    else if (a.g.mord == 3) k_flux_gp<NGP, 3><<<grid, 128, 0, s>>>(a, w);
    else k_flux_gp<NGP, 1><<<grid, 128, 0, s>>>(a, w);
}

int launch_flux_all(const StageArgs& a, const GpWeights& w, cudaStream_t s) {
#if !GPM_EXACT
    if (a.uniform_order && a.g.num_flux == 100 && a.g.mord >= 3 && (a.g.ngp == 2 || a.g.ngp == 3) &&
        w.orb[a.g.mord / 2 - 1].ok) {
        if (a.g.mord == 5 && a.g.ngp == 3) launch_flux_xy<5, 3>(a, w, s);
        else if (a.g.mord == 5) launch_flux_xy<5, 2>(a, w, s);
        else if (a.g.ngp == 3) launch_flux_xy<3, 3>(a, w, s);
        else launch_flux_xy<3, 2>(a, w, s);
        return 1;
    }
#endif
    switch (a.g.ngp) {
    case 1: launch_flux_ngp<1>(a, w, s); break;
    case 2: launch_flux_ngp<2>(a, w, s); break;
    case 3: launch_flux_ngp<3>(a, w, s); break;
    case 4: launch_flux_ngp<4>(a, w, s); break;
    default: launch_flux_ngp<5>(a, w, s); break;
    }
    return 1;
}

// ---------------------------------------------------------------------------
// Flux-difference update of one cell in the reference's accumulation order
// (the n-outer, l-inner face loop of mod_FE.f90:75-145 visits, for cell
// (l,n): the y face below, the x face to the left, the x face to the right,
// the y face above).
__device__ __forceinline__ Cell cell_update(const GridGeom& g, const double* __restrict__ uin,
                                            const double* __restrict__ fx, const double* __restrict__ fy,
                                            size_t c, double qx, double qy) {
    const Cell u = ld_cell(uin + 4 * c);
    const Cell fb = ld_cell_cg(fy + 4 * (c - g.nx));
    const Cell fl = ld_cell_cg(fx + 4 * (c - 1));
    const Cell fr = ld_cell_cg(fx + 4 * c);
    const Cell ft = ld_cell_cg(fy + 4 * c);
    Cell o;
    o.r = u.r + qy * fb.r;    o.mx = u.mx + qy * fb.mx;   o.my = u.my + qy * fb.my;   o.e = u.e + qy * fb.e;
    o.r = o.r + qx * fl.r;    o.mx = o.mx + qx * fl.mx;   o.my = o.my + qx * fl.my;   o.e = o.e + qx * fl.e;
    o.r = o.r - qx * fr.r;    o.mx = o.mx - qx * fr.mx;   o.my = o.my - qx * fr.my;   o.e = o.e - qx * fr.e;
    o.r = o.r - qy * ft.r;    o.mx = o.mx - qy * ft.mx;   o.my = o.my - qy * ft.my;   o.e = o.e - qy * ft.e;
    return o;
}

// Warp-aggregated append of flagged cells to a list.
__device__ __forceinline__ void list_append(bool flag, int* __restrict__ list, int* __restrict__ count, int value) {
    const unsigned act = __activemask();
    const unsigned m = __ballot_sync(act, flag);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(act) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(act, base, leader);
    if (flag) list[base + __popc(m & ((1u << lane) - 1))] = value;
}

// Position of the calling thread in an order that fills whole warps with
// consecutive work items and deals the warps round-robin over the CTAs (one
// or a few per SM).  An FP64 instruction costs the SM the same time whether
// 1 or 32 lanes of the warp are active, so a short list must pack its items
// into as few warps as possible, and spread those warps over the SMs.
__device__ __forceinline__ int pack_tid() {
    return (((threadIdx.x >> 5) * gridDim.x + blockIdx.x) << 5) + (threadIdx.x & 31);
}

// Face item i of the 4*nt faces of nt troubled cells: the x faces come first
// (item 2j: left face of cell j, 2j+1: its right face), then the y faces
// (below, above), so the lanes of a warp share one direction.
__device__ __forceinline__ int face_item(int i, int nt, int* dir, int* side) {
    const int x = i < 2 * nt ? 1 : 0;
    const int j = x ? i : i - 2 * nt;
    *dir = x ? 0 : 1;
    *side = j & 1;
    return j >> 1;
}

// The order cascade of a troubled cell, mod_subroutine_MOOD.f90:159-163
// (5 -> 3, 3 -> 1).  It is applied by the thread that finds the cell troubled,
// when it lists the cell: no other thread reads that cell's order before the
// next pass's faces, which come after a grid barrier or a kernel boundary.
__device__ __forceinline__ void cascade_order(int8_t* o) {
    const int v = *o;
    *o = (int8_t)(v == 3 ? 1 : (v > 3 ? 3 : v));
}

// Uout of every cell and DETECTION on it (mood_troubled's decision).  The
// cells whose new density breaks the DMP bound (mood_uout_part 2) need up to
// ~150 more FP64 instructions; run by the threads that found them they cost
// their whole warp that much (34.6 us of a 256^2 2DRP3 stage), so a CTA lists
// them in shared memory and runs the remaining tests on full warps: both
// halves of the shock detector at once on different warps, then both U2 tests
// of the cells that it left.
struct DetectSmem {
    int n[2];               // cells in each list
    short list[2][256];     // candidates; those left by the shock detector
    bool hit[2][256];       // shock_flow, shock_grad; U2 smooth in x, in y
    bool troubled[256];
};

__global__ void __launch_bounds__(256) k_update_detect(StageArgs a, const __grid_constant__ GpWeights w, int cur) {
    __shared__ DetectSmem sm;
    const GridGeom& g = a.g;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const int l = 1 + blockIdx.x * 32 + threadIdx.x, n = 1 + blockIdx.y * 8 + threadIdx.y;
    const bool in = l <= g.lf && n <= g.nf;
    const bool mood = g.method == 2 || g.method == 203;
    const size_t c = cidx(g, l, n);
    if (tid < 2) sm.n[tid] = 0;
    int part = 0;
    if (in) {
        const Cell uo = cell_update(g, a.uin, a.fx, a.fy, c, a.sc->qx, a.sc->qy);
        st_cell(a.uout + 4 * c, uo);
        if (mood) {
            const int o = a.uniform_order ? g.mord : (int)a.order[c];
            if (o > 1) part = mood_uout_part(uo, a.uin + 4 * c, g.nx, g);
            else if (inadmissible(uo)) atomicOr(&a.sc->status, GPM_STATUS_NAN);
        }
    }
    bool trb = part == 1;
    if (mood && __syncthreads_or(part == 2)) {  // most CTAs have none and leave with this one barrier
        sm.troubled[tid] = false;
        if (part == 2) sm.list[0][atomicAdd(&sm.n[0], 1)] = (short)tid;
        __syncthreads();
        // two tests at a time on the listed cells, one per warp: test t of chunk i is warp task 2*i + t
        const int warp = tid >> 5, lane = tid & 31;
#pragma unroll 1
        for (int round = 0; round < 2; round++) {
            const int m = sm.n[round];
            for (int task = warp; task < 2 * ((m + 31) / 32); task += 8) {
                const int t = task & 1, j = (task >> 1) * 32 + lane;
                if (j < m) {
                    const int i = sm.list[round][j];
                    const double* u = a.uin + 4 * cidx(g, 1 + blockIdx.x * 32 + (i & 31), 1 + blockIdx.y * 8 + (i >> 5));
                    if (round == 0)
                        sm.hit[t][j] = t == 0 ? mood_shock_flow_part(u, g.nx, g) : mood_shock_grad_part(u, g.nx, g);
                    else
                        sm.hit[t][j] = t == 0 ? mood_u2_smooth<0>(u, g.nx, g, w.d2x) : mood_u2_smooth<1>(u, g.nx, g, w.d2y);
                }
            }
            __syncthreads();
            if (tid < m) {
                const int i = sm.list[round][tid];
                if (round == 0) {
                    if (sm.hit[0][tid] && sm.hit[1][tid]) {
                        if (g.u2) sm.list[1][atomicAdd(&sm.n[1], 1)] = (short)i;
                        else sm.troubled[i] = true;
                    }
                } else {
                    sm.troubled[i] = !(sm.hit[0][tid] || sm.hit[1][tid]);
                }
            }
            __syncthreads();
        }
        trb = trb || sm.troubled[tid];
    }
    if (in) {
        if (a.uniform_order) a.order[c] = (int8_t)(!trb ? g.mord : g.mord == 3 ? 1 : 3);  // CellGPO = mord, :48, lowered
        else if (trb) cascade_order(&a.order[c]);
    }
    list_append(trb, a.tlist[cur], &a.sc->ntrb[cur], (int)c);
}

void launch_update_detect(const StageArgs& a, const GpWeights& w, int cur, cudaStream_t s) {
    const dim3 grid((a.g.lf + 31) / 32, (a.g.nf + 7) / 8), blk(32, 8);
    k_update_detect<<<grid, blk, 0, s>>>(a, w, cur);
}

// ---------------------------------------------------------------------------
// MOOD passes 2, 3, ... on the troubled list only.

constexpr int LIST_CTAS_PER_SM = 4;

// The MOOD face phase, split by Gauss point.  A pass's face list is short
// (the faces of the cells lowered in the previous pass), so the SMs hold one
// or two warps each and a pass waits on one warp's chain of dependent FP64
// instructions.  NGP consecutive lanes share a face: each reconstructs both
// sides at its own Gauss point (gp_recon_at, the per-point sum of
// mod_GP_MOOD.f90:61) and solves that point's Riemann problem; the face's
// lanes gather the NGP fluxes by shuffles and sum them in Gauss-point order
// with quad_flux's expression, and the first lane stores the face.  The chain
// is one Gauss point's work instead of the face's.  A listed cell was lowered
// when it was listed, so its faces are at order <= 3; the 13-point branch only
// keeps the function total.
struct FaceGp {
    double F[4];        // this lane's Gauss-point flux
    double* out;        // the face's stored flux
    const double* gw;   // Gauss weights
};

// The two face states of one Gauss point at order NP (stencil straight from
// global memory).
template <int DIR, int NP>
__device__ __forceinline__ void face_gp_states(const GridGeom& g, const GpWeights& w, int o,
                                               const double* __restrict__ uin, size_t c0, int gp, double* uL,
                                               double* uR, const float* ccw) {
    constexpr int FL = DIR == 0 ? 2 : 1;
    constexpr int FH = DIR == 0 ? 0 : 3;
    constexpr int hx = DIR == 0 ? 1 : 0, hy = DIR == 0 ? 0 : 1;
    const ptrdiff_t row = g.nx;
    const size_t c1 = DIR == 0 ? c0 + 1 : c0 + g.nx;
    const int l0 = (int)(c0 % (size_t)g.nx) - 3, n0 = (int)(c0 / (size_t)g.nx) - 3;  // low cell (l, n)
    {
        Cell q[NP];
#pragma unroll
        for (int m = 0; m < NP; m++) q[m] = ld_cell(uin + 4 * (c0 + st_ox(m) + row * st_oy(m)));
        gp_recon_at<NP>(&w.zt[o][FL][gp][0], q, uL);
        if (ccw) {
            double v1, v2;
            cc_weights(g, ccw, l0, n0, &v1, &v2);
            cc_blend<NP>(v1, v2, q[0], uL);
        }
    }
    {
        Cell q[NP];
#pragma unroll
        for (int m = 0; m < NP; m++) q[m] = ld_cell(uin + 4 * (c1 + st_ox(m) + row * st_oy(m)));
        gp_recon_at<NP>(&w.zt[o][FH][gp][0], q, uR);
        if (ccw) {
            double v1, v2;
            cc_weights(g, ccw, l0 + hx, n0 + hy, &v1, &v2);
            cc_blend<NP>(v1, v2, q[0], uR);
        }
    }
}

// Lanes of one warp may hold faces of different orders: only the
// reconstruction branches on the order, and the Riemann solve runs once for
// the whole warp after the branches rejoin (an FP64 warp instruction costs
// its SM partition ~64 cycles however many lanes are active, so a solve in
// each branch would double the pass's critical path).
template <int DIR, class M = FaceMath>
__device__ __forceinline__ void face_gp_any(const StageArgs& a, const GpWeights& w, size_t c0, int gp, FaceGp& f) {
    const GridGeom& g = a.g;
    const size_t c1 = DIR == 0 ? c0 + 1 : c0 + g.nx;
    const int o = min((int)a.order[c0], (int)a.order[c1]);
    double uL[4], uR[4];
    if (o >= 5) face_gp_states<DIR, 13>(g, w, 2, a.uin, c0, gp, uL, uR, nullptr);
    else if (o >= 3) face_gp_states<DIR, 5>(g, w, 1, a.uin, c0, gp, uL, uR, a.ccw);
    else face_gp_states<DIR, 1>(g, w, 0, a.uin, c0, gp, uL, uR, a.ccw);
    M::template solve<DIR>(g.num_flux, uL, uR, f.F);
    f.out = (DIR == 0 ? a.fx : a.fy) + 4 * c0;
    f.gw = w.gw;
}

// Faces 0 .. nf-1 dealt to whole warps (stid: pack_tid, gstride: threads of
// the grid); item(i, gp, f) fills face i's Gauss point gp.  Faces 0 .. n0-1
// (the x faces) and n0 .. nf-1 (the y faces) start on warp boundaries, so no
// warp runs both directions' code.  Every lane of a warp runs the same trip
// count, so the shuffles see full warps.
template <int NGP, class Item>
__device__ __forceinline__ void face_phase_gp(int nf, int n0, int stid, int gstride, Item item) {
    constexpr int FPW = 32 / NGP;  // faces per warp
    const int lane = threadIdx.x & 31, fl = lane / NGP, gp = lane - fl * NGP, lead = lane - gp;
    const int w0 = (n0 + FPW - 1) / FPW, nw = w0 + (nf - n0 + FPW - 1) / FPW;
    for (int wi = stid >> 5; wi < nw; wi += gstride >> 5) {
        const int i = wi < w0 ? wi * FPW + fl : n0 + (wi - w0) * FPW + fl;
        const bool act = fl < FPW && i < (wi < w0 ? n0 : nf);
        FaceGp f;
        f.F[0] = f.F[1] = f.F[2] = f.F[3] = 0.0;
        f.out = nullptr;
        f.gw = nullptr;
        if (act) item(i, gp, f);
        double acc[4];
#pragma unroll
        for (int j = 0; j < NGP; j++) {
            const int src = min(lead + j, 31);
            const double wj = act ? f.gw[j] : 0.0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double v = __shfl_sync(0xffffffffu, f.F[k], src);
                acc[k] = (j == 0) ? v * wj : acc[k] + v * wj;
            }
        }
        if (act && gp == 0) {
#if GPM_EXACT
#pragma unroll
            for (int k = 0; k < 4; k++) acc[k] = plus_zero(acc[k]);
#endif
            st_cell(f.out, Cell{acc[0], acc[1], acc[2], acc[3]});
        }
    }
}

template <int NGP>
__global__ void __launch_bounds__(128) k_mood_faces(StageArgs a, const __grid_constant__ GpWeights w, int cur) {
    const int nt = a.sc->ntrb[cur];
    // 4 faces per troubled cell: x faces (l-1,n), (l,n), y faces (l,n-1), (l,n)
    face_phase_gp<NGP>(4 * nt, 2 * nt, pack_tid(), gridDim.x * blockDim.x, [&](int i, int gp, FaceGp& f) {
        int dir, side;
        const size_t c = (size_t)a.tlist[cur][face_item(i, nt, &dir, &side)];
        if (dir == 0) face_gp_any<0>(a, w, side == 0 ? c - 1 : c, gp, f);
        else face_gp_any<1>(a, w, side == 0 ? c - a.g.nx : c, gp, f);
    });
}

// ---------------------------------------------------------------------------
// The whole MOOD loop on the device: one cooperative launch runs passes 2, 3,
// ... until the troubled list is empty, with a grid barrier after each of the
// two phases of a pass (faces, crosses; the cascade is applied when a cell is
// listed).  Every CTA is co-resident
// (cooperative launch), so the barrier cannot wait on an unscheduled CTA; its
// spin is still bounded, and a timeout records GPM_STATUS_BARRIER and makes
// every CTA leave.

// Threads per CTA of the cooperative MOOD loops: one 16-warp CTA per SM
// keeps the barrier's arrival count at the SM count.
constexpr int MOOD_THREADS = 512;

// Arrivals are counted up and never reset: every launch adds a multiple of the
// grid's size, and before its first barrier opens a CTA can see at most one
// grid's worth of arrivals above that, so the count rounded down to a multiple
// is where the launch began.  One release-add and polls of the same word: two
// trips to L2 instead of the four of a count, a reset and a generation word
// (4.8k cycles a barrier at best before).
struct GridWait {
    unsigned long long next;  // arrivals that open the next barrier
};

__device__ __forceinline__ GridWait grid_start(GridBar* b) {
    unsigned long long c;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(&b->count) : "memory");
    return GridWait{(c / gridDim.x + 1) * gridDim.x};
}

__device__ __forceinline__ bool grid_sync(GridBar* b, GridWait& w) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const int lim = *(volatile int*)&b->limit;
        const long long max_it = lim > 0 ? lim : (1LL << 22);  // ~1 s: far beyond any pass
        __threadfence();
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&b->count), "l"(1ull) : "memory");
        long long it = 0;
        for (;;) {
            unsigned long long c;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(&b->count) : "memory");
            if (c >= w.next) break;
            if (++it > max_it) {
                atomicExch(&b->err, 1);
                break;
            }
        }
        __threadfence();
    }
    w.next += gridDim.x;
    __syncthreads();
    return *(volatile int*)&b->err == 0;
}

// One-CTA passes of the batched loop: a pass with at most BatchArgs::mood_solo
// cells runs in CTA 0 alone with CTA barriers.  Every CTA reads the same count
// after a grid barrier, so all take the switch at the same pass; the others
// leave and CTA 0 runs the loop to its end (a list that grows again is still
// done, by one CTA's threads).
__device__ __forceinline__ bool mood_sync(GridBar* b, GridWait& w, bool solo) {
    if (solo) {
        __syncthreads();
        return true;
    }
    return grid_sync(b, w);
}

// A pass of the MOOD loop.  It is a few chains of dependent FP64 instructions,
// each ~64 cycles for a lone warp however few of its lanes are active, and
// trips to L2 of ~1k cycles, so the chains are cut over lanes and warps:
//  * a face's Gauss point takes two lanes, one per side: each reconstructs its
//    side's state and its primitive quantities; they swap them by shuffles,
//    both run the Riemann join, and the face's lanes sum the quadrature, one
//    variable a lane (~70 instructions in a row for ~112 on one lane; measured
//    in a pass of 3 cells: sums 1.9k cycles, side 1.0k, join 2.0k, quadrature 0.8k,
//    the same through shared memory);
//  * what a cross needs of Uin alone (the shock detector's halves, U2 in x and
//    in y; in the team also the density bounds and which list entry takes a
//    shared cell) runs beside the faces on warps of its own, so that after the
//    barrier only the update, positivity and two comparisons are left, one lane
//    a cross cell or, for up to TEAM_QUAD of them, one a variable.
// Passes over more than GridGeom::mood_solo cells run on all SMs with grid
// barriers (k_mood_loop).  Shorter ones run on one thread-block cluster (the
// "team", k_mood_team) with cluster barriers (~1k cycles with what they wait for, against ~4k):
// 8 SMs take 32 warps side by side, and CTA 0 runs the cells.  The team's lists
// live in every member's shared memory (and in the global list, which a longer
// one is read from), the tests' results in CTA 0's, through distributed shared
// memory.  A 512x128 DMR, 30 steps, 42 ms with one-CTA passes: 22.5 ms so; 23.8
// with 4 CTAs, 24.3 with lists of up to 160 cells here, 22.7 with up to 60.
constexpr int TEAM = 8;                  // CTAs of the cluster
constexpr int TEAM_CROSS = 512;          // cross cells whose tests run beside the faces (one per thread of CTA 0)
constexpr int TEAM_LIST_CAP = 1024;
// Up to here a cross cell is updated by four lanes (4 FP64 instructions in a row
// for 16, the tests after it on every lane): at most two warps per SM quarter; 128
// is as fast.
constexpr int TEAM_QUAD = 64;

struct TeamSmem {
    int list[2][TEAM_LIST_CAP];
    int count[2];                        // the team's count: appended to in CTA 0, then copied to every member
    bool flag[4][TEAM_CROSS];            // shock flow half, pressure-jump half, U2 smooth in x, in y
    int cross[TEAM_CROSS];               // the cross cell; -1: outside, or another entry's
    Bound lo[TEAM_CROSS], hi[TEAM_CROSS];  // its density bounds; lo > hi: none
    double z3[4][GPM_MAXGP][5];          // order-3 weights, read by lanes of mixed faces and Gauss points
    double z1[4][GPM_MAXGP];             // order 1
};

__device__ __forceinline__ void team_sync() {  // every thread arrives for itself: no assumption on convergence
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
    __syncwarp();
}

// The Uin-only test t of a cross cell.
__device__ __forceinline__ bool cross_test(const GridGeom& g, const GpWeights& w, const double* u, int t) {
    return t == 0   ? mood_shock_flow_part(u, g.nx, g)
           : t == 1 ? mood_shock_grad_part(u, g.nx, g)
           : t == 2 ? mood_u2_smooth<0>(u, g.nx, g, w.d2x)
                    : mood_u2_smooth<1>(u, g.nx, g, w.d2y);
}

// Warp task `task` of the 4*nt faces of the listed cells.
template <int NGP>
__device__ __forceinline__ void team_faces(const StageArgs& a, const GpWeights& w, const TeamSmem& sm, const int* lst,
                                           int nt, int task) {
    constexpr int LPF = 2 * NGP, FPW = 32 / LPF;  // lanes per face, faces per warp
    const GridGeom& g = a.g;
    const int lane = threadIdx.x & 31, fl = lane / LPF, j = lane - fl * LPF, gp = j >> 1, side = j & 1;
    const int base = lane - j, i = task * FPW + fl;
    const bool act = fl < FPW && i < 4 * nt;
    int dir, sd;
    // idle lanes repeat the warp's last face: another face's order would cost the
    // warp that order's sums too (one at order 5: 52 instructions, 3.3k cycles)
    const int lcell = *(volatile const int*)(lst + face_item(min(task * FPW + min(fl, FPW - 1), 4 * nt - 1), nt, &dir, &sd));
    const size_t step = dir == 0 ? (size_t)1 : (size_t)g.nx;
    const size_t c0 = (size_t)lcell - (sd == 0 ? step : 0);
    const size_t cs = c0 + (side ? step : 0);                                     // this lane's cell
    const int face = dir == 0 ? (side ? 0 : 2) : (side ? 3 : 1);
    const ptrdiff_t row = g.nx;
    Cell q[5];  // in flight with the orders: listed cells' faces are at order 3 or 1
#pragma unroll
    for (int m = 0; m < 5; m++) q[m] = ld_cell(a.uin + 4 * (cs + st_ox(m) + row * st_oy(m)));
    const int o = min((int)__ldcg(a.order + c0), (int)__ldcg(a.order + c0 + step));
    double u[4];
    if (o >= 5) {  // not reached by listed cells; keeps the function total
        Cell q5[13];
#pragma unroll
        for (int m = 0; m < 13; m++) q5[m] = ld_cell(a.uin + 4 * (cs + st_ox(m) + row * st_oy(m)));
        gp_recon_at<13>(&w.zt[2][face][gp][0], q5, u);
    } else {
        if (o >= 3) gp_recon_at<5>(&sm.z3[face][gp][0], q, u);
        else gp_recon_at<1>(&sm.z1[face][gp], q, u);
        if (a.ccw) {
            double v1, v2;
            cc_weights(g, a.ccw, (int)(cs % (size_t)g.nx) - 3, (int)(cs / (size_t)g.nx) - 3, &v1, &v2);
            if (o >= 3) cc_blend<5>(v1, v2, q[0], u);
            else cc_blend<1>(v1, v2, q[0], u);
        }
    }
    auto swap = [](double x) { return __shfl_xor_sync(0xffffffffu, x, 1); };  // the other side's lane
    double F[4];
    if (g.num_flux == 100) {
#if GPM_EXACT
        const Prim mine = c2p_dyn(u, dir);
        Prim other;
        other.vn = swap(mine.vn);
        other.vt = swap(mine.vt);
        other.p = swap(mine.p);
        other.c = swap(mine.c);
        other.vx = swap(mine.vx);
        other.adm = __shfl_xor_sync(0xffffffffu, (int)mine.adm, 1) != 0;
        double uo[4], ul[4], ur[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uo[k] = swap(u[k]);
            ul[k] = side ? uo[k] : u[k];
            ur[k] = side ? u[k] : uo[k];
        }
        hllc_join(ul, ur, side ? other : mine, side ? mine : other, dir, F);
#else
        const Side mine = hllc_side(u[0], dir ? u[2] : u[1], dir ? u[1] : u[2], u[3]);
        const Side other{swap(mine.r), swap(mine.n), swap(mine.t), swap(mine.e),
                         swap(mine.v), swap(mine.w), swap(mine.p), swap(mine.c)};
        NormalFlux f;
        hllc_join(side ? other : mine, side ? mine : other, f);
        F[0] = f.r;
        F[1] = dir ? f.t : f.n;
        F[2] = dir ? f.n : f.t;
        F[3] = f.e;
        nan_flux(!(side_ok(mine) && side_ok(other)), F);
#endif
    } else {
        double ul[4], ur[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const double x = swap(u[k]);
            ul[k] = side ? x : u[k];
            ur[k] = side ? u[k] : x;
        }
        if (dir == 0) riemann<0>(g.num_flux, ul, ur, F);
        else riemann<1>(g.num_flux, ul, ur, F);
    }
    // quadrature (quad_flux's expression): variable k on lane k of the face; two rounds of two with one Gauss point
#pragma unroll
    for (int k0 = 0; k0 < 4; k0 += (LPF < 4 ? LPF : 4)) {
        double acc = 0.;
#pragma unroll
        for (int gg = 0; gg < NGP; gg++) {
            double x = 0.;
#pragma unroll
            for (int k = 0; k < (LPF < 4 ? LPF : 4); k++) {
                const double y = __shfl_sync(0xffffffffu, F[k0 + k], min(base + 2 * gg, 31));
                if (j == k) x = y;
            }
            acc = gg == 0 ? x * w.gw[0] : acc + x * w.gw[gg];
        }
#if GPM_EXACT
        acc = plus_zero(acc);
#endif
        if (act && j < (LPF < 4 ? LPF : 4)) __stcg((dir == 0 ? a.fx : a.fy) + 4 * c0 + k0 + j, acc);
    }
}

// Cross cell k of listed cell t; false outside the interior.
__device__ __forceinline__ bool cross_cell(const GridGeom& g, int t, int k, int* c) {
    *c = k == 0 ? t - g.nx : k == 1 ? t - 1 : k == 2 ? t : k == 3 ? t + 1 : t + g.nx;
    const int n = *c / g.nx - 3, l = *c - (n + 3) * g.nx - 3;
    return l >= 1 && l <= g.lf && n >= 1 && n <= g.nf;
}

// The update of one cross cell and the decision on it: the last half of
// mood_troubled.  flags: the Uin-only tests' results as bits, or -1 to run them
// here.  Returns whether the cell is troubled (its order is lowered then).
__device__ __forceinline__ bool cross_update(const StageArgs& a, const GpWeights& w, int c, int flags, double qx,
                                             double qy) {
    const GridGeom& g = a.g;
    const double* uin = a.uin + 4 * (size_t)c;
    const int o = (int)__ldcg(a.order + c);
    const Cell uo = cell_update(g, a.uin, a.fx, a.fy, (size_t)c, qx, qy);
    st_cell(a.uout + 4 * (size_t)c, uo);
    if (o <= 1) {
        if (inadmissible(uo)) atomicOr(&a.sc->status, GPM_STATUS_NAN);
        return false;
    }
    const int r = mood_uout_part(uo, uin, g.nx, g);
    bool trb = r == 1;
    if (r == 2) {
        if (flags >= 0) trb = (flags & 3) == 3 && !(g.u2 && (flags & 12));
        else trb = mood_shock_part(uin, g.nx, g) && !(g.u2 && (mood_u2_smooth<0>(uin, g.nx, g, w.d2x) ||
                                                               mood_u2_smooth<1>(uin, g.nx, g, w.d2y)));
    }
    if (trb) __stcg(a.order + c, (int8_t)(o == 3 ? 1 : 3));  // the cascade of cascade_order
    return trb;
}

// What a team pass needs of cross i before the fluxes: its cell, if this entry
// takes it, and the density bounds.  A cross cell that several listed cells share
// is taken by the first of them (a scan of a short list), or by whoever stamps
// it first.
__device__ __forceinline__ bool team_own(const StageArgs& a, const int* lst, int nt, int i, unsigned pid, int* c) {
    const int q = i / 5, nx = a.g.nx;
    if (!cross_cell(a.g, lst[q], i - 5 * q, c)) return false;
    if (nt > 24) return atomicExch(&a.stamp[*c], pid) != pid;
    bool own = true;
    for (int q2 = 0; q2 < q; q2++) {
        const int d = *c - lst[q2];
        if (d == 0 || d == 1 || d == -1 || d == nx || d == -nx) own = false;
    }
    return own;
}
__device__ __forceinline__ void team_prepare(const StageArgs& a, TeamSmem* sm0, const int* lst, int nt, int i,
                                             unsigned pid) {
    int c;
    const bool own = team_own(a, lst, nt, i, pid, &c);
    sm0->cross[i] = own ? c : -1;
    if (!own) return;
    Bound lo = 0, hi = 0;
    const bool dmp = a.g.dmp && mood_bounds(a.uin + 4 * (size_t)c, a.g.nx, a.g, &lo, &hi);
    sm0->lo[i] = dmp ? lo : (Bound)1;
    sm0->hi[i] = dmp ? hi : (Bound)0;
}

// cross_update of a prepared cross i by L lanes (1 or 4, this one's variable k);
// all return the same.
template <int L>
__device__ __forceinline__ bool cross_finish(const StageArgs& a, const TeamSmem& sm, int i, int k, double qx,
                                             double qy) {
    const GridGeom& g = a.g;
    const int c = sm.cross[i], o = (int)__ldcg(a.order + c);
    Cell uo;
    if (L == 4) {  // cell_update's sum for variable k
        const size_t at = 4 * (size_t)c + k, row = 4 * (size_t)g.nx;
        const double fb = __ldcg(a.fy + at - row), fl = __ldcg(a.fx + at - 4);
        const double fr = __ldcg(a.fx + at), ft = __ldcg(a.fy + at);
        double x = __ldg(a.uin + at);
        x = x + qy * fb;
        x = x + qx * fl;
        x = x - qx * fr;
        x = x - qy * ft;
        a.uout[at] = x;
        const unsigned m = 0xfu << (threadIdx.x & 28);
        uo.r = __shfl_sync(m, x, 0, 4);
        uo.mx = __shfl_sync(m, x, 1, 4);
        uo.my = __shfl_sync(m, x, 2, 4);
        uo.e = __shfl_sync(m, x, 3, 4);
    } else {
        uo = cell_update(g, a.uin, a.fx, a.fy, (size_t)c, qx, qy);
        st_cell(a.uout + 4 * (size_t)c, uo);
    }
    if (o <= 1) {
        if (inadmissible(uo)) atomicOr(&a.sc->status, GPM_STATUS_NAN);
        return false;
    }
    bool trb = !mood_positive(uo);
    const Bound key = bound_key(uo.r);
    if (!trb && sm.lo[i] <= sm.hi[i] && (key > sm.hi[i] || key < sm.lo[i]))
        trb = sm.flag[0][i] && sm.flag[1][i] && !(g.u2 && (sm.flag[2][i] || sm.flag[3][i]));
    if (trb && k == 0) __stcg(a.order + c, (int8_t)(o == 3 ? 1 : 3));  // the cascade of cascade_order
    return trb;
}

// The crosses of a team pass, by CTA 0; those from ncross on were not prepared.
__device__ __forceinline__ void team_cells(const StageArgs& a, const GpWeights& w, TeamSmem& sm, const int* lst,
                                           int cur, int nt, int ncross, unsigned pid, double qx, double qy) {
    const int nxt = cur ^ 1, total = 5 * nt, lane = threadIdx.x & 31;
    const int quad = total <= TEAM_QUAD && ncross == total ? 2 : 0;  // log2 of the lanes per cell
    for (int i0 = (int)threadIdx.x - lane; i0 < total << quad; i0 += MOOD_THREADS) {
        const int i = (i0 + lane) >> quad, k = quad ? lane & 3 : 0;
        bool trb = false;
        int c = 0;
        if (i < ncross) {
            c = sm.cross[i];
            if (c >= 0) trb = quad ? cross_finish<4>(a, sm, i, k, qx, qy) : cross_finish<1>(a, sm, i, k, qx, qy);
        } else if (i < total && team_own(a, lst, nt, i, pid, &c)) {
            trb = cross_update(a, w, c, -1, qx, qy);
        }
        trb = trb && k == 0;
        // warp-aggregated append to the next list, of every member and global
        const unsigned m = __ballot_sync(0xffffffffu, trb);
        if (m) {
            int b0 = 0;
            if (lane == 0) b0 = atomicAdd(&sm.count[nxt], __popc(m));
            b0 = __shfl_sync(0xffffffffu, b0, 0);
            if (trb) {
                const int idx = b0 + __popc(m & ((1u << lane) - 1));
                __stcg(a.tlist[nxt] + idx, c);
                if (idx < TEAM_LIST_CAP)
#pragma unroll
                    for (int r = 0; r < TEAM; r++)
                        cooperative_groups::this_cluster().map_shared_rank(&sm, r)->list[nxt][idx] = c;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x >= 1 && threadIdx.x < TEAM)
        cooperative_groups::this_cluster().map_shared_rank(&sm, (int)threadIdx.x)->count[nxt] = sm.count[nxt];
}

// Order-3 and order-1 weights into shared memory.
template <int NGP>
__device__ __forceinline__ void team_weights(TeamSmem& sm, const GpWeights& w) {
    for (int i = (int)threadIdx.x; i < 4 * NGP * 5; i += MOOD_THREADS) {
        const int f = i / (5 * NGP), gp = (i / 5) % NGP, m = i % 5;
        sm.z3[f][gp][m] = w.zt[1][f][gp][m];
        if (m == 0) sm.z1[f][gp] = w.zt[0][f][gp][0];
    }
}

// Passes 2, 3, ... over lists of more than GridGeom::mood_solo cells, on all SMs
// (a cooperative launch).  Leaves the list, which of the two it is and the
// pass count for k_mood_team.
template <int NGP>
__global__ void __launch_bounds__(MOOD_THREADS, 1) k_mood_loop(StageArgs a, const __grid_constant__ GpWeights w, GridBar* bar,
                                                      int max_pass) {
    __shared__ TeamSmem sm;
    const GridGeom& g = a.g;
    const double qx = a.sc->qx, qy = a.sc->qy;
    const unsigned epoch = a.sc->stamp_epoch;  // stamps epoch+2, epoch+3, ... are new
    const int tid = (int)threadIdx.x, lane = tid & 31, gtid = blockIdx.x * MOOD_THREADS + tid;
    const int slot = (tid >> 5) * (int)gridDim.x + (int)blockIdx.x;  // warp tasks are dealt over the SMs first
    const int slots = (MOOD_THREADS / 32) * (int)gridDim.x;
    constexpr int FPW = 32 / (2 * NGP);
    int cur = 0, pass = 1;  // pass 1 (all faces) ran before this kernel
    int nt = *(volatile int*)&a.sc->ntrb[cur];
    GridWait wait = grid_start(bar);
    if (nt > g.mood_solo) team_weights<NGP>(sm, w);
    __syncthreads();
    while (nt > g.mood_solo && pass < max_pass) {
        pass++;
        // the listed cells' orders were lowered when they were listed
        if (gtid == 0) {
            a.sc->ntrb[cur ^ 1] = 0;  // nobody appends to it before the next barrier
            a.sc->detected_step += (unsigned long long)nt;
        }
        const int* lst = a.tlist[cur];
        const int nface = (4 * nt + FPW - 1) / FPW, total = 5 * nt, chunks = (total + 31) / 32;
        for (int task = slot; task < nface + 4 * chunks; task += slots) {
            if (task < nface) {
                team_faces<NGP>(a, w, sm, lst, nt, task);
            } else {  // a cell's results are the same from whichever cross they come
                const int t = (task - nface) & 3, i = ((task - nface) >> 2) * 32 + lane;
                int c;
                if (i < total && cross_cell(g, __ldcg(lst + i / 5), i % 5, &c))
                    __stcg(a.tests + 4 * (size_t)c + t, (unsigned char)cross_test(g, w, a.uin + 4 * (size_t)c, t));
            }
        }
        if (!grid_sync(bar, wait)) return;
        // the 5-point crosses: Uout from Uin and the current fluxes, DETECTION
        const unsigned pid = epoch + (unsigned)pass;
        const int nxt = cur ^ 1;
        for (int task = slot; task < chunks; task += slots) {
            const int i = task * 32 + lane;
            bool trb = false;
            int c = 0;
            if (i < total && cross_cell(g, __ldcg(lst + i / 5), i % 5, &c)) {
                const unsigned f = __ldcg(reinterpret_cast<const unsigned*>(a.tests) + c);
                const int flags = (int)((f & 1) | (f >> 7 & 2) | (f >> 14 & 4) | (f >> 21 & 8));
                if (atomicExch(&a.stamp[c], pid) != pid) trb = cross_update(a, w, c, flags, qx, qy);
            }
            list_append(trb, a.tlist[nxt], &a.sc->ntrb[nxt], c);
        }
        if (!grid_sync(bar, wait)) return;
        cur ^= 1;
        nt = *(volatile int*)&a.sc->ntrb[cur];
    }
    if (gtid == 0) {
        a.sc->mood_cur = cur;
        a.sc->mood_pass = pass;
    }
}

// The rest of the loop, on one cluster (a launch of TEAM CTAs) until the list is
// empty or max_pass is reached, and the loop's results.
template <int NGP>
__global__ void __launch_bounds__(MOOD_THREADS, 1) k_mood_team(StageArgs a, const __grid_constant__ GpWeights w,
                                                      const GridBar* bar, int max_pass, int stage) {
    __shared__ TeamSmem sm;
    if (bar->err) {  // a grid barrier ran out: the host reports it after the step's other stages, whose lists start empty
        if (blockIdx.x == 0 && threadIdx.x == 0) a.sc->ntrb[0] = a.sc->ntrb[1] = 0;
        return;
    }
    const double qx = a.sc->qx, qy = a.sc->qy;
    const unsigned epoch = a.sc->stamp_epoch;
    const int rank = (int)blockIdx.x, tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int FPW = 32 / (2 * NGP);
    TeamSmem* sm0 = cooperative_groups::this_cluster().map_shared_rank(&sm, 0);
    int cur = a.sc->mood_cur, pass = a.sc->mood_pass;
    int nt = a.sc->ntrb[cur];
    if (nt != 0) {
        team_weights<NGP>(sm, w);
        for (int i = tid; i < nt && i < TEAM_LIST_CAP; i += MOOD_THREADS) sm.list[cur][i] = __ldcg(a.tlist[cur] + i);
        if (tid == 0) sm.count[cur] = nt;
        team_sync();
        while (nt != 0 && pass < max_pass) {
            pass++;
            if (rank == 0 && tid == 0) {
                sm.count[cur ^ 1] = 0;  // read last before the two barriers of the pass before
                a.sc->detected_step += (unsigned long long)nt;
            }
            const int* lst = nt <= TEAM_LIST_CAP ? sm.list[cur] : a.tlist[cur];
            const int nface = (4 * nt + FPW - 1) / FPW, ncross = a.g.solo_split ? min(5 * nt, TEAM_CROSS) : 0;
            const int chunks = (ncross + 31) / 32;
            for (int task = warp * TEAM + rank; task < nface + 5 * chunks; task += (MOOD_THREADS / 32) * TEAM) {
                if (task < nface) {
                    team_faces<NGP>(a, w, sm, lst, nt, task);
                } else {
                    const int t = (task - nface) % 5, i = (task - nface) / 5 * 32 + lane;
                    int c;
                    if (t == 4) {
                        if (i < ncross) team_prepare(a, sm0, lst, nt, i, epoch + (unsigned)pass);
                    } else if (i < ncross && cross_cell(a.g, lst[i / 5], i % 5, &c)) {
                        sm0->flag[t][i] = cross_test(a.g, w, a.uin + 4 * (size_t)c, t);
                    }
                }
            }
            team_sync();
            if (rank == 0) team_cells(a, w, sm, lst, cur, nt, ncross, epoch + (unsigned)pass, qx, qy);
            team_sync();
            cur ^= 1;
            nt = *(volatile int*)&sm.count[cur];
        }
        team_sync();  // a member's shared memory stays until no one writes to it
    }
    if (rank == 0 && tid == 0) {
        if (nt != 0) a.sc->status |= GPM_STATUS_MOODCAP;
        a.sc->passes_stage[stage] = pass;
        a.sc->stamp_epoch = epoch + (unsigned)pass + 1u;
        a.sc->ntrb[0] = a.sc->ntrb[1] = 0;  // for the next stage
    }
}

template <int NGP>
static int launch_mood_loop_n(const StageArgs& a, const GpWeights& w, GridBar* bar, int max_pass, int stage,
                              cudaStream_t s) {
    static std::atomic<int> grids[GPM_MAX_DEVICES];
    const int dev = gpm_device();
    int grid = grids[dev].load(std::memory_order_relaxed);
    if (!grid) {
        int sms = 0, occ = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_mood_loop<NGP>, MOOD_THREADS, 0);
        grid = sms * (occ > 0 ? occ : 1);
        grids[dev].store(grid, std::memory_order_relaxed);
    }
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(MOOD_THREADS);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k_mood_loop<NGP>, a, w, bar, max_pass) != cudaSuccess) return -1;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = TEAM;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(TEAM);
    return cudaLaunchKernelEx(&cfg, k_mood_team<NGP>, a, w, (const GridBar*)bar, max_pass, stage) == cudaSuccess ? 0 : -1;
}

int launch_mood_loop(const StageArgs& a, const GpWeights& w, GridBar* bar, int max_pass, int stage,
                     cudaStream_t s) {
    switch (a.g.ngp) {
    case 1: return launch_mood_loop_n<1>(a, w, bar, max_pass, stage, s);
    case 2: return launch_mood_loop_n<2>(a, w, bar, max_pass, stage, s);
    case 3: return launch_mood_loop_n<3>(a, w, bar, max_pass, stage, s);
    case 4: return launch_mood_loop_n<4>(a, w, bar, max_pass, stage, s);
    default: return launch_mood_loop_n<5>(a, w, bar, max_pass, stage, s);
    }
}

static int list_grid(int max_items, int threads) {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int need = (max_items + threads - 1) / threads;
    const int cap = sms * LIST_CTAS_PER_SM;
    return need < 1 ? 1 : (need < cap ? need : cap);
}


void launch_mood_faces(const StageArgs& a, const GpWeights& w, int cur, int max_trb, cudaStream_t s) {
    const int gr = list_grid(4 * max_trb, 128);
    switch (a.g.ngp) {
    case 1: k_mood_faces<1><<<gr, 128, 0, s>>>(a, w, cur); break;
    case 2: k_mood_faces<2><<<gr, 128, 0, s>>>(a, w, cur); break;
    case 3: k_mood_faces<3><<<gr, 128, 0, s>>>(a, w, cur); break;
    case 4: k_mood_faces<4><<<gr, 128, 0, s>>>(a, w, cur); break;
    default: k_mood_faces<5><<<gr, 128, 0, s>>>(a, w, cur); break;
    }
}


// The gate's extras repair (optional): a gated cell whose update from the
// uniform first pass (every face at mord, already stored) passes DETECTION is
// given mord back before the gated cells' faces are recomputed, so that only
// cells plain MOOD would also flag in its first pass start lowered.  The
// a-priori count drops by the cells given back.
__global__ void __launch_bounds__(256) k_gate_repair(StageArgs a, const __grid_constant__ GpWeights w) {
    const GridGeom& g = a.g;
    const int n = a.sc->ntrb[1];
    const double qx = a.sc->qx, qy = a.sc->qy;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const size_t c = (size_t)a.tlist[1][i];
        const Cell uo = cell_update(g, a.uin, a.fx, a.fy, c, qx, qy);
        if (!mood_troubled(uo, a.uin + 4 * c, g.nx, g, w.d2x, w.d2y)) {
            a.order[c] = (int8_t)g.mord;
            atomicAdd(&a.sc->apriori_step, ~0ull);  // minus one
        }
    }
}

void launch_gate_repair(const StageArgs& a, const GpWeights& w, int max_items, cudaStream_t s) {
    k_gate_repair<<<list_grid(max_items, 256), 256, 0, s>>>(a, w);
}

// ---------------------------------------------------------------------------
// Setdt (physics.f90:78-129): min over every cell, ghosts included, of
// 1/(1/(dx/(|u|+c)) + 1/(dy/(|v|+c))).  Reduced with fmin inside a CTA and an
// atomicMin on the bit pattern across CTAs (positive doubles order like their
// bits); NaN cells are ignored (IEEE minNum, as in the CPU restatement).

#if GPM_EXACT
__device__ __forceinline__ double cell_dt(const Cell& u, double dx, double dy) {
    const double vx = u.mx / u.r;
    const double vy = u.my / u.r;
    const double p = pressure(u);
    const double c = sqrt(GPM_GAMMA * p / u.r);
    return 1.0 / (1.0 / (dx / (fabs(vx) + c)) + 1.0 / (dy / (fabs(vy) + c)));
}
#else
// Fast mode: dx*dy / ((|u|+c)*dy + (|v|+c)*dx) with gpm_fast_rcp and
// the fast square root, equal to the form above up to rounding (a NaN or
// non-positive cell still gives NaN or a non-positive value, which the
// reduction skips).
__device__ __forceinline__ double cell_dt(const Cell& u, double dx, double dy) {
    const double ir = gpm_fast_rcp(u.r);
    const double vx = u.mx * ir, vy = u.my * ir;
    const double c = gpm_fast_sqrt(GPM_GAMMA * pressure_ir(u, ir) * ir);
    return dx * dy * gpm_fast_rcp((fabs(vx) + c) * dy + (fabs(vy) + c) * dx);
}
#endif

__device__ __forceinline__ void dt_reduce(double v, DevScalars* sc) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    __shared__ double wmin[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) wmin[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = lane < (int)(blockDim.x >> 5) ? wmin[lane] : 1.0e30;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0 && v > 0.0 && v < 1.0e30)  // NaN fails both tests
            atomicMin(&sc->dtmin_bits, (unsigned long long)__double_as_longlong(v));
    }
}

__global__ void __launch_bounds__(256) k_cfl(GridGeom g, const double* __restrict__ u, DevScalars* sc) {
    const size_t ncell = (size_t)g.nx * g.ny;
    double v = 1.0e30;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < ncell; c += (size_t)gridDim.x * blockDim.x)
        v = fmin(v, cell_dt(ld_cell(u + 4 * c), g.dx, g.dy));
    dt_reduce(v, sc);
}

void launch_cfl(const GridGeom& g, const double* u, DevScalars* sc, cudaStream_t s) {
    k_cfl<<<list_grid(g.nx * g.ny, 256), 256, 0, s>>>(g, u, sc);
}

// SSP-RK3 combination y = a*x + b*y over every cell (ghosts included, as the
// reference's whole-array expressions); optionally the Setdt reduction of y.
__global__ void __launch_bounds__(256) k_combine(GridGeom g, const double* __restrict__ x, double* __restrict__ y,
                                                 double ca, double cb, int with_cfl, DevScalars* sc) {
    const size_t ncell = (size_t)g.nx * g.ny;
    double v = 1.0e30;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < ncell; c += (size_t)gridDim.x * blockDim.x) {
        const Cell a = ld_cell(x + 4 * c);
        const Cell b = ld_cell_cg(y + 4 * c);
        Cell o;
        o.r = ca * a.r + cb * b.r;
        o.mx = ca * a.mx + cb * b.mx;
        o.my = ca * a.my + cb * b.my;
        o.e = ca * a.e + cb * b.e;
        st_cell(y + 4 * c, o);
        if (with_cfl) v = fmin(v, cell_dt(o, g.dx, g.dy));
    }
    if (with_cfl) dt_reduce(v, sc);
}

// The same combination out = a*x + b*y of a stage's y before Boundary_C(y):
// a ghost cell of y is Boundary_C's value (bc_cell; stage selects t_rk), so the
// stage needs no Boundary_C launch of its own.  out is neither x nor y.
__global__ void __launch_bounds__(256) k_combine_bc(GridGeom g, const double* __restrict__ x,
                                                    const double* __restrict__ y, double* __restrict__ out, double ca,
                                                    double cb, int with_cfl, DevScalars* sc, int stage) {
    const unsigned ncell = (unsigned)g.nx * (unsigned)g.ny;
    double v = 1.0e30;
    for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
        const int n = (int)(c / (unsigned)g.nx) - 3, l = (int)(c - (unsigned)(n + 3) * g.nx) - 3;
        const Cell a = ld_cell(x + 4 * (size_t)c);
        const bool inner = l >= 1 && l <= g.lf && n >= 1 && n <= g.nf;
        const Cell b = inner ? ld_cell(y + 4 * (size_t)c) : bc_cell(g, y, sc, stage, l, n);
        Cell o;
        o.r = ca * a.r + cb * b.r;
        o.mx = ca * a.mx + cb * b.mx;
        o.my = ca * a.my + cb * b.my;
        o.e = ca * a.e + cb * b.e;
        st_cell(out + 4 * (size_t)c, o);
        if (with_cfl) v = fmin(v, cell_dt(o, g.dx, g.dy));
    }
    if (with_cfl) dt_reduce(v, sc);
}

// y = c[0]*x[0] + c[1]*x[1] + ... (n terms, summed left to right as the
// reference's whole-array expressions of mod_SSP_RK4.f90:25-36 and
// mod_FE.f90:188), over every cell; y may be one of the x.
struct LinComb {
    const double* x[5];
    double c[5];
    int n;
};

__global__ void __launch_bounds__(256) k_lincomb(GridGeom g, double* y, LinComb lc, int with_cfl, DevScalars* sc) {
    const size_t ncell = (size_t)g.nx * g.ny;
    double v = 1.0e30;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < ncell; c += (size_t)gridDim.x * blockDim.x) {
        const Cell a = ld_cell_cg(lc.x[0] + 4 * c);
        Cell o{lc.c[0] * a.r, lc.c[0] * a.mx, lc.c[0] * a.my, lc.c[0] * a.e};
        for (int i = 1; i < lc.n; i++) {
            const Cell b = ld_cell_cg(lc.x[i] + 4 * c);
            o.r = o.r + lc.c[i] * b.r;
            o.mx = o.mx + lc.c[i] * b.mx;
            o.my = o.my + lc.c[i] * b.my;
            o.e = o.e + lc.c[i] * b.e;
        }
        st_cell(y + 4 * c, o);
        if (with_cfl) v = fmin(v, cell_dt(o, g.dx, g.dy));
    }
    if (with_cfl) dt_reduce(v, sc);
}

void launch_lincomb(const GridGeom& g, double* y, int n, const double* const* x, const double* c, int with_cfl,
                    DevScalars* sc, cudaStream_t s) {
    LinComb lc{};
    lc.n = n;
    for (int i = 0; i < n; i++) {
        lc.x[i] = x[i];
        lc.c[i] = c[i];
    }
    k_lincomb<<<list_grid(g.nx * g.ny, 256), 256, 0, s>>>(g, y, lc, with_cfl, sc);
}

void launch_combine(const GridGeom& g, const double* x, double* y, double a, double b, int with_cfl, DevScalars* sc,
                    cudaStream_t s) {
    k_combine<<<list_grid(g.nx * g.ny, 256), 256, 0, s>>>(g, x, y, a, b, with_cfl, sc);
}

void launch_combine_bc(const GridGeom& g, const double* x, const double* y, double* out, double a, double b,
                       int with_cfl, DevScalars* sc, int stage, cudaStream_t s) {
    k_combine_bc<<<list_grid(g.nx * g.ny, 256), 256, 0, s>>>(g, x, y, out, a, b, with_cfl, sc, stage);
}

// dt = CFL * min, clipped to dtfinal (physics.f90:292-296); qx = dt/dx.
// dtfinal < 0 selects tmax - t (main.f90:149).
__global__ void k_dt_finalize(GridGeom g, DevScalars* sc, double dtfinal_in) {
    double dt = __longlong_as_double((long long)sc->dtmin_bits);
    dt = dt * sc->cfl;
    const double dtfinal = dtfinal_in < 0.0 ? sc->tmax - sc->t : dtfinal_in;
    if (dt > dtfinal) dt = dtfinal;
    sc->dt = dt;
    sc->qx = dt / g.dx;
    sc->qy = dt / g.dy;
    sc->dtmin_bits = (unsigned long long)__double_as_longlong(1.0e30);
    if (!(dt > 0.0) || is_nan(dt) || dt == __longlong_as_double(0x7ff0000000000000LL)) sc->status |= GPM_STATUS_DT;
    sc->detected_step = 0;
}

void launch_dt_finalize(const GridGeom& g, DevScalars* sc, double dtfinal, cudaStream_t s) {
    k_dt_finalize<<<1, 1, 0, s>>>(g, sc, dtfinal);
}

// The start of a step of the device-resident loop (main.f90:149-160) at time
// t: Setdt's dt, and the step's counters.
__global__ void k_step_begin(GridGeom g, DevScalars* sc, double t) {
    sc->t = t;
    double dt = __longlong_as_double((long long)sc->dtmin_bits);
    dt = dt * sc->cfl;
    const double dtfinal = sc->tmax - t;
    if (dt > dtfinal) dt = dtfinal;
    sc->dt = dt;
    sc->qx = dt / g.dx;
    sc->qy = dt / g.dy;
    sc->dtmin_bits = (unsigned long long)__double_as_longlong(1.0e30);
    sc->detected_step = 0;
    sc->apriori_step = 0;
    sc->ntrb[0] = sc->ntrb[1] = 0;  // calls between steps (nn_predict, nn_gate_logits) list cells too
    sc->status = 0;
}

void launch_step_begin(const GridGeom& g, DevScalars* sc, double t, cudaStream_t s) {
    k_step_begin<<<1, 1, 0, s>>>(g, sc, t);
}

const KernelTable table = {launch_bc,       launch_flux_all, launch_update_detect, launch_mood_faces,
                           launch_combine,  launch_combine_bc, launch_cfl,         launch_dt_finalize,
                           launch_step_begin, launch_mood_loop, launch_lincomb,    launch_gate_repair};

}  // namespace GPM_NS

// ===========================================================================
// Batched stepping: many independent problems of uneven size (batch_common.h).
// Every phase of an RK stage is one persistent launch over all problems'
// work items, so a whole step has a fixed launch sequence that is captured
// once as a CUDA graph.  Per-problem arithmetic is the single-problem path's in
// the exact mode, and its own in the fast mode (batch_fast.cuh).
#include "batch_common.h"

namespace GPM_NS {

#if GPM_EXACT
using EnsMath = FaceMath;
namespace ens {
using GPM_NS::cell_dt;
}
#else
#include "batch_fast.cuh"
struct EnsMath {
    template <int DIR, int NGP>
    static __device__ __forceinline__ void quad(const double (*uL)[4], const double (*uR)[4], const double* gw,
                                                double* F, int nflux) {
        ens::quad_flux<DIR, NGP>(uL, uR, gw, F, nflux);
    }
    template <int DIR>
    static __device__ __forceinline__ void solve(int nflux, const double* uL, const double* uR, double* F) {
        ens::solve<DIR>(nflux, uL, uR, F);
    }
};
#endif

__device__ __forceinline__ GridGeom bgeom(const BatchArgs& a, const BProb& p) {
    GridGeom g;
    g.lf = p.lf; g.nf = p.nf; g.nx = p.nx; g.ny = p.ny;
    g.dx = p.dx; g.dy = p.dy;
    g.bc_type = a.bc_type; g.ngp = a.ngp; g.mord = a.mord; g.method = a.method;
    g.dmp = a.dmp; g.u2 = a.u2; g.u2_tol = a.u2_tol; g.u2_fd = 0; g.num_flux = a.num_flux;
    g.mood_solo = a.mood_solo;
    g.flux_tma = 0;
    g.solo_split = 0;
    g.cc_col = -1;
    return g;
}

// Boundary_C of every problem: blockIdx.y is the problem.
__global__ void kb_bc_x(BatchArgs a, double* __restrict__ u) {
    const BProb P = a.prob[blockIdx.y];
    const GridGeom g = bgeom(a, P);
    const int n = 1 + blockIdx.x * blockDim.y + threadIdx.y, k = threadIdx.x;
    if (n > g.nf || k >= 2 * GPM_NGC) return;
    double* ub = u + 4 * P.off;
    const bool right = k >= GPM_NGC;
    const int j = right ? k - GPM_NGC : k;
    const int l = right ? g.lf + 1 + j : -j;
    double* dst = ub + 4 * cidx(g, l, n);
    if (g.bc_type == 17) {
        const double* src = ub + 4 * cidx(g, right ? g.lf : 1, n);
        for (int v = 0; v < 4; v++) dst[v] = src[v];
    } else if (g.bc_type == 18) {
        const double* src = ub + 4 * cidx(g, right ? 1 + j : g.lf - j, n);
        for (int v = 0; v < 4; v++) dst[v] = src[v];
    } else if (g.bc_type == 20) {
        const double* src = ub + 4 * cidx(g, right ? g.lf - j : 1 + j, n);
        dst[0] = src[0]; dst[1] = -src[1]; dst[2] = src[2]; dst[3] = src[3];
    }
}

__global__ void kb_bc_y(BatchArgs a, double* __restrict__ u) {
    const BProb P = a.prob[blockIdx.y];
    const GridGeom g = bgeom(a, P);
    const int l = (int)(blockIdx.x * blockDim.y + threadIdx.y) - 3, k = threadIdx.x;
    if (l > g.lf + GPM_NGC || k >= 2 * GPM_NGC) return;
    double* ub = u + 4 * P.off;
    const bool top = k >= GPM_NGC;
    const int j = top ? k - GPM_NGC : k;
    const int n = top ? g.nf + 1 + j : -j;
    double* dst = ub + 4 * cidx(g, l, n);
    if (g.bc_type == 17) {
        const double* src = ub + 4 * cidx(g, l, top ? g.nf : 1);
        for (int v = 0; v < 4; v++) dst[v] = src[v];
    } else if (g.bc_type == 18) {
        const double* src = ub + 4 * cidx(g, l, top ? 1 + j : g.nf - j);
        for (int v = 0; v < 4; v++) dst[v] = src[v];
    } else if (g.bc_type == 20) {
        const double* src = ub + 4 * cidx(g, l, top ? g.nf - j : 1 + j);
        dst[0] = src[0]; dst[1] = src[1]; dst[2] = -src[2]; dst[3] = src[3];
    }
}

static int g_max_nx = 0;  // set by the batch host code before launches (largest nx/ny of the batch)

void blaunch_bc(const BatchArgs& a, double* u, cudaStream_t s) {
    const dim3 blk(8, 32);
    kb_bc_x<<<dim3((g_max_nx + 31) / 32, a.nprob), blk, 0, s>>>(a, u);
    kb_bc_y<<<dim3((g_max_nx + 31) / 32, a.nprob), blk, 0, s>>>(a, u);
}

// Face tiles of every problem: a persistent CTA walks the tile list.  Tile
// shape TXB x TYB is a template parameter chosen by the autotuner.
template <int DIR, int NP, int NGP, int HXB>
__device__ __forceinline__ void face_tile_b(const GpWeights& w, int o, const Cell* tile, int tx, int ty, double* F,
                                            int nflux) {
    constexpr int FL = DIR == 0 ? 2 : 1;
    constexpr int FH = DIR == 0 ? 0 : 3;
    double uL[NGP][4], uR[NGP][4];
    {
        Cell q[NP];
#pragma unroll
        for (int m = 0; m < NP; m++) q[m] = tile[(ty + st_oy(m)) * HXB + tx + st_ox(m)];
        recon_face<DIR, NP, NGP>(w, o, FL, q, uL);
    }
    {
        constexpr int hx = DIR == 0 ? 1 : 0, hy = DIR == 0 ? 0 : 1;
        Cell q[NP];
#pragma unroll
        for (int m = 0; m < NP; m++) q[m] = tile[(ty + hy + st_oy(m)) * HXB + tx + hx + st_ox(m)];
        recon_face<DIR, NP, NGP>(w, o, FH, q, uR);
    }
    EnsMath::template quad<DIR, NGP>(uL, uR, w.gw, F, nflux);
}

template <int TXB, int TYB, int NGP, int ORD>
__global__ void __launch_bounds__(TXB* TYB) kb_flux(BatchArgs a) {
    constexpr int HXB = TXB + 5, HYB = TYB + 5;
    __shared__ Cell tile[HXB * HYB];
    const int tid = threadIdx.y * TXB + threadIdx.x;
    for (int item = blockIdx.x; item < a.nftiles; item += gridDim.x) {
        const int4 it = a.ftiles[item];
        const BProb P = a.prob[it.x];
        const GridGeom g = bgeom(a, P);
        const GpWeights& w = a.wtab[P.wc];
        const double* ub = a.uin + 4 * P.off;
        __syncthreads();  // the previous tile's faces are done with the buffer
        for (int i = tid; i < HXB * HYB; i += TXB * TYB) {
            const int cy = i / HXB, cx = i - cy * HXB;
            const int l = it.z - 2 + cx, n = it.w - 2 + cy;
            if (l >= -3 && l <= g.lf + 4 && n >= -3 && n <= g.nf + 4) tile[i] = ld_cell(ub + 4 * cidx(g, l, n));
        }
        __syncthreads();
        const int l = it.z + threadIdx.x, n = it.w + threadIdx.y;
        if (l > g.lf || n > g.nf) continue;
        double F[4];
        if (it.y == 0)
            face_tile_b<0, np_of(ORD), NGP, HXB>(w, ORD / 2, tile, threadIdx.x + 2, threadIdx.y + 2, F, g.num_flux);
        else face_tile_b<1, np_of(ORD), NGP, HXB>(w, ORD / 2, tile, threadIdx.x + 2, threadIdx.y + 2, F, g.num_flux);
        st_cell((it.y == 0 ? a.fx : a.fy) + 4 * (P.off + (long long)cidx(g, l, n)), Cell{F[0], F[1], F[2], F[3]});
    }
}

#if !GPM_EXACT
// The two-direction cell tiles of every problem (xy_tile), persistent CTAs.
__global__ void __launch_bounds__(XT * XY, 2) kb_flux_xy(BatchArgs a) {
    extern __shared__ __align__(16) unsigned char xy_raw[];
    ens::XySmem& sm = *reinterpret_cast<ens::XySmem*>(xy_raw);
    for (int item = blockIdx.x; item < a.nftiles; item += gridDim.x) {
        const int4 it = a.ftiles[item];
        const BProb P = a.prob[it.x];
        __syncthreads();  // the previous tile is done with the shared buffers
        ens::xy_tile(bgeom(a, P), a.wtab[P.wc], a.uin + 4 * P.off, a.fx + 4 * P.off, a.fy + 4 * P.off, it.z, it.w, sm);
    }
}

// The edge items (problem, 3, k0, 0) of every problem.
__global__ void __launch_bounds__(EDGE_T) kb_flux_edge(BatchArgs a) {
    for (int item = blockIdx.x; item < a.netiles; item += gridDim.x) {
        const int4 it = a.etiles[item];
        const BProb P = a.prob[it.x];
        edge_faces<EnsMath>(bgeom(a, P), a.wtab[P.wc], a.uin + 4 * P.off, a.fx + 4 * P.off, a.fy + 4 * P.off, it.z);
    }
}
#endif

template <int TXB, int TYB, int NGP>
static void blaunch_flux_t(const BatchArgs& a, cudaStream_t s) {
    const int grid = a.nftiles < sm_count() * 4 ? a.nftiles : sm_count() * 4;
    const dim3 blk(TXB, TYB);
    if (a.mord == 5) kb_flux<TXB, TYB, NGP, 5><<<grid, blk, 0, s>>>(a);
    else if (a.mord == 3) kb_flux<TXB, TYB, NGP, 3><<<grid, blk, 0, s>>>(a);
    else kb_flux<TXB, TYB, NGP, 1><<<grid, blk, 0, s>>>(a);
}

template <int NGP>
static void blaunch_flux_n(const BatchArgs& a, cudaStream_t s) {
#if !GPM_EXACT
    if (a.tile == GPM_TILE_XY && NGP == 3 && a.mord == 5) {
        static std::atomic<bool> attr[GPM_MAX_DEVICES];
        const int dev = gpm_device();
        if (!attr[dev].load(std::memory_order_relaxed)) {
            cudaFuncSetAttribute(kb_flux_xy, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ens::XySmem));
            attr[dev].store(true, std::memory_order_relaxed);
        }
        const int grid = a.nftiles < sm_count() * 2 ? a.nftiles : sm_count() * 2;
        kb_flux_xy<<<grid, dim3(XT, XY), sizeof(ens::XySmem), s>>>(a);
        const int ge = a.netiles < sm_count() * 16 ? a.netiles : sm_count() * 16;
        if (ge > 0) kb_flux_edge<<<ge, EDGE_T, 0, s>>>(a);
        return;
    }
#endif
    switch (a.tile) {
    case 0: blaunch_flux_t<32, 8, NGP>(a, s); break;
    case 1: blaunch_flux_t<32, 4, NGP>(a, s); break;
    case 2: blaunch_flux_t<16, 16, NGP>(a, s); break;
    default: blaunch_flux_t<64, 4, NGP>(a, s); break;
    }
}

void blaunch_flux(const BatchArgs& a, cudaStream_t s) {
    switch (a.ngp) {
    case 1: blaunch_flux_n<1>(a, s); break;
    case 2: blaunch_flux_n<2>(a, s); break;
    case 3: blaunch_flux_n<3>(a, s); break;
    case 4: blaunch_flux_n<4>(a, s); break;
    default: blaunch_flux_n<5>(a, s); break;
    }
}

__device__ __forceinline__ void list_append2(bool flag, int2* __restrict__ list, int* __restrict__ count, int2 value) {
    const unsigned act = __activemask();
    const unsigned m = __ballot_sync(act, flag);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(act) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(act, base, leader);
    if (flag) list[base + __popc(m & ((1u << lane) - 1))] = value;
}

// First-pass update + DETECTION: persistent over blocks of 256 interior cells.
__global__ void __launch_bounds__(256) kb_update(BatchArgs a) {
    for (int item = blockIdx.x; item < a.ncblocks; item += gridDim.x) {
        const int2 it = a.cblocks[item];
        const BProb P = a.prob[it.x];
        const GridGeom g = bgeom(a, P);
        const int k = it.y + threadIdx.x;
        bool trb = false;
        int cl = 0;
        if (k < g.lf * g.nf) {
            const int l = 1 + k % g.lf, n = 1 + k / g.lf;
            const size_t c = cidx(g, l, n);
            const double* ub = a.uin + 4 * P.off;
            const Cell uo = cell_update(g, ub, a.fx + 4 * P.off, a.fy + 4 * P.off, c, a.sc[it.x].qx, a.sc[it.x].qy);
            st_cell(a.uout + 4 * (P.off + (long long)c), uo);
            if (a.method == 2 && g.mord > 1)
                trb = mood_troubled(uo, ub + 4 * c, g.nx, g, a.wtab[P.wc].d2x, a.wtab[P.wc].d2y);
            else if (a.method == 2 && inadmissible(uo))
                atomicOr(&a.ntrb[6], 1);
            cl = (int)c;
        }
        if (trb) cascade_order(a.order + P.off + cl);
        list_append2(trb, a.tlist[0], &a.ntrb[0], make_int2(it.x, cl));
    }
}

void blaunch_update(const BatchArgs& a, cudaStream_t s) {
    const int grid = a.ncblocks < sm_count() * 8 ? a.ncblocks : sm_count() * 8;
    kb_update<<<grid, 256, 0, s>>>(a);
}

// Face i of the batch's face list at Gauss point gp (face_phase_gp item).
__device__ __forceinline__ void kb_face_gp(const BatchArgs& a, int cur, int nt, int i, int gp, FaceGp& f) {
    int dir, side;
    const int2 e = a.tlist[cur][face_item(i, nt, &dir, &side)];
    const BProb P = a.prob[e.x];
    StageArgs sa;
    sa.ccw = nullptr;
    sa.g = bgeom(a, P);
    sa.uin = a.uin + 4 * P.off;
    sa.fx = a.fx + 4 * P.off;
    sa.fy = a.fy + 4 * P.off;
    sa.order = a.order + P.off;
    const GpWeights& w = a.wtab[P.wc];
    const size_t c = (size_t)e.y;
    if (dir == 0) face_gp_any<0, EnsMath>(sa, w, side == 0 ? c - 1 : c, gp, f);
    else face_gp_any<1, EnsMath>(sa, w, side == 0 ? c - sa.g.nx : c, gp, f);
}

// The batch's whole MOOD loop in one cooperative launch: passes run until every
// problem's list is empty, on all SMs and, once it is short, in CTA 0 (mood_sync).  ntrb[2] is the stamp epoch,
// ntrb[4] the detected-cell total, ntrb[5] the pass count of the last stage.
template <int NGP>
__global__ void __launch_bounds__(MOOD_THREADS, 1) kb_mood_loop(BatchArgs a, GridBar* bar, int max_pass) {
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gstride = gridDim.x * blockDim.x;
    int stid = pack_tid(), wstride = gstride;
    GridWait wait = grid_start(bar);
    bool solo = false;
    int cur = 0, pass = 1;
    for (;;) {
        const int nt = *(volatile int*)&a.ntrb[cur];
        if (nt == 0) break;
        if (pass >= max_pass) {
            if (gtid == 0) a.ntrb[3] = 1;
            break;
        }
        if (!solo && nt <= a.mood_solo) {
            if (blockIdx.x != 0) return;
            solo = true;
            stid = threadIdx.x;
            wstride = blockDim.x;
        }
        pass++;
        // the listed cells' orders were lowered when they were listed
        if (gtid == 0) {
            a.ntrb[cur ^ 1] = 0;  // nobody appends to it before the next barrier
            a.ntrb[2] += 1;       // stamp epoch, read after the next barrier
            a.ntrb[4] += nt;
        }
        const int total = 5 * nt;
        face_phase_gp<NGP>(4 * nt, 2 * nt, stid, wstride,
                           [&](int i, int gp, FaceGp& f) { kb_face_gp(a, cur, nt, i, gp, f); });
        if (solo) {
            // The crosses' Uin-only tests beside the faces, on the warps after theirs.  On a long list
            // they stay behind the update, for the few cells that need them: 48 problems, 3 steps, the loop's
            // nine launches take 6.87 ms with all tests behind it, 7.13 with all beside the faces, 6.51 so.
            constexpr int FPW = 32 / NGP;
            const int chunks = (total + 31) / 32, nwarp = wstride >> 5;
            const int first = 2 * ((2 * nt + FPW - 1) / FPW) % nwarp;
            for (int task = ((stid >> 5) + nwarp - first) % nwarp; task < 4 * chunks; task += nwarp) {
                const int t = task & 3, i = (task >> 2) * 32 + (threadIdx.x & 31);
                int c;
                if (i < total) {
                    const int2 e = a.tlist[cur][i / 5];
                    const BProb P = a.prob[e.x];
                    const GridGeom g = bgeom(a, P);
                    if (cross_cell(g, e.y, i % 5, &c))
                        __stcg(a.tests + 4 * (P.off + c) + t,
                               (unsigned char)cross_test(g, a.wtab[P.wc], a.uin + 4 * (P.off + c), t));
                }
            }
        }
        if (!mood_sync(bar, wait, solo)) return;
        const unsigned epoch = (unsigned)*(volatile int*)&a.ntrb[2];
        const int nxt = cur ^ 1;
        const int lim = ((total + wstride - 1) / wstride) * wstride;
        for (int base = 0; base < lim; base += wstride) {
            const int i = base + stid;
            bool trb = false;
            int2 val = make_int2(0, 0);
            if (i < total) {
                const int2 e = a.tlist[cur][i / 5];
                const BProb P = a.prob[e.x];
                const GridGeom g = bgeom(a, P);
                int c;
                if (cross_cell(g, e.y, i % 5, &c) && atomicExch(&a.stamp[P.off + c], epoch) != epoch) {
                    const double* ub = a.uin + 4 * P.off;
                    const Cell uo = cell_update(g, ub, a.fx + 4 * P.off, a.fy + 4 * P.off, (size_t)c, a.sc[e.x].qx,
                                                a.sc[e.x].qy);
                    st_cell(a.uout + 4 * (P.off + c), uo);
                    if (a.order[P.off + c] > 1) {
                        const int r = solo ? mood_uout_part(uo, ub + 4 * (size_t)c, g.nx, g) : 0;
                        if (r == 2) {
                            const unsigned f = __ldcg(reinterpret_cast<const unsigned*>(a.tests) + P.off + c);
                            trb = (f & 0x101) == 0x101 && !(g.u2 && (f & 0x1010000));
                        } else {
                            trb = solo ? r == 1 : mood_troubled(uo, ub + 4 * (size_t)c, g.nx, g, a.wtab[P.wc].d2x, a.wtab[P.wc].d2y);
                        }
                    } else if (inadmissible(uo)) {
                        atomicOr(&a.ntrb[6], 1);
                    }
                    val = make_int2(e.x, c);
                }
            }
            if (trb) cascade_order(a.order + a.prob[val.x].off + val.y);
            list_append2(trb, a.tlist[nxt], &a.ntrb[nxt], val);
        }
        if (!mood_sync(bar, wait, solo)) return;
        cur ^= 1;
    }
    if (gtid == 0) a.ntrb[5] = pass;
}

template <int NGP>
static int blaunch_mood_loop_n(const BatchArgs& a, GridBar* bar, int max_pass, cudaStream_t s) {
    static std::atomic<int> grids[GPM_MAX_DEVICES];
    const int dev = gpm_device();
    int grid = grids[dev].load(std::memory_order_relaxed);
    if (!grid) {
        int occ = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kb_mood_loop<NGP>, MOOD_THREADS, 0);
        grid = sm_count() * (occ > 0 ? occ : 1);
        grids[dev].store(grid, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(MOOD_THREADS);
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kb_mood_loop<NGP>, a, bar, max_pass) == cudaSuccess ? 0 : -1;
}

int blaunch_mood_loop(const BatchArgs& a, GridBar* bar, int max_pass, cudaStream_t s) {
    switch (a.ngp) {
    case 1: return blaunch_mood_loop_n<1>(a, bar, max_pass, s);
    case 2: return blaunch_mood_loop_n<2>(a, bar, max_pass, s);
    case 3: return blaunch_mood_loop_n<3>(a, bar, max_pass, s);
    case 4: return blaunch_mood_loop_n<4>(a, bar, max_pass, s);
    default: return blaunch_mood_loop_n<5>(a, bar, max_pass, s);
    }
}

// Per-problem CFL minimum: every block of padded cells belongs to one problem.
__device__ __forceinline__ void bdt_reduce(double v, BScal* sc) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    __shared__ double wmin[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) wmin[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = lane < (int)(blockDim.x >> 5) ? wmin[lane] : 1.0e30;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0 && v > 0.0 && v < 1.0e30) atomicMin(&sc->dtmin_bits, (unsigned long long)__double_as_longlong(v));
    }
}

__global__ void __launch_bounds__(256) kb_combine(BatchArgs a, const double* __restrict__ x, double* __restrict__ y,
                                                  double ca, double cb, int with_cfl, int only_cfl) {
    for (int item = blockIdx.x; item < a.npblocks; item += gridDim.x) {
        const int2 it = a.pblocks[item];
        const BProb P = a.prob[it.x];
        const int k = it.y + threadIdx.x;
        double v = 1.0e30;
        if (k < P.nx * P.ny) {
            const long long c = P.off + k;
            if (only_cfl) {
                v = ens::cell_dt(ld_cell(x + 4 * c), P.dx, P.dy);
            } else {
                const Cell p = ld_cell(x + 4 * c);
                const Cell q = ld_cell_cg(y + 4 * c);
                Cell o;
                o.r = ca * p.r + cb * q.r;
                o.mx = ca * p.mx + cb * q.mx;
                o.my = ca * p.my + cb * q.my;
                o.e = ca * p.e + cb * q.e;
                st_cell(y + 4 * c, o);
                if (with_cfl) v = ens::cell_dt(o, P.dx, P.dy);
            }
        }
        if (with_cfl || only_cfl) bdt_reduce(v, &a.sc[it.x]);
    }
}

void blaunch_combine(const BatchArgs& a, const double* x, double* y, double ca, double cb, int with_cfl, cudaStream_t s) {
    const int grid = a.npblocks < sm_count() * 8 ? a.npblocks : sm_count() * 8;
    kb_combine<<<grid, 256, 0, s>>>(a, x, y, ca, cb, with_cfl, 0);
}

void blaunch_cfl(const BatchArgs& a, const double* u, cudaStream_t s) {
    const int grid = a.npblocks < sm_count() * 8 ? a.npblocks : sm_count() * 8;
    kb_combine<<<grid, 256, 0, s>>>(a, u, nullptr, 0.0, 0.0, 1, 1);
}

__global__ void kb_dt_finalize(BatchArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nprob) return;
    BScal& sc = a.sc[i];
    double dt = __longlong_as_double((long long)sc.dtmin_bits);
    dt = dt * sc.cfl;
    const double dtfinal = sc.tmax - sc.t;
    if (dt > dtfinal) dt = dtfinal;
    sc.dt = dt;
    sc.qx = dt / a.prob[i].dx;
    sc.qy = dt / a.prob[i].dy;
    sc.dtmin_bits = (unsigned long long)__double_as_longlong(1.0e30);
    if (!(dt > 0.0) || is_nan(dt)) sc.status |= GPM_STATUS_DT;
}

__global__ void kb_advance_t(BatchArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.nprob) a.sc[i].t = a.sc[i].t + a.sc[i].dt;
}

void blaunch_dt_finalize(const BatchArgs& a, cudaStream_t s) { kb_dt_finalize<<<(a.nprob + 127) / 128, 128, 0, s>>>(a); }
void blaunch_advance_t(const BatchArgs& a, cudaStream_t s) { kb_advance_t<<<(a.nprob + 127) / 128, 128, 0, s>>>(a); }

void batch_set_max_nx(int nx) { g_max_nx = nx; }

const BatchTable batch_table = {blaunch_bc,  blaunch_flux,        blaunch_update,    blaunch_combine,
                                blaunch_cfl, blaunch_dt_finalize, blaunch_advance_t, blaunch_mood_loop};

}  // namespace GPM_NS
