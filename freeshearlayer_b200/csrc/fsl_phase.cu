// fsl_phase.cu -- one kernel per reference phase of the explicit step (FP64).
//
// These are the unfused path behind the per-phase C-ABI entry points
// (fsl_ghost_bc, fsl_reconstruct, ...).  They keep the reference's data flow
// (face-state arrays between reconstruction and fluxes) so each phase can be
// checked on its own against the CPU oracle.  Compiled with --fmad=false:
// results equal the reference's serial FP64 code bit for bit.
#include <algorithm>

#define FSL_CHK_UNIT FSL_CHK_PHASE
#include "fsl_check.cuh"
#include "fsl_dyn.cuh"
#include "fsl_internal.h"
#include "fsl_phys.cuh"
#include "fsl_stage.cuh"

FSL_CHK_EXPORT(phase)

namespace fsl {

namespace {

__device__ __forceinline__ long long ixf(int L, int H, int D, int i, int j, int k)
{
    return FSL_FACE(((long long)i * H + j) * D + k, (long long)(L + 1) * H * D);
}
__device__ __forceinline__ long long iyf(int L, int H, int D, int i, int j, int k)
{
    return FSL_FACE(((long long)i * (H + 1) + j) * D + k, (long long)L * (H + 1) * D);
}
__device__ __forceinline__ long long izf(int L, int H, int D, int i, int j, int k)
{
    return FSL_FACE(((long long)i * H + j) * (D + 1) + k, (long long)L * H * (D + 1));
}

// ---------------------------------------------------------------------------
// A1 ghost cells (src/boundCondInGhostCells.c:10-96), one thread per cell.
// ---------------------------------------------------------------------------
__global__ void k_ghost(Grid g, int setup, double *__restrict__ u)
{
    follow();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < stage::ghost_cells(g)) stage::ghost_cell(g, setup == FSL_SETUP_SPATIAL, u, t);
}

// Blocks of the per-phase kernels: kPlaneThreads consecutive entries of one
// plane's nb x nc list, so short and ragged rows fill their warps (rows of 40
// left 24 of every 64 lanes idle); block -> (plane a, row b, column c).
// ---------------------------------------------------------------------------
constexpr int kPlaneThreads = 128;
__host__ __device__ inline unsigned plane_blocks(int nb, int nc)
{
    return ((unsigned)nb * (unsigned)nc + kPlaneThreads - 1) / kPlaneThreads;
}
__device__ __forceinline__ bool plane_cell(int nb, int nc, unsigned block, int &a, int &b, int &c)
{
    const unsigned per = plane_blocks(nb, nc), p = block / per;
    const unsigned t = (block - p * per) * kPlaneThreads + threadIdx.x, r = t / (unsigned)nc;
    a = (int)p;
    b = (int)r;
    c = (int)(t - r * (unsigned)nc);
    return b < nb;
}

// ---------------------------------------------------------------------------
// A2 reconstruction (src/reconstruction.c:26-345): one thread per interior
// cell, all three sweeps, six face states written to the face arrays.  With
// PPM, a sweep whose four neighbours exist (the cell is not next to the
// domain boundary in that direction) uses ppm_* instead.  FP64 arithmetic in a
// chain of three sweeps: five blocks an SM (102 registers) where 132 registers
// left three, and full warps; 96x72x40 29 -> 20 us with both.
// ---------------------------------------------------------------------------
template <bool PPM>
__global__ void __launch_bounds__(kPlaneThreads, 5) k_recon(Grid g, const double *__restrict__ u, Faces f)
{
    follow();
    const int L = g.L, H = g.H, D = g.D;
    int i, j, k;
    if (!plane_cell(H, D, blockIdx.x, i, j, k)) return;
    i++; j++; k++;
    const long long fs = g.fstride;
    const long long c0 = g.idx(i, j, k);
    if (!FSL_SPAN(c0, -g.pi, g.pi, fs)) return; // the one-neighbour stencil in x, the widest
    CellC<double> c;
#pragma unroll
    for (int q = 0; q < 5; q++) c.u[q] = u[q * fs + c0];
    cell_consts(c);
    double fw[5], bw[5], hi[5], lo[5];
    // x
    {
        const long long a = c0 + g.pi, b = c0 - g.pi;
#pragma unroll
        for (int q = 0; q < 5; q++) { fw[q] = u[q * fs + a]; bw[q] = u[q * fs + b]; }
        if (PPM && i >= 2 && i <= L - 1) {
            double m2[5], p2[5];
#pragma unroll
            for (int q = 0; q < 5; q++) { p2[q] = u[q * fs + a + g.pi]; m2[q] = u[q * fs + b - g.pi]; }
            ppm_x(c, m2, bw, fw, p2, hi, lo);
        } else {
            recon_x(c, fw, bw, hi, lo);
        }
        const long long fh = ixf(L, H, D, i, j - 1, k - 1), fl = ixf(L, H, D, i - 1, j - 1, k - 1);
#pragma unroll
        for (int q = 0; q < 5; q++) { f.x[0][q][fh] = hi[q]; f.x[1][q][fl] = lo[q]; }
    }
    // y: (rho, rho v, rho w, rho u, E)
    {
        const long long a = c0 + g.pk, b = c0 - g.pk;
        const int perm[5] = {0, 2, 3, 1, 4};
#pragma unroll
        for (int q = 0; q < 5; q++) { fw[q] = u[perm[q] * fs + a]; bw[q] = u[perm[q] * fs + b]; }
        if (PPM && j >= 2 && j <= H - 1) {
            double m2[5], p2[5];
#pragma unroll
            for (int q = 0; q < 5; q++) { p2[q] = u[perm[q] * fs + a + g.pk]; m2[q] = u[perm[q] * fs + b - g.pk]; }
            ppm_y(c, m2, bw, fw, p2, hi, lo);
        } else {
            recon_y(c, fw, bw, hi, lo);
        }
        const long long fh = iyf(L, H, D, i - 1, j, k - 1), fl = iyf(L, H, D, i - 1, j - 1, k - 1);
#pragma unroll
        for (int q = 0; q < 5; q++) { f.y[0][q][fh] = hi[q]; f.y[1][q][fl] = lo[q]; }
    }
    // z: (rho, rho w, rho u, rho v, E)
    {
        const long long a = c0 + 1, b = c0 - 1;
        const int perm[5] = {0, 3, 1, 2, 4};
#pragma unroll
        for (int q = 0; q < 5; q++) { fw[q] = u[perm[q] * fs + a]; bw[q] = u[perm[q] * fs + b]; }
        if (PPM && k >= 2 && k <= D - 1) {
            double m2[5], p2[5];
#pragma unroll
            for (int q = 0; q < 5; q++) { p2[q] = u[perm[q] * fs + a + 1]; m2[q] = u[perm[q] * fs + b - 1]; }
            ppm_z(c, m2, bw, fw, p2, hi, lo);
        } else {
            recon_z(c, fw, bw, hi, lo);
        }
        const long long fh = izf(L, H, D, i - 1, j - 1, k), fl = izf(L, H, D, i - 1, j - 1, k - 1);
#pragma unroll
        for (int q = 0; q < 5; q++) { f.z[0][q][fh] = hi[q]; f.z[1][q][fl] = lo[q]; }
    }
}

// ---------------------------------------------------------------------------
// A3 boundary face states (src/bounCondOnInterfaces.c:11-110).
// ---------------------------------------------------------------------------
__global__ void k_ifbc(Grid g, int setup, int BL_HIG, Disturb d, Faces f)
{
    follow();
    const int L = g.L, H = g.H, D = g.D;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nx = (long long)H * D, ny = (long long)L * D, nz = (long long)L * H;
    const bool spatial = (setup == FSL_SETUP_SPATIAL);
    typedef Kc<double> kc;
    if (t < nx) {
        const int j = (int)((unsigned)t / (unsigned)D), k = (int)((unsigned)t % (unsigned)D);
        const long long f0 = ixf(L, H, D, 0, j, k), fL = ixf(L, H, D, L, j, k);
        if (spatial) {
            const double P = 100000., R = 1.0;
            double U, V = 0., W = 0.;
            double v[5];
            if (j < H / 2) { // :17-29
                U = 76.4;
                v[0] = R; v[1] = R * U; v[2] = 0.; v[3] = 0.; v[4] = P / kc::K_1 + 0.5 * R * (U * U);
            } else if (j < H / 2 + BL_HIG) { // :31-49
                const unsigned ku = (unsigned)k;
                bool dist;
                if (d.k_max > d.k_min) dist = (ku >= d.k_min && ku < d.k_max);
                else dist = !(ku >= d.k_max && ku < d.k_min);
                if (dist) { U = 200. + d.Ud; V = d.Vd; W = d.Wd; }
                else { U = 200.; V = W = 0.; }
                v[0] = R; v[1] = R * U; v[2] = R * V; v[3] = R * W;
                v[4] = P / kc::K_1 + 0.5 * R * (U * U + V * V + W * W);
            } else { // :51-60
                U = 200.;
                v[0] = R; v[1] = R * U; v[2] = 0.; v[3] = 0.; v[4] = P / kc::K_1 + 0.5 * R * (U * U);
            }
#pragma unroll
            for (int q = 0; q < 5; q++) f.x[0][q][f0] = v[q];
            // :62-71 outflow
            const double r = f.x[0][0][fL], mu_ = f.x[0][1][fL], mv = f.x[0][2][fL], mw = f.x[0][3][fL];
            f.x[1][0][fL] = r; f.x[1][1][fL] = mu_; f.x[1][2][fL] = mv; f.x[1][3][fL] = mw;
            f.x[1][4][fL] = P / kc::K_1 + 0.5 * (mu_ * mu_ + mv * mv + mw * mw) / r;
        } else {
#pragma unroll
            for (int q = 0; q < 5; q++) {
                f.x[0][q][f0] = f.x[0][q][fL];
                f.x[1][q][fL] = f.x[1][q][f0];
            }
        }
    } else if ((t -= nx) < ny) { // :75-90
        const int i = (int)((unsigned)t / (unsigned)D), k = (int)((unsigned)t % (unsigned)D);
        const long long f0 = iyf(L, H, D, i, 0, k), fH = iyf(L, H, D, i, H, k);
#pragma unroll
        for (int q = 0; q < 5; q++) {
            if (q == 2 && spatial) {
                f.y[0][q][f0] = -f.y[1][q][f0];
                f.y[1][q][fH] = -f.y[0][q][fH];
            } else {
                f.y[0][q][f0] = f.y[1][q][f0];
                f.y[1][q][fH] = f.y[0][q][fH];
            }
        }
    } else if ((t -= ny) < nz) { // :94-109
        const int i = (int)((unsigned)t / (unsigned)H), j = (int)((unsigned)t % (unsigned)H);
        const long long f0 = izf(L, H, D, i, j, 0), fD = izf(L, H, D, i, j, D);
#pragma unroll
        for (int q = 0; q < 5; q++) {
            f.z[0][q][f0] = f.z[0][q][fD];
            f.z[1][q][fD] = f.z[1][q][f0];
        }
    }
}

// ---------------------------------------------------------------------------
// A4 fluxes (src/fluxes.c:57-571): one thread per face, the three directions in
// one launch.  The flux overwrites the minus-side state array, as in the
// reference.  Bound by FP64 arithmetic and the latency of its chain: the eight
// tangential reciprocals are formed without a branch (rcp_rn, divisions when one
// is out of its range).  96x72x40: 92 us in three launches -> 44 us (four blocks
// an SM 50 us, six 45).
// ---------------------------------------------------------------------------
__device__ __noinline__ double inverse(double x) { return 1. / x; }

// sgs: FSL_SGS_STATIC forms the face viscosity from the face gradients and
// the two cells' densities (src/fluxes.c:193-205, :362-374, :533-545),
// FSL_SGS_NONE uses zero, any other mode the mu_SGS field.
template <int N>
__device__ __forceinline__ void flux_face(const Grid &g, const Consts &kc, const double *__restrict__ u,
                                          const double *__restrict__ mu, const Faces &f, int sgs, unsigned block)
{
    const int H = g.H, D = g.D;
    const int nb = H + (N == 2), nc = D + (N == 3);
    int a, b, c;
    if (!plane_cell(nb, nc, block, a, b, c)) return;
    const long long fs = g.fstride;
    long long fi;
    double *const *mS;
    double *const *pS;
    long long plus, dn, dt1, dt2;
    double rdn, rt1, rt2;
    if (N == 1) {
        fi = ((long long)a * nb + b) * nc + c;
        mS = f.x[0]; pS = f.x[1];
        plus = g.idx(a + 1, b + 1, c + 1); dn = g.pi; dt1 = g.pk; dt2 = 1;
        rdn = kc.rdx; rt1 = kc.r4dy; rt2 = kc.r4dz;
    } else if (N == 2) {
        fi = ((long long)a * nb + b) * nc + c;
        mS = f.y[0]; pS = f.y[1];
        plus = g.idx(a + 1, b + 1, c + 1); dn = g.pk; dt1 = g.pi; dt2 = 1;
        rdn = kc.rdy; rt1 = kc.r4dx; rt2 = kc.r4dz;
    } else {
        fi = ((long long)a * nb + b) * nc + c;
        mS = f.z[0]; pS = f.z[1];
        plus = g.idx(a + 1, b + 1, c + 1); dn = 1; dt1 = g.pi; dt2 = g.pk;
        rdn = kc.rdz; rt1 = kc.r4dx; rt2 = kc.r4dy;
    }
    const long long minus = plus - dn;
    // the neighbours read: plus and minus, each with both tangential offsets
    if (!FSL_SPAN(plus, -dn - (dt1 > dt2 ? dt1 : dt2), dt1 > dt2 ? dt1 : dt2, fs)) return;
    fi = FSL_FACE(fi, (long long)(g.L + (N == 1)) * nb * nc);
    double Lm[5], Rp[5];
#pragma unroll
    for (int q = 0; q < 5; q++) { Lm[q] = mS[q][fi]; Rp[q] = pS[q][fi]; }
    double Rho, P, vel[3];
    riemann<double, N>(Lm, Rp, Rho, P, vel);
    double vp[3], vm[3], Tp, Tm;
    vel_div(u[plus], u[fs + plus], u[2 * fs + plus], u[3 * fs + plus], u[4 * fs + plus], vp, Tp);
    vel_div(u[minus], u[fs + minus], u[2 * fs + minus], u[3 * fs + minus], u[4 * fs + minus], vm, Tm);
    // tangential neighbours: the plus and the minus cell's, at +/- both offsets,
    // with the rounded reciprocal density of src/fluxes.c:124-142
    const long long at[8] = {plus + dt1, minus + dt1, plus - dt1, minus - dt1,
                             plus + dt2, minus + dt2, plus - dt2, minus - dt2};
    double ru[8];
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const double r = u[at[q]];
        ru[q] = rcp_rn(r);
        ok = ok && range_ok(r) && !ones(r);
    }
    if (!ok) {
#pragma unroll
        for (int q = 0; q < 8; q++) ru[q] = inverse(u[at[q]]);
    }
    double s1[3], s2[3]; // sums over the two faces' cells of the tangential differences
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const double *m = u + (q + 1) * fs;
        s1[q] = m[at[0]] * ru[0] + m[at[1]] * ru[1] - m[at[2]] * ru[2] - m[at[3]] * ru[3];
        s2[q] = m[at[4]] * ru[4] + m[at[5]] * ru[5] - m[at[6]] * ru[6] - m[at[7]] * ru[7];
    }
    // g[a][b] = d u_a / d x_b
    double gr[3][3];
    const int n0 = N - 1;
    const int t1 = (N == 1) ? 1 : 0;   // first tangential axis
    const int t2 = (N == 3) ? 1 : 2;   // second tangential axis
#pragma unroll
    for (int q = 0; q < 3; q++) {
        gr[q][n0] = (vp[q] - vm[q]) * rdn;
        gr[q][t1] = s1[q] * rt1;
        gr[q][t2] = s2[q] * rt2;
    }
    // SGS viscosity at the face: x uses the two adjacent cells (:191); the y
    // and z sweeps average the plus cell with its x-neighbour (:360, :531).
    double mu_T;
    if (sgs == FSL_SGS_STATIC) mu_T = static_mu_t<double>(gr, 0.5 * (u[plus] + u[minus]), kc.CsDD);
    else if (sgs == FSL_SGS_NONE) mu_T = 0.0;
    else mu_T = 0.5 * (mu[plus] + mu[plus - g.pi]);
    double F[5];
    face_flux<double, N>(Rho, P, vel, gr, vp, vm, Tp, Tm, kc.mu_L, mu_T, kc.lambda_L, kc.cp_Pr_T, rdn, F);
#pragma unroll
    for (int q = 0; q < 5; q++) mS[q][fi] = F[q];
}

// blocks [0, bx) the x faces, [bx, by) the y faces, the others the z faces
__global__ void __launch_bounds__(kPlaneThreads, 5) k_flux(Grid g, Consts kc, const double *__restrict__ u,
                                                        const double *__restrict__ mu, Faces f, int sgs, unsigned bx,
                                                        unsigned by)
{
    follow();
    if (blockIdx.x < bx) flux_face<1>(g, kc, u, mu, f, sgs, blockIdx.x);
    else if (blockIdx.x < by) flux_face<2>(g, kc, u, mu, f, sgs, blockIdx.x - bx);
    else flux_face<3>(g, kc, u, mu, f, sgs, blockIdx.x - by);
}

// ---------------------------------------------------------------------------
// A7 TVD Runge-Kutta (src/evolution.c:15-245).  mode: 1..3 = RK3 stage,
// 4 = the nStages == 2 chain of stage 1, 5 = the chain of stage 2 (RK2 stage
// 2 followed by RK3 stage 2 on the updated U, src/evolution.c:19-23).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kPlaneThreads) k_evolution(Grid g, int mode, const DevScalars *__restrict__ ds, double *__restrict__ U,
                            double *__restrict__ Up, Faces f)
{
    follow();
    const int L = g.L, H = g.H, D = g.D;
    int i, j, k;
    if (!plane_cell(H, D, blockIdx.x, i, j, k)) return;
    i++; j++; k++;
    const double dtx = ds->dtx, dty = ds->dty, dtz = ds->dtz;
    const double one_third = 1. / 3., two_thirds = 2. / 3.;
    const long long fs = g.fstride, c = FSL_CELL(g.idx(i, j, k), fs);
    const long long xm = ixf(L, H, D, i - 1, j - 1, k - 1), xp = ixf(L, H, D, i, j - 1, k - 1);
    const long long ym = iyf(L, H, D, i - 1, j - 1, k - 1), yp = iyf(L, H, D, i - 1, j, k - 1);
    const long long zm = izf(L, H, D, i - 1, j - 1, k - 1), zp = izf(L, H, D, i - 1, j - 1, k);
#pragma unroll
    for (int q = 0; q < 5; q++) {
        const double X = dtx * (f.x[0][q][xm] - f.x[0][q][xp]);
        const double Y = dty * (f.y[0][q][ym] - f.y[0][q][yp]);
        const double Z = dtz * (f.z[0][q][zm] - f.z[0][q][zp]);
        double *u = U + q * fs, *up = Up + q * fs;
        if (mode == 1 || mode == 4) {
            up[c] = u[c] + X + Y + Z;
        } else if (mode == 2) {
            up[c] = 0.75 * u[c] + 0.25 * (up[c] + X + Y + Z);
        } else if (mode == 3) {
            u[c] = one_third * u[c] + two_thirds * (up[c] + X + Y + Z);
        } else { // mode 5
            const double un = 0.5 * (u[c] + up[c] + X + Y + Z);
            u[c] = un;
            up[c] = 0.75 * un + 0.25 * (up[c] + X + Y + Z);
        }
    }
}

// ---------------------------------------------------------------------------
// A8 Courant maximum (src/helpers.c:23-52).  NaN never wins a comparison, as
// in the reference's `(CoNum = U*deltaT_X) > maxCo`, so the maximum is
// independent of reduction order.
// ---------------------------------------------------------------------------
__global__ void k_courant_partial(Grid g, Consts kc, const double *__restrict__ U,
                                  const DevScalars *__restrict__ ds, double *__restrict__ partials,
                                  DevScalars *__restrict__ dsw, int i0, int i1)
{
    const int H = g.H, D = g.D;
    const long long n = (long long)(i1 - i0 + 1) * H * D; // planes i0..i1
    const long long fs = g.fstride;
    const double dtx = ds->dtx, dty = ds->dty, dtz = ds->dtz;
    double m = 0.0;
    unsigned bad = 0;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t % D) + 1;
        const long long r = t / D;
        const int j = (int)(r % H) + 1;
        const int i = (int)(r / H) + i0;
        const long long c = FSL_CELL(g.idx(i, j, k), g.fstride);
        const double R = U[c];
        const double Co = cell_courant(kc.cfl_mode, R, U[fs + c], kc.cfl_mode == FSL_CFL_ACOUSTIC ? U[2 * fs + c] : 0.,
                                       kc.cfl_mode == FSL_CFL_ACOUSTIC ? U[3 * fs + c] : 0.,
                                       kc.cfl_mode == FSL_CFL_ACOUSTIC ? U[4 * fs + c] : 0., dtx, dty, dtz);
        m = (Co > m) ? Co : m;
        if (!(R > 0.0)) bad = 1;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, m, o);
        m = (x > m) ? x : m;
    }
    __shared__ double sm[32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sm[w] = m;
    if (bad) atomicOr(&dsw->status, 2u);
    __syncthreads();
    if (w == 0) {
        m = (l < (int)(blockDim.x >> 5)) ? sm[l] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double x = __shfl_xor_sync(0xffffffffu, m, o);
            m = (x > m) ? x : m;
        }
        if (l == 0) partials[blockIdx.x] = m;
    }
}

// dt rescale of src/helpers.c:47-50; clears the fused accumulator for the
// next stage 3
__device__ __forceinline__ void apply_courant(const Consts &kc, double maxCo, DevScalars *ds)
{
    double dt = ds->dt;
    dt *= (kc.maxCoNum / maxCo);
    ds->dt = dt;
    ds->dtx = dt / kc.deltaX;
    ds->dty = dt / kc.deltaY;
    ds->dtz = dt / kc.deltaZ;
    ds->maxCo = maxCo;
    ds->co_bits = 0ull;
    if (!(maxCo > 0.0) || !isfinite(maxCo) || !isfinite(dt)) ds->status |= 1u;
}

// Final reduction and the dt rescale of src/helpers.c:47-50.
__global__ void k_courant_final(Consts kc, const double *__restrict__ partials, int np, DevScalars *ds)
{
    double m = 0.0;
    for (int t = threadIdx.x; t < np; t += blockDim.x) {
        const double x = partials[t];
        m = (x > m) ? x : m;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, m, o);
        m = (x > m) ? x : m;
    }
    __shared__ double sm[32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sm[w] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        m = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) m = (sm[q] > m) ? sm[q] : m;
        apply_courant(kc, m, ds);
    }
}

// The maximum of the partials as the accumulator's bit pattern, without the
// dt update (the Courant maximum of a slab, to be combined across slabs).
__global__ void k_courant_to_bits(const double *__restrict__ partials, int np, DevScalars *ds)
{
    if (threadIdx.x != 0) return;
    double m = 0.0;
    for (int t = 0; t < np; t++) m = (partials[t] > m) ? partials[t] : m;
    ds->co_bits = (unsigned long long)__double_as_longlong(m);
}

// The same dt update from the maximum the fused stage 3 of the previous step
// accumulated over the state it wrote (that state is this step's U^n).
__global__ void k_courant_apply(Consts kc, DevScalars *ds)
{
    follow();
    if (threadIdx.x == 0) apply_courant(kc, __longlong_as_double((long long)ds->co_bits), ds);
}

// Per y row: sums over the x-z plane of a, b, (a-b)^2 and b^2 (two padded
// fields) -- the judgement of the learned closure, over the band two cells
// away from every boundary (nearer, the dynamic procedure's values carry the
// zero padding of the reference's test filter); rows outside it are zero.
template <typename TA, typename TB>
__global__ void k_judge_rows(Grid g, const TA *__restrict__ a, const TB *__restrict__ b,
                             double *__restrict__ rows)
{
    const int j = blockIdx.x + 1;
    const int bL = g.L - 4, bD = g.D - 4;
    const long long n = (j >= 3 && j <= g.H - 2) ? (long long)bL * bD : 0;
    double s[4] = {0, 0, 0, 0};
    for (long long t = threadIdx.x; t < n; t += blockDim.x) {
        const int k = (int)(t % bD) + 3;
        const int i = (int)(t / bD) + 3;
        const long long c = FSL_CELL(g.idx(i, j, k), g.fstride);
        const double x = a[c], y = b[c];
        s[0] += x; s[1] += y; s[2] += (x - y) * (x - y); s[3] += y * y;
    }
    __shared__ double sm[4][32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        double x = s[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (l == 0) sm[q][w] = x;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double x = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) x += sm[threadIdx.x][q];
        rows[(long long)blockIdx.x * 4 + threadIdx.x] = x;
    }
}

// ---------------------------------------------------------------------------
// state transfer and diagnostics
// ---------------------------------------------------------------------------
// Planes i0 .. i0+ni-1 (1-based interior planes) between the padded fields and
// the state layout, one warp per row of DEP values, four loads in flight per
// lane, pairs of values where every packed row starts on 16 bytes.  Bound by
// memory: 512x256x256 928 us -> 430 us a direction (three 64-bit divisions per
// value before).
template <bool GATHER, typename V>
__global__ void __launch_bounds__(256) k_state_rows(Grid g, double *__restrict__ fields, double *__restrict__ packed,
                                                    int i0, unsigned nrows)
{
    constexpr int W = sizeof(V) / sizeof(double), UN = 4;
    const unsigned H = (unsigned)g.H, n = (unsigned)g.D / W, l = threadIdx.x & 31;
    for (unsigned row = blockIdx.x * 8u + (threadIdx.x >> 5); row < nrows; row += gridDim.x * 8u) {
        const unsigned ij = row / 5u, v = row - ij * 5u, ii = ij / H, j = ij - ii * H;
        const long long c = g.idx((int)ii + i0, (int)j + 1, 1);
        (void)FSL_CELL(c, g.fstride);
        (void)FSL_CELL(c + g.D - 1, g.fstride);
        V *f = reinterpret_cast<V *>(fields + v * g.fstride + c);
        V *p = reinterpret_cast<V *>(packed + (long long)row * g.D);
        const V *src = GATHER ? f : p;
        V *dst = GATHER ? p : f;
        for (unsigned k = l; k < n; k += 32 * UN) {
            V x[UN];
#pragma unroll
            for (int q = 0; q < UN; q++)
                if (k + 32 * q < n) x[q] = src[k + 32 * q];
#pragma unroll
            for (int q = 0; q < UN; q++)
                if (k + 32 * q < n) dst[k + 32 * q] = x[q];
        }
    }
}

// Deterministic block partial sums of the five conserved variables over
// the interior planes i0 .. i0+ni-1.
__global__ void k_sums_partial(Grid g, int i0, int ni, const double *__restrict__ U, double *__restrict__ partials)
{
    const long long n = (long long)ni * g.H * g.D;
    double s[5] = {0, 0, 0, 0, 0};
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t % g.D) + 1;
        const long long r = t / g.D;
        const int j = (int)(r % g.H) + 1;
        const int i = (int)(r / g.H) + i0;
        const long long c = FSL_CELL(g.idx(i, j, k), g.fstride);
#pragma unroll
        for (int q = 0; q < 5; q++) s[q] += U[q * g.fstride + c];
    }
    __shared__ double sm[5][32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 5; q++) {
        double x = s[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (l == 0) sm[q][w] = x;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        double x = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) x += sm[threadIdx.x][q];
        partials[blockIdx.x * 5 + threadIdx.x] = x;
    }
}

__global__ void k_sums_final(const double *__restrict__ partials, int np, double vol, double *__restrict__ out)
{
    if (threadIdx.x < 5) {
        double x = 0;
        for (int b = 0; b < np; b++) x += partials[b * 5 + threadIdx.x];
        out[threadIdx.x] = x * vol;
    }
}

// Block (y row, segment of the planes i0 .. i0+ni-1): sums over its cells of
// rho, rho u, rho v, rho w, rho uu, rho vv, rho ww, rho uv; a warp per plane.
__global__ void __launch_bounds__(256) k_plane_sums(Grid g, int i0, int ni, int seg, const double *__restrict__ U,
                                                    double *__restrict__ parts)
{
    const int j = blockIdx.x + 1, w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int ib = (int)blockIdx.y * seg, ie = min(ni, ib + seg);
    const long long fs = g.fstride;
    double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = ib + w; i < ie; i += 8) {
        const long long c0 = g.idx(i + i0, j, 1);
#pragma unroll 2
        for (int k = l; k < g.D; k += 32) {
            const long long c = FSL_CELL(c0 + k, fs);
            const double r = U[c], m1 = U[fs + c], m2 = U[2 * fs + c], m3 = U[3 * fs + c];
            const double u = m1 / r, v = m2 / r, ww = m3 / r;
            s[0] += r; s[1] += r * u; s[2] += r * v; s[3] += r * ww;
            s[4] += r * u * u; s[5] += r * v * v; s[6] += r * ww * ww; s[7] += r * u * v;
        }
    }
    __shared__ double sm[8][8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        double x = s[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (l == 0) sm[q][w] = x;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        double x = 0;
#pragma unroll
        for (int q = 0; q < 8; q++) x += sm[threadIdx.x][q];
        parts[((long long)blockIdx.y * g.H + blockIdx.x) * 8 + threadIdx.x] = x;
    }
}

// the segments' sums of every row, in order
__global__ void k_plane_sums_final(int n, int nseg, const double *__restrict__ parts, double *__restrict__ rows)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double x = 0;
    for (int q = 0; q < nseg; q++) x += parts[(long long)q * n + t];
    rows[t] = x;
}

} // namespace

// ---- launchers -------------------------------------------------------------

void launch_ghost(Ctx &c, double *cur)
{
    const Grid &g = c.g;
    const long long n = stage::ghost_cells(g);
    prof_begin(c, FSL_K_BC);
    launch_following(k_ghost, dim3((unsigned)((n + 255) / 256)), 256, 0, c.stream, g, c.k.setup, cur);
    prof_end(c, FSL_K_BC, 1);
}

void launch_recon(Ctx &c, const double *cur)
{
    const Grid &g = c.g;
    const unsigned n = (unsigned)g.L * plane_blocks(g.H, g.D);
    prof_begin(c, FSL_K_RECON);
    if (c.p.recon == FSL_RECON_PPM) launch_following(k_recon<true>, dim3(n), kPlaneThreads, 0, c.stream, g, cur, c.f);
    else launch_following(k_recon<false>, dim3(n), kPlaneThreads, 0, c.stream, g, cur, c.f);
    prof_end(c, FSL_K_RECON, 1);
}

void launch_ifbc(Ctx &c, const Disturb &d)
{
    const Grid &g = c.g;
    const long long n = (long long)g.H * g.D + (long long)g.L * g.D + (long long)g.L * g.H;
    prof_begin(c, FSL_K_BC);
    launch_following(k_ifbc, dim3((unsigned)((n + 255) / 256)), 256, 0, c.stream, g, c.k.setup, c.k.BL_HIG, d, c.f);
    prof_end(c, FSL_K_BC, 1);
}

void launch_fluxes(Ctx &c, const double *cur)
{
    const Grid &g = c.g;
    const unsigned bx = (unsigned)(g.L + 1) * plane_blocks(g.H, g.D);
    const unsigned by = bx + (unsigned)g.L * plane_blocks(g.H + 1, g.D);
    const unsigned n = by + (unsigned)g.L * plane_blocks(g.H, g.D + 1);
    prof_begin(c, FSL_K_FLUX);
    launch_following(k_flux, dim3(n), kPlaneThreads, 0, c.stream, g, c.k, cur, c.mu, c.f, c.p.sgs, bx, by);
    prof_end(c, FSL_K_FLUX, 1);
}

void launch_evolution(Ctx &c, int nstages, int stage)
{
    const Grid &g = c.g;
    int mode = stage >= 3 ? 3 : stage;
    if (nstages == 2) mode = (stage == 1) ? 4 : 5;
    const unsigned n = (unsigned)g.L * plane_blocks(g.H, g.D);
    prof_begin(c, FSL_K_EVOL);
    launch_following(k_evolution, dim3(n), kPlaneThreads, 0, c.stream, g, mode, c.ds, c.U, c.Up, c.f);
    prof_end(c, FSL_K_EVOL, 1);
}

int launch_dynsmag(Ctx &c, const double *U, float *cd)
{
    prof_begin(c, FSL_K_SGS);
    const int e = dyn::march<double>(c.g, c.k, U, c.mu, cd, c.dyn_cut, c.dyn_seg, c.stream);
    prof_end(c, FSL_K_SGS, 1);
    if (!e) return FSL_OK;
    c.err = "dynamic procedure: kernel launch";
    return FSL_ERR_CUDA;
}

void launch_courant(Ctx &c)
{
    const Grid &g = c.g;
    prof_begin(c, FSL_K_CFL);
    k_courant_partial<<<c.npartials, 256, 0, c.stream>>>(g, c.k, c.U, c.ds, c.partials, c.ds, c.co_i0, c.co_i1);
    k_courant_final<<<1, 1024, 0, c.stream>>>(c.k, c.partials, c.npartials, c.ds);
    prof_end(c, FSL_K_CFL, 2);
}

void launch_courant_to_bits(Ctx &c)
{
    prof_begin(c, FSL_K_CFL);
    k_courant_partial<<<c.npartials, 256, 0, c.stream>>>(c.g, c.k, c.U, c.ds, c.partials, c.ds, c.co_i0, c.co_i1);
    k_courant_to_bits<<<1, 32, 0, c.stream>>>(c.partials, c.npartials, c.ds);
    prof_end(c, FSL_K_CFL, 2);
}

void launch_courant_apply(Ctx &c)
{
    prof_begin(c, FSL_K_CFL);
    launch_following(k_courant_apply, dim3(1), 32, 0, c.stream, c.k, c.ds);
    prof_end(c, FSL_K_CFL, 1);
}

template <bool GATHER> static void state_rows(Ctx &c, double *fields, double *packed, int i0, int ni)
{
    if (ni <= 0) return;
    const Grid &g = c.g;
    const long long batch = rows_batch(g.H);
    prof_begin(c, FSL_K_OTHER);
    int launches = 0;
    for (long long b = 0; b < ni; b += batch, launches++) {
        const unsigned nrows = (unsigned)(std::min(batch, ni - b) * g.H * 5);
        const unsigned nblk = std::min((nrows + 7u) / 8u, kRowBlocks);
        double *p = packed + b * g.H * 5 * g.D;
        if (g.D % 2 == 0 && (uintptr_t)p % 16 == 0)
            k_state_rows<GATHER, double2><<<nblk, 256, 0, c.stream>>>(g, fields, p, i0 + (int)b, nrows);
        else k_state_rows<GATHER, double><<<nblk, 256, 0, c.stream>>>(g, fields, p, i0 + (int)b, nrows);
    }
    prof_end(c, FSL_K_OTHER, launches);
}

void launch_state_scatter(Ctx &c, double *dst, const double *packed, int i0, int ni)
{
    state_rows<false>(c, dst, const_cast<double *>(packed), i0, ni);
}

void launch_state_gather(Ctx &c, const double *src, double *packed, int i0, int ni)
{
    state_rows<true>(c, const_cast<double *>(src), packed, i0, ni);
}

void launch_sums(Ctx &c, const double *U, int i0, int ni, double *out5)
{
    const int nb = 148 * 4;
    prof_begin(c, FSL_K_OTHER);
    k_sums_partial<<<nb, 256, 0, c.stream>>>(c.g, i0, ni, U, c.partials);
    const double vol = c.p.deltaX * c.p.deltaY * c.p.deltaZ;
    k_sums_final<<<1, 32, 0, c.stream>>>(c.partials, nb, vol, out5);
    prof_end(c, FSL_K_OTHER, 2);
}

template <typename TA, typename TB> static void judge_rows_t(Ctx &c, const TA *a, const TB *b, double *rows)
{
    prof_begin(c, FSL_K_OTHER);
    k_judge_rows<TA, TB><<<c.g.H, 256, 0, c.stream>>>(c.g, a, b, rows);
    prof_end(c, FSL_K_OTHER, 1);
}
void launch_judge_rows(Ctx &c, const float *a, const float *b, double *rows) { judge_rows_t(c, a, b, rows); }
void launch_judge_rows(Ctx &c, const float *a, const double *b, double *rows) { judge_rows_t(c, a, b, rows); }
void launch_judge_rows(Ctx &c, const double *a, const double *b, double *rows) { judge_rows_t(c, a, b, rows); }

// rows: 8 HIG doubles, followed by scratch for the segments (8 HIG doubles each,
// at most LEN / 2 of them).  One block per row left most SMs a single block's
// latency: 512x256x256 871 -> 250 us.
void launch_plane_sums(Ctx &c, const double *U, int i0, int ni, double *rows)
{
    const int H = c.g.H;
    const int want = std::max(1, std::min((8 * c.sms + H - 1) / H, ni / 2)); // eight blocks an SM
    const int seg = (ni + want - 1) / want, nseg = (ni + seg - 1) / seg;
    prof_begin(c, FSL_K_OTHER);
    k_plane_sums<<<dim3(H, nseg), 256, 0, c.stream>>>(c.g, i0, ni, seg, U, rows + 8 * (size_t)H);
    k_plane_sums_final<<<(8 * H + 127) / 128, 128, 0, c.stream>>>(8 * H, nseg, rows + 8 * (size_t)H, rows);
    prof_end(c, FSL_K_OTHER, 2);
}

} // namespace fsl

// ---------------------------------------------------------------------------
// Allocation-free SGS viscosity (fsl_dynamic_smagorinsky_noalloc).
//
// Callers that cannot allocate device memory hand in their own input and
// output buffers; the procedure's 40 scratch fields live in this fixed static
// device array instead of cudaMalloc'd memory.  Every GPU that loads the
// library holds the array until the process exits.  On the host the symbol
// name only stands in for the array; the device address is looked up once per
// device with cudaGetSymbolAddress (that device current) and cached.
// ---------------------------------------------------------------------------
#include <cmath>
#include <mutex>

static __device__ __align__(256) double fsl_noalloc_scratch[FSL_NOALLOC_SCRATCH_BYTES / sizeof(double)];

namespace {

constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mutex;
double *g_noalloc_ptr[kNoallocMaxDevices] = {nullptr};

// Device address of the scratch array on the current device.
int noalloc_scratch(double **out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return FSL_ERR_NODEVICE;
    if (dev < 0 || dev >= kNoallocMaxDevices) return FSL_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, fsl_noalloc_scratch);
        if (e != cudaSuccess || !p) return FSL_ERR_CUDA;
        g_noalloc_ptr[dev] = static_cast<double *>(p);
    }
    *out = g_noalloc_ptr[dev];
    return FSL_OK;
}

// The dynamic procedure's unfused nine-launch sequence (dyn::sequence: the
// seven-pass filters and the coefficient, each field in its own scratch
// array), on explicit buffers and stream.  The context path runs the fused
// form (dyn::march) without scratch; both give the same bits.
void noalloc_dyn_sequence(const fsl::Grid &g, const fsl::Consts &k, const fsl::dyn::Scratch<double> &s,
                          const double *U, double *mu, cudaStream_t st)
{
    fsl::dyn::sequence<double>(g, k, s, U, mu, nullptr, st);
}

} // namespace

extern "C" int fsl_dynamic_smagorinsky_noalloc(const double *U, double *mu, int LEN, int HIG, int DEP,
                                                double deltaX, double deltaY, double deltaZ, void *stream)
{
    if (!U || !mu || LEN < 2 || HIG < 2 || DEP < 2 || !(deltaX > 0) || !(deltaY > 0) || !(deltaZ > 0))
        return FSL_ERR_ARG;
    // each extent widened before the +2, so no int arithmetic can overflow
    const long long n = ((long long)LEN + 2) * ((long long)HIG + 2) * ((long long)DEP + 2);
    if (n <= 0) return FSL_ERR_ARG;
    if (n > (long long)FSL_NOALLOC_MAX_CELLS) return FSL_ERR_TOO_LARGE;
    // an error left pending by the caller's earlier work is not this call's:
    // report it without clearing it and without starting any work
    if (cudaPeekAtLastError() != cudaSuccess) return FSL_ERR_CUDA;
    double *s = nullptr;
    int rc = noalloc_scratch(&s);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the scratch address belongs to the current device: a stream of another
    // device would run the work against that device's copy of the array
    if (st) {
        int sdev = -1, dev = -1;
        if (cudaStreamGetDevice(st, &sdev) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) return FSL_ERR_ARG;
        if (sdev != dev) return FSL_ERR_ARG;
    }
    fsl::Grid g;
    g.L = LEN; g.H = HIG; g.D = DEP;
    g.pk = DEP + 2;
    g.pi = (long long)(DEP + 2) * (HIG + 2);
    g.off = 0;
    g.fstride = n;
    // derived constants exactly as fsl_init computes them (src/initialize.c:67-94)
    fsl::Consts k{};
    k.r4dx = 1. / (4 * deltaX); k.r4dy = 1. / (4 * deltaY); k.r4dz = 1. / (4 * deltaZ);
    k.r2dx = k.r4dx + k.r4dx; k.r2dy = k.r4dy + k.r4dy; k.r2dz = k.r4dz + k.r4dz;
    k.DD = pow(deltaX * deltaY * deltaZ, 0.666666666666667);
    fsl::dyn::Scratch<double> d;
    d.vel = s; d.t1 = s + 3 * n; d.t2 = s + 12 * n; d.A = s + 21 * n;
    d.Lst = s + 27 * n; d.B = s + 33 * n; d.S = s + 39 * n;
    // zero bands of the filter passes and the A ghost layer must start at 0;
    // the previous call left its values in the shared scratch
    if (cudaMemsetAsync(s, 0, (size_t)(40 * n) * sizeof(double), st) != cudaSuccess) return FSL_ERR_CUDA;
    if (cudaMemsetAsync(mu, 0, (size_t)n * sizeof(double), st) != cudaSuccess) return FSL_ERR_CUDA;
    noalloc_dyn_sequence(g, k, d, U, mu, st);
    if (cudaGetLastError() != cudaSuccess) return FSL_ERR_CUDA;
    return FSL_OK;
}
