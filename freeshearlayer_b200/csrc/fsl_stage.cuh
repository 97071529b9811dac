// fsl_stage.cuh -- fused RK3 stage kernel and boundary-face pass, templated on
// the compute type T.  Instantiated for T = double (fsl_fused.cu, compiled
// with --fmad=false: the plain method, bit-identical to the reference) and
// T = float (fsl_fused32.cu: FP32 bulk, FP64 stage accumulation).
//
// Decomposition ("2.5-D" streaming): a block owns a tile of (TJE-2) x 30
// cell columns in (y, z) plus a one-cell halo ring (TJE rows = warps, 32
// lanes along the contiguous k axis) and marches along x over `seg` planes.
// Per plane it stages in shared memory the current-stage state (two planes,
// halo 2), the two velocity forms the viscous stencil reads (src/fluxes.c
// divides for the two cells adjacent to a face, :117-122, and multiplies by a
// reciprocal for the eight tangential neighbours, :124-142), temperature and
// the face-averaged SGS viscosity.  Every face flux of the tile is computed
// once (x faces in registers carried along the march, y faces through shared
// memory, z faces through warp shuffles); the state is read once and the
// stage result written once.  Plane i+2 (PPM: i+3) is asked for at the top of
// iteration i, which hides its latency behind the flux work: in FP64 by asynchronous
// copies into a ring slot of its own, in FP32 into registers that are converted and
// stored to shared memory at the iteration's end.  Domain-boundary faces take their outer state
// from the boundary pass (k_boundary), which applies the reference's interface
// rules (src/bounCondOnInterfaces.c:11-110) to the reconstructed boundary cells.
#pragma once

#include "fsl_check.cuh"
#include "fsl_internal.h"
#include "fsl_phys.cuh"

namespace fsl {
namespace stage {

template <typename T> struct BF {
    T *x0, *xL, *y0, *yH, *z0, *zD;
};

template <typename T>
__device__ __forceinline__ void load5(const double *__restrict__ u, long long fs, long long c, T *v)
{
#pragma unroll
    for (int q = 0; q < 5; q++) v[q] = T(u[q * fs + FSL_CELL(c, fs)]);
}

// reconstruction sweep DIR (0 x, 1 y, 2 z) of the padded cell c
template <typename T, int DIR>
__device__ __forceinline__ void recon_at(const Grid &g, const double *__restrict__ u, long long c, T *hi, T *lo)
{
    const long long fs = g.fstride;
    CellC<T> cc;
    load5(u, fs, c, cc.u);
    cell_consts(cc);
    const long long d = DIR == 0 ? g.pi : DIR == 1 ? (long long)g.pk : 1LL;
    const int p1 = DIR == 0 ? 1 : DIR == 1 ? 2 : 3;
    const int p2 = DIR == 0 ? 2 : DIR == 1 ? 3 : 1;
    const int p3 = DIR == 0 ? 3 : DIR == 1 ? 1 : 2;
    T fw[5], bw[5];
    const long long cf = FSL_CELL(c + d, fs), cb = FSL_CELL(c - d, fs);
    fw[0] = T(u[cf]); fw[1] = T(u[p1 * fs + cf]); fw[2] = T(u[p2 * fs + cf]);
    fw[3] = T(u[p3 * fs + cf]); fw[4] = T(u[4 * fs + cf]);
    bw[0] = T(u[cb]); bw[1] = T(u[p1 * fs + cb]); bw[2] = T(u[p2 * fs + cb]);
    bw[3] = T(u[p3 * fs + cb]); bw[4] = T(u[4 * fs + cb]);
    if (DIR == 0) recon_x(cc, fw, bw, hi, lo);
    else if (DIR == 1) recon_y(cc, fw, bw, hi, lo);
    else recon_z(cc, fw, bw, hi, lo);
}

// PPM x-sweep of the padded cell c (planes c-2 .. c+2 from global memory)
template <typename T>
__device__ __forceinline__ void ppm_at_x(const Grid &g, const double *__restrict__ u, long long c, T *hi, T *lo)
{
    const long long fs = g.fstride, d = g.pi;
    CellC<T> cc;
    T m2[5], m1[5], p1[5], p2[5];
    load5(u, fs, c, cc.u);
    load5(u, fs, c - 2 * d, m2);
    load5(u, fs, c - d, m1);
    load5(u, fs, c + d, p1);
    load5(u, fs, c + 2 * d, p2);
    cell_consts(cc);
    ppm_x(cc, m2, m1, p1, p2, hi, lo);
}

// State on the outer face of the boundary cell c in direction DIR: the upper
// face (UP) or the lower one, from the cell, its inner neighbour and the ghost
// value g5 beyond the face (FP64, natural order).
template <typename T, int DIR, bool UP>
__device__ __forceinline__ void edge_state(const Grid &g, const double *__restrict__ u, long long c, const double *g5,
                                           T *out)
{
    const long long fs = g.fstride;
    CellC<T> cc;
    load5(u, fs, c, cc.u);
    cell_consts(cc);
    const long long d = DIR == 0 ? g.pi : DIR == 1 ? (long long)g.pk : 1LL;
    const int p1 = DIR == 0 ? 1 : DIR == 1 ? 2 : 3;
    const int p2 = DIR == 0 ? 2 : DIR == 1 ? 3 : 1;
    const int p3 = DIR == 0 ? 3 : DIR == 1 ? 1 : 2;
    T in[5], go[5], other[5];
    const long long ci = FSL_CELL(UP ? c - d : c + d, fs);
    in[0] = T(u[ci]); in[1] = T(u[p1 * fs + ci]); in[2] = T(u[p2 * fs + ci]);
    in[3] = T(u[p3 * fs + ci]); in[4] = T(u[4 * fs + ci]);
    go[0] = T(g5[0]); go[1] = T(g5[p1]); go[2] = T(g5[p2]); go[3] = T(g5[p3]); go[4] = T(g5[4]);
    T *hi = UP ? out : other, *lo = UP ? other : out;
    const T *fw = UP ? go : in, *bw = UP ? in : go;
    if (DIR == 0) recon_x(cc, fw, bw, hi, lo);
    else if (DIR == 1) recon_y(cc, fw, bw, hi, lo);
    else recon_z(cc, fw, bw, hi, lo);
}

// The ghost value beyond the interior boundary cell s in direction DIR, before
// the other directions' copies (src/boundCondInGhostCells.c:10-96): `c` the cell
// it copies, with the spatial setup's slip wall and outflow.  Explicitly rounded,
// so both precisions' translation units form the ghost pass's bits.
__device__ __forceinline__ void ghost_value(const double *__restrict__ u, long long fs, long long c, bool flip,
                                            bool outflow, double *v)
{
#pragma unroll
    for (int q = 0; q < 5; q++) v[q] = u[q * fs + c];
    if (outflow) { // :44-52: momenta copied, E rebuilt at P = 1e5
        const double q = __dadd_rn(__dadd_rn(__dmul_rn(v[1], v[1]), __dmul_rn(v[2], v[2])), __dmul_rn(v[3], v[3]));
        v[4] = __dadd_rn(__ddiv_rn(100000., 0.4), __ddiv_rn(__dmul_rn(0.5, q), v[0]));
    }
    if (flip) v[2] = -v[2];
}

// Ghost cell t of the ghost layer (x planes, y rows and z columns in turn).  The
// reference fills x, then z over all i, then y over all i and k; every ghost
// value is therefore a composition of copies of one interior cell (or of the
// inflow profile), which is evaluated here for one cell, edges and corners
// included.  32-bit divisions: no list is longer than 2^32 on 2^31 cells.
__device__ __forceinline__ void ghost_cell(const Grid &g, bool spatial, double *__restrict__ u, long long t)
{
    const int L = g.L, H = g.H, D = g.D;
    const long long ax = (long long)(H + 2) * (D + 2), ay = (long long)L * (D + 2), az = (long long)L * H;
    int i, j, k;
    if (t < 2 * ax) {
        const bool up = t >= ax;
        const unsigned r = (unsigned)(up ? t - ax : t), w = (unsigned)D + 2u;
        i = up ? L + 1 : 0;
        j = (int)(r / w);
        k = (int)(r - (unsigned)j * w);
    } else if ((t -= 2 * ax) < 2 * ay) {
        const bool up = t >= ay;
        const unsigned r = (unsigned)(up ? t - ay : t), w = (unsigned)D + 2u, q = r / w;
        j = up ? H + 1 : 0;
        i = 1 + (int)q;
        k = (int)(r - q * w);
    } else {
        t -= 2 * ay;
        const bool up = t >= az;
        const unsigned r = (unsigned)(up ? t - az : t), w = (unsigned)H, q = r / w;
        k = up ? D + 1 : 0;
        i = 1 + (int)q;
        j = 1 + (int)(r - q * w);
    }
    const int jj = j == 0 ? 1 : j == H + 1 ? H : j, kk = k == 0 ? D : k == D + 1 ? 1 : k;
    const bool flip = spatial && jj != j;
    const long long fs = g.fstride;
    double v[5];
    if (i == 0 && spatial) {
        // inflow step profile, :17-40
        const double P = 100000., R = 1.0;
        const double U = (jj <= H / 2) ? 76.4 : 200;
        v[0] = R; v[1] = R * U; v[2] = 0.; v[3] = 0.;
        v[4] = __dadd_rn(P / 0.4, __dmul_rn(0.5 * R, __dmul_rn(U, U)));
        if (flip) v[2] = -v[2];
    } else {
        const int si = i == 0 ? L : i == L + 1 ? (spatial ? L : 1) : i;
        ghost_value(u, fs, FSL_CELL(g.idx(si, jj, kk), fs), flip, spatial && i == L + 1, v);
    }
    const long long d = FSL_CELL(g.idx(i, j, k), fs);
#pragma unroll
    for (int q = 0; q < 5; q++) u[q * fs + d] = v[q];
}
__host__ __device__ inline long long ghost_cells(const Grid &g)
{
    return 2LL * (g.H + 2) * (g.D + 2) + 2LL * g.L * (g.D + 2) + 2LL * g.L * g.H;
}

// Outer states of one domain-boundary face (src/bounCondOnInterfaces.c:11-110):
// face t of the x (HIG DEP), y (LEN DEP) and z (LEN HIG) boundary lists, the lower
// boundary's face or (upper) the other's.
template <typename T>
__device__ __forceinline__ void bface_one(const Grid &g, bool spatial, int BL_HIG, const Disturb &d,
                                          const double *__restrict__ u, const BF<T> &bf, long long t, bool upper)
{
    const int L = g.L, H = g.H, D = g.D;
    const long long nx = (long long)H * D, ny = (long long)L * D, nz = (long long)L * H, fs = g.fstride;
    typedef Kc<T> kc;
    T o[5];
    double gv[5];
    if (t < nx) {
        const unsigned r = (unsigned)t;
        const int jf = (int)(r / (unsigned)D), kf = (int)(r - (unsigned)jf * (unsigned)D);
        const int j = jf + 1, k = kf + 1;
        const long long fo = FSL_FACE(t, nx);
        if (spatial && !upper) {
            // inflow profile in the reference's FP64 arithmetic (:17-60)
            const double P = 100000., R = 1.0;
            double U, V = 0., W = 0., v[5];
            if (jf < H / 2) {
                U = 76.4;
                v[0] = R; v[1] = R * U; v[2] = 0.; v[3] = 0.; v[4] = P / 0.4 + 0.5 * R * (U * U);
            } else if (jf < H / 2 + BL_HIG) {
                const unsigned ku = (unsigned)kf;
                bool dist;
                if (d.k_max > d.k_min) dist = (ku >= d.k_min && ku < d.k_max);
                else dist = !(ku >= d.k_max && ku < d.k_min);
                if (dist) { U = 200. + d.Ud; V = d.Vd; W = d.Wd; }
                else { U = 200.; V = W = 0.; }
                v[0] = R; v[1] = R * U; v[2] = R * V; v[3] = R * W;
                v[4] = P / 0.4 + 0.5 * R * (U * U + V * V + W * W);
            } else {
                U = 200.;
                v[0] = R; v[1] = R * U; v[2] = 0.; v[3] = 0.; v[4] = P / 0.4 + 0.5 * R * (U * U);
            }
#pragma unroll
            for (int q = 0; q < 5; q++) bf.x0[q * nx + fo] = T(v[q]);
        } else if (spatial) {
            // :62-71 outflow from the minus state of face LEN
            const long long c = g.idx(L, j, k);
            ghost_value(u, fs, FSL_CELL(c, fs), false, true, gv);
            edge_state<T, 0, true>(g, u, c, gv, o);
            const T r_ = o[0], mu_ = o[1], mv = o[2], mw = o[3];
            const T P_ = T(100000.);
            bf.xL[fo] = r_; bf.xL[nx + fo] = mu_; bf.xL[2 * nx + fo] = mv; bf.xL[3 * nx + fo] = mw;
            bf.xL[4 * nx + fo] = P_ / kc::K_1 + T(0.5) * (mu_ * mu_ + mv * mv + mw * mw) / r_;
        } else if (!upper) { // periodic x, the reference's z rule (:94-109)
            ghost_value(u, fs, FSL_CELL(g.idx(1, j, k), fs), false, false, gv);
            edge_state<T, 0, true>(g, u, g.idx(L, j, k), gv, o);
#pragma unroll
            for (int q = 0; q < 5; q++) bf.x0[q * nx + fo] = o[q];
        } else {
            ghost_value(u, fs, FSL_CELL(g.idx(L, j, k), fs), false, false, gv);
            edge_state<T, 0, false>(g, u, g.idx(1, j, k), gv, o);
#pragma unroll
            for (int q = 0; q < 5; q++) bf.xL[q * nx + fo] = o[q];
        }
    } else if ((t -= nx) < ny) { // :75-90
        const unsigned r = (unsigned)t, q_ = r / (unsigned)D;
        const int i = (int)q_ + 1, k = (int)(r - q_ * (unsigned)D) + 1;
        const long long c = g.idx(i, upper ? H : 1, k), fo = FSL_FACE(t, ny);
        ghost_value(u, fs, FSL_CELL(c, fs), spatial, false, gv);
        if (upper) edge_state<T, 1, true>(g, u, c, gv, o);
        else edge_state<T, 1, false>(g, u, c, gv, o);
        T *dst = upper ? bf.yH : bf.y0;
#pragma unroll
        for (int q = 0; q < 5; q++) dst[q * ny + fo] = (q == 2 && spatial) ? -o[q] : o[q];
    } else if ((t -= ny) < nz) { // :94-109
        const unsigned r = (unsigned)t, q_ = r / (unsigned)H;
        const int i = (int)q_ + 1, j = (int)(r - q_ * (unsigned)H) + 1;
        const long long fo = FSL_FACE(t, nz);
        if (!upper) {
            ghost_value(u, fs, FSL_CELL(g.idx(i, j, 1), fs), false, false, gv);
            edge_state<T, 2, true>(g, u, g.idx(i, j, D), gv, o);
        } else {
            ghost_value(u, fs, FSL_CELL(g.idx(i, j, D), fs), false, false, gv);
            edge_state<T, 2, false>(g, u, g.idx(i, j, 1), gv, o);
        }
        T *dst = upper ? bf.zD : bf.z0;
#pragma unroll
        for (int q = 0; q < 5; q++) dst[q * nz + fo] = o[q];
    }
}

// The boundary pass before a fused stage: the ghost layer of u and the outer
// states of the boundary faces, in one launch -- the faces form the ghost values
// they need from the interior, so neither waits for the other (two dependent
// launches of 5 and 9 us at 100x80x35 before).
template <typename T>
__global__ void __launch_bounds__(128) k_boundary(Grid g, int setup, int BL_HIG, Disturb d, double *__restrict__ u,
                                                  BF<T> bf)
{
    follow();
    const long long nf = (long long)g.H * g.D + (long long)g.L * g.D + (long long)g.L * g.H;
    const bool spatial = setup == FSL_SETUP_SPATIAL;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 2 * nf) {
        const bool upper = t >= nf;
        bface_one<T>(g, spatial, BL_HIG, d, u, bf, upper ? t - nf : t, upper);
    } else if ((t -= 2 * nf) < ghost_cells(g)) {
        ghost_cell(g, spatial, u, t);
    }
}

template <typename T, int TJE, bool PPM = false> struct Smem {
    static constexpr int HW = PPM ? 2 : 1; // y/z halo width of the state planes
    // FP64 planes arrive in shared memory by asynchronous copies, into a slot of
    // their own (in registers, as the FP32 bulk's conversion needs them, a plane in
    // flight costs 20 of the 128 a thread has); FP32 planes replace a slot whose
    // readers are done
    static constexpr bool ASYNC = sizeof(T) == 8;
    static constexpr int NS = (PPM ? 4 : 2) + (ASYNC ? 1 : 0); // x-planes in the state ring
    __device__ static __forceinline__ int slot(int p) { return ASYNC ? (p + NS) % NS : p & (NS - 1); }
    // current-stage state: planes i, i+1 (PPM: i-1 .. i+2; FP64: and the next) as
    // a ring, with HW halo rows and lanes
    T U[NS][TJE + 2 * HW][32 + 2 * HW][5];
    T R[3][TJE][32][3];     // velocities by reciprocal, planes i-1, i, i+1 (ring)
    T Dv[2][TJE][32][5];    // velocities by division, temperature, mu face average, planes i, i+1
    T Lo[TJE][32][5];       // y sweep: state on the face below each cell
    T Fy[TJE][32][5];       // y flux on the face above each row
    // FP64: sound speed, 1/(2C) and 1/(2C)/C of planes i, i+1 (with R the roots
    // of the cell's characteristic transform), formed once per cell instead of
    // by the y and z sweeps and again by the x sweep a plane earlier
    static constexpr bool ROOTS = sizeof(T) == 8;
    T C[2][ROOTS ? TJE : 1][32][3];
};

template <typename T> struct Args {
    const double *cur; // current-stage state, ghost layer filled
    const double *un;  // U^n
    double *out;
    const T *mu;
    BF<T> bf;
    const DevScalars *ds;
    unsigned long long *co; // non-null: accumulate the Courant maximum of `out` (stage 3)
    int co_i0, co_i1;       // over planes co_i0..co_i1 only
    unsigned int *status;   // bit 1 set on a non-positive output density (with co)
    int stage;
    int seg;
    // non-null (full-lane tile, temporal setup): also write the FP32 velocities
    // of `out`, ghost cells included, as the closure's velocity pass forms them
    float *vel;
};

// Own column of plane `pl` (and, on the tile edge, the halo neighbour the y
// and z sweeps need) from global memory into registers.
// Kept in the storage type (FP64) while in flight: a conversion at load
// time would wait on the load immediately.
struct PlaneLoad {
    double own[5], halo[5], halo2[5]; // halo2: the second halo cell (PPM)
};

// FP64: straight into the plane's ring slot; else into registers.
__device__ __forceinline__ void copy5_async(double *dst, const double *__restrict__ u, long long fs, long long c)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const double *src = u + FSL_CELL(c, fs);
#pragma unroll
    for (int q = 0; q < 5; q++)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + q * 8u), "l"(src + q * fs) : "memory");
}
__device__ __forceinline__ void copies_done()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

template <typename T, int TJE, bool PPM>
__device__ __forceinline__ void plane_issue(Smem<T, TJE, PPM> &s, const Grid &g, const double *__restrict__ cu, int pl,
                                            int r, int l, int j, int k, bool live, PlaneLoad &p)
{
    constexpr int HW = Smem<T, TJE, PPM>::HW;
    const long long fs = g.fstride;
    if (!live || pl > g.L + 1) return;
    const long long c = g.idx(pl, j, k);
    auto get = [&](double *reg, int rr, int ll, long long cell) {
        if constexpr (Smem<T, TJE, PPM>::ASYNC)
            copy5_async(s.U[Smem<T, TJE, PPM>::slot(pl)][rr][ll], cu, fs, cell);
        else load5(cu, fs, cell, reg);
    };
    get(p.own, r + HW, l + HW, c);
    if (r == 0 && j >= 1) {
        get(p.halo, HW - 1, l + HW, c - g.pk);
        if (PPM && j >= 2) get(p.halo2, 0, l + HW, c - 2 * g.pk);
    } else if (r == TJE - 1 && j <= g.H) {
        get(p.halo, TJE + HW, l + HW, c + g.pk);
        if (PPM && j <= g.H - 1) get(p.halo2, TJE + HW + 1, l + HW, c + 2 * g.pk);
    } else if (l == 0 && k >= 1) {
        get(p.halo, r + HW, HW - 1, c - 1);
        if (PPM && k >= 2) get(p.halo2, r + HW, 0, c - 2);
    } else if (l == 31 && k <= g.D) {
        get(p.halo, r + HW, 32 + HW, c + 1);
        if (PPM && k <= g.D - 1) get(p.halo2, r + HW, 33 + HW, c + 2);
    }
}

template <typename T, int TJE, bool PPM>
__device__ __forceinline__ void plane_store(Smem<T, TJE, PPM> &s, int slot, int r, int l, int j, int k, int H, int D,
                                            bool live, const PlaneLoad &p)
{
    constexpr int HW = Smem<T, TJE, PPM>::HW;
    if constexpr (Smem<T, TJE, PPM>::ASYNC) return; // already there
    if (!live) return;
#pragma unroll
    for (int q = 0; q < 5; q++) s.U[slot][r + HW][l + HW][q] = T(p.own[q]);
    T *h = nullptr, *h2 = nullptr;
    if (r == 0 && j >= 1) {
        h = s.U[slot][HW - 1][l + HW];
        if (PPM && j >= 2) h2 = s.U[slot][0][l + HW];
    } else if (r == TJE - 1 && j <= H) {
        h = s.U[slot][TJE + HW][l + HW];
        if (PPM && j <= H - 1) h2 = s.U[slot][TJE + HW + 1][l + HW];
    } else if (l == 0 && k >= 1) {
        h = s.U[slot][r + HW][HW - 1];
        if (PPM && k >= 2) h2 = s.U[slot][r + HW][0];
    } else if (l == 31 && k <= D) {
        h = s.U[slot][r + HW][32 + HW];
        if (PPM && k <= D - 1) h2 = s.U[slot][r + HW][33 + HW];
    }
    if (h) {
#pragma unroll
        for (int q = 0; q < 5; q++) h[q] = T(p.halo[q]);
    }
    if (PPM && h2) {
#pragma unroll
        for (int q = 0; q < 5; q++) h2[q] = T(p.halo2[q]);
    }
}

// Velocities of plane `pl` (own column, from the shared ring) into the
// reciprocal ring and the division plane with the face-averaged viscosity.
template <typename T, int TJE, bool PPM, bool SST>
__device__ __forceinline__ void plane_prims(Smem<T, TJE, PPM> &s, int pl, int r, int l, T mu_pl, T mu_prev)
{
    constexpr int HW = Smem<T, TJE, PPM>::HW;
    const T *u = s.U[Smem<T, TJE, PPM>::slot(pl)][r + HW][l + HW];
    T dv[4];
    if constexpr (Smem<T, TJE, PPM>::ROOTS) {
        CellC<T> c;
#pragma unroll
        for (int q = 0; q < 5; q++) c.u[q] = u[q];
        cell_prims64(c, dv); // U, V, W are the reciprocal velocities of vel_rcp
        T *v = s.R[pl % 3][r][l], *k = s.C[pl & 1][r][l];
        v[0] = c.U; v[1] = c.V; v[2] = c.W;
        k[0] = c.C; k[1] = c.ll; k[2] = c.ee;
    } else {
        vel_rcp(u[0], u[1], u[2], u[3], s.R[pl % 3][r][l]);
        vdiv(u, dv);
    }
    T *o = s.Dv[pl & 1][r][l];
    o[0] = dv[0]; o[1] = dv[1]; o[2] = dv[2]; o[3] = dv[3];
    if constexpr (!SST) o[4] = T(0.5) * (mu_pl + mu_prev);
}

// The characteristic transform of the own cell of plane `pl` (state cell u),
// from the stored roots or from the state.
template <typename T, int TJE, bool PPM>
__device__ __forceinline__ void ring_consts(const Smem<T, TJE, PPM> &s, const T *u, int pl, int r, int l, CellC<T> &c)
{
#pragma unroll
    for (int q = 0; q < 5; q++) c.u[q] = u[q];
    if constexpr (Smem<T, TJE, PPM>::ROOTS) {
        const T *v = s.R[pl % 3][r][l], *k = s.C[pl & 1][r][l];
        c.U = v[0]; c.V = v[1]; c.W = v[2];
        c.C = k[0]; c.ll = k[1]; c.ee = k[2];
        cell_products(c);
    } else {
        cell_consts(c);
    }
}

// The FP32 kernels' results depend in their last bits on where a march begins (its
// prologue and its loop are compiled apart).  A march is therefore cut into `split`
// parts for the SMs a small grid leaves idle without moving its beginning: a part
// that begins inside computes WARM planes before the first it writes, so that all
// it takes over -- the flux of face i - 1/2, the x sweep's state and the velocities
// of plane i-1 -- was formed by the loop, and the cut shows in no bit.
constexpr int WARM = 3;

// First plane of part p of a march of n planes in `split` parts of equal cost, each
// but the first paying for its WARM planes.
__host__ __device__ inline long long part_begin(long long n, int p, int split)
{
    if (p == 0) return 0;
    return n < WARM ? n : (n + WARM * (split - 1)) * p / split - (long long)WARM * (p - 1);
}

// SST: static Smagorinsky (the face viscosity from the face gradients and the
// two cells' densities; no mu field is read).  SPLIT: the blocks of a segment along
// z are its parts (their number follows from the grid: one more argument made the
// FP64 kernels' compilation spill, 1.6 % and with PPM 4 % of their time).
template <typename T, int TJE, int MINB, bool PPM, bool SST, bool SPLIT = false>
__global__ void __launch_bounds__(TJE * 32, MINB) k_stage(Grid g, Consts kc, Args<T> a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    typedef Smem<T, TJE, PPM> SM;
    SM &s = *reinterpret_cast<SM *>(smraw);
    constexpr int HW = SM::HW;
    const int L = g.L, H = g.H, D = g.D;
    constexpr int TJ = TJE - 2;
    const int r = threadIdx.y, l = threadIdx.x;
    const int j = blockIdx.y * TJ + r;
    const int k = blockIdx.x * 30 + l;
    const int split = SPLIT ? (int)gridDim.z / ((L + a.seg - 1) / a.seg) : 1;
    int i0 = 1 + (SPLIT ? blockIdx.z / split : blockIdx.z) * a.seg;
    int i1 = min(L, i0 + a.seg - 1), iw = i0; // iw: the first plane written
    if constexpr (SPLIT) {
        const int n = i1 - i0 + 1, p = (int)blockIdx.z % split, b = i0;
        iw = b + (int)part_begin(n, p, split);
        i1 = b + (int)part_begin(n, p + 1, split) - 1;
        if (iw > i1) return;
        i0 = max(b, iw - WARM);
    }
    const bool live = (j <= H + 1) && (k <= D + 1);
    const bool inter = live && r >= 1 && r <= TJE - 2 && l >= 1 && l <= 30 && j <= H && k <= D;
    const bool ycol = live && l >= 1 && l <= 30 && k <= D;     // column takes part in y faces
    const bool zrow = live && r >= 1 && r <= TJE - 2 && j <= H; // row takes part in z faces
    const long long fs = g.fstride;
    const double *__restrict__ cu = a.cur;
    const T *__restrict__ mu = a.mu;
    const long long nxf = (long long)H * D, nyf = (long long)L * D, nzf = (long long)L * H;
    const long long cj = g.idx(0, j, k); // column base (plane 0)

    T hix[5], Fxp[5];
#pragma unroll
    for (int q = 0; q < 5; q++) hix[q] = Fxp[q] = T(0.);
    T mu0 = 0, mu1 = 0, mu2 = 0; // mu of planes i, i+1, i+2 (own column)
    PlaneLoad pl;
#pragma unroll
    for (int q = 0; q < 5; q++) pl.own[q] = pl.halo[q] = pl.halo2[q] = 0.;
    double base[5], unv[5]; // FP64 operands of the stage combination, fetched early
#pragma unroll
    for (int q = 0; q < 5; q++) base[q] = unv[q] = 0.;

    // ---- prologue: planes i0-1 .. i0+1 (PPM: .. i0+2), flux of face i0 - 1/2 ----
    {
        T Um[5] = {0, 0, 0, 0, 0}, mum = 0;
        plane_issue<T, TJE, PPM>(s, g, cu, i0, r, l, j, k, live, pl);
        plane_store<T, TJE, PPM>(s, SM::slot(i0), r, l, j, k, H, D, live, pl);
        plane_issue<T, TJE, PPM>(s, g, cu, i0 + 1, r, l, j, k, live, pl);
        plane_store<T, TJE, PPM>(s, SM::slot(i0 + 1), r, l, j, k, H, D, live, pl);
        if constexpr (PPM) {
            plane_issue<T, TJE, PPM>(s, g, cu, i0 + 2, r, l, j, k, live, pl);
            plane_store<T, TJE, PPM>(s, SM::slot(i0 + 2), r, l, j, k, H, D, live && i0 + 2 <= L + 1, pl);
        }
        if constexpr (SM::ASYNC) copies_done(); // the own cell's copies; the barrier below shows the others'
        if (live) {
            load5(cu, fs, cj + (long long)(i0 - 1) * g.pi, Um);
            if constexpr (PPM) {
                // plane i0-1 (own column): the x sweep of cell i0+1 reads it
#pragma unroll
                for (int q = 0; q < 5; q++) s.U[SM::slot(i0 - 1)][r + HW][l + HW][q] = Um[q];
            }
            vel_rcp(Um[0], Um[1], Um[2], Um[3], s.R[(i0 - 1) % 3][r][l]);
            if constexpr (!SST) {
                mum = mu[FSL_CELL(cj + (long long)(i0 - 1) * g.pi, fs)];
                mu0 = mu[FSL_CELL(cj + (long long)i0 * g.pi, fs)];
                mu1 = mu[FSL_CELL(cj + (long long)(i0 + 1) * g.pi, fs)];
            }
            plane_prims<T, TJE, PPM, SST>(s, i0, r, l, mu0, mum);
            plane_prims<T, TJE, PPM, SST>(s, i0 + 1, r, l, mu1, mu0);
        }
        __syncthreads();
        if (inter) {
            T hm[5], lo[5], hin[5], dm[4], tmp[5];
            const T *Uc = s.U[SM::slot(i0)][r + HW][l + HW], *Un = s.U[SM::slot(i0 + 1)][r + HW][l + HW];
            {
                CellC<T> cc;
#pragma unroll
                for (int q = 0; q < 5; q++) cc.u[q] = Uc[q];
                cell_consts(cc);
                if (PPM && i0 >= 2 && i0 <= L - 1) {
                    T m2[5];
                    load5(cu, fs, cj + (long long)(i0 - 2) * g.pi, m2);
                    ppm_x(cc, m2, Um, Un, s.U[SM::slot(i0 + 2)][r + HW][l + HW], hin, lo);
                } else {
                    recon_x(cc, Un, Um, hin, lo);
                }
            }
            if (i0 == 1) {
                const long long fo = (long long)(j - 1) * D + (k - 1);
#pragma unroll
                for (int q = 0; q < 5; q++) hm[q] = a.bf.x0[q * nxf + FSL_FACE(fo, nxf)];
            } else if (PPM && i0 - 1 >= 2 && i0 - 1 <= L - 1) {
                ppm_at_x<T>(g, cu, cj + (long long)(i0 - 1) * g.pi, hm, tmp);
            } else {
                recon_at<T, 0>(g, cu, cj + (long long)(i0 - 1) * g.pi, hm, tmp);
            }
            vdiv(Um, dm);
            const T *dc = s.Dv[i0 & 1][r][l];
            const int sb = (i0 - 1) % 3, sf = i0 % 3;
            const T m_f = SST ? T(0.5) * (Uc[0] + Um[0]) : dc[4];
            fused_face<T, 1, SST>(hm, lo, dm, dm[3], dc, dc[3], s.R[sf][r + 1][l], s.R[sb][r + 1][l],
                                  s.R[sf][r - 1][l], s.R[sb][r - 1][l], s.R[sf][r][l + 1], s.R[sb][r][l + 1],
                                  s.R[sf][r][l - 1], s.R[sb][r][l - 1], m_f, kc, Fxp);
#pragma unroll
            for (int q = 0; q < 5; q++) hix[q] = hin[q];
        }
    }
    const double dtx = a.ds->dtx, dty = a.ds->dty, dtz = a.ds->dtz;
    const double one_third = 1. / 3., two_thirds = 2. / 3.;
    // Courant maximum of the cells this thread wrote (with a.co); in shared
    // memory rather than registers, which the FP64 16-row tile has none left of
    __shared__ double comax[TJE][32];
    comax[r][l] = 0.0;
    __syncthreads();

    for (int i = i0; i <= i1; i++) {
        const int sm1 = (i + 2) % 3, s0 = i % 3, sp1 = (i + 1) % 3;
        const int u0 = i & 1, u1 = (i + 1) & 1;                   // Dv ring
        const int q0 = SM::slot(i), q1 = SM::slot(i + 1);         // state ring: planes i, i+1
        // (a) issue plane i+2 (PPM: i+3) loads (the velocities of plane i+1
        // were formed at the end of the previous iteration, or in the prologue)
        plane_issue<T, TJE, PPM>(s, g, cu, i + (PPM ? 3 : 2), r, l, j, k, live, pl);
        if (inter) {
            const long long c = FSL_CELL(cj + (long long)i * g.pi, fs);
            // FP64 takes the combination's stage state from the ring and U^n at
            // its end, from L2 where it is asked for here
            if (sizeof(T) == 8 && a.stage != 1) {
#pragma unroll
                for (int q = 0; q < 5; q++) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.un + q * fs + c));
            }
            // FP32 bulk keeps only a converted copy of the state in shared
            // memory; the FP64 operands of the combination are fetched here
            if (sizeof(T) != 8) {
#pragma unroll
                for (int q = 0; q < 5; q++) base[q] = cu[q * fs + c];
                if (a.stage != 1 && (!SPLIT || i >= iw)) { // (the planes before iw are another block's)
#pragma unroll
                    for (int q = 0; q < 5; q++) unv[q] = a.un[q * fs + c];
                }
            }
        }
        if (!SST && live && i + 2 <= L + 1) mu2 = mu[FSL_CELL(cj + (long long)(i + 2) * g.pi, fs)];
        // (b) y and z reconstruction of cell (i, j, k): reads the state ring
        // only (plane i, stored two iterations ago)
        T hy[5], hz[5], lz[5];
#pragma unroll
        for (int q = 0; q < 5; q++) hy[q] = hz[q] = lz[q] = T(0.);
        {
            const bool ry = ycol && j >= 1 && j <= H;
            const bool rz = zrow && k >= 1 && k <= D;
            if (ry || rz) {
                CellC<T> cc;
                ring_consts<T, TJE, PPM>(s, s.U[q0][r + HW][l + HW], i, r, l, cc);
                T fw[5], bw[5], lo[5];
                if (ry) {
                    const T *a1 = s.U[q0][r + HW + 1][l + HW], *b1 = s.U[q0][r + HW - 1][l + HW];
                    fw[0] = a1[0]; fw[1] = a1[2]; fw[2] = a1[3]; fw[3] = a1[1]; fw[4] = a1[4];
                    bw[0] = b1[0]; bw[1] = b1[2]; bw[2] = b1[3]; bw[3] = b1[1]; bw[4] = b1[4];
                    if (PPM && j >= 2 && j <= H - 1) {
                        const T *a2 = s.U[q0][r + HW + 2][l + HW], *b2 = s.U[q0][r + HW - 2][l + HW];
                        T f2[5], b2v[5];
                        f2[0] = a2[0]; f2[1] = a2[2]; f2[2] = a2[3]; f2[3] = a2[1]; f2[4] = a2[4];
                        b2v[0] = b2[0]; b2v[1] = b2[2]; b2v[2] = b2[3]; b2v[3] = b2[1]; b2v[4] = b2[4];
                        ppm_y(cc, b2v, bw, fw, f2, hy, lo);
                    } else {
                        recon_y(cc, fw, bw, hy, lo);
                    }
#pragma unroll
                    for (int q = 0; q < 5; q++) s.Lo[r][l][q] = lo[q];
                }
                if (rz) {
                    const T *a1 = s.U[q0][r + HW][l + HW + 1], *b1 = s.U[q0][r + HW][l + HW - 1];
                    fw[0] = a1[0]; fw[1] = a1[3]; fw[2] = a1[1]; fw[3] = a1[2]; fw[4] = a1[4];
                    bw[0] = b1[0]; bw[1] = b1[3]; bw[2] = b1[1]; bw[3] = b1[2]; bw[4] = b1[4];
                    if (PPM && k >= 2 && k <= D - 1) {
                        const T *a2 = s.U[q0][r + HW][l + HW + 2], *b2 = s.U[q0][r + HW][l + HW - 2];
                        T f2[5], b2v[5];
                        f2[0] = a2[0]; f2[1] = a2[3]; f2[2] = a2[1]; f2[3] = a2[2]; f2[4] = a2[4];
                        b2v[0] = b2[0]; b2v[1] = b2[3]; b2v[2] = b2[1]; b2v[3] = b2[2]; b2v[4] = b2[4];
                        ppm_z(cc, b2v, bw, fw, f2, hz, lz);
                    } else {
                        recon_z(cc, fw, bw, hz, lz);
                    }
                }
            }
            if (ycol && j == 0) {
                const long long fo = (long long)(i - 1) * D + (k - 1);
#pragma unroll
                for (int q = 0; q < 5; q++) hy[q] = a.bf.y0[q * nyf + FSL_FACE(fo, nyf)];
            }
            if (ycol && j == H + 1) {
                const long long fo = (long long)(i - 1) * D + (k - 1);
#pragma unroll
                for (int q = 0; q < 5; q++) s.Lo[r][l][q] = a.bf.yH[q * nyf + FSL_FACE(fo, nyf)];
            }
            if (zrow && k == 0) {
                const long long fo = (long long)(i - 1) * H + (j - 1);
#pragma unroll
                for (int q = 0; q < 5; q++) hz[q] = a.bf.z0[q * nzf + FSL_FACE(fo, nzf)];
            }
            if (zrow && k == D + 1) {
                const long long fo = (long long)(i - 1) * H + (j - 1);
#pragma unroll
                for (int q = 0; q < 5; q++) lz[q] = a.bf.zD[q * nzf + FSL_FACE(fo, nzf)];
            }
        }
        __syncthreads();
        // (c) y face above the cell: (i, j + 1/2), j in [0, HIG]
        if (ycol && r <= TJE - 2 && j <= H) {
            T F[5];
            const T *vm = s.Dv[u0][r][l], *vp = s.Dv[u0][r + 1][l];
            const T m_f = SST ? T(0.5) * (s.U[q0][r + 1 + HW][l + HW][0] + s.U[q0][r + HW][l + HW][0]) : vp[4];
            fused_face<T, 2, SST>(hy, s.Lo[r + 1][l], vm, vm[3], vp, vp[3], s.R[sp1][r + 1][l], s.R[sp1][r][l],
                                  s.R[sm1][r + 1][l], s.R[sm1][r][l], s.R[s0][r + 1][l + 1], s.R[s0][r][l + 1],
                                  s.R[s0][r + 1][l - 1], s.R[s0][r][l - 1], m_f, kc, F);
#pragma unroll
            for (int q = 0; q < 5; q++) s.Fy[r][l][q] = F[q];
        }
        // (d) z face nearer than the cell: (i, j, k + 1/2), k in [0, DEP]
        T Fz[5], Fzm[5];
        {
            T lzn[5];
#pragma unroll
            for (int q = 0; q < 5; q++) lzn[q] = __shfl_down_sync(0xffffffffu, lz[q], 1);
#pragma unroll
            for (int q = 0; q < 5; q++) Fz[q] = T(0.);
            if (zrow && l <= 30 && k <= D) {
                const T *vm = s.Dv[u0][r][l], *vp = s.Dv[u0][r][l + 1];
                const T m_f = SST ? T(0.5) * (s.U[q0][r + HW][l + 1 + HW][0] + s.U[q0][r + HW][l + HW][0]) : vp[4];
                fused_face<T, 3, SST>(hz, lzn, vm, vm[3], vp, vp[3], s.R[sp1][r][l + 1], s.R[sp1][r][l],
                                      s.R[sm1][r][l + 1], s.R[sm1][r][l], s.R[s0][r + 1][l + 1], s.R[s0][r + 1][l],
                                      s.R[s0][r - 1][l + 1], s.R[s0][r - 1][l], m_f, kc, Fz);
            }
#pragma unroll
            for (int q = 0; q < 5; q++) Fzm[q] = __shfl_up_sync(0xffffffffu, Fz[q], 1);
        }
        // (e) x face (i + 1/2, j, k): reconstruct cell i+1, flux
        T Fx[5], hin[5];
#pragma unroll
        for (int q = 0; q < 5; q++) Fx[q] = hin[q] = T(0.);
        if constexpr (SM::ASYNC) copies_done(); // the next plane's own cell
        if (inter) {
            T lo[5];
            if (i + 1 <= L) {
                CellC<T> cc;
                ring_consts<T, TJE, PPM>(s, s.U[q1][r + HW][l + HW], i + 1, r, l, cc);
                if constexpr (PPM) {
                    // planes i-1 .. i+2 from the ring (own column), i+3 in flight
                    const T *Um1 = s.U[SM::slot(i - 1)][r + HW][l + HW], *U0 = s.U[q0][r + HW][l + HW];
                    const T *Up2 = s.U[SM::slot(i + 2)][r + HW][l + HW];
                    if (i + 1 <= L - 1) {
                        T p2[5];
#pragma unroll
                        for (int q = 0; q < 5; q++)
                            p2[q] = SM::ASYNC ? s.U[SM::slot(i + 3)][r + HW][l + HW][q] : T(pl.own[q]);
                        ppm_x(cc, Um1, U0, Up2, p2, hin, lo);
                    } else {
                        recon_x(cc, Up2, U0, hin, lo);
                    }
                } else {
                    T fw2[5];
#pragma unroll
                    for (int q = 0; q < 5; q++)
                        fw2[q] = SM::ASYNC ? s.U[SM::slot(i + 2)][r + HW][l + HW][q] : T(pl.own[q]);
                    recon_x(cc, fw2, s.U[q0][r + HW][l + HW], hin, lo);
                }
            } else {
                const long long fo = (long long)(j - 1) * D + (k - 1);
#pragma unroll
                for (int q = 0; q < 5; q++) lo[q] = a.bf.xL[q * nxf + FSL_FACE(fo, nxf)];
            }
            const T *dc = s.Dv[u0][r][l], *dn = s.Dv[u1][r][l];
            const T m_f = SST ? T(0.5) * (s.U[q1][r + HW][l + HW][0] + s.U[q0][r + HW][l + HW][0]) : dn[4];
            fused_face<T, 1, SST>(hix, lo, dc, dc[3], dn, dn[3], s.R[sp1][r + 1][l], s.R[s0][r + 1][l],
                                  s.R[sp1][r - 1][l], s.R[s0][r - 1][l], s.R[sp1][r][l + 1], s.R[s0][r][l + 1],
                                  s.R[sp1][r][l - 1], s.R[s0][r][l - 1], m_f, kc, Fx);
        }
        __syncthreads();
        // (f) divergence and stage combination (src/evolution.c:29-161), FP64
        if (inter && (!SPLIT || i >= iw)) {
            const long long c = FSL_CELL(cj + (long long)i * g.pi, fs);
            const T *Uc = s.U[q0][r + HW][l + HW];
            (void)Uc;
#pragma unroll
            for (int q = 0; q < 5; q++) {
                double o;
                if constexpr (sizeof(T) == 8) {
                    // the reference's order, ((b0 + X) + Y) + Z, on the stage
                    // state itself (the shared copy is exact for T = double)
                    const double X = dtx * ((double)Fxp[q] - (double)Fx[q]);
                    const double Y = dty * ((double)s.Fy[r - 1][l][q] - (double)s.Fy[r][l][q]);
                    const double Z = dtz * ((double)Fzm[q] - (double)Fz[q]);
                    const double b0 = (double)Uc[q];
                    if (a.stage != 1) unv[q] = a.un[q * fs + c];
                    if (a.stage == 1) o = b0 + X + Y + Z;
                    else if (a.stage == 2) o = 0.75 * unv[q] + 0.25 * (b0 + X + Y + Z);
                    else o = one_third * unv[q] + two_thirds * (b0 + X + Y + Z);
                } else {
                    // FP32 bulk: the divergence in FP32 (one conversion), the
                    // stage combination in FP64 on the FP64 stage state
                    const T X = T(dtx) * (Fxp[q] - Fx[q]);
                    const T Y = T(dty) * (s.Fy[r - 1][l][q] - s.Fy[r][l][q]);
                    const T Z = T(dtz) * (Fzm[q] - Fz[q]);
                    const double inc = (double)(X + Y + Z);
                    if (a.stage == 1) o = base[q] + inc;
                    else if (a.stage == 2) o = 0.75 * unv[q] + 0.25 * (base[q] + inc);
                    else o = one_third * unv[q] + two_thirds * (base[q] + inc);
                }
                a.out[q * fs + c] = o;
                base[q] = o; // the new state, for the Courant number below
            }
            if (a.co && i >= a.co_i0 && i <= a.co_i1) {
                // the next step's check of src/helpers.c:23-52 on this state
                const double Co = cell_courant(kc.cfl_mode, base[0], base[1], base[2], base[3], base[4], dtx, dty, dtz);
                const double m = comax[r][l];
                comax[r][l] = (Co > m) ? Co : m;
                if (!(base[0] > 0.0)) atomicOr(a.status, 2u);
            }
        }
        // (g) FP32: plane i+2 (PPM: i+3) into the ring slot of plane i (PPM: i-1; all
        // its readers passed the barrier above); FP64 planes are there already.  The
        // velocities of plane i+2 into the slots of planes i-1 (reciprocal ring) and
        // i (division planes), read next after the next iteration's barrier; advance
        // the march
        if constexpr (PPM)
            plane_store<T, TJE, PPM>(s, SM::slot(i + 3), r, l, j, k, H, D, live && i + 3 <= L + 1, pl);
        else
            plane_store<T, TJE, PPM>(s, q0, r, l, j, k, H, D, live && i + 2 <= L + 1, pl);
        if (live && i < i1) plane_prims<T, TJE, PPM, SST>(s, i + 2, r, l, mu2, mu1);
#pragma unroll
        for (int q = 0; q < 5; q++) {
            Fxp[q] = Fx[q];
            hix[q] = hin[q];
        }
        mu0 = mu1;
        mu1 = mu2;
    }
    if (a.co) {
        __syncthreads();
        double m = comax[r][l];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double x = __shfl_xor_sync(0xffffffffu, m, o);
            m = (x > m) ? x : m;
        }
        __syncthreads();
        if (l == 0) comax[r][0] = m;
        __syncthreads();
        if (r == 0 && l == 0) {
            m = 0.0;
#pragma unroll
            for (int q = 0; q < TJE; q++) m = (comax[q][0] > m) ? comax[q][0] : m;
            // non-negative doubles order like their bit patterns
            atomicMax(a.co, (unsigned long long)__double_as_longlong(m));
        }
    }
}

// Parts of each march: as many as fill the SMs the grid's blocks leave idle, down
// to two planes a part.  Used where no bit may change (the FP32 PPM tile).  Three
// stages at 64x32x32 983 -> 172 us, 128x64x64 993 -> 395 us, 110x48x80 998 -> 333 us;
// with more than half the SMs at work in the one wave a second part has no SM to run
// on.  (Several waves are not cut, though the last may be uneven: 300 marches on 148 SMs
// at 256x128x128 end after 100 planes where an even share is 90.)
inline int march_split(const Grid &g, int nb, int seg, int sms)
{
    return std::max(1, std::min(sms / nb, std::min(seg, g.L) / 2));
}

template <typename T, int TJE, int MINB, bool PPM = false, bool SST = false>
int launch_stage_t(Ctx &c, int stage, const double *cur, const double *un, double *out, const T *mu, BF<T> bf,
                   bool courant, int seg = 0)
{
    const Grid &g = c.g;
    Args<T> a;
    a.cur = cur; a.un = un; a.out = out; a.mu = mu; a.bf = bf; a.ds = c.ds; a.stage = stage;
    a.co = courant ? &c.ds->co_bits : nullptr;
    a.co_i0 = c.co_i0;
    a.co_i1 = c.co_i1;
    a.status = &c.ds->status;
    a.seg = seg > 0 ? seg : c.stage_seg;
    a.vel = nullptr;
    const size_t smem = sizeof(Smem<T, TJE, PPM>);
    static std::atomic<uint64_t> attr{0};
    if (!smem_limit_once((const void *)k_stage<T, TJE, MINB, PPM, SST>, smem, attr)) return -1;
    dim3 b(32, TJE, 1);
    dim3 gr((g.D + 29) / 30, (g.H + TJE - 3) / (TJE - 2), (g.L + a.seg - 1) / a.seg);
    if constexpr (sizeof(T) == 4 && PPM && TJE == 16) {
        const long long nb = (long long)gr.x * gr.y * gr.z;
        const int split = nb * 2 <= c.sms ? march_split(g, (int)nb, a.seg, c.sms) : 1;
        if (split > 1) {
            static std::atomic<uint64_t> attr_split{0};
            if (!smem_limit_once((const void *)k_stage<T, TJE, MINB, PPM, SST, true>, smem, attr_split)) return -1;
            gr.z *= split;
            prof_begin(c, FSL_K_STAGE);
            k_stage<T, TJE, MINB, PPM, SST, true><<<gr, b, smem, c.stream>>>(g, c.k, a);
            prof_end(c, FSL_K_STAGE, 1);
            return cudaGetLastError() == cudaSuccess ? 0 : -1;
        }
    }
    prof_begin(c, FSL_K_STAGE);
    k_stage<T, TJE, MINB, PPM, SST><<<gr, b, smem, c.stream>>>(g, c.k, a);
    prof_end(c, FSL_K_STAGE, 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <typename T> void launch_boundary_t(Ctx &c, double *cur, const Disturb &d, BF<T> bf)
{
    const Grid &g = c.g;
    const long long n =
        2 * ((long long)g.H * g.D + (long long)g.L * g.D + (long long)g.L * g.H) + ghost_cells(g);
    prof_begin(c, FSL_K_BC);
    launch_following(k_boundary<T>, dim3((unsigned)((n + 127) / 128)), 128, 0, c.stream, g, c.k.setup, c.k.BL_HIG, d, cur, bf);
    prof_end(c, FSL_K_BC, 1);
}

} // namespace stage
} // namespace fsl
