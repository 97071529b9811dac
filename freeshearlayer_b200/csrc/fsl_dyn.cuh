// fsl_dyn.cuh -- the dynamic Smagorinsky procedure (src/turbulence.c:17-507),
// as one marching kernel and as separate passes, templated on the arithmetic type T: T = double in
// fsl_phase.cu (the plain method, compiled with --fmad=false, bit-identical to
// the reference) and T = float in fsl_dyn32.cu (the FP32-bulk path's
// filtering and coefficient).  The conserved state U stays FP64 in both.
#pragma once

#include "fsl_check.cuh"
#include "fsl_internal.h"
#include "fsl_phys.cuh"

namespace fsl {
namespace dyn {

constexpr double H3 = 1. / 3.; // box test-filter weight, src/turbulence.c:113

// ---------------------------------------------------------------------------
// A5/A6 (src/turbulence.c:17-507).
// The filter keeps the reference's three sweeps (y, z, x), each
// t = 0; t += a h; t += b h; t += c h, on zero-initialised scratch whose never
// written bands stay zero (the oracle convention for src/turbulence.c:44-45).
// ---------------------------------------------------------------------------
template <typename T> __global__ void k_dyn_vel(Grid g, const double *__restrict__ U, T *__restrict__ vel)
{
    const long long n = (long long)(g.L + 2) * g.pi;
    const long long fs = g.fstride;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        const long long c = FSL_CELL(g.off + t, fs);
        const T rr = T(1.) / T(U[c]); // :201-205
        vel[c] = T(U[fs + c]) * rr;
        vel[fs + c] = T(U[2 * fs + c]) * rr;
        vel[2 * fs + c] = T(U[3 * fs + c]) * rr;
    }
}

// y sweep (:47-61) of u, v, w and their six products (:213-230), computed
// on the fly; i in [0,LEN], j in [1,HIG], k in [0,DEP].
template <typename T> __global__ void k_filt_y_vel(Grid g, const T *__restrict__ vel, T *__restrict__ t1)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int i = blockIdx.z;
    if (k > g.D || j > g.H) return;
    const long long fs = g.fstride, c = g.idx(i, j, k);
    if (!FSL_SPAN(c, -(long long)g.pk, (long long)g.pk, fs)) return;
    T a[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const long long s = c + (r - 1) * (long long)g.pk;
        a[r][0] = vel[s]; a[r][1] = vel[fs + s]; a[r][2] = vel[2 * fs + s];
    }
    T q[3][9];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const T uu = a[r][0], vv = a[r][1], ww = a[r][2];
        q[r][0] = uu; q[r][1] = vv; q[r][2] = ww;
        q[r][3] = uu * uu; q[r][4] = uu * vv; q[r][5] = uu * ww;
        q[r][6] = vv * vv; q[r][7] = vv * ww; q[r][8] = ww * ww;
    }
#pragma unroll
    for (int m = 0; m < 9; m++) {
        T t = 0.;
        t += q[0][m] * T(H3); t += q[1][m] * T(H3); t += q[2][m] * T(H3);
        t1[m * fs + c] = t;
    }
}

// generic y sweep of nf fields
template <typename T> __global__ void k_filt_y(Grid g, int nf, const T *__restrict__ src, T *__restrict__ t1)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int i = blockIdx.z;
    if (k > g.D || j > g.H) return;
    const long long fs = g.fstride, c = g.idx(i, j, k);
    if (!FSL_SPAN(c, -(long long)g.pk, (long long)g.pk, fs)) return;
    for (int m = 0; m < nf; m++) {
        const T *s = src + m * fs;
        T t = 0.;
        t += s[c - g.pk] * T(H3); t += s[c] * T(H3); t += s[c + g.pk] * T(H3);
        t1[m * fs + c] = t;
    }
}

// z sweep (:63-77): i in [0,LEN], j in [0,HIG], k in [1,DEP]
template <typename T> __global__ void k_filt_z(Grid g, int nf, const T *__restrict__ t1, T *__restrict__ t2)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k > g.D || j > g.H) return;
    const long long fs = g.fstride, c = g.idx(i, j, k);
    if (!FSL_SPAN(c, -1LL, 1LL, fs)) return;
    for (int m = 0; m < nf; m++) {
        const T *s = t1 + m * fs;
        T t = 0.;
        t += s[c - 1] * T(H3); t += s[c] * T(H3); t += s[c + 1] * T(H3);
        t2[m * fs + c] = t;
    }
}

// x sweep (:80-95) back into the pass-1 buffer: i in [1,LEN], j in [0,HIG],
// k in [0,DEP]
template <typename T> __global__ void k_filt_x(Grid g, int nf, const T *__restrict__ t2, T *__restrict__ t1)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z + 1;
    if (k > g.D || j > g.H) return;
    const long long fs = g.fstride, c = g.idx(i, j, k);
    if (!FSL_SPAN(c, -g.pi, g.pi, fs)) return;
    for (int m = 0; m < nf; m++) {
        const T *s = t2 + m * fs;
        T t = 0.;
        t += s[c - g.pi] * T(H3); t += s[c] * T(H3); t += s[c + g.pi] * T(H3);
        t1[m * fs + c] = t;
    }
}

// Interior: Leonard stress, |S|, A_ij = |S| S_ij, B_ij = |S^| S^_ij
// (:250-382).  Field order of the symmetric tensors: 11 12 13 22 23 33.
template <typename T>
__global__ void k_dyn_mid(Grid g, Consts kc, const T *__restrict__ vel, const T *__restrict__ F, T *__restrict__ Lst,
                          T *__restrict__ A, T *__restrict__ B, T *__restrict__ Smag)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int i = blockIdx.z + 1;
    if (k > g.D || j > g.H) return;
    const long long fs = g.fstride, c = g.idx(i, j, k);
    if (!FSL_SPAN(c, -g.pi, g.pi, fs)) return;
    const T f0 = F[c], f1 = F[fs + c], f2 = F[2 * fs + c];
    Lst[c] = F[3 * fs + c] - f0 * f0;
    Lst[fs + c] = F[4 * fs + c] - f0 * f1;
    Lst[2 * fs + c] = F[5 * fs + c] - f0 * f2;
    Lst[3 * fs + c] = F[6 * fs + c] - f1 * f1;
    Lst[4 * fs + c] = F[7 * fs + c] - f1 * f2;
    Lst[5 * fs + c] = F[8 * fs + c] - f2 * f2;
    const long long dI = g.pi, dJ = g.pk;
#pragma unroll
    for (int pass = 0; pass < 2; pass++) {
        const T *uu = pass ? F : vel;
        const T *vv = uu + fs, *ww = uu + 2 * fs;
        const T du_dx = (uu[c + dI] - uu[c - dI]) * T(kc.r2dx);
        const T du_dy = (uu[c + dJ] - uu[c - dJ]) * T(kc.r2dy);
        const T du_dz = (uu[c + 1] - uu[c - 1]) * T(kc.r2dz);
        const T dv_dx = (vv[c + dI] - vv[c - dI]) * T(kc.r2dx);
        const T dv_dy = (vv[c + dJ] - vv[c - dJ]) * T(kc.r2dy);
        const T dv_dz = (vv[c + 1] - vv[c - 1]) * T(kc.r2dz);
        const T dw_dx = (ww[c + dI] - ww[c - dI]) * T(kc.r2dx);
        const T dw_dy = (ww[c + dJ] - ww[c - dJ]) * T(kc.r2dy);
        const T dw_dz = (ww[c + 1] - ww[c - 1]) * T(kc.r2dz);
        const T S11 = du_dx, S12 = 0.5 * (du_dy + dv_dx), S13 = 0.5 * (du_dz + dw_dx);
        const T S21 = S12, S22 = dv_dy, S23 = 0.5 * (dv_dz + dw_dy);
        const T S31 = S13, S32 = S23, S33 = dw_dz;
        const T S = sqrt(2 * (S11 * S11 + S12 * S12 + S13 * S13 + S21 * S21 + S22 * S22 + S23 * S23 +
                                   S31 * S31 + S32 * S32 + S33 * S33));
        T *o = pass ? B : A;
        o[c] = S * S11; o[fs + c] = S * S12; o[2 * fs + c] = S * S13;
        o[3 * fs + c] = S * S22; o[4 * fs + c] = S * S23; o[5 * fs + c] = S * S33;
        if (!pass) Smag[c] = S;
    }
}

// M_ij, Germano-Lilly coefficient with clipping to [0, 0.15], mu_SGS
// (:398-445).
template <typename T>
__global__ void k_dyn_final(Grid g, Consts kc, const double *__restrict__ rho, const T *__restrict__ Lst,
                            const T *__restrict__ B, const T *__restrict__ Ahat, const T *__restrict__ Smag,
                            T *__restrict__ mu, float *__restrict__ cd)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int i = blockIdx.z + 1;
    if (k > g.D || j > g.H) return;
    const long long fs = g.fstride, c = g.idx(i, j, k);
    if (!FSL_SPAN(c, 0LL, 0LL, fs)) return;
    const T DD = T(kc.DD);
    const T M11 = DD * (4 * B[c] - Ahat[c]);
    const T M12 = DD * (4 * B[fs + c] - Ahat[fs + c]);
    const T M13 = DD * (4 * B[2 * fs + c] - Ahat[2 * fs + c]);
    const T M22 = DD * (4 * B[3 * fs + c] - Ahat[3 * fs + c]);
    const T M23 = DD * (4 * B[4 * fs + c] - Ahat[4 * fs + c]);
    const T M33 = DD * (4 * B[5 * fs + c] - Ahat[5 * fs + c]);
    T L11 = Lst[c], L12 = Lst[fs + c], L13 = Lst[2 * fs + c];
    T L22 = Lst[3 * fs + c], L23 = Lst[4 * fs + c], L33 = Lst[5 * fs + c];
    const T tr = -(1.0 / 3.0) * (L11 + L22 + L33);
    L11 += tr; L22 += tr; L33 += tr;
    const T LLMM = (L11 * M11 + L12 * M12 + L13 * M13 + L12 * M12 + L22 * M22 + L23 * M23 +
                         L13 * M13 + L23 * M23 + L33 * M33);
    const T MMMM = (M11 * M11 + M12 * M12 + M13 * M13 + M12 * M12 + M22 * M22 + M23 * M23 +
                         M13 * M13 + M23 * M23 + M33 * M33);
    T Cd = -0.5 * (LLMM / (MMMM + 1e-30));
    if (Cd > 0.15) Cd = 0.15;
    else if (Cd < 0.0) Cd = 0.0;
    mu[c] = T(rho[c]) * Cd * DD * Smag[c];
    if (cd) cd[c] = (float)Cd; // Cs^2 for the learned closure's harvest and judgement
}


// ---------------------------------------------------------------------------
// Fused evaluation: the same arithmetic in one kernel that marches along x.
//
// A block owns DYN_J rows x DYN_K columns of output cells; its warps are the
// rows with a one-row halo and its lanes the columns with a two-column halo, so
// every neighbour along z is a lane and every neighbour along y a row of shared
// memory.  Per plane p of velocities it forms
//   - the box filter of u, v, w and their six products: the y pass from the rows'
//     values h q in shared memory, the z pass by shuffles of h t1, the x pass as
//     two running sums -- each sum as 0 + a h + b h + c h, each product by h
//     formed once (the reference forms it three times; the same value);
//   - the filtered velocities and the Leonard stress of plane p-1, and the
//     strain rate and A = |S| S of plane p-1, filtered the same way;
//   - from these |S^| S^, M, the clipped coefficient and mu_SGS of plane p-2
//     (src/turbulence.c:250-445).
// The filter's write regions are the reference's (pass 1: i in [0,L], j in
// [1,H], k in [0,D]; pass 2: k in [1,D]; pass 3: i in [1,L]; plane 0 keeps the
// y-pass value, src/turbulence.c:44-95), zero elsewhere; A is zero outside the
// interior.
//
// Four streaming kernels (velocities, filter, strain, filter of A) with 19
// scratch fields went before: 376 B of traffic a cell and a march of 32 planes
// per block whatever the grid.  This one reads the state once per block, keeps
// everything else on chip (no scratch fields), and cuts the march so that the
// blocks fill the SMs.  It is bound by the latency of shared memory, shuffles and
// dependent arithmetic at 16 warps an SM (issue slots 46 % busy in FP64, 60 %
// in FP32).  The own row's summands come from registers, not shared memory, and
// FP64 forms its two quotients without a branch (3.15 -> 3.00 ms).  Measured:
// FP64 512x256x256 4.21 -> 3.00 ms, 64x32x32 177 -> 33 us; FP32 203x97x75 195 ->
// 74 us.
// ---------------------------------------------------------------------------
constexpr int DYN_W = 16, DYN_J = DYN_W - 2, DYN_K = 28; // warps, output rows, output columns

template <typename T> struct DynSmem {
    double raw[4][DYN_W * 32 + 64];  // rho, rho u, rho v, rho w of the next plane, in flight (own slots)
    T Q[DYN_W + 2][32][9];           // h times u v w uu uv uw vv vw ww of plane p
    T V[2][DYN_W + 2][32][3];        // velocities of planes p, p-1
    T F[2][DYN_W][32][3];            // filtered velocities of planes p-1, p-2
    T A[DYN_W][6][32];               // h A of plane p-1
    // running x sums of the nine filters: FP64 in shared memory (own slots), as
    // registers they would spill at 128 a thread; FP32 in registers
    static constexpr bool XS = sizeof(T) == 8;
    T X[XS ? 18 : 1][DYN_W * 32];
    T t0[XS ? 3 : 1][DYN_W * 32]; // the y pass of plane 0, kept as the sums are
};

template <typename T> __device__ __forceinline__ T sh_up(T v) { return __shfl_up_sync(0xffffffffu, v, 1); }
template <typename T> __device__ __forceinline__ T sh_dn(T v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// |S| and S (11 12 13 22 23 33) from the differences d[a][x] of velocity
// component a along axis x (src/turbulence.c:273-311, :316-366)
template <typename T> __device__ __forceinline__ T strain_of(const T (*d)[3], T *S)
{
    S[0] = d[0][0];
    S[1] = T(0.5) * (d[0][1] + d[1][0]);
    S[2] = T(0.5) * (d[0][2] + d[2][0]);
    S[3] = d[1][1];
    S[4] = T(0.5) * (d[1][2] + d[2][1]);
    S[5] = d[2][2];
    const T S21 = S[1], S31 = S[2], S32 = S[4];
    return sqrt(2 * (S[0] * S[0] + S[1] * S[1] + S[2] * S[2] + S21 * S21 + S[3] * S[3] + S[4] * S[4] + S31 * S31 +
                     S32 * S32 + S[5] * S[5]));
}

// 1/x and a/b rounded as by division; in FP64 without its branch where the
// operands allow (the bounds of quot_rn, b in [2^-100, 2^120) as the 1e-30 added to
// the coefficient's denominator leaves it)
static __device__ __noinline__ double divided(double a, double b) { return a / b; }
__device__ __forceinline__ float inverse_of(float x) { return 1.f / x; }
__device__ __forceinline__ double inverse_of(double x)
{
    double y = rcp_rn(x);
    if (!range_ok(x) || ones(x)) y = divided(1., x);
    return y;
}
__device__ __forceinline__ float ratio_of(float a, float b) { return a / b; }
__device__ __forceinline__ double ratio_of(double a, double b)
{
    double q = quot_signed(a, b, rcp_rn(b));
    const bool in = (unsigned)(__double2hiint(b) - 0x39b00000) < 0x0dc00000u;
    if (!in || !zero_or_range_ok(a) || ones(b)) q = divided(a, b);
    return q;
}

template <typename T>
__global__ void __launch_bounds__(DYN_W * 32, 1)
    k_dyn_march(Grid g, Consts kc, int seg, const double *__restrict__ U, T *__restrict__ mu, float *__restrict__ cd)
{
    follow();
    extern __shared__ __align__(16) unsigned char smraw[];
    DynSmem<T> &s = *reinterpret_cast<DynSmem<T> *>(smraw);
    const int L = g.L, H = g.H, D = g.D;
    const int t = threadIdx.x, l = t & 31, r = t >> 5;
    const int j = (int)blockIdx.y * DYN_J + r, k = (int)blockIdx.x * DYN_K + l - 1; // row 1, lane 2: the first output cell
    const int i0 = 1 + (int)blockIdx.z * seg, i1 = min(L, i0 + seg - 1);
    const long long fs = g.fstride;
    const T h = T(H3), r2x = T(kc.r2dx), r2y = T(kc.r2dy), r2z = T(kc.r2dz);
    // the rows below warp 0's and above the last warp's: an extra cell of those warps
    const bool edge = r == 0 || r == DYN_W - 1;
    const int je = r == 0 ? j - 1 : j + 1;
    const bool kin = k >= 0 && k <= D + 1;
    const bool in = kin && j <= H + 1, ein = edge && kin && je >= 0 && je <= H + 1;
    const long long c0 = in ? g.idx(0, j, k) : 0, ce = ein ? g.idx(0, je, k) : 0;
    const bool y1 = j >= 1 && j <= H && k >= 0 && k <= D; // pass 1 writes here
    const bool z1 = y1 && k >= 1;                         // pass 2, and the interior
    const bool own = z1 && r >= 1 && r <= DYN_J && l >= 2 && l <= DYN_K + 1;

    auto fetch = [&](int p) {
        if (p >= 0 && p <= L + 1) {
#pragma unroll
            for (int w = 0; w < 2; w++) {
                if (w ? !ein : !in) continue;
                const long long c = FSL_CELL((w ? ce : c0) + p * g.pi, fs);
                const int slot = w ? DYN_W * 32 + (r ? 32 : 0) + l : t;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                     (uint32_t)__cvta_generic_to_shared(&s.raw[q][slot])),
                                 "l"(U + q * fs + c)
                                 : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    T v1[3] = {}, v2[3] = {};       // own velocities of planes p-1, p-2
    T f1[3] = {}, f2[3] = {};       // own filtered velocities of planes p-2, p-3
    T Lst[6] = {};                  // Leonard stress of plane p-2
    T a1[6] = {}, a2[6] = {};       // running x sums of the filter of A
    T S1 = T(0.);                   // |S| of plane p-2
    T t0[3] = {};                   // the y pass of plane 0 (FP32)
    double r1 = 0., r2 = 0.;        // density of planes p-1, p-2
    T x1[9] = {}, x2[9] = {};       // running x sums of the nine filters (FP32)
    if constexpr (DynSmem<T>::XS) {
#pragma unroll
        for (int m = 0; m < 18; m++) s.X[m][t] = T(0.);
    }
    const int pb = max(i0 - 2, 0);
    fetch(pb);
    for (int p = pb; p <= i1 + 2; p++) {
        asm volatile("cp.async.wait_group 0;" ::: "memory"); // own copies only: no barrier
        // ---- velocities and h q of plane p
        T v0[3] = {};
        double rho = 0.;
        const bool pin = p <= L + 1;
#pragma unroll
        for (int w = 0; w < 2; w++) {
            if (w && !edge) continue;
            T v[3] = {};
            if (pin && (w ? ein : in)) {
                const int slot = w ? DYN_W * 32 + (r ? 32 : 0) + l : t;
                const double rw = s.raw[0][slot];
                const T rr = inverse_of(T(rw));
                v[0] = T(s.raw[1][slot]) * rr;
                v[1] = T(s.raw[2][slot]) * rr;
                v[2] = T(s.raw[3][slot]) * rr;
                if (!w) rho = rw;
            }
            const int row = w ? (r ? DYN_W + 1 : 0) : r + 1;
            T *q = s.Q[row][l], *o = s.V[p & 1][row][l];
            o[0] = v[0]; o[1] = v[1]; o[2] = v[2];
            q[0] = v[0] * h; q[1] = v[1] * h; q[2] = v[2] * h;
            q[3] = v[0] * v[0] * h; q[4] = v[0] * v[1] * h; q[5] = v[0] * v[2] * h;
            q[6] = v[1] * v[1] * h; q[7] = v[1] * v[2] * h; q[8] = v[2] * v[2] * h;
            if (!w) { v0[0] = v[0]; v0[1] = v[1]; v0[2] = v[2]; }
        }
        __syncthreads();
        if (p < i1 + 2) fetch(p + 1);
        // ---- the nine filters: F of plane p-1
        T fn[3], Ln[6];
        {
            const bool yp = y1 && p <= L, zp = z1 && p <= L;
            T F[9];
            // the own row's values, formed again rather than read or kept
            const T oq[9] = {v0[0] * h, v0[1] * h, v0[2] * h, v0[0] * v0[0] * h, v0[0] * v0[1] * h,
                             v0[0] * v0[2] * h, v0[1] * v0[1] * h, v0[1] * v0[2] * h, v0[2] * v0[2] * h};
#pragma unroll
            for (int m = 0; m < 9; m++) {
                T t1 = T(0.) + s.Q[r][l][m];
                t1 += oq[m];
                t1 += s.Q[r + 2][l][m];
                if (!yp) t1 = T(0.);
                const T th = t1 * h;
                T t2 = T(0.) + sh_up(th);
                t2 += th;
                t2 += sh_dn(th);
                if (!zp) t2 = T(0.);
                const T x = t2 * h;
                if constexpr (DynSmem<T>::XS) {
                    F[m] = s.X[9 + m][t] + x;
                    s.X[9 + m][t] = s.X[m][t] + x;
                    s.X[m][t] = T(0.) + x;
                } else {
                    F[m] = x2[m] + x;
                    x2[m] = x1[m] + x;
                    x1[m] = T(0.) + x;
                }
                if (m < 3) {
                    // plane 0 keeps the y pass
                    if constexpr (DynSmem<T>::XS) {
                        if (p == 1) F[m] = s.t0[m][t];
                        if (p == 0) s.t0[m][t] = t1;
                    } else {
                        if (p == 1) F[m] = t0[m];
                        if (p == 0) t0[m] = t1;
                    }
                }
            }
            const bool none = p > L + 1 || p == 0; // nothing is written on plane L+1 (and none precedes plane 0)
#pragma unroll
            for (int m = 0; m < 3; m++) {
                fn[m] = none ? T(0.) : F[m];
                s.F[(p + 1) & 1][r][l][m] = fn[m];
            }
            Ln[0] = F[3] - F[0] * F[0]; Ln[1] = F[4] - F[0] * F[1]; Ln[2] = F[5] - F[0] * F[2];
            Ln[3] = F[6] - F[1] * F[1]; Ln[4] = F[7] - F[1] * F[2]; Ln[5] = F[8] - F[2] * F[2];
        }
        // ---- strain rate of plane p-1: A and |S|
        T S0 = T(0.), oa[6];
        {
            T d[3][3], A[6];
            const T(*V)[32][3] = s.V[(p + 1) & 1];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                d[a][0] = (v0[a] - v2[a]) * r2x;
                d[a][1] = (V[r + 2][l][a] - V[r][l][a]) * r2y;
                const T up = sh_dn(v1[a]), dn = sh_up(v1[a]);
                d[a][2] = (up - dn) * r2z;
            }
            const bool ap = z1 && p >= 2 && p <= L + 1;
            S0 = strain_of(d, A);
#pragma unroll
            for (int m = 0; m < 6; m++) s.A[r][m][l] = oa[m] = ap ? S0 * A[m] * h : T(0.);
        }
        __syncthreads();
        // ---- the filter of A, and plane p-2
        const bool mid = r >= 1 && r <= DYN_J;
        if (mid) {
            T Ah[6];
#pragma unroll
            for (int m = 0; m < 6; m++) {
                T t1 = T(0.) + s.A[r - 1][m][l];
                t1 += oa[m];
                t1 += s.A[r + 1][m][l];
                if (!y1) t1 = T(0.);
                const T th = t1 * h;
                T t2 = T(0.) + sh_up(th);
                t2 += th;
                t2 += sh_dn(th);
                const T x = (p >= 2 && p <= L + 1) ? t2 * h : T(0.);
                Ah[m] = a2[m] + x;
                a2[m] = a1[m] + x;
                a1[m] = T(0.) + x;
            }
            T d[3][3], Sh_[6];
            const T(*F)[32][3] = s.F[p & 1];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                d[a][0] = (fn[a] - f2[a]) * r2x;
                d[a][1] = (F[r + 1][l][a] - F[r - 1][l][a]) * r2y;
                const T up = sh_dn(f1[a]), dn = sh_up(f1[a]);
                d[a][2] = (up - dn) * r2z;
            }
            const int io = p - 2;
            if (own && io >= i0) {
                const T Sh = strain_of(d, Sh_);
                const T DD = T(kc.DD);
                const T M11 = DD * (4 * (Sh * Sh_[0]) - Ah[0]);
                const T M12 = DD * (4 * (Sh * Sh_[1]) - Ah[1]);
                const T M13 = DD * (4 * (Sh * Sh_[2]) - Ah[2]);
                const T M22 = DD * (4 * (Sh * Sh_[3]) - Ah[3]);
                const T M23 = DD * (4 * (Sh * Sh_[4]) - Ah[4]);
                const T M33 = DD * (4 * (Sh * Sh_[5]) - Ah[5]);
                T L11 = Lst[0], L22 = Lst[3], L33 = Lst[5];
                const T L12 = Lst[1], L13 = Lst[2], L23 = Lst[4];
                const T tr = T(-(1.0 / 3.0)) * (L11 + L22 + L33);
                L11 += tr; L22 += tr; L33 += tr;
                const T LLMM = (L11 * M11 + L12 * M12 + L13 * M13 + L12 * M12 + L22 * M22 + L23 * M23 + L13 * M13 +
                                L23 * M23 + L33 * M33);
                const T MMMM = (M11 * M11 + M12 * M12 + M13 * M13 + M12 * M12 + M22 * M22 + M23 * M23 + M13 * M13 +
                                M23 * M23 + M33 * M33);
                T Cd = T(-0.5) * ratio_of(LLMM, MMMM + T(1e-30));
                if (Cd > T(0.15)) Cd = T(0.15);
                else if (Cd < T(0.0)) Cd = T(0.0);
                const long long c = FSL_CELL(c0 + io * g.pi, fs);
                mu[c] = T(r2) * Cd * DD * S1;
                if (cd) cd[c] = (float)Cd;
            }
        }
        S1 = S0;
        r2 = r1;
        r1 = rho;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            v2[a] = v1[a];
            v1[a] = v0[a];
            f2[a] = f1[a];
            f1[a] = fn[a];
        }
#pragma unroll
        for (int m = 0; m < 6; m++) Lst[m] = Ln[m];
    }
}

inline dim3 cells_grid3(dim3 b, int ni, int nj, int nk)
{
    return dim3((unsigned)((nk + b.x - 1) / b.x), (unsigned)((nj + b.y - 1) / b.y), (unsigned)ni);
}

// Scratch fields of one evaluation (each `fstride` elements of T).
template <typename T> struct Scratch {
    T *vel, *t1, *t2, *A, *Lst, *B, *S;
};

// The nine launches of one evaluation on `st`: velocities, the filter of the
// velocities and their products (y, z, x), Leonard stress, |S| S and |S^| S^,
// the filter of A (y, z, x) and the coefficient; mu in T, Cd as FP32 (or not).
template <typename T>
void sequence(const Grid &g, const Consts &k, const Scratch<T> &s, const double *U, T *mu, float *cd,
              cudaStream_t st)
{
    const long long ncell = (long long)(g.L + 2) * g.pi;
    k_dyn_vel<T><<<(unsigned)std::min<long long>((ncell + 255) / 256, 148LL * 16), 256, 0, st>>>(g, U, s.vel);
    const dim3 b(32, 4, 1);
    // velocity and product filters: y over i in [0,L] j in [1,H] k in [0,D]
    k_filt_y_vel<T><<<cells_grid3(b, g.L + 1, g.H, g.D + 1), b, 0, st>>>(g, s.vel, s.t1);
    k_filt_z<T><<<cells_grid3(b, g.L + 1, g.H + 1, g.D), b, 0, st>>>(g, 9, s.t1, s.t2);
    k_filt_x<T><<<cells_grid3(b, g.L, g.H + 1, g.D + 1), b, 0, st>>>(g, 9, s.t2, s.t1);
    k_dyn_mid<T><<<cells_grid3(b, g.L, g.H, g.D), b, 0, st>>>(g, k, s.vel, s.t1, s.Lst, s.A, s.B, s.S);
    // filter of A (pass-1 buffer reused; its zero bands are preserved)
    k_filt_y<T><<<cells_grid3(b, g.L + 1, g.H, g.D + 1), b, 0, st>>>(g, 6, s.A, s.t1);
    k_filt_z<T><<<cells_grid3(b, g.L + 1, g.H + 1, g.D), b, 0, st>>>(g, 6, s.t1, s.t2);
    k_filt_x<T><<<cells_grid3(b, g.L, g.H + 1, g.D + 1), b, 0, st>>>(g, 6, s.t2, s.t1);
    k_dyn_final<T><<<cells_grid3(b, g.L, g.H, g.D), b, 0, st>>>(g, k, U, s.Lst, s.B, s.t1, s.S, mu, cd);
}

// Planes of tiles of one evaluation.
inline long long march_units(const Grid &g)
{
    return (long long)((g.D + DYN_K - 1) / DYN_K) * ((g.H + DYN_J - 1) / DYN_J) * g.L;
}

// The march is cut so that the blocks fill
// the SMs in whole waves: a segment of n planes costs n + 4 (the planes its
// filters reach), and the number of waves times that is least.
inline int march_cut(const Grid &g, int sms)
{
    const long long tiles = march_units(g) / g.L;
    int seg = 1;
    long long best = -1;
    for (int n = 1; n <= g.L; n++) {
        const long long segs = (g.L + n - 1) / n;
        if (n > 1 && segs == (g.L + n - 2) / (n - 1)) continue; // the same number of blocks with longer segments
        const long long cost = (tiles * segs + sms - 1) / sms * (n + 4);
        if (best < 0 || cost < best) {
            best = cost;
            seg = n;
        }
    }
    return seg;
}

// The fused evaluation: one launch, marches of `cut` planes.  A domain that does
// not have the SMs to itself is given the length of its longest march instead, which
// its marches share evenly (longest 0: not given).
template <typename T>
int march(const Grid &g, const Consts &k, const double *U, T *mu, float *cd, int cut, int longest, cudaStream_t st)
{
    static std::atomic<uint64_t> attr{0};
    if (!smem_limit_once((const void *)k_dyn_march<T>, sizeof(DynSmem<T>), attr)) return -1;
    const unsigned nk = (unsigned)((g.D + DYN_K - 1) / DYN_K), nj = (unsigned)((g.H + DYN_J - 1) / DYN_J);
    int seg = cut;
    if (longest > 0) {
        const int segs = (g.L + longest - 1) / longest;
        seg = (g.L + segs - 1) / segs;
    }
    launch_following(k_dyn_march<T>, dim3(nk, nj, (unsigned)((g.L + seg - 1) / seg)), DYN_W * 32, sizeof(DynSmem<T>), st, g,
                     k, seg, U, mu, cd);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

} // namespace dyn
} // namespace fsl
