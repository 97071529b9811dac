// fsl_phys.cuh -- device arithmetic of the explicit step, templated on the
// compute type T (double for the plain method, float for the FP32 bulk).
//
// Every expression keeps the reference's evaluation order; translation units
// that instantiate T = double are compiled with --fmad=false so that the plain
// method rounds exactly like the reference's serial CPU code (IEEE division
// and square root are the CUDA defaults for double).
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

// Arithmetic templates callable from host code too (an instrumented
// instantiation counts their operations; the kernels use T = double, float).
#define FSL_HD __host__ __device__ __forceinline__

namespace fsl {

// gas and scheme constants, src/def.h:25-45
template <typename T> struct Kc {
    static constexpr T K = T(1.4);
    static constexpr T K_1 = T(0.4);
    static constexpr T NK_1 = T(-0.4);
    static constexpr T K05 = T(0.7);
    static constexpr T K_K_1 = T(3.5);
    static constexpr T K_1_2 = T(0.2);
    static constexpr T H_K_1 = T(1.25);
    static constexpr T R_VOZD = T(287.10);
    static constexpr T C1 = T(0.333333333333333);
    static constexpr T C2 = T(0.166666666666667);
    static constexpr T TWO_THIRDS = T(0.666666666666667);
};

// Chakravarthy-Osher minmod, compression 4 (src/reconstruction.c:17-24),
// written as selects: the same comparisons on the same values, so the same
// result, without data-dependent branches that split a warp.  (y = 0 never
// reaches |4y|: x y = 0 returns 0 first.)
template <typename T> FSL_HD T minmod(T x, T y)
{
    const T y4 = y * T(4.0);
    const T ay = (y4 > T(0)) ? y4 : -y4;
    const T r = (x > T(0)) ? ((x < ay) ? x : ay) : ((-x < ay) ? x : -ay);
    return (x * y <= T(0)) ? T(0) : r;
}

// minmod(a, b) and minmod(b, a) at once: both are 0 when a b <= 0, else
// sign(a) min(|a|, 4|b|) and sign(b) min(|b|, 4|a|) -- exactly the values of
// the select form above (min, |.|, x4 and the sign copy are exact; in FP64, where one
// of the two is NaN, so is one result in either form, and the sweep adds the two), with
// one product and one sign test for the pair.  FP64 takes the minimum as a compare
// and a select and the sign by bits, which keeps the FP64 pipe to six
// instructions a pair instead of fourteen (with the stored roots of the ring
// tile, stage::Smem::C, the FP64 stage went from 8.35 to 7.30 ms a launch at
// 512x256x256).
template <typename T> FSL_HD void minmod2(T a, T b, T &ab, T &ba)
{
    const bool z = a * b <= T(0);
    const T fa = fabs(a), fb = fabs(b);
    if constexpr (std::is_same<T, float>::value) {
        const T m1 = copysign(fmin(fa, T(4) * fb), a);
        const T m2 = copysign(fmin(fb, T(4) * fa), b);
        ab = z ? T(0) : m1;
        ba = z ? T(0) : m2;
    } else {
        const T fa4 = T(4.0) * fa, fb4 = T(4.0) * fb;
        const T m1 = copysign((fa < fb4) ? fa : fb4, a);
        const T m2 = copysign((fb < fa4) ? fb : fa4, b);
        ab = z ? T(0) : m1;
        ba = z ? T(0) : m2;
    }
}

// The pair as the reference-order sweep takes it: minmod2 in FP64 (the same
// values), the two calls the reference writes for any other number type (the
// operation counter's).
template <typename T> FSL_HD void minmod_pair(T a, T b, T &ab, T &ba)
{
    if constexpr (std::is_same<T, double>::value) {
        minmod2(a, b, ab, ba);
    } else {
        ab = minmod(a, b);
        ba = minmod(b, a);
    }
}

// ---------------------------------------------------------------------------
// Correctly rounded FP64 reciprocals and quotients without branches (device).
// The FP64 stage's time goes with its IEEE divisions (53 a cell): each expands
// into a guarded sequence whose branch cuts the compiler's schedule, so that the
// chains of a face's divisions do not overlap.  Here the range is checked once for
// a whole group (a face's Riemann solve, a cell's primitives) and quotients by one
// denominator share its reciprocal.
//
// rcp_rn: Newton's iteration from the gross reciprocal (20 bits); the last step,
// from within an ulp, gives the rounded reciprocal unless b's significand is all
// ones (Markstein, IBM J. Res. Dev. 34 (1990) 111).  (Two steps would do for a
// quotient unless b lies just below a power of two -- as densities near 1 do.)
//
// quot_rn: a y corrected twice by its exact remainder a - b q.  After the first
// correction q is within 1/2 + 2^-52 ulp of a/b, so before its rounding the second
// is off by at most (1/2 + 2^-52) |b y - 1| ulp, |b y - 1| <= 2^-54 m with m the
// significand of b in [1, 2); a/b lies at least 2^-53 / m ulp from a midpoint of two
// doubles (its numerator there is a nonzero integer over 2 b), so the rounding is
// right for every significand but all ones.  No step may leave the normal range.
// The callers check both (range_ok, zero_or_range_ok, ones) and divide otherwise;
// quot_signed also keeps the sign of a zero numerator.
// ---------------------------------------------------------------------------
#ifdef __CUDACC__
__device__ __forceinline__ double rcp_rn(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    return __fma_rn(y, __fma_rn(-b, y, 1.0), y);
}
__device__ __forceinline__ double quot_rn(double a, double b, double y)
{
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}
__device__ __forceinline__ double quot_signed(double a, double b, double y)
{
    const double q = quot_rn(a, b, y);
    const int sign = (__double2hiint(a) ^ __double2hiint(b)) & 0x80000000;
    return __hiloint2double(__double2hiint(q) | sign, __double2loint(q));
}
// positive and in [2^-60, 2^60)
__device__ __forceinline__ bool range_ok(double x) { return (unsigned)(__double2hiint(x) - 0x3c300000) < 0x07800000u; }
// zero, or of magnitude in [2^-512, 2^120) (the high word twice drops the sign)
__device__ __forceinline__ bool zero_or_range_ok(double x)
{
    return 2u * (unsigned)__double2hiint(x) - 0x3fe00000u < 0x4f000000u || x == 0.0;
}
// a significand whose low word is all ones
__device__ __forceinline__ bool ones(double x) { return __double2loint(x) == -1; }
#endif

// Per-cell quantities shared by the three sweeps (src/reconstruction.c:63-88,
// :104, :142-145).
template <typename T> struct CellC {
    T u[5];
    T U, V, W, C;
    T aa, ll, ee, gg, hh, nn, S11;
    T bb, cc, dd;
    T u_hh, v_hh, w_hh, u_ee, v_ee, w_ee;
};

// What costs divisions and the square root: velocities, sound speed, 1/(2C)
// and 1/(2C)/C, from the conserved state c.u.
template <typename T> FSL_HD void cell_roots_div(CellC<T> &c)
{
    typedef Kc<T> k;
    T R = T(1.) / c.u[0];
    c.U = c.u[1] * R;
    c.V = c.u[2] * R;
    c.W = c.u[3] * R;
    T P = (c.u[4] - T(0.5) * (c.u[1] * c.u[1] + c.u[2] * c.u[2] + c.u[3] * c.u[3]) * R) * k::K_1;
    c.C = sqrt(k::K * P * R);
    c.ll = T(1.) / (c.C + c.C);
    c.ee = c.ll / c.C;
}

#ifdef __CUDACC__
struct Roots64 {
    double U, V, W, C, ll, ee;
};
__device__ __noinline__ inline Roots64 cell_roots_by_division(double u0, double u1, double u2, double u3, double u4)
{
    CellC<double> c;
    c.u[0] = u0; c.u[1] = u1; c.u[2] = u2; c.u[3] = u3; c.u[4] = u4;
    cell_roots_div(c);
    return Roots64{c.U, c.V, c.W, c.C, c.ll, c.ee};
}
// the same values from R = rcp_rn(c.u[0]); 1/(C+C) is half of the rounded 1/C
__device__ __forceinline__ void cell_roots64(CellC<double> &c, double R)
{
    typedef Kc<double> k;
    c.U = c.u[1] * R;
    c.V = c.u[2] * R;
    c.W = c.u[3] * R;
    const double P = (c.u[4] - 0.5 * (c.u[1] * c.u[1] + c.u[2] * c.u[2] + c.u[3] * c.u[3]) * R) * k::K_1;
    c.C = sqrt(k::K * P * R);
    const double y = rcp_rn(c.C);
    c.ll = 0.5 * y;
    c.ee = quot_rn(c.ll, c.C, y);
    if (!range_ok(c.u[0]) || !range_ok(P) || ones(c.u[0]) || ones(c.C)) {
        const Roots64 o = cell_roots_by_division(c.u[0], c.u[1], c.u[2], c.u[3], c.u[4]);
        c.U = o.U; c.V = o.V; c.W = o.W; c.C = o.C; c.ll = o.ll; c.ee = o.ee;
    }
}
#endif

template <typename T> FSL_HD void cell_roots(CellC<T> &c)
{
#ifdef __CUDA_ARCH__
    if constexpr (std::is_same<T, double>::value) {
        cell_roots64(c, rcp_rn(c.u[0]));
        return;
    }
#endif
    cell_roots_div(c);
}

// The products of those.
template <typename T> FSL_HD void cell_products(CellC<T> &c)
{
    typedef Kc<T> k;
    T ff = c.U * c.U + c.V * c.V + c.W * c.W;
    c.aa = k::K_1_2 * ff;
    c.bb = k::NK_1 * c.U;
    c.cc = k::NK_1 * c.V;
    c.dd = k::NK_1 * c.W;
    c.gg = -ff * c.ee;
    c.hh = -(c.ee + c.ee);
    c.S11 = c.aa - c.C * c.C;
    c.u_hh = c.U * c.hh;
    c.v_hh = c.V * c.hh;
    c.w_hh = c.W * c.hh;
    c.u_ee = c.U * c.ee;
    c.v_ee = c.V * c.ee;
    c.w_ee = c.W * c.ee;
    c.nn = T(-0.5) * c.gg;
}

template <typename T> FSL_HD void cell_consts(CellC<T> &c)
{
    cell_roots(c);
    cell_products(c);
}

// The sweep below with its characteristic rows and face coefficients
// regrouped, for the FP32 bulk (which does not follow the reference's
// rounding): with d the forward (or backward) differences,
//   A = aa d1 + bn d2 + K_1 d5 + bt1 d3 + bt2 d4,  B = C (d2 - vn d1),
//   M1 = A - C^2 d1,  M4 = A + B,  M5 = A - B
// (S41 = aa - C vn, S42 = bn + C, S51 = aa + C vn, S52 = bn - C, S11 = aa - C^2),
// and on the faces n_ee (k4 + k5) + ll (k4 - k5) for _S24 k4 + _S25 k5 and
// (nn + H_K_1)(k4 + k5) + mm (k4 - k5) for _S54 k4 + _S55 k5.  The same
// scheme in fewer operations.
template <typename T, int N, int T1, int T2>
FSL_HD void recon_sweep_grouped(const CellC<T> &c, T vn, T vt1, T vt2, T bn, T bt1, T bt2, T n_hh, T t1_hh,
                                T t2_hh, T n_ee, T t1_ee, T t2_ee, const T *fw, const T *bw, T *hi, T *lo)
{
    typedef Kc<T> k;
    const T *u = c.u;
    const T C = c.C, C2 = c.aa - c.S11;
    T M[5], W[5];
    {
        const T d1 = fw[0] - u[0], d2 = fw[1] - u[N], d3 = fw[2] - u[T1], d4 = fw[3] - u[T2], d5 = fw[4] - u[4];
        const T A = c.aa * d1 + bn * d2 + k::K_1 * d5 + bt1 * d3 + bt2 * d4;
        const T B = C * (d2 - vn * d1);
        M[0] = A - C2 * d1; M[1] = d3 - vt1 * d1; M[2] = d4 - vt2 * d1; M[3] = A + B; M[4] = A - B;
    }
    {
        const T d1 = u[0] - bw[0], d2 = u[N] - bw[1], d3 = u[T1] - bw[2], d4 = u[T2] - bw[3], d5 = u[4] - bw[4];
        const T A = c.aa * d1 + bn * d2 + k::K_1 * d5 + bt1 * d3 + bt2 * d4;
        const T B = C * (d2 - vn * d1);
        W[0] = A - C2 * d1; W[1] = d3 - vt1 * d1; W[2] = d4 - vt2 * d1; W[3] = A + B; W[4] = A - B;
    }
    T Ml[5], Wl[5];
#pragma unroll
    for (int q = 0; q < 5; q++) minmod2(M[q], W[q], Ml[q], Wl[q]);
    const T mm = vn * c.ll, e45 = c.nn + k::H_K_1;
    {
        const T k1 = Ml[0] * k::C1 + Wl[0] * k::C2, k2 = Ml[1] * k::C1 + Wl[1] * k::C2;
        const T k3 = Ml[2] * k::C1 + Wl[2] * k::C2, k4 = Ml[3] * k::C1 + Wl[3] * k::C2;
        const T k5 = Ml[4] * k::C1 + Wl[4] * k::C2;
        const T ks = k4 + k5, kd = k4 - k5;
        hi[0] = u[0] + c.hh * k1 + c.ee * ks;
        hi[N] = u[N] + n_hh * k1 + n_ee * ks + c.ll * kd;
        hi[T1] = u[T1] + t1_hh * k1 + k2 + t1_ee * ks;
        hi[T2] = u[T2] + t2_hh * k1 + k3 + t2_ee * ks;
        hi[4] = u[4] + c.gg * k1 + vt1 * k2 + vt2 * k3 + e45 * ks + mm * kd;
    }
    {
        const T k1 = Ml[0] * k::C2 + Wl[0] * k::C1, k2 = Ml[1] * k::C2 + Wl[1] * k::C1;
        const T k3 = Ml[2] * k::C2 + Wl[2] * k::C1, k4 = Ml[3] * k::C2 + Wl[3] * k::C1;
        const T k5 = Ml[4] * k::C2 + Wl[4] * k::C1;
        const T ks = k4 + k5, kd = k4 - k5;
        lo[0] = u[0] - (c.hh * k1 + c.ee * ks);
        lo[N] = u[N] - (n_hh * k1 + n_ee * ks + c.ll * kd);
        lo[T1] = u[T1] - (t1_hh * k1 + k2 + t1_ee * ks);
        lo[T2] = u[T2] - (t2_hh * k1 + k3 + t2_ee * ks);
        lo[4] = u[4] - (c.gg * k1 + vt1 * k2 + vt2 * k3 + e45 * ks + mm * kd);
    }
}

// One sweep of the characteristic reconstruction.  N = index of the normal
// momentum in u[] (1..3); T1, T2 = tangential momenta in the reference's
// permuted order (x: 2 3 4 -> 1 2 3; y: 3 4 2 -> 2 3 1; z: 4 2 3 -> 3 1 2).
// fw/bw: forward/backward neighbour values in the order (rho, N, T1, T2, E).
// hi: state on the face towards the forward neighbour, lo: towards the
// backward neighbour, natural variable order.  t2_ee is the coefficient the
// reference applies to the T2 momentum (the z sweep uses w_ee for rho v,
// src/reconstruction.c:328,340).
template <typename T, int N, int T1, int T2>
FSL_HD void recon_sweep(const CellC<T> &c, T vn, T vt1, T vt2, T bn, T bt1, T bt2,
                                            T n_hh, T t1_hh, T t2_hh, T n_ee, T t1_ee, T t2_ee,
                                            const T *fw, const T *bw, T *hi, T *lo)
{
    if constexpr (std::is_same<T, float>::value) {
        recon_sweep_grouped<T, N, T1, T2>(c, vn, vt1, vt2, bn, bt1, bt2, n_hh, t1_hh, t2_hh, n_ee, t1_ee, t2_ee,
                                          fw, bw, hi, lo);
        return;
    }
    typedef Kc<T> k;
    const T *u = c.u;
    const T C = c.C;
    T m1, m2, m3, m4, m5, w1, w2, w3, w4, w5;
    T M1, M2, M3, M4, M5, W1, W2, W3, W4, W5;
    T _M1, _M2, _M3, _M4, _M5, _W1, _W2, _W3, _W4, _W5;
    T S12, S41, S42, S51, S52, _S24, _S25, _S54, _S55;
    T k1, k2, k3, k4, k5, kk, mm;
    mm = vn * c.ll;
    m1 = fw[0] - u[0]; m2 = fw[1] - u[N]; m3 = fw[2] - u[T1]; m4 = fw[3] - u[T2]; m5 = fw[4] - u[4];
    w1 = u[0] - bw[0]; w2 = u[N] - bw[1]; w3 = u[T1] - bw[2]; w4 = u[T2] - bw[3]; w5 = u[4] - bw[4];
    S41 = c.aa - (kk = C * vn);
    S51 = c.aa + kk;
    S12 = S42 = S52 = bn;
    S42 += C;
    S52 -= C;
    kk = k::K_1 * m5; k2 = bt1 * m3; k3 = bt2 * m4;
    M1 = c.S11 * m1 + S12 * m2 + k2 + k3 + kk;
    M2 = -vt1 * m1 + m3;
    M3 = -vt2 * m1 + m4;
    M4 = S41 * m1 + S42 * m2 + k2 + k3 + kk;
    M5 = S51 * m1 + S52 * m2 + k2 + k3 + kk;
    kk = k::K_1 * w5; k2 = bt1 * w3; k3 = bt2 * w4;
    W1 = c.S11 * w1 + S12 * w2 + k2 + k3 + kk;
    W2 = -vt1 * w1 + w3;
    W3 = -vt2 * w1 + w4;
    W4 = S41 * w1 + S42 * w2 + k2 + k3 + kk;
    W5 = S51 * w1 + S52 * w2 + k2 + k3 + kk;
    minmod_pair(M1, W1, _M1, _W1); minmod_pair(M2, W2, _M2, _W2); minmod_pair(M3, W3, _M3, _W3);
    minmod_pair(M4, W4, _M4, _W4); minmod_pair(M5, W5, _M5, _W5);
    _S24 = n_ee + c.ll; _S25 = n_ee - c.ll;
    _S54 = _S55 = c.nn + k::H_K_1;
    _S54 += mm; _S55 -= mm;
    k1 = _M1 * k::C1 + _W1 * k::C2; k2 = _M2 * k::C1 + _W2 * k::C2; k3 = _M3 * k::C1 + _W3 * k::C2;
    k4 = _M4 * k::C1 + _W4 * k::C2; k5 = _M5 * k::C1 + _W5 * k::C2;
    kk = k4 + k5;
    hi[0] = u[0] + c.hh * k1 + c.ee * kk;
    hi[N] = u[N] + n_hh * k1 + _S24 * k4 + _S25 * k5;
    hi[T1] = u[T1] + t1_hh * k1 + k2 + t1_ee * kk;
    hi[T2] = u[T2] + t2_hh * k1 + k3 + t2_ee * kk;
    hi[4] = u[4] + c.gg * k1 + vt1 * k2 + vt2 * k3 + _S54 * k4 + _S55 * k5;
    k1 = _M1 * k::C2 + _W1 * k::C1; k2 = _M2 * k::C2 + _W2 * k::C1; k3 = _M3 * k::C2 + _W3 * k::C1;
    k4 = _M4 * k::C2 + _W4 * k::C1; k5 = _M5 * k::C2 + _W5 * k::C1;
    kk = k4 + k5;
    lo[0] = u[0] - c.hh * k1 - c.ee * kk;
    lo[N] = u[N] - n_hh * k1 - _S24 * k4 - _S25 * k5;
    lo[T1] = u[T1] - t1_hh * k1 - k2 - t1_ee * kk;
    lo[T2] = u[T2] - t2_hh * k1 - k3 - t2_ee * kk;
    lo[4] = u[4] - c.gg * k1 - vt1 * k2 - vt2 * k3 - _S54 * k4 - _S55 * k5;
}

// x, y and z sweeps with the reference's permutations.
template <typename T> FSL_HD void recon_x(const CellC<T> &c, const T *fw, const T *bw, T *hi, T *lo)
{
    recon_sweep<T, 1, 2, 3>(c, c.U, c.V, c.W, c.bb, c.cc, c.dd, c.u_hh, c.v_hh, c.w_hh, c.u_ee, c.v_ee,
                            c.w_ee, fw, bw, hi, lo);
}
template <typename T> FSL_HD void recon_y(const CellC<T> &c, const T *fw, const T *bw, T *hi, T *lo)
{
    recon_sweep<T, 2, 3, 1>(c, c.V, c.W, c.U, c.cc, c.dd, c.bb, c.v_hh, c.w_hh, c.u_hh, c.v_ee, c.w_ee,
                            c.u_ee, fw, bw, hi, lo);
}
template <typename T> FSL_HD void recon_z(const CellC<T> &c, const T *fw, const T *bw, T *hi, T *lo)
{
    recon_sweep<T, 3, 1, 2>(c, c.W, c.U, c.V, c.dd, c.bb, c.cc, c.w_hh, c.u_hh, c.v_hh, c.w_ee, c.u_ee,
                            c.w_ee, fw, bw, hi, lo);
}

// PPM (project extension; the reference has only the scheme above): Colella
// & Woodward (1984) on the same characteristic variables, with cell i's
// transform (src/reconstruction.c:104-129) and inverse (:148-158).  Per
// characteristic field: monotonised-central slopes (CW84 eq. 1.8) of cells
// i-1, i, i+1, edge values a_{i+1/2} - a_i = 1/2 d_{i+1/2} - (da_{i+1} -
// da_i)/6 and a_{i-1/2} - a_i = -1/2 d_{i-1/2} - (da_i - da_{i-1})/6 (eq.
// 1.6), the monotonicity limiter (eq. 1.10); the same arithmetic as the
// oracle's restatement.
template <typename T> FSL_HD T ppm_mc(T a, T b)
{
    if constexpr (std::is_same<T, float>::value) {
        // FP32 bulk: the same value as a min and a sign copy
        const T m = fmin(fmin(T(0.5) * fabs(a + b), T(2.0) * fabs(a)), T(2.0) * fabs(b));
        return (a * b <= T(0.0)) ? T(0.0) : copysign(m, a);
    }
    T m = T(0.5) * fabs(a + b);
    const T ta = T(2.0) * fabs(a), tb = T(2.0) * fabs(b);
    m = (ta < m) ? ta : m;
    m = (tb < m) ? tb : m;
    return (a * b <= T(0.0)) ? T(0.0) : ((a > T(0.0)) ? m : -m);
}

template <typename T>
FSL_HD void char_fwd(const CellC<T> &c, T vn, T vt1, T vt2, T bn, T bt1, T bt2, const T *d, T *M)
{
    typedef Kc<T> k;
    if constexpr (std::is_same<T, float>::value) {
        // FP32 bulk: the rows regrouped as in recon_sweep_grouped
        const T A = c.aa * d[0] + bn * d[1] + k::K_1 * d[4] + bt1 * d[2] + bt2 * d[3];
        const T B = c.C * (d[1] - vn * d[0]);
        M[0] = A - (c.aa - c.S11) * d[0];
        M[1] = d[2] - vt1 * d[0];
        M[2] = d[3] - vt2 * d[0];
        M[3] = A + B;
        M[4] = A - B;
        return;
    }
    const T C = c.C;
    T S12, S41, S42, S51, S52, kk, k2, k3;
    S41 = c.aa - (kk = C * vn);
    S51 = c.aa + kk;
    S12 = S42 = S52 = bn;
    S42 += C;
    S52 -= C;
    kk = k::K_1 * d[4]; k2 = bt1 * d[2]; k3 = bt2 * d[3];
    M[0] = c.S11 * d[0] + S12 * d[1] + k2 + k3 + kk;
    M[1] = -vt1 * d[0] + d[2];
    M[2] = -vt2 * d[0] + d[3];
    M[3] = S41 * d[0] + S42 * d[1] + k2 + k3 + kk;
    M[4] = S51 * d[0] + S52 * d[1] + k2 + k3 + kk;
}

template <typename T, int N, int T1, int T2>
FSL_HD void char_inv(const CellC<T> &c, T vn, T vt1, T vt2, T n_hh, T t1_hh, T t2_hh, T n_ee,
                                         T t1_ee, T t2_ee, const T *q, T *out)
{
    typedef Kc<T> k;
    const T *u = c.u;
    if constexpr (std::is_same<T, float>::value) {
        // FP32 bulk: the face coefficients as sums and differences
        const T ks = q[3] + q[4], kd = q[3] - q[4];
        out[0] = u[0] + c.hh * q[0] + c.ee * ks;
        out[N] = u[N] + n_hh * q[0] + n_ee * ks + c.ll * kd;
        out[T1] = u[T1] + t1_hh * q[0] + q[1] + t1_ee * ks;
        out[T2] = u[T2] + t2_hh * q[0] + q[2] + t2_ee * ks;
        out[4] = u[4] + c.gg * q[0] + vt1 * q[1] + vt2 * q[2] + (c.nn + k::H_K_1) * ks + (vn * c.ll) * kd;
        return;
    }
    const T mm = vn * c.ll;
    T _S24, _S25, _S54, _S55, kk;
    _S24 = n_ee + c.ll; _S25 = n_ee - c.ll;
    _S54 = _S55 = c.nn + k::H_K_1;
    _S54 += mm; _S55 -= mm;
    kk = q[3] + q[4];
    out[0] = u[0] + c.hh * q[0] + c.ee * kk;
    out[N] = u[N] + n_hh * q[0] + _S24 * q[3] + _S25 * q[4];
    out[T1] = u[T1] + t1_hh * q[0] + q[1] + t1_ee * kk;
    out[T2] = u[T2] + t2_hh * q[0] + q[2] + t2_ee * kk;
    out[4] = u[4] + c.gg * q[0] + vt1 * q[1] + vt2 * q[2] + _S54 * q[3] + _S55 * q[4];
}

// x / 6, correctly rounded.  PPM divides by 6 thirty times a cell, a third of its
// divisions.  On the device in FP64: the product with the rounded reciprocal is
// within an ulp of the quotient, and one correction by its exact remainder
// gives the rounded quotient (Markstein 1990; for division by a constant,
// Brisebarre and Muller 2008) -- three instructions instead of a division's
// expansion and the branch that guards it: the FP64 PPM stages of a step 8.47 -> 5.59
// ms at 256x128x128.  Outside the range where the
// remainder is exact (and for infinities and NaN) the division itself.
#ifdef __CUDACC__
__device__ __noinline__ inline double sixth_by_division(double x) { return x / 6.0; }
#endif
template <typename T> FSL_HD T sixth(T x)
{
#ifdef __CUDA_ARCH__
    if constexpr (std::is_same<T, double>::value) {
        // not of magnitude in [2^-959, 2^993), nor zero
        if (2u * (unsigned)__double2hiint(x) - 0x08000000u >= 0xf4000000u && x != 0.0) return sixth_by_division(x);
        constexpr double y = 1.0 / 6.0;
        const double q = __dmul_rn(x, y);
        return __fma_rn(__fma_rn(6.0, q, -x), -y, q); // (in this order -0 gives -0)
    }
#endif
    return x / T(6.0);
}

// m2, m1, p1, p2: the neighbours at -2, -1, +1, +2 in the sweep's order
// (rho, normal, t1, t2, E); hi, lo as recon_sweep.
template <typename T, int N, int T1, int T2>
FSL_HD void ppm_sweep(const CellC<T> &c, T vn, T vt1, T vt2, T bn, T bt1, T bt2, T n_hh,
                                          T t1_hh, T t2_hh, T n_ee, T t1_ee, T t2_ee, const T *m2, const T *m1,
                                          const T *p1, const T *p2, T *hi, T *lo)
{
    const T *u = c.u;
    const T uc[5] = {u[0], u[N], u[T1], u[T2], u[4]};
    T d[5], W0[5], W1[5], W2[5], W3[5], qR[5], qL[5];
#pragma unroll
    for (int v = 0; v < 5; v++) d[v] = m1[v] - m2[v];
    char_fwd(c, vn, vt1, vt2, bn, bt1, bt2, d, W0);
#pragma unroll
    for (int v = 0; v < 5; v++) d[v] = uc[v] - m1[v];
    char_fwd(c, vn, vt1, vt2, bn, bt1, bt2, d, W1);
#pragma unroll
    for (int v = 0; v < 5; v++) d[v] = p1[v] - uc[v];
    char_fwd(c, vn, vt1, vt2, bn, bt1, bt2, d, W2);
#pragma unroll
    for (int v = 0; v < 5; v++) d[v] = p2[v] - p1[v];
    char_fwd(c, vn, vt1, vt2, bn, bt1, bt2, d, W3);
#pragma unroll
    for (int v = 0; v < 5; v++) {
        const T dm = ppm_mc(W0[v], W1[v]), d0 = ppm_mc(W1[v], W2[v]), dp = ppm_mc(W2[v], W3[v]);
        T r = T(0.5) * W2[v] - sixth(dp - d0), l = T(-0.5) * W1[v] - sixth(d0 - dm);
        if constexpr (std::is_same<T, float>::value) {
            // FP32 bulk: |r| > 2|l| and |l| > 2|r| exclude each other unless
            // both are zero, which the flat case covers
            const bool flat = r * l >= T(0.0);
            const T ar = fabs(r), al = fabs(l);
            qR[v] = flat ? T(0.0) : (ar > T(2.0) * al ? T(-2.0) * l : r);
            qL[v] = flat ? T(0.0) : (al > T(2.0) * ar ? T(-2.0) * r : l);
            continue;
        }
        const bool flat = r * l >= T(0.0);
        const bool capR = !flat && fabs(r) > T(2.0) * fabs(l);
        const bool capL = !flat && !capR && fabs(l) > T(2.0) * fabs(r);
        const T r2 = flat ? T(0.0) : (capR ? T(-2.0) * l : r);
        const T l2 = flat ? T(0.0) : (capL ? T(-2.0) * r : l);
        qR[v] = r2;
        qL[v] = l2;
    }
    char_inv<T, N, T1, T2>(c, vn, vt1, vt2, n_hh, t1_hh, t2_hh, n_ee, t1_ee, t2_ee, qR, hi);
    char_inv<T, N, T1, T2>(c, vn, vt1, vt2, n_hh, t1_hh, t2_hh, n_ee, t1_ee, t2_ee, qL, lo);
}

template <typename T>
FSL_HD void ppm_x(const CellC<T> &c, const T *m2, const T *m1, const T *p1, const T *p2, T *hi, T *lo)
{
    ppm_sweep<T, 1, 2, 3>(c, c.U, c.V, c.W, c.bb, c.cc, c.dd, c.u_hh, c.v_hh, c.w_hh, c.u_ee, c.v_ee, c.w_ee, m2, m1,
                          p1, p2, hi, lo);
}
template <typename T>
FSL_HD void ppm_y(const CellC<T> &c, const T *m2, const T *m1, const T *p1, const T *p2, T *hi, T *lo)
{
    ppm_sweep<T, 2, 3, 1>(c, c.V, c.W, c.U, c.cc, c.dd, c.bb, c.v_hh, c.w_hh, c.u_hh, c.v_ee, c.w_ee, c.u_ee, m2, m1,
                          p1, p2, hi, lo);
}
template <typename T>
FSL_HD void ppm_z(const CellC<T> &c, const T *m2, const T *m1, const T *p1, const T *p2, T *hi, T *lo)
{
    ppm_sweep<T, 3, 1, 2>(c, c.W, c.U, c.V, c.dd, c.bb, c.cc, c.w_hh, c.u_hh, c.v_hh, c.w_ee, c.u_ee, c.w_ee, m2, m1,
                          p1, p2, hi, lo);
}

// Linearised characteristic Riemann solve on one face (src/fluxes.c:61-113,
// :230-282, :401-453).  N = normal direction 1..3.  Lm/Rp: minus/plus
// conserved states.  Returns interface density, pressure and velocity (the
// normal component from the solve, the tangential ones upwinded by its sign).
template <typename T, int N>
FSL_HD void riemann_div(const T *Lm, const T *Rp, T &Rho, T &Pr, T *vel)
{
    typedef Kc<T> k;
    T _R, _P, _C, _jo, _jp, _jm, RU, R_, P_, C_, jo_, jp_, jm_;
    T lv[3], rv[3];
    T Un, C, C_p, C_m, C_o, al_p, al_m, al_o, J_p, J_m, J_o, P;
    _R = Lm[0];
    lv[0] = Lm[1] / _R; lv[1] = Lm[2] / _R; lv[2] = Lm[3] / _R;
    _P = (Lm[4] - T(0.5) * _R * (lv[0] * lv[0] + lv[1] * lv[1] + lv[2] * lv[2])) * k::K_1;
    _C = sqrt(k::K * _P / _R);
    _jo = k::NK_1 * _P;
    _jp = lv[N - 1] + (RU = _P / (_R * _C));
    _jm = lv[N - 1] - RU;
    R_ = Rp[0];
    rv[0] = Rp[1] / R_; rv[1] = Rp[2] / R_; rv[2] = Rp[3] / R_;
    P_ = (Rp[4] - T(0.5) * R_ * (rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2])) * k::K_1;
    C_ = sqrt(k::K * P_ / R_);
    jo_ = k::NK_1 * P_;
    jp_ = rv[N - 1] + (RU = P_ / (R_ * C_));
    jm_ = rv[N - 1] - RU;
    Un = T(0.5) * (lv[N - 1] + rv[N - 1]);
    C = T(0.5) * (_C + C_);
    C_p = Un + C; C_m = Un - C; C_o = Un;
    // upwind choices of src/fluxes.c:90-108 as operand selects (one division
    // each on the chosen operands: the same arithmetic as the branches)
    const bool pp = C_p > T(0.), pm = C_m > T(0.), po = C_o > T(0.);
    al_p = k::K_1_2 * (pp ? (_jm - _jp) : (jm_ - jp_)) / (pp ? _jo : jo_);
    J_p = pp ? _jp : jp_;
    al_m = k::K_1_2 * (pm ? (_jp - _jm) : (jp_ - jm_)) / (pm ? _jo : jo_);
    J_m = pm ? _jm : jm_;
    al_o = k::K05 * (po ? (_jp - _jm) : (jp_ - jm_));
    al_o = -al_o * al_o;
    J_o = po ? _jo : jo_;
    P = (J_p - J_m) / (al_p - al_m);
    Un = J_p - al_p * P;
    Rho = (J_o - P) / al_o;
    Pr = P;
    const bool up = Un > T(0);
    vel[0] = up ? lv[0] : rv[0];
    vel[1] = up ? lv[1] : rv[1];
    vel[2] = up ? lv[2] : rv[2];
    vel[N - 1] = Un;
}

#ifdef __CUDACC__
struct Riemann64 {
    double Rho, P, v0, v1, v2;
};
template <int N>
__device__ __noinline__ Riemann64 riemann_by_division(double l0, double l1, double l2, double l3, double l4, double r0,
                                                      double r1, double r2, double r3, double r4)
{
    const double Lm[5] = {l0, l1, l2, l3, l4}, Rp[5] = {r0, r1, r2, r3, r4};
    double Rho, P, v[3];
    riemann_div<double, N>(Lm, Rp, Rho, P, v);
    return Riemann64{Rho, P, v[0], v[1], v[2]};
}
// One side of the solve with shared reciprocals; p, q, r: the squares of the
// velocities in the order their sum takes.  false: divide instead.
__device__ __forceinline__ bool riemann_side64(double R, double m0, double m1, double m2, double &v0, double &v1,
                                               double &v2, double &y)
{
    y = rcp_rn(R);
    v0 = quot_signed(m0, R, y);
    v1 = quot_signed(m1, R, y);
    v2 = quot_signed(m2, R, y);
    return range_ok(R) && !ones(R) && zero_or_range_ok(m0) && zero_or_range_ok(m1) && zero_or_range_ok(m2);
}
__device__ __forceinline__ bool riemann_side64(double R, double P, double y, double &C, double &RU)
{
    C = sqrt(quot_rn(Kc<double>::K * P, R, y));
    const double RC = R * C;
    RU = quot_rn(P, RC, rcp_rn(RC));
    return range_ok(P) && !ones(RC);
}
// The upwinded middle of the solve (src/fluxes.c:85-113) from both sides' n
// velocity, P, C and RU.  With the sides' ranges checked every quotient here is
// normal or of a zero numerator; false: divide instead.
__device__ __forceinline__ bool riemann_mid64(double ln, double lP, double lC, double lRU, double rn, double rP,
                                              double rC, double rRU, double &Rho, double &P, double &vn)
{
    typedef Kc<double> k;
    const double ljo = k::NK_1 * lP, ljp = ln + lRU, ljm = ln - lRU;
    const double rjo = k::NK_1 * rP, rjp = rn + rRU, rjm = rn - rRU;
    const double Un = 0.5 * (ln + rn), C = 0.5 * (lC + rC);
    const bool pp = Un + C > 0., pm = Un - C > 0., po = Un > 0.;
    const double bp = pp ? ljo : rjo, bm = pm ? ljo : rjo;
    const double al_p = quot_rn(k::K_1_2 * (pp ? (ljm - ljp) : (rjm - rjp)), bp, rcp_rn(bp));
    const double al_m = quot_rn(k::K_1_2 * (pm ? (ljp - ljm) : (rjp - rjm)), bm, rcp_rn(bm));
    const double Jp = pp ? ljp : rjp, Jm = pm ? ljm : rjm, Jo = po ? ljo : rjo;
    double al_o = k::K05 * (po ? (ljp - ljm) : (rjp - rjm));
    al_o = -al_o * al_o;
    const double da = al_p - al_m;
    P = quot_rn(Jp - Jm, da, rcp_rn(da));
    vn = Jp - al_p * P;
    Rho = quot_rn(Jo - P, al_o, rcp_rn(al_o));
    return !(ones(bp) || ones(bm) || ones(da) || ones(al_o));
}
#endif

template <typename T, int N>
FSL_HD void riemann(const T *Lm, const T *Rp, T &Rho, T &Pr, T *vel)
{
#ifdef __CUDA_ARCH__
    if constexpr (std::is_same<T, double>::value) {
        typedef Kc<double> k;
        double l[3], r[3], ly, ry, lC, lRU, rC, rRU;
        bool ok = riemann_side64(Lm[0], Lm[1], Lm[2], Lm[3], l[0], l[1], l[2], ly);
        ok = riemann_side64(Rp[0], Rp[1], Rp[2], Rp[3], r[0], r[1], r[2], ry) && ok;
        const double lP = (Lm[4] - 0.5 * Lm[0] * (l[0] * l[0] + l[1] * l[1] + l[2] * l[2])) * k::K_1;
        const double rP = (Rp[4] - 0.5 * Rp[0] * (r[0] * r[0] + r[1] * r[1] + r[2] * r[2])) * k::K_1;
        ok = riemann_side64(Lm[0], lP, ly, lC, lRU) && ok;
        ok = riemann_side64(Rp[0], rP, ry, rC, rRU) && ok;
        double vn;
        ok = riemann_mid64(l[N - 1], lP, lC, lRU, r[N - 1], rP, rC, rRU, Rho, Pr, vn) && ok;
        const bool up = vn > 0.;
        vel[0] = up ? l[0] : r[0];
        vel[1] = up ? l[1] : r[1];
        vel[2] = up ? l[2] : r[2];
        vel[N - 1] = vn;
        if (!ok) {
            const Riemann64 o = riemann_by_division<N>(Lm[0], Lm[1], Lm[2], Lm[3], Lm[4], Rp[0], Rp[1], Rp[2], Rp[3],
                                                       Rp[4]);
            Rho = o.Rho; Pr = o.P;
            vel[0] = o.v0; vel[1] = o.v1; vel[2] = o.v2;
        }
        return;
    }
#endif
    riemann_div<T, N>(Lm, Rp, Rho, Pr, vel);
}

// Velocities by reciprocal, RU = 1./rho (src/fluxes.c:124-142).
template <typename T> FSL_HD void vel_rcp(T r, T mu_, T mv, T mw, T *o)
{
    T RU = T(1.) / r;
    o[0] = mu_ * RU; o[1] = mv * RU; o[2] = mw * RU;
}

// Velocities and temperature by division (src/fluxes.c:117-122).
template <typename T> FSL_HD void vel_div_div(T R_, T mu_, T mv, T mw, T E, T *o, T &Tt)
{
    typedef Kc<T> k;
    T U_ = mu_ / R_, V_ = mv / R_, W_ = mw / R_;
    T P_ = (E - T(0.5) * R_ * (U_ * U_ + V_ * V_ + W_ * W_)) * k::K_1;
    Tt = P_ / (k::R_VOZD * R_);
    o[0] = U_; o[1] = V_; o[2] = W_;
}

#ifdef __CUDACC__
struct VelT64 {
    double u, v, w, T;
};
__device__ __noinline__ inline VelT64 vel_by_division(double R, double m0, double m1, double m2, double E)
{
    VelT64 o;
    double v[3];
    vel_div_div(R, m0, m1, m2, E, v, o.T);
    o.u = v[0]; o.v = v[1]; o.w = v[2];
    return o;
}
// the same values; y = rcp_rn(R)
__device__ __forceinline__ void vel_div64(double R, double m0, double m1, double m2, double E, double y, double *o,
                                          double &Tt)
{
    typedef Kc<double> k;
    o[0] = quot_signed(m0, R, y);
    o[1] = quot_signed(m1, R, y);
    o[2] = quot_signed(m2, R, y);
    const double P = (E - 0.5 * R * (o[0] * o[0] + o[1] * o[1] + o[2] * o[2])) * k::K_1;
    const double den = k::R_VOZD * R;
    Tt = quot_rn(P, den, rcp_rn(den));
    if (!(range_ok(R) && range_ok(P) && zero_or_range_ok(m0) && zero_or_range_ok(m1) && zero_or_range_ok(m2)) ||
        ones(R) || ones(den)) {
        const VelT64 q = vel_by_division(R, m0, m1, m2, E);
        o[0] = q.u; o[1] = q.v; o[2] = q.w;
        Tt = q.T;
    }
}
#endif

template <typename T> FSL_HD void vel_div(T R_, T mu_, T mv, T mw, T E, T *o, T &Tt)
{
#ifdef __CUDA_ARCH__
    if constexpr (std::is_same<T, double>::value) {
        vel_div64(R_, mu_, mv, mw, E, rcp_rn(R_), o, Tt);
        return;
    }
#endif
    vel_div_div(R_, mu_, mv, mw, E, o, Tt);
}

// Flux assembly of one face from the Riemann state, the face velocity
// gradient and the cell-centre velocities of the two adjacent cells
// (src/fluxes.c:185-220, :353-391, :524-568).  N = normal direction.
// g[a][b] = d u_a / d x_b.  fw/bw: velocities of the plus/minus cell.
template <typename T, int N>
FSL_HD void face_flux(T Rho, T P, const T *vel, const T (*g)[3], const T *fw, const T *bw,
                                          T Tp, T Tm, T mu_L, T mu_T, T lambda_L, T cp_Pr_T, T rdn, T *F)
{
    typedef Kc<T> k;
    T uu = T(0.5) * (fw[0] + bw[0]), vv = T(0.5) * (fw[1] + bw[1]), ww = T(0.5) * (fw[2] + bw[2]);
    T mu_E = mu_L + mu_T;
    T s0, s1, s2; // sigma_N{x,y,z}
    if (N == 1) {
        s0 = k::TWO_THIRDS * mu_E * (g[0][0] + g[0][0] - g[1][1] - g[2][2]);
        s1 = mu_E * (g[0][1] + g[1][0]);
        s2 = mu_E * (g[0][2] + g[2][0]);
    } else if (N == 2) {
        s0 = mu_E * (g[1][0] + g[0][1]);
        s1 = k::TWO_THIRDS * mu_E * (g[1][1] + g[1][1] - g[0][0] - g[2][2]);
        s2 = mu_E * (g[1][2] + g[2][1]);
    } else {
        s0 = mu_E * (g[2][0] + g[0][2]);
        s1 = mu_E * (g[2][1] + g[1][2]);
        s2 = k::TWO_THIRDS * mu_E * (g[2][2] + g[2][2] - g[0][0] - g[1][1]);
    }
    T lambda_E = lambda_L + mu_T * cp_Pr_T;
    T q = -lambda_E * (Tp - Tm) * rdn;
    T RU = Rho * vel[N - 1];
    F[0] = RU;
    F[1] = RU * vel[0] - s0;
    F[2] = RU * vel[1] - s1;
    F[3] = RU * vel[2] - s2;
    if (N == 1) F[1] = RU * vel[0] + P - s0;
    if (N == 2) F[2] = RU * vel[1] + P - s1;
    if (N == 3) F[3] = RU * vel[2] + P - s2;
    F[4] = vel[N - 1] * (k::K_K_1 * P + T(0.5) * Rho * (vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2])) -
           uu * s0 - vv * s1 - ww * s2 + q;
}

// The static Smagorinsky viscosity of one face (the reference's
// DynamicSmagorinskySGS 0 branch, src/fluxes.c:193-205 x, :362-374 y,
// :533-545 z; live in src-par/def.h:47): the mean density of the two cells
// beside the face times CsDD = Cs (dx dy dz)^(2/3) times |S| from the face
// velocity gradients g[a][b] = d u_a / d x_b, in the reference's order.
template <typename T> FSL_HD T static_mu_t(const T (*g)[3], T rr, T CsDD)
{
    const T S12 = T(0.5) * (g[0][1] + g[1][0]);
    const T S13 = T(0.5) * (g[0][2] + g[2][0]);
    const T S23 = T(0.5) * (g[1][2] + g[2][1]);
    const T S = sqrt(T(2) * (g[0][0] * g[0][0] + g[1][1] * g[1][1] + g[2][2] * g[2][2] +
                             T(2) * (S12 * S12 + S13 * S13 + S23 * S23)));
    return rr * CsDD * S;
}

// Flux of one face (src/fluxes.c): Riemann state from the two face states,
// viscous and heat flux from the two adjacent cells (vm/Tm minus side, vp/Tp
// plus side, by division) and the eight tangential neighbours (by
// reciprocal; P/M = plus/minus cell, h/l = +/- along the first (1) and
// second (2) tangential axis).  kc: grid spacings and transport constants
// (rdx.., r4dx.., mu_L, lambda_L, cp_Pr_T, CsDD).  muT is the face's SGS
// viscosity; with SST (static Smagorinsky) it is the mean density of the two
// cells beside the face, and the viscosity is formed here from the gradients.
template <typename T, int N, bool SST = false, typename KC>
FSL_HD void fused_face(const T *Lm, const T *Rp, const T *vm, T Tm, const T *vp, T Tp, const T *Ph1, const T *Mh1,
                       const T *Pl1, const T *Ml1, const T *Ph2, const T *Mh2, const T *Pl2, const T *Ml2, T muT,
                       const KC &kc, T *F)
{
    T Rho, P, vel[3];
    riemann<T, N>(Lm, Rp, Rho, P, vel);
    const int n0 = N - 1;
    const int t1 = (N == 1) ? 1 : 0;
    const int t2 = (N == 3) ? 1 : 2;
    const T rdn = T(N == 1 ? kc.rdx : N == 2 ? kc.rdy : kc.rdz);
    const T rt1 = T(N == 1 ? kc.r4dy : kc.r4dx);
    const T rt2 = T(N == 3 ? kc.r4dy : kc.r4dz);
    T gr[3][3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        gr[q][n0] = (vp[q] - vm[q]) * rdn;
        gr[q][t1] = (Ph1[q] + Mh1[q] - Pl1[q] - Ml1[q]) * rt1;
        gr[q][t2] = (Ph2[q] + Mh2[q] - Pl2[q] - Ml2[q]) * rt2;
    }
    if constexpr (SST) muT = static_mu_t<T>(gr, muT, T(kc.CsDD));
    face_flux<T, N>(Rho, P, vel, gr, vp, vm, Tp, Tm, T(kc.mu_L), muT, T(kc.lambda_L), T(kc.cp_Pr_T), rdn, F);
}

template <typename T> FSL_HD void vdiv(const T *U, T *o)
{
    T Tt;
    vel_div(U[0], U[1], U[2], U[3], U[4], o, Tt);
    o[3] = Tt;
}

#ifdef __CUDACC__
// A cell's characteristic roots and its velocities and temperature by division
// (dv), sharing 1/rho.
__device__ __forceinline__ void cell_prims64(CellC<double> &c, double *dv)
{
    const double y = rcp_rn(c.u[0]);
    cell_roots64(c, y);
    vel_div64(c.u[0], c.u[1], c.u[2], c.u[3], c.u[4], y, dv, dv[3]);
}
#endif

// Courant number of one cell from its conserved variables: the reference's
// streamwise u dt/dx (src/helpers.c:31-43) or the acoustic sum
// dt((|u|+c)/dx + (|v|+c)/dy + (|w|+c)/dz) (a project extension, formed with
// the reciprocal ir = 1/rho: one division instead of four).  Every operation
// is an explicitly rounded FP64 intrinsic, so the value does not depend on
// the contraction flags of the translation unit: the standalone reduction and
// the fused stage kernels (FP64 and FP32 bulk) produce the same bits.
__device__ __forceinline__ double cell_courant_ir(int mode, double R, double ir, double mu, double mv, double mw,
                                                  double E, double dtx, double dty, double dtz)
{
    if (mode != 1) return __dmul_rn(__ddiv_rn(mu, R), dtx);
    const double Uv = __dmul_rn(mu, ir), V = __dmul_rn(mv, ir), W = __dmul_rn(mw, ir);
    const double q = __dadd_rn(__dadd_rn(__dmul_rn(Uv, Uv), __dmul_rn(V, V)), __dmul_rn(W, W));
    const double P = __dmul_rn(__dsub_rn(E, __dmul_rn(__dmul_rn(0.5, R), q)), 0.4);
    const double Cs = __dsqrt_rn(__dmul_rn(__dmul_rn(1.4, P), ir));
    return __dadd_rn(__dadd_rn(__dmul_rn(__dadd_rn(fabs(Uv), Cs), dtx), __dmul_rn(__dadd_rn(fabs(V), Cs), dty)),
                     __dmul_rn(__dadd_rn(fabs(W), Cs), dtz));
}
__device__ __forceinline__ double cell_courant(int mode, double R, double mu, double mv, double mw, double E,
                                               double dtx, double dty, double dtz)
{
    return cell_courant_ir(mode, R, mode == 1 ? __ddiv_rn(1.0, R) : 0.0, mu, mv, mw, E, dtx, dty, dtz);
}

} // namespace fsl
