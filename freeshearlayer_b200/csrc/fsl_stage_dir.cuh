// fsl_stage_dir.cuh -- the plain method's (FP64) fused RK3 stage kernel with
// one group of warps per sweep direction, for the reference reconstruction
// (src/reconstruction.c:26-345) and fluxes (src/fluxes.c:57-571).
//
// The ring tile (fsl_stage.cuh) takes a cell through its three directions in one
// thread: 128 registers, 11 us a plane of 14 x 30 cells however few SMs a small
// grid fills.  Here three threads share a cell, one per direction, on tiles of 4
// (y) x 32 (z) cells whose lanes all own a cell, so a plane takes 5 us and a small
// grid spreads over three times as many blocks (64x32x32: 48 -> 34 us a stage, and
// no boundary passes on the temporal setup).  What bounds it is the latency of
// one warp's chain of dependent FP64 arithmetic, sweep then face; per cell it
// issues a third more instructions than the ring (its operands come from shared
// memory through computed offsets), so large grids keep the ring (fsl_fused.cu).
//
// Group d of warps sweeps and solves the faces of direction d = x, y, z; three
// halo warps do the tile's neighbouring rows and columns and its first y and z
// faces, so that no warp has two tasks in a row.  All run the same code: operands
// are addressed through direction-dependent offsets in the frame (rho, normal,
// first and second tangential, E), and where the reference sums the three
// velocity components the terms are put back in natural order, so every value
// rounds as in the reference.  One copy of the sweep and one of the face also
// keep the code in the instruction cache (a full-lane tile with a copy per
// direction and halo task overran it: 13.8 ms a launch at 512x256x256).
//
// A block marches along x.  Per plane i: group x sweeps cell i+1, groups y and
// z the cells of plane i; then every group solves its faces (x: i+1/2; y, z:
// beyond each cell); after a barrier group x combines the stage while the others
// form the velocities and characteristic roots of plane i+2.  Plane i+3 arrives
// in shared memory by asynchronous copies meanwhile.  A segment starts two
// planes early with group x alone, which gives the first face's flux without a
// second copy of the code.
#pragma once

#include "fsl_stage.cuh"

namespace fsl {
namespace dirs {

using stage::BF;

constexpr int WJ = 4;            // tile rows (warps of a group)
constexpr int WK = 32;           // tile columns (lanes)
constexpr int NT = (3 * WJ + 3) * WK; // threads of a block: three groups and three halo warps

struct Smem {
    double U[4][WJ + 4][WK + 4][5];  // state of planes i .. i+3 (ring): rows -2..5, cols -2..33
    double R[3][WJ + 2][WK + 2][3];  // velocities by reciprocal, planes i-1, i, i+1 (ring): rows -1..4, cols -1..32
    double Dv[2][WJ + 2][WK + 2][5]; // velocities by division, T, face-averaged mu: planes i, i+1
    double K[2][WJ + 2][WK + 2][4];  // C, 1/(2C), 1/(2C)/C, |u|^2: planes i, i+1
    double SL[3][WJ + 1][WK + 1][5]; // per direction, state on the face before each cell (row 4, column 32: halo)
    double SF[2][WJ + 1][WK + 1][5]; // y, z fluxes of the face before each cell
    double co[WJ];                   // Courant maxima, per warp of group x
};

struct DirArgs {
    Grid g;
    Consts kc;
    const double *cur, *un;
    double *out;
    const double *mu;
    BF<double> bf;
    const DevScalars *ds;
    unsigned long long *co; // non-null: accumulate the Courant maximum of `out` (stage 3)
    unsigned int *status;
    int co_i0, co_i1;
    int stage;
    int seg; // planes of a block
};

// a natural-order sum x0 + x1 + x2 from the frame's values (n, a, b); natural
// order is n a b in x, a n b in y, a b n in z
__device__ __forceinline__ double nat3(int d, double n, double a, double b)
{
    const double p = d == 2 ? b : n, q = d == 2 ? n : b;
    return a + p + q;
}

// stage::riemann in the frame (src/fluxes.c:61-113)
struct FaceState {
    double Rho, P, vn, va, vb;
};
__device__ __noinline__ FaceState face_by_division(int d, double l0, double l1, double l2, double l3, double l4,
                                                   double r0, double r1, double r2, double r3, double r4)
{
    // the frame's components in natural order: n a b, a n b, a b n
    const double L[5] = {l0, d == 0 ? l1 : l2, d == 0 ? l2 : d == 1 ? l1 : l3, d == 2 ? l1 : l3, l4};
    const double R[5] = {r0, d == 0 ? r1 : r2, d == 0 ? r2 : d == 1 ? r1 : r3, d == 2 ? r1 : r3, r4};
    FaceState o;
    double v[3];
    if (d == 0) {
        riemann_div<double, 1>(L, R, o.Rho, o.P, v);
        o.vn = v[0]; o.va = v[1]; o.vb = v[2];
    } else if (d == 1) {
        riemann_div<double, 2>(L, R, o.Rho, o.P, v);
        o.vn = v[1]; o.va = v[0]; o.vb = v[2];
    } else {
        riemann_div<double, 3>(L, R, o.Rho, o.P, v);
        o.vn = v[2]; o.va = v[0]; o.vb = v[1];
    }
    return o;
}

__device__ __forceinline__ void face_riemann(int d, const double *Lm, const double *Rp, double &Rho, double &P,
                                             double &vn, double &va, double &vb)
{
    typedef Kc<double> k;
    double ln, la, lb, ly, lC, lRU, rn, ra, rb, ry, rC, rRU;
    bool ok = riemann_side64(Lm[0], Lm[1], Lm[2], Lm[3], ln, la, lb, ly);
    ok = riemann_side64(Rp[0], Rp[1], Rp[2], Rp[3], rn, ra, rb, ry) && ok;
    const double lP = (Lm[4] - 0.5 * Lm[0] * nat3(d, ln * ln, la * la, lb * lb)) * k::K_1;
    const double rP = (Rp[4] - 0.5 * Rp[0] * nat3(d, rn * rn, ra * ra, rb * rb)) * k::K_1;
    ok = riemann_side64(Lm[0], lP, ly, lC, lRU) && ok;
    ok = riemann_side64(Rp[0], rP, ry, rC, rRU) && ok;
    ok = riemann_mid64(ln, lP, lC, lRU, rn, rP, rC, rRU, Rho, P, vn) && ok;
    const bool up = vn > 0.;
    va = up ? la : ra;
    vb = up ? lb : rb;
    if (!ok) {
        const FaceState o = face_by_division(d, Lm[0], Lm[1], Lm[2], Lm[3], Lm[4], Rp[0], Rp[1], Rp[2], Rp[3], Rp[4]);
        Rho = o.Rho; P = o.P;
        vn = o.vn; va = o.va; vb = o.vb;
    }
}

template <bool SST>
__global__ void __launch_bounds__(NT, 1) k_stage_dir(DirArgs A)
{
    follow();
    extern __shared__ __align__(16) unsigned char smraw[];
    Smem &s = *reinterpret_cast<Smem *>(smraw);
    typedef Kc<double> kk;
    const Grid &g = A.g;
    const Consts &kc = A.kc;
    const int L = g.L, H = g.H, D = g.D;
    const int t = threadIdx.x, l = t & 31;
    // warp-uniform: direction and tile row
    const int wid = __shfl_sync(0xffffffffu, t >> 5, 0);
    // halo warps: 0 row -1 and the tile's first y faces, 1 row WJ (direction y);
    // 2 columns -1 and 32 and the first z faces (direction z)
    const int hw = wid - 3 * WJ;
    const int d = hw < 0 ? wid / WJ : hw < 2 ? 1 : 2;
    const int r = hw < 0 ? wid % WJ : hw == 0 ? -1 : hw == 1 ? WJ : (l & (WJ - 1));
    const int cl = hw < 2 ? l : l < WJ ? -1 : WK; // tile column of this thread's sweep
    const int y_threads = (WJ + 2) * WK, z_threads = (WJ + 1) * WK;
    const long long fs = g.fstride;
    const double *__restrict__ cu = A.cur;
    const bool tpl = kc.setup == FSL_SETUP_TEMPORAL;
    const double dtx = A.ds->dtx, dty = A.ds->dty, dtz = A.ds->dtz;
    if (t < WJ) s.co[t] = 0.0;

    // the frame: components (0 u, 1 v, 2 w) of the normal and the tangentials in
    // the sweep's order (x: u v w, y: v w u, z: w u v) and in the face's (a < b)
    const int cn = d, ct1 = d == 2 ? 0 : d + 1, ct2 = d == 0 ? 2 : d - 1;
    const int ca = d == 0 ? 1 : 0, cb = d == 2 ? 1 : 2;
    const double rdn = d == 0 ? kc.rdx : d == 1 ? kc.rdy : kc.rdz;
    const double r4a = d == 0 ? kc.r4dy : kc.r4dx, r4b = d == 2 ? kc.r4dy : kc.r4dz;
    // element strides of the shared arrays
    constexpr int UR = (WK + 4) * 5, UP = (WJ + 4) * UR;
    constexpr int RR = (WK + 2) * 3, RP = (WJ + 2) * RR;
    constexpr int VR = (WK + 2) * 5, VP = (WJ + 2) * VR;
    constexpr int KR = (WK + 2) * 4, KP = (WJ + 2) * KR;
    constexpr int SR = (WK + 1) * 5;
    double *const U0 = &s.U[0][2][2][0], *const R0 = &s.R[0][1][1][0], *const V0 = &s.Dv[0][1][1][0],
                 *const K0 = &s.K[0][1][1][0];
    double *const SLd = &s.SL[d][0][0][0], *const SFd = &s.SF[d == 2][0][0][0];

    const int ntk = (D + WK - 1) / WK, ntj = (H + WJ - 1) / WJ;
    // block b: segment b / ntiles of tile b % ntiles
    {
        const int tile = (int)(blockIdx.x % (unsigned)(ntk * ntj));
        const int i0 = 1 + (int)(blockIdx.x / (unsigned)(ntk * ntj)) * A.seg, i1 = min(L, i0 + A.seg - 1);
        const int k0 = (int)(tile % ntk) * WK + 1, j0 = (int)(tile / ntk) * WJ + 1;
        const int j = j0 + r, k = k0 + cl;
        const bool own = hw < 0 && j <= H && k <= D;
        
        // one plane of the tile and its halo into the state ring, one cell per
        // thread.  Temporal setup: the planes -1 and L+2 and the columns -1 and
        // D+2 hold the periodic images (planes L-1 and 2, columns D-1 and 2);
        // elsewhere they are not read
        const int lr = t / (WK + 4) - 2, lc = t % (WK + 4) - 2;
        const int lj = j0 + lr, lk = k0 + lc, lz = lk < 0 ? D - 1 : lk == D + 2 ? 2 : lk;
        const bool loads = t < (WJ + 4) * (WK + 4) && lj >= 0 && lj <= H + 1 && lz <= D + 1 && (lz == lk || tpl);
        const long long lcell = loads ? g.idx(0, lj, lz) : 0;
        const uint32_t ldst = (uint32_t)__cvta_generic_to_shared(U0 + (loads ? lr * UR + lc * 5 : 0));
        auto load_plane = [&](int p) {
            const int gp = p < 0 ? L - 1 : p > L + 1 ? 2 : p;
            if (loads && (gp == p || tpl)) {
                const long long c = FSL_CELL(lcell + gp * g.pi, fs);
                const uint32_t dst = ldst + (uint32_t)((p & 3) * UP) * 8u;
#pragma unroll
                for (int q = 0; q < 5; q++)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + q * 8u), "l"(cu + q * fs + c)
                                 : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        // this thread's cell of the velocity ring: group z (own cells) and the
        // halo warps (rows -1, WJ; columns -1, 32 and the corners)
        int pr = r, pc = cl;
        bool prim = d == 2 || hw >= 0;
        if (hw == 2) {
            if (l < 2 * WJ) {
                pc = l < WJ ? -1 : WK;
            } else {
                const int h = l - 2 * WJ;
                pr = (h & 1) ? WJ : -1;
                pc = h >= 2 ? WK : -1;
                prim = l < 2 * WJ + 4;
            }
        }
        const int pj = j0 + pr, pk = k0 + pc;
        prim = prim && pj >= 0 && pj <= H + 1 && pk <= D + 1;
        const double *mup = SST ? nullptr : A.mu + g.idx(0, prim ? pj : 0, prim ? pk : 0);
        double mu_prev = 0., mu_next = 0.;
        auto prims = [&](int p) {
            CellC<double> c;
            const double *u = U0 + (p & 3) * UP + pr * UR + pc * 5;
#pragma unroll
            for (int q = 0; q < 5; q++) c.u[q] = u[q];
            double dv[4];
            cell_prims64(c, dv);
            double *v = R0 + ((p + 3) % 3) * RP + pr * RR + pc * 3, *o = V0 + (p & 1) * VP + pr * VR + pc * 5,
                   *w = K0 + (p & 1) * KP + pr * KR + pc * 4;
            v[0] = c.U; v[1] = c.V; v[2] = c.W;
            w[0] = c.C; w[1] = c.ll; w[2] = c.ee;
            w[3] = c.U * c.U + c.V * c.V + c.W * c.W;
            o[0] = dv[0]; o[1] = dv[1]; o[2] = dv[2]; o[3] = dv[3];
            if constexpr (!SST) o[4] = 0.5 * (mu_next + mu_prev);
        };

        double hi[5], carry[5], Fxp[5];
#pragma unroll
        for (int q = 0; q < 5; q++) hi[q] = carry[q] = Fxp[q] = 0.;

        load_plane(i0 - 2);
        load_plane(i0 - 1);
        load_plane(i0);
        if constexpr (!SST) {
            if (prim) mu_next = mup[(long long)(i0 - 1) * g.pi];
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (prim) prims(i0 - 1);
        __syncthreads();

        for (int i = i0 - 2; i <= i1; i++) {
            const bool full = i >= i0;
            if (i + 3 <= i1 + 2) load_plane(i + 3);
            const bool next = prim && i + 2 <= i1 + 1; // prims(i+2) after the faces
            if constexpr (!SST) {
                mu_prev = mu_next;
                if (next) mu_next = mup[(long long)(i + 2) * g.pi];
            }
            const int rs = (i + 3) % 3, rn = (i + 4) % 3, rb = (i + 2) % 3; // R slots of planes i, i+1, i-1
            // ---- sweeps
            if (d == 0 || full) {
                // offsets of the forward and backward neighbours; x sweeps plane i+1
                const int ps = d == 0 ? i + 1 : i;
                const int uf = d == 0 ? (((ps + 1) & 3) - (ps & 3)) * UP : d == 1 ? UR : 5;
                const int ub = d == 0 ? (((ps - 1) & 3) - (ps & 3)) * UP : d == 1 ? -UR : -5;
                // the cells swept, or the outer state of a boundary face from the
                // boundary pass (bsrc); where the states go: the face before the
                // cell, or for row -1 and column -1 the face beyond it
                bool act, low = false;
                const double *bsrc = nullptr;
                long long bst = 0;
                if (d == 0) {
                    act = own;
                    if (!tpl && own && (ps < 1 || ps > L)) {
                        act = false;
                        bst = (long long)H * D;
                        bsrc = (ps < 1 ? A.bf.x0 : A.bf.xL) + FSL_FACE((long long)(j - 1) * D + (k - 1), bst);
                    }
                } else if (d == 1) {
                    low = r < 0;
                    const bool in = k <= D;
                    act = in && j <= H && j >= 1;
                    if (!act && in && !tpl && (j == 0 || j == H + 1)) {
                        bst = (long long)L * D;
                        bsrc = (low ? A.bf.y0 : A.bf.yH) + FSL_FACE((long long)(i - 1) * D + (k - 1), bst);
                    }
                } else {
                    low = hw >= 0 && l < WJ;
                    const bool in = j <= H && (hw < 0 || l < 2 * WJ);
                    act = in && (k >= 1 || tpl) && (k <= D || (tpl && k == D + 1));
                    if (!act && in && !tpl && (k == 0 || k == D + 1)) {
                        bst = (long long)L * H;
                        bsrc = (low ? A.bf.z0 : A.bf.zD) + FSL_FACE((long long)(i - 1) * H + (j - 1), bst);
                    }
                }
                {
                    const int sr = r, sc = cl;
                    double lo[5];
                    if (act) {
                        const double *u = U0 + (ps & 3) * UP + sr * UR + sc * 5;
                        const double *vr = R0 + ((ps + 3) % 3) * RP + sr * RR + sc * 3;
                        const double *w = K0 + (ps & 1) * KP + sr * KR + sc * 4;
                        const double *f = u + uf, *bk = u + ub;
                        CellC<double> c;
                        c.u[0] = u[0]; c.u[1] = u[1 + cn]; c.u[2] = u[1 + ct1]; c.u[3] = u[1 + ct2]; c.u[4] = u[4];
                        const double fw[5] = {f[0], f[1 + cn], f[1 + ct1], f[1 + ct2], f[4]};
                        const double bw[5] = {bk[0], bk[1 + cn], bk[1 + ct1], bk[1 + ct2], bk[4]};
                        const double vn = vr[cn], v1 = vr[ct1], v2 = vr[ct2], ff = w[3];
                        c.C = w[0]; c.ll = w[1]; c.ee = w[2];
                        c.aa = kk::K_1_2 * ff;
                        c.gg = -ff * c.ee;
                        c.hh = -(c.ee + c.ee);
                        c.S11 = c.aa - c.C * c.C;
                        c.nn = -0.5 * c.gg;
                        const double n_ee = vn * c.ee;
                        recon_sweep<double, 1, 2, 3>(c, vn, v1, v2, kk::NK_1 * vn, kk::NK_1 * v1, kk::NK_1 * v2,
                                                     vn * c.hh, v1 * c.hh, v2 * c.hh, n_ee, v1 * c.ee,
                                                     d == 2 ? n_ee : v2 * c.ee, fw, bw, hi, lo);
                        if (d == 1) { // the sweep's tangentials are w, u; the face's u, w
                            double x = hi[2];
                            hi[2] = hi[3]; hi[3] = x;
                            x = lo[2];
                            lo[2] = lo[3]; lo[3] = x;
                        }
                    } else if (bsrc) {
                        hi[0] = bsrc[0]; hi[1] = bsrc[(1 + cn) * bst]; hi[2] = bsrc[(1 + ca) * bst];
                        hi[3] = bsrc[(1 + cb) * bst]; hi[4] = bsrc[4 * bst];
#pragma unroll
                        for (int q = 0; q < 5; q++) lo[q] = hi[q];
                    }
                    if ((act || bsrc) && !low) {
                        double *dst = SLd + sr * SR + sc * 5;
#pragma unroll
                        for (int q = 0; q < 5; q++) dst[q] = lo[q];
                    }
                }
            }
            // the y rows' and z columns' states meet within their groups
            if (full) {
                if (d == 1) asm volatile("bar.sync 1, %0;" ::"r"(y_threads) : "memory");
                else if (d == 2) asm volatile("bar.sync 2, %0;" ::"r"(z_threads) : "memory");
            }
            // ---- faces: beyond the own cell; halo warps 0 and 2 the tile's first
            // y and z faces
            double F[5];
            if (d == 0 ? i >= i0 - 1 : full) {
                // from the cell to the one beyond the face, in each ring
                const int nR = d == 0 ? (rn - rs) * RP : d == 1 ? RR : 3;
                const int nV = d == 0 ? (((i + 1) & 1) - (i & 1)) * VP : d == 1 ? VR : 5;
                // along the tangentials: a is x (y, z faces) or y, b is z or y
                const int ahi = d == 0 ? RR : (rn - rs) * RP, alo = d == 0 ? -RR : (rb - rs) * RP;
                const int bhi = d == 2 ? RR : 3, blo = -bhi;
                const int fr = r, fc = cl;
                const bool act = own || (hw == 0 && k <= D) || (hw == 2 && l < WJ && j <= H);
                double Lm[5];
#pragma unroll
                for (int q = 0; q < 5; q++) {
                    Lm[q] = d == 0 ? carry[q] : hi[q];
                    carry[q] = hi[q];
                }
                if (act) {
                    const double *Rs = SLd + fr * SR + fc * 5 + (d == 0 ? 0 : d == 1 ? SR : 5);
                    // zero-gradient y: both sides of a boundary face are the cell's own state
                    const bool top = tpl && d == 1 && j == H, bottom = tpl && d == 1 && j == 0;
                    double Rp[5];
#pragma unroll
                    for (int q = 0; q < 5; q++) {
                        const double x = top ? Lm[q] : Rs[q];
                        Rp[q] = x;
                        Lm[q] = bottom ? x : Lm[q];
                    }
                    double Rho, P, vn, va, vb;
                    face_riemann(d, Lm, Rp, Rho, P, vn, va, vb);
                    const double *vm = V0 + (i & 1) * VP + fr * VR + fc * 5, *vp = vm + nV;
                    const double *rm = R0 + rs * RP + fr * RR + fc * 3, *rp = rm + nR;
                    const double vmn = vm[cn], vma = vm[ca], vmb = vm[cb], vpn = vp[cn], vpa = vp[ca], vpb = vp[cb];
                    const double gnn = (vpn - vmn) * rdn, gan = (vpa - vma) * rdn, gbn = (vpb - vmb) * rdn;
                    const double gna = (rp[ahi + cn] + rm[ahi + cn] - rp[alo + cn] - rm[alo + cn]) * r4a;
                    const double gaa = (rp[ahi + ca] + rm[ahi + ca] - rp[alo + ca] - rm[alo + ca]) * r4a;
                    const double gnb = (rp[bhi + cn] + rm[bhi + cn] - rp[blo + cn] - rm[blo + cn]) * r4b;
                    const double gbb = (rp[bhi + cb] + rm[bhi + cb] - rp[blo + cb] - rm[blo + cb]) * r4b;
                    double mu_T;
                    if constexpr (SST) { // static_mu_t in the frame
                        const double gba = (rp[ahi + cb] + rm[ahi + cb] - rp[alo + cb] - rm[alo + cb]) * r4a;
                        const double gab = (rp[bhi + ca] + rm[bhi + ca] - rp[blo + ca] - rm[blo + ca]) * r4b;
                        const double Sa = 0.5 * (gna + gan), Sb = 0.5 * (gnb + gbn), Sx = 0.5 * (gab + gba);
                        const double na = Sa * Sa, nb_ = Sb * Sb, ab = Sx * Sx;
                        const double y1 = d == 0 ? nb_ : ab, y2 = d == 0 ? ab : nb_;
                        const double S = sqrt(2 * (nat3(d, gnn * gnn, gaa * gaa, gbb * gbb) + 2 * (na + y1 + y2)));
                        const double *u = U0 + (i & 3) * UP + fr * UR + fc * 5;
                        const int nU = d == 0 ? (((i + 1) & 3) - (i & 3)) * UP : d == 1 ? UR : 5;
                        mu_T = 0.5 * (u[nU] + u[0]) * kc.CsDD * S;
                    } else {
                        mu_T = vp[4];
                    }
                    const double mu_E = kc.mu_L + mu_T;
                    const double sn = kk::TWO_THIRDS * mu_E * (gnn + gnn - gaa - gbb);
                    const double sa = mu_E * (gna + gan), sb = mu_E * (gnb + gbn);
                    const double lambda_E = kc.lambda_L + mu_T * kc.cp_Pr_T;
                    const double qn = -lambda_E * (vp[3] - vm[3]) * rdn;
                    const double RU = Rho * vn;
                    F[0] = RU;
                    F[1] = RU * vn + P - sn;
                    F[2] = RU * va - sa;
                    F[3] = RU * vb - sb;
                    // the work of the stresses, subtracted in natural order
                    const double tn = 0.5 * (vpn + vmn) * sn, ta = 0.5 * (vpa + vma) * sa, tb = 0.5 * (vpb + vmb) * sb;
                    const double x1 = d == 0 ? tn : ta, x2 = d == 0 ? ta : d == 1 ? tn : tb, x3 = d == 2 ? tn : tb;
                    F[4] = vn * (kk::K_K_1 * P + 0.5 * Rho * nat3(d, vn * vn, va * va, vb * vb)) - x1 - x2 - x3 + qn;
                    if (d != 0) {
                        // slot (row, column) holds the face before cell (row, column)
                        double *dst = SFd + fr * SR + fc * 5 + (d == 1 ? SR : 5);
#pragma unroll
                        for (int q = 0; q < 5; q++) dst[q] = F[q];
                    }
                }
            } else if (d == 0) {
#pragma unroll
                for (int q = 0; q < 5; q++) carry[q] = hi[q];
            }
            double unv[5];
            long long c = 0;
            if (d == 0 && full && own) {
                c = FSL_CELL(g.idx(i, j, k), fs);
                if (A.stage != 1) {
#pragma unroll
                    for (int q = 0; q < 5; q++) unv[q] = A.un[q * fs + c];
                }
            }
            __syncthreads();
            if (d != 0) {
                // ---- groups y, z: velocities and roots of plane i+2
                if (next) prims(i + 2);
            } else if (i >= i0 - 1) {
                // ---- group x: divergence and stage combination (src/evolution.c:29-161)
                double co = 0.0;
                if (full && own) {
                    const double one_third = 1. / 3., two_thirds = 2. / 3.;
                    const double *u = U0 + (i & 3) * UP + r * UR + l * 5;
                    const double *fy = &s.SF[0][r][l][0], *fz = &s.SF[1][r][l][0];
                    double o[5];
#pragma unroll
                    for (int q = 0; q < 5; q++) {
                        const int qy = q == 1 ? 2 : q == 2 ? 1 : q, qz = q == 1 ? 2 : q == 2 ? 3 : q == 3 ? 1 : q;
                        const double X = dtx * (Fxp[q] - F[q]);
                        const double Y = dty * (fy[qy] - fy[SR + qy]);
                        const double Z = dtz * (fz[qz] - fz[5 + qz]);
                        const double b1 = u[q] + X + Y + Z;
                        if (A.stage == 1) o[q] = b1;
                        else if (A.stage == 2) o[q] = 0.75 * unv[q] + 0.25 * b1;
                        else o[q] = one_third * unv[q] + two_thirds * b1;
                        A.out[q * fs + c] = o[q];
                    }
                    const bool bx = i == 1 || i == L, by = j == 1 || j == H, bz = k == 1 || k == D;
                    if (tpl && A.stage != 3 && (bx || by || bz)) {
                        // the ghost cells that copy this cell (the ghost pass's periodic
                        // x and z and zero-gradient y rules, edges and corners included);
                        // U^{n+1} keeps the ghost layer of U^n, as the reference's
                        // stages leave it to its Output()
                        const int xi[2] = {i, i == L ? 0 : (i == 1 ? L + 1 : -1)};
                        const int yj[2] = {j, j == 1 ? 0 : (j == H ? H + 1 : -1)};
                        const int zk[2] = {k, k == D ? 0 : (k == 1 ? D + 1 : -1)};
#pragma unroll 1
                        for (int e = 1; e < 8; e++) {
                            const int gi = xi[e & 1], gj = yj[(e >> 1) & 1], gk = zk[e >> 2];
                            if (gi < 0 || gj < 0 || gk < 0) continue;
                            const long long gc = FSL_CELL(g.idx(gi, gj, gk), fs);
#pragma unroll
                            for (int q = 0; q < 5; q++) A.out[q * fs + gc] = o[q];
                        }
                    }
                    if (A.co && i >= A.co_i0 && i <= A.co_i1) {
                        co = cell_courant(kc.cfl_mode, o[0], o[1], o[2], o[3], o[4], dtx, dty, dtz);
                        if (!(o[0] > 0.0)) atomicOr(A.status, 2u);
                    }
                }
                if (A.co && full) {
                    // (a NaN is ignored, as by the standalone reduction)
#pragma unroll
                    for (int w = 16; w > 0; w >>= 1) {
                        const double x = __shfl_xor_sync(0xffffffffu, co, w);
                        co = (x > co) ? x : co;
                    }
                    if (l == 0 && co > s.co[r]) s.co[r] = co;
                }
#pragma unroll
                for (int q = 0; q < 5; q++) Fxp[q] = F[q];
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
        }
    }
    if (A.co) {
        __syncthreads();
        if (t == 0) {
            double m = 0.0;
#pragma unroll
            for (int q = 0; q < WJ; q++) m = (s.co[q] > m) ? s.co[q] : m;
            // non-negative doubles order like their bit patterns
            atomicMax(A.co, (unsigned long long)__double_as_longlong(m));
        }
    }
}

template <bool SST>
int launch_stage_dir(Ctx &c, int stage, const double *cur, const double *un, double *out, const double *mu,
                     BF<double> bf, bool courant, int seg)
{
    static std::atomic<uint64_t> attr{0};
    if (!smem_limit_once((const void *)k_stage_dir<SST>, sizeof(Smem), attr)) return -1;
    DirArgs a;
    a.g = c.g;
    a.kc = c.k;
    a.cur = cur; a.un = un; a.out = out; a.mu = mu; a.bf = bf; a.ds = c.ds;
    a.co = courant ? &c.ds->co_bits : nullptr;
    a.status = &c.ds->status;
    a.co_i0 = c.co_i0;
    a.co_i1 = c.co_i1;
    a.stage = stage;
    a.seg = seg;
    const unsigned tiles = (unsigned)(((c.g.D + WK - 1) / WK) * ((c.g.H + WJ - 1) / WJ));
    prof_begin(c, FSL_K_STAGE);
    launch_following(k_stage_dir<SST>, dim3(tiles * (unsigned)((c.g.L + seg - 1) / seg)), NT, sizeof(Smem), c.stream, a);
    prof_end(c, FSL_K_STAGE, 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

} // namespace dirs
} // namespace fsl
