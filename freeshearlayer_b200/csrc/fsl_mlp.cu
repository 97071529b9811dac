// fsl_mlp.cu -- learned subgrid closure: a per-cell MLP 8 -> 64 -> 64 -> 64 -> 1
// (SiLU) mapping local strain-rate and density invariants to the Smagorinsky
// coefficient Cs^2 (the quantity the dynamic procedure computes as Cd,
// src/turbulence.c:433-440), trained on that procedure's output.
//
// All three hidden layers run on the 5th-generation tensor cores (tcgen05,
// BF16 operands, FP32 accumulation in tensor memory), 128 cells per tile (one
// cell per thread and TMEM lane).  Training keeps the pre-activations in TMEM
// for the backward pass; the data gradients (dz W) and the weight gradients
// (dz^T a, over the 128 cells of a tile, accumulated across a block's tiles)
// are tensor-core GEMMs too.  Weight-gradient operands are staged transposed
// and zero-padded to 128 rows so every product has the one verified shape
// M = 128 with K-major operands.
#include <cuda_bf16.h>

#define FSL_CHK_UNIT FSL_CHK_MLP
#include "fsl_check.cuh"
#include "fsl_internal.h"
#include "fsl_mlp.h"
#include "fsl_umma.cuh"

FSL_CHK_EXPORT(mlp)

namespace fsl {
namespace mlp {

constexpr uint32_t kWaitLimit = 1u << 24; // mbarrier polls before giving up

// ---- features (shared by inference and harvest) ------------------------------
// Strain rate from central differences of u = rho u * (1/rho), as the dynamic
// procedure forms it (src/turbulence.c:201-205, :273-301), in FP32.
__device__ __forceinline__ void cell_features(const Grid &g, const double *__restrict__ U, long long c,
                                              const ClosureScales &sc, float *f, float &rho, float &Smag)
{
    const long long fs = g.fstride;
    float u[7], v[7], w[7];
    const long long off[7] = {0, g.pi, -g.pi, (long long)g.pk, -(long long)g.pk, 1, -1};
#pragma unroll
    for (int n = 0; n < 7; n++) {
        const long long a = c + off[n];
        const double r = U[a];
        const float rr = (float)(1. / r);
        u[n] = (float)U[fs + a] * rr;
        v[n] = (float)U[2 * fs + a] * rr;
        w[n] = (float)U[3 * fs + a] * rr;
        if (n == 0) rho = (float)r;
    }
    const float ax = sc.r2dx, ay = sc.r2dy, az = sc.r2dz;
    const float du_dx = (u[1] - u[2]) * ax, du_dy = (u[3] - u[4]) * ay, du_dz = (u[5] - u[6]) * az;
    const float dv_dx = (v[1] - v[2]) * ax, dv_dy = (v[3] - v[4]) * ay, dv_dz = (v[5] - v[6]) * az;
    const float dw_dx = (w[1] - w[2]) * ax, dw_dy = (w[3] - w[4]) * ay, dw_dz = (w[5] - w[6]) * az;
    const float S11 = du_dx, S22 = dv_dy, S33 = dw_dz;
    const float S12 = 0.5f * (du_dy + dv_dx), S13 = 0.5f * (du_dz + dw_dx), S23 = 0.5f * (dv_dz + dw_dy);
    const float S = sqrtf(2.f * (S11 * S11 + S22 * S22 + S33 * S33 + 2.f * (S12 * S12 + S13 * S13 + S23 * S23)));
    Smag = S;
    const float inv = 1.f / (S + 1e-30f);
    f[0] = log1pf(S * sc.t_ref);
    f[1] = S11 * inv;
    f[2] = S22 * inv;
    f[3] = S12 * inv;
    f[4] = S13 * inv;
    f[5] = S23 * inv;
    f[6] = rho;
    f[7] = sc.delta_ratio;
}

// FP32 velocities of every padded cell, formed exactly as cell_features forms
// them (rho u as float times the float of the FP64 reciprocal), so features
// computed from this field equal cell_features bit for bit.
__global__ void k_closure_vel(Grid g, const double *__restrict__ U, float *__restrict__ vel)
{
    const long long fs = g.fstride;
    const long long n = (long long)(g.L + 2) * g.pi;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        if ((int)(t % g.pk) >= g.D + 2) continue; // row padding
        const long long a = FSL_CELL(g.off + t, fs);
        const double r = U[a];
        const float rr = (float)(1. / r);
        vel[a] = (float)U[fs + a] * rr;
        vel[fs + a] = (float)U[2 * fs + a] * rr;
        vel[2 * fs + a] = (float)U[3 * fs + a] * rr;
    }
}

// The raw inputs of one cell's features: the six neighbours' velocities and
// the cell's density, loaded one tile ahead of their use.
struct FeatIn {
    float u[7], v[7], w[7];
    double r;
    long long c;
    bool valid;
};

__device__ __forceinline__ void feat_load(const Grid &g, const double *__restrict__ U, const float *__restrict__ vel,
                                          long long cell, long long ncell, FeatIn &p)
{
    p.valid = cell < ncell;
    p.c = 0;
    if (!p.valid) return;
    // 32-bit index arithmetic (the launcher refuses grids of 2^31 cells or
    // more): an unsigned 32-bit division is a short inline sequence, a 64-bit
    // one a long subroutine, in a kernel whose issue slots are the limit
    const unsigned cu = (unsigned)cell, D = (unsigned)g.D, H = (unsigned)g.H;
    const unsigned rr = cu / D, ii = rr / H;
    const int k = (int)(cu - rr * D) + 1;
    const int j = (int)(rr - ii * H) + 1, i = (int)ii + 1;
    const long long c = g.idx(i, j, k), fs = g.fstride;
    const long long off[7] = {0, g.pi, -g.pi, (long long)g.pk, -(long long)g.pk, 1, -1};
#pragma unroll
    for (int n = 1; n < 7; n++) {
        const long long a = FSL_CELL(c + off[n], fs);
        p.u[n] = vel[a];
        p.v[n] = vel[fs + a];
        p.w[n] = vel[2 * fs + a];
    }
    p.r = U[FSL_CELL(c, fs)];
    p.c = c;
}

__device__ __forceinline__ void cell_features_v(const FeatIn &p, const ClosureScales &sc, float *f, float &rho,
                                                float &Smag)
{
    const float *u = p.u, *v = p.v, *w = p.w;
    rho = (float)p.r;
    const float ax = sc.r2dx, ay = sc.r2dy, az = sc.r2dz;
    const float du_dx = (u[1] - u[2]) * ax, du_dy = (u[3] - u[4]) * ay, du_dz = (u[5] - u[6]) * az;
    const float dv_dx = (v[1] - v[2]) * ax, dv_dy = (v[3] - v[4]) * ay, dv_dz = (v[5] - v[6]) * az;
    const float dw_dx = (w[1] - w[2]) * ax, dw_dy = (w[3] - w[4]) * ay, dw_dz = (w[5] - w[6]) * az;
    const float S11 = du_dx, S22 = dv_dy, S33 = dw_dz;
    const float S12 = 0.5f * (du_dy + dv_dx), S13 = 0.5f * (du_dz + dw_dx), S23 = 0.5f * (dv_dz + dw_dy);
    const float S = sqrtf(2.f * (S11 * S11 + S22 * S22 + S33 * S33 + 2.f * (S12 * S12 + S13 * S13 + S23 * S23)));
    Smag = S;
    const float inv = 1.f / (S + 1e-30f);
    f[0] = log1pf(S * sc.t_ref);
    f[1] = S11 * inv;
    f[2] = S22 * inv;
    f[3] = S12 * inv;
    f[4] = S13 * inv;
    f[5] = S23 * inv;
    f[6] = rho;
    f[7] = sc.delta_ratio;
}

// SiLU and its derivative with sigmoid(x) = 0.5 tanh(x/2) + 0.5
__device__ __forceinline__ float tanh_fast(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sigm(float x) { return 0.5f * tanh_fast(0.5f * x) + 0.5f; }
__device__ __forceinline__ float silu(float x) { return x * sigm(x); }
__device__ __forceinline__ float dsilu(float x)
{
    const float s = sigm(x);
    return s + x * s * (1.f - s);
}

// ---- weights in shared memory ------------------------------------------------
struct SmemW {
    alignas(128) __nv_bfloat16 W1[64 * 16];
    alignas(128) __nv_bfloat16 W2[64 * 64];
    alignas(128) __nv_bfloat16 W3[64 * 64];
    alignas(16) float b1[64];
    float b2[64], b3[64], w4[64], b4;
};

__device__ __forceinline__ void stage_weights(SmemW &s, const float *__restrict__ P, int t, int nt)
{
    for (int e = t; e < 64 * 16; e += nt) {
        const int o = e / 16, i = e % 16;
        s.W1[umma::tile_off(o, i, 16) / 2] = __float2bfloat16_rn(P[kOffW1 + o * 16 + i]);
    }
    for (int e = t; e < 64 * 64; e += nt) {
        const int o = e / 64, i = e % 64;
        s.W2[umma::tile_off(o, i, 64) / 2] = __float2bfloat16_rn(P[kOffW2 + e]);
        s.W3[umma::tile_off(o, i, 64) / 2] = __float2bfloat16_rn(P[kOffW3 + e]);
    }
    for (int e = t; e < 64; e += nt) {
        s.b1[e] = P[kOffB1 + e];
        s.b2[e] = P[kOffB2 + e];
        s.b3[e] = P[kOffB3 + e];
        s.w4[e] = P[kOffW4 + e];
    }
    if (t == 0) s.b4 = P[kOffB4];
}

// ---- inference -----------------------------------------------------------------
// The inference tiles fold everything linear into the tensor-core products:
// each layer's operand carries two constant-one columns (K = 16 for the
// features, 80 = 64 + 16 for the hidden layers) against the bias split into a
// BF16 high and low part, and weights and biases of the hidden layers are
// pre-scaled by 1/2, so the accumulator holds h = (z + b) / 2 and
// silu(z + b) = h + h tanh(h) needs no further FP32 work.  The output layer
// is a fourth product with N = 16 (row 0 live, K = 64) plus b4 in FP32.
// The feature tile (128 x 16) occupies the first 4 KB of the activation
// tile, which the first layer's epilogue overwrites only after the first
// product has read it: 45 KB per block, five blocks per SM.
constexpr int kKH = 80; // K of the hidden-layer operands

struct SmemInfer {
    alignas(128) __nv_bfloat16 W1[64 * 16];
    alignas(128) __nv_bfloat16 W2[64 * kKH];
    alignas(128) __nv_bfloat16 W3[64 * kKH];
    alignas(128) __nv_bfloat16 W4[16 * 64];
    // activations (K-major; columns 64, 65 one, 66..79 zero); before the
    // first product, the features (K = 16; columns 8, 9 one, 10..15 zero)
    alignas(128) __nv_bfloat16 A[128 * kKH];
    uint64_t mbar;
    uint32_t tholder;
    float b4;
};

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16 &hi, __nv_bfloat16 &lo)
{
    hi = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}

// element (o, i) of a K-major operand of width K
__device__ __forceinline__ __nv_bfloat16 &tile_el(__nv_bfloat16 *T, int o, int i, int K)
{
    return T[umma::tile_off(o, i, K) / 2];
}

__device__ __forceinline__ void stage_infer_weights(SmemInfer &s, const float *__restrict__ P, int t, int nt)
{
    const __nv_bfloat16 z = __float2bfloat16_rn(0.f);
    for (int e = t; e < 64 * 16; e += nt) {
        const int o = e / 16, i = e % 16;
        __nv_bfloat16 v = z;
        if (i < 8) v = __float2bfloat16_rn(0.5f * P[kOffW1 + o * 16 + i]);
        tile_el(s.W1, o, i, 16) = v;
    }
    for (int e = t; e < 64 * kKH; e += nt) {
        const int o = e / kKH, i = e % kKH;
        __nv_bfloat16 v2 = z, v3 = z;
        if (i < 64) {
            v2 = __float2bfloat16_rn(0.5f * P[kOffW2 + o * 64 + i]);
            v3 = __float2bfloat16_rn(0.5f * P[kOffW3 + o * 64 + i]);
        }
        tile_el(s.W2, o, i, kKH) = v2;
        tile_el(s.W3, o, i, kKH) = v3;
    }
    for (int e = t; e < 16 * 64; e += nt) {
        const int o = e / 64, i = e % 64;
        tile_el(s.W4, o, i, 64) = o == 0 ? __float2bfloat16_rn(P[kOffW4 + i]) : z;
    }
    if (t == 0) s.b4 = P[kOffB4];
    __syncthreads(); // the bias columns below overwrite zeros written above
    if (t < 64) {
        __nv_bfloat16 hi, lo;
        split_bf16(0.5f * P[kOffB1 + t], hi, lo);
        tile_el(s.W1, t, 8, 16) = hi;
        tile_el(s.W1, t, 9, 16) = lo;
        split_bf16(0.5f * P[kOffB2 + t], hi, lo);
        tile_el(s.W2, t, 64, kKH) = hi;
        tile_el(s.W2, t, 65, kKH) = lo;
        split_bf16(0.5f * P[kOffB3 + t], hi, lo);
        tile_el(s.W3, t, 64, kKH) = hi;
        tile_el(s.W3, t, 65, kKH) = lo;
    }
}

// silu of two values in packed BF16 arithmetic from h = (z + b) / 2 given in
// FP32: silu = h + h tanh(h), one MUFU operation per pair.  h is cut to BF16
// by truncation (a byte permute on the integer pipe).  Result: element 0 in
// the low half (the lower k of a K-major tile row).
__device__ __forceinline__ uint32_t silu2_bf16(float h0, float h1)
{
    uint32_t th, y;
    const uint32_t hp = __byte_perm(__float_as_uint(h0), __float_as_uint(h1), 0x7632);
    asm("tanh.approx.bf16x2 %0, %1;" : "=r"(th) : "r"(hp));
    asm("fma.rn.bf16x2 %0, %1, %2, %1;" : "=r"(y) : "r"(hp), "r"(th));
    return y;
}

// silu of two values on the FMA pipe (the MUFU pipe runs the others): tanh
// from an odd polynomial of degree 13 on [-3.3, 3.3], h clamped there,
// coefficients this project fitted near-minimax on Chebyshev nodes with
// Lawson's iteratively reweighted least squares (max |error| 1.4e-3,
// including the clamp; the BF16 result rounds at 2^-9 relative), then
// silu = h + h tanh(h) and one rounding to BF16.  The pair is evaluated in
// packed FP32 arithmetic (sm_100 issues two FP32 FMAs per instruction),
// written with the compiler's packed builtins rather than inline PTX so the
// compiler sees the coefficient pairs as constants (the same roundings; the
// step 0.7 % faster than the inline-PTX form).
__device__ __forceinline__ uint32_t silu2_poly(float h0, float h1)
{
    const float2 x = make_float2(fminf(fmaxf(h0, -3.3f), 3.3f), fminf(fmaxf(h1, -3.3f), 3.3f));
    const float2 h = make_float2(h0, h1), x2 = __fmul2_rn(x, x);
    float2 p = __ffma2_rn(make_float2(2.460764335e-06f, 2.460764335e-06f), x2,
                          make_float2(-1.012231442e-04f, -1.012231442e-04f));
    p = __ffma2_rn(p, x2, make_float2(1.705276780e-03f, 1.705276780e-03f));
    p = __ffma2_rn(p, x2, make_float2(-1.538222842e-02f, -1.538222842e-02f));
    p = __ffma2_rn(p, x2, make_float2(8.308345824e-02f, 8.308345824e-02f));
    p = __ffma2_rn(p, x2, make_float2(-2.995448709e-01f, -2.995448709e-01f));
    p = __ffma2_rn(p, x2, make_float2(9.929457903e-01f, 9.929457903e-01f));
    const float2 y = __ffma2_rn(h, __fmul2_rn(p, x), h);
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y.y), "f"(y.x));
    return r;
}

// one tensor-core layer: D = A W^T into TMEM, wait; returns false on timeout
__device__ __forceinline__ bool layer_mma(uint32_t tmem, uint32_t a, int Ka, uint32_t b, int Kb, int K, int N,
                                          uint64_t *mbar, uint32_t &phase, int t)
{
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (t == 0) {
        umma::gemm_issue2(tmem, a, Ka, b, Kb, K, N);
        umma::commit(mbar);
    }
    bool ok = umma::mbar_wait(mbar, phase, kWaitLimit);
    phase ^= 1u;
    ok = __syncthreads_and(ok) != 0;
    umma::fence_after_sync();
    return ok;
}

// SiLU of this thread's TMEM accumulator row (64 columns, h = (z + b) / 2)
// into row t of the next activation tile (K = 80), 8 BF16 per 16-byte store.
// Of each chunk's 8 pairs, the first kPolyPairs take the FMA-pipe tanh and
// the rest the MUFU one: the MUFU pipe sets the kernel's pace, and a MUFU
// tanh of a warp's 64 values leaves ~13 issue slots free on its scheduler
// (FSL_TUNE_CLOSURE_POLY picks the split).
template <int kPolyPairs, bool kOnes>
__device__ __forceinline__ void epilogue_to_tile(uint32_t taddr, unsigned char *A, int t)
{
    const uint32_t row = (uint32_t)(t >> 3) * (uint32_t)(kKH * 16) + (uint32_t)(t & 7) * 16u;
    if constexpr (kOnes) {
        // columns 64..79 = (1, 1, 0, ...): the feature tile overlaid them
        *reinterpret_cast<uint4 *>(A + row + 8u * 128u) = make_uint4(0x3F803F80u, 0u, 0u, 0u);
        *reinterpret_cast<uint4 *>(A + row + 9u * 128u) = make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
        float v[16];
        umma::tmem_ld16(taddr + (uint32_t)(c * 16), v);
        umma::tmem_wait_ld();
        uint32_t y[8];
#pragma unroll
        for (int q = 0; q < 8; q++)
            y[q] = q < kPolyPairs ? silu2_poly(v[2 * q], v[2 * q + 1]) : silu2_bf16(v[2 * q], v[2 * q + 1]);
#pragma unroll
        for (int half = 0; half < 2; half++)
            *reinterpret_cast<uint4 *>(A + row + (uint32_t)(c * 2 + half) * 128u) =
                make_uint4(y[4 * half], y[4 * half + 1], y[4 * half + 2], y[4 * half + 3]);
    }
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// Persistent: each block (one warpgroup) walks tiles of 128 interior cells in
// (i, j, k) order; mu = rho Cs^2 DD |S| (the reference's formula,
// src/turbulence.c:442) with Cs^2 from the MLP clipped to [0, 0.15].  The
// hidden-layer SiLU runs in packed BF16 (its results are BF16 operands of the
// next product either way); the last layer's dot product with w4 is FP32.
template <typename MT, int NP>
__global__ void __launch_bounds__(128, NP <= 3 ? 5 : 4) k_closure_infer(Grid g, ClosureScales sc, const double *__restrict__ U,
                                                          const float *__restrict__ vel,
                                                          const float *__restrict__ P, MT *__restrict__ mu,
                                                          float *__restrict__ cs2_out, int *err)
{
    extern __shared__ __align__(1024) unsigned char smraw[];
    SmemInfer &s = *reinterpret_cast<SmemInfer *>(smraw);
    const int t = threadIdx.x, wp = t >> 5;
    stage_infer_weights(s, P, t, 128);
    unsigned char *A = reinterpret_cast<unsigned char *>(s.A);
    const uint32_t one2 = 0x3F803F80u; // two BF16 ones
    // feature row t (the 128 x 16 tile at the start of A): columns 0..7 at
    // +0, columns 8..15 = (1, 1, 0, ...) at +128
    const uint32_t frow = (uint32_t)(t >> 3) * 256u + (uint32_t)(t & 7) * 16u;
    if (t == 0) umma::mbar_init(&s.mbar, 1);
    if (wp == 0) umma::tmem_alloc(&s.tholder, 64);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = s.tholder;
    const uint32_t lane_addr = tmem + ((uint32_t)(32 * wp) << 16);
    const uint32_t aA = umma::smem_u32(s.A), aW1 = umma::smem_u32(s.W1), aW2 = umma::smem_u32(s.W2),
                   aW3 = umma::smem_u32(s.W3), aW4 = umma::smem_u32(s.W4);
    const float b4 = s.b4;
    uint32_t phase = 0;
    bool ok = true;
    const long long ncell = (long long)g.L * g.H * g.D;
    const long long ntile = (ncell + 127) / 128;
    FeatIn in;
    feat_load(g, U, vel, (long long)blockIdx.x * 128 + t, ncell, in);
    for (long long tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
        const bool valid = in.valid;
        const long long c = in.c;
        float f[8] = {0, 0, 0, 0, 0, 0, 0, 0}, rho = 0.f, Smag = 0.f;
        if (valid) cell_features_v(in, sc, f, rho, Smag);
        *reinterpret_cast<uint4 *>(A + frow) =
            make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
        *reinterpret_cast<uint4 *>(A + frow + 128u) = make_uint4(one2, 0u, 0u, 0u);
        // the next tile's inputs load while this tile is on the tensor cores
        feat_load(g, U, vel, (tile + gridDim.x) * 128 + t, ncell, in);
        ok = layer_mma(tmem, aA, 16, aW1, 16, 16, 64, &s.mbar, phase, t);
        if (!ok) break;
        epilogue_to_tile<NP, true>(lane_addr, A, t);
        ok = layer_mma(tmem, aA, kKH, aW2, kKH, kKH, 64, &s.mbar, phase, t);
        if (!ok) break;
        epilogue_to_tile<NP, false>(lane_addr, A, t);
        ok = layer_mma(tmem, aA, kKH, aW3, kKH, kKH, 64, &s.mbar, phase, t);
        if (!ok) break;
        epilogue_to_tile<NP, false>(lane_addr, A, t);
        ok = layer_mma(tmem, aA, kKH, aW4, 64, 64, 16, &s.mbar, phase, t);
        if (!ok) break;
        float v[16];
        umma::tmem_ld16(lane_addr, v);
        umma::tmem_wait_ld();
        const float cs2 = fminf(fmaxf(v[0] + b4, 0.f), 0.15f);
        if (valid) {
            const long long cc = FSL_CELL(c, g.fstride);
            mu[cc] = (MT)(rho * cs2 * sc.DD * Smag);
            if (cs2_out) cs2_out[cc] = cs2;
        }
    }
    if (!ok) {
        atomicExch(err, 1);
        umma::mbar_wait(&s.mbar, phase ^ 1u, kWaitLimit);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (wp == 0) umma::tmem_free(tmem, 64);
}

// ---- harvest -------------------------------------------------------------------
// Every `stride`-th cell of the band two cells away from every boundary
// (i in [3, LEN-2], likewise j, k): its 8 features and the dynamic
// procedure's Cs^2 (cd, a padded FP32 field written by the SGS pass).  Within
// two cells of a boundary the dynamic Cs^2 carries the zero padding of the
// reference's test filter (src/turbulence.c:44-95) rather than the flow.
__global__ void k_harvest(Grid g, ClosureScales sc, const double *__restrict__ U, const float *__restrict__ cd,
                          long long stride, long long offset, float *__restrict__ X, float *__restrict__ Y,
                          long long cap, long long base)
{
    const int bL = g.L - 4, bH = g.H - 4, bD = g.D - 4;
    const long long ncell = (long long)bL * bH * bD;
    const long long nsamp = (ncell - offset + stride - 1) / stride;
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < nsamp;
         s += (long long)gridDim.x * blockDim.x) {
        const long long dst = base + s;
        if (dst >= cap) return;
        const long long cell = offset + s * stride;
        const int k = (int)(cell % bD) + 3;
        const long long rr = cell / bD;
        const int j = (int)(rr % bH) + 3, i = (int)(rr / bH) + 3;
        const long long c = g.idx(i, j, k);
        float f[8], rho, Smag;
        cell_features(g, U, c, sc, f, rho, Smag);
#pragma unroll
        for (int q = 0; q < 8; q++) X[dst * 8 + q] = f[q];
        Y[dst] = cd[c];
    }
}

// ---- training --------------------------------------------------------------------
// TMEM columns of one training block
constexpr uint32_t kZ1 = 0, kZ2 = 64, kZ3 = 128, kGW1 = 192, kGW2 = 256, kGW3 = 320, kDG = 384;

constexpr int kTrainThreads = 512; // four per cell of a tile

struct SmemTrain {
    SmemW w;
    alignas(128) __nv_bfloat16 W2T[64 * 64]; // B operand of the data gradient: [in][out]
    alignas(128) __nv_bfloat16 W3T[64 * 64];
    alignas(128) __nv_bfloat16 A0[128 * 16];  // features, [cell][16]
    alignas(128) __nv_bfloat16 A0T[16 * 128]; // features, [in][cell]
    alignas(128) __nv_bfloat16 A1[128 * 64];
    alignas(128) __nv_bfloat16 A2[128 * 64];
    alignas(128) __nv_bfloat16 A1T[64 * 128];
    alignas(128) __nv_bfloat16 A2T[64 * 128];
    alignas(128) __nv_bfloat16 DZ[128 * 64];   // dz, [cell][out]
    alignas(128) __nv_bfloat16 DZT[128 * 128]; // dz, [out (64, zero-padded to 128)][cell]
    float gsum[4][4][64];            // per warp: the gradients of b1, b2, b3, w4
    float gone[4][2];                // per warp: the gradient of b4, the loss
    float ypart[4][128];             // the four threads' parts of a cell's output
    uint64_t mbar;
    uint32_t tholder;
};

__device__ __forceinline__ void mma_wait(SmemTrain &s, uint32_t &phase, bool &ok)
{
    ok = ok && umma::mbar_wait(&s.mbar, phase, kWaitLimit);
    phase ^= 1u;
    ok = __syncthreads_and(ok) != 0;
    umma::fence_after_sync();
}

__device__ __forceinline__ void sync_for_mma()
{
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
}

// 16 consecutive columns (from column c0, a multiple of 8) of row t of a K-major
// tile of width 64, as two 16-byte stores.
__device__ __forceinline__ void store_row16(__nv_bfloat16 *A, int t, int c0, const float *v)
{
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t p[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(v[8 * h + 2 * q], v[8 * h + 2 * q + 1]);
            p[q] = *reinterpret_cast<const uint32_t *>(&b);
        }
        *reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(A) + umma::tile_off(t, c0 + 8 * h, 64)) =
            make_uint4(p[0], p[1], p[2], p[3]);
    }
}

// This warp's 32 rows x 16 columns (chunk c) of the 128 x 64 tile A (K-major,
// width 64) into the transposed tile AT (rows = A's columns, width 128): 8 x 8
// core matrices through ldmatrix.trans / stmatrix, four at a time.
__device__ __forceinline__ void transpose_chunk(const __nv_bfloat16 *A, __nv_bfloat16 *AT, int wp, int c, int l)
{
    __syncwarp();
    const uint32_t src = umma::smem_u32(A) + (uint32_t)(wp * 4 + (l >> 3)) * 1024u + (uint32_t)(l & 7) * 16u;
    const uint32_t dst = umma::smem_u32(AT) + (uint32_t)(wp * 4 + (l >> 3)) * 128u + (uint32_t)(l & 7) * 16u;
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
        const uint32_t ob = 2u * (uint32_t)c + h;
        uint32_t r0, r1, r2, r3;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                     : "r"(src + ob * 128u)
                     : "memory");
        asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(dst + ob * 2048u), "r"(r0),
                     "r"(r1), "r"(r2), "r"(r3)
                     : "memory");
    }
}

// Sums over the warp's lanes of 16 values per lane: lane l receives the sum of
// value l & 15 (a halving butterfly: 16 shuffles instead of 16 x 5).
__device__ __forceinline__ float warp_colsum16(const float *in, int l)
{
    float v[16];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = in[q];
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        const bool up = (l & h) != 0;
#pragma unroll
        for (int q = 0; q < h; q++) {
            const float give = up ? v[q] : v[q + h], keep = up ? v[q + h] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, give, h);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

// Gradient of the mean squared error over n samples for the parameters P,
// accumulated per block into Gpart[blockIdx.x][kNParams]; loss_part holds
// the block's summed squared error.  Each block handles tiles
// [blockIdx.x * tpb, (blockIdx.x + 1) * tpb).  TMEM (448 of 512 columns) allows
// one block per SM, so the chain of six waits for eight products and their epilogues bounds
// it; four threads share a cell (a TMEM lane), each with 16 of a layer's 64
// columns, so that four warps a scheduler hide the epilogues' latency (a
// gradient of 2^20 samples: 0.85 ms with one thread a cell, 0.51 ms now).  The bias,
// w4 and loss sums are taken over a warp's lanes with shuffles and kept in
// registers from tile to tile: as atomic adds to one shared word per column they
// serialised a tile's cells 256 times over (75 ms).
__global__ void __launch_bounds__(kTrainThreads, 1) k_train_grad(const float *__restrict__ X, const float *__restrict__ Yt,
                                                       long long n, int tpb, const float *__restrict__ P,
                                                       float *__restrict__ Gpart, float *__restrict__ loss_part,
                                                       int *err, float inv_wmean)
{
    extern __shared__ __align__(1024) unsigned char smraw[];
    SmemTrain &s = *reinterpret_cast<SmemTrain *>(smraw);
    const int gave_up = threadIdx.x == 0 ? *err : 0; // in flight while the weights are staged
    // cell (TMEM lane) t of the tile, columns 16 c .. 16 c + 15
    const int x = threadIdx.x, t = x & 127, c = x >> 7, wp = t >> 5, l = t & 31, c0 = c * 16;
    stage_weights(s.w, P, x, kTrainThreads);
    for (int e = x; e < 64 * 64; e += kTrainThreads) {
        const int o = e / 64, i = e % 64; // W[o][i] -> WT[i][o]
        s.W2T[umma::tile_off(i, o, 64) / 2] = __float2bfloat16_rn(P[kOffW2 + e]);
        s.W3T[umma::tile_off(i, o, 64) / 2] = __float2bfloat16_rn(P[kOffW3 + e]);
    }
    // the padding: rows 64..127 of dz^T, inputs 8..15 of the features
    for (int e = x; e < 128 * 128; e += kTrainThreads) s.DZT[e] = __float2bfloat16_rn(0.f);
    for (int e = x; e < 128 * 16; e += kTrainThreads) s.A0[e] = s.A0T[e] = __float2bfloat16_rn(0.f);
    if (x == 0) umma::mbar_init(&s.mbar, 1);
    float gb1 = 0.f, gb2 = 0.f, gb3 = 0.f, gw4 = 0.f, gb4 = 0.f, loss = 0.f;
    // an earlier pass gave up: its caller reports it.  One thread's reading for all: a
    // block of this launch may set the flag while others start
    if (__syncthreads_or(gave_up)) return;
    if (x < 32) umma::tmem_alloc(&s.tholder, 512);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = s.tholder;
    const uint32_t lane = tmem + ((uint32_t)(32 * wp) << 16);
    const uint32_t aA0 = umma::smem_u32(s.A0), aA0T = umma::smem_u32(s.A0T), aA1 = umma::smem_u32(s.A1),
                   aA2 = umma::smem_u32(s.A2), aA1T = umma::smem_u32(s.A1T), aA2T = umma::smem_u32(s.A2T),
                   aDZ = umma::smem_u32(s.DZ), aDZT = umma::smem_u32(s.DZT), aW1 = umma::smem_u32(s.w.W1),
                   aW2 = umma::smem_u32(s.w.W2), aW3 = umma::smem_u32(s.w.W3), aW2T = umma::smem_u32(s.W2T),
                   aW3T = umma::smem_u32(s.W3T);
    const float scale = 2.f / (float)n;
    uint32_t phase = 0;
    bool ok = true;
    const long long ntile = (n + 127) / 128;
    float4 x0, x1; // the sample of this thread (each is 32 bytes, so 16-byte aligned)
    float yt;
    auto fetch = [&](long long tile, bool more) {
        const long long m = tile * 128 + t;
        x0 = x1 = make_float4(0.f, 0.f, 0.f, 0.f);
        yt = 0.f;
        if (more && m < n) {
            x0 = reinterpret_cast<const float4 *>(X)[2 * m];
            x1 = reinterpret_cast<const float4 *>(X)[2 * m + 1];
            yt = Yt[m];
        }
    };
    fetch((long long)blockIdx.x * tpb, true);
    for (int tt = 0; tt < tpb && ok; tt++) {
        const long long tile = (long long)blockIdx.x * tpb + tt;
        if (tile >= ntile) break; // uniform across the block
        const bool acc = tt > 0;
        const bool valid = tile * 128 + t < n;
        const float f[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
        const float target = yt;
        fetch(tile + 1, tt + 1 < tpb); // the next tile's samples, in flight during this one
        if (c == 0) {
            uint32_t p[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const __nv_bfloat162 b = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
                p[q] = *reinterpret_cast<const uint32_t *>(&b);
                s.A0T[umma::tile_off(2 * q, t, 128) / 2] = __low2bfloat16(b);
                s.A0T[umma::tile_off(2 * q + 1, t, 128) / 2] = __high2bfloat16(b);
            }
            *reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(s.A0) + umma::tile_off(t, 0, 16)) =
                make_uint4(p[0], p[1], p[2], p[3]);
        }
        // ---- forward: z1, z2, z3 stay in TMEM ----
        sync_for_mma();
        if (x == 0) { umma::gemm_issue(tmem + kZ1, aA0, aW1, 16, 64, false); umma::commit(&s.mbar); }
        mma_wait(s, phase, ok);
        if (!ok) break;
        {
            float v[16];
            umma::tmem_ld16(lane + kZ1 + c0, v);
            umma::tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = silu(v[q] + s.w.b1[c0 + q]);
            store_row16(s.A1, t, c0, v);
            transpose_chunk(s.A1, s.A1T, wp, c, l);
        }
        sync_for_mma();
        if (x == 0) { umma::gemm_issue(tmem + kZ2, aA1, aW2, 64, 64, false); umma::commit(&s.mbar); }
        mma_wait(s, phase, ok);
        if (!ok) break;
        {
            float v[16];
            umma::tmem_ld16(lane + kZ2 + c0, v);
            umma::tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = silu(v[q] + s.w.b2[c0 + q]);
            store_row16(s.A2, t, c0, v);
            transpose_chunk(s.A2, s.A2T, wp, c, l);
        }
        sync_for_mma();
        if (x == 0) { umma::gemm_issue(tmem + kZ3, aA2, aW3, 64, 64, false); umma::commit(&s.mbar); }
        mma_wait(s, phase, ok);
        if (!ok) break;
        // ---- output, loss gradient, layer 3 backward ----
        float z3[16], y = 0.f;
        umma::tmem_ld16(lane + kZ3 + c0, z3);
        umma::tmem_wait_ld();
#pragma unroll
        for (int q = 0; q < 16; q++) {
            z3[q] += s.w.b3[c0 + q];
            y += s.w.w4[c0 + q] * silu(z3[q]);
        }
        s.ypart[c][t] = y;
        __syncthreads();
        y = s.w.b4 + s.ypart[0][t] + s.ypart[1][t] + s.ypart[2][t] + s.ypart[3][t];
        // sample weight: 1, or (rho |S| t_ref)^2 over its dataset mean, which
        // makes the loss the squared error of mu_SGS = rho Cs^2 DD |S|
        float wgt = 1.f;
        if (inv_wmean > 0.f) {
            const float st = expm1f(f[0]) * f[6];
            wgt = st * st * inv_wmean;
        }
        const float e = valid ? (y - target) : 0.f;
        const float dy = scale * wgt * e;
        if (c == 0) {
            loss += wgt * e * e;
            gb4 += dy;
        }
        {
            float v[16], g4[16];
#pragma unroll
            for (int q = 0; q < 16; q++) {
                g4[q] = dy * silu(z3[q]);
                v[q] = dy * s.w.w4[c0 + q] * dsilu(z3[q]);
            }
            gw4 += warp_colsum16(g4, l);
            gb3 += warp_colsum16(v, l);
            store_row16(s.DZ, t, c0, v);
            transpose_chunk(s.DZ, s.DZT, wp, c, l);
        }
        // dW3 += dz3^T a2 ; da2 = dz3 W3
        sync_for_mma();
        if (x == 0) {
            umma::gemm_issue(tmem + kGW3, aDZT, aA2T, 128, 64, acc);
            umma::gemm_issue(tmem + kDG, aDZ, aW3T, 64, 64, false);
            umma::commit(&s.mbar);
        }
        mma_wait(s, phase, ok);
        if (!ok) break;
        {
            float v[16], zz[16];
            umma::tmem_ld16(lane + kDG + c0, v);
            umma::tmem_ld16(lane + kZ2 + c0, zz);
            umma::tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = valid ? v[q] * dsilu(zz[q] + s.w.b2[c0 + q]) : 0.f;
            gb2 += warp_colsum16(v, l);
            store_row16(s.DZ, t, c0, v);
            transpose_chunk(s.DZ, s.DZT, wp, c, l);
        }
        // dW2 += dz2^T a1 ; da1 = dz2 W2
        sync_for_mma();
        if (x == 0) {
            umma::gemm_issue(tmem + kGW2, aDZT, aA1T, 128, 64, acc);
            umma::gemm_issue(tmem + kDG, aDZ, aW2T, 64, 64, false);
            umma::commit(&s.mbar);
        }
        mma_wait(s, phase, ok);
        if (!ok) break;
        {
            float v[16], zz[16];
            umma::tmem_ld16(lane + kDG + c0, v);
            umma::tmem_ld16(lane + kZ1 + c0, zz);
            umma::tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = valid ? v[q] * dsilu(zz[q] + s.w.b1[c0 + q]) : 0.f;
            gb1 += warp_colsum16(v, l);
            store_row16(s.DZ, t, c0, v);
            transpose_chunk(s.DZ, s.DZT, wp, c, l);
        }
        // dW1 += dz1^T a0
        sync_for_mma();
        if (x == 0) {
            umma::gemm_issue(tmem + kGW1, aDZT, aA0T, 128, 16, acc);
            umma::commit(&s.mbar);
        }
        mma_wait(s, phase, ok);
        if (!ok) break;
    }
    // the warps' sums to shared memory (lanes 0..15 hold the chunk's 16 columns)
    if (l < 16) {
        s.gsum[wp][0][c0 + l] = gb1;
        s.gsum[wp][1][c0 + l] = gb2;
        s.gsum[wp][2][c0 + l] = gb3;
        s.gsum[wp][3][c0 + l] = gw4;
    }
    if (c == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            loss += __shfl_xor_sync(0xffffffffu, loss, o);
            gb4 += __shfl_xor_sync(0xffffffffu, gb4, o);
        }
        if (l == 0) { s.gone[wp][0] = gb4; s.gone[wp][1] = loss; }
    }
    // ---- block partial gradients ----
    float *G = Gpart + (long long)blockIdx.x * kNParams;
    if (ok) {
        if (wp < 2) { // TMEM lanes 0..63 hold the weight-gradient rows (output features)
            const int o = t;
            float v[16];
            umma::tmem_ld16(lane + kGW2 + c0, v);
            umma::tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; q++) G[kOffW2 + o * 64 + c0 + q] = v[q];
            umma::tmem_ld16(lane + kGW3 + c0, v);
            umma::tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; q++) G[kOffW3 + o * 64 + c0 + q] = v[q];
            if (c == 0) {
                umma::tmem_ld16(lane + kGW1, v);
                umma::tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < 16; q++) G[kOffW1 + o * 16 + q] = (q < 8) ? v[q] : 0.f;
            }
        }
        __syncthreads();
        for (int e = x; e < 4 * 64; e += kTrainThreads) {
            const int which = e >> 6, o = e & 63;
            const int at = which == 0 ? kOffB1 : which == 1 ? kOffB2 : which == 2 ? kOffB3 : kOffW4;
            G[at + o] = s.gsum[0][which][o] + s.gsum[1][which][o] + s.gsum[2][which][o] + s.gsum[3][which][o];
        }
        if (x == 0) {
            G[kOffB4] = s.gone[0][0] + s.gone[1][0] + s.gone[2][0] + s.gone[3][0];
            loss_part[blockIdx.x] = s.gone[0][1] + s.gone[1][1] + s.gone[2][1] + s.gone[3][1];
        }
    } else {
        if (x == 0) atomicExch(err, 1);
        umma::mbar_wait(&s.mbar, phase ^ 1u, kWaitLimit);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (x < 32) umma::tmem_free(tmem, 512);
}

// Deterministic sum of the block partials and an Adam step (FP32 master
// weights), counted in err[1]; no step after a pass that gave up.  The partials are read eight
// at a time (a serial chain of loads per parameter otherwise) and added in
// block order.
__global__ void k_reduce_adam(const float *__restrict__ Gpart, int nblk, float *__restrict__ P,
                              float *__restrict__ Mo, float *__restrict__ Vo, float *__restrict__ Gout, float lr,
                              float b1t, float b2t, int *err)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kNParams || *err) return;
    float g = 0.f;
    for (int b = 0; b < nblk; b += 8) {
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = b + q < nblk ? Gpart[(long long)(b + q) * kNParams + p] : 0.f;
#pragma unroll
        for (int q = 0; q < 8; q++) g += v[q];
    }
    if (Gout) Gout[p] = g;
    if (lr <= 0.f) return;
    if (p == 0) err[1]++;
    const bool padded = (p >= kOffW1 && p < kOffW1 + 64 * 16 && ((p - kOffW1) % 16) >= 8);
    if (padded) return;
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    const float m = beta1 * Mo[p] + (1.f - beta1) * g;
    const float v = beta2 * Vo[p] + (1.f - beta2) * g * g;
    Mo[p] = m;
    Vo[p] = v;
    P[p] -= lr * (m / (1.f - b1t)) / (sqrtf(v / (1.f - b2t)) + eps);
}

} // namespace mlp

// ---- launchers -----------------------------------------------------------------
size_t closure_infer_smem() { return sizeof(mlp::SmemInfer); }
size_t closure_train_smem() { return sizeof(mlp::SmemTrain); }

template <int NP>
static int infer_np(Ctx &c, const double *U, double *mu64, float *mu32, float *cs2_out, const float *P, int *err)
{
    const size_t smem = sizeof(mlp::SmemInfer);
    static std::atomic<uint64_t> attr64{0}, attr32{0};
    if (!smem_limit_once((const void *)mlp::k_closure_infer<double, NP>, smem, attr64) ||
        !smem_limit_once((const void *)mlp::k_closure_infer<float, NP>, smem, attr32))
        return -1;
    // five blocks per SM (45 KB of shared memory and at most 96 registers a
    // thread each, with all of the SM's unified memory as shared memory);
    // four for the wider polynomial splits, whose registers allow four
    static std::atomic<bool> carve{false};
    if (!carve.load()) {
        if (cudaFuncSetAttribute((const void *)mlp::k_closure_infer<float, NP>,
                                 cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
                cudaSuccess ||
            cudaFuncSetAttribute((const void *)mlp::k_closure_infer<double, NP>,
                                 cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
                cudaSuccess)
            return -1;
        carve.store(true);
    }
    const int blocks = c.sms * (NP <= 3 ? 5 : 4);
    prof_begin(c, FSL_K_SGS);
    if (mu32)
        mlp::k_closure_infer<float, NP><<<blocks, 128, smem, c.stream>>>(c.g, c.cls, U, c.cl_vel, P, mu32, cs2_out,
                                                                         err);
    else
        mlp::k_closure_infer<double, NP><<<blocks, 128, smem, c.stream>>>(c.g, c.cls, U, c.cl_vel, P, mu64, cs2_out,
                                                                          err);
    prof_end(c, FSL_K_SGS, 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_closure_infer(Ctx &c, const double *U, double *mu64, float *mu32, float *cs2_out, const float *P, int *err)
{
    if ((long long)c.g.L * c.g.H * c.g.D >= (1LL << 31)) return -1; // feat_load's 32-bit indices
    if (!(c.vel_fresh && U == c.U)) {
        prof_begin(c, FSL_K_SGS);
        mlp::k_closure_vel<<<148 * 8, 256, 0, c.stream>>>(c.g, U, c.cl_vel);
        prof_end(c, FSL_K_SGS, 1);
    }
    switch (c.infer_poly) {
    case 0: return infer_np<0>(c, U, mu64, mu32, cs2_out, P, err);
    case 3: return infer_np<3>(c, U, mu64, mu32, cs2_out, P, err);
    case 4: return infer_np<4>(c, U, mu64, mu32, cs2_out, P, err);
    case 5: return infer_np<5>(c, U, mu64, mu32, cs2_out, P, err);
    case 6: return infer_np<6>(c, U, mu64, mu32, cs2_out, P, err);
    default: return infer_np<2>(c, U, mu64, mu32, cs2_out, P, err);
    }
}

void launch_harvest(Ctx &c, const float *cd, long long stride, long long offset, float *X, float *Y, long long cap,
                    long long base)
{
    prof_begin(c, FSL_K_OTHER);
    mlp::k_harvest<<<148 * 8, 256, 0, c.stream>>>(c.g, c.cls, c.U, cd, stride, offset, X, Y, cap, base);
    prof_end(c, FSL_K_OTHER, 1);
}

int launch_train_grad(cudaStream_t st, const float *X, const float *Y, long long n, int tpb, const float *P,
                      float *Gpart, float *loss_part, int *err, int *nblk_out, float inv_wmean)
{
    const size_t smem = sizeof(mlp::SmemTrain);
    static std::atomic<uint64_t> attr{0};
    if (!smem_limit_once((const void *)mlp::k_train_grad, smem, attr)) return -1;
    const long long ntile = (n + 127) / 128;
    const int nblk = (int)((ntile + tpb - 1) / tpb);
    mlp::k_train_grad<<<nblk, mlp::kTrainThreads, smem, st>>>(X, Y, n, tpb, P, Gpart, loss_part, err, inv_wmean);
    *nblk_out = nblk;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

void launch_reduce_adam(cudaStream_t st, const float *Gpart, int nblk, float *P, float *M, float *V, float *Gout,
                        float lr, float b1t, float b2t, int *err)
{
    mlp::k_reduce_adam<<<(kNParams + 63) / 64, 64, 0, st>>>(Gpart, nblk, P, M, V, Gout, lr, b1t, b2t, err);
}

namespace {
// One 128 x N x K GEMM through the tensor cores (diagnostic of the descriptor
// and TMEM plumbing).  A: 128 x K, B: N x K, row-major FP32 in global memory
// (rounded to BF16 on staging); D: 128 x N FP32.
__global__ void __launch_bounds__(128) k_umma_selftest(const float *__restrict__ A, const float *__restrict__ B,
                                                       float *__restrict__ D, int K, int N, int *err)
{
    __shared__ __align__(1024) __nv_bfloat16 sA[128 * 80];
    __shared__ __align__(1024) __nv_bfloat16 sB[64 * 80];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tholder;
    const int t = threadIdx.x, w = t >> 5;
    for (int k = 0; k < K; k++) sA[umma::tile_off(t, k, K) / 2] = __float2bfloat16_rn(A[t * K + k]);
    if (t < N)
        for (int k = 0; k < K; k++) sB[umma::tile_off(t, k, K) / 2] = __float2bfloat16_rn(B[t * K + k]);
    if (t == 0) umma::mbar_init(&mbar, 1);
    if (w == 0) umma::tmem_alloc(&tholder, 64);
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tholder;
    if (t == 0) {
        umma::gemm_issue(tmem, umma::smem_u32(sA), umma::smem_u32(sB), K, N, false);
        umma::commit(&mbar);
    }
    bool ok = umma::mbar_wait(&mbar, 0, mlp::kWaitLimit);
    ok = __all_sync(0xffffffffu, ok);
    umma::fence_after_sync();
    if (ok) {
        for (int c = 0; c < N / 16; c++) {
            float v[16];
            umma::tmem_ld16(tmem + ((uint32_t)(32 * w) << 16) + (uint32_t)(c * 16), v);
            umma::tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; q++) D[t * N + c * 16 + q] = v[q];
        }
    } else {
        atomicExch(err, 1);
        umma::mbar_wait(&mbar, 0, mlp::kWaitLimit); // let an MMA still in flight finish
    }
    umma::fence_before_sync();
    __syncthreads();
    if (w == 0) umma::tmem_free(tmem, 64);
}
} // namespace

} // namespace fsl

using namespace fsl;

// Diagnostic: D = A B^T for A 128 x K, B N x K (host FP32 arrays, rounded to
// BF16), K in {16, 32, 48, 64}, N in {16, 32, 48, 64}.
extern "C" int fsl_selftest_tensor_gemm(const float *A, const float *B, float *D, int K, int N)
{
    if (!A || !B || !D || K < 16 || K > 80 || (K % 16) || N < 16 || N > 64 || (N % 16)) return FSL_ERR_ARG;
    int dev = 0;
    cudaDeviceProp prop;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaGetDeviceProperties(&prop, dev) != cudaSuccess ||
        prop.major != 10)
        return FSL_ERR_NODEVICE;
    float *dA = nullptr, *dB = nullptr, *dD = nullptr;
    int *dErr = nullptr, herr = 0;
    int rc = FSL_OK;
    if (cudaMalloc((void **)&dA, 128 * K * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void **)&dB, N * K * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void **)&dD, 128 * N * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void **)&dErr, sizeof(int)) != cudaSuccess) {
        rc = FSL_ERR_NOMEM;
    }
    if (!rc) {
        cudaMemcpy(dA, A, 128 * K * sizeof(float), cudaMemcpyHostToDevice);
        cudaMemcpy(dB, B, N * K * sizeof(float), cudaMemcpyHostToDevice);
        cudaMemset(dErr, 0, sizeof(int));
        k_umma_selftest<<<1, 128>>>(dA, dB, dD, K, N, dErr);
        if (cudaDeviceSynchronize() != cudaSuccess) rc = FSL_ERR_CUDA;
        else {
            cudaMemcpy(D, dD, 128 * N * sizeof(float), cudaMemcpyDeviceToHost);
            cudaMemcpy(&herr, dErr, sizeof(int), cudaMemcpyDeviceToHost);
            if (herr) rc = FSL_ERR_TIMEOUT;
        }
    }
    cudaFree(dA); cudaFree(dB); cudaFree(dD); cudaFree(dErr);
    return rc;
}
