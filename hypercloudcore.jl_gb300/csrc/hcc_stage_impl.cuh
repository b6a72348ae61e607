// hcc_stage_impl.cuh — the per-stage kernels, templated on the arithmetic type T (double: plain FP64 path,
// float: FP32 bulk path), the dimension D, the number of state components M, the physics module PDE and the
// reconstruction degree RDEG. Included per precision, degree and physics by hcc_stage_f{64,32}_r{1,2}[_linear].cu (the
// Euler modules and the linear ones compile side by side).
//
// Thread per particle over slot-major neighbour arrays: the 32 threads of a warp read slot k of 32 consecutive
// particles from consecutive addresses; neighbour states, gradients and orders are gathered through L1/L2
// (the Morton numbering keeps a warp's stencils overlapping).
#pragma once
#include <algorithm>

#include "hcc_internal.cuh"

// Launch shape of the flux pass (threads per block, minimum resident blocks per SM for the register budget): the
// HCC_FLUX_* constants of hcc_internal.cuh.

namespace hcc {

// ----------------------------------------------------------------------------------- physics (device)
template <typename T> struct Accum;    // FP32: Kahan-compensated sums; FP64: plain sums
template <> struct Accum<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double x) { s = s + x; }
    __device__ __forceinline__ double value() const { return s; }
};
template <> struct Accum<float> {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x) {
        float y = x - c;
        float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ float value() const { return s; }
};

// FP32 component vectors in pairs: the packed FP32x2 instructions of sm_100+ (per component identical to the scalar
// operations; a - b as fma(b, -1, a) is the same rounding of the same exact value). HCC_FP32_PACKED=0 builds the
// same arithmetic from scalar instructions (identical results; which form runs faster is measured).
#if HCC_FP32_PACKED
__device__ __forceinline__ float2 p_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 p_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 p_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 p_sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
#else
__device__ __forceinline__ float2 p_add(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
__device__ __forceinline__ float2 p_mul(float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
__device__ __forceinline__ float2 p_fma(float2 a, float2 b, float2 c) {
    return make_float2(__fmaf_rn(a.x, b.x, c.x), __fmaf_rn(a.y, b.y, c.y));
}
__device__ __forceinline__ float2 p_sub(float2 a, float2 b) { return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y)); }
#endif
__device__ __forceinline__ float2 p_bc(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 p_ld(const float *x, int q) { return make_float2(x[2 * q], x[2 * q + 1]); }
__device__ __forceinline__ void p_st(float *x, int q, float2 v) { x[2 * q] = v.x; x[2 * q + 1] = v.y; }

// Per-component sums of the flux pass: FP64 plain; FP32 Kahan-compensated, in pairs (scalar tail for odd M).
template <typename T, int M> struct AccumV {
    T s[M];
    __device__ __forceinline__ AccumV() {
#pragma unroll
        for (int m = 0; m < M; ++m) s[m] = T(0);
    }
    __device__ __forceinline__ void add(const T *t) {
#pragma unroll
        for (int m = 0; m < M; ++m) s[m] = s[m] + t[m];
    }
};
template <int M> struct AccumV<float, M> {
    float s[M], c[M];
    __device__ __forceinline__ AccumV() {
#pragma unroll
        for (int m = 0; m < M; ++m) { s[m] = 0.0f; c[m] = 0.0f; }
    }
    __device__ __forceinline__ void add(const float *t) {
#pragma unroll
        for (int q = 0; q < M / 2; ++q) {
            const float2 y = p_sub(p_ld(t, q), p_ld(c, q));
            const float2 u = p_add(p_ld(s, q), y);
            p_st(c, q, p_sub(p_sub(u, p_ld(s, q)), y));
            p_st(s, q, u);
        }
        if constexpr (M & 1) {
            const float y = t[M - 1] - c[M - 1];
            const float u = s[M - 1] + y;
            c[M - 1] = (u - s[M - 1]) - y;
            s[M - 1] = u;
        }
    }
};

// Compensated sums of the tile-staged flux pass in blocks: NB slot terms summed plainly, then the block's sum added
// with compensation (NB = 1: every term compensated, as AccumV). `flush` adds a partial block; `sum` then holds
// the compensated sums.
template <int M, int NB> struct BlockAccum {
    AccumV<float, M> sum;
    float p[M];
    int n;
    __device__ __forceinline__ BlockAccum() : n(0) {
#pragma unroll
        for (int m = 0; m < M; ++m) p[m] = 0.0f;
    }
    __device__ __forceinline__ void add(const float *t) {
        if constexpr (NB == 1) {
            sum.add(t);
        } else {
#pragma unroll
            for (int m = 0; m < M; ++m) p[m] = p[m] + t[m];
            if (++n == NB) flush();
        }
    }
    __device__ __forceinline__ void flush() {
        if constexpr (NB > 1) {
            if (n > 0) {
                sum.add(p);
#pragma unroll
                for (int m = 0; m < M; ++m) p[m] = 0.0f;
                n = 0;
            }
        }
    }
};

template <typename T> __device__ __forceinline__ T floatmin_of();
template <> __device__ __forceinline__ double floatmin_of<double>() { return 2.2250738585072014e-308; }
template <> __device__ __forceinline__ float floatmin_of<float>() { return 1.17549435e-38f; }

// Arithmetic kernels of the two paths. FP64 (plain path): IEEE division and square root — the oracle's exact
// sequence. FP32 (bulk path, compiled with denormals flushed to zero): the reciprocal of the special-function unit (1 ulp)
// and x rsqrt(x) (0 at 0, NaN below). sqrt.approx has the smaller error of one root (0.24 against 0.36 units of 2^-23
// rms) but twice the bias (-0.093 against -0.041), which the sums over the slots keep: 1.6 % more error of the
// right-hand side on 12^3 points, 0.1 % on 70^2, and no time gained (3-D Euler, 343k points: 1528 us a step against
// 1544). The results are compared
// with the FP64 oracle to tolerance. Both keep Julia's NaN-propagating min/max:
// a reconstruction with negative pressure has a NaN sound speed, and the NaN must reach the candidate so that the
// admissibility check flags it (fmaxf would drop it and keep the high order).
template <typename T> __device__ __forceinline__ T recip(T x) { return T(1) / x; }
template <> __device__ __forceinline__ float recip<float>(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
template <typename T> __device__ __forceinline__ T root(T x) { return sqrt(x); }
template <> __device__ __forceinline__ float root<float>(float x) {
    return x == 0.0f ? 0.0f : x * rsqrtf(x);
}
template <typename T> __device__ __forceinline__ T vmin(T x, T y) { return jmin(x, y); }
template <typename T> __device__ __forceinline__ T vmax(T x, T y) { return jmax(x, y); }
// FP32: the NaN-propagating forms of the min/max instructions (one instruction each)
template <> __device__ __forceinline__ float vmin<float>(float x, float y) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
    return r;
}
template <> __device__ __forceinline__ float vmax<float>(float x, float y) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
    return r;
}

// Load N contiguous elements with 16-byte vectors (8-byte for two floats) where the layout guarantees the alignment
// (particle-major arrays of N elements a row from a 256-byte-aligned base).
template <typename T, int N>
__device__ __forceinline__ void load_vec(const T *__restrict__ p, T *out) {
    if constexpr (sizeof(T) == 4 && N % 4 == 0) {
#pragma unroll
        for (int q = 0; q < N / 4; ++q) {
            float4 v = reinterpret_cast<const float4 *>(p)[q];
            out[4 * q] = v.x; out[4 * q + 1] = v.y; out[4 * q + 2] = v.z; out[4 * q + 3] = v.w;
        }
    } else if constexpr (sizeof(T) == 4 && N == 2) {
        float2 v = *reinterpret_cast<const float2 *>(p);
        out[0] = v.x; out[1] = v.y;
    } else if constexpr (sizeof(T) == 8 && N % 2 == 0) {
#pragma unroll
        for (int q = 0; q < N / 2; ++q) {
            double2 v = reinterpret_cast<const double2 *>(p)[q];
            out[2 * q] = v.x; out[2 * q + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int q = 0; q < N; ++q) out[q] = p[q];
    }
}

// Store N contiguous elements with 16-byte vectors under the same alignment guarantee.
template <typename T, int N>
__device__ __forceinline__ void store_vec(T *__restrict__ p, const T *v) {
    if constexpr (sizeof(T) == 4 && N % 4 == 0) {
#pragma unroll
        for (int q = 0; q < N / 4; ++q)
            reinterpret_cast<float4 *>(p)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    } else if constexpr (sizeof(T) == 4 && N == 2) {
        *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
    } else if constexpr (sizeof(T) == 8 && N % 2 == 0) {
#pragma unroll
        for (int q = 0; q < N / 2; ++q) reinterpret_cast<double2 *>(p)[q] = make_double2(v[2 * q], v[2 * q + 1]);
    } else {
#pragma unroll
        for (int q = 0; q < N; ++q) p[q] = v[q];
    }
}

// a + f x with f a power of two (or zero) and sign: FP64 as one fused multiply-add, which rounds the same sum of the
// same exact product as a multiply and an add (f x is exact), in one FP64 instruction instead of two.
template <typename T> __device__ __forceinline__ T add_scaled(T a, T f, T x) { return a + f * x; }
template <> __device__ __forceinline__ double add_scaled<double>(double a, double f, double x) { return __fma_rn(f, x, a); }
// x > 0 without the FP64 unit (NaN: false)
template <typename T> __device__ __forceinline__ bool positive(T x) { return x > T(0); }
template <> __device__ __forceinline__ bool positive<double>(double x) {
    return (unsigned long long)(__double_as_longlong(x) - 1) < 0x7ff0000000000000ull;
}
// |a| >= |b| and neither a NaN; FP64 as integers (magnitudes order like their words, a NaN's above infinity's).
template <typename T> __device__ __forceinline__ bool covers(T a, T b) { return fabs(a) >= fabs(b); }
template <> __device__ __forceinline__ bool covers<double>(double a, double b) {
    const unsigned long long m = 0x7fffffffffffffffull, inf = 0x7ff0000000000000ull;
    const unsigned long long wa = __double_as_longlong(a) & m, wb = __double_as_longlong(b) & m;
    return wa >= wb && wa <= inf;
}
// x or -x by the sign bit
__device__ __forceinline__ double negate_if(double x, bool neg) {
    return __longlong_as_double(__double_as_longlong(x) ^ (neg ? (long long)0x8000000000000000ull : 0ll));
}

// Elements of a particle's gradient row for N slope components: rows of 12 or more that are not whole 16-byte groups
// (3-D Euler: 15) are padded to them, so that a neighbour's row comes in 16-byte loads (four instead of fifteen).
// hcc_internal.cuh's grad_row_elements is the host's form.
template <typename T, int N> constexpr int grad_row() { return grad_row_elements(N, int(sizeof(T))); }
// N elements of a 16-byte-aligned row of S >= N elements (S a multiple of the group, or S = N).
template <typename T, int N, int S> __device__ __forceinline__ void load_row(const T *__restrict__ p, T *out) {
    if constexpr (S == N) {
        load_vec<T, N>(p, out);
    } else {
        T v[S];
        load_vec<T, S>(p, v);
#pragma unroll
        for (int q = 0; q < N; ++q) out[q] = v[q];
    }
}
template <typename T, int N, int S> __device__ __forceinline__ void store_row(T *__restrict__ p, const T *v) {
    if constexpr (S == N) {
        store_vec<T, N>(p, v);
    } else {
        T w[S];
#pragma unroll
        for (int q = 0; q < S; ++q) w[q] = q < N ? v[q < N ? q : 0] : T(0);
        store_vec<T, S>(p, w);
    }
}

// Euler primitives: inv_rho = 1/rho, u_d = m_d inv_rho, p = (gamma-1)(E - 0.5 (rho |u|^2)), c = sqrt(gamma p inv_rho).
template <typename T, int D>
__device__ __forceinline__ T euler_internal(const T *U, T &inv_rho, T *u) {
    T rho = U[0];
    inv_rho = recip(rho);
    T q2 = T(0);
#pragma unroll
    for (int d = 0; d < D; ++d) {
        u[d] = U[1 + d] * inv_rho;
        q2 = (d == 0) ? u[d] * u[d] : q2 + u[d] * u[d];
    }
    return add_scaled<T>(U[D + 1], T(-0.5), rho * q2);
}
template <typename T, int D>
__device__ __forceinline__ void euler_prim(const PhysParams<T> &ph, const T *U, T &inv_rho, T *u, T &p) {
    p = ph.gm1 * euler_internal<T, D>(U, inv_rho, u);
}

// flux(eq, U) (API.jl:23) for the compiled-in modules; lam[d] = max_eigenvalue(eq, U, d) (API.jl:38).
// On a moving grid (w != nullptr) the flux and speeds of ALEFrame(eq, w) (GridMovers.jl:77-83): F_d - w_d U and
// max_eigenvalue(eq, U, d, w_d) (API.jl:51-58): |u_d - w_d| + c (Euler), |c_d - w_d| (scalar advection,
// test/PDEs/linear_advection.jl:35), else max_eigenvalue + |w_d|.
template <typename T, int D, int M, int PDE>
__device__ __forceinline__ void flux_and_speed(const PhysParams<T> &ph, const T *U, T (*F)[M], T *lam,
                                               const T *w = nullptr) {
    if constexpr (PDE == HCC_PDE_EULER) {
        T inv_rho, u[D], p;
        euler_prim<T, D>(ph, U, inv_rho, u, p);
        T c = root(ph.gamma * p * inv_rho);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            F[d][0] = U[1 + d];
#pragma unroll
            for (int e = 0; e < D; ++e) {
                T v = U[1 + e] * u[d];
                F[d][1 + e] = (e == d) ? v + p : v;
            }
            F[d][D + 1] = (U[D + 1] + p) * u[d];
            lam[d] = fabs(w ? u[d] - w[d] : u[d]) + c;
        }
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d) {
#pragma unroll
            for (int m = 0; m < M; ++m) F[d][m] = ph.c[d][m] * U[m];
            lam[d] = !w ? ph.amax[d]
                        : ((PDE == HCC_PDE_ADVECTION && M == 1) ? fabs(ph.c[d][0] - w[d]) : ph.amax[d] + fabs(w[d]));
        }
    }
    if (w) {
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
            for (int m = 0; m < M; ++m) F[d][m] = F[d][m] - w[d] * U[m];
    }
}

// FP32 Euler on a fixed grid, the flux contracted with a weight vector w: Fw(U) = sum_d w_d F_d(U) =
// (m.w, (u.w) m + p w, (E + p)(u.w)), and the axis speeds |u_d| + c of flux_and_speed. One contracted flux
// replaces the D axis fluxes and their contraction in the flux pass (the Rusanov flux is linear in the F_d).
template <int D>
__device__ __forceinline__ void euler_projected(const PhysParams<float> &ph, const float *U, const float *w,
                                                float *Fn, float *lam) {
    float inv_rho, u[D], p;
    euler_prim<float, D>(ph, U, inv_rho, u, p);
    const float c = root(ph.gamma * p * inv_rho);
    float un = u[0] * w[0], mw = U[1] * w[0];
#pragma unroll
    for (int d = 1; d < D; ++d) { un = un + u[d] * w[d]; mw = mw + U[1 + d] * w[d]; }
    Fn[0] = mw;
#pragma unroll
    for (int e = 0; e < D; ++e) Fn[1 + e] = un * U[1 + e] + p * w[e];
    Fn[D + 1] = (U[D + 1] + p) * un;
#pragma unroll
    for (int d = 0; d < D; ++d) lam[d] = fabsf(u[d]) + c;
}

// Whether the flux pass takes the contracted Euler form (FP32, fixed grid, no moment correction).
template <typename T, int PDE, bool ALE, bool MOM> constexpr bool projected_flux() {
    return sizeof(T) == 4 && PDE == HCC_PDE_EULER && !ALE && !MOM;
}

// The own flux a flux pass keeps for particle i: F(f_i) per axis (FP64), doubled (FP32, the scaled Rusanov form),
// or for the contracted Euler form the constants 2 Fw(f_i) is formed from in every slot, in the first row:
// (2u, 2p, E + p).
template <typename T, int D, int M, int PDE, bool ALE, bool MOM>
__device__ __forceinline__ void own_flux(const PhysParams<T> &ph, const T *fi, T (*Fi)[M], const T *wp) {
    if constexpr (projected_flux<T, PDE, ALE, MOM>()) {
        T inv_rho, u[D], p;
        euler_prim<T, D>(ph, fi, inv_rho, u, p);
#pragma unroll
        for (int d = 0; d < D; ++d) Fi[0][d] = T(2) * u[d];
        Fi[0][D] = T(2) * p;
        Fi[0][D + 1] = fi[D + 1] + p;
    } else {
        T lam[D];
        flux_and_speed<T, D, M, PDE>(ph, fi, Fi, lam, wp);
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int d = 0; d < D; ++d)
#pragma unroll
                for (int m = 0; m < M; ++m) Fi[d][m] = T(2) * Fi[d][m];
        }
    }
}

// grid_velocity (GridMovers.jl:60-63) of particle i: fluid velocity (Euler m_d / rho, scalar advection c_d), scaled,
// or the prescribed field velocity + omega x (x - center) at its current position
template <typename T, int D, int M, int PDE>
__device__ __forceinline__ void grid_velocity(const StageArgs<T> &a, int64_t i, const T *U, T *w) {
    if (a.mover == HCC_MOVER_PRESCRIBED) {
        double r[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int d = 0; d < D; ++d) r[d] = a.pos[int64_t(d) * a.g.npad + i] - a.mv_c[d];
        if constexpr (D == 1) {
            w[0] = T(a.mv_v[0]);
        } else if constexpr (D == 2) {
            w[0] = T(a.mv_v[0] - a.mv_om[2] * r[1]);
            w[1] = T(a.mv_v[1] + a.mv_om[2] * r[0]);
        } else {
            w[0] = T(a.mv_v[0] + (a.mv_om[1] * r[2] - a.mv_om[2] * r[1]));
            w[1] = T(a.mv_v[1] + (a.mv_om[2] * r[0] - a.mv_om[0] * r[2]));
            w[2] = T(a.mv_v[2] + (a.mv_om[0] * r[1] - a.mv_om[1] * r[0]));
        }
        return;
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
        if constexpr (PDE == HCC_PDE_EULER) w[d] = U[1 + d] / U[0];
        else w[d] = a.ph.c[d][0];
        if (a.mover == HCC_MOVER_SCALED) w[d] = a.mv_alpha * w[d];
    }
}

// The axis speeds of the CFL step. FP32: correctly rounded reciprocal and root, once a particle or union entry; the own
// speed is in most of a particle's terms, so its error is the step's.
template <typename T, int D, int M, int PDE>
__device__ __forceinline__ void speeds(const PhysParams<T> &ph, const T *U, T *lam) {
    if constexpr (PDE == HCC_PDE_EULER) {
        T inv_rho, u[D], c;
        if constexpr (sizeof(T) == 4) {
            inv_rho = __frcp_rn(U[0]);
            T q2 = T(0);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                u[d] = U[1 + d] * inv_rho;
                q2 = q2 + U[1 + d] * u[d];
            }
            c = __fsqrt_rn(ph.gamma * ph.gm1 * (U[D + 1] - T(0.5) * q2) * inv_rho);
        } else {
            T p;
            euler_prim<T, D>(ph, U, inv_rho, u, p);
            c = root(ph.gamma * p * inv_rho);
        }
#pragma unroll
        for (int d = 0; d < D; ++d) lam[d] = fabs(u[d]) + c;
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d) lam[d] = ph.amax[d];
    }
}

// is_admissible (API.jl:48): finite; Euler also rho > 0 and p > 0.
template <typename T, int D, int M, int PDE>
__device__ __forceinline__ bool admissible(const PhysParams<T> &ph, const T *U) {
    bool ok = true;
#pragma unroll
    for (int m = 0; m < M; ++m) ok = ok && isfinite(U[m]);
    if constexpr (PDE == HCC_PDE_EULER) {
        if (!ok) return false;
        T inv_rho, u[D], p;
        euler_prim<T, D>(ph, U, inv_rho, u, p);
        return U[0] > T(0) && p > T(0);
    }
    return ok;
}

// BGK Maxwellian of the single macro moment (evaluate_source / implicit_solve, test/kinetic_source.jl:67-104).
template <typename T, int D, int M>
__device__ __forceinline__ void maxwellian(const PhysParams<T> &ph, const T *U, T *Mk) {
    T u = U[0];
#pragma unroll
    for (int k = 1; k < M; ++k) u = u + U[k];
    T F[D];
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] = ph.a_macro[d] * u;
#pragma unroll
    for (int k = 0; k < M; ++k) {
        T fd = F[0] * ph.sinv[k][0];
#pragma unroll
        for (int d = 1; d < D; ++d) fd = fd + F[d] * ph.sinv[k][d];
        Mk[k] = ph.coeff * (u + fd);
    }
}

// Implicit part of a stage (TimeSteppers.jl:427-444): mode 1 solves U_out - dt a_ii S(U_out) = U_in and sets
// K_I = (U_out - U_in) / (dt a_ii); mode 2 evaluates K_I = S(Y) explicitly.
template <typename T, int D, int M, int PDE>
__device__ __forceinline__ void implicit_part(const StageArgs<T> &a, int64_t i, T *Y, T *KIout) {
    if constexpr (PDE == HCC_PDE_BGK) {
        T Mk[M];
        maxwellian<T, D, M>(a.ph, Y, Mk);
        if (a.implicit_mode == 1) {
            const StageCoeffs<T> *cf = coef_of(a, i);
            T dto = cf->dt_ii * a.ph.inv_eps;
            T denom = T(1) / (T(1) + dto);
            const T inv_dt_ii = cf->inv_dt_ii;
#pragma unroll
            for (int k = 0; k < M; ++k) {
                T out = (Y[k] + dto * Mk[k]) * denom;
                KIout[k] = (out - Y[k]) * inv_dt_ii;
                Y[k] = out;
            }
        } else {
#pragma unroll
            for (int k = 0; k < M; ++k) KIout[k] = (Mk[k] - Y[k]) * a.ph.inv_eps;
        }
    } else {
#pragma unroll
        for (int k = 0; k < M; ++k) KIout[k] = T(0);
    }
}

// ----------------------------------------------------------------------------------- slope limiters
// limiter_phi (Limiter.jl:35-46): Barth-Jespersen min(1, r); Venkatakrishnan (r² + 2r)/(r² + r + 2), for r > 1 in
// s = 1/r.
template <typename T>
__device__ __forceinline__ T limiter_phi(int lim, T r) {
    if (lim == HCC_LIMITER_BJ_SOFT || lim == HCC_LIMITER_BJ_HARD) return vmin(T(1), r);
    const T rp = vmax(T(0), r);
    if (rp > T(1)) {
        const T sv = T(1) / rp;
        return (T(1) + T(2) * sv) / (T(1) + sv + T(2) * (sv * sv));
    }
    return (rp * rp + T(2) * rp) / (rp * rp + rp + T(2));
}

// Positive numbers from 2^-900 (FP32: 2^-90) up, no NaN nor infinity; x < y of such (FP64 as integers).
__device__ __forceinline__ bool in_range(double x) {
    const unsigned hi = unsigned(__double2hiint(x));
    return hi >= ((1023u - 900u) << 20) && hi < 0x7ff00000u;
}
__device__ __forceinline__ bool in_range(float x) { return x >= 8.0779357e-28f && x <= 3.0e38f; }
__device__ __forceinline__ bool below(double x, double y) { return __double_as_longlong(x) < __double_as_longlong(y); }
__device__ __forceinline__ bool below(float x, float y) { return x < y; }

// Venkatakrishnan's coefficient over the slots: phi grows with r = room / recon up to r = 4.8, so the least r gives the
// least phi, and the quotients are compared by their cross products (two multiplications where the quotient and phi take
// three divisions, which a warp executes as soon as one of its lanes has such a slot). Ratios too close for the rounded
// phi to follow their order (1e-13, FP32 1e-5; its rounding is some 1e-15 and its slope at least a quarter), and products
// out of range, are evaluated one by one, so the minimum keeps its bits.
template <typename T> struct LeastRatio {
    T room, recon;                                // of the least ratio so far; recon 0: none
    __device__ __forceinline__ LeastRatio() : room(T(0)), recon(T(0)) {}
    __device__ __forceinline__ void add(int lim, T rm, T rc, T &phi) {       // magnitudes; rc > 0
        constexpr T near = T(1) - (sizeof(T) == 8 ? T(1e-13) : T(1e-5));
        if (rm == T(0)) { phi = T(0); return; }   // (phi(0) = 0, no other is less)
        if (recon == T(0)) { room = rm; recon = rc; return; }
        const T a = rm * recon, b = room * rc;
        if (in_range(a) && in_range(b)) {
            if (below(a, b * near)) { room = rm; recon = rc; return; }
            if (below(b, a * near)) return;
        }
        if (rm == room && rc == recon) return;
        phi = vmin(phi, limiter_phi<T>(lim, rm / rc));
    }
    __device__ __forceinline__ void finish(int lim, T &phi) const {
        if (recon != T(0)) phi = vmin(phi, limiter_phi<T>(lim, room / recon));
    }
};

template <typename T> __device__ __forceinline__ T eps16();
template <> __device__ __forceinline__ double eps16<double>() { return 16.0 * 2.220446049250313e-16; }
template <> __device__ __forceinline__ float eps16<float>() { return 16.0f * 1.1920929e-7f; }

// Local extrema over {i} u N(i) (_local_extrema, Limiter.jl:61-69), one neighbour at a time.
template <typename T, int M> __device__ __forceinline__ void extend_extrema(const T *f, T *umin, T *umax) {
#pragma unroll
    for (int m = 0; m < M; ++m) { umax[m] = vmax(umax[m], f[m]); umin[m] = vmin(umin[m], f[m]); }
}

// _limit_slopes for BJ / VK (Limiter.jl:120-143): with the local extrema of the reconstruction's own neighbour loop, the
// bounding coefficient over the interface reconstructions (_bounding_phi / _update_phi, :76-100), then the
// gradient terms (hard: every term; soft: the first-degree ones) scaled by it. The coefficient only falls below 1
// where the distance to the bound is under twice the reconstructed step (Venkatakrishnan; (r^2 + 2r) >= (r^2 + r + 2)
// from r = 2 on, computed as 1 or more) or under the step (Barth-Jespersen), so the divisions of the other slots, most
// of them in a resolved field, are left out.
template <typename T, int D, int M, int RDEG>
__device__ __forceinline__ void limit_slopes(const StageArgs<T> &a, int64_t i, int cnt, const T *fi, const T *umin,
                                             const T *umax, T (*out)[M]) {
    constexpr int BR = RBasis<D, RDEG>::B;
    const int64_t np = a.g.npad;
    T phi[M];
#pragma unroll
    for (int m = 0; m < M; ++m) phi[m] = T(1);
    const T tol16 = eps16<T>();
    const bool bj = a.sc.limiter == HCC_LIMITER_BJ_SOFT || a.sc.limiter == HCC_LIMITER_BJ_HARD;
    const T reach = bj ? T(1) : T(2.01);
    // out.p(dk / 2) with the halves and quarters in the coefficients (powers of two: the same bits), the distances to the
    // bounds formed once and the reach compared as integers: 17 -> 13 FP64 instructions a slot and variable
    LeastRatio<T> least[M];
    T half[BR][M], up[M], down[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        up[m] = umax[m] - fi[m];
        down[m] = umin[m] - fi[m];
#pragma unroll
        for (int b = 0; b < BR; ++b) half[b][m] = out[b][m] * (b < D ? T(0.5) : T(0.25));
    }
#pragma unroll 2
    for (int k = 0; k < cnt; ++k) {
        T x[D], p[BR];
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = a.g.dist[(int64_t(k) * D + d) * np + i];
        recon_basis<D, RDEG, T>(x, p);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            T recon = half[0][m] * p[0];
#pragma unroll
            for (int b = 1; b < BR; ++b) recon = recon + half[b][m] * p[b];
            const bool pos = positive(recon);
            const T room = pos ? up[m] : down[m], bound = pos ? umax[m] : umin[m];
            if (covers(room, reach * recon)) continue;            // (a NaN goes on)
            const T tol = tol16 * vmax(fabs(fi[m]), fabs(bound));
            if (!(fabs(recon) > tol)) continue;
            // (room and recon have the same sign: the ratio is that of their magnitudes)
            if (bj) phi[m] = vmin(phi[m], limiter_phi<T>(a.sc.limiter, room / recon));
            else least[m].add(a.sc.limiter, fabs(room), fabs(recon), phi[m]);
        }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) least[m].finish(a.sc.limiter, phi[m]);
    const bool hard = a.sc.limiter == HCC_LIMITER_BJ_HARD || a.sc.limiter == HCC_LIMITER_VK_HARD;
#pragma unroll
    for (int b = 0; b < BR; ++b)
        if (hard || b < D) {
#pragma unroll
            for (int m = 0; m < M; ++m) out[b][m] = out[b][m] * phi[m];
        }
}

// The particle of entry q of a full pass, or -1 past its end.
template <typename T> __device__ __forceinline__ int64_t full_particle(const StageArgs<T> &a, int64_t q) {
    return q >= a.nfull ? -1 : (a.ilist ? int64_t(a.ilist[q]) : q);
}

// ----------------------------------------------------------------------------------- gather pass
// update_content! of MUSCL (MUSCL.jl:351-384) with NoLimiter: starved-order lowering, cached full-order fit
// (apply_weights, Interpolators.jl:585-602), dynamic lower-degree fit, or zero (order 1).
// LIM: a slope limiter is on (its extrema are kept in the neighbour loop; without it they cost no registers).
template <typename T, int D, int M, int PDE, int RDEG, bool LIM>
__device__ __forceinline__ void gather_one(const StageArgs<T> &a, const int64_t i) {
    constexpr int BR = RBasis<D, RDEG>::B;
    if (a.g.bnd[i]) return;
    const int cnt = a.g.cnt[i];
    const int64_t np = a.g.npad;
    int p = a.orders[i];
    const int p0 = p;
    while (p > 1 && cnt < basis_count(D, p - 1)) --p;
    if (p < p0) a.orders[i] = int8_t(p);
    T *g = a.grad + i * grad_row<T, BR * M>();
    T fi[M];
#pragma unroll
    for (int m = 0; m < M; ++m) fi[m] = a.U[i * M + m];
    T out[BR][M];
#pragma unroll
    for (int b = 0; b < BR; ++b)
#pragma unroll
        for (int m = 0; m < M; ++m) out[b][m] = T(0);
    const T invL = a.g.invL;
    bool done = false;
    const bool lim = LIM && p > 1;
    T umin[M], umax[M];                               // of the neighbour loop below (limiter only)
#pragma unroll
    for (int m = 0; m < M; ++m) umin[m] = umax[m] = fi[m];
    if constexpr (sizeof(T) == 4 && RDEG == 1) {
        // FP32, degree 1: the cached fit as one weight vector per slot (nidx + D floats per slot)
        if (p == a.sc.max_order && p > 1 && a.g.ok_r[i] && a.g.gw) {
            // slots in groups of G: the states of a group, and the indices and weights of the next, are in flight
            // while the group is summed (an index is what its state's load waits for). Two with the extrema of a limited
            // pair of variables: four of them spill within the bound of gather_min_blocks (449 us a step, 428 with two).
            constexpr int G = LIM && M == 2 ? 2 : 4;
            int32_t j[G];
            T gk[G][D];
            auto stream = [&](int k, int32_t *jk, T(*g)[D]) {
#pragma unroll
                for (int q = 0; q < G; ++q) {
                    const bool on = k + q < cnt;
                    jk[q] = on ? a.g.nidx[int64_t(k + q) * np + i] : int32_t(i);
#pragma unroll
                    for (int d = 0; d < D; ++d) g[q][d] = on ? a.g.gw[(int64_t(k + q) * D + d) * np + i] : T(0);
                }
            };
            stream(0, j, gk);
            for (int k = 0; k < cnt; k += G) {
                T df[G][M], gn[G][D];
                int32_t jn[G];
#pragma unroll
                for (int q = 0; q < G; ++q) load_vec<T, M>(a.U + int64_t(j[q]) * M, df[q]);
                stream(k + G, jn, gn);
#pragma unroll
                for (int q = 0; q < G; ++q) {
                    if (k + q < cnt) {
                        if (lim) extend_extrema<T, M>(df[q], umin, umax);
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            const T dm = df[q][m] - fi[m];
#pragma unroll
                            for (int b = 0; b < BR; ++b) out[b][m] = out[b][m] + gk[q][b] * dm;
                        }
                    }
                    j[q] = jn[q];
#pragma unroll
                    for (int d = 0; d < D; ++d) gk[q][d] = gn[q][d];
                }
            }
            done = true;
        }
    }
    if (done) {
    } else if (p == a.sc.max_order && p > 1 && a.g.ok_r[i]) {
        T bs[BR][M];
#pragma unroll
        for (int b = 0; b < BR; ++b)
#pragma unroll
            for (int m = 0; m < M; ++m) bs[b][m] = T(0);
        // slots in groups, as above: one at a time for several variables, two for a 3-D scalar (registers; four of them in
        // 3-D: 1979 us a step with limiter, two 1762)
        constexpr int G = M == 1 ? (D == 3 ? 2 : 4) : 1;
        int32_t j[G];
        T dk[G][D], wk[G];
        auto stream = [&](int k, int32_t *jk, T(*d)[D], T *w) {
#pragma unroll
            for (int q = 0; q < G; ++q) {
                const bool on = k + q < cnt;
                const int64_t s1 = int64_t(k + q) * np + i;
                jk[q] = on ? a.g.nidx[s1] : int32_t(i);
                w[q] = on ? a.g.wt[s1] : T(0);
#pragma unroll
                for (int e = 0; e < D; ++e) d[q][e] = on ? a.g.dist[(int64_t(k + q) * D + e) * np + i] : T(0);
            }
        };
        stream(0, j, dk, wk);
        for (int k = 0; k < cnt; k += G) {
            T df[G][M], x[G][D], w[G];
#pragma unroll
            for (int q = 0; q < G; ++q) {
                load_vec<T, M>(a.U + int64_t(j[q]) * M, df[q]);
                w[q] = wk[q];
#pragma unroll
                for (int d = 0; d < D; ++d) x[q][d] = dk[q][d] * invL;
            }
            stream(k + G, j, dk, wk);
#pragma unroll
            for (int q = 0; q < G; ++q) {
                if (k + q >= cnt) break;
                T pb[BR];
                recon_basis<D, RDEG, T>(x[q], pb);
                if (lim) extend_extrema<T, M>(df[q], umin, umax);
#pragma unroll
                for (int m = 0; m < M; ++m) df[q][m] = df[q][m] - fi[m];
#pragma unroll
                for (int b = 0; b < BR; ++b)
#pragma unroll
                    for (int m = 0; m < M; ++m) bs[b][m] = bs[b][m] + w[q] * (pb[b] * df[q][m]);
            }
        }
        const T *inv = a.g.inv_r + i * (BR * BR);
        T invm[BR][BR];
#pragma unroll
        for (int b = 0; b < BR; ++b)
#pragma unroll
            for (int c = 0; c < BR; ++c) invm[b][c] = inv[b * BR + c];
#pragma unroll
        for (int b = 0; b < BR; ++b) {
            const T sc = recon_scale<D, RDEG, T>(b, invL);
#pragma unroll
            for (int m = 0; m < M; ++m) {
                T acc = invm[b][0] * bs[0][m];
#pragma unroll
                for (int c = 1; c < BR; ++c) acc = acc + invm[b][c] * bs[c][m];
                out[b][m] = acc * sc;
            }
        }
    } else if (p > 1 && p - 1 < RDEG) {
        // Interpolator{D, 1, 1} (_mls_solve, Interpolators.jl:372-400): moment matrix and Cholesky in FP64
        constexpr int B1 = D;
        double N[B1 * B1];
        T bs[B1][M];
#pragma unroll
        for (int q = 0; q < B1 * B1; ++q) N[q] = 0.0;
#pragma unroll
        for (int b = 0; b < B1; ++b)
#pragma unroll
            for (int m = 0; m < M; ++m) bs[b][m] = T(0);
        const double invLd = double(invL);
        for (int k = 0; k < cnt; ++k) {
            const int64_t s = int64_t(k) * np + i;
            const int32_t j = a.g.nidx[s];
            double xd[D];
            T xt[D];
#pragma unroll
            for (int d = 0; d < D; ++d) {
                T dk = a.g.dist[(int64_t(k) * D + d) * np + i];
                xd[d] = double(dk) * invLd;
                xt[d] = dk * invL;
            }
            const T w = a.g.wt[s];
            const double wd = double(w);
#pragma unroll
            for (int r = 0; r < B1; ++r)
#pragma unroll
                for (int c = 0; c < B1; ++c) N[r * B1 + c] = N[r * B1 + c] + wd * (xd[r] * xd[c]);
#pragma unroll
            for (int b = 0; b < B1; ++b)
#pragma unroll
                for (int m = 0; m < M; ++m) bs[b][m] = bs[b][m] + w * (xt[b] * (a.U[int64_t(j) * M + m] - fi[m]));
        }
        // _cholesky_moment
        double U[B1 * B1];
        bool ok = true;
        for (int attempt = 0; attempt < 2; ++attempt) {
            ok = true;
            for (int r = 0; r < B1 * B1; ++r) U[r] = 0.0;
            for (int r = 0; r < B1 && ok; ++r)
                for (int c = r; c < B1; ++c) {
                    double sm = N[r * B1 + c];
                    for (int q = 0; q < r; ++q) sm = sm - U[q * B1 + r] * U[q * B1 + c];
                    if (r == c) {
                        if (!(sm > 0.0)) { ok = false; break; }
                        U[r * B1 + r] = sqrt(sm);
                    } else U[r * B1 + c] = sm / U[r * B1 + r];
                }
            if (attempt == 0 && ok) {
                for (int q = 0; q < B1; ++q) {
                    double u = U[q * B1 + q];
                    if (!(u * u > 10.0 * 2.220446049250313e-16 * N[q * B1 + q])) { ok = false; break; }
                }
                if (ok) break;
            }
            if (attempt == 0) {
                double tr = 0.0;
                for (int q = 0; q < B1; ++q) tr = tr + N[q * B1 + q];
                double er = 1.4901161193847656e-08 * tr / double(B1);
                for (int q = 0; q < B1; ++q) N[q * B1 + q] = N[q * B1 + q] + er;
            }
        }
        if (ok) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                double y[B1], x[B1];
                for (int r = 0; r < B1; ++r) {
                    double t = double(bs[r][m]);
                    for (int q = 0; q < r; ++q) t = t - U[q * B1 + r] * y[q];
                    y[r] = t / U[r * B1 + r];
                }
                for (int r = B1 - 1; r >= 0; --r) {
                    double t = y[r];
                    for (int q = r + 1; q < B1; ++q) t = t - U[r * B1 + q] * x[q];
                    x[r] = t / U[r * B1 + r];
                }
#pragma unroll
                for (int b = 0; b < B1; ++b) out[b][m] = T(x[b] * invLd);
            }
        }
    }
    if (lim) {
        if (!done && !(p == a.sc.max_order && a.g.ok_r[i]))       // a lowered order's fit (or none): its own loop
            for (int k = 0; k < cnt; ++k) {
                T f[M];
                load_vec<T, M>(a.U + int64_t(a.g.nidx[int64_t(k) * np + i]) * M, f);
                extend_extrema<T, M>(f, umin, umax);
            }
        limit_slopes<T, D, M, RDEG>(a, i, cnt, fi, umin, umax, out);
    }
    store_row<T, BR * M, grad_row<T, BR * M>()>(g, &out[0][0]);
}

// Warps of a block of the FP32 worklist passes, and how many of them share a tile of nt listed tiles. A tile's slots
// are dealt to its warps, so a warp's serial chain (a dependent index -> state -> gradient load a slot, about 1.4 us
// each at 66 slots in 3-D) is the slots over the warps. Short lists leave most SMs idle and take the whole block a
// tile; longer ones keep four warps a tile, whose partial sums cost less to combine. The line depends on the list
// alone, so results do not depend on the launch shape. States of 8 and more components keep blocks of four warps
// (shared memory of their partial sums), and so does the flux pass in 1-D and 2-D: about 20 slots are few for 16 warps
// (15.7 us a pass with 16 warps, 12.9 with four; the reconstruction pass 8.8 against 12.5). Third-order systems in 3-D have
// eight in the flux pass: a slot takes up to 192 registers, and 16 warps leave 128 (188 bytes spilled). 3-D Euler, us a
// step with 16 / eight: blast at 64k interior particles 3902 / 3793, 343k 9923 / 9825 (limiter 4707 / 4582, 12960 / 12870);
// smooth, where lists are short, 2525 / 2483 and 6715 / 6816.
template <int M> constexpr int split_warps() { return M >= 8 ? 4 : 16; }
template <int D, int M, int RDEG> constexpr int flux_split_warps() { return M >= 8 || D < 3 ? 4 : RDEG >= 2 && M > 2 ? 8 : 16; }
template <int NW> __device__ __forceinline__ int split_share(unsigned nt) {
    return NW > 4 && nt <= HCC_SPLIT_WIDE_TILES ? NW : 4;
}

// FP32 degree-1 worklist pass of the reconstruction with several warps per tile: the tile's first warp lowers starved
// orders and picks the path; on the cached gradient-weight path warp w of W sums the slots k = w, w + W, ... and marks
// their neighbours' reach, the first warp adds the partial sums in a fixed order, applies the limiter and stores the
// gradients; any other particle has zero slopes (with a limiter: is reconstructed whole by the first warp).
template <typename T, int D, int M, int PDE, int RDEG, bool LIM>
__global__ void __launch_bounds__(32 * split_warps<M>()) k_gather_tiles(const StageArgs<T> a) {
    constexpr int BR = RBasis<D, RDEG>::B, NW = split_warps<M>();
    __shared__ T parts[NW][32][BR * M];
    __shared__ int path[NW / 4][32];
    const int lane = int(threadIdx.x & 31), wb = int(threadIdx.x >> 5);
    const unsigned nt = *a.wcount;
    const int W = split_share<NW>(nt);             // warps per tile
    const int group = wb / W, w = wb % W, first = group * W;
    const unsigned step = unsigned(NW / W) * gridDim.x;
    const int64_t np = a.g.npad;
    for (unsigned q0 = blockIdx.x * unsigned(NW / W); q0 < nt; q0 += step) {
        const unsigned q = q0 + unsigned(group);
        const int32_t tile = q < nt ? a.wtiles[q] : 0;
        const uint32_t word = q < nt ? a.wmask[tile] : 0u;
        const int64_t i = int64_t(tile) * 32 + lane;
        const bool live = ((word >> lane) & 1u) && !a.g.bnd[i];
        const int cnt = live ? a.g.cnt[i] : 0;
        if (w == 0) {
            int gp = 0;
            if (live) {
                int p = a.orders[i];
                const int p0 = p;
                while (p > 1 && cnt < basis_count(D, p - 1)) --p;
                if (p < p0) a.orders[i] = int8_t(p);
                gp = (p == a.sc.max_order && p > 1 && a.g.ok_r[i] && a.g.gw) ? 1 : 0;
            }
            path[group][lane] = gp;
        }
        __syncthreads();
        const int gp = path[group][lane];
        {
            // warp-uniform slot loop over every live member (the reach marks, combined across the warp); the
            // cached-fit members also accumulate their gradients here
            const int myc = (live && gp) ? cnt : 0;
            const int myr = (live && a.rmask) ? cnt : myc;
            const int kw = __reduce_max_sync(0xffffffffu, myr);
            T fi[M], out[BR * M];
            if (myc > 0) load_vec<T, M>(a.U + i * M, fi);
#pragma unroll
            for (int b = 0; b < BR * M; ++b) out[b] = T(0);
            for (int k = w; k < kw; k += W) {
                const int32_t j = k < myr ? a.g.nidx[int64_t(k) * np + i] : -1;
                if (k < myc) {
                    T gk[D], df[M];
#pragma unroll
                    for (int d = 0; d < D; ++d) gk[d] = a.g.gw[(int64_t(k) * D + d) * np + i];
                    load_vec<T, M>(a.U + int64_t(j) * M, df);
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const T dm = df[m] - fi[m];
#pragma unroll
                        for (int b = 0; b < BR; ++b) out[b * M + m] = out[b * M + m] + gk[b] * dm;
                    }
                }
                if (a.rmask) reach_mark_warp(a.rmask, a.rtiles, a.rcount, a.rlist, a.rlcount, j);
            }
            if (myc > 0 || (live && gp))
#pragma unroll
                for (int b = 0; b < BR * M; ++b) parts[wb][lane][b] = out[b];
        }
        __syncthreads();
        if (w == 0 && a.rmask) reach_mark_warp(a.rmask, a.rtiles, a.rcount, a.rlist, a.rlcount, live ? int32_t(i) : -1);
        if (w == 0 && live) {
            if (gp) {
                T fi[M], out[BR][M];
                load_vec<T, M>(a.U + i * M, fi);
#pragma unroll
                for (int b = 0; b < BR; ++b)
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        T sm = parts[first][lane][b * M + m];
                        for (int v = 1; v < W; ++v) sm = sm + parts[first + v][lane][b * M + m];
                        out[b][m] = sm;
                    }
                if constexpr (LIM) {
                    T umin[M], umax[M];
#pragma unroll
                    for (int m = 0; m < M; ++m) umin[m] = umax[m] = fi[m];
                    for (int k = 0; k < cnt; ++k) {
                        T f[M];
                        load_vec<T, M>(a.U + int64_t(a.g.nidx[int64_t(k) * np + i]) * M, f);
                        extend_extrema<T, M>(f, umin, umax);
                    }
                    limit_slopes<T, D, M, RDEG>(a, i, cnt, fi, umin, umax, out);
                }
                store_row<T, BR * M, grad_row<T, BR * M>()>(a.grad + i * grad_row<T, BR * M>(), &out[0][0]);
            } else {
                if constexpr (LIM) {
                    gather_one<T, D, M, PDE, RDEG, true>(a, i);
                } else {                           // off the cached fit: zero slopes
                    T z[BR * M];
#pragma unroll
                    for (int b = 0; b < BR * M; ++b) z[b] = T(0);
                    store_row<T, BR * M, grad_row<T, BR * M>()>(a.grad + i * grad_row<T, BR * M>(), z);
                }
            }
        }
        if (w == 0 && lane == 0 && q < nt && a.clear_wmask) a.wmask[tile] = 0u;   // every lane read the word before the barrier
        __syncthreads();
    }
}

// Blocks an SM of the stream-fed reconstruction pass in FP32. One variable: nine in 1-D and 2-D (flux_min_blocks), eight in
// 3-D, where a slot's basis is longer and nine spilled up to 540 bytes a thread. 3-D, 343k interior particles, order 3, us
// a step: 1938 (limiter 1711) with eight here and seven in the flux pass, 2754 (2257) with nine in both, 2483 (2213)
// when one slot was in flight. Two variables in 2-D: ten (48 registers; a warp waits for its gathers); 360k particles, us a
// step with Barth-Jespersen limiter / without: 423 / 414 with ten, 461 / 415 with eight, 501 / 425 unbounded (80 and 76
// registers), 442 / 433 with one thread's slots in three sweeps.
template <typename T, int D, int M> constexpr int gather_min_blocks() {
    if (sizeof(T) == 8) return 1;
    return M == 1 ? (D == 3 ? 8 : 9) : M == 2 && D == 2 ? 10 : 1;
}

// A full pass (one thread per particle) or a worklist pass over tiles (the members of a word) that also marks the one-hop
// reach of each member in rmask / rtiles. Most listed members have dropped to order 1 and have nothing to fit: the pass
// is bound by the marks, slot after slot, so a list of no more tiles than warps gives each tile a block, whose warps
// share the slots, and a longer one a warp: all passes of an FP64 3-D step 707 -> 307 us (65.6 k interior particles, a
// third of them listed), of a moving 2-D one 123 -> 46 us.
template <typename T, int D, int M, int PDE, int RDEG, bool LIM>
__global__ void __launch_bounds__(128, gather_min_blocks<T, D, M>()) k_gather(const StageArgs<T> a) {
    if (a.full) {
        const int64_t i = full_particle(a, int64_t(blockIdx.x) * blockDim.x + threadIdx.x);
        if (i >= 0) gather_one<T, D, M, PDE, RDEG, LIM>(a, i);
        return;
    }
    const unsigned nt = *a.wcount;
    const int64_t np = a.g.npad;
    const int lane = int(threadIdx.x & 31), wb = int(threadIdx.x >> 5), warps = int(blockDim.x >> 5);
    const bool share = nt <= gridDim.x * warps;
    const int w = share ? wb : 0, step = share ? warps : 1;
    const unsigned first = share ? blockIdx.x : blockIdx.x * warps + wb, stride = share ? gridDim.x : gridDim.x * warps;
    for (unsigned q = first; q < nt; q += stride) {
        const int32_t tile = a.wtiles[q];
        const uint32_t word = a.wmask[tile];
        if (share) __syncthreads();                // (q is the block's) every warp has read the word
        else __syncwarp();
        if (a.clear_wmask && w == 0 && lane == 0) a.wmask[tile] = 0u;     // the changed list is consumed here
        const bool mem = (word >> lane) & 1u;
        const int32_t i = tile * 32 + lane;
        if (mem && w == 0) gather_one<T, D, M, PDE, RDEG, LIM>(a, i);
        if (a.rmask) {
            // the reach (members and their neighbours), slot by slot across the warp with combined atomics
            if (w == 0) reach_mark_warp(a.rmask, a.rtiles, a.rcount, a.rlist, a.rlcount, mem ? i : -1);
            const int c = mem ? a.g.cnt[i] : 0;
            const int kw = __reduce_max_sync(0xffffffffu, c);
            for (int k = w; k < kw; k += step)
                reach_mark_warp(a.rmask, a.rtiles, a.rcount, a.rlist, a.rlcount, k < c ? a.g.nidx[int64_t(k) * np + i] : -1);
        }
    }
}

// Epilogue of a flux pass for particle i: K_E[s] stored, the next candidate formed (_stage_predictor!,
// TimeSteppers.jl:400-421, and the implicit part), the Euler substep (:511-518) and the MOOD check of the next
// checkpoint (_mood_flag!, MOOD.jl:289-295) against the extrema mn/mx of {i} ∪ N(i) of the stage state.
// MOODu2 override (_u2_fails, MOOD.jl:241-271), for the DMP-violating components of a particle of order >= 3: per
// axis the curvature terms (reconstruction terms D + d) over {i} ∪ N(i) keep one sign, and over the neighbours within
// 1.5h comparable magnitudes, or are negligible; otherwise the candidate is flagged. A rare path (DMP violators only).
template <typename T, int D, int M, int RDEG>
__device__ __noinline__ bool u2_curvature_fails(const StageArgs<T> &a, int64_t i, const bool *viol) {
    constexpr int GS = grad_row<T, RBasis<D, RDEG>::B * M>();
    const int cnt = a.g.cnt[i];
    const int64_t np = a.g.npad;
    const T h = a.u2_h, h2 = h * h, r15 = T(1.5) * h, near_sq = r15 * r15, dl = a.delta;
    for (int d = 0; d < D; ++d) {
        const int b = D + d;
        T mini[M], maxi[M], minA[M], maxA[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const T ci = a.grad[i * GS + b * M + m];
            mini[m] = maxi[m] = ci;
            minA[m] = maxA[m] = fabs(ci);
        }
        for (int k = 0; k < cnt; ++k) {
            const int64_t j = a.g.nidx[int64_t(k) * np + i];
            T r2 = T(0);
#pragma unroll
            for (int e = 0; e < D; ++e) {
                const T x = a.g.dist[(int64_t(k) * D + e) * np + i];
                r2 = (e == 0) ? x * x : r2 + x * x;
            }
            const bool near = r2 <= near_sq;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const T cj = a.grad[j * GS + b * M + m];
                mini[m] = vmin(mini[m], cj);
                maxi[m] = vmax(maxi[m], cj);
                if (near) { minA[m] = vmin(minA[m], fabs(cj)); maxA[m] = vmax(maxA[m], fabs(cj)); }
            }
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
            if (!viol[m]) continue;
            if (vmax(fabs(mini[m]), fabs(maxi[m])) * h2 < dl) continue;    // negligible curvature
            const bool same_sign = (mini[m] * h2) * (maxi[m] * h2) > -(dl * dl);
            const bool comparable = a.u2_ratio <= T(0) || minA[m] >= a.u2_ratio * maxA[m];
            if (!(same_sign && comparable)) return true;
        }
    }
    return false;
}

template <typename T, int D, int M, int PDE, int RDEG = 0>
__device__ __forceinline__ bool stage_epilogue(const StageArgs<T> &a, int64_t i, const T *fi, const T *Kv,
                                               const T *mn, const T *mx) {
    store_vec<T, M>(a.K + i * M, Kv);
    if (!a.form_next) return false;
    // _stage_predictor! for the next candidate
    T Y[M];
    load_vec<T, M>(a.Un + i * M, Y);
    const StageCoeffs<T> *cf = coef_of(a, i);
    for (int j = 0; j < a.n_prev; ++j) {
        const T hE = cf->hE[j], hI = cf->hI[j];
        if (hE != T(0)) {
            const T h = hE;
            if (j == a.self_slot) {
#pragma unroll
                for (int m = 0; m < M; ++m) Y[m] = Y[m] + h * Kv[m];
            } else {
                T kv[M];
                load_vec<T, M>(a.KE[j] + i * M, kv);
#pragma unroll
                for (int m = 0; m < M; ++m) Y[m] = Y[m] + h * kv[m];
            }
        }
        if (hI != T(0)) {
            const T h = hI;
            T kv[M];
            load_vec<T, M>(a.KI[j] + i * M, kv);
#pragma unroll
            for (int m = 0; m < M; ++m) Y[m] = Y[m] + h * kv[m];
        }
    }
    if (a.implicit_mode) {
        T KIo[M];
        implicit_part<T, D, M, PDE>(a, i, Y, KIo);
        store_vec<T, M>(a.KInext + i * M, KIo);
    }
    store_vec<T, M>(a.Ynext + i * M, Y);
    if (a.Xnext) {
        // moving grid: the next stage positions X = x_n + Σ_j dt ã_j K_X[j] (_stage_predictor!, :403-421)
        const int64_t np = a.g.npad;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            double X = a.x_n[int64_t(d) * np + i];
            for (int j = 0; j < a.n_prev; ++j) {
                const double h = cf->hEd[j];
                if (h != 0.0) {
                    const double kx = (j == a.self_slot) ? a.KXout[int64_t(d) * np + i] : a.KX[j][int64_t(d) * np + i];
                    X = X + h * kx;
                }
            }
            a.Xnext[int64_t(d) * np + i] = X;
        }
    }
    if (!a.check) return false;
    T cand[M];
    if (a.check_substep) {
        if (a.KIs) {
#pragma unroll
            for (int m = 0; m < M; ++m) cand[m] = fi[m] + cf->h_sub * (Kv[m] + a.KIs[i * M + m]);
        } else {
#pragma unroll
            for (int m = 0; m < M; ++m) cand[m] = fi[m] + cf->h_sub * Kv[m];
        }
    } else {
#pragma unroll
        for (int m = 0; m < M; ++m) cand[m] = Y[m];
    }
    const bool adm = admissible<T, D, M, PDE>(a.ph, cand);
    bool flag = !adm;
    if (a.sc.criterion == HCC_MOOD_ONLY) flag = true;
    else if (a.sc.criterion == HCC_MOOD_U1 && !flag) {
        const T dl = a.delta, d3 = dl * dl * dl;
        if constexpr (sizeof(T) == 8) {
#pragma unroll
            for (int m = 0; m < M; ++m)
                if (fabs(mx[m] - mn[m]) >= d3 && (cand[m] < mn[m] - dl || cand[m] > mx[m] + dl)) flag = true;
        } else {
            // FP32: the bounds are padded by 16 unit round-offs of their magnitude on top of delta, so the round-off
            // of the FP32 update (a few units on a flat state) is not read as a new extremum.
            constexpr T kPad = T(16) * T(1.1920928955078125e-7);
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const T pad = dl + kPad * vmax(fabs(mn[m]), fabs(mx[m]));
                if (fabs(mx[m] - mn[m]) >= d3 && (cand[m] < mn[m] - pad || cand[m] > mx[m] + pad)) flag = true;
            }
        }
    }
    else if (a.sc.criterion == HCC_MOOD_U2 && !flag) {
        // DMP violators that are not a plateau (the u1 test, plus max - min < plateau x global range)
        const T dl = a.delta, d3 = dl * dl * dl;
        bool viol[M], any = false;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            T pad = dl;
            if constexpr (sizeof(T) == 4) pad = dl + T(16) * T(1.1920928955078125e-7) * vmax(fabs(mn[m]), fabs(mx[m]));
            bool v = fabs(mx[m] - mn[m]) >= d3 && (cand[m] < mn[m] - pad || cand[m] > mx[m] + pad);
            if (v && a.u2_range) {
                const unsigned long long nanbits = a.u2_range[2 * M];
                const T range = ((nanbits >> m) & 1ull) ? T(NAN)
                                                        : T(order_value(a.u2_range[M + m])) - T(order_value(a.u2_range[m]));
                v = !(mx[m] - mn[m] < a.u2_plateau * range);
            }
            viol[m] = v;
            any = any || v;
        }
        if (any) {
            if constexpr (RDEG >= 2) {
                flag = (a.sc.max_order < 3 || a.orders[i] < 3) ? true : u2_curvature_fails<T, D, M, RDEG>(a, i, viol);
            } else {
                flag = true;
            }
        }
    }
    a.inadm[i] = !adm;
    return flag;
}

// ----------------------------------------------------------------------------------- flux pass
// Number of reconstruction terms an interface of order o keeps (mask_basis, Interpolators.jl:265-284):
// basis_count(D, o - 1) for 2 <= o <= RDEG + 1, else 0 — compile-time values, no integer division per slot.
template <int D, int RDEG>
__device__ __forceinline__ int interface_terms(int o) {
    constexpr int b1 = cbasis_count(D, 1), b2 = cbasis_count(D, 2);
    return (o == 2) ? b1 : ((o == 3 && RDEG >= 2) ? b2 : 0);
}

// Resident blocks per SM the flux kernel is compiled for: as many as its registers allow without spilling
// (FP32 2-D Euler and 3-D scalars: 72 registers; wider states and FP64 need more), but for 1-D and 2-D scalars.
template <typename T, int D, int M> constexpr int flux_min_blocks() {
    if (sizeof(T) == 8) return M >= 8 ? 1 : (D * M >= 12 ? 2 : HCC_FLUX_MINB64);
    // one variable in 1-D and 2-D: a slot is few instructions and three dependent gathers, so the pass waits, and 36 warps an
    // SM wait better than 28 (56 registers, 46 to 68 bytes spilled in 2-D at order 3; with limiter, 1.0 M: 3857 us for four
    // steps with nine blocks an SM in this pass and the reconstruction, 3926 with eight, 4222 with seven, 4441 with ten). In
    // 3-D the spills cost more than the warps give: see gather_min_blocks.
    return M >= 8 ? HCC_FLUX_MINB_MANY : (D * M >= 12 ? HCC_FLUX_MINB_WIDE : M == 1 && D < 3 ? 9 : HCC_FLUX_MINB);
}

// The MUSCL functor (MUSCL.jl:390-508) in its streamed form: per slot, EPD interface reconstruction, physical
// fluxes, Rusanov (FluxFunctions.jl:66-76) with sort_flux (Utils.jl:95-102), the flux difference ΔF and its
// contraction with the divergence weights; K_E = -2 Σ c·ΔF (TimeSteppers.jl:354). Fused epilogue: the next
// candidate (_stage_predictor!, :400-421, and the implicit part), the Euler substep (:511-518) and the MOOD
// check of the next checkpoint (_mood_flag!, MOOD.jl:289-295; the extrema come from this loop's neighbour reads).
// Partial sums of a particle's slots handled by one warp of a split tile (FP32 worklist passes).
template <typename T, int M> struct FluxPart {
    T s[M], c[M], mn[M], mx[M];
};

// A slot's term on its own (the ordered split adds it later).
template <int M> struct SlotTerm {
    double t[M];
    __device__ __forceinline__ void add(const double *x) {
#pragma unroll
        for (int m = 0; m < M; ++m) t[m] = x[m];
    }
};

// One slot k of the flux pass of particle i (the MUSCL functor's slot body, MUSCL.jl:463-508): interface orders oi,
// oj and the sort orientation `below` are the caller's; the interface reconstructions, the physical fluxes, the
// Rusanov flux of the pair sorted by the signs of the axis offsets (sort_flux, Utils.jl:95-102; FluxFunctions.jl:66-76)
// and its flux difference contracted with the slot's divergence weights wk go into acc.
template <typename T, int D, int M, int PDE, int RDEG, bool ALE, bool MOM, class Acc>
__device__ __forceinline__ void flux_slot(const StageArgs<T> &a, const T *fi, const T (*gi)[M], const T (*Fi)[M],
                                          const T *wp, const T *fj, const T *gj, const int oi, const int oj,
                                          const bool below, const T *dk, const T *wk, Acc &acc,
                                          const int64_t i, const int k) {
    constexpr int BR = RBasis<D, RDEG>::B;
    constexpr bool kFast = sizeof(T) == 4;   // FP32: scaled Rusanov form
    const int64_t np = a.g.npad;
    (void)np; (void)i; (void)k; (void)wp;
    // (FP64, degree 1: the reconstruction below scales the contraction with the whole offset)
    T pi[BR], pj[BR];
    if constexpr (kFast && RDEG == 1) {
        // degree 1: an interface of order 2 keeps the linear terms, order 1 none (the midpoint offsets
        // ±dk/2 scaled by 0 or ±1/2)
        const T si = oi >= 2 ? T(0.5) : T(0), sj = oj >= 2 ? T(-0.5) : T(0);
#pragma unroll
        for (int d = 0; d < D; ++d) { pi[d] = si * dk[d]; pj[d] = sj * dk[d]; }
    } else if constexpr (RDEG > 1) {
        const int keep_i = interface_terms<D, RDEG>(oi);
        const int keep_j = interface_terms<D, RDEG>(oj);
        T hx[D], pb[BR];
#pragma unroll
        for (int d = 0; d < D; ++d) hx[d] = T(0.5) * dk[d];
        recon_basis<D, RDEG, T>(hx, pb);
        // the basis at -hx: the first-degree terms change sign, the second-degree ones do not
#pragma unroll
        for (int b = 0; b < BR; ++b) {
            pi[b] = b < keep_i ? pb[b] : T(0);
            pj[b] = b < keep_j ? (b < D ? -pb[b] : pb[b]) : T(0);
        }
    }
    if constexpr (kFast && PDE != HCC_PDE_EULER && !ALE) {
        // FP32, linear fluxes F_d(f)_m = c_dm f_m with constant speeds (advection, BGK), fixed grid: the
        // doubled Rusanov difference per component on the fly, without flux arrays (registers:
        // 2 (F_n - F_i)_m = sum_d w_d (c_dm (f_ij + f_ji - 2 f_i) - s_d max(λ_d) (f_ji - f_ij)))
        T sw[D];
#pragma unroll
        for (int d = 0; d < D; ++d)
            sw[d] = (below ? wk[d] : dk[d]) > T(0) ? a.ph.amax[d] : -a.ph.amax[d];
        T t[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            T si = gi[0][m] * pi[0];
            T sj = gj[m] * pj[0];
#pragma unroll
            for (int b = 1; b < BR; ++b) {
                si = si + gi[b][m] * pi[b];
                sj = sj + gj[b * M + m] * pj[b];
            }
            const T fij = fi[m] + si, fji = fj[m] + sj;
            const T sum = (fij + fji) - T(2) * fi[m], jump = fji - fij;
            T tm = wk[0] * (a.ph.c[0][m] * sum - sw[0] * jump);
#pragma unroll
            for (int d = 1; d < D; ++d) tm = tm + wk[d] * (a.ph.c[d][m] * sum - sw[d] * jump);
            t[m] = tm;
            if constexpr (MOM) {
                T se = a.ph.amax[0] * a.g.mw[(int64_t(k) * D) * np + i];
#pragma unroll
                for (int d = 1; d < D; ++d) se = se + a.ph.amax[d] * a.g.mw[(int64_t(k) * D + d) * np + i];
                t[m] = t[m] - se * jump;
            }
        }
        acc.add(t);
        return;
    }
    T fij[M], fji[M];
    if constexpr (kFast) {
#pragma unroll
        for (int q = 0; q < M / 2; ++q) {
            float2 si = p_mul(p_ld(gi[0], q), p_bc(pi[0]));
            float2 sj = p_mul(p_ld(gj, q), p_bc(pj[0]));
#pragma unroll
            for (int b = 1; b < BR; ++b) {
                si = p_fma(p_ld(gi[b], q), p_bc(pi[b]), si);
                sj = p_fma(p_ld(gj + b * M, q), p_bc(pj[b]), sj);
            }
            p_st(fij, q, p_add(p_ld(fi, q), si));
            p_st(fji, q, p_add(p_ld(fj, q), sj));
        }
    }
    if constexpr (!kFast && RDEG == 1) {
        // g.(±dk/2) = ±(g.dk)/2 exactly (a power of two), added in one rounding: 2 M + 2 D fewer FP64 instructions a
        // slot than with the scaled offsets
        const T si = oi >= 2 ? T(0.5) : T(0), sj = oj >= 2 ? T(-0.5) : T(0);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            T ci = gi[0][m] * dk[0], cj = gj[m] * dk[0];
#pragma unroll
            for (int b = 1; b < D; ++b) {
                ci = ci + gi[b][m] * dk[b];
                cj = cj + gj[b * M + m] * dk[b];
            }
            fij[m] = add_scaled<T>(fi[m], si, ci);
            fji[m] = add_scaled<T>(fj[m], sj, cj);
        }
    }
#pragma unroll
    for (int m = kFast ? (M / 2) * 2 : (RDEG == 1 ? M : 0); m < M; ++m) {
        T si = gi[0][m] * pi[0];
        T sj = gj[m] * pj[0];
#pragma unroll
        for (int b = 1; b < BR; ++b) {
            si = si + gi[b][m] * pi[b];
            sj = sj + gj[b * M + m] * pj[b];
        }
        fij[m] = fi[m] + si;
        fji[m] = fj[m] + sj;
    }
    if constexpr (projected_flux<T, PDE, ALE, MOM>()) {
        // FP32 Euler, fixed grid: the doubled Rusanov difference contracted with the slot's divergence weights,
        //   sum_d w_d [(F_d(f_ij) + F_d(f_ji)) - s_d max(λ_d) (f_ji - f_ij) - 2 F_d(f_i)]
        //     = Fw(f_ij) + Fw(f_ji) - S (f_ji - f_ij) - 2 Fw(f_i),   S = sum_d w_d s_d max(λ_d)
        // with Fw(U) = sum_d w_d F_d(U) (euler_projected) and 2 Fw(f_i) = (rho (2u.w), (2u.w) m + 2p w,
        // (E + p)(2u.w)) from the own constants of own_flux.
        T Fa[M], Fb[M], la[D], lb[D];
        euler_projected<D>(a.ph, fij, wk, Fa, la);
        euler_projected<D>(a.ph, fji, wk, Fb, lb);
        T S = T(0), un2 = T(0);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const T sd = vmax(la[d], lb[d]);
            const T ssd = (below ? wk[d] : dk[d]) > T(0) ? sd : -sd;
            S = (d == 0) ? wk[0] * ssd : S + wk[d] * ssd;
            un2 = (d == 0) ? wk[0] * Fi[0][0] : un2 + wk[d] * Fi[0][d];
        }
        T t[M], own[M];
        own[0] = fi[0] * un2;
#pragma unroll
        for (int e = 0; e < D; ++e) own[1 + e] = un2 * fi[1 + e] + Fi[0][D] * wk[e];
        own[D + 1] = Fi[0][D + 1] * un2;
#pragma unroll
        for (int m = 0; m < M; ++m) t[m] = ((Fa[m] + Fb[m]) - S * (fji[m] - fij[m])) - own[m];
        acc.add(t);
        return;
    }
    T Fij[D][M], Fji[D][M], lij[D], lji[D];
    flux_and_speed<T, D, M, PDE>(a.ph, fij, Fij, lij, wp);
    flux_and_speed<T, D, M, PDE>(a.ph, fji, Fji, lji, wp);
    T t[M];
    if constexpr (kFast) {
        // FP32: 2 (F_n - F_i) = (F_ij + F_ji) - s_d max(λ) (f_ji - f_ij) - 2 F_i with s_d = sign of the
        // axis component (the sort_flux orientation folded into the speed); the factor 2 leaves K = -Σ.
        // (pairs of components with the packed instructions, a scalar tail for odd M)
        T jump[M];
#pragma unroll
        for (int q = 0; q < M / 2; ++q) p_st(jump, q, p_sub(p_ld(fji, q), p_ld(fij, q)));
        if constexpr (M & 1) jump[M - 1] = fji[M - 1] - fij[M - 1];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const T ssd = (below ? wk[d] : dk[d]) > T(0) ? vmax(lij[d], lji[d]) : -vmax(lij[d], lji[d]);
            const float2 nssd = p_bc(-ssd), w2 = p_bc(wk[d]);
#pragma unroll
            for (int q = 0; q < M / 2; ++q) {
                const float2 Fs = p_add(p_ld(Fij[d], q), p_ld(Fji[d], q));
                const float2 dF2 = p_sub(p_fma(nssd, p_ld(jump, q), Fs), p_ld(Fi[d], q));
                p_st(t, q, (d == 0) ? p_mul(w2, dF2) : p_fma(w2, dF2, p_ld(t, q)));
            }
            if constexpr (M & 1) {
                const T dF2 = ((Fij[d][M - 1] + Fji[d][M - 1]) - ssd * jump[M - 1]) - Fi[d][M - 1];
                t[M - 1] = (d == 0) ? wk[0] * dF2 : t[M - 1] + wk[d] * dF2;
            }
        }
    } else {
        // sort_flux + Rusanov without per-component selects: F_L + F_R is Fij + Fji in either order (IEEE addition
        // commutes), max(λ_L, λ_R) is symmetric, and the orientation of f_R - f_L is the sign of the speed. The
        // halving is exact, so F_n - F_i is one fused multiply-add. The pass is bound by the FP64 unit, so only the
        // number of its instructions counts: with the fused scalings and the integer-key extrema the 3-D Euler pass
        // takes 3.48 ms on 103k particles (4.52 ms with separate multiplies and FP64 compares), the 2-D one 0.50 ms
        // on 68k (0.67 ms). Sums, products, divisions and roots are those of the oracle, in its order.
        T jump[M];
#pragma unroll
        for (int m = 0; m < M; ++m) jump[m] = fji[m] - fij[m];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const T sdd = negate_if(vmax(lij[d], lji[d]), !positive<T>(below ? wk[d] : dk[d]));
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const T dF = add_scaled<T>(-Fi[d][m], T(0.5), (Fij[d][m] + Fji[d][m]) - sdd * jump[m]);
                t[m] = (d == 0) ? wk[0] * dF : t[m] + wk[d] * dF;
            }
        }
    }
    acc.add(t);
    if constexpr (MOM) {
        // moment correction of a first-order scheme (MUSCL.jl:501-505): -1/2 sum_d s_d e^d_ij (f_ji - f_ij),
        // the speeds s_d = max(λ_d) of the pair (FP32: the doubled form of the scaled Rusanov flux)
        T se = vmax(lij[0], lji[0]) * a.g.mw[(int64_t(k) * D) * np + i];
#pragma unroll
        for (int d = 1; d < D; ++d) se = se + vmax(lij[d], lji[d]) * a.g.mw[(int64_t(k) * D + d) * np + i];
        const T corr = kFast ? se : T(0.5) * se;
        T t2[M];
#pragma unroll
        for (int m = 0; m < M; ++m) t2[m] = -(corr * (fji[m] - fij[m]));
        acc.add(t2);
    }
}

// The flux pass of particle i over its slots: the whole pass and its epilogue, or with SPLIT (FP32) the slots
// k0, k0 + kstep, ..., whose partial sums and extrema go to `part` for the caller to combine.
template <typename T, int D, int M, int PDE, int RDEG, bool ALE, bool SPLIT = false, bool MOM = false>
__device__ __forceinline__ bool flux_one(const StageArgs<T> &a, const int64_t i, const int first_slot = 0,
                                         const int split_step = 1, FluxPart<T, M> *part = nullptr,
                                         bool *rough = nullptr) {
    const int k0 = SPLIT ? first_slot : 0, kstep = SPLIT ? split_step : 1;
    constexpr int BR = RBasis<D, RDEG>::B;
    if (a.g.bnd[i]) {
        if (a.full) {
#pragma unroll
            for (int m = 0; m < M; ++m) a.K[i * M + m] = T(0);
            if (a.mover)
#pragma unroll
                for (int d = 0; d < D; ++d) a.KXout[int64_t(d) * a.g.npad + i] = 0.0;
        }
        return false;
    }
    const int cnt = a.g.cnt[i];
    const int64_t np = a.g.npad;
    const T invL = a.g.invL;
    (void)invL;
    T fi[M], gi[BR][M], Fi[D][M];
    load_vec<T, M>(a.U + i * M, fi);
    constexpr int GS = grad_row<T, BR * M>();
    load_row<T, BR * M, GS>(a.grad + i * GS, &gi[0][0]);
    // moving grid: this particle's grid velocity (K_X of the stage) and every flux in its frame
    T wv[D];
    const T *wp = nullptr;
    if constexpr (ALE) {
        grid_velocity<T, D, M, PDE>(a, i, fi, wv);
        wp = wv;
        if (k0 == 0)
#pragma unroll
            for (int d = 0; d < D; ++d) a.KXout[int64_t(d) * a.g.npad + i] = double(wv[d]);
    }
    own_flux<T, D, M, PDE, ALE, MOM>(a.ph, fi, Fi, wp);
    constexpr bool kFast = sizeof(T) == 4;   // FP32: scaled Rusanov form (flux_slot)
    const int oi_own = a.orders[i];
    const int didx = divergence_index(a.sc.DO, D, oi_own, cnt);
    const bool cached = a.g.ok_d[i] && didx == divergence_index(a.sc.DO, D, a.sc.max_order, cnt);
    const T *wsl = cached ? a.g.dw : a.g.dw1;
    const bool wok = cnt > 0 && (cached || (a.g.dw1 != nullptr && didx == 2 && a.g.ok_1[i]));
    const bool need_ext = a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2);
    const int nbmin_i = (a.sc.strategy == HCC_EPD2) ? a.nbmin[i] : 0;
    AccumV<T, M> acc;
    T mn[M], mx[M];
#pragma unroll
    for (int m = 0; m < M; ++m) { mn[m] = fi[m]; mx[m] = fi[m]; }

    // one slot: its neighbour's state, gradient and order, the interface orders, the flux
    auto slot = [&](const int32_t j, const T *dk, const T *wk, const int k) {
        T fj[M];
        load_vec<T, M>(a.U + int64_t(j) * M, fj);
        T gj[BR * M];
        load_row<T, BR * M, GS>(a.grad + int64_t(j) * GS, gj);
        if (need_ext) {
#pragma unroll
            for (int m = 0; m < M; ++m) { mn[m] = vmin(mn[m], fj[m]); mx[m] = vmax(mx[m], fj[m]); }
        }
        const int oj_own = a.orders[j];
        int oi, oj;
        if (a.sc.strategy == HCC_EPD1) { oi = oj = (oi_own < oj_own ? oi_own : oj_own); }
        else if (a.sc.strategy == HCC_EPD2) { int nj = a.nbmin[j]; oi = oj = (nbmin_i < nj ? nbmin_i : nj); }
        else { oi = oi_own; oj = oj_own; }
        // AlignedRusanovFlux (MUSCL.jl:331-338): where either particle is below the full order (every pair at
        // order 1) the states are sorted by the signs of the slot's divergence weights instead of the distance
        const bool below = a.sc.aligned && (a.sc.max_order == 1 || oi_own < a.sc.max_order ||
                                            oj_own < a.sc.max_order);
        flux_slot<T, D, M, PDE, RDEG, ALE, MOM>(a, fi, gi, Fi, wp, fj, gj, oi, oj, below, dk, wk, acc, i, k);
    };
    // FP32 full passes: the slots in groups of UF, the next group's slot data in flight while this group is
    // computed (the slot body unrolled over the group); otherwise a one-deep software pipeline
    constexpr int UF = (kFast && !SPLIT) ? HCC_FLUX_STREAM_GROUP : 1;
    if (UF > 1 && wok && k0 < cnt) {
        int32_t jb[UF];
        T dkb[UF][D], wkb[UF][D];
#pragma unroll
        for (int u = 0; u < UF; ++u) {
            const int ku = k0 + u;
            jb[u] = ku < cnt ? a.g.nidx[int64_t(ku) * np + i] : 0;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                dkb[u][d] = ku < cnt ? a.g.dist[(int64_t(ku) * D + d) * np + i] : T(0);
                wkb[u][d] = ku < cnt ? wsl[(int64_t(ku) * D + d) * np + i] : T(0);
            }
        }
        for (int k = k0; k < cnt; k += UF) {
            int32_t jn[UF];
            T dkn[UF][D], wkn[UF][D];
#pragma unroll
            for (int u = 0; u < UF; ++u) {
                const int kn = k + UF + u;
                jn[u] = kn < cnt ? a.g.nidx[int64_t(kn) * np + i] : 0;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    dkn[u][d] = kn < cnt ? a.g.dist[(int64_t(kn) * D + d) * np + i] : T(0);
                    wkn[u][d] = kn < cnt ? wsl[(int64_t(kn) * D + d) * np + i] : T(0);
                }
            }
#pragma unroll
            for (int u = 0; u < UF; ++u) {
                if (k + u >= cnt) break;
                slot(jb[u], dkb[u], wkb[u], k + u);
            }
#pragma unroll
            for (int u = 0; u < UF; ++u) {
                jb[u] = jn[u];
#pragma unroll
                for (int d = 0; d < D; ++d) { dkb[u][d] = dkn[u][d]; wkb[u][d] = wkn[u][d]; }
            }
        }
    } else if (wok && k0 < cnt) {
        // slot data of the next slot are loaded while this one is computed (one-deep software pipeline)
        int32_t jn = a.g.nidx[int64_t(k0) * np + i];
        T dkn[D], wkn[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            dkn[d] = a.g.dist[(int64_t(k0) * D + d) * np + i];
            wkn[d] = wsl[(int64_t(k0) * D + d) * np + i];
        }
        for (int k = k0; k < cnt; k += kstep) {
            const int32_t j = jn;
            T dk[D], wk[D];
#pragma unroll
            for (int d = 0; d < D; ++d) { dk[d] = dkn[d]; wk[d] = wkn[d]; }
            if (k + kstep < cnt) {
                jn = a.g.nidx[int64_t(k + kstep) * np + i];
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    dkn[d] = a.g.dist[(int64_t(k + kstep) * D + d) * np + i];
                    wkn[d] = wsl[(int64_t(k + kstep) * D + d) * np + i];
                }
            }
            slot(j, dk, wk, k);
        }
    } else if (need_ext) {
        for (int k = k0; k < cnt; k += kstep) {
            const int32_t j = a.g.nidx[int64_t(k) * np + i];
#pragma unroll
            for (int m = 0; m < M; ++m) {
                T fj = a.U[int64_t(j) * M + m];
                mn[m] = vmin(mn[m], fj);
                mx[m] = vmax(mx[m], fj);
            }
        }
    }
    if constexpr (SPLIT) {
        static_assert(sizeof(T) == 4, "split tiles are the FP32 path");
#pragma unroll
        for (int m = 0; m < M; ++m) {
            part->s[m] = acc.s[m];
            part->c[m] = acc.c[m];
            part->mn[m] = mn[m];
            part->mx[m] = mx[m];
        }
        return false;
    }
    T Kv[M];
#pragma unroll
    for (int m = 0; m < M; ++m) Kv[m] = kFast ? -acc.s[m] : -(T(2) * acc.s[m]);
    if (rough) {
        // the stencil of the stage state is not flat in some component (without the extrema: assume not flat)
        bool r = !need_ext;
#pragma unroll
        for (int m = 0; m < M; ++m) r = r || (mx[m] - mn[m]) > T(1e-6) * (fabs(mx[m]) + fabs(mn[m]));
        *rough = r;
    }
    return stage_epilogue<T, D, M, PDE, RDEG>(a, i, fi, Kv, mn, mx);
}

// Failed candidates of one tile (a warp's ballot) into the t list.
template <typename T> __device__ __forceinline__ void tile_failures(const StageArgs<T> &a, int64_t tile, bool f) {
    const unsigned b = __ballot_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && b) {
        a.tmask[tile] = b;
        a.ttiles[atomicAdd(a.tcount, 1u)] = int32_t(tile);
    }
}

// Failed candidates of a warp of particles from anywhere (i: this lane's particle): their bits, and each tile once. The
// words are clear between passes (k_drop_decide clears those it reads).
template <typename T> __device__ __forceinline__ void list_failures(const StageArgs<T> &a, int64_t i, bool f) {
    if (f && atomicOr(&a.tmask[i >> 5], 1u << (i & 31)) == 0u) list_append(a.ttiles, a.tcount, int32_t(i >> 5));
}

// ... of a warp of a full pass: its tile's, or each particle's own of an interior list.
template <typename T> __device__ __forceinline__ void full_failures(const StageArgs<T> &a, int64_t i, bool f) {
    if (a.ilist) list_failures(a, i, f);
    else tile_failures(a, i >> 5, f);              // (lane 0's, the only one used: every lane of a tile is in its warp)
}
// The predictor's rough marks of a warp of a full pass (an interior list's words are cleared before the pass).
template <typename T> __device__ __forceinline__ void full_rough(const StageArgs<T> &a, int64_t i, bool rough) {
    if (a.ilist) {
        if (rough) atomicOr(&a.rough_words[i >> 5], 1u << (i & 31));
        return;
    }
    const unsigned b = __ballot_sync(0xffffffffu, rough);
    if ((threadIdx.x & 31) == 0 && i >= 0) a.rough_words[i >> 5] = b;
}

// A full pass (one thread per particle; each warp reports the failed candidates of its tile) or an FP64 worklist pass over
// the particles of the reach, 32 to a warp. The members of a listed tile are few of its 32 (7 to 9 around the extrema of
// a smooth field, 22 around a front), and a warp instruction of the FP64 unit costs the same for any number of them. (The
// FP32 worklist pass, k_flux_tiles, keeps the tiles: it gains less from full warps than it loses to scattered slot
// loads.) The reach marks are cleared once read.
template <typename T, int D, int M, int PDE, int RDEG, bool ALE, bool MOM = false>
__global__ void __launch_bounds__(HCC_FLUX_BLOCK, flux_min_blocks<T, D, M>()) k_flux(const StageArgs<T> a) {
    if (a.full) {
        const int64_t i = full_particle(a, int64_t(blockIdx.x) * blockDim.x + threadIdx.x);
        bool rough = false;
        const bool f = (i >= 0) ? flux_one<T, D, M, PDE, RDEG, ALE, false, MOM>(a, i, 0, 1, nullptr,
                                                                                   a.rough_words ? &rough : nullptr)
                                   : false;
        if (a.check) full_failures(a, i, f);
        if (a.rough_words) full_rough(a, i, rough);
        return;
    }
    const unsigned nm = *a.wcount;
    const unsigned first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (unsigned q = first; q < nm; q += step) {
        const int64_t i = a.wlist[q];
        if (a.clear_wmask) a.wmask[i >> 5] = 0u;
        const bool f = flux_one<T, D, M, PDE, RDEG, ALE, false, MOM>(a, i);
        if (a.check) list_failures(a, i, f);
    }
}

// ----------------------------------------------------------------------------------- ordered slot split (FP64)
// FP64 passes of small clouds and short worklists: eight lanes share a particle. Lane h computes the terms of the slots
// h, h + 8, ... and leaves them in shared memory, and the lanes then add the round's terms in slot order, one component
// each, so every sum has the order of the one-thread pass and the result its bits. A warp instruction occupies the FP64
// unit for 16 cycles and its result is some 40 cycles away, so the one-thread pass wants about four warps an SM
// (20,000 particles on 152 SMs) before the unit is busy rather than the chain of one slot after another.
// 2.7 k particles, 2-D, one variable: flux 54 -> 18 us, reconstruction 23 -> 11 us. With 66 slots a particle (3-D Euler)
// the split also spreads the last wave, and no size is slower: a step of 22 k, 39 k, 64 k, 125 k, 216 k interior
// particles took 6.08, 11.1, 14.5, 23.3, 37.0 ms with one thread in the full flux pass and 6.08, 9.55, 13.7, 23.1, 36.9
// with eight lanes. With 20 slots the last round of eight is half empty, and large 2-D clouds keep one thread.
constexpr int kSplit64 = 8;

// Adds the round's terms (term[lane * E + e] of the slots k0 ... k0 + 7 of the warp's four particles) to this lane's
// share of the sums: entry h + 8 j in sum[j].
template <int E>
__device__ __forceinline__ void ordered_round(const double *term, int lane, int k0, int cnt, double *sum) {
    const int h = lane % kSplit64, g = lane - h;
#pragma unroll
    for (int j = 0; j < (E + kSplit64 - 1) / kSplit64; ++j) {
        const int e = h + kSplit64 * j;
        if (e < E) {
#pragma unroll
            for (int q = 0; q < kSplit64; ++q)
                if (k0 + q < cnt) sum[j] = sum[j] + term[(g + q) * E + e];
        }
    }
}
// The particle of this lane's group in entry `g` of a full pass (every particle) or a worklist pass, or -1.
template <typename T> __device__ __forceinline__ int64_t split_particle(const StageArgs<T> &a, unsigned g, unsigned count) {
    return a.full ? full_particle(a, int64_t(g)) : (g < count ? int64_t(a.wlist[g]) : -1);
}

// flux_one with the slots shared by eight lanes (no moment correction, no marks for the predictor).
template <int D, int M, int PDE, int RDEG, bool ALE>
__global__ void __launch_bounds__(128) k_flux_split(const StageArgs<double> a) {
    constexpr int BR = RBasis<D, RDEG>::B, GS = grad_row<double, BR * M>();
    __shared__ double terms[4][32 * M];
    double *term = terms[threadIdx.x >> 5];
    const int lane = int(threadIdx.x & 31), h = lane % kSplit64;
    const int64_t np = a.g.npad;
    const unsigned count = a.full ? unsigned(a.nfull) : *a.wcount;
    const unsigned step = gridDim.x * blockDim.x / kSplit64;
    const bool need_ext = a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2);
    for (unsigned g0 = (blockIdx.x * blockDim.x + threadIdx.x - lane) / kSplit64; g0 < count; g0 += step) {
        const int64_t i = split_particle(a, g0 + unsigned(lane / kSplit64), count);
        const bool bnd = i >= 0 && a.g.bnd[i];
        const bool live = i >= 0 && !bnd;
        if (bnd && a.full && h == 0) {
#pragma unroll
            for (int m = 0; m < M; ++m) a.K[i * M + m] = 0.0;
            if (ALE)
#pragma unroll
                for (int d = 0; d < D; ++d) a.KXout[int64_t(d) * np + i] = 0.0;
        }
        const int cnt = live ? a.g.cnt[i] : 0;
        double fi[M], gi[BR][M], Fi[D][M], wv[D], mn[M], mx[M], sum[1] = {0.0};
        const double *wp = nullptr, *wsl = nullptr;
        bool wok = false;
        int oi_own = 1, nbmin_i = 0;
        if (live) {
            load_vec<double, M>(a.U + i * M, fi);
            load_row<double, BR * M, GS>(a.grad + i * GS, &gi[0][0]);
            if constexpr (ALE) {
                grid_velocity<double, D, M, PDE>(a, i, fi, wv);
                wp = wv;
                if (h == 0)
#pragma unroll
                    for (int d = 0; d < D; ++d) a.KXout[int64_t(d) * np + i] = wv[d];
            }
            own_flux<double, D, M, PDE, ALE, false>(a.ph, fi, Fi, wp);
            oi_own = a.orders[i];
            const int didx = divergence_index(a.sc.DO, D, oi_own, cnt);
            const bool cached = a.g.ok_d[i] && didx == divergence_index(a.sc.DO, D, a.sc.max_order, cnt);
            wsl = cached ? a.g.dw : a.g.dw1;
            wok = cnt > 0 && (cached || (a.g.dw1 != nullptr && didx == 2 && a.g.ok_1[i]));
            if (a.sc.strategy == HCC_EPD2) nbmin_i = a.nbmin[i];
#pragma unroll
            for (int m = 0; m < M; ++m) { mn[m] = fi[m]; mx[m] = fi[m]; }
        }
        const int kw = __reduce_max_sync(0xffffffffu, cnt);
        for (int k0 = 0; k0 < kw; k0 += kSplit64) {
            const int k = k0 + h;
            if (k < cnt) {
                const int64_t j = a.g.nidx[int64_t(k) * np + i];
                double fj[M];
                load_vec<double, M>(a.U + j * M, fj);
                if (need_ext) {
#pragma unroll
                    for (int m = 0; m < M; ++m) { mn[m] = vmin(mn[m], fj[m]); mx[m] = vmax(mx[m], fj[m]); }
                }
                if (wok) {
                    double gj[BR * M], dk[D], wk[D];
                    load_row<double, BR * M, GS>(a.grad + j * GS, gj);
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        dk[d] = a.g.dist[(int64_t(k) * D + d) * np + i];
                        wk[d] = wsl[(int64_t(k) * D + d) * np + i];
                    }
                    const int oj_own = a.orders[j];
                    int oi = oi_own, oj = oj_own;
                    if (a.sc.strategy == HCC_EPD1) oi = oj = (oi_own < oj_own ? oi_own : oj_own);
                    else if (a.sc.strategy == HCC_EPD2) { const int nj = a.nbmin[j]; oi = oj = (nbmin_i < nj ? nbmin_i : nj); }
                    const bool below = a.sc.aligned && (a.sc.max_order == 1 || oi_own < a.sc.max_order ||
                                                        oj_own < a.sc.max_order);
                    SlotTerm<M> t;
                    flux_slot<double, D, M, PDE, RDEG, ALE, false>(a, fi, gi, Fi, wp, fj, gj, oi, oj, below, dk, wk, t,
                                                                   i, k);
#pragma unroll
                    for (int m = 0; m < M; ++m) term[lane * M + m] = t.t[m];
                }
            }
            __syncwarp();
            if constexpr (M <= kSplit64) {
                if (wok) ordered_round<M>(term, lane, k0, cnt, sum);
            }
            __syncwarp();
        }
        // the sums to the particle's first lane, the extrema over its lanes (exact in any order)
        if (live && h < M) term[(lane - h) * M + h] = sum[0];
        __syncwarp();
        if (need_ext) {
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int o = 1; o < kSplit64; o <<= 1) {
                    mn[m] = vmin(mn[m], __shfl_xor_sync(0xffffffffu, mn[m], o));
                    mx[m] = vmax(mx[m], __shfl_xor_sync(0xffffffffu, mx[m], o));
                }
        }
        if (live && h == 0) {
            double Kv[M];
#pragma unroll
            for (int m = 0; m < M; ++m) Kv[m] = -(2.0 * term[lane * M + m]);
            const bool f = stage_epilogue<double, D, M, PDE, RDEG>(a, i, fi, Kv, mn, mx);
            if (a.check) list_failures(a, i, f);
        }
        if (i >= 0 && h == 0 && !a.full && a.clear_wmask) a.wmask[i >> 5] = 0u;
        __syncwarp();
    }
}

// gather_one's cached fit with the slots shared by eight lanes; the other cases (no cached fit) go through gather_one
// in the particle's first lane. Full passes without a limiter.
template <int D, int M, int PDE, int RDEG>
__global__ void __launch_bounds__(128) k_gather_split(const StageArgs<double> a) {
    constexpr int BR = RBasis<D, RDEG>::B, E = BR * M, GS = grad_row<double, E>(), NE = (E + kSplit64 - 1) / kSplit64;
    __shared__ double terms[4][32 * E];
    double *term = terms[threadIdx.x >> 5];
    const int lane = int(threadIdx.x & 31), h = lane % kSplit64;
    const int64_t np = a.g.npad;
    const int64_t i = full_particle(a, (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) / kSplit64);
    const bool live = i >= 0 && !a.g.bnd[i];
    int cnt = 0;
    bool cached = false;
    double fi[M], sum[NE];
#pragma unroll
    for (int q = 0; q < NE; ++q) sum[q] = 0.0;
    if (live) {
        cnt = a.g.cnt[i];
        int p = a.orders[i];
        while (p > 1 && cnt < basis_count(D, p - 1)) --p;
        cached = p == a.sc.max_order && p > 1 && a.g.ok_r[i];
        load_vec<double, M>(a.U + i * M, fi);
    }
    if (!cached) cnt = 0;
    const int kw = __reduce_max_sync(0xffffffffu, cnt);
    for (int k0 = 0; k0 < kw; k0 += kSplit64) {
        const int k = k0 + h;
        if (k < cnt) {
            const int64_t s = int64_t(k) * np + i;
            double x[D], pb[BR], df[M];
            load_vec<double, M>(a.U + int64_t(a.g.nidx[s]) * M, df);
#pragma unroll
            for (int d = 0; d < D; ++d) x[d] = a.g.dist[(int64_t(k) * D + d) * np + i] * a.g.invL;
            const double w = a.g.wt[s];
            recon_basis<D, RDEG, double>(x, pb);
#pragma unroll
            for (int m = 0; m < M; ++m) df[m] = df[m] - fi[m];
#pragma unroll
            for (int b = 0; b < BR; ++b)
#pragma unroll
                for (int m = 0; m < M; ++m) term[lane * E + b * M + m] = w * (pb[b] * df[m]);
        }
        __syncwarp();
        ordered_round<E>(term, lane, k0, cnt, sum);
        __syncwarp();
    }
#pragma unroll
    for (int q = 0; q < NE; ++q)
        if (h + kSplit64 * q < E) term[(lane - h) * E + h + kSplit64 * q] = sum[q];
    __syncwarp();
    if (!live) return;
    if (!cached) {
        if (h == 0) gather_one<double, D, M, PDE, RDEG, false>(a, i);
        return;
    }
    // the inverse moments applied entry by entry: g_bm = (sum_c inv_bc bs_cm) scale_b, in gather_one's order
    const double *inv = a.g.inv_r + i * (BR * BR), *bs = term + (lane - h) * E;
    for (int e = h; e < E; e += kSplit64) {
        const int b = e / M, m = e % M;
        double acc = inv[b * BR] * bs[m];
        for (int c = 1; c < BR; ++c) acc = acc + inv[b * BR + c] * bs[c * M + m];
        a.grad[i * GS + e] = acc * recon_scale<D, RDEG, double>(b, a.g.invL);
    }
}

// FP32 worklist pass with several warps per tile (split_share): warp w of W takes the slots k = w, w + W, ... of every
// member of the tile (a share of the serial slot chain, the latency that bounds the short worklist passes), the tile's
// first warp combines the compensated partial sums (Kahan over the partials, minus their compensations) and the
// extrema, and runs the epilogue. Block-stride over the list.
template <typename T, int D, int M, int PDE, int RDEG, bool ALE, bool MOM = false>
__global__ void __launch_bounds__(32 * flux_split_warps<D, M, RDEG>()) k_flux_tiles(const StageArgs<T> a) {
    constexpr int NW = flux_split_warps<D, M, RDEG>();
    __shared__ FluxPart<T, M> parts[NW][32];
    const int lane = int(threadIdx.x & 31), wb = int(threadIdx.x >> 5);
    const unsigned nt = *a.wcount;
    const int W = split_share<NW>(nt);             // warps per tile
    const int group = wb / W, w = wb % W, first = group * W;
    const unsigned step = unsigned(NW / W) * gridDim.x;
    for (unsigned q0 = blockIdx.x * unsigned(NW / W); q0 < nt; q0 += step) {
        const unsigned q = q0 + unsigned(group);
        const int32_t tile = q < nt ? a.wtiles[q] : 0;
        const uint32_t word = q < nt ? a.wmask[tile] : 0u;
        const int64_t i = int64_t(tile) * 32 + lane;
        const bool live = ((word >> lane) & 1u) && !a.g.bnd[i];
        if (live) flux_one<T, D, M, PDE, RDEG, ALE, true, MOM>(a, i, w, W, &parts[wb][lane]);
        __syncthreads();
        if (w == 0 && q < nt) {
            bool f = false;
            if (live) {
                T Kv[M], mn[M], mx[M], fi[M];
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    T sm = T(0), cm = T(0), comp = T(0);
                    mn[m] = parts[first][lane].mn[m];
                    mx[m] = parts[first][lane].mx[m];
                    for (int v = 0; v < W; ++v) {
                        const T y = parts[first + v][lane].s[m] - cm;
                        const T u = sm + y;
                        cm = (u - sm) - y;
                        sm = u;
                        comp = comp + parts[first + v][lane].c[m];
                        mn[m] = vmin(mn[m], parts[first + v][lane].mn[m]);
                        mx[m] = vmax(mx[m], parts[first + v][lane].mx[m]);
                    }
                    Kv[m] = -(sm - comp);
                }
                load_vec<T, M>(a.U + i * M, fi);
                f = stage_epilogue<T, D, M, PDE, RDEG>(a, i, fi, Kv, mn, mx);
            }
            if (a.check) tile_failures(a, tile, f);
            if (lane == 0 && a.clear_wmask) a.wmask[tile] = 0u;
        }
        __syncthreads();
    }
}

// ----------------------------------------------------------------------------------- tile-staged full passes (FP32)
// Full gather and flux passes of an FP32 context with tile tables (TileView): one block per tile of HCC_TILE
// consecutive particles first copies the tile's neighbour union into shared memory -- positions (and orders), states,
// and for the flux pass the gradients; a thread copies whole entries, and the ascending union ids make a warp's loads
// cover contiguous runs -- then every slot reads its neighbour from shared memory with 16-byte loads. Offsets
// x_j - x_i are (in 3-D) exact differences of the quantised union positions, rounded once to FP32; the weight w(|x|^2) and
// the slot's gradient and divergence weights follow from the particle's FP32 fit rows. The arithmetic after that is
// flux_slot / the cached gather of the stream-fed passes. Each thread loads the union place of its next slot while
// it computes the current one.

// Shared-memory layout. Gather pass: one row per union entry, the position (D ints) then the state. Flux pass: an
// int4 array of positions (the order in .w), then one row per entry of the state and the gradient; without positions
// (1-D, 2-D) the rows, then the orders. Rows are whole
// 16-byte groups, an odd number of them, so the rows that the lanes of a warp read spread over the banks.
constexpr int tile_odd_groups(int words) {
    const int g = (words + 3) / 4;
    return (g % 2 == 1) ? g : g + 1;
}
template <int D, int M> constexpr int tile_gather_row() { return 4 * tile_odd_groups(D + M); }
template <int D, int M> constexpr int tile_flux_row() { return 4 * tile_odd_groups(M + D * M); }

// Exponential weight of a squared distance (MLSWeightFunctions.jl:68-82: 1 / the degree-4 Taylor sum of e^y,
// y = alpha r^2 / R^2), FP32.
__device__ __forceinline__ float tile_weight(float r2, float wscale) {
    const float y = r2 * wscale;
    return recip<float>(1.0f + y * (1.0f + y * (0.5f + y * (0.16666667f + y * 0.041666668f))));
}

template <int D>
__device__ __forceinline__ void tile_offset(const int *qj, const int *qi, float qt, float *x) {
#pragma unroll
    for (int d = 0; d < D; ++d) x[d] = float(qj[d] - qi[d]) * qt;
}

// N words of a 16-byte-aligned shared-memory row as whole 16-byte loads.
template <int N>
__device__ __forceinline__ void lds_words(const float *row, float *out) {
    constexpr int G = (N + 3) / 4;
    const float4 *r4 = reinterpret_cast<const float4 *>(row);
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const float4 v = r4[g];
        if (4 * g + 0 < N) out[4 * g + 0] = v.x;
        if (4 * g + 1 < N) out[4 * g + 1] = v.y;
        if (4 * g + 2 < N) out[4 * g + 2] = v.z;
        if (4 * g + 3 < N) out[4 * g + 3] = v.w;
    }
}

// N words into a 16-byte-aligned shared-memory row (the padding of the last group is written as zero).
template <int N>
__device__ __forceinline__ void sts_words(float *row, const float *in) {
    constexpr int G = (N + 3) / 4;
    float4 *r4 = reinterpret_cast<float4 *>(row);
#pragma unroll
    for (int g = 0; g < G; ++g)
        r4[g] = make_float4(in[4 * g], 4 * g + 1 < N ? in[4 * g + 1] : 0.0f, 4 * g + 2 < N ? in[4 * g + 2] : 0.0f,
                            4 * g + 3 < N ? in[4 * g + 3] : 0.0f);
}

// Reconstruction pre-pass, two threads per particle of the tile (slots k = h, h + 2, ... for h = 0, 1): the cached
// degree-1 fit of gather_one with the gradient weights recomputed per slot, the second thread's partial sums added by
// the first through shared memory (the fit's rows applied once, to the sums of w x (f_j - f_i), take no less time, 1534
// against 1529 us a step of 3-D Euler at 343k points, and round more: the right-hand side's error grows by 0.3 % on a box,
// by 1.0 % on a cloud squeezed along its diagonal); every other case (boundary, starved or lowered order, failed fit, limiter) goes
// through gather_one itself.
// Union entries a thread stages per round in the tile passes (all their loads in flight before the first store):
// HCC_TILE_STAGE_UNROLL for rows of up to 12 words, half as many for wider rows (registers).
template <int RW> constexpr int tile_stage_unroll() {
    return RW <= 12 ? HCC_TILE_STAGE_UNROLL : (HCC_TILE_STAGE_UNROLL + 1) / 2;
}

// LIM: slope limiters, which go through gather_one. Without one, a particle off the cached fit (an order below the full
// one, a failed fit) has zero slopes, and the kernel does without gather_one's registers.
// Two blocks an SM with a limiter (three spilled 104 bytes): 3-D Euler, us a step with three / two, Barth-Jespersen at 64k
// interior particles 1360 / 1149 (blast 1325 / 1165), at 343k 3872 / 3787 (3938 / 3913); Venkatakrishnan 1426 / 1240
// (1300 / 1152), 4154 / 4176 (3933 / 3906).
template <int D, int M, int PDE, bool LIM>
__global__ void __launch_bounds__(2 * HCC_TILE, LIM ? 2 : 3) k_gather_tile(const StageArgs<float> a) {
    extern __shared__ __align__(16) float sm[];
    constexpr int W = tile_gather_row<D, M>(), GS = grad_row<float, D * M>();
    const int64_t t = blockIdx.x;
    {
        const int64_t u0 = a.tv.ustart[t];
        const int nu = int(a.tv.ustart[t + 1] - u0);
        // SU entries per thread and round: their ids first, then every load of the round in flight, then the stores
        constexpr int SU = tile_stage_unroll<D + M>();
        const int nt = int(blockDim.x);
        for (int e0 = threadIdx.x; e0 < nu; e0 += SU * nt) {
            int32_t jj[SU];
#pragma unroll
            for (int u = 0; u < SU; ++u) jj[u] = e0 + u * nt < nu ? a.tv.uid[u0 + e0 + u * nt] : 0;
            float v[SU][D + M];
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                if (e0 + u * nt >= nu) break;
                const int4 q = a.tv.upos[u0 + e0 + u * nt];
                v[u][0] = __int_as_float(q.x);
                if constexpr (D > 1) v[u][1] = __int_as_float(q.y);
                if constexpr (D > 2) v[u][2] = __int_as_float(q.z);
#pragma unroll
                for (int m = 0; m < M; ++m) v[u][D + m] = a.U[int64_t(jj[u]) * M + m];
            }
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                if (e0 + u * nt >= nu) break;
                sts_words<D + M>(sm + (e0 + u * nt) * W, v[u]);
            }
        }
    }
    float *parts = sm + a.tv.umax * W;           // [HCC_TILE][D * M] partial gradients of the second threads
    __syncthreads();
    const int pl = int(threadIdx.x) % HCC_TILE, h = int(threadIdx.x) / HCC_TILE;
    const int64_t i = full_particle(a, t * HCC_TILE + pl);
    int mode = 0;                                 // 1: the cached fit here, 2: gather_one (first thread)
    int cnt = 0;
    if (i >= 0 && !a.g.bnd[i]) {
        cnt = a.g.cnt[i];
        int q = a.orders[i];
        while (q > 1 && cnt < basis_count(D, q - 1)) --q;
        if (!LIM && h == 0 && q < a.orders[i]) a.orders[i] = int8_t(q);   // starved (gather_one lowers it itself)
        mode = (q == a.sc.max_order && q > 1 && a.g.ok_r[i] && !LIM) ? 1 : 2;
    }
    float out[D][M];
#pragma unroll
    for (int b = 0; b < D; ++b)
#pragma unroll
        for (int m = 0; m < M; ++m) out[b][m] = 0.0f;
    if (mode == 1) {
        const int64_t np = a.g.npad;
        float own[D + M];
        lds_words<D + M>(sm + int(a.tv.lself[i]) * W, own);
        int qi[D];
#pragma unroll
        for (int d = 0; d < D; ++d) qi[d] = __float_as_int(own[d]);
        float G[D][D];
        const float *cf = a.tv.coef + i * a.tv.cw + D + D * D;
#pragma unroll
        for (int b = 0; b < D; ++b)
#pragma unroll
            for (int c = 0; c < D; ++c) G[b][c] = cf[b * D + c];
        const float qt = a.tv.quantum[t], ws = a.tv.wscale;
        // this thread's slots h, h + 2, ...: their union places in groups of PF, the next group's loads in flight
        // while this group is summed
        constexpr int PF = HCC_TILE_GATHER_GROUP;
        const int mine = cnt > h ? (cnt - h + 1) / 2 : 0;
        const uint16_t *lp = a.tv.lidx + int64_t(h) * np + i;
        const int64_t step = 2 * np;
        int lbuf[PF];
#pragma unroll
        for (int q = 0; q < PF; ++q) lbuf[q] = q < mine ? int(lp[int64_t(q) * step]) : 0;
        for (int k0 = 0; k0 < mine; k0 += PF) {
            int lnext[PF];
#pragma unroll
            for (int q = 0; q < PF; ++q) lnext[q] = k0 + PF + q < mine ? int(lp[int64_t(k0 + PF + q) * step]) : 0;
#pragma unroll
            for (int q = 0; q < PF; ++q) {
                if (k0 + q >= mine) break;
                float r[D + M];
                lds_words<D + M>(sm + lbuf[q] * W, r);
                int qj[D];
#pragma unroll
                for (int d = 0; d < D; ++d) qj[d] = __float_as_int(r[d]);
                float x[D];
                tile_offset<D>(qj, qi, qt, x);
                float r2 = x[0] * x[0];
#pragma unroll
                for (int d = 1; d < D; ++d) r2 = r2 + x[d] * x[d];
                const float w = tile_weight(r2, ws);
                float gk[D];
#pragma unroll
                for (int b = 0; b < D; ++b) {
                    float v = G[b][0] * x[0];
#pragma unroll
                    for (int c = 1; c < D; ++c) v = v + G[b][c] * x[c];
                    gk[b] = w * v;
                }
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float dm = r[D + m] - own[D + m];
#pragma unroll
                    for (int b = 0; b < D; ++b) out[b][m] = out[b][m] + gk[b] * dm;
                }
            }
#pragma unroll
            for (int q = 0; q < PF; ++q) lbuf[q] = lnext[q];
        }
        if (h == 1)
#pragma unroll
            for (int b = 0; b < D; ++b)
#pragma unroll
                for (int m = 0; m < M; ++m) parts[pl * (D * M) + b * M + m] = out[b][m];
    }
    __syncthreads();
    if (h == 1) return;
    if (mode == 2) {
        if constexpr (LIM) gather_one<float, D, M, PDE, 1, true>(a, i);
        else store_row<float, D * M, GS>(a.grad + i * GS, &out[0][0]);
    } else if (mode == 1) {
#pragma unroll
        for (int b = 0; b < D; ++b)
#pragma unroll
            for (int m = 0; m < M; ++m) out[b][m] = out[b][m] + parts[pl * (D * M) + b * M + m];
        store_row<float, D * M, GS>(a.grad + i * GS, &out[0][0]);
    }
}

// Flux pass, two threads per particle of the tile in 3-D (slots k = h, h + 2, ... for h = 0, 1); the second writes its
// compensated partial sums and extrema to shared memory, the first combines them and runs the epilogue. (Four threads and
// one block an SM where that saves a wave: never faster on 11 k to 290 k interior particles, at most 12 % slower.)
// In 2-D and 1-D one thread: with 20 slots the combination and the idle half of the epilogue cost more than the second
// thread gives. There the offsets and divergence weights come from the FP32 slot streams, and every slot is compensated on
// its own, so the results have the bits of the stream-fed pass (in 2-D): only the neighbours' rows come from shared
// memory. 2-D Euler, us a step with tiles / stream-fed: 167 / 178 at 4.4 k interior particles, 189 / 199 at 10 k,
// 228 / 234 at 53 k, 263 / 262 at 90 k, 362 / 393 at 160 k, 679 / 711 at 518 k, 1045 / 1120 at 1.0 M. (Offsets and weights
// recomputed from the quantised positions, sums compensated in blocks of four: no faster, and up to 0.5 % more error of the
// right-hand side. Four blocks an SM 1144, six 1117 at 1.0 M.)
template <int D> constexpr int tile_flux_threads() { return D == 3 ? 2 : 1; }
template <int D> constexpr int tile_flux_min_blocks() { return D == 3 ? 2 : 5; }
template <int D> constexpr bool tile_flux_streams() { return D < 3; }

// PLAIN: EPD1 interface orders and the plain Rusanov flux (the usual configuration), known at compile time.
template <int D, int M, int PDE, bool PLAIN>
__global__ void __launch_bounds__(tile_flux_threads<D>() * HCC_TILE, tile_flux_min_blocks<D>()) k_flux_tile(const StageArgs<float> a) {
    extern __shared__ __align__(16) float sm[];
    constexpr int W = tile_flux_row<D, M>();
    constexpr int RW = M + D * M;                 // used words of a row: the state, then the gradient
    constexpr int GS = grad_row<float, D * M>(), HT = tile_flux_threads<D>();
    constexpr bool STREAMS = tile_flux_streams<D>();
    const int64_t t = blockIdx.x;
    const int64_t u0 = a.tv.ustart[t];
    const int nu = int(a.tv.ustart[t + 1] - u0);
    int4 *spos = reinterpret_cast<int4 *>(sm);    // positions and orders, then the rows; without positions the rows,
    float *srow = sm + (STREAMS ? 0 : 4 * a.tv.umax);                                      // then the orders
    int *sord = reinterpret_cast<int *>(srow + a.tv.umax * W);
    FluxPart<float, M> *parts = reinterpret_cast<FluxPart<float, M> *>(sm);   // over the union, once it has been read
    // the particle's own global loads (count, union place, fit rows, the first union places of its slots) are issued
    // before the staging so that their latency overlaps it; none of them reads shared memory
    const int pl = int(threadIdx.x) % HCC_TILE, h = int(threadIdx.x) / HCC_TILE;
    const int64_t i = full_particle(a, t * HCC_TILE + pl);
    const bool live = i >= 0 && !a.g.bnd[i];
    const int64_t np = a.g.npad;
    // this thread's slots h, h + HT, ...: union places PF slots ahead (a rotating window), or in groups of PF with the
    // next group in flight (HCC_TILE_FLUX_GROUP > 0: the slot body unrolled over the group)
    constexpr int GROUP = STREAMS ? HCC_TILE_STREAM_GROUP : HCC_TILE_FLUX_GROUP;
    constexpr int PF = GROUP > 0 ? GROUP : HCC_TILE_FLUX_PF;
    const int64_t lstep = HT * np;
    const uint16_t *lp = a.tv.lidx + int64_t(h) * np + i;
    int cnt = 0, li = 0, mine = 0;
    bool wok = false;
    int lb[PF];
    float A[D], B[D][D];
    float xb[PF][D], wb[PF][D];                   // the offsets and divergence weights of a group's slots (STREAMS)
    auto stream = [&](int s, float *x, float *w) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            x[d] = s < mine ? a.g.dist[(int64_t(s) * D + d) * np + i] : 0.0f;
            w[d] = s < mine ? a.g.dw[(int64_t(s) * D + d) * np + i] : 0.0f;
        }
    };
    if (live) {
        cnt = a.g.cnt[i];
        li = int(a.tv.lself[i]);
        wok = cnt > 0 && a.g.ok_d[i];
        if constexpr (!STREAMS) {
            const float *cf = a.tv.coef + i * a.tv.cw;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                A[d] = cf[d];
#pragma unroll
                for (int e = 0; e < D; ++e) B[d][e] = cf[D + d * D + e];
            }
        }
        mine = cnt > h ? (cnt - h + HT - 1) / HT : 0;
#pragma unroll
        for (int q = 0; q < PF; ++q) {
            lb[q] = q < mine ? int(lp[int64_t(q) * lstep]) : 0;
            if constexpr (STREAMS) stream(q, xb[q], wb[q]);
        }
        lp += int64_t(PF) * lstep;
    }
    {
        // SU entries per thread and round: their ids first, then every load of the round in flight, then the stores
        constexpr int SU = tile_stage_unroll<RW>();
        const int nt = int(blockDim.x);
        for (int e0 = threadIdx.x; e0 < nu; e0 += SU * nt) {
            int32_t jj[SU];
#pragma unroll
            for (int u = 0; u < SU; ++u) jj[u] = e0 + u * nt < nu ? a.tv.uid[u0 + e0 + u * nt] : 0;
            int4 qq[SU];
            float v[SU][RW];
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                if (e0 + u * nt >= nu) break;
                const int64_t j = jj[u];
                if constexpr (!STREAMS) qq[u] = a.tv.upos[u0 + e0 + u * nt];
                qq[u].w = a.orders[j];
#pragma unroll
                for (int m = 0; m < M; ++m) v[u][m] = a.U[j * M + m];
                load_row<float, D * M, GS>(a.grad + j * GS, v[u] + M);
            }
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                if (e0 + u * nt >= nu) break;
                if constexpr (STREAMS) sord[e0 + u * nt] = qq[u].w;
                else spos[e0 + u * nt] = qq[u];
                sts_words<RW>(srow + (e0 + u * nt) * W, v[u]);
            }
        }
    }
    __syncthreads();
    const bool need_ext = a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2);
    // (with the streams each slot is compensated on its own, as in the stream-fed pass)
    BlockAccum<M, STREAMS ? 1 : HCC_FLUX_KAHAN_BLOCK> blk;
    AccumV<float, M> &acc = blk.sum;
    float mn[M], mx[M], fi[M];
    float gi[D][M], Fi[D][M];
    if (live) {
        int qi[3] = {0, 0, 0}, oi_own;
        if constexpr (STREAMS) {
            oi_own = sord[li];
        } else {
            const int4 q4 = spos[li];
            qi[0] = q4.x; qi[1] = q4.y; qi[2] = q4.z;
            oi_own = q4.w;
        }
        {
            float own[RW];
            lds_words<RW>(srow + li * W, own);
#pragma unroll
            for (int m = 0; m < M; ++m) { fi[m] = own[m]; mn[m] = fi[m]; mx[m] = fi[m]; }
#pragma unroll
            for (int b = 0; b < D; ++b)
#pragma unroll
                for (int m = 0; m < M; ++m) gi[b][m] = own[M + b * M + m];
        }
        own_flux<float, D, M, PDE, false, false>(a.ph, fi, Fi, nullptr);
        if (wok) {
            const float qt = STREAMS ? 0.0f : a.tv.quantum[t], ws = a.tv.wscale;
            auto slot = [&](const int l, const float *xs, const float *wsl, const int k) {
                float dk[D], wk[D];
                int oj_own;
                if constexpr (STREAMS) {
                    oj_own = sord[l];
#pragma unroll
                    for (int d = 0; d < D; ++d) { dk[d] = xs[d]; wk[d] = wsl[d]; }
                } else {
                    const int4 qj4 = spos[l];
                    const int qj[3] = {qj4.x, qj4.y, qj4.z};
                    oj_own = qj4.w;
                    tile_offset<D>(qj, qi, qt, dk);
                    float r2 = dk[0] * dk[0];
#pragma unroll
                    for (int d = 1; d < D; ++d) r2 = r2 + dk[d] * dk[d];
                    const float w = tile_weight(r2, ws);
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        float v = A[d];
#pragma unroll
                        for (int e = 0; e < D; ++e) v = v + B[d][e] * dk[e];
                        wk[d] = w * v;
                    }
                }
                float r[RW];
                lds_words<RW>(srow + l * W, r);
                if (need_ext) {
#pragma unroll
                    for (int m = 0; m < M; ++m) { mn[m] = vmin(mn[m], r[m]); mx[m] = vmax(mx[m], r[m]); }
                }
                int oi, oj;
                if (PLAIN || a.sc.strategy == HCC_EPD1) { oi = oj = (oi_own < oj_own ? oi_own : oj_own); }
                else { oi = oi_own; oj = oj_own; }
                const bool below = !PLAIN && a.sc.aligned && (a.sc.max_order == 1 || oi_own < a.sc.max_order ||
                                                              oj_own < a.sc.max_order);
                flux_slot<float, D, M, PDE, 1, false, false>(a, fi, gi, Fi, nullptr, r, r + M, oi, oj, below, dk,
                                                             wk, blk, i, k);
            };
            if constexpr (GROUP > 0) {
                for (int s0 = 0; s0 < mine; s0 += PF) {
                    int ln[PF];
                    float xn[PF][D], wn[PF][D];
#pragma unroll
                    for (int q = 0; q < PF; ++q) {
                        ln[q] = s0 + PF + q < mine ? int(lp[int64_t(q) * lstep]) : 0;
                        if constexpr (STREAMS) stream(s0 + PF + q, xn[q], wn[q]);
                    }
                    lp += int64_t(PF) * lstep;
#pragma unroll
                    for (int q = 0; q < PF; ++q) {
                        if (s0 + q >= mine) break;
                        slot(lb[q], xb[q], wb[q], h + HT * (s0 + q));
                    }
#pragma unroll
                    for (int q = 0; q < PF; ++q) {
                        lb[q] = ln[q];
                        if constexpr (STREAMS)
#pragma unroll
                            for (int d = 0; d < D; ++d) { xb[q][d] = xn[q][d]; wb[q][d] = wn[q][d]; }
                    }
                }
            } else {
                static_assert(!STREAMS || GROUP > 0, "the streams come in groups");
                for (int s = 0; s < mine; ++s) {
                    const int l = lb[0];
#pragma unroll
                    for (int q = 0; q + 1 < PF; ++q) lb[q] = lb[q + 1];
                    lb[PF - 1] = s + PF < mine ? int(*lp) : 0;
                    lp += lstep;
                    slot(l, nullptr, nullptr, h + HT * s);
                }
            }
            blk.flush();
        } else if (need_ext) {
            for (int s = 0; s < mine; ++s) {
                const int l = lb[0];
#pragma unroll
                for (int q = 0; q + 1 < PF; ++q) lb[q] = lb[q + 1];
                lb[PF - 1] = s + PF < mine ? int(*lp) : 0;
                lp += lstep;
                float r[M];
                lds_words<M>(srow + l * W, r);
#pragma unroll
                for (int m = 0; m < M; ++m) { mn[m] = vmin(mn[m], r[m]); mx[m] = vmax(mx[m], r[m]); }
            }
        }
    }
    if constexpr (HT == 2) {
        __syncthreads();
        if (h == 1 && live) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                parts[pl].s[m] = acc.s[m];
                parts[pl].c[m] = acc.c[m];
                parts[pl].mn[m] = mn[m];
                parts[pl].mx[m] = mx[m];
            }
        }
        __syncthreads();
        if (h == 1) return;
    }
    bool f = false, rough = false;
    if (i >= 0) {
        if (a.g.bnd[i]) {
            float z[M];
#pragma unroll
            for (int m = 0; m < M; ++m) z[m] = 0.0f;
            store_vec<float, M>(a.K + i * M, z);
        } else {
            // the two compensated partials: their sum, minus both compensations and the rounding error of that sum
            float Kv[M];
#pragma unroll
            for (int m = 0; m < M; ++m) {
                if constexpr (HT == 1) {
                    Kv[m] = -acc.s[m];
                } else {
                    const float s1 = parts[pl].s[m];
                    const float u = acc.s[m] + s1;
                    const float cm = (u - acc.s[m]) - s1;
                    Kv[m] = -(u - ((acc.c[m] + parts[pl].c[m]) + cm));
                    mn[m] = vmin(mn[m], parts[pl].mn[m]);
                    mx[m] = vmax(mx[m], parts[pl].mx[m]);
                }
            }
            if (a.rough_words) {
                bool r = !need_ext;
#pragma unroll
                for (int m = 0; m < M; ++m) r = r || (mx[m] - mn[m]) > 1e-6f * (fabsf(mx[m]) + fabsf(mn[m]));
                rough = r;
            }
            f = stage_epilogue<float, D, M, PDE, 1>(a, i, fi, Kv, mn, mx);
        }
    }
    if (a.check) full_failures(a, i, f);
    if (a.rough_words) full_rough(a, i, rough);
}

// ----------------------------------------------------------------------------------- wide linear systems (FP32)
// Full flux pass of an FP32 linear system with many components (the 16-velocity kinetic model): a block takes a tile of
// HCC_TILE particles, stages the rows of its neighbour union in shared memory and gives every particle M / 4 lanes, four
// components each, half of the tile at a time. A row is 64 bytes of state and 128 of gradient, read about 20 times: with
// one thread per particle and the rows gathered through the caches, a thread held 112 numbers of state, gradient, sums
// and extrema (219 registers, two blocks an SM) and waited for the twelve loads of a slot that its index load had to
// precede. Here a lane holds a quarter of that, the rows come from shared memory, and the slot streams (place in the
// union, offsets, divergence weights: the FP32 streams of the stream-fed pass) do not depend on one another; the four
// lanes load one of a slot's four stream words each and exchange them, two slots ahead of the sums (four: 72 bytes
// spilled at three blocks an SM, 7883 us for two steps of 1.0 M particles against 6505; without spills at two: 6806).
template <int M> constexpr int wide_lanes() { return M / 4; }
template <typename T, int M, int PDE> constexpr bool wide_system() {
    return sizeof(T) == 4 && PDE != HCC_PDE_EULER && M >= 8 && M % 4 == 0 && 32 % (M / 4) == 0;
}
constexpr int kWideThreads = 256;
// the flux row: state, gradient, the order in the word after them
template <int D, int M> constexpr int wide_flux_row() { return 4 * tile_odd_groups(M + D * M + 1); }

// stage_epilogue for the four components `off` ... of the lanes of a particle; every lane of the warp calls it (the
// Maxwellian's sum and the flags cross the lanes), `live` marks those with a particle.
template <int D, int M, int PDE>
__device__ __forceinline__ bool wide_epilogue(const StageArgs<float> &a, int64_t i, int off, bool live, const float *fi,
                                              const float *Kv, const float *mn, const float *mx) {
    constexpr int L = wide_lanes<M>();
    const int64_t row = i * M + off;
    if (live) store_vec<float, 4>(a.K + row, Kv);
    if (!a.form_next) return false;
    float Y[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const StageCoeffs<float> *cf = live ? coef_of(a, i) : a.coef;
    if (live) {
        load_vec<float, 4>(a.Un + row, Y);
        for (int j = 0; j < a.n_prev; ++j) {
            const float hE = cf->hE[j], hI = cf->hI[j];
            if (hE != 0.0f) {
                float kv[4];
                if (j != a.self_slot) load_vec<float, 4>(a.KE[j] + row, kv);
#pragma unroll
                for (int m = 0; m < 4; ++m) Y[m] = Y[m] + hE * (j == a.self_slot ? Kv[m] : kv[m]);
            }
            if (hI != 0.0f) {
                float kv[4];
                load_vec<float, 4>(a.KI[j] + row, kv);
#pragma unroll
                for (int m = 0; m < 4; ++m) Y[m] = Y[m] + hI * kv[m];
            }
        }
    }
    if (a.implicit_mode) {
        float KIo[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if constexpr (PDE == HCC_PDE_BGK) {
            // the sum over all components in their order, handed from lane to lane (as maxwellian adds them)
            float u = ((Y[0] + Y[1]) + Y[2]) + Y[3];
#pragma unroll
            for (int s = 1; s < L; ++s) {
                const float before = __shfl_sync(0xffffffffu, u, s - 1, L);
                if (4 * s == off) u = (((before + Y[0]) + Y[1]) + Y[2]) + Y[3];
            }
            u = __shfl_sync(0xffffffffu, u, L - 1, L);
            const float dto = cf->dt_ii * a.ph.inv_eps, denom = 1.0f / (1.0f + dto), inv_dt_ii = cf->inv_dt_ii;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                float fd = (a.ph.a_macro[0] * u) * a.ph.sinv[off + m][0];
#pragma unroll
                for (int d = 1; d < D; ++d) fd = fd + (a.ph.a_macro[d] * u) * a.ph.sinv[off + m][d];
                const float Mk = a.ph.coeff * (u + fd);
                if (a.implicit_mode == 1) {
                    const float o = (Y[m] + dto * Mk) * denom;
                    KIo[m] = (o - Y[m]) * inv_dt_ii;
                    Y[m] = o;
                } else {
                    KIo[m] = (Mk - Y[m]) * a.ph.inv_eps;
                }
            }
        }
        if (live) store_vec<float, 4>(a.KInext + row, KIo);
    }
    if (live) store_vec<float, 4>(a.Ynext + row, Y);
    if (!a.check) return false;
    float cand[4];
    if (a.check_substep) {
        float ki[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (a.KIs && live) load_vec<float, 4>(a.KIs + row, ki);
#pragma unroll
        for (int m = 0; m < 4; ++m) cand[m] = fi[m] + cf->h_sub * (a.KIs ? Kv[m] + ki[m] : Kv[m]);
    } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) cand[m] = Y[m];
    }
    bool adm = true, flag = false;
    const float dl = a.delta, d3 = dl * dl * dl;
    constexpr float kPad = 16.0f * 1.1920928955078125e-7f;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        adm = adm && isfinite(cand[m]);
        const float pad = dl + kPad * vmax(fabsf(mn[m]), fabsf(mx[m]));
        bool v = fabsf(mx[m] - mn[m]) >= d3 && (cand[m] < mn[m] - pad || cand[m] > mx[m] + pad);
        if (a.sc.criterion == HCC_MOOD_U2 && v && a.u2_range) {
            const unsigned long long nanbits = a.u2_range[2 * M];
            const float range = ((nanbits >> (off + m)) & 1ull)
                                    ? float(NAN)
                                    : float(order_value(a.u2_range[M + off + m])) - float(order_value(a.u2_range[off + m]));
            v = !(mx[m] - mn[m] < a.u2_plateau * range);
        }
        flag = flag || v;
    }
    // over the particle's lanes
    const unsigned lanes = ((1u << L) - 1u) << ((threadIdx.x & 31u) / L * L);
    adm = (__ballot_sync(0xffffffffu, !adm) & lanes) == 0u;
    flag = (__ballot_sync(0xffffffffu, flag) & lanes) != 0u;
    if (live && off == 0) a.inadm[i] = !adm;
    if (!live) return false;
    if (a.sc.criterion == HCC_MOOD_ONLY || !adm) return true;
    return (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2) && flag;
}

// Reconstruction of a wide linear system (no limiter): L lanes a particle, four components each, as in the flux pass. A
// lane loads the index and weights of one of L slots and the lanes exchange them; the states of the next L slots (whole
// rows: a thread a particle took a quarter of a sector from each of 32 lines a load) and the stream words of the ones
// after are in flight while L slots are summed. 218 us against 241 on 1.0 M
// particles of 16 components.
template <int D, int M, int PDE> __device__ __noinline__ void gather_apart(const StageArgs<float> &a, int64_t i) {
    gather_one<float, D, M, PDE, 1, false>(a, i);  // (its registers are not the loop's)
}
template <int D, int M, int PDE>
__global__ void __launch_bounds__(kWideThreads, 4) k_gather_wide(const StageArgs<float> a) {
    constexpr int L = wide_lanes<M>();
    const int c = int(threadIdx.x) % L, off = 4 * c;
    const int64_t i = full_particle(a, (int64_t(blockIdx.x) * kWideThreads + threadIdx.x) / L);
    const bool live = i >= 0 && !a.g.bnd[i];
    const int64_t np = a.g.npad;
    bool cached = false;
    int cnt = 0;
    if (live) {
        cnt = a.g.cnt[i];
        int p = a.orders[i];
        while (p > 1 && cnt < basis_count(D, p - 1)) --p;
        cached = p == a.sc.max_order && p > 1 && a.g.ok_r[i];
        if (!cached && c == 0) gather_apart<D, M, PDE>(a, i);
    }
    if (!cached) cnt = 0;
    float fi[4] = {}, out[D][4] = {};
    if (cached) load_vec<float, 4>(a.U + i * M + off, fi);
    int32_t jn = 0;
    float gn[D];
    auto stream = [&](int k) {                     // slot k + c
        const bool on = k + c < cnt;
        jn = on ? a.g.nidx[int64_t(k + c) * np + i] : 0;
#pragma unroll
        for (int d = 0; d < D; ++d) gn[d] = on ? a.g.gw[(int64_t(k + c) * D + d) * np + i] : 0.0f;
    };
    float f[L][4], g[D];
    auto rows = [&](int k) {                       // the states of slots k ... of the words loaded last
#pragma unroll
        for (int d = 0; d < D; ++d) g[d] = gn[d];
#pragma unroll
        for (int s = 0; s < L; ++s) {
            const int32_t j = __shfl_sync(0xffffffffu, jn, s, L);
            if (k + s < cnt) load_vec<float, 4>(a.U + int64_t(j) * M + off, f[s]);
        }
    };
    const int kw = __reduce_max_sync(0xffffffffu, cnt);
    stream(0);
    rows(0);
    stream(L);
    for (int k = 0; k < kw; k += L) {
        float df[L][4], w[D];
#pragma unroll
        for (int d = 0; d < D; ++d) w[d] = g[d];
#pragma unroll
        for (int s = 0; s < L; ++s)
#pragma unroll
            for (int m = 0; m < 4; ++m) df[s][m] = f[s][m];
        rows(k + L);
        stream(k + 2 * L);
#pragma unroll
        for (int s = 0; s < L; ++s) {
            float ws[D];
#pragma unroll
            for (int d = 0; d < D; ++d) ws[d] = __shfl_sync(0xffffffffu, w[d], s, L);
            if (k + s < cnt) {
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const float dm = df[s][m] - fi[m];
#pragma unroll
                    for (int d = 0; d < D; ++d) out[d][m] = out[d][m] + ws[d] * dm;
                }
            }
        }
    }
    if (!cached) return;
    float *row = a.grad + i * grad_row<float, D * M>() + off;
#pragma unroll
    for (int d = 0; d < D; ++d) store_vec<float, 4>(row + d * M, out[d]);
}

// flux_one for a linear system on a fixed grid, degree-1 reconstruction. (The term of a slot from differences of the
// states, (cw + S) (f_ij - f_i) + (cw - S) (f_ji - f_i) with cw = sum_d w_d c_dm and S = sum_d w_d s_d max lambda_d, takes
// fewer instructions (700 against 865 us, both with four slots ahead) and rounds less; but MOOD then decides otherwise for a few candidates at a
// bound, which moves a state more than the rounding does.)
template <int D, int M, int PDE>
__global__ void __launch_bounds__(kWideThreads, 3) k_flux_wide(const StageArgs<float> a) {
    extern __shared__ __align__(16) float sm[];
    constexpr int L = wide_lanes<M>(), W = wide_flux_row<D, M>(), RG = (D + 1) * L;   // 16-byte groups of a row
    constexpr int G = 2, P = kWideThreads / L;     // slots a group, particles at a time
    static_assert(L == 2 * D, "one of a slot's 2 D offsets and weights a lane");
    __shared__ unsigned rough[HCC_TILE / 32];
    const int64_t t = blockIdx.x, u0 = a.tv.ustart[t], np = a.g.npad;
    const int nu = int(a.tv.ustart[t + 1] - u0);
    if (threadIdx.x < HCC_TILE / 32) rough[threadIdx.x] = 0u;
    for (int e = threadIdx.x; e < nu * RG; e += kWideThreads) {
        const int64_t j = a.tv.uid[u0 + e / RG];
        const int g = e % RG;
        float v[4];
        load_vec<float, 4>(g < L ? a.U + j * M + 4 * g : a.grad + j * (D * M) + 4 * (g - L), v);
        store_vec<float, 4>(sm + (e / RG) * W + 4 * g, v);
    }
    for (int e = threadIdx.x; e < nu; e += kWideThreads)
        sm[e * W + (D + 1) * M] = __int_as_float(int(a.orders[a.tv.uid[u0 + e]]));
    const int c = int(threadIdx.x) % L, off = 4 * c, lane0 = int(threadIdx.x & 31) - c;
    const bool need_ext = a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2);
    float cm[D][4];
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
        for (int m = 0; m < 4; ++m) cm[d][m] = a.ph.c[d][off + m];
    __syncthreads();
    for (int pl = int(threadIdx.x) / L; pl < HCC_TILE; pl += P) {
        const int64_t i = full_particle(a, t * HCC_TILE + pl);
        const bool bnd = i >= 0 && a.g.bnd[i];
        const bool live = i >= 0 && !bnd;
        float fi[4] = {0.0f, 0.0f, 0.0f, 0.0f}, mn[4], mx[4], Kv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (bnd) store_vec<float, 4>(a.K + i * M + off, Kv);
        const int cnt = live ? a.g.cnt[i] : 0;
        const bool wok = cnt > 0 && a.g.ok_d[i];
        // this lane's stream word of each slot, and the neighbour's place: the next group's in flight
        const float *sp = (c < D ? a.g.dist + int64_t(c) * np : a.g.dw + int64_t(c - D) * np) + i;
        const uint16_t *lp = a.tv.lidx + i;
        float v[G];
        int l[G];
#pragma unroll
        for (int q = 0; q < G; ++q) {
            v[q] = q < cnt ? sp[int64_t(q) * (D * np)] : 0.0f;
            l[q] = q < cnt ? int(lp[int64_t(q) * np]) : 0;
        }
        float gi[D][4] = {};
        int oi_own = 1;
        if (live) {
            const float *own = sm + int(a.tv.lself[i]) * W;
            oi_own = __float_as_int(own[(D + 1) * M]);
            load_vec<float, 4>(own + off, fi);
#pragma unroll
            for (int d = 0; d < D; ++d) load_vec<float, 4>(own + (d + 1) * M + off, gi[d]);
        }
        AccumV<float, 4> acc;
#pragma unroll
        for (int m = 0; m < 4; ++m) { mn[m] = fi[m]; mx[m] = fi[m]; }
        const int kw = __reduce_max_sync(0xffffffffu, cnt);
        for (int k0 = 0; k0 < kw; k0 += G) {
            sp += int64_t(G) * (D * np);
            lp += int64_t(G) * np;
            float vn[G];
            int ln[G];
#pragma unroll
            for (int q = 0; q < G; ++q) {
                vn[q] = k0 + G + q < cnt ? sp[int64_t(q) * (D * np)] : 0.0f;
                ln[q] = k0 + G + q < cnt ? int(lp[int64_t(q) * np]) : 0;
            }
#pragma unroll
            for (int q = 0; q < G; ++q) {
                float dk[D], wk[D];
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    dk[d] = __shfl_sync(0xffffffffu, v[q], lane0 + d);
                    wk[d] = __shfl_sync(0xffffffffu, v[q], lane0 + D + d);
                }
                if (k0 + q >= cnt) continue;
                const float *row = sm + l[q] * W;
                float fj[4];
                load_vec<float, 4>(row + off, fj);
                if (need_ext) {
#pragma unroll
                    for (int m = 0; m < 4; ++m) { mn[m] = vmin(mn[m], fj[m]); mx[m] = vmax(mx[m], fj[m]); }
                }
                if (!wok) continue;
                const int oj_own = __float_as_int(row[(D + 1) * M]);
                float gj[D][4];
#pragma unroll
                for (int d = 0; d < D; ++d) load_vec<float, 4>(row + (d + 1) * M + off, gj[d]);
                const bool epd1 = a.sc.strategy == HCC_EPD1;       // (EPD2 has no tile tables)
                const int lo = oi_own < oj_own ? oi_own : oj_own;
                const float si = (epd1 ? lo : oi_own) >= 2 ? 0.5f : 0.0f, sj = (epd1 ? lo : oj_own) >= 2 ? -0.5f : 0.0f;
                const bool below = a.sc.aligned && (a.sc.max_order == 1 || lo < a.sc.max_order);
                // the slot's term in flux_slot's form and order: the results keep the stream-fed pass's bits
                float sw[D], pi[D], pj[D], t[4];
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    sw[d] = (below ? wk[d] : dk[d]) > 0.0f ? a.ph.amax[d] : -a.ph.amax[d];
                    pi[d] = si * dk[d];
                    pj[d] = sj * dk[d];
                }
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    float ri = gi[0][m] * pi[0], rj = gj[0][m] * pj[0];
#pragma unroll
                    for (int d = 1; d < D; ++d) { ri = ri + gi[d][m] * pi[d]; rj = rj + gj[d][m] * pj[d]; }
                    const float fij = fi[m] + ri, fji = fj[m] + rj;
                    const float sum = (fij + fji) - 2.0f * fi[m], jump = fji - fij;
                    float tm = wk[0] * (cm[0][m] * sum - sw[0] * jump);
#pragma unroll
                    for (int d = 1; d < D; ++d) tm = tm + wk[d] * (cm[d][m] * sum - sw[d] * jump);
                    t[m] = tm;
                }
                acc.add(t);
            }
#pragma unroll
            for (int q = 0; q < G; ++q) { v[q] = vn[q]; l[q] = ln[q]; }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) Kv[m] = -acc.s[m];
        if (live && a.rough_words) {
            bool r = !need_ext;
#pragma unroll
            for (int m = 0; m < 4; ++m) r = r || (mx[m] - mn[m]) > 1e-6f * (fabsf(mx[m]) + fabsf(mn[m]));
            if (r) atomicOr(&rough[pl >> 5], 1u << (pl & 31));
        }
        if (wide_epilogue<D, M, PDE>(a, i, off, live, fi, Kv, mn, mx) && c == 0) list_failures(a, i, true);
    }
    if (!a.rough_words) return;
    __syncthreads();
    for (int pl = int(threadIdx.x); pl < HCC_TILE; pl += kWideThreads)      // (whole warps)
        full_rough(a, full_particle(a, t * HCC_TILE + pl), (rough[pl >> 5] >> (pl & 31)) & 1u);
}

// The opt-in shared-memory limit of a block on the current device (the tile passes' dynamic allocation may go up
// to it).
inline int tile_smem_optin() {
    int dev = 0, v = 48 * 1024;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

// Dynamic shared memory of the tile passes for the largest union.
template <int D, int M> inline size_t tile_gather_smem(int umax) {
    return (size_t(umax) * tile_gather_row<D, M>() + size_t(HCC_TILE) * D * M) * sizeof(float);
}
template <int D, int M> inline size_t tile_flux_smem(int umax) {
    return std::max(size_t(umax) * ((tile_flux_streams<D>() ? 1 : 4) + tile_flux_row<D, M>()) * sizeof(float),
                    size_t(tile_flux_threads<D>() - 1) * HCC_TILE * sizeof(FluxPart<float, M>));
}

// ----------------------------------------------------------------------------------- WENO (scalar)
// _cholesky_moment (Interpolators.jl:31-64) and C \ b for a fixed basis size B (FP64).
template <int B>
__device__ __forceinline__ bool chol_upper_fixed(const double *A, double *U) {
    for (int q = 0; q < B * B; ++q) U[q] = 0.0;
    for (int r = 0; r < B; ++r)
        for (int c = r; c < B; ++c) {
            double sm = A[r * B + c];
            for (int q = 0; q < r; ++q) sm = sm - U[q * B + r] * U[q * B + c];
            if (r == c) {
                if (!(sm > 0.0)) return false;
                U[r * B + r] = sqrt(sm);
            } else {
                U[r * B + c] = sm / U[r * B + r];
            }
        }
    return true;
}
template <int B>
__device__ __forceinline__ bool chol_moment_fixed(double *N, double *U) {
    bool ok = chol_upper_fixed<B>(N, U);
    if (ok) {
        for (int q = 0; q < B; ++q) {
            const double u = U[q * B + q];
            if (!(u * u > 10.0 * 2.220446049250313e-16 * N[q * B + q])) { ok = false; break; }
        }
    }
    if (ok) return true;
    double tr = 0.0;
    for (int q = 0; q < B; ++q) tr = tr + N[q * B + q];
    const double er = 1.4901161193847656e-08 * tr / double(B);
    for (int q = 0; q < B; ++q) N[q * B + q] = N[q * B + q] + er;
    return chol_upper_fixed<B>(N, U);
}
template <int B>
__device__ __forceinline__ void chol_solve_fixed(const double *U, const double *b, double *x) {
    double y[B];
    for (int r = 0; r < B; ++r) {
        double t = b[r];
        for (int q = 0; q < r; ++q) t = t - U[q * B + r] * y[q];
        y[r] = t / U[r * B + r];
    }
    for (int r = B - 1; r >= 0; --r) {
        double t = y[r];
        for (int q = r + 1; q < B; ++q) t = t - U[r * B + q] * x[q];
        x[r] = t / U[r * B + r];
    }
}

// _mls_solve_masked of degree Q (Interpolators.jl:412-443) over the slots of particle i, all of them (dsel < 0) or
// the one-sided stencil along axis dsel: side 1 x_d < 0, side 2 x_d >= 0 (WENO's upwind sides), side 3 x_d <= 0
// (Tiwari's upwind side for v_d > 0), of the per-particle field g (fi = its value at i); out[0..D) = the
// first-derivative coefficients (scaled by invL). Returns the factorisation status (out = 0 when it fails).
template <typename T, int D, int Q, typename Field>
__device__ bool weno_fit_f(const StageArgs<T> &a, int64_t i, int cnt, int dsel, int side, double fi, Field g,
                           double *out) {
    constexpr int B = ExpTable<D, Q>::B;
    const int64_t np = a.g.npad;
    double N[B * B], bs[B];
    for (int q = 0; q < B * B; ++q) N[q] = 0.0;
    for (int q = 0; q < B; ++q) bs[q] = 0.0;
    for (int k = 0; k < cnt; ++k) {
        if (dsel >= 0) {
            const double dd = double(a.g.dist[(int64_t(k) * D + dsel) * np + i]);
            if (!(side == 1 ? dd < 0.0 : side == 2 ? dd >= 0.0 : dd <= 0.0)) continue;
        }
        const int64_t s = int64_t(k) * np + i;
        double x[D], p[B];
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = double(a.g.dist[(int64_t(k) * D + d) * np + i]) * a.g.invL64;
        table_basis<D, Q, double>(x, p);
        const double w = double(a.g.wt[s]);
        const double df = g(int64_t(a.g.nidx[s])) - fi;
        for (int r = 0; r < B; ++r)
            for (int c = 0; c < B; ++c) N[r * B + c] = N[r * B + c] + w * (p[r] * p[c]);
        for (int r = 0; r < B; ++r) bs[r] = bs[r] + w * (p[r] * df);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) out[d] = 0.0;
    double U[B * B], xs[B];
    if (!chol_moment_fixed<B>(N, U)) return false;
    chol_solve_fixed<B>(U, bs, xs);
#pragma unroll
    for (int d = 0; d < D; ++d) out[d] = xs[d] * a.g.invL64;   // degree-1 scale factors
    return true;
}

template <typename T, int D, int Q>
__device__ bool weno_fit(const StageArgs<T> &a, int64_t i, int cnt, int dsel, int side, double fi, double *out) {
    return weno_fit_f<T, D, Q>(a, i, cnt, dsel, side, fi, [&a](int64_t j) { return double(a.U[j]); }, out);
}

template <typename T, int D>
__device__ __forceinline__ void weno_fit_q(int q, const StageArgs<T> &a, int64_t i, int cnt, int dsel, int side,
                                           double fi, double *out) {
    if (q == 1) weno_fit<T, D, 1>(a, i, cnt, dsel, side, fi, out);
    else if (q == 2) weno_fit<T, D, 2>(a, i, cnt, dsel, side, fi, out);
    else weno_fit<T, D, 3>(a, i, cnt, dsel, side, fi, out);
}

// Position of the upper-triangle entry (r, c), r <= c, of a B x B matrix stored packed by rows.
template <int B> __host__ __device__ constexpr int packed_upper(int r, int c) { return r * B - r * (r - 1) / 2 + (c - r); }
// chol_solve_fixed with the factor packed: the same entries, the same operations in the same order.
template <int B>
__device__ __forceinline__ void chol_solve_packed(const double *U, const double *b, double *x) {
    double y[B];
    for (int r = 0; r < B; ++r) {
        double t = b[r];
        for (int q = 0; q < r; ++q) t = t - U[packed_upper<B>(q, r)] * y[q];
        y[r] = t / U[packed_upper<B>(r, r)];
    }
    for (int r = B - 1; r >= 0; --r) {
        double t = y[r];
        for (int q = r + 1; q < B; ++q) t = t - U[packed_upper<B>(r, q)] * x[q];
        x[r] = t / U[packed_upper<B>(r, r)];
    }
}

// weno_fit_f with the moment matrix's Cholesky factor taken from the geometry pass (k_weno_geom64: the same matrix,
// the same factorisation): only the right-hand side is summed here, in the same order, so the fit is bit for bit
// that of weno_fit_f.
template <typename T, int D, int Q, typename Field>
__device__ bool weno_fit_cached(const StageArgs<T> &a, int64_t i, int cnt, int dsel, int side, double fi, Field g,
                                const double *Up, bool ok, double *out) {
    constexpr int B = ExpTable<D, Q>::B;
    const int64_t np = a.g.npad;
    double bs[B];
    for (int q = 0; q < B; ++q) bs[q] = 0.0;
    for (int k = 0; k < cnt; ++k) {
        if (dsel >= 0) {
            const double dd = double(a.g.dist[(int64_t(k) * D + dsel) * np + i]);
            if (!(side == 1 ? dd < 0.0 : side == 2 ? dd >= 0.0 : dd <= 0.0)) continue;
        }
        const int64_t s = int64_t(k) * np + i;
        double x[D], p[B];
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = double(a.g.dist[(int64_t(k) * D + d) * np + i]) * a.g.invL64;
        table_basis<D, Q, double>(x, p);
        const double w = double(a.g.wt[s]);
        const double df = g(int64_t(a.g.nidx[s])) - fi;
        for (int r = 0; r < B; ++r) bs[r] = bs[r] + w * (p[r] * df);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) out[d] = 0.0;
    if (!ok) return false;
    double xs[B];
    chol_solve_packed<B>(Up, bs, xs);
#pragma unroll
    for (int d = 0; d < D; ++d) out[d] = xs[d] * a.g.invL64;
    return true;
}

// The WENO functor (WENO.jl:55-165): central fit over the whole stencil and one upwind one-sided fit per axis,
// blended with w_S = 1 / (1 + (a_S / a_C)^2) on smoothness indicators IS = Σ_d (∂_d u)^2 h^2 normalised by
// max(u_i^2, IS_C); the result is Σ_d v_d ∂_d u and K_E = -that. Fits in FP64 in both paths.
template <typename T, int D>
__device__ __forceinline__ bool weno_one(const StageArgs<T> &a, const int64_t i) {
    if (a.g.bnd[i]) {
        if (a.full) a.K[i] = T(0);
        return false;
    }
    const int cnt = a.g.cnt[i];
    const int64_t np = a.g.npad;
    const T fiT = a.U[i];
    T mn = fiT, mx = fiT;
    if (a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2))
        for (int k = 0; k < cnt; ++k) {
            const T fj = a.U[a.g.nidx[int64_t(k) * np + i]];
            mn = vmin(mn, fj);
            mx = vmax(mx, fj);
        }
    const double fi = double(fiT);
    double div_total = 0.0;
    int p_order = a.orders[i];
    while (p_order > 1 && cnt < basis_count(D, p_order)) --p_order;
    if (cnt >= basis_count(D, p_order)) {
        const int DO = a.sc.DO;
        const double dx2 = a.g.h64 * a.g.h64;
        double resC[D];
        weno_fit_q<T, D>(DO == 0 ? p_order : (DO < p_order ? DO : p_order), a, i, cnt, -1, 0, fi, resC);
        double smoothC = (resC[0] * resC[0]) * dx2;
#pragma unroll
        for (int d = 1; d < D; ++d) smoothC = smoothC + (resC[d] * resC[d]) * dx2;
        double s2 = jmax(fi * fi, smoothC);
        s2 = s2 > 0.0 ? s2 : 1.0;
        const double aC = smoothC / s2 + 1e-12;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const double vel = double(a.ph.c[d][0]);
            const bool use_left = vel > 0.0;
            int stencil = 0;
            for (int k = 0; k < cnt; ++k) {
                const double dd = double(a.g.dist[(int64_t(k) * D + d) * np + i]);
                stencil += (use_left && dd < 0.0) || (!use_left && dd >= 0.0);
            }
            int p_d = p_order;
            while (p_d > 1 && stencil < basis_count(D, p_d)) --p_d;
            if (stencil < basis_count(D, p_d)) {
                div_total = div_total + resC[d] * vel;
                continue;
            }
            double resS[D];
            weno_fit_q<T, D>(DO == 0 ? p_d : (DO < p_d ? DO : p_d), a, i, cnt, d, use_left ? 1 : 2, fi, resS);
            double smoothS = (resS[0] * resS[0]) * dx2;
#pragma unroll
            for (int e = 1; e < D; ++e) smoothS = smoothS + (resS[e] * resS[e]) * dx2;
            const double q = (smoothS / s2 + 1e-12) / aC;
            const double wS = 1.0 / (1.0 + q * q);
            const double wC = 1.0 - wS;
            const double div_d = wS * resS[d] + wC * resC[d];
            div_total = div_total + div_d * vel;
        }
    }
    const T Kv = T(-div_total);
    return stage_epilogue<T, D, 1, HCC_PDE_ADVECTION>(a, i, &fiT, &Kv, &mn, &mx);
}

// A full pass or a worklist pass over tiles, as the MUSCL flux pass.
template <typename T, int D>
__global__ void __launch_bounds__(128) k_weno(const StageArgs<T> a) {
    const int lane = int(threadIdx.x & 31);
    if (a.full) {
        const int64_t i = full_particle(a, int64_t(blockIdx.x) * blockDim.x + threadIdx.x);
        const bool f = (i >= 0) ? weno_one<T, D>(a, i) : false;
        if (a.check) full_failures(a, i, f);
        return;
    }
    const unsigned nt = *a.wcount;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned q = warp; q < nt; q += nwarps) {
        const int32_t tile = a.wtiles[q];
        const uint32_t word = a.wmask[tile];
        const int64_t i = int64_t(tile) * 32 + lane;
        const bool f = ((word >> lane) & 1u) ? weno_one<T, D>(a, i) : false;
        if (a.check) tile_failures(a, tile, f);
        if (lane == 0 && a.clear_wmask) a.wmask[tile] = 0u;
    }
}

template <typename T, int D, typename Field>
__device__ __forceinline__ void weno_fit_qf(int q, const StageArgs<T> &a, int64_t i, int cnt, int dsel, int side,
                                            double fi, Field g, double *out) {
    if (q == 1) weno_fit_f<T, D, 1>(a, i, cnt, dsel, side, fi, g, out);
    else weno_fit_f<T, D, 2>(a, i, cnt, dsel, side, fi, g, out);
}

// Component-wise meshless WENO of a system (an extension of the scalar functor WENO.jl:55-165, which the reference
// defines for M = 1 only), orders 1 and 2: the central and one-sided fits, smoothness indicators and weights of the
// scalar scheme applied to one field at a time. Linear fluxes F_d(U)_m = c_dm U_m (advection, the kinetic model):
// field U_m, upwind side by the sign of c_dm, divergence sum_d c_dm d_d U_m. Euler: local Lax-Friedrichs splitting
// F_d^+- = (F_d(U) +- alpha_d U) / 2 with alpha_d the largest lambda_d over {i} u N(i); d_d F_d^+ from the
// left-biased one-sided fit (x_d < 0), d_d F_d^- from the right-biased one (x_d >= 0). Fits in FP64 in both paths.
template <typename T, int D, int M, int PDE>
__device__ __forceinline__ bool weno_sys_one(const StageArgs<T> &a, const int64_t i) {
    if (a.g.bnd[i]) {
        if (a.full) {
            T z[M];
#pragma unroll
            for (int m = 0; m < M; ++m) z[m] = T(0);
            store_vec<T, M>(a.K + i * M, z);
        }
        return false;
    }
    const int cnt = a.g.cnt[i];
    const int64_t np = a.g.npad;
    T fiT[M], mn[M], mx[M];
    load_vec<T, M>(a.U + i * M, fiT);
#pragma unroll
    for (int m = 0; m < M; ++m) mn[m] = mx[m] = fiT[m];
    if (a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2))
        for (int k = 0; k < cnt; ++k) {
            const int64_t j = a.g.nidx[int64_t(k) * np + i];
#pragma unroll
            for (int m = 0; m < M; ++m) { mn[m] = vmin(mn[m], a.U[j * M + m]); mx[m] = vmax(mx[m], a.U[j * M + m]); }
        }
    double div[M];
#pragma unroll
    for (int m = 0; m < M; ++m) div[m] = 0.0;
    int p_order = a.orders[i];
    while (p_order > 1 && cnt < basis_count(D, p_order)) --p_order;
    if (cnt >= basis_count(D, p_order)) {
        const int DO = a.sc.DO;
        const double dx2 = a.g.h64 * a.g.h64;
        const int qC = DO == 0 ? p_order : (DO < p_order ? DO : p_order);
        // fit degree of the one-sided stencil of axis d (side 1: x_d < 0, side 2: x_d >= 0), 0 when too small
        auto one_sided = [&](int d, int side) {
            int stencil = 0;
            if (a.g.wcnt) {
                stencil = a.g.wcnt[i * (2 * D) + 2 * d + side - 1];
            } else {
                for (int k = 0; k < cnt; ++k) {
                    const double dd = double(a.g.dist[(int64_t(k) * D + d) * np + i]);
                    stencil += side == 1 ? (dd < 0.0) : (dd >= 0.0);
                }
            }
            int p_d = p_order;
            while (p_d > 1 && stencil < basis_count(D, p_d)) --p_d;
            if (stencil < basis_count(D, p_d)) return 0;
            return DO == 0 ? p_d : (DO < p_d ? DO : p_d);
        };
        auto smooth = [&](const double *r) {
            double sm = (r[0] * r[0]) * dx2;
#pragma unroll
            for (int d = 1; d < D; ++d) sm = sm + (r[d] * r[d]) * dx2;
            return sm;
        };
        if constexpr (PDE != HCC_PDE_EULER) {
            for (int m = 0; m < M; ++m) {
                auto g = [&a, m](int64_t j) { return double(a.U[j * M + m]); };
                const double fi = double(fiT[m]);
                double resC[D];
                weno_fit_qf<T, D>(qC, a, i, cnt, -1, 0, fi, g, resC);
                const double smoothC = smooth(resC);
                double s2 = jmax(fi * fi, smoothC);
                s2 = s2 > 0.0 ? s2 : 1.0;
                const double aC = smoothC / s2 + 1e-12;
                double div_total = 0.0;
                for (int d = 0; d < D; ++d) {
                    const double vel = double(a.ph.c[d][m]);
                    const int side = vel > 0.0 ? 1 : 2;
                    const int qS = one_sided(d, side);
                    if (qS == 0) {
                        div_total = div_total + resC[d] * vel;
                        continue;
                    }
                    double resS[D];
                    weno_fit_qf<T, D>(qS, a, i, cnt, d, side, fi, g, resS);
                    const double smoothS = smooth(resS);
                    const double q = (smoothS / s2 + 1e-12) / aC;
                    const double wS = 1.0 / (1.0 + q * q);
                    const double wC = 1.0 - wS;
                    const double div_d = wS * resS[d] + wC * resC[d];
                    div_total = div_total + div_d * vel;
                }
                div[m] = div_total;
            }
        } else {
            const double gamma = double(a.ph.gamma), gm1 = double(a.ph.gm1);
            // Euler primitives and lambda_d of a state in FP64 (euler_prim and speeds, operation for operation)
            auto prim = [gm1](const double *Uj, double &inv_rho, double *u, double &p) {
                const double rho = Uj[0];
                inv_rho = 1.0 / rho;
                double q2 = 0.0;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    u[d] = Uj[1 + d] * inv_rho;
                    q2 = (d == 0) ? u[d] * u[d] : q2 + u[d] * u[d];
                }
                p = gm1 * (Uj[D + 1] - 0.5 * (rho * q2));
            };
            auto lam = [&](const double *Uj, int d) {
                double inv_rho, u[D], p;
                prim(Uj, inv_rho, u, p);
                return fabs(u[d]) + sqrt(gamma * p * inv_rho);
            };
            double Ui[M];
#pragma unroll
            for (int m = 0; m < M; ++m) Ui[m] = double(fiT[m]);
            // with the geometry pass's factors and this stage's flux table (k_weno_prep64): the same values, each
            // computed once instead of once per fit
            const bool cached = a.g.wchol != nullptr && a.wflux64 != nullptr;
            constexpr int FW = D * (M + 1);                 // flux table row: F_d(U)_m then lambda_d, per axis
            double alpha[D];
            for (int d = 0; d < D; ++d) {
                alpha[d] = cached ? a.wflux64[i * FW + d * (M + 1) + M] : lam(Ui, d);
                for (int k = 0; k < cnt; ++k) {
                    const int64_t j = a.g.nidx[int64_t(k) * np + i];
                    if (cached) {
                        alpha[d] = jmax(alpha[d], a.wflux64[j * FW + d * (M + 1) + M]);
                        continue;
                    }
                    double Uj[M];
#pragma unroll
                    for (int m = 0; m < M; ++m) Uj[m] = double(a.U[j * M + m]);
                    alpha[d] = jmax(alpha[d], lam(Uj, d));
                }
            }
            constexpr int B2 = cbasis_count(D, 2), PK = B2 * (B2 + 1) / 2, NS = 2 * D + 1;
            auto fit = [&](int q, int dsel, int side, double fi, auto g, double *res) {
                if (!cached) {
                    weno_fit_qf<T, D>(q, a, i, cnt, dsel, side, fi, g, res);
                    return;
                }
                const int st = dsel < 0 ? 0 : 1 + 2 * dsel + side - 1;
                const int64_t slot = (i * 2 + (q - 1)) * NS + st;
                if (q == 1) weno_fit_cached<T, D, 1>(a, i, cnt, dsel, side, fi, g, a.g.wchol + slot * PK, a.g.wok[slot], res);
                else weno_fit_cached<T, D, 2>(a, i, cnt, dsel, side, fi, g, a.g.wchol + slot * PK, a.g.wok[slot], res);
            };
            for (int d = 0; d < D; ++d)
                for (int sg = 0; sg < 2; ++sg) {
                    const int side = sg == 0 ? 1 : 2;
                    const int qS = one_sided(d, side);
                    for (int m = 0; m < M; ++m) {
                        // F_d^+-(U_j)_m, the physical flux component as flux_and_speed forms it
                        auto g = [&a, &prim, &alpha, d, m, sg, cached](int64_t j) {
                            double F, Ujm;
                            if (cached) {
                                F = a.wflux64[j * FW + d * (M + 1) + m];
                                Ujm = double(a.U[j * M + m]);
                            } else {
                                double Uj[M];
#pragma unroll
                                for (int c = 0; c < M; ++c) Uj[c] = double(a.U[j * M + c]);
                                double inv_rho, u[D], p;
                                prim(Uj, inv_rho, u, p);
                                if (m == 0) F = Uj[1 + d];
                                else if (m <= D) F = (m - 1 == d) ? Uj[m] * u[d] + p : Uj[m] * u[d];
                                else F = (Uj[D + 1] + p) * u[d];
                                Ujm = Uj[m];
                            }
                            const double aU = alpha[d] * Ujm;
                            return sg == 0 ? 0.5 * (F + aU) : 0.5 * (F - aU);
                        };
                        const double fi = g(i);
                        double resC[D];
                        fit(qC, -1, 0, fi, g, resC);
                        double deriv = resC[d];
                        if (qS > 0) {
                            const double smoothC = smooth(resC);
                            double s2 = jmax(fi * fi, smoothC);
                            s2 = s2 > 0.0 ? s2 : 1.0;
                            const double aC = smoothC / s2 + 1e-12;
                            double resS[D];
                            fit(qS, d, side, fi, g, resS);
                            const double smoothS = smooth(resS);
                            const double q = (smoothS / s2 + 1e-12) / aC;
                            const double wS = 1.0 / (1.0 + q * q);
                            const double wC = 1.0 - wS;
                            deriv = wS * resS[d] + wC * resC[d];
                        }
                        div[m] = div[m] + deriv;
                    }
                }
        }
    }
    T Kv[M];
#pragma unroll
    for (int m = 0; m < M; ++m) Kv[m] = T(-div[m]);
    return stage_epilogue<T, D, M, PDE>(a, i, fiT, Kv, mn, mx);
}

template <typename T, int D, int M, int PDE>
__global__ void __launch_bounds__(128) k_weno_sys(const StageArgs<T> a) {
    const int lane = int(threadIdx.x & 31);
    if (a.full) {
        const int64_t i = full_particle(a, int64_t(blockIdx.x) * blockDim.x + threadIdx.x);
        const bool f = (i >= 0) ? weno_sys_one<T, D, M, PDE>(a, i) : false;
        if (a.check) full_failures(a, i, f);
        return;
    }
    const unsigned nt = *a.wcount;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned q = warp; q < nt; q += nwarps) {
        const int32_t tile = a.wtiles[q];
        const uint32_t word = a.wmask[tile];
        const int64_t i = int64_t(tile) * 32 + lane;
        const bool f = ((word >> lane) & 1u) ? weno_sys_one<T, D, M, PDE>(a, i) : false;
        if (a.check) tile_failures(a, tile, f);
        if (lane == 0 && a.clear_wmask) a.wmask[tile] = 0u;
    }
}

// UpwindDivergence (Upwind.jl), scalar advection, first order. Tiwari (:158-202): per axis d the gradient fit on
// the upwind side v_d x_d <= 0 (order lowered while that side has fewer than basis_count(D, p) points; an axis
// without enough contributes 0), summed as v_d (d_d u). Praveen (:205-249, 2-D): from the moment matrix
// N = sum w (x/L)(x/L)^T, per slot c = N^-1 (w x/L) / L, the edge normal n and tangent s, the coefficient
// (n . c) min(v . n, 0) + min((s . c)(v . s), 0) on u_j - u_i, summed and doubled. K_E = -that. FP64 fits.
template <typename T, int D, int ALG>
__device__ __forceinline__ bool upwind_one(const StageArgs<T> &a, const int64_t i) {
    if (a.g.bnd[i]) {
        if (a.full) a.K[i] = T(0);
        return false;
    }
    const int cnt = a.g.cnt[i];
    const int64_t np = a.g.npad;
    const T fiT = a.U[i];
    T mn = fiT, mx = fiT;
    if (a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2))
        for (int k = 0; k < cnt; ++k) {
            const T fj = a.U[a.g.nidx[int64_t(k) * np + i]];
            mn = vmin(mn, fj);
            mx = vmax(mx, fj);
        }
    const double fi = double(fiT);
    double total = 0.0;
    if constexpr (ALG == HCC_UPWIND_TIWARI) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const double vel = double(a.ph.c[d][0]);
            int stencil = 0;
            for (int k = 0; k < cnt; ++k)
                stencil += vel * double(a.g.dist[(int64_t(k) * D + d) * np + i]) <= 0.0;
            int p_d = a.orders[i];
            while (p_d > 1 && stencil < basis_count(D, p_d)) --p_d;
            if (stencil < basis_count(D, p_d)) continue;
            const int q = a.sc.DO == 0 ? p_d : (a.sc.DO < p_d ? a.sc.DO : p_d);
            // v_d x_d <= 0: x_d <= 0 for v_d > 0, x_d >= 0 for v_d < 0, every slot for v_d = 0
            double res[D];
            weno_fit_q<T, D>(q, a, i, cnt, vel == 0.0 ? -1 : d, vel > 0.0 ? 3 : 2, fi, res);
            total = total + res[d] * vel;
        }
    } else if constexpr (D == 2) {
        if (cnt >= 3 && a.g.h64 >= 1e-14) {
            const double iL = a.g.invL64;
            const double vx = double(a.ph.c[0][0]), vy = double(a.ph.c[1][0]);
            double n11 = 0.0, n12 = 0.0, n22 = 0.0;
            for (int k = 0; k < cnt; ++k) {
                const double w = double(a.g.wt[int64_t(k) * np + i]);
                const double x = double(a.g.dist[(int64_t(k) * 2) * np + i]) * iL;
                const double y = double(a.g.dist[(int64_t(k) * 2 + 1) * np + i]) * iL;
                n11 = n11 + w * (x * x);
                n12 = n12 + w * (x * y);
                n22 = n22 + w * (y * y);
            }
            const double det = n11 * n22 - n12 * n12;
            const double tr = n11 + n22;
            if (!(fabs(det) <= 4.0 * 2.220446049250313e-16 * (tr * tr))) {
                double div = 0.0;
                for (int k = 0; k < cnt; ++k) {
                    const double w = double(a.g.wt[int64_t(k) * np + i]);
                    const double dx = double(a.g.dist[(int64_t(k) * 2) * np + i]);
                    const double dy = double(a.g.dist[(int64_t(k) * 2 + 1) * np + i]);
                    const double bx = w * dx * iL, by = w * dy * iL;
                    const double cx = ((n22 * bx - n12 * by) / det) * iL;
                    const double cy = ((n11 * by - n12 * bx) / det) * iL;
                    const double hyp = sqrt(dx * dx + dy * dy);
                    double nx = 1.0, ny = 0.0;
                    if (!(hyp <= 2.220446049250313e-16 * a.g.h64)) { nx = dx / hyp; ny = dy / hyp; }
                    const double sx = -ny, sy = nx;
                    const double alfa = nx * cx + ny * cy;
                    const double beta = sx * cx + sy * cy;
                    const double vn = vx * nx + vy * ny;
                    const double vs = vx * sx + vy * sy;
                    const double bv = beta * vs;
                    const double cij = alfa * (vn < 0.0 ? vn : 0.0) + (bv < 0.0 ? bv : 0.0);
                    div = div + cij * (double(a.U[a.g.nidx[int64_t(k) * np + i]]) - fi);
                }
                total = 2.0 * div;
            }
        }
    }
    const T Kv = T(-total);
    return stage_epilogue<T, D, 1, HCC_PDE_ADVECTION>(a, i, &fiT, &Kv, &mn, &mx);
}

template <typename T, int D, int ALG>
__global__ void __launch_bounds__(128) k_upwind(const StageArgs<T> a) {
    const int lane = int(threadIdx.x & 31);
    if (a.full) {
        const int64_t i = full_particle(a, int64_t(blockIdx.x) * blockDim.x + threadIdx.x);
        const bool f = (i >= 0) ? upwind_one<T, D, ALG>(a, i) : false;
        if (a.check) full_failures(a, i, f);
        return;
    }
    const unsigned nt = *a.wcount;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned q = warp; q < nt; q += nwarps) {
        const int32_t tile = a.wtiles[q];
        const uint32_t word = a.wmask[tile];
        const int64_t i = int64_t(tile) * 32 + lane;
        const bool f = ((word >> lane) & 1u) ? upwind_one<T, D, ALG>(a, i) : false;
        if (a.check) tile_failures(a, tile, f);
        if (lane == 0 && a.clear_wmask) a.wmask[tile] = 0u;
    }
}

// CentralDivergence (Central.jl:45-88): the particle's order, lowered while it has fewer than basis_count(D, p) + 1
// neighbours (zero divergence if even order 1 lacks them), capped by div_order, selects the degree-q intercept fit
// of the flux differences F(f_j) - F(f_i); its per-slot weights (the geometry cache) are applied slot by slot.
// K_E = -div; the MOOD check of the next candidate runs in the shared epilogue.
template <typename T, int D, int M, int PDE>
__device__ __forceinline__ bool central_one(const StageArgs<T> &a, const int64_t i) {
    if (a.g.bnd[i]) {
        if (a.full) {
            T z[M];
#pragma unroll
            for (int m = 0; m < M; ++m) z[m] = T(0);
            store_vec<T, M>(a.K + i * M, z);
        }
        return false;
    }
    const int cnt = a.g.cnt[i];
    const int64_t np = a.g.npad;
    T fi[M], mn[M], mx[M];
    load_vec<T, M>(a.U + i * M, fi);
#pragma unroll
    for (int m = 0; m < M; ++m) mn[m] = mx[m] = fi[m];
    const bool ext = a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2);
    int p = a.orders[i];
    while (p > 1 && cnt < basis_count(D, p) + 1) --p;
    const int q = a.sc.DO == 0 ? p : (a.sc.DO < p ? a.sc.DO : p);
    const T *wq = (cnt >= basis_count(D, p) + 1 && a.g.okc[q - 1][i]) ? a.g.dwc[q - 1] : nullptr;
    T Fi[D][M], lam[D], div[M];
    flux_and_speed<T, D, M, PDE>(a.ph, fi, Fi, lam);
#pragma unroll
    for (int m = 0; m < M; ++m) div[m] = T(0);
    for (int k = 0; k < cnt; ++k) {
        const int64_t j = a.g.nidx[int64_t(k) * np + i];
        T fj[M];
        load_vec<T, M>(a.U + j * M, fj);
        if (ext) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                mn[m] = vmin(mn[m], fj[m]);
                mx[m] = vmax(mx[m], fj[m]);
            }
        }
        if (wq) {
            T Fj[D][M], lj[D];
            flux_and_speed<T, D, M, PDE>(a.ph, fj, Fj, lj);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const T c = wq[(int64_t(k) * D + d) * np + i];
#pragma unroll
                for (int m = 0; m < M; ++m) div[m] = div[m] + c * (Fj[d][m] - Fi[d][m]);
            }
        }
    }
    T Kv[M];
#pragma unroll
    for (int m = 0; m < M; ++m) Kv[m] = -div[m];
    return stage_epilogue<T, D, M, PDE>(a, i, fi, Kv, mn, mx);
}

// Whether full passes go over the interior list: in FP64, whose unit bounds them. The FP32 pass waits for its slot streams,
// which a list takes out of step with the warps: 3-D Euler at 343k interior and 109k ghosts 948 us a step over the list,
// 934 over all particles; FP64 at 47k and 30k 1990 and 2619.
template <typename T> constexpr bool central_lists() { return sizeof(T) == 8; }

// A full pass or a worklist pass over tiles (the changed particles: no order reach), as the MUSCL flux pass.
template <typename T, int D, int M, int PDE>
__global__ void __launch_bounds__(128) k_central(const StageArgs<T> a) {
    const int lane = int(threadIdx.x & 31);
    if (a.full) {
        const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
        if constexpr (central_lists<T>()) {
            const int64_t i = full_particle(a, q);
            const bool f = (i >= 0) ? central_one<T, D, M, PDE>(a, i) : false;
            if (a.check) full_failures(a, i, f);
        } else {
            const bool f = (q < a.g.n) ? central_one<T, D, M, PDE>(a, q) : false;
            if (a.check) tile_failures(a, q >> 5, f);
        }
        return;
    }
    const unsigned nt = *a.wcount;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned q = warp; q < nt; q += nwarps) {
        const int32_t tile = a.wtiles[q];
        const uint32_t word = a.wmask[tile];
        const int64_t i = int64_t(tile) * 32 + lane;
        const bool f = ((word >> lane) & 1u) ? central_one<T, D, M, PDE>(a, i) : false;
        if (a.check) tile_failures(a, tile, f);
        if (lane == 0 && a.clear_wmask) a.wmask[tile] = 0u;
    }
}

// The start of a step: orders, flags, worklist counts and statistics reset, and form_candidate!(ts, eq, pg, 1, dt, t)
// (TimeSteppers.jl:365-397) for stage 1: Y_1 = Uⁿ (interior; then the implicit part) and the boundary conditions of the
// boundary (apply_boundary_conditions!, BoundaryConditions.jl:43-130): the donor's start-of-step state or their own.
// (Stages whose implicit part changes Y_1 take the donors' states from a pass after this one.) One launch: the three
// resets, the fill, the copy and the boundary pass it replaces were about 2 us each in a step's graph.
template <typename T, int D, int M, int PDE, int RDEG>
__global__ void k_stage1(const StageArgs<T> a) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i == 0) {
        *a.lists = ListCounts{};
        *a.stats = MoodStats{};
    }
    if (i >= a.g.n) return;
    a.orders[i] = int8_t(a.sc.max_order);
    a.trig_step[i] = 0;
    const bool bnd = a.g.bnd[i];
    const int32_t root = bnd ? a.root[i] : -1;
    T Y[M];
    load_vec<T, M>(a.Un + (root >= 0 ? int64_t(root) : i) * M, Y);
    if (!bnd && a.implicit_mode) {
        T KIo[M];
        implicit_part<T, D, M, PDE>(a, i, Y, KIo);
        store_vec<T, M>(a.KInext + i * M, KIo);
    }
    store_vec<T, M>(a.Ynext + i * M, Y);
}

// Spacing of the speed table's rows: whole vectors.
template <int D> constexpr int lam_stride() { return D == 3 ? 4 : D; }

// s + x with the rounding error of the sum kept in c (FP32 CFL sums: a group of slots at a time). A sum that overflows stays
// infinite (there is no error to keep): its step is zero, not unbounded.
template <typename T> __device__ __forceinline__ void compensated(T &s, T &c, T x) {
    const T y = x - c, u = s + y, e = (u - s) - y;
    c = isfinite(e) ? e : T(0);
    s = u;
}

// The axis speeds of every particle's state (Euler), for k_cfl: a speed takes a division and a square root, and every
// particle is a neighbour about 20 (2-D) or 66 (3-D) times.
template <typename T, int D, int M, int PDE>
__global__ void k_speeds(const StageArgs<T> a) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.g.n) return;
    constexpr int LS = lam_stride<D>();
    T U[M], L[LS];
    load_vec<T, M>(a.U + i * M, U);
#pragma unroll
    for (int d = 0; d < LS; ++d) L[d] = T(0);
    speeds<T, D, M, PDE>(a.ph, U, L);
    store_vec<T, LS>(a.lam + i * LS, L);
}

// _cfl_weights_body! (ParticleGrids.jl:439-450) + the minimum over particles (:414). Bound by the slot streams; the
// neighbours' speeds come from the table of k_speeds (Euler) or are constants (linear fluxes), and a group of slots is
// in flight at once. The sum runs over the slots in order; in FP32 a group at a time, compensated (the step's error against
// 64 bits 4.1e-8 rms instead of 8.0e-8 on 70^2 points, 5.8e-8 instead of 1.27e-7 on 31^3, at the same time). With the
// table: FP64 3-D, 103k particles, 117 us (723 with the speeds recomputed in every slot); FP64 2-D, 68k, 31 us (122);
// FP32 2-D, 1.01M, 83 us (107). FP32: five blocks an SM leave a group's loads their registers (3-D stream-fed, the call on
// 33k / 373k interior particles: 30 / 114 us, 51 / 163 with the 32 registers of the unbounded kernel).
template <typename T, int D, int M, int PDE, int RDEG>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 256 : 1024, sizeof(T) == 4 ? 5 : 1) k_cfl(const StageArgs<T> a, unsigned long long *dt_bits) {
    const int64_t i = full_particle(a, int64_t(blockIdx.x) * blockDim.x + threadIdx.x);
    double dti = INFINITY;
    if (i >= 0 && !a.g.bnd[i]) {
        const int cnt = a.g.cnt[i];
        if (cnt > 0) {
            constexpr int LS = lam_stride<D>(), G = 4;
            constexpr bool kTable = PDE == HCC_PDE_EULER;
            const int64_t np = a.g.npad;
            T Li[LS];
            if constexpr (kTable) load_vec<T, LS>(a.lam + i * LS, Li);
            T sum_c = T(0), comp = T(0);
            for (int k0 = 0; k0 < cnt; k0 += G) {
                T w[G][D], Lj[G][LS], part = T(0);
#pragma unroll
                for (int q = 0; q < G; ++q) {
                    const int k = k0 + q < cnt ? k0 + q : cnt - 1;
#pragma unroll
                    for (int d = 0; d < D; ++d) w[q][d] = a.g.dw[(int64_t(k) * D + d) * np + i];
                    if constexpr (kTable)
                        load_vec<T, LS>(a.lam + int64_t(a.g.nidx[int64_t(k) * np + i]) * LS, Lj[q]);
                }
#pragma unroll
                for (int q = 0; q < G; ++q) {
                    T dot = T(0);
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        T top;
                        if constexpr (kTable) top = vmax(Li[d], Lj[q][d]);
                        else top = a.ph.amax[d];
                        const T pr = fabs(w[q][d]) * top;
                        dot = (d == 0) ? pr : dot + pr;
                    }
                    if constexpr (sizeof(T) == 4) part = part + (k0 + q < cnt ? dot : T(0));
                    else if (k0 + q < cnt) sum_c = sum_c + dot;
                }
                if constexpr (sizeof(T) == 4) compensated(sum_c, comp, part);
            }
            if (sum_c > floatmin_of<T>()) dti = double((T(1) / T(D)) / sum_c);
        }
    }
    // positive doubles order like their bit patterns
    unsigned long long b = __double_as_longlong(dti);
    int cl = 0;
    bool whole_warp = true;
    if (a.cloud_id) {   // one minimum per cloud of a batch (a warp straddling two clouds: one atomic per lane)
        cl = i >= 0 ? a.cloud_id[i] : -1;
        whole_warp = __match_any_sync(0xffffffffu, cl) == 0xffffffffu;
        if (!whole_warp) {
            if (cl >= 0) atomicMin(dt_bits + cl, b);
            return;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long ob = __shfl_down_sync(0xffffffffu, b, o);
        b = ob < b ? ob : b;
    }
    if ((threadIdx.x & 31) == 0 && cl >= 0) atomicMin(dt_bits + cl, b);
}

// The CFL step of an FP32 context with tile tables (the same formula as k_cfl): per tile of HCC_TILE particles the
// union's quantised positions and the axis speeds of its states are staged in shared memory, one speed evaluation per
// union entry instead of one per slot, and each slot reads only its neighbour's union place; the slot offsets and
// divergence weights are recomputed from the positions and the particle's fit rows as in the tile flux pass. Two
// threads per particle (alternate slots, the second's partial sum through shared memory), the per-particle loads
// issued before the staging, every staging load of a thread in flight at once, union places in groups of four. One
// minimum for the whole cloud (batches with a minimum per cloud take k_cfl).
template <int D, int M, int PDE>
__global__ void __launch_bounds__(2 * HCC_TILE) k_cfl_tile(const StageArgs<float> a, unsigned long long *dt_bits) {
    extern __shared__ __align__(16) float sm[];
    int4 *spos = reinterpret_cast<int4 *>(sm);
    float4 *sspd = reinterpret_cast<float4 *>(sm + 4 * a.tv.umax);
    float *parts = sm + 8 * a.tv.umax;           // [HCC_TILE] partial sums of the second threads
    const int64_t t = blockIdx.x;
    const int64_t u0 = a.tv.ustart[t];
    const int nu = int(a.tv.ustart[t + 1] - u0);
    const int pl = int(threadIdx.x) % HCC_TILE, h = int(threadIdx.x) / HCC_TILE;
    const int64_t i = full_particle(a, t * HCC_TILE + pl);
    const int64_t np = a.g.npad;
    constexpr int PF = 4;
    const int64_t lstep = 2 * np;
    const uint16_t *lp = a.tv.lidx + int64_t(h) * np + i;
    int li = 0, mine = 0;
    int lb[PF];
    float A[D], B[D][D];
    if (i >= 0 && !a.g.bnd[i]) {
        const int cnt = a.g.cnt[i];
        if (cnt > 0 && a.g.ok_d[i]) {
            li = int(a.tv.lself[i]);
            const float *cf = a.tv.coef + i * a.tv.cw;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                A[d] = cf[d];
#pragma unroll
                for (int e = 0; e < D; ++e) B[d][e] = cf[D + d * D + e];
            }
            mine = cnt > h ? (cnt - h + 1) / 2 : 0;
#pragma unroll
            for (int q = 0; q < PF; ++q) lb[q] = q < mine ? int(lp[int64_t(q) * lstep]) : 0;
            lp += int64_t(PF) * lstep;
        }
    }
    {
        constexpr int SU = 4;
        const int nt = int(blockDim.x);
        for (int e0 = threadIdx.x; e0 < nu; e0 += SU * nt) {
            int32_t jj[SU];
#pragma unroll
            for (int u = 0; u < SU; ++u) jj[u] = e0 + u * nt < nu ? a.tv.uid[u0 + e0 + u * nt] : 0;
            int4 qq[SU];
            float U[SU][M];
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                if (e0 + u * nt >= nu) break;
                qq[u] = a.tv.upos[u0 + e0 + u * nt];
#pragma unroll
                for (int m = 0; m < M; ++m) U[u][m] = a.U[int64_t(jj[u]) * M + m];
            }
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                if (e0 + u * nt >= nu) break;
                float L[D];
                speeds<float, D, M, PDE>(a.ph, U[u], L);
                spos[e0 + u * nt] = qq[u];
                sspd[e0 + u * nt] = make_float4(L[0], D > 1 ? L[D > 1 ? 1 : 0] : 0.0f,
                                                D > 2 ? L[D > 2 ? 2 : 0] : 0.0f, 0.0f);
            }
        }
    }
    __syncthreads();
    float sum_c = 0.0f, comp = 0.0f;
    if (mine > 0) {
        const int4 q4 = spos[li];
        const int qi[3] = {q4.x, q4.y, q4.z};
        const float4 l4 = sspd[li];
        const float Li[3] = {l4.x, l4.y, l4.z};
        const float qt = a.tv.quantum[t], ws = a.tv.wscale;
        auto slot = [&](const int l, float &part) {
            const int4 qj4 = spos[l];
            const int qj[3] = {qj4.x, qj4.y, qj4.z};
            const float4 lj4 = sspd[l];
            const float Lj[3] = {lj4.x, lj4.y, lj4.z};
            float dk[D];
            tile_offset<D>(qj, qi, qt, dk);
            float r2 = dk[0] * dk[0];
#pragma unroll
            for (int d = 1; d < D; ++d) r2 = r2 + dk[d] * dk[d];
            const float w = tile_weight(r2, ws);
            float dot = 0.0f;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                float v = A[d];
#pragma unroll
                for (int e = 0; e < D; ++e) v = v + B[d][e] * dk[e];
                const float pr = fabsf(w * v) * jmax(Li[d], Lj[d]);
                dot = (d == 0) ? pr : dot + pr;
            }
            part = part + dot;
        };
        // groups of PF union places, the next group in flight while this one is summed (the slot body unrolled)
        for (int s0 = 0; s0 < mine; s0 += PF) {
            int ln[PF];
#pragma unroll
            for (int q = 0; q < PF; ++q) ln[q] = s0 + PF + q < mine ? int(lp[int64_t(q) * lstep]) : 0;
            lp += int64_t(PF) * lstep;
            float part = 0.0f;
#pragma unroll
            for (int q = 0; q < PF; ++q) {
                if (s0 + q >= mine) break;
                slot(lb[q], part);
            }
            compensated(sum_c, comp, part);
#pragma unroll
            for (int q = 0; q < PF; ++q) lb[q] = ln[q];
        }
    }
    if (h == 1) parts[pl] = sum_c - comp;
    __syncthreads();
    if (h == 1) return;
    double dti = INFINITY;
    if (i >= 0 && !a.g.bnd[i]) {
        sum_c = (sum_c - comp) + parts[pl];
        if (sum_c > floatmin_of<float>()) dti = double((1.0f / float(D)) / sum_c);
    }
    // positive doubles order like their bit patterns
    unsigned long long b = __double_as_longlong(dti);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long ob = __shfl_down_sync(0xffffffffu, b, o);
        b = ob < b ? ob : b;
    }
    if ((threadIdx.x & 31) == 0) atomicMin(dt_bits, b);
}

// ----------------------------------------------------------------------------------- FP32 meshless WENO of Euler
// The fits of the component-wise WENO (weno_sys_one) are linear in the fitted field: out_s = sum_k c_{s,k} df_k with
// c_{s,k} = invL R_s (w_k p_k), R_s the first D rows of the inverse moment matrix of stencil s (the central stencil
// and, per axis, the slots with x_d < 0 and with x_d >= 0). The moment matrices depend on the geometry only: this
// pass assembles and factorises them once in FP64 (degree 2; the degree-1 matrix is its leading block, the same
// products), and stores R_s for both degrees in FP32, with the one-sided stencil sizes. A failed factorisation
// stores zeros (the fit returns zero, as in weno_fit_f).
template <int D>
__global__ void k_weno_geom(const WenoGeomArgs g) {
    constexpr int B1 = cbasis_count(D, 1), B2 = cbasis_count(D, 2), NS = 2 * D + 1;
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    float *out = g.ops + i * int64_t(2 * NS * D * B2);
    for (int q = 0; q < 2 * NS * D * B2; ++q) out[q] = 0.0f;
    if (g.bnd[i]) return;
    const int cnt = g.cnt[i];
    const int64_t np = g.npad;
    for (int st = 0; st < NS; ++st) {
        const int dsel = st == 0 ? -1 : (st - 1) / 2, side = st == 0 ? 0 : 1 + (st - 1) % 2;
        double N[B2 * B2];
        for (int q = 0; q < B2 * B2; ++q) N[q] = 0.0;
        int members = 0;
        for (int k = 0; k < cnt; ++k) {
            if (dsel >= 0) {
                const double dd = g.dist[(int64_t(k) * D + dsel) * np + i];
                if (!(side == 1 ? dd < 0.0 : dd >= 0.0)) continue;
            }
            ++members;
            double x[D], p[B2];
#pragma unroll
            for (int d = 0; d < D; ++d) x[d] = g.dist[(int64_t(k) * D + d) * np + i] * g.invL64;
            table_basis<D, 2, double>(x, p);
            const double w = g.w[int64_t(k) * np + i];
            for (int r = 0; r < B2; ++r)
                for (int c = r; c < B2; ++c) N[r * B2 + c] = N[r * B2 + c] + w * (p[r] * p[c]);
        }
        for (int r = 1; r < B2; ++r)
            for (int c = 0; c < r; ++c) N[r * B2 + c] = N[c * B2 + r];
        if (st > 0) g.wcnt[i * (2 * D) + (st - 1)] = members;
        {   // degree 1: the leading block
            double N1[B1 * B1], U1[B1 * B1];
            for (int r = 0; r < B1; ++r)
                for (int c = 0; c < B1; ++c) N1[r * B1 + c] = N[r * B2 + c];
            if (chol_moment_fixed<B1>(N1, U1)) {
                float *o = out + (0 * NS + st) * D * B2;
                for (int b = 0; b < B1; ++b) {
                    double e[B1], xs[B1];
                    for (int r = 0; r < B1; ++r) e[r] = r == b ? 1.0 : 0.0;
                    chol_solve_fixed<B1>(U1, e, xs);
#pragma unroll
                    for (int d = 0; d < D; ++d) o[d * B2 + b] = float(xs[d] * g.invL64);
                }
            }
        }
        {   // degree 2
            double U2[B2 * B2];
            if (chol_moment_fixed<B2>(N, U2)) {
                float *o = out + (1 * NS + st) * D * B2;
                for (int b = 0; b < B2; ++b) {
                    double e[B2], xs[B2];
                    for (int r = 0; r < B2; ++r) e[r] = r == b ? 1.0 : 0.0;
                    chol_solve_fixed<B2>(U2, e, xs);
#pragma unroll
                    for (int d = 0; d < D; ++d) o[d * B2 + b] = float(xs[d] * g.invL64);
                }
            }
        }
    }
}

// The FP64 path's counterpart of k_weno_geom: the same masked moment matrices (upper triangles, the same products
// in the same order), factorised by chol_moment_fixed as weno_fit_f does at every stage, stored packed with their
// flags; and the one-sided stencil sizes. weno_sys_one then sums only the right-hand sides.
template <int D>
__global__ void k_weno_geom64(const WenoGeomArgs g) {
    constexpr int B1 = cbasis_count(D, 1), B2 = cbasis_count(D, 2), NS = 2 * D + 1;
    constexpr int PK = B2 * (B2 + 1) / 2;
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    double *out = g.chol + i * int64_t(2 * NS * PK);
    uint8_t *okf = g.ok + i * int64_t(2 * NS);
    for (int q = 0; q < 2 * NS * PK; ++q) out[q] = 0.0;
    for (int q = 0; q < 2 * NS; ++q) okf[q] = 0;
    if (g.bnd[i]) return;
    const int cnt = g.cnt[i];
    const int64_t np = g.npad;
    for (int st = 0; st < NS; ++st) {
        const int dsel = st == 0 ? -1 : (st - 1) / 2, side = st == 0 ? 0 : 1 + (st - 1) % 2;
        double N[B2 * B2];
        for (int q = 0; q < B2 * B2; ++q) N[q] = 0.0;
        int members = 0;
        for (int k = 0; k < cnt; ++k) {
            if (dsel >= 0) {
                const double dd = g.dist[(int64_t(k) * D + dsel) * np + i];
                if (!(side == 1 ? dd < 0.0 : dd >= 0.0)) continue;
            }
            ++members;
            double x[D], p[B2];
#pragma unroll
            for (int d = 0; d < D; ++d) x[d] = g.dist[(int64_t(k) * D + d) * np + i] * g.invL64;
            table_basis<D, 2, double>(x, p);
            const double w = g.w[int64_t(k) * np + i];
            for (int r = 0; r < B2; ++r)
                for (int c = r; c < B2; ++c) N[r * B2 + c] = N[r * B2 + c] + w * (p[r] * p[c]);
        }
        if (st > 0) g.wcnt[i * (2 * D) + (st - 1)] = members;
        {   // degree 1: the leading block (the degree-1 basis is the degree-2 basis's first B1 terms)
            double N1[B1 * B1], U1[B1 * B1];
            for (int r = 0; r < B1; ++r)
                for (int c = 0; c < B1; ++c) N1[r * B1 + c] = N[r * B2 + c];
            const bool ok = chol_moment_fixed<B1>(N1, U1);
            okf[0 * NS + st] = ok;
            double *o = out + (0 * NS + st) * PK;
            for (int r = 0; r < B1; ++r)
                for (int c = r; c < B1; ++c) o[packed_upper<B1>(r, c)] = U1[r * B1 + c];
        }
        {   // degree 2
            double U2[B2 * B2];
            const bool ok = chol_moment_fixed<B2>(N, U2);
            okf[1 * NS + st] = ok;
            double *o = out + (1 * NS + st) * PK;
            for (int r = 0; r < B2; ++r)
                for (int c = r; c < B2; ++c) o[packed_upper<B2>(r, c)] = U2[r * B2 + c];
        }
    }
}

// The FP64 flux table of one stage for weno_sys_one: per particle F_d(U)_m and lambda_d, each by the same
// operations as the fits' field functions compute them.
template <int D>
__global__ void k_weno_prep64(const StageArgs<double> a) {
    constexpr int M = D + 2, FW = D * (M + 1);
    const int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= a.g.n) return;
    const double gamma = double(a.ph.gamma), gm1 = double(a.ph.gm1);
    double Uj[M];
#pragma unroll
    for (int m = 0; m < M; ++m) Uj[m] = double(a.U[j * M + m]);
    const double rho = Uj[0];
    const double inv_rho = 1.0 / rho;
    double u[D], q2 = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        u[d] = Uj[1 + d] * inv_rho;
        q2 = (d == 0) ? u[d] * u[d] : q2 + u[d] * u[d];
    }
    const double p = gm1 * (Uj[D + 1] - 0.5 * (rho * q2));
    double *row = a.wflux64 + j * FW;
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            double F;
            if (m == 0) F = Uj[1 + d];
            else if (m <= D) F = (m - 1 == d) ? Uj[m] * u[d] + p : Uj[m] * u[d];
            else F = (Uj[D + 1] + p) * u[d];
            row[d * (M + 1) + m] = F;
        }
        row[d * (M + 1) + M] = fabs(u[d]) + sqrt(gamma * p * inv_rho);
    }
}

// The component-wise WENO of weno_sys_one for Euler in FP32 with the cached operators. One pass over the slots
// accumulates, with the central operator and per axis d the operator of the slot's side, the gradients of the
// differences U_j,m - U_i,m and F_d(U_j)_m - F_d(U_i)_m and the largest lambda_d of the stencil (alpha_d); the split
// fields F_d^+- = (F_d +- alpha_d U) / 2 are linear in those, so their central and one-sided gradients, smoothness
// indicators and WENO weights follow without another pass. Same degree and stencil rules as weno_sys_one.
// M lanes share a particle (30 of a warp's 32 in 3-D). In a round each forms the operator coefficients and the
// primitives of one slot and leaves them as a record in shared memory; then each sums its variable m over the round's
// records, in slot order. A thread a particle kept 90 sums of one axis (223 registers, 8 warps an SM, 35 % of the issue
// slots used), formed the basis, the primitives and the central coefficients once per axis, and ran both sides'
// branches: 740 us against 517 us for the full pass over 104 k particles, 129 against 45 us for a short
// list.
constexpr int kWenoWarps = 4, kWenoRec = 36;      // warps a block; words of a record (an odd number of 16-byte groups)
// Operator rows of a particle in shared memory, each padded to 16-byte groups, an odd number of them in all.
template <int D> constexpr int weno_op_words() { return (D * cbasis_count(D, 2) + 3) / 4 * 4; }
template <int D> constexpr int weno_op_row() { return 4 * (((2 * D + 1) * weno_op_words<D>() / 4) | 1); }
template <int D> struct WenoShared {
    static constexpr int P = 32 / (D + 2);        // particles a warp
    __align__(16) float ops[kWenoWarps * P * weno_op_row<D>()];
    __align__(16) float rec[kWenoWarps * 32 * kWenoRec];
};

// The warp's particles: i of this lane's group (-1: none), c its lane in the group, `ops` and `rec` the group's operator
// rows and records, `mine` this lane's record. Every lane of the warp calls it. True on the first lane of a failed candidate's group.
template <int D>
__device__ __forceinline__ bool weno_euler_lanes(const StageArgs<float> &a, const int64_t i, const int c, float *ops,
                                                 const float *rec, float *mine) {
    constexpr int M = D + 2, B2 = cbasis_count(D, 2), NS = 2 * D + 1, R = D * B2, RP = weno_op_words<D>();
    // a record: cC[D], the internal energy e (p = (gamma - 1) e) at 3; u[D] at 4; per axis the D coefficients of side 1, then of side 2 (the slot's own side,
    // zeros for the other) from 8; rho at 26; rho u[D], E from 28
    constexpr int CS = 8, RHO = 26, MOM = 28;
    static_assert(CS + 2 * D * D <= RHO && MOM + D < kWenoRec, "record layout");
    const bool bnd = i >= 0 && a.g.bnd[i];
    const bool live = i >= 0 && !bnd;
    if (bnd && a.full) a.K[i * M + c] = 0.0f;
    const int64_t np = a.g.npad;
    const int cnt = live ? a.g.cnt[i] : 0;
    const bool need_ext = a.check && (a.sc.criterion == HCC_MOOD_U1 || a.sc.criterion == HCC_MOOD_U2);
    const int DO = a.sc.DO;
    int p_order = 1;
    bool fit = false;
    unsigned sided = 0u;                          // the one-sided fits there are (bit 2 d + side - 1)
    if (live) {
        p_order = a.orders[i];
        while (p_order > 1 && cnt < basis_count(D, p_order)) --p_order;
        fit = cnt >= basis_count(D, p_order);
    }
    if (fit) {
        const int qC = DO == 0 ? p_order : (DO < p_order ? DO : p_order);
        const float *src = a.g.wops + i * int64_t(2 * NS * R) + (qC - 1) * NS * R;
        for (int q = c; q < R; q += M) ops[q] = src[q];
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
            for (int sg = 0; sg < 2; ++sg) {
                const int stencil = a.g.wcnt[i * (2 * D) + 2 * d + sg];
                int p_d = p_order;
                while (p_d > 1 && stencil < basis_count(D, p_d)) --p_d;
                const int qd = stencil < basis_count(D, p_d) ? 0 : DO == 0 ? p_d : (DO < p_d ? DO : p_d);
                if (qd > 0) sided |= 1u << (2 * d + sg);
                const int st = 1 + 2 * d + sg;
                const float *from = a.g.wops + i * int64_t(2 * NS * R) + ((qd > 0 ? qd - 1 : 0) * NS + st) * R;
                for (int q = c; q < R; q += M) ops[st * RP + q] = from[q];
            }
    }
    // this lane's variable: its own value and fluxes. F_d(U)_m = v_d s + (m == 1 + d ? p : 0) with v = rho u, s = 1 for
    // the density and v = u, s = U_m (+ p for the energy) for the others; p = (gamma - 1) e enters both sums by a fused
    // multiply-add. (Rounded on its own first, it costs 0.9 to 2 % more error of the right-hand side on 24^3 and 46^3
    // points: p is the largest term of the momentum flux. The same time: 1685 and 1679 us a step on 46^3.)
    float alpha[D], Uim = 0.0f, Fi[D], g_momentum[D];
    const float g_energy = c == M - 1 ? a.ph.gm1 : 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        alpha[d] = Fi[d] = 0.0f;
        g_momentum[d] = c == 1 + d ? a.ph.gm1 : 0.0f;
    }
    if (live) {
        float Ui[M], inv_rho, u_i[D];
        load_vec<float, M>(a.U + i * M, Ui);
        const float e_i = euler_internal<float, D>(Ui, inv_rho, u_i);
        const float c_i = root(a.ph.gamma * (a.ph.gm1 * e_i) * inv_rho);
#pragma unroll
        for (int m = 0; m < M; ++m) Uim = c == m ? Ui[m] : Uim;
        const float s = c == 0 ? 1.0f : __fmaf_rn(g_energy, e_i, Uim);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            alpha[d] = fabsf(u_i[d]) + c_i;
            Fi[d] = __fmaf_rn(g_momentum[d], e_i, __fmul_rn(c == 0 ? Ui[1 + d] : u_i[d], s));
        }
    }
    float gCU[D], gCF[D][D], gSU[D][2][D], gSF[D][2][D], mn = Uim, mx = Uim;
#pragma unroll
    for (int e = 0; e < D; ++e) {
        gCU[e] = 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            gCF[d][e] = 0.0f;
            gSU[d][0][e] = gSU[d][1][e] = gSF[d][0][e] = gSF[d][1][e] = 0.0f;
        }
    }
    // the stream words of the next round, and its states, are in flight while a round is summed
    int32_t jn = 0;
    float xn[D], wn = 0.0f, Un[M];
    auto stream = [&](int k) {
        const int64_t s = int64_t(k) * np + i;
        jn = a.g.nidx[s];
        wn = a.g.wt[s];
#pragma unroll
        for (int e = 0; e < D; ++e) xn[e] = a.g.dist[(int64_t(k) * D + e) * np + i];
    };
    if (c < cnt) {
        stream(c);
        load_vec<float, M>(a.U + int64_t(jn) * M, Un);
    }
    const float *vec = rec + (c == 0 ? MOM : 4), *val = rec + (c == 0 ? RHO : MOM + c - 1);
    const int kw = __reduce_max_sync(0xffffffffu, cnt);
    __syncwarp();
    for (int k0 = 0; k0 < kw; k0 += M) {
        const int k = k0 + c;
        if (k < cnt) {
            mine[RHO] = Un[0];
            sts_words<D + 1>(mine + MOM, Un + 1);
        }
        if (k < cnt && fit) {
            float inv_rho, u[4] = {}, cp[4] = {}, x[D], pb[B2], o[RP];
            cp[3] = euler_internal<float, D>(Un, inv_rho, u);
            const float cs = root(a.ph.gamma * (a.ph.gm1 * cp[3]) * inv_rho);
#pragma unroll
            for (int d = 0; d < D; ++d) alpha[d] = vmax(alpha[d], fabsf(u[d]) + cs);
            sts_words<4>(mine + 4, u);
#pragma unroll
            for (int e = 0; e < D; ++e) x[e] = xn[e] * a.g.invL;
            table_basis<D, 2, float>(x, pb);
#pragma unroll
            for (int b = 0; b < B2; ++b) pb[b] = wn * pb[b];
            lds_words<RP>(ops, o);
#pragma unroll
            for (int e = 0; e < D; ++e) {
                float v = 0.0f;
#pragma unroll
                for (int b = 0; b < B2; ++b) v = v + o[e * B2 + b] * pb[b];
                cp[e] = v;
            }
            sts_words<4>(mine, cp);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const bool left = x[d] < 0.0f;
                float *at = mine + CS + 2 * D * d;
                lds_words<RP>(ops + (left ? 1 + 2 * d : 2 + 2 * d) * RP, o);
#pragma unroll
                for (int e = 0; e < D; ++e) {
                    float v = 0.0f;
#pragma unroll
                    for (int b = 0; b < B2; ++b) v = v + o[e * B2 + b] * pb[b];
                    at[e] = left ? v : 0.0f;
                    at[D + e] = left ? 0.0f : v;
                }
            }
        } else {                                   // past the end (or no fit): no contribution
            const float zero[RHO] = {};
            sts_words<CS + 2 * D * D>(mine, zero);
            if (k >= cnt) {
                mine[RHO] = 0.0f;
                sts_words<D + 1>(mine + MOM, zero);
            } else {
                mine[RHO] = Un[0];
            }
        }
        if (k + M < cnt) {
            stream(k + M);
            load_vec<float, M>(a.U + int64_t(jn) * M, Un);
        }
        __syncwarp();
#pragma unroll 1
        for (int s = 0; s < M; ++s) {
            const float *r = rec + s * kWenoRec;
            float cp[4], v[D], cs[2 * D * D];
            lds_words<4>(r, cp);
            lds_words<D>(vec + s * kWenoRec, v);
            lds_words<2 * D * D>(r + CS, cs);
            const float Um = val[s * kWenoRec], e_j = cp[3];
            const float dU = Um - Uim, sc = c == 0 ? 1.0f : __fmaf_rn(g_energy, e_j, Um);
            if (need_ext && k0 + s < cnt) { mn = vmin(mn, Um); mx = vmax(mx, Um); }
            float dF[D];
#pragma unroll
            for (int d = 0; d < D; ++d) dF[d] = __fmaf_rn(g_momentum[d], e_j, __fmul_rn(v[d], sc)) - Fi[d];
#pragma unroll
            for (int e = 0; e < D; ++e) {
                gCU[e] = gCU[e] + cp[e] * dU;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    gCF[d][e] = gCF[d][e] + cp[e] * dF[d];
#pragma unroll
                    for (int sg = 0; sg < 2; ++sg) {
                        const float w = cs[2 * D * d + D * sg + e];
                        gSU[d][sg][e] = gSU[d][sg][e] + w * dU;
                        gSF[d][sg][e] = gSF[d][sg][e] + w * dF[d];
                    }
                }
            }
        }
        __syncwarp();
    }
    // alpha_d of the group
#pragma unroll
    for (int d = 0; d < D; ++d) mine[d] = alpha[d];
    __syncwarp();
#pragma unroll
    for (int s = 0; s < M; ++s)
#pragma unroll
        for (int d = 0; d < D; ++d) alpha[d] = vmax(alpha[d], rec[s * kWenoRec + d]);
    __syncwarp();
    float div = 0.0f;
    if (fit) {
        const float dx2 = float(a.g.h64 * a.g.h64);
        // the split fields F_d^+ (side 1: x_d < 0) and F_d^- (side 2)
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
            for (int sg = 0; sg < 2; ++sg) {
                const float sgn = sg == 0 ? 1.0f : -1.0f;
                const float fi = 0.5f * (Fi[d] + sgn * alpha[d] * Uim);
                float gC[D];
#pragma unroll
                for (int e = 0; e < D; ++e) gC[e] = 0.5f * (gCF[d][e] + sgn * alpha[d] * gCU[e]);
                float deriv = gC[d];
                if ((sided >> (2 * d + sg)) & 1u) {
                    float smoothC = (gC[0] * gC[0]) * dx2;
#pragma unroll
                    for (int e = 1; e < D; ++e) smoothC = smoothC + (gC[e] * gC[e]) * dx2;
                    float s2 = vmax(fi * fi, smoothC);
                    s2 = s2 > 0.0f ? s2 : 1.0f;
                    const float aC = smoothC / s2 + 1e-12f;
                    float gS[D];
#pragma unroll
                    for (int e = 0; e < D; ++e) gS[e] = 0.5f * (gSF[d][sg][e] + sgn * alpha[d] * gSU[d][sg][e]);
                    float smoothS = (gS[0] * gS[0]) * dx2;
#pragma unroll
                    for (int e = 1; e < D; ++e) smoothS = smoothS + (gS[e] * gS[e]) * dx2;
                    const float qq = (smoothS / s2 + 1e-12f) / aC;
                    const float wS = 1.0f / (1.0f + qq * qq);
                    deriv = wS * gS[d] + (1.0f - wS) * gC[d];
                }
                div = div + deriv;
            }
    }
    // the epilogue takes all variables in one lane
    mine[0] = -div;
    mine[1] = mn;
    mine[2] = mx;
    __syncwarp();
    bool f = false;
    if (live && c == 0) {
        float Ui[M], Kv[M], lo[M], hi[M];
        load_vec<float, M>(a.U + i * M, Ui);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            Kv[m] = rec[m * kWenoRec];
            lo[m] = rec[m * kWenoRec + 1];
            hi[m] = rec[m * kWenoRec + 2];
        }
        f = stage_epilogue<float, D, M, HCC_PDE_EULER>(a, i, Ui, Kv, lo, hi);
    }
    __syncwarp();
    return f;
}

// A full pass: consecutive particles to a block, P to a warp; a worklist pass: a block takes a listed tile and its warps
// P of the members at a time.
template <int D>
__global__ void __launch_bounds__(32 * kWenoWarps, 4) k_weno_euler_f32(const StageArgs<float> a) {
    constexpr int M = D + 2, P = WenoShared<D>::P;
    __shared__ WenoShared<D> sh;
    const int warp = int(threadIdx.x) >> 5, lane = int(threadIdx.x & 31), g = lane / M, c = lane % M;
    const bool on = g < P;                        // (two lanes of a warp have no particle in 1-D and 3-D)
    float *ops = sh.ops + (warp * P + (on ? g : 0)) * weno_op_row<D>();
    float *mine = sh.rec + (warp * 32 + lane) * kWenoRec;
    const float *rec = sh.rec + (warp * 32 + (on ? g * M : 0)) * kWenoRec;
    if (a.full) {
        const int64_t i = on ? full_particle(a, (int64_t(blockIdx.x) * kWenoWarps + warp) * P + g) : -1;
        const bool f = weno_euler_lanes<D>(a, i, c, ops, rec, mine);
        if (a.check) list_failures(a, i, f);
        return;
    }
    const unsigned nt = *a.wcount;
    for (unsigned q = blockIdx.x; q < nt; q += gridDim.x) {
        const int32_t tile = a.wtiles[q];
        const uint32_t word = a.wmask[tile];
        const int members = __popc(word);
        for (int m0 = warp * P; m0 < members; m0 += kWenoWarps * P) {
            uint32_t rest = word;                 // without its first m0 + g members
            for (int b = 0; b < m0 + g; ++b) rest &= rest - 1u;
            const int64_t i = on && rest ? int64_t(tile) * 32 + (__ffs(int(rest)) - 1) : -1;
            const bool f = weno_euler_lanes<D>(a, i, c, ops, rec, mine);
            if (a.check) list_failures(a, i, f);
        }
        __syncthreads();                          // every warp has read the word
        if (threadIdx.x == 0 && a.clear_wmask) a.wmask[tile] = 0u;
    }
}

// ----------------------------------------------------------------------------------- launchers / registry
template <typename T, int D, int M, int PDE, int RDEG>
struct StageInst {
    static unsigned grid(int64_t n, int bs) { return unsigned((n + bs - 1) / bs); }
    static unsigned pass_grid(const StageArgs<T> &a, int bs) {
        const unsigned g = std::max(1u, grid(a.nfull, bs));
        return a.full ? g : std::max(1u, std::min(g, unsigned(a.list_blocks)));
    }
    // blocks of an FP32 split worklist pass (list_blocks counts blocks of four warps)
    static unsigned split_grid(const StageArgs<T> &a, int warps) {
        return std::max(1u, unsigned(a.list_blocks) * 4u / unsigned(warps));
    }
    // block of a full pass of the other flux-like schemes (the tuned flux block); worklist passes keep 128
    static int fbs(const StageArgs<T> &a) { return a.full ? a.flux_block : 128; }
    static void gather(const void *args, int64_t n, cudaStream_t s) {
        const StageArgs<T> &a = *static_cast<const StageArgs<T> *>(args);
        if constexpr (sizeof(T) == 4 && RDEG == 1) {
            if constexpr (D == 3 && !wide_system<T, M, PDE>()) {
                // FP32 full pass with tile tables: neighbours staged in shared memory (in 2-D the slot streams are
                // the faster form: 893 against 1027 us a step, 2-D Euler at 1.0M)
                if (a.full && a.tile) {
                    const size_t smem = tile_gather_smem<D, M>(a.tv.umax);
                    if (a.sc.limiter != HCC_LIMITER_NONE)
                        k_gather_tile<D, M, PDE, true><<<unsigned(a.tv.ntiles), 2 * HCC_TILE, smem, s>>>(a);
                    else
                        k_gather_tile<D, M, PDE, false><<<unsigned(a.tv.ntiles), 2 * HCC_TILE, smem, s>>>(a);
                    return;
                }
            }
            if constexpr (wide_system<T, M, PDE>()) {
                if (a.full && a.sc.limiter == HCC_LIMITER_NONE && a.g.gw) {
                    k_gather_wide<D, M, PDE><<<std::max(1u, grid(a.nfull * wide_lanes<M>(), kWideThreads)), kWideThreads, 0,
                                               s>>>(a);
                    return;
                }
            }
            if (!a.full) {   // FP32 degree-1 worklist pass: split tiles
                if (a.sc.limiter != HCC_LIMITER_NONE)
                    k_gather_tiles<T, D, M, PDE, RDEG, true><<<split_grid(a, split_warps<M>()), 32 * split_warps<M>(), 0, s>>>(a);
                else
                    k_gather_tiles<T, D, M, PDE, RDEG, false><<<split_grid(a, split_warps<M>()), 32 * split_warps<M>(), 0, s>>>(a);
                return;
            }
        }
        if constexpr (sizeof(T) == 8 && M <= kSplit64) {
            if (a.full && a.sc.limiter == HCC_LIMITER_NONE && (D == 3 || a.nfull <= HCC_SPLIT64_GATHER)) {
                k_gather_split<D, M, PDE, RDEG><<<std::max(1u, grid(a.nfull * kSplit64, 128)), 128, 0, s>>>(a);
                return;
            }
        }
        const int bs = a.full ? a.gather_block : 128;
        if (a.sc.limiter != HCC_LIMITER_NONE)
            k_gather<T, D, M, PDE, RDEG, true><<<pass_grid(a, bs), bs, 0, s>>>(a);
        else
            k_gather<T, D, M, PDE, RDEG, false><<<pass_grid(a, bs), bs, 0, s>>>(a);
    }
    template <bool MOM> static void flux_mom(const StageArgs<T> &a, int64_t n, cudaStream_t s) {
        if constexpr (sizeof(T) == 4) {
            if (!a.full) {
                const unsigned g = split_grid(a, flux_split_warps<D, M, RDEG>()), nth = 32 * flux_split_warps<D, M, RDEG>();
                if (a.mover) k_flux_tiles<T, D, M, PDE, RDEG, true, MOM><<<g, nth, 0, s>>>(a);
                else k_flux_tiles<T, D, M, PDE, RDEG, false, MOM><<<g, nth, 0, s>>>(a);
                return;
            }
        }
        const int bs = a.full ? a.flux_block : HCC_FLUX_BLOCK;
        if (a.mover)
            k_flux<T, D, M, PDE, RDEG, true, MOM><<<pass_grid(a, bs), bs, 0, s>>>(a);
        else
            k_flux<T, D, M, PDE, RDEG, false, MOM><<<pass_grid(a, bs), bs, 0, s>>>(a);
    }
    static void flux(const void *args, int64_t n, cudaStream_t s) {
        const StageArgs<T> &a = *static_cast<const StageArgs<T> *>(args);
        // first-order MUSCL with the moment correction: its own instantiation (the per-slot correction costs the
        // plain pass registers)
        if constexpr (RDEG == 1) {
            if (a.g.mw) { flux_mom<true>(a, n, s); return; }
        }
        if constexpr (sizeof(T) == 4) {
            if constexpr (RDEG == 1) {
                if (a.full && a.tile) {   // full pass with tile tables: neighbours staged in shared memory
                    if constexpr (wide_system<T, M, PDE>()) {
                        const size_t smem = size_t(a.tv.umax) * wide_flux_row<D, M>() * sizeof(float);
                        k_flux_wide<D, M, PDE><<<unsigned(a.tv.ntiles), kWideThreads, smem, s>>>(a);
                    } else {
                        auto go = [&](auto kernel) {
                            kernel<<<unsigned(a.tv.ntiles), tile_flux_threads<D>() * HCC_TILE, tile_flux_smem<D, M>(a.tv.umax),
                                     s>>>(a);
                        };
                        const bool plain = a.sc.strategy == HCC_EPD1 && !a.sc.aligned;
                        if (plain) go(k_flux_tile<D, M, PDE, true>);
                        else go(k_flux_tile<D, M, PDE, false>);
                    }
                    return;
                }
            }
            if (!a.full) {   // FP32 worklist pass: split tiles
                const unsigned g = split_grid(a, flux_split_warps<D, M, RDEG>()), nth = 32 * flux_split_warps<D, M, RDEG>();
                if (a.mover) k_flux_tiles<T, D, M, PDE, RDEG, true><<<g, nth, 0, s>>>(a);
                else k_flux_tiles<T, D, M, PDE, RDEG, false><<<g, nth, 0, s>>>(a);
                return;
            }
        }
        if constexpr (sizeof(T) == 8 && M <= kSplit64) {
            if ((D == 3 || a.nfull <= (a.full ? HCC_SPLIT64_FLUX : HCC_SPLIT64_LIST)) && !(a.full && a.rough_words)) {
                const unsigned g = a.full ? std::max(1u, grid(a.nfull * kSplit64, 128)) : std::max(1u, unsigned(a.list_blocks));
                if (a.mover) k_flux_split<D, M, PDE, RDEG, true><<<g, 128, 0, s>>>(a);
                else k_flux_split<D, M, PDE, RDEG, false><<<g, 128, 0, s>>>(a);
                return;
            }
        }
        const int bs = a.full ? a.flux_block : HCC_FLUX_BLOCK;
        if (a.mover)     // moving grid: the ALE-frame instantiation (grid velocities, shifted fluxes and speeds)
            k_flux<T, D, M, PDE, RDEG, true><<<pass_grid(a, bs), bs, 0, s>>>(a);
        else
            k_flux<T, D, M, PDE, RDEG, false><<<pass_grid(a, bs), bs, 0, s>>>(a);
    }
    static void stage1(const void *args, int64_t n, cudaStream_t s) {
        k_stage1<T, D, M, PDE, RDEG><<<grid(n, 256), 256, 0, s>>>(*static_cast<const StageArgs<T> *>(args));
    }
    static int cfl(const void *args, int64_t n, unsigned long long *dt_bits, cudaStream_t s) {
        const StageArgs<T> &a = *static_cast<const StageArgs<T> *>(args);
        if constexpr (sizeof(T) == 4 && RDEG == 1 && D == 3) {
            // FP32 with tile tables: the union's speeds staged in shared memory (in 2-D the streams and the table of
            // speeds are faster: 78 against 88 us at 1.0M)
            if (a.tile && !a.cloud_id) {
                const size_t smem = (size_t(a.tv.umax) * 8 + HCC_TILE) * sizeof(float);
                k_cfl_tile<D, M, PDE><<<unsigned(a.tv.ntiles), 2 * HCC_TILE, smem, s>>>(a, dt_bits);
                return 1;
            }
        }
        if constexpr (PDE == HCC_PDE_EULER) k_speeds<T, D, M, PDE><<<grid(n, 256), 256, 0, s>>>(a);
        k_cfl<T, D, M, PDE, RDEG><<<std::max(1u, grid(a.nfull, 256)), 256, 0, s>>>(a, dt_bits);
        return PDE == HCC_PDE_EULER ? 2 : 1;
    }
    static void weno(const void *args, int64_t n, cudaStream_t s) {
        const StageArgs<T> &a = *static_cast<const StageArgs<T> *>(args);
        if constexpr (sizeof(T) == 4 && PDE == HCC_PDE_EULER && RDEG == 1) {
            if (a.g.wops) {   // FP32 Euler with the cached operators
                constexpr int NB = kWenoWarps * WenoShared<D>::P;
                const unsigned g = std::max(1u, a.full ? grid(a.nfull, NB) : unsigned(a.list_blocks));
                k_weno_euler_f32<D><<<g, 32 * kWenoWarps, 0, s>>>(a);
                return;
            }
        }
        if constexpr (sizeof(T) == 8 && PDE == HCC_PDE_EULER && RDEG == 1) {
            // the stage's flux table, once per stage state (the MOOD worklist passes reuse it)
            if (a.full && a.wflux64) k_weno_prep64<D><<<grid(n, 256), 256, 0, s>>>(a);
        }
        if constexpr (M == 1 && PDE == HCC_PDE_ADVECTION) {
            k_weno<T, D><<<pass_grid(a, fbs(a)), fbs(a), 0, s>>>(a);
        } else if constexpr (RDEG == 1) {       // systems (one instantiation: WENO has no reconstruction degree)
            k_weno_sys<T, D, M, PDE><<<pass_grid(a, fbs(a)), fbs(a), 0, s>>>(a);
        }
    }
    static void upwind(const void *args, int64_t n, cudaStream_t s) {
        if constexpr (M == 1 && PDE == HCC_PDE_ADVECTION) {
            const StageArgs<T> &a = *static_cast<const StageArgs<T> *>(args);
            if (a.sc.upwind_alg == HCC_UPWIND_TIWARI)
                k_upwind<T, D, HCC_UPWIND_TIWARI><<<pass_grid(a, fbs(a)), fbs(a), 0, s>>>(a);
            else if constexpr (D == 2)
                k_upwind<T, D, HCC_UPWIND_PRAVEEN><<<pass_grid(a, fbs(a)), fbs(a), 0, s>>>(a);
        }
    }
    static void weno_geom(const WenoGeomArgs &g, cudaStream_t s) {
        if constexpr (PDE == HCC_PDE_EULER && RDEG == 1) {
            if (g.n <= 0) return;
            if constexpr (sizeof(T) == 4) k_weno_geom<D><<<unsigned((g.n + 127) / 128), 128, 0, s>>>(g);
            else k_weno_geom64<D><<<unsigned((g.n + 127) / 128), 128, 0, s>>>(g);
        }
    }
    static void central(const void *args, int64_t n, cudaStream_t s) {
        const StageArgs<T> &a = *static_cast<const StageArgs<T> *>(args);
        const unsigned g = a.full && !central_lists<T>() ? std::max(1u, grid(n, fbs(a))) : pass_grid(a, fbs(a));
        k_central<T, D, M, PDE><<<g, fbs(a), 0, s>>>(a);
    }
    // The opt-in shared memory of the tile passes. The attribute belongs to a kernel on a device: it is set when the tables
    // of a context are built, on the device that will run them.
    static cudaError_t tile_setup() {
        cudaError_t err = cudaSuccess;
        if constexpr (sizeof(T) == 4 && RDEG == 1) {
            const int most = tile_smem_optin();
            auto allow = [&](auto kernel, int bytes) {
                if (err == cudaSuccess) err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            };
            if constexpr (wide_system<T, M, PDE>()) {
                allow(k_flux_wide<D, M, PDE>, most - 1024);        // (it has a static part)
            } else {
                allow(k_flux_tile<D, M, PDE, true>, most);
                allow(k_flux_tile<D, M, PDE, false>, most);
            }
            if constexpr (D == 3 && !wide_system<T, M, PDE>()) {
                allow(k_gather_tile<D, M, PDE, true>, most);
                allow(k_gather_tile<D, M, PDE, false>, most);
            }
            if constexpr (D == 3) allow(k_cfl_tile<D, M, PDE>, most);
        }
        return err;
    }
    static const StageOps *ops() {
        static const StageOps o = {D, M, PDE, RDEG, RBasis<D, RDEG>::B, &gather, &flux, &stage1, &cfl,
                                   ((M == 1 && PDE == HCC_PDE_ADVECTION) || RDEG == 1) ? &weno : nullptr,
                                   RDEG == 1 ? &central : nullptr,
                                   (RDEG == 1 && M == 1 && PDE == HCC_PDE_ADVECTION) ? &upwind : nullptr,
                                   (PDE == HCC_PDE_EULER && RDEG == 1) ? &weno_geom : nullptr, &tile_setup};
        return &o;
    }
};

template <typename T, int RDEG>
const StageOps *lookup_euler(int D, int M) {
    if (D == 1 && M == 3) return StageInst<T, 1, 3, HCC_PDE_EULER, RDEG>::ops();
    if (D == 2 && M == 4) return StageInst<T, 2, 4, HCC_PDE_EULER, RDEG>::ops();
    if (D == 3 && M == 5) return StageInst<T, 3, 5, HCC_PDE_EULER, RDEG>::ops();
    return nullptr;
}
template <typename T, int RDEG>
const StageOps *lookup_linear(int D, int M, int pde) {
    if (pde == HCC_PDE_BGK) {
        if (D == 2 && M == 16) return StageInst<T, 2, 16, HCC_PDE_BGK, RDEG>::ops();
        if (D == 1 && M == 2) return StageInst<T, 1, 2, HCC_PDE_BGK, RDEG>::ops();
        return nullptr;
    }
    if (D == 1 && M == 1) return StageInst<T, 1, 1, HCC_PDE_ADVECTION, RDEG>::ops();
    if (D == 2 && M == 1) return StageInst<T, 2, 1, HCC_PDE_ADVECTION, RDEG>::ops();
    if (D == 3 && M == 1) return StageInst<T, 3, 1, HCC_PDE_ADVECTION, RDEG>::ops();
    if (D == 2 && M == 2) return StageInst<T, 2, 2, HCC_PDE_ADVECTION, RDEG>::ops();
    return nullptr;
}

}  // namespace hcc
