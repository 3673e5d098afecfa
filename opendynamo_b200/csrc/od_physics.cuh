// Pointwise compressible Navier-Stokes physics for the FR P=3 step path.
//
// Same mathematics as the reference's device library
// (src/cuda/device_functions.cuh): ideal gas gamma = 1.4, Pr = 0.72,
// Stokes hypothesis, heat flux -mu*gamma/(Pr*(gamma-1)) * grad(p/rho),
// pressure clamped at 1e-7 in the inviscid fluxes and sound speeds, and the
// Rusanov / AUSM+ / SLAU2 interface fluxes on axis-aligned normals.
//
// Laid out for the GPU rather than per call: the primitive variables of a
// point (1/rho, velocity, pressure) are formed once and shared by the Euler
// flux, the viscous flux of all three directions and the Riemann solvers.
// Normals are axis-aligned, so the direction is a template argument and the
// normal velocity is a register pick, not a dot product.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace od {

enum Flux : int { kSlau2 = 0, kAusmPlus = 1, kRusanov = 2 };

// Division / reciprocal / square root policy. MathIeee: correctly rounded
// (the reference with fast_math = false, and every f64 operation).
// MathFast: for f32 operands the approximate PTX forms (rcp.approx,
// sqrt.approx, ~1-2 ulp), the arithmetic of the reference's default
// --use_fast_math build; f64 operands stay IEEE (fast math does not touch them).
struct MathIeee {
    static constexpr bool kSutherland = false;
    static constexpr bool kWideState = false;
    template <class T>
    static __device__ __forceinline__ T rcp(T x) { return (T)1.0 / x; }
    template <class T>
    static __device__ __forceinline__ T div(T a, T b) { return a / b; }
    template <class T>
    static __device__ __forceinline__ T sqrt(T x) { return ::sqrt(x); }
};

struct MathFast {
    static constexpr bool kSutherland = false;
    static constexpr bool kWideState = false;
    template <class T>
    static __device__ __forceinline__ T rcp(T x) {
        if constexpr (sizeof(T) == 4) {
            float r;
            asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
            return r;
        } else {
            return (T)1.0 / x;
        }
    }
    template <class T>
    static __device__ __forceinline__ T div(T a, T b) {
        if constexpr (sizeof(T) == 4) return a * rcp(b);
        else return a / b;
    }
    template <class T>
    static __device__ __forceinline__ T sqrt(T x) {
        if constexpr (sizeof(T) == 4) {
            float r;
            asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
            return r;
        } else {
            return ::sqrt(x);
        }
    }
};

// A math policy with Sutherland's law switched on (a separate kernel variant,
// so the constant-viscosity kernels carry no trace of it).
template <class Base>
struct WithSutherland : Base {
    static constexpr bool kSutherland = true;
};

// A math policy for f32 flux arithmetic under an f64 state (the u64/c32 and
// mixed pipelines). Such a state shows every rounding of the fluxes (at 1e-8,
// where an f32 state rounds them away), so these pipelines keep the formulas'
// operation order that their states, checkpoints and restarts have always
// had; the other pipelines take the forms with fewer operations.
template <class Base>
struct WideState : Base {
    static constexpr bool kWideState = true;
};

template <class C>
struct Gas {
    static __device__ __forceinline__ C gamma() { return (C)1.4; }
    static __device__ __forceinline__ C gm1() { return (C)1.4 - (C)1.0; }
    static __device__ __forceinline__ C pr() { return (C)0.72; }
};

template <class C>
__device__ __forceinline__ C cmax(C a, C b) { return a > b ? a : b; }
template <class C>
__device__ __forceinline__ C cmin(C a, C b) { return a < b ? a : b; }

// Raw pressure (gamma-1)(E - |m|^2 / (2 rho)); the viscous flux uses it unclamped.
template <class M, class P>
__device__ __forceinline__ P raw_pressure(P r, P m0, P m1, P m2, P E) {
    P ke = M::div((P)0.5 * (m0 * m0 + m1 * m1 + m2 * m2), r);
    return Gas<P>::gm1() * (E - ke);
}

template <class C>
__device__ __forceinline__ C clamp_p(C p) { return cmax((C)1e-7, p); }

// State of a point in compute type: conserved variables, 1/rho, velocity, the
// clamped pressure, and what the viscous flux needs: kinetic and internal
// energy per volume, or (kWideState) the unclamped pressure.
template <class C>
struct FaceState {
    C q[5];
    C ir;
    C vel[3];
    C ke;     // |m|^2 / (2 rho)
    C ein;    // E - ke
    C praw;   // (gamma - 1) ein
    C p;      // praw clamped (the inviscid fluxes and sound speeds)
};

// 1/x in f64 from an f32 estimate r0 of it (rcp.approx: relative error below
// 2^-22): one step of the third-order iteration r0 (1 + e + e^2), e = 1 - r0 x
// (Householder's method for f(r) = 1/r - x), error e^3 below 2^-66 before
// rounding. x in the f32 range.
__device__ __forceinline__ double rcp_refined(double x, float r0) {
    const double r = (double)r0;
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// kWideState: the pressure recovered in the state arithmetic's precision P
// (f64 in the mixed form, whose f64 division of the kinetic energy, 17 of them
// a thread, is a product with the refined reciprocal: 96^3 step 14.9 -> 14.2 ms).
// Otherwise the kinetic energy comes from the velocity (one reciprocal per
// point, no second division).
template <class M, class C, class P>
__device__ __forceinline__ FaceState<C> make_face_state(const P* qp) {
    FaceState<C> s;
#pragma unroll
    for (int v = 0; v < 5; ++v) s.q[v] = (C)qp[v];
    s.ir = M::rcp(s.q[0]);
    if constexpr (M::kWideState) {
        if constexpr (sizeof(P) == 8) {
            const P ke = ((P)0.5 * (qp[1] * qp[1] + qp[2] * qp[2] + qp[3] * qp[3])) * rcp_refined(qp[0], s.ir);
            s.praw = (C)(Gas<P>::gm1() * (qp[4] - ke));
        } else {
            s.praw = raw_pressure<M, P>(qp[0], qp[1], qp[2], qp[3], qp[4]);
        }
        s.p = clamp_p<C>(s.praw);
    }
    s.vel[0] = s.q[1] * s.ir;
    s.vel[1] = s.q[2] * s.ir;
    s.vel[2] = s.q[3] * s.ir;
    if constexpr (!M::kWideState) {
        s.ke = (C)0.5 * (s.q[1] * s.vel[0] + s.q[2] * s.vel[1] + s.q[3] * s.vel[2]);
        s.ein = s.q[4] - s.ke;
        s.p = clamp_p<C>(Gas<C>::gm1() * s.ein);
    }
    return s;
}

// Inviscid flux along axis D.
template <int D, class C>
__device__ __forceinline__ void euler_flux(const FaceState<C>& s, C* f) {
    C vn = s.vel[D];
    f[0] = s.q[1 + D];
    f[1] = s.q[1] * vn;
    f[2] = s.q[2] * vn;
    f[3] = s.q[3] * vn;
    f[1 + D] += s.p;
    f[4] = vn * (s.q[4] + s.p);
}

// sqrt(gamma p / max(rho, 1e-7)); not kWideState: with the reciprocal of rho
// at hand (NaN for a NaN density)
template <class M, class C>
__device__ __forceinline__ C sound_speed(const FaceState<C>& s) {
    if constexpr (M::kWideState) {
        return M::sqrt(cmax((C)0.0, M::div(Gas<C>::gamma() * s.p, cmax((C)1e-7, s.q[0]))));
    } else {
        const C ir = (C)1e-7 > s.q[0] ? (C)1e7 : s.ir;
        return M::sqrt(cmax((C)0.0, Gas<C>::gamma() * s.p * ir));
    }
}

// Dynamic viscosity at a point. Policies without kSutherland: constant mu
// (the reference's MU_REF, src/cuda/constants.cuh:42). Otherwise Sutherland's law
//   mu = mu_ref * T^(3/2) * (1 + S) / (T + S),
// T = gamma * p / rho the temperature in units of the reference temperature
// (rho = 1, c = 1 there) and S = s_suth / t_ref (config.toml [physics]).
// An extension: the reference parses viscosity_model but no kernel reads it.
template <class M, class C>
__device__ __forceinline__ C viscosity(C mu, C suth, const FaceState<C>& s) {
    if constexpr (!M::kSutherland) {
        return mu;
    } else {
        const C T = Gas<C>::gamma() * s.p * s.ir;
        return mu * T * M::sqrt(T) * M::div((C)1.0 + suth, T + suth);
    }
}

// The viscous terms, arranged so that every factor 1/rho is applied once.
// With w_ab = d(rho u_a)/dx_b - u_a d(rho)/dx_b = rho du_a/dx_b:
//   tau_ab = (mu / rho) (w_ab + w_ba - 2/3 delta_ab tr w)
// and the heat flux -mu gamma / (Pr (gamma - 1)) d(p/rho)/dx_b, p = (gamma - 1)
// ein, whose gradient needs no pressure:
//   -heat_b = (mu / rho) (gamma / Pr)
//             (dE/dx_b - u . d(rho u)/dx_b + (ke - ein) / rho d(rho)/dx_b)
// 28 operations a face and 77 a point for all three directions (with every
// velocity gradient, pressure gradient and kinetic-energy gradient formed on
// its own: about 45 and 150). With the one reciprocal per point, the shared
// flux rows and the folded jumps: phase A 1948 -> 1779 warp instructions per
// element in f32 (85.1 -> 82.1 us at 32^3), 269 -> 243 us in f64.

// the bracket of -heat_b; ce = (ke - ein) / rho
template <class C>
__device__ __forceinline__ C heat_bracket(const FaceState<C>& s, const C* g, C ce, int b) {
    return g[12 + b] + ce * g[b] - s.vel[0] * g[3 + b] - s.vel[1] * g[6 + b] - s.vel[2] * g[9 + b];
}

template <class C>
__device__ __forceinline__ constexpr C gamma_over_pr() { return (C)(1.4 / 0.72); }

// Viscous flux along axis D at a face point from the state and the
// 15-component conserved gradient g[3*var + axis] (only the 11 components
// the D-flux reads are touched).
template <int D, class C>
__device__ __forceinline__ void viscous_flux(const FaceState<C>& s, const C* g, C mu, C* f) {
    auto w = [&](int a, int b) -> C { return g[3 * (1 + a) + b] - s.vel[a] * g[b]; };
    const C mi = mu * s.ir;
    const C tr = (w(0, 0) + w(1, 1) + w(2, 2)) * ((C)2.0 / (C)3.0);
    C tau[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (a == D)
            tau[a] = mi * ((C)2.0 * w(D, D) - tr);
        else
            tau[a] = mi * (w(a, D) + w(D, a));
    }
    f[0] = (C)0.0;
    f[1] = tau[0];
    f[2] = tau[1];
    f[3] = tau[2];
    f[4] = mi * gamma_over_pr<C>() * heat_bracket(s, g, (s.ke - s.ein) * s.ir, D) + s.vel[0] * tau[0] +
           s.vel[1] * tau[1] + s.vel[2] * tau[2];
}

// Volume fluxes F_euler - F_viscous of all three directions at a solution
// point. The momentum fluxes rho u_a u_b + p delta_ab - tau_ab are symmetric
// (m[a][b], b >= a); the mass flux along d is the momentum q[1 + d].
template <class C>
struct VolumeFluxes {
    C m00, m11, m22, m01, m02, m12;
    C e[3];
};

template <class C>
__device__ __forceinline__ VolumeFluxes<C> volume_fluxes(const FaceState<C>& s, const C* g, C mu) {
    auto w = [&](int a, int b) -> C { return g[3 * (1 + a) + b] - s.vel[a] * g[b]; };
    const C mi = mu * s.ir;
    const C w00 = w(0, 0), w11 = w(1, 1), w22 = w(2, 2);
    const C tr = (w00 + w11 + w22) * ((C)2.0 / (C)3.0);
    const C t00 = mi * ((C)2.0 * w00 - tr), t11 = mi * ((C)2.0 * w11 - tr), t22 = mi * ((C)2.0 * w22 - tr);
    const C t01 = mi * (w(0, 1) + w(1, 0)), t02 = mi * (w(0, 2) + w(2, 0)), t12 = mi * (w(1, 2) + w(2, 1));
    const C u = s.vel[0], v = s.vel[1], x = s.vel[2];
    VolumeFluxes<C> f;
    f.m00 = s.q[1] * u + s.p - t00;
    f.m11 = s.q[2] * v + s.p - t11;
    f.m22 = s.q[3] * x + s.p - t22;
    f.m01 = s.q[1] * v - t01;
    f.m02 = s.q[1] * x - t02;
    f.m12 = s.q[2] * x - t12;
    const C h = s.q[4] + s.p, ce = (s.ke - s.ein) * s.ir, k = mi * gamma_over_pr<C>();
    // the viscous terms first: h u is orders of magnitude above them, and every
    // term added to it would round at its size
    f.e[0] = h * u - (k * heat_bracket(s, g, ce, 0) + u * t00 + v * t01 + x * t02);
    f.e[1] = h * v - (k * heat_bracket(s, g, ce, 1) + u * t01 + v * t11 + x * t12);
    f.e[2] = h * x - (k * heat_bracket(s, g, ce, 2) + u * t02 + v * t12 + x * t22);
    return f;
}

// The same at two points at once in packed f32 arithmetic (FFMA2: two lanes an
// instruction; the kernels are bound by instruction issue, not by the FP32
// pipe). Every multiply-add is explicit.
struct F2 {
    float2 v;
    __device__ __forceinline__ F2() {}
    __device__ __forceinline__ F2(float a) : v{a, a} {}
    __device__ __forceinline__ F2(float a, float b) : v{a, b} {}
    __device__ __forceinline__ F2(float2 a) : v(a) {}
};
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return __fmul2_rn(a.v, b.v); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return __fadd2_rn(a.v, b.v); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { return __ffma2_rn(a.v, b.v, c.v); }
__device__ __forceinline__ F2 neg2(F2 a) { return F2(-a.v.x, -a.v.y); }

struct VolumeFluxes2 {
    F2 m00, m11, m22, m01, m02, m12;
    F2 e[3];
};

// q(v), g(c): the conserved variables and gradient components of the two points
template <class M, class QF, class GF>
__device__ __forceinline__ VolumeFluxes2 volume_fluxes2(QF q, GF g, float mu0, float suth) {
    const F2 q0 = q(0), q1 = q(1), q2 = q(2), q3 = q(3), q4 = q(4);
    const F2 ir(M::rcp(q0.v.x), M::rcp(q0.v.y));
    const F2 nir = neg2(ir);
    const F2 u = q1 * ir, v = q2 * ir, x = q3 * ir;
    const F2 nu = q1 * nir, nv = q2 * nir, nx = q3 * nir;
    const F2 s2 = fma2(q3, x, fma2(q2, v, q1 * u));   // 2 ke
    const F2 ein = fma2(s2, F2(-0.5f), q4);
    const F2 pr = ein * F2(Gas<float>::gm1());
    const F2 p(clamp_p<float>(pr.v.x), clamp_p<float>(pr.v.y));
    F2 mu(mu0);
    if constexpr (M::kSutherland) {
        FaceState<float> a, b;
        a.p = p.v.x; a.ir = ir.v.x;
        b.p = p.v.y; b.ir = ir.v.y;
        mu = F2(viscosity<M>(mu0, suth, a), viscosity<M>(mu0, suth, b));
    }
    const F2 nmi = mu * nir;                       // -mu / rho
    const F2 ce = fma2(s2, F2(0.5f), neg2(ein)) * ir;   // (ke - ein) / rho
    const F2 h = q4 + p;
    VolumeFluxes2 f;
    const F2 r0 = g(0), r1 = g(1), r2 = g(2);      // gradient of rho
    const F2 a00 = g(3), a10 = g(6), a20 = g(9);   // d/dx of the momenta
    const F2 a01 = g(4), a11 = g(7), a21 = g(10);
    const F2 a02 = g(5), a12 = g(8), a22 = g(11);
    const F2 w00 = fma2(nu, r0, a00), w11 = fma2(nv, r1, a11), w22 = fma2(nx, r2, a22);
    const F2 ntr = (w00 + w11 + w22) * F2(-2.0f / 3.0f);
    // -tau
    const F2 t00 = nmi * fma2(w00, F2(2.0f), ntr), t11 = nmi * fma2(w11, F2(2.0f), ntr),
             t22 = nmi * fma2(w22, F2(2.0f), ntr);
    const F2 t01 = nmi * (fma2(nu, r1, a01) + fma2(nv, r0, a10));
    const F2 t02 = nmi * (fma2(nu, r2, a02) + fma2(nx, r0, a20));
    const F2 t12 = nmi * (fma2(nv, r2, a12) + fma2(nx, r1, a21));
    f.m00 = fma2(q1, u, t00) + p;
    f.m11 = fma2(q2, v, t11) + p;
    f.m22 = fma2(q3, x, t22) + p;
    f.m01 = fma2(q1, v, t01);
    f.m02 = fma2(q1, x, t02);
    f.m12 = fma2(q2, x, t12);
    const F2 nk = nmi * F2(gamma_over_pr<float>());
    const F2 b0 = fma2(nx, a20, fma2(nv, a10, fma2(nu, a00, fma2(ce, r0, g(12)))));
    f.e[0] = fma2(h, u, fma2(x, t02, fma2(v, t01, fma2(u, t00, nk * b0))));
    const F2 b1 = fma2(nx, a21, fma2(nv, a11, fma2(nu, a01, fma2(ce, r1, g(13)))));
    f.e[1] = fma2(h, v, fma2(x, t12, fma2(v, t11, fma2(u, t01, nk * b1))));
    const F2 b2 = fma2(nx, a22, fma2(nv, a12, fma2(nu, a02, fma2(ce, r2, g(14)))));
    f.e[2] = fma2(h, x, fma2(x, t22, fma2(v, t12, fma2(u, t02, nk * b2))));
    return f;
}

// ---- the viscous terms of the kWideState pipelines, in the reference's order
// (device_functions.cuh)

// Inviscid flux along axis d (d known after unrolling).
template <class C>
__device__ __forceinline__ void euler_flux_dyn(const FaceState<C>& s, int d, C* f) {
    C vn = s.vel[d];
    f[0] = s.q[1 + d];
    f[1] = s.q[1] * vn;
    f[2] = s.q[2] * vn;
    f[3] = s.q[3] * vn;
    f[1 + d] += s.p;
    f[4] = vn * (s.q[4] + s.p);
}

// kWideState: heat-flux coefficient mu gamma / (Pr (gamma - 1)), in the reference's
// operation order (device_functions.cuh:44). Constant viscosity: the value
// formed once per launch on the host with the same IEEE operations
// (kappa_const, heat_coeff_host); Sutherland's law: per point.
template <class M, class C>
__device__ __forceinline__ C heat_coeff(C mu, C kappa_const) {
    if constexpr (!M::kSutherland)
        return kappa_const;
    else
        return mu * Gas<C>::gamma() / (Gas<C>::pr() * Gas<C>::gm1());
}

template <class C>
__host__ inline C heat_coeff_host(C mu) {
    return mu * (C)1.4 / ((C)0.72 * ((C)1.4 - (C)1.0));
}

// Viscous flux along axis D at a face point (see viscous_flux).
template <int D, class C>
__device__ __forceinline__ void viscous_flux_wide(const FaceState<C>& s, const C* g, C mu, C kappa, C* f) {
    const C ir = s.ir;
    // d(vel_a)/d(x_b) for the pairs the D-flux needs
    auto dv = [&](int a, int b) -> C { return (g[3 * (1 + a) + b] - s.vel[a] * g[b]) * ir; };
    C div = dv(0, 0) + dv(1, 1) + dv(2, 2);
    C tau[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (a == D)
            tau[a] = mu * ((C)2.0 * dv(D, D) - (C)2.0 / (C)3.0 * div);
        else
            tau[a] = mu * (dv(a, D) + dv(D, a));
    }
    C ke = (C)0.5 * (s.q[1] * s.vel[0] + s.q[2] * s.vel[1] + s.q[3] * s.vel[2]);
    C dke = (s.q[1] * g[3 + D] + s.q[2] * g[6 + D] + s.q[3] * g[9 + D]) * ir - ke * g[D] * ir;
    C dp = Gas<C>::gm1() * (g[12 + D] - dke);
    C heat = -kappa * (dp * ir - s.praw * g[D] * ir * ir);
    f[0] = (C)0.0;
    f[1] = tau[0];
    f[2] = tau[1];
    f[3] = tau[2];
    f[4] = s.vel[0] * tau[0] + s.vel[1] * tau[1] + s.vel[2] * tau[2] - heat;
}

// Volume fluxes of all three directions at a solution point:
// out[d][v] = F_euler,d - F_viscous,d.
template <class C>
__device__ __forceinline__ void volume_fluxes_wide(const FaceState<C>& s, const C* g, C mu, C kappa, C out[3][5]) {
    const C ir = s.ir;
    C dvel[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) dvel[a][b] = (g[3 * (1 + a) + b] - s.vel[a] * g[b]) * ir;
    C div = dvel[0][0] + dvel[1][1] + dvel[2][2];
    C tau[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        tau[a][a] = mu * ((C)2.0 * dvel[a][a] - (C)2.0 / (C)3.0 * div);
#pragma unroll
        for (int b = a + 1; b < 3; ++b) {
            C t = mu * (dvel[a][b] + dvel[b][a]);
            tau[a][b] = t;
            tau[b][a] = t;
        }
    }
    C ke = (C)0.5 * (s.q[1] * s.vel[0] + s.q[2] * s.vel[1] + s.q[3] * s.vel[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        C vn = s.vel[d];
        C dke = (s.q[1] * g[3 + d] + s.q[2] * g[6 + d] + s.q[3] * g[9 + d]) * ir - ke * g[d] * ir;
        C dp = Gas<C>::gm1() * (g[12 + d] - dke);
        C heat = -kappa * (dp * ir - s.praw * g[d] * ir * ir);
        // (F_euler) - (F_viscous), each formed first as the reference does
        C fe[5];
        euler_flux_dyn(s, d, fe);
        out[d][0] = fe[0];
        out[d][1] = fe[1] - tau[0][d];
        out[d][2] = fe[2] - tau[1][d];
        out[d][3] = fe[3] - tau[2][d];
        out[d][4] = fe[4] - (s.vel[0] * tau[0][d] + s.vel[1] * tau[1][d] + s.vel[2] * tau[2][d] - heat);
    }
}

// ---- interface fluxes (axis-aligned normal D, left state L, right state R) ----

template <class M, int D, class C>
__device__ __forceinline__ void rusanov(const FaceState<C>& L, const FaceState<C>& R, C* f) {
    C vnL = L.vel[D], vnR = R.vel[D];
    C smax = cmax(fabs(vnL) + sound_speed<M>(L), fabs(vnR) + sound_speed<M>(R));
    C fL[5], fR[5];
    euler_flux<D>(L, fL);
    euler_flux<D>(R, fR);
#pragma unroll
    for (int v = 0; v < 5; ++v) f[v] = (C)0.5 * (fL[v] + fR[v] - smax * (R.q[v] - L.q[v]));
}

template <class M, int D, class C>
__device__ __forceinline__ void ausm_plus(const FaceState<C>& L, const FaceState<C>& R, C* f) {
    const C alpha = (C)0.1875, beta = (C)0.125;
    C cm = cmax(sound_speed<M>(L), sound_speed<M>(R));
    C icm = M::rcp(cm);
    C mL = L.vel[D] * icm, mR = R.vel[D] * icm;
    C mp, pp, mm, pm;
    if (fabs(mL) >= (C)1.0) {
        mp = (C)0.5 * (mL + fabs(mL));
        pp = mL > (C)0.0 ? (C)1.0 : (C)0.0;
    } else {
        C a = mL + (C)1.0, b = mL * mL - (C)1.0;
        mp = (C)0.25 * a * a + beta * b * b;
        pp = (C)0.25 * a * a * ((C)2.0 - mL) + alpha * mL * b * b;
    }
    if (fabs(mR) >= (C)1.0) {
        mm = (C)0.5 * (mR - fabs(mR));
        pm = mR < (C)0.0 ? (C)1.0 : (C)0.0;
    } else {
        C a = mR - (C)1.0, b = mR * mR - (C)1.0;
        mm = -(C)0.25 * a * a - beta * b * b;
        pm = (C)0.25 * a * a * ((C)2.0 + mR) - alpha * mR * b * b;
    }
    C m = mp + mm;
    C pf = pp * L.p + pm * R.p;
    const bool up = m > (C)0.0;
    const FaceState<C>& W = up ? L : R;
    C mdot = m * cm * W.q[0];
    f[0] = mdot;
    f[1] = mdot * W.vel[0];
    f[2] = mdot * W.vel[1];
    f[3] = mdot * W.vel[2];
    f[1 + D] += pf;
    f[4] = mdot * ((W.q[4] + W.p) * W.ir);
}

template <class M, int D, class C>
__device__ __forceinline__ void slau2(const FaceState<C>& L, const FaceState<C>& R, C* f) {
    C rL = L.q[0], rR = R.q[0];
    C vnL = L.vel[D], vnR = R.vel[D];
    C q2L = L.vel[0] * L.vel[0] + L.vel[1] * L.vel[1] + L.vel[2] * L.vel[2];
    C q2R = R.vel[0] * R.vel[0] + R.vel[1] * R.vel[1] + R.vel[2] * R.vel[2];
    C cf = (C)0.5 * (sound_speed<M>(L) + sound_speed<M>(R));
    C icf = M::rcp(cf);
    C mL = vnL * icf, mR = vnR * icf;
    C qbar = M::sqrt((C)0.5 * (q2L + q2R));
    C mtil = cmin((C)1.0, icf * qbar);
    C chi = ((C)1.0 - mtil) * ((C)1.0 - mtil);
    C g = -cmax(cmin(mL, (C)0.0), (C)-1.0) * cmin(cmax(mR, (C)0.0), (C)1.0);
    C vbar = M::div(rL * fabs(vnL) + rR * fabs(vnR), rL + rR);
    C vbL = ((C)1.0 - g) * vbar + g * fabs(vnL);
    C vbR = ((C)1.0 - g) * vbar + g * fabs(vnR);
    C mdot = (C)0.5 * (rL * (vnL + vbL) + rR * (vnR - vbR) - (chi * icf) * (R.p - L.p));
    C bL = fabs(mL) < (C)1.0 ? (C)0.25 * ((C)2.0 - mL) * (mL + (C)1.0) * (mL + (C)1.0)
                             : (mL >= (C)0.0 ? (C)1.0 : (C)0.0);
    C bR = fabs(mR) < (C)1.0 ? (C)0.25 * ((C)2.0 + mR) * (mR - (C)1.0) * (mR - (C)1.0)
                             : (mR >= (C)0.0 ? (C)0.0 : (C)1.0);
    C pf = (C)0.5 * (L.p + R.p) + (C)0.5 * (bL - bR) * (L.p - R.p);
    pf += qbar * (bL + bR - (C)1.0) * cf * (C)0.5 * (rL + rR);
    const bool up = mdot > (C)0.0;
    const FaceState<C>& W = up ? L : R;
    f[0] = mdot;
    f[1] = mdot * W.vel[0];
    f[2] = mdot * W.vel[1];
    f[3] = mdot * W.vel[2];
    f[1 + D] += pf;
    f[4] = mdot * ((W.q[4] + W.p) * W.ir);
}

template <class M, int FLUX, int D, class C>
__device__ __forceinline__ void interface_flux(const FaceState<C>& L, const FaceState<C>& R, C* f) {
    if constexpr (FLUX == kSlau2)
        slau2<M, D>(L, R, f);
    else if constexpr (FLUX == kAusmPlus)
        ausm_plus<M, D>(L, R, f);
    else
        rusanov<M, D>(L, R, f);
}

// Scheme chosen at run time (ensembles that mix schemes in one launch).
constexpr int kFluxRuntime = -1;

template <class M, int D, class C>
__device__ __forceinline__ void interface_flux_rt(int flux, const FaceState<C>& L, const FaceState<C>& R, C* f) {
    if (flux == kSlau2)
        slau2<M, D>(L, R, f);
    else if (flux == kAusmPlus)
        ausm_plus<M, D>(L, R, f);
    else
        rusanov<M, D>(L, R, f);
}

}  // namespace od
