// FR P=3 stage kernels for sm_100a.
//
// One SSP-RK3 stage of the reference (src/solver.rs:262-317) is a volume
// kernel, three face kernels (+ the y-wall kernel) and an RK kernel
// (src/cuda/rhs.cu:344-739, src/cuda/rk.cu:85-115): seven passes over HBM
// with 6 gradient-slice and 6 face-correction arrays in between. Here a
// stage is two element-local kernels.
//
// Phase A — 16 threads per element; in the pass of direction d each thread
// owns the d-line through face point l (l = j+4k for x, i+4k for y, i+4j for
// z, the reference's face-point numbering), so 1-D operators act on four
// registers:
//   P1  the element state (x-lines, 128-bit loads) -> smem; each thread
//        keeps its own x-line for the x pass
//   P2-4 per direction (x, y, then z after a barrier): own and neighbour
//        face values (BR1 common solution, slip-wall mirror
//        rhs.cu:111-114), corrected gradient along the line
//        (rhs.cu:373-461); at the minus face of the line the interface flux
//        F_I is solved once for both sides (j = F_I - Fe_own here, F_I kept
//        in registers); at the plus face j = -Fe_own (slip wall:
//        j = [0,0,p_w,0,0] - Fe, complete). The y neighbours' traces come
//        from one 128-bit load per variable and side and a lane
//        reduce-scatter; the z pass also does P5 for the z faces.
//   P5  x / y faces: gradient at the face (11 components), own viscous
//        flux Fv; j += 1/2 Fv_own; to the face buffer for the neighbours:
//        F_I - 1/2 Fv_own at the minus faces (all the minus neighbour still
//        needs at its plus face), Fv_own at the plus faces
//   P6  x-threads: pointwise Euler - viscous fluxes of their 4 points
//        (rhs.cu:229-266), two at a time in packed arithmetic in the all-f32
//        kernels; F_y, F_z -> smem, the x-divergence of the thread's own
//        x-line accumulated in registers
//   P7  divergence of F_y / F_z and the lifting -(j_L g_L' + j_R g_R') jac
//        (rk.cu:12-25) of the faces: the thread's own y-line, then z-line, then
//        x-line, the partial updates handed on through smem (kLineUpdate); the
//        pipelines with f32 fluxes under an f64 state instead update a whole
//        x-line from the x-lines of its k-plane and j-column
//   P8  x-threads: RHS + forcing (rhs.cu:505-509), RK combination
//        a*u0 + b*u + c*(RHS + lift) (rk.cu:27-83), 128-bit stores.
//   An element's 16 threads are half of a warp: the passes are separated by
//   warp barriers only.
//   The face correction of the reference, j = F_I - 1/2(Fv_L + Fv_R) -
//   (Fe_own - Fv_own), is then complete except for the terms that belong to
//   the neighbour: F_I at the plus faces and -1/2 Fv_nbr at every non-wall
//   face.
// Phase B — reads those from the face buffer records of the +x/+y/+z
// neighbours (F_I - 1/2 Fv_nbr) and -x/-y/-z neighbours (Fv_nbr) and adds
// their lifted contribution. With an f32 state
// phase A stores the unrounded RHS instead of the new state and phase B
// performs the RK combination, so the state is rounded once per stage:
// phase B's increments are often below half an f32 ulp of E and rho*u, and
// rounding the state before adding them would drop them systematically.
// Phase B always runs (the plus-face F_I comes from the neighbour even when
// mu == 0).
//
// Types: S = stored state, P = state arithmetic (face values, pressure
// recovery, RK accumulation), C = flux arithmetic. Reference-compatible
// pipelines use P == C; the mixed-precision form uses S = P = double with
// C = float.
#pragma once

#include <cuda_bf16.h>

#include "od_launch.h"
#include "od_physics.cuh"

namespace od {

constexpr int NP = 4;   // points per direction
constexpr int NF = 16;  // points per face
constexpr int NE = 64;  // points per element
constexpr int NV = 5;   // conserved variables
constexpr int LPE = 16; // threads (lines) per element

template <class T>
struct Tab {
    T D[16];   // D[a*4+m] = l'_m(x_a)
    T eL[4];   // l_m(-1)
    T eR[4];   // l_m(+1)
    T gL[4];   // Radau g_L'(x_a)
    T gR[4];   // Radau g_R'(x_a)
};

// The operators of each direction scaled by its Jacobian 2/h (products
// rounded in T), with the signs and halves of their uses folded in, so that
// the corrected gradient, the divergence and the lifting are pure FMA chains:
//   d[dir][a*4+m] = D[a*4+m] jac        gradient
//   hl / hr[dir][a] = g_L' / g_R'(x_a) jac / 2   times the jump at the face
//   nd = -d                              divergence
//   nl / nr = -g_L' / g_R' jac           lifting
template <class T>
struct ScaledTab {
    T d[3][16], nd[3][16];
    T hl[3][4], hr[3][4];
    T nl[3][4], nr[3][4];
};

template <class T, class TabT>
__host__ ScaledTab<T> scale_tab(const TabT& t, const T* jac) {
    ScaledTab<T> r;
    for (int dir = 0; dir < 3; ++dir) {
        for (int i = 0; i < 16; ++i) {
            r.d[dir][i] = (T)(t.D[i] * jac[dir]);
            r.nd[dir][i] = -r.d[dir][i];
        }
        for (int a = 0; a < 4; ++a) {
            r.nl[dir][a] = -(T)(t.gL[a] * jac[dir]);
            r.nr[dir][a] = -(T)(t.gR[a] * jac[dir]);
            r.hl[dir][a] = (T)-0.5 * r.nl[dir][a];
            r.hr[dir][a] = (T)-0.5 * r.nr[dir][a];
        }
    }
    return r;
}

// Division of a 32-bit unsigned value by a divisor fixed for the launch: a
// multiply-high and two shifts instead of the integer division sequence
// (Granlund & Montgomery, "Division by invariant integers using
// multiplication", PLDI 1994, section 4): with l = ceil(log2 d) and
// m = floor(2^32 (2^l - d) / d) + 1, n / d = (t + ((n - t) >> min(l, 1))) >>
// max(l - 1, 0) where t = mulhi(m, n), for every n and d in [1, 2^32).
struct FastDiv {
    unsigned m, s1, s2;
};

__host__ inline FastDiv make_fastdiv(unsigned d) {
    unsigned l = 0;
    while (l < 32 && (1ull << l) < d) ++l;
    FastDiv f;
    f.m = (unsigned)(((1ull << 32) * ((1ull << l) - d)) / d + 1);
    f.s1 = l < 1 ? l : 1;
    f.s2 = l > 0 ? l - 1 : 0;
    return f;
}

__device__ __forceinline__ unsigned fast_div(unsigned n, const FastDiv& f) {
    const unsigned t = __umulhi(f.m, n);
    return (t + ((n - t) >> f.s1)) >> f.s2;
}

// Element indices are below 2^31 (od_create rejects larger meshes).
struct Mesh {
    int nx, ny, nz, y_wall;
    long long nelem, npts;
    FastDiv fx, fy;   // division by nx and by ny
};

__host__ inline void mesh_set_div(Mesh& m) {
    m.fx = make_fastdiv((unsigned)m.nx);
    m.fy = make_fastdiv((unsigned)m.ny);
}

// (ex, ey, ez) of element e = ex + nx (ey + ny ez)
__device__ __forceinline__ void elem_coords(const Mesh& m, long long e, int& ex, int& ey, int& ez) {
    const unsigned u = (unsigned)e;
    const unsigned q = fast_div(u, m.fx);
    const unsigned q2 = fast_div(q, m.fy);
    ex = (int)(u - q * (unsigned)m.nx);
    ey = (int)(q - q2 * (unsigned)m.ny);
    ez = (int)q2;
}

// point index inside an element: i + 4 j + 16 k
__device__ __forceinline__ constexpr int pid(int i, int j, int k) { return i + NP * j + NF * k; }

// point m of the direction-D line through face point fp
template <int D>
__device__ __forceinline__ int line_pt(int fp, int m) {
    if constexpr (D == 0) return m + NP * fp;                  // fp = j + 4k
    else if constexpr (D == 1) return (fp & 3) + NP * m + NF * (fp >> 2);  // fp = i + 4k
    else return fp + NF * m;                                   // fp = i + 4j
}

// Face value from the four samples of a line; one fixed FMA chain so that the
// two elements sharing a face compute bit-identical face states.
template <class T, class CC>
__device__ __forceinline__ T trace4(const T* q, const CC& c) {
    return fma(q[3], c[3], fma(q[2], c[2], fma(q[1], c[1], q[0] * c[0])));
}

// Face values at both ends of a line (trace4 with cL and with cR).
template <class T, class CL, class CR>
__device__ __forceinline__ void trace4_lr(const T* q, const CL& cL, const CR& cR, T& oL, T& oR) {
    oL = trace4(q, cL);
    oR = trace4(q, cR);
}

// Sum over the four lanes of an aligned lane group (4g .. 4g+3) of p[q], for
// lane q = lane & 3 of the group: a reduce-scatter in two shuffle rounds
// (partner lane ^ 2 for the pair of components a lane keeps, then lane ^ 1).
// Every lane forms (p_q + p_q^2) + (p_q^1 + p_q^3), which by commutativity is
// the same value, (p_0 + p_2) + (p_1 + p_3), for all four. All 32 lanes of
// the warp must call it together.
template <class T>
__device__ __forceinline__ T sum4_scatter(const T (&p)[4], int q) {
    const bool hi = (q & 2) != 0;
    const T a0 = hi ? p[2] : p[0], a1 = hi ? p[3] : p[1];
    const T b0 = hi ? p[0] : p[2], b1 = hi ? p[1] : p[3];
    const T c0 = a0 + __shfl_xor_sync(0xffffffffu, b0, 2);
    const T c1 = a1 + __shfl_xor_sync(0xffffffffu, b1, 2);
    const bool odd = (q & 1) != 0;
    const T d = odd ? c1 : c0, e = odd ? c0 : c1;
    return d + __shfl_xor_sync(0xffffffffu, e, 1);
}

// neighbour across face (d, side) or -1 for a slip wall (element indices are below 2^31)
__device__ __forceinline__ int neighbour(const Mesh& m, int ex, int ey, int ez, int d, int side) {
    int c0 = ex, c1 = ey, c2 = ez;
    if (d == 0) {
        c0 += side ? 1 : -1;
        c0 = c0 < 0 ? c0 + m.nx : (c0 >= m.nx ? c0 - m.nx : c0);
    } else if (d == 1) {
        c1 += side ? 1 : -1;
        if (m.y_wall && (c1 < 0 || c1 >= m.ny)) return -1;
        c1 = c1 < 0 ? c1 + m.ny : (c1 >= m.ny ? c1 - m.ny : c1);
    } else {
        c2 += side ? 1 : -1;
        c2 = c2 < 0 ? c2 + m.nz : (c2 >= m.nz ? c2 - m.nz : c2);
    }
    return c0 + m.nx * (c1 + m.ny * c2);
}

// ---- 4-wide loads / stores (16-byte aligned for float, 32-byte for double)
template <class T>
__device__ __forceinline__ void ld4s(const T* p, T* q) {
    if constexpr (sizeof(T) == 4) {
        float4 v = *reinterpret_cast<const float4*>(p);
        q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
    } else {
        double2 a = reinterpret_cast<const double2*>(p)[0];
        double2 b = reinterpret_cast<const double2*>(p)[1];
        q[0] = a.x; q[1] = a.y; q[2] = b.x; q[3] = b.y;
    }
}

template <class T>
__device__ __forceinline__ void st4s(T* p, const T* q) {
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(p) = make_float4(q[0], q[1], q[2], q[3]);
    } else {
        reinterpret_cast<double2*>(p)[0] = make_double2(q[0], q[1]);
        reinterpret_cast<double2*>(p)[1] = make_double2(q[2], q[3]);
    }
}

// Global loads of state, records and right-hand sides. They are coherent
// (ld.global, never ld.global.nc or __ldg) and, where written as assembly,
// volatile with a memory clobber: these kernels are resident while the kernel
// before them still writes what they read (programmatic dependents), so nothing
// may be read through a path that assumes read-only data, or moved above the
// griddepcontrol.wait in dependent_start.

// 4-wide load of S values converted to P
template <class S, class P>
__device__ __forceinline__ void ldc4(const S* p, P* q) {
    S w[4];
    ld4s(p, w);
#pragma unroll
    for (int a = 0; a < 4; ++a) q[a] = (P)w[a];
}

// One value, as assembly, so that the strided loads of a y- or z-line and the
// 256-bit ones stay in the order they are written in (plain loads: 48^3 f32 and
// 24^3 closure steps 0.7% slower, 96^3 mixed 0.2%).
template <class P, class S>
__device__ __forceinline__ P ldc1(const S* p) {
    S a;
    if constexpr (sizeof(S) == 8)
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(a) : "l"(p) : "memory");
    else
        asm volatile("ld.global.f32 %0, [%1];" : "=f"(a) : "l"(p) : "memory");
    return (P)a;
}

// 256-bit load / store of a 32-byte aligned f64 line
template <class S, class P>
__device__ __forceinline__ void ld4wide(const S* p, P* q) {
    double a, b, c, d;
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p) : "memory");
    q[0] = (P)a; q[1] = (P)b; q[2] = (P)c; q[3] = (P)d;
}

// 4-wide load, of a 32-byte aligned f64 line in one 256-bit load (W): two
// 128-bit loads of a warp's 16-byte halves touch every sector twice
template <bool W, class S, class P>
__device__ __forceinline__ void ldc4w(const S* p, P* q) {
    if constexpr (W && sizeof(S) == 8)
        ld4wide<S, P>(p, q);
    else
        ldc4<S, P>(p, q);
}

template <class S, class P>
__device__ __forceinline__ void st4wide(S* p, const P* q) {
    asm volatile("st.global.v4.f64 [%4], {%0,%1,%2,%3};" ::"d"((double)q[0]), "d"((double)q[1]), "d"((double)q[2]),
                 "d"((double)q[3]), "l"(p)
                 : "memory");
}

template <class S, class P>
__device__ __forceinline__ void stg4(S* p, const P* q) {
    if constexpr (sizeof(S) == 4) {
        *reinterpret_cast<float4*>(p) = make_float4((float)q[0], (float)q[1], (float)q[2], (float)q[3]);
    } else {
        reinterpret_cast<double2*>(p)[0] = make_double2((double)q[0], (double)q[1]);
        reinterpret_cast<double2*>(p)[1] = make_double2((double)q[2], (double)q[3]);
    }
}

// gradient components the direction-D viscous flux reads
// (x omits 8,10,13,14; y omits 5,9,12,14; z omits 4,6,12,13 — rhs.cu:129,151,169)
template <int D>
__device__ __forceinline__ constexpr bool grad_used(int c) {
    constexpr unsigned omit = D == 0 ? ((1u << 8) | (1u << 10) | (1u << 13) | (1u << 14))
                            : D == 1 ? ((1u << 5) | (1u << 9) | (1u << 12) | (1u << 14))
                                     : ((1u << 4) | (1u << 6) | (1u << 12) | (1u << 13));
    return !((omit >> c) & 1u);
}

// ---- shared-memory point layout
// 4-byte rows: points of an element are stored at p ^ (((p >> 3) & 4) | par << 3):
// the j index is XOR-swizzled with bit 1 of k and with the element's parity
// inside its warp (two elements per warp), and every element slot is a
// multiple of 32 words plus 16. With these, the three access patterns of a
// half-warp (16 x-lines as 128-bit vectors, 16 y-lines and 16 z-lines as
// scalars) hit 32 distinct banks across the whole warp.
// 8-byte rows: an access phase is one element's half-warp of 8-byte words (16
// bank pairs), or 8 lanes of a 128-bit one. j is XORed with all of k, so that
// the 16 y-lines, 4 values of i for each k, fall on distinct banks, and the
// halves of an x-line are swapped for odd k, so that the 128-bit halves of
// the 8 lines of two k's do. (With the 4-byte swizzle 31% of the wavefronts
// of the f64 kernel were conflicts; 40^3 f64 step 1.64 -> 1.60 ms, 96^3 mixed
// 15.6 -> 15.0.)
template <class T>
__device__ __forceinline__ int sw(int p, int swz) {
    if constexpr (sizeof(T) == 4)
        return p ^ (((p >> 3) & 4) | swz);
    else
        return p ^ ((p >> 2) & 12) ^ ((p >> 3) & 2);
}

// the x-line stored at offset x (sw of its first point) of a row
template <class T>
__device__ __forceinline__ void ld_xline(const T* row, int x, T* q) {
    if constexpr (sizeof(T) == 4) {
        ld4s(row + x, q);
    } else {
        const double2 a = *reinterpret_cast<const double2*>(row + x), b = *reinterpret_cast<const double2*>(row + (x ^ 2));
        q[0] = a.x; q[1] = a.y; q[2] = b.x; q[3] = b.y;
    }
}

template <class T>
__device__ __forceinline__ void st_xline(T* row, int x, const T* q) {
    if constexpr (sizeof(T) == 4) {
        st4s(row + x, q);
    } else {
        *reinterpret_cast<double2*>(row + x) = make_double2(q[0], q[1]);
        *reinterpret_cast<double2*>(row + (x ^ 2)) = make_double2(q[2], q[3]);
    }
}

// Whether every face correction of a line stays in its thread's registers (all
// but the kWideState pipelines, whose operation order the other update keeps):
// the update then works on the thread's own y- and z-lines, one row line in
// and one out per variable, where the update of a whole x-line loads the four
// x-lines of its k-plane and of its j-column and the corrections of four lines
// (a third of the kernel's shared-memory traffic). 48^3 f32 step 1.10 -> 1.06
// ms, 40^3 f64 1.55 -> 1.46.
template <class M, class P, class C>
constexpr bool kLineUpdate = !M::kWideState && sizeof(P) == sizeof(C);

template <class P, class C, bool J>
struct SlotBytes {
    static constexpr int base =
        15 * NE * (int)sizeof(C) + NV * NE * (int)sizeof(P) + (J ? 4 * NV * NF * (int)sizeof(C) : 0);
    static constexpr int words = base / 4;
    static constexpr int pad_words = ((16 - words % 32) + 32) % 32 == 0 ? 32 : ((16 - words % 32) + 32) % 32;
};

// y / z face corrections without -1/2 Fv_nbr [face - 2][var][face pt]; the x
// faces of a line belong to its own thread and stay in registers
template <class C, bool J>
struct SlotJ {
    C j[4][NV][NF];
};
template <class C>
struct SlotJ<C, false> {};

// Shared-memory slot of one element in phase A.
template <class P, class C, bool J>
struct alignas(16) SlotA : SlotJ<C, J> {
    C g[15][NE];          // gradient; from P6: fluxes (and partial updates) in the first rows
    P u[NV][NE];          // state
    float pad[SlotBytes<P, C, J>::pad_words];
};

template <class M, class P, class C>
using SlotFor = SlotA<P, C, !kLineUpdate<M, P, C>>;

template <class S, class P, class C>
struct StageAParams {
    using S_t = S;
    using P_t = P;
    using C_t = C;
    const S* u_in;
    const S* u0;
    S* u_out;       // new state, or the RHS when phase B performs the RK combination
    C* fv;          // [elem][dir 3][var 4][face pt 16]: own viscous flux (components 1..4) at the plus faces
    C* fi;          // [elem][dir 3][var 5][face pt 16]: F_I - 1/2 Fv_own at the minus faces
    Mesh m;
    Tab<P> tp;
    Tab<C> tc;
    ScaledTab<C> sc;
    C jac[3];
    P ra, rb, rc;
    C mu, forcing;
    C suth;             // Sutherland S = s_suth / t_ref, < 0: constant mu
    C kappa;            // kWideState: heat-flux coefficient of the constant mu (heat_coeff_host)
    int flags;
    int flux;           // scheme id, read when the kernel's FLUX is kFluxRuntime
    long long e0, e1;   // element range of this launch
    StageFeatures feat; // the closure's features, written by the FEAT kernels (f32)
};


// P1b of phase A with the closure attached: the features of the element's
// input state at the thread's four points (the same operations, in the same
// order, as the closure's features kernel: x derivatives from the thread's
// x-line, y / z derivatives from the x-lines of its k-plane / j-column),
// staged as bf16 in the gradient rows (not written before P2) and stored in
// the fused inference kernel's tile layout as 16-byte chunks.
template <class PA, class Slot, class P = typename PA::P_t, class C = typename PA::C_t>
__device__ __forceinline__ void stage_a_features(const PA& A, Slot& sm, long long e, int l, int swz,
                                                 bool live, const P (&qx)[NV][4]) {
    // Points (0, 1) and (2, 3) of the line side by side in packed arithmetic,
    // each value by the features kernel's operations; the clip follows the bf16
    // rounding (8 is a bf16 value, so the order makes no difference), and a
    // channel's four points are one 8-byte store (24^3 closure step 0.262 ms
    // with scalar arithmetic and 2-byte stores, 0.257 so).
    const StageFeatures& fp = A.feat;
    const int j = l & 3, k = l >> 2;
    F2 d[4][3][2];   // [var][direction][pair]
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        float sx[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            sx[i] = 0.f;
#pragma unroll
            for (int m = 0; m < 4; ++m) sx[i] = fma(fp.D[i * 4 + m], qx[v][m], sx[i]);
        }
        F2 sy[2] = {F2(0.f), F2(0.f)}, sz[2] = {F2(0.f), F2(0.f)};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            float ly[4], lz[4];   // the x-lines (m, k) and (j, m)
            ld_xline(sm.u[v], sw<P>(4 * (m + 4 * k), swz), ly);
            ld_xline(sm.u[v], sw<P>(4 * (j + 4 * m), swz), lz);
            const F2 cy(fp.D[j * 4 + m]), cz(fp.D[k * 4 + m]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                sy[h] = fma2(cy, F2(ly[2 * h], ly[2 * h + 1]), sy[h]);
                sz[h] = fma2(cz, F2(lz[2 * h], lz[2 * h + 1]), sz[h]);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            d[v][0][h] = F2(sx[2 * h], sx[2 * h + 1]) * F2(fp.jac[0]);
            d[v][1][h] = sy[h] * F2(fp.jac[1]);
            d[v][2][h] = sz[h] * F2(fp.jac[2]);
        }
    }
    __nv_bfloat16* st = reinterpret_cast<__nv_bfloat16*>(&sm.g[0][0]);   // [channel][64 points]
    F2 ir[2], nir[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        ir[h] = F2(1.0f / qx[0][2 * h], 1.0f / qx[0][2 * h + 1]);
        nir[h] = neg2(ir[h]);
    }
    const __nv_bfloat162 lo = __float2bfloat162_rn(-kFeatClip), hi = __float2bfloat162_rn(kFeatClip);
    auto put = [&](int c, const F2 (&x)[2]) {   // x: the channel minus its mean
        uint32_t w[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const F2 y = x[h] * F2(fp.inv_scale[c]);
            const __nv_bfloat162 r = __hmin2(__hmax2(__floats2bfloat162_rn(y.v.x, y.v.y), lo), hi);
            w[h] = *reinterpret_cast<const uint32_t*>(&r);
        }
        *reinterpret_cast<uint2*>(&st[c * 64 + 4 * l]) = make_uint2(w[0], w[1]);
    };
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const F2 nm(-fp.mean[v]);
        const F2 x[2] = {F2(qx[v][0], qx[v][1]) + nm, F2(qx[v][2], qx[v][3]) + nm};
        put(v, x);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        F2 nv[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) nv[h] = F2(qx[1 + a][2 * h], qx[1 + a][2 * h + 1]) * nir[h];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const F2 nm(-fp.mean[5 + 3 * a + b]);
            F2 x[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) x[h] = fma2(fma2(nv[h], d[0][b][h], d[1 + a][b][h]), ir[h], nm);
            put(5 + 3 * a + b, x);
        }
    }
    __syncwarp();
    if (live) {
        // tile (e / 128), channel c: a 128 x 64 block, row e % 128, 16-byte
        // chunk kc at ((row / 8) * 1024 + kc * 128 + (row % 8) * 16) bytes
        char* tile = reinterpret_cast<char*>(fp.X) + (size_t)(e >> 7) * (128 * 64 * 2 * kFeatChan);
        const int r = (int)(e & 127);
        for (int q8 = l; q8 < kFeatChan * 8; q8 += 16) {
            const int c = q8 >> 3, kc = q8 & 7;
            *reinterpret_cast<uint4*>(tile + (size_t)c * (128 * 64 * 2) + (r >> 3) * 1024 + kc * 128 + (r & 7) * 16) =
                *reinterpret_cast<const uint4*>(&st[c * 64 + 8 * kc]);
        }
    }
    __syncwarp();   // the gradient rows are P2's from here
}

// Inviscid part of the face corrections at the two faces of a line. Each
// face's interface flux F_I is solved once, by the element on its plus side
// (the face is that element's minus face): there j = F_I - Fe_own and F_I is
// stored for the neighbour; on the element's plus face j = -Fe_own here and
// phase B adds the neighbour's F_I. Slip walls (rhs.cu:311-339) are complete
// here: j = [0, 0, p_wall, 0, 0] - Fe_own with p_wall from the own flux.
template <class M, int D, class P, class C>
__device__ __forceinline__ void wall_face(const FaceState<C>& so, const C* fe, C* j) {
    const C pw = fe[2] - so.q[2] * so.q[2] * so.ir;
#pragma unroll
    for (int v = 0; v < NV; ++v) j[v] = -fe[v];
    j[2] = pw - fe[2];
}

// so: the own face state (make_face_state of the own face values).
template <class M, int FLUX, int D, class P, class C>
__device__ __forceinline__ void minus_face(const FaceState<C>& so, const P* nbr, bool wall, C* j, C* fi, int rflux) {
    C fe[NV];
    euler_flux<D>(so, fe);
    if (wall) {
        wall_face<M, D, P, C>(so, fe, j);
        return;
    }
    const FaceState<C> sn = make_face_state<M, C, P>(nbr);
    if constexpr (FLUX == kFluxRuntime)
        interface_flux_rt<M, D>(rflux, sn, so, fi);
    else
        interface_flux<M, FLUX, D>(sn, so, fi);
#pragma unroll
    for (int v = 0; v < NV; ++v) j[v] = fi[v] - fe[v];
}

template <class M, int D, class P, class C>
__device__ __forceinline__ void plus_face(const FaceState<C>& so, bool wall, C* j) {
    C fe[NV];
    euler_flux<D>(so, fe);
    if (wall) {
        wall_face<M, D, P, C>(so, fe, j);
        return;
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) j[v] = -fe[v];
}

// Swizzled row offsets of the three lines of thread l, computed once per
// tile: x-line start, the four y-line points and the z-line points (4-byte
// rows: the bases of points mm < 2 and mm >= 2, + 16 mm).
template <class T>
struct LineIdx {
    int x;
    int y[4];
    int z[sizeof(T) == 4 ? 2 : 4];
};

template <class T>
__device__ __forceinline__ LineIdx<T> line_idx(int l, int swz) {
    LineIdx<T> li;
    li.x = sw<T>(4 * l, swz);
#pragma unroll
    for (int mm = 0; mm < 4; ++mm) li.y[mm] = sw<T>(line_pt<1>(l, mm), swz);
    if constexpr (sizeof(T) == 4) {
        li.z[0] = sw<T>(line_pt<2>(l, 0), swz);
        li.z[1] = sw<T>(line_pt<2>(l, 2), swz) - 32;
    } else {
#pragma unroll
        for (int mm = 0; mm < 4; ++mm) li.z[mm] = sw<T>(line_pt<2>(l, mm), swz);
    }
    return li;
}

template <int D, class T>
__device__ __forceinline__ int line_off(const LineIdx<T>& li, int mm) {
    if constexpr (D == 1) return li.y[mm];
    else if constexpr (sizeof(T) == 4) return li.z[mm >> 1] + 16 * mm;
    else return li.z[mm];
}

// the offsets in rows of the state type and of the flux type
template <class P, class C>
struct LineSet {
    LineIdx<P> p;
    LineIdx<C> c;
    template <class T>
    __device__ __forceinline__ const auto& of() const {
        if constexpr (sizeof(T) == sizeof(P)) return p;
        else return c;
    }
};

// load / store the 4 samples of the thread's direction-D line of a swizzled row
template <int D, class T, class L>
__device__ __forceinline__ void row_line_load(const T* row, const L& ls, T* w) {
    const auto& li = ls.template of<T>();
    if constexpr (D == 0) {
        ld_xline(row, li.x, w);
    } else {
#pragma unroll
        for (int mm = 0; mm < 4; ++mm) w[mm] = row[line_off<D>(li, mm)];
    }
}

template <int D, class T, class L>
__device__ __forceinline__ void row_line_store(T* row, const L& ls, const T* w) {
    const auto& li = ls.template of<T>();
    if constexpr (D == 0) {
        st_xline(row, li.x, w);
    } else {
#pragma unroll
        for (int mm = 0; mm < 4; ++mm) row[line_off<D>(li, mm)] = w[mm];
    }
}

// Viscous part at one face point: j += 1/2 Fv_own; to the face buffer for
// the neighbour's phase B: F_I - 1/2 Fv_own at a minus face (fi: the
// interface flux solved in the line pass), Fv_own (components 1..4) at a
// plus face.
// REG: the face's correction j is in registers (jreg), else in shared memory.
// s: the face state (make_face_state of the face values).
template <class M, int D, bool REG, class PA, class Slot, class P = typename PA::P_t, class C = typename PA::C_t>
__device__ __forceinline__ void viscous_face(const PA& A, Slot& sm, long long e, int l, int side,
                                             const FaceState<C>& s, const C* gt, bool live, C* jreg,
                                             const C* fi) {
    const int f = 2 * D + side;
    C fv[NV];
    const C mu = viscosity<M>(A.mu, A.suth, s);
    if constexpr (M::kWideState)
        viscous_flux_wide<D>(s, gt, mu, heat_coeff<M>(mu, A.kappa), fv);
    else
        viscous_flux<D>(s, gt, mu, fv);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if constexpr (REG)
            jreg[v] += (C)0.5 * fv[v];
        else
            sm.j[f - 2][v][l] += (C)0.5 * fv[v];
    }
    if (!live) return;
    if (side == 0) {
        C* out = A.fi + ((e * 3 + D) * NV) * NF + l;
        out[0] = fi[0];
#pragma unroll
        for (int v = 1; v < NV; ++v) out[v * NF] = fi[v] - (C)0.5 * fv[v];
    } else {
        C* out = A.fv + ((e * 3 + D) * 4) * NF + l;
#pragma unroll
        for (int v = 1; v < NV; ++v) out[(v - 1) * NF] = fv[v];
    }
}

// P2-P4: one direction of the gradient / face-value pass for line l.
// jd: the corrections at the line's two faces, where they stay in registers.
// qx: the thread's own x-line as P1 loaded it (used by the x pass instead of
// reading it back from shared memory). The z pass (the last one, run after
// the x and y gradients are in shared memory) also does the z faces' viscous
// part (P5 for z): its normal gradient components are traced from registers
// and the z-face corrections are stored once, complete.
template <class M, int FLUX, int D, bool W, class PA, class Slot, class P = typename PA::P_t, class C = typename PA::C_t>
__device__ __forceinline__ void line_pass(const PA& A, Slot& sm, long long e, int l, const LineSet<P, C>& li,
                                          bool live, const long long nb0, const long long nb1, bool xpair, P* oL, P* oR,
                                          C (&jd)[2][NV], C* fi, const P (&qx)[NV][4]) {
    using S = typename PA::S_t;
    const Mesh& m = A.m;
    P q[NV][4];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if constexpr (D == 0) {
#pragma unroll
            for (int a = 0; a < 4; ++a) q[v][a] = qx[v][a];
        } else {
            row_line_load<D>(sm.u[v], li, q[v]);
        }
    }
    P nL[NV], nR[NV];
    if constexpr (D == 1) {
        // y neighbours: the neighbour's x-line l (points (0..3, j, k), j = l & 3,
        // k = l >> 2) in one 128-bit load per variable, weighted with the trace
        // coefficient of row j and summed over the four rows of the k-plane by
        // the four lanes that hold them, so that lane l ends with the trace at
        // face point (i, k) = (l & 3, l >> 2), its own y-line. Slip walls (no
        // neighbour) load nothing and mirror the own face value instead.
        const int q4 = l & 3;
        const P cm = A.tp.eR[q4], cp = A.tp.eL[q4];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            trace4_lr(q[v], A.tp.eL, A.tp.eR, oL[v], oR[v]);
            const P refl = (v > 0 && v < 4) ? (P)-1.0 : (P)1.0;
            P wm[4] = {(P)0, (P)0, (P)0, (P)0}, wp[4] = {(P)0, (P)0, (P)0, (P)0};
            if (nb0 >= 0) ldc4w<W, S, P>(A.u_in + v * m.npts + nb0 * NE + 4 * l, wm);
            if (nb1 >= 0) ldc4w<W, S, P>(A.u_in + v * m.npts + nb1 * NE + 4 * l, wp);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                wm[a] *= cm;
                wp[a] *= cp;
            }
            const P sL = sum4_scatter(wm, q4);
            const P sR = sum4_scatter(wp, q4);
            nL[v] = nb0 >= 0 ? sL : oL[v] * refl;
            nR[v] = nb1 >= 0 ? sR : oR[v] * refl;
        }
    } else if (D == 0 && sizeof(P) == 4 && xpair) {
        // the warp's two elements are neighbours: each has the other's trace at
        // their common face already (the same FMA chain), so only the outer
        // neighbours are read (u64/c32 4.5% faster, 24^3 closure step 1.1%; f64
        // traces take two shuffles each and lost 0.3 to 0.9%)
        const bool odd = (threadIdx.x & LPE) != 0;
        P cm[4];
#pragma unroll
        for (int mm = 0; mm < 4; ++mm) cm[mm] = odd ? A.tp.eL[mm] : A.tp.eR[mm];
        const S* outer = A.u_in + (odd ? nb1 : nb0) * NE + 4 * l;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            trace4_lr(q[v], A.tp.eL, A.tp.eR, oL[v], oR[v]);
            P w[4];
            ldc4w<W, S, P>(outer + v * m.npts, w);
            const P t = trace4(w, cm);
            const P c = __shfl_xor_sync(0xffffffffu, odd ? oL[v] : oR[v], LPE);
            nL[v] = odd ? c : t;
            nR[v] = odd ? t : c;
        }
    } else {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        trace4_lr(q[v], A.tp.eL, A.tp.eR, oL[v], oR[v]);
        const P refl = (v > 0 && v < 4) ? (P)-1.0 : (P)1.0;
        if (D != 1 || nb0 >= 0) {   // only y can have walls: x and z neighbours always exist
            P w[4];
            const S* base = A.u_in + v * m.npts + nb0 * NE;
            if constexpr (D == 0) {
                ldc4w<W, S, P>(base + 4 * l, w);
            } else {
#pragma unroll
                for (int mm = 0; mm < 4; ++mm) w[mm] = ldc1<P>(base + line_pt<D>(l, mm));
            }
            nL[v] = trace4(w, A.tp.eR);
        } else {
            nL[v] = oL[v] * refl;
        }
        if (D != 1 || nb1 >= 0) {
            P w[4];
            const S* base = A.u_in + v * m.npts + nb1 * NE;
            if constexpr (D == 0) {
                ldc4w<W, S, P>(base + 4 * l, w);
            } else {
#pragma unroll
                for (int mm = 0; mm < 4; ++mm) w[mm] = ldc1<P>(base + line_pt<D>(l, mm));
            }
            nR[v] = trace4(w, A.tp.eL);
        } else {
            nR[v] = oR[v] * refl;
        }
    }
    }
    // corrected gradient along the line (BR1): the jump to the common value is
    // half the difference across the face; (n_L - o_L) g_L'/2 + (n_R - o_R)
    // g_R'/2 + D q, all scaled by the Jacobian, as one FMA chain per point
    // (kWideState: the jump formed from the common value, times g_L', g_R')
    C gnL[NV], gnR[NV];   // z pass: face values of the normal gradient components
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        C jl, jr;
        if constexpr (M::kWideState) {
            jl = (C)((P)0.5 * (nL[v] + oL[v]) - oL[v]);
            jr = (C)((P)0.5 * (nR[v] + oR[v]) - oR[v]);
        } else {
            jl = (C)(nL[v] - oL[v]);
            jr = (C)(nR[v] - oR[v]);
        }
        C gv[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            C gg = M::kWideState ? fma(-jr, A.sc.nr[D][a], -jl * A.sc.nl[D][a])
                                 : fma(jr, A.sc.hr[D][a], jl * A.sc.hl[D][a]);
#pragma unroll
            for (int mm = 0; mm < 4; ++mm) gg = fma(A.sc.d[D][a * 4 + mm], (C)q[v][mm], gg);
            if constexpr (sizeof(C) == 8) {
                if (A.flags & kRoundQ) gg = (C)(float)gg;
            }
            gv[a] = gg;
        }
        row_line_store<D>(sm.g[3 * v + D], li, gv);
        if constexpr (D == 2) trace4_lr(gv, A.tc.eL, A.tc.eR, gnL[v], gnR[v]);
    }
    // inviscid parts at the two faces of this line; F_I stays in registers
    // until the minus face's viscous flux is known (P5)
    C j0[NV], j1[NV];
    const FaceState<C> sL = make_face_state<M, C, P>(oL);
    const FaceState<C> sR = make_face_state<M, C, P>(oR);
    minus_face<M, FLUX, D, P, C>(sL, nL, D == 1 && nb0 < 0, j0, fi, A.flux);
    plus_face<M, D, P, C>(sR, D == 1 && nb1 < 0, j1);
    if constexpr (D == 2) {
        // z faces (never walls): the 11 gradient components the z flux reads,
        // the normal ones from registers, the x / y ones from shared memory
        C gL[15], gR[15];
#pragma unroll
        for (int c = 0; c < 15; ++c) {
            if (!grad_used<2>(c)) {
                gL[c] = (C)0;
                gR[c] = (C)0;
            } else if (c % 3 == 2) {
                gL[c] = gnL[c / 3];
                gR[c] = gnR[c / 3];
            } else {
                C w[4];
                row_line_load<2>(sm.g[c], li, w);
                trace4_lr(w, A.tc.eL, A.tc.eR, gL[c], gR[c]);
            }
        }
        viscous_face<M, 2, true>(A, sm, e, l, 0, sL, gL, live, j0, fi);
        viscous_face<M, 2, true>(A, sm, e, l, 1, sR, gR, live, j1, fi);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if constexpr (D == 0 || kLineUpdate<M, P, C>) {
            jd[0][v] = j0[v];
            jd[1][v] = j1[v];
        } else {
            sm.j[2 * D - 2][v][l] = j0[v];
            sm.j[2 * D - 1][v][l] = j1[v];
        }
    }
}

// The reference's y-face gradient slice multiplies with __fmul_rn, a float
// intrinsic, also in its f64 build (rhs.cu:145-160): products and pair sums
// in f32. Reproduced on request (kRefYSlice) for bit-level drop-in parity.
template <class C, class CC>
__device__ __forceinline__ C ref_y_slice(const C* w, const CC& c) {
    const float a = __fadd_rn(__fmul_rn((float)w[0], (float)c[0]), __fmul_rn((float)w[1], (float)c[1]));
    const float b = __fadd_rn(__fmul_rn((float)w[2], (float)c[2]), __fmul_rn((float)w[3], (float)c[3]));
    return (C)__fadd_rn(a, b);
}

// P5: face values and face gradient along the D-line of thread l, viscous
// flux at both faces of the line.
template <class M, int D, class PA, class Slot, class P = typename PA::P_t, class C = typename PA::C_t>
__device__ __forceinline__ void face_grad_pass(const PA& A, Slot& sm, long long e, int l,
                                               const LineSet<P, C>& li, bool wall0, bool wall1, bool live, const P* tL,
                                               const P* tR, C (&jd)[2][NV], const C* fi) {
    if (wall0 && wall1) return;
    C gL[15], gR[15];
    const bool ref_y = D == 1 && sizeof(C) == 8 && (A.flags & kRefYSlice);
#pragma unroll
    for (int c = 0; c < 15; ++c) {
        if (!grad_used<D>(c)) {
            gL[c] = (C)0;
            gR[c] = (C)0;
            continue;
        }
        C w[4];
        row_line_load<D>(sm.g[c], li, w);
        if (ref_y) {
            gL[c] = ref_y_slice(w, A.tc.eL);
            gR[c] = ref_y_slice(w, A.tc.eR);
        } else {
            trace4_lr(w, A.tc.eL, A.tc.eR, gL[c], gR[c]);
        }
    }
    // face values: kept in registers from the line pass (f32), else recomputed
    P qL[NV], qR[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if constexpr (sizeof(P) == 4) {
            qL[v] = tL[v];
            qR[v] = tR[v];
        } else {
            P w[4];
            row_line_load<D>(sm.u[v], li, w);
            trace4_lr(w, A.tp.eL, A.tp.eR, qL[v], qR[v]);
        }
    }
    if (!wall0) {
        const FaceState<C> st = make_face_state<M, C, P>(qL);
        viscous_face<M, D, D == 0 || kLineUpdate<M, P, C>>(A, sm, e, l, 0, st, gL, live, jd[0], fi);
    }
    if (!wall1) {
        const FaceState<C> st = make_face_state<M, C, P>(qR);
        viscous_face<M, D, D == 0 || kLineUpdate<M, P, C>>(A, sm, e, l, 1, st, gR, live, jd[1], fi);
    }
}

// Rows of the dead gradient that hold F_y and F_z between P6 and P7. F_y of
// rho w is F_z of rho v, and the mass fluxes are the momenta, read from the
// state. (kWideState: all ten fluxes, F_y in rows 0-4 and F_z in rows 5-9.)
constexpr int kFy1 = 0, kFy2 = 1, kFy3 = 2, kFy4 = 3, kFz1 = 4, kFz2 = kFy3, kFz3 = 5, kFz4 = 6;

template <int D, class Slot>
__device__ __forceinline__ const auto* flux_row(const Slot& sm, int v) {
    if constexpr (D == 1)
        return v == 0 ? &sm.u[2][0] : &sm.g[v == 1 ? kFy1 : v == 2 ? kFy2 : v == 3 ? kFy3 : kFy4][0];
    else
        return v == 0 ? &sm.u[3][0] : &sm.g[v == 1 ? kFz1 : v == 2 ? kFz2 : v == 3 ? kFz3 : kFz4][0];
}

// RK combination a*u0 + b*u + c*R of variable v on the x-line, or (deferred
// RK) the unrounded R for phase B. u is still in shared memory (x: the line's
// offset there): a global load here would wait for the stores of the variable
// before, which may alias it (96^3 mixed step 1.6% slower).
template <class PA, class Slot, class P = typename PA::P_t, class C = typename PA::C_t>
__device__ __forceinline__ void store_update(const PA& A, const Slot& sm, int x, long long ec, int l, int v,
                                             const C (&rt)[4]) {
    using S = typename PA::S_t;
    const Mesh& m = A.m;
    const bool defer = (A.flags & kDeferRK) != 0;
    S* dst = A.u_out + v * m.npts + ec * NE + 4 * l;
    if (defer) {
        stg4<S, C>(dst, rt);
        return;
    }
    P un[4], u0v[4], out[4];
    ld_xline(sm.u[v], x, un);
    if (A.flags & kHasU0) ldc4<S, P>(A.u0 + v * m.npts + ec * NE + 4 * l, u0v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        P o = A.rb * un[i] + A.rc * (P)rt[i];
        if (A.flags & kHasU0) o = A.ra * u0v[i] + A.rb * un[i] + A.rc * (P)rt[i];
        out[i] = o;
    }
    stg4<S, P>(dst, out);
}

// P7 + P8 of phase A for one live element: the y / z divergences of the
// x-line's four points, RHS = -div + forcing, own-face lifting
// -(j_L g_L' + j_R g_R') jac, then the RK combination, or (deferred RK) the
// unrounded RHS + own lift for phase B.
// The y derivative at (i, j, k) reads F_y at (i, 0..3, k): the four x-lines of
// the thread's k-plane; the z derivative reads F_z at (i, j, 0..3): the four
// x-lines of its j-column. Each is one 128-bit shared load per x-line (lanes
// of the same plane / column load the same line: broadcasts), so no pass
// along y and z lines and no barrier before the update. Operation order per
// point as a derivative along the line: D[a][0] F_0, then FMAs for m = 1..3.
template <class M, class PA, class Slot, class P = typename PA::P_t, class C = typename PA::C_t>
__device__ __forceinline__ void stage_a_update(const PA& A, Slot& sm, long long ec, int l, int swz,
                                               const C (&divx)[NV][4], const C (&jx)[2][NV]) {
    static_assert(M::kWideState && sizeof(C) == 4, "every other pipeline updates by lines");
    const int lj = l & 3, lk = l >> 2;   // this x-line's (j, k)
    C cy[4], cz[4];   // derivative rows of this thread's j (y) and k (z)
#pragma unroll
    for (int mm = 0; mm < 4; ++mm) {
        cy[mm] = A.sc.d[1][lj * 4 + mm];
        cz[mm] = A.sc.d[2][lk * 4 + mm];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        C rt[4], dy[4], dz[4], jy0[4], jy1[4], jz0[4], jz1[4];
        const C* fy = sm.g[v];
        const C* fz = sm.g[5 + v];
#pragma unroll
        for (int mm = 0; mm < 4; ++mm) {
            C f[4];
            ld_xline(fy, sw<C>(4 * (mm + 4 * lk), swz), f);
#pragma unroll
            for (int i = 0; i < 4; ++i) dy[i] = mm == 0 ? cy[0] * f[i] : fma(cy[mm], f[i], dy[i]);
        }
#pragma unroll
        for (int mm = 0; mm < 4; ++mm) {
            C f[4];
            ld_xline(fz, sw<C>(4 * (lj + 4 * mm), swz), f);
#pragma unroll
            for (int i = 0; i < 4; ++i) dz[i] = mm == 0 ? cz[0] * f[i] : fma(cz[mm], f[i], dz[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            rt[i] = -((divx[v][i] + dy[i]) + dz[i]);
            if (v == 1) rt[i] += A.forcing;
        }
        ld4s(&sm.j[0][v][4 * lk], jy0);
        ld4s(&sm.j[1][v][4 * lk], jy1);
        ld4s(&sm.j[2][v][4 * lj], jz0);
        ld4s(&sm.j[3][v][4 * lj], jz1);
        const C jx0 = jx[0][v], jx1 = jx[1][v];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            C r = rt[i];
            // lifting -(j_L g_L' + j_R g_R') jac of the six faces (rk.cu:12-25)
            r = fma(jx0, A.sc.nl[0][i], r);
            r = fma(jx1, A.sc.nr[0][i], r);
            r = fma(jy0[i], A.sc.nl[1][lj], r);
            r = fma(jy1[i], A.sc.nr[1][lj], r);
            r = fma(jz0[i], A.sc.nl[2][lk], r);
            rt[i] = fma(jz1[i], A.sc.nr[2][lk], r);
        }
        store_update(A, sm, sw<P>(4 * l, swz), ec, l, v, rt);
    }
}

// P7 + P8 with the face corrections in registers (kLineUpdate): the thread's
// y-line takes the y divergence and the lifting of its two faces into rows
// kR.., its z-line adds the z terms, and the x-line adds divx and the x lifting.
// One line of four values in and out of shared memory per variable and
// direction. Called by whole warps.
constexpr int kR = 7;   // first row of the partial updates (rows 0-6: the fluxes)

// The divergence (DIV) and / or the lifting (LIFT) of the thread's direction-D
// line of variable v, added to r (FRESH: r is set); f: the line's fluxes, j0, j1:
// its faces' corrections. A direction's terms are summed on their own, the
// divergence first, and added to r once: with the lifting first and the
// divergence chained onto r the sums took more roundings at the size of one
// direction's terms (error of an f64 right-hand side 1.02 times as large, f32
// 1.05).
template <int D, bool FRESH, bool DIV, bool LIFT, class PA, class C>
__device__ __forceinline__ void line_terms(const PA& A, const C* f, C j0, C j1, C* r) {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if constexpr (DIV) {
            C d = A.sc.nd[D][a * 4] * f[0];
#pragma unroll
            for (int mm = 1; mm < 4; ++mm) d = fma(A.sc.nd[D][a * 4 + mm], f[mm], d);
            if constexpr (LIFT) {
                d = fma(j0, A.sc.nl[D][a], d);
                d = fma(j1, A.sc.nr[D][a], d);
            }
            r[a] = FRESH ? d : r[a] + d;
        } else if constexpr (LIFT) {
            r[a] = fma(j0, A.sc.nl[D][a], r[a]);
            r[a] = fma(j1, A.sc.nr[D][a], r[a]);
        }
    }
}

// One pass of the update over the thread's direction-D lines (y or z): rows kR..
// FRESH: they start here.
template <class M, int D, bool FRESH, bool DIV, bool LIFT, class PA, class Slot, class L, class C>
__device__ __forceinline__ void update_pass(const PA& A, Slot& sm, const L& li, const C (&j)[2][NV]) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        C f[4], r[4];
        if constexpr (DIV) row_line_load<D>(flux_row<D>(sm, v), li, f);
        if constexpr (!FRESH) row_line_load<D>(&sm.g[kR + v][0], li, r);
        line_terms<D, FRESH, DIV, LIFT>(A, f, j[0][v], j[1][v], r);
        row_line_store<D>(&sm.g[kR + v][0], li, r);
    }
    __syncwarp();
}

template <class M, class PA, class Slot, class P = typename PA::P_t, class C = typename PA::C_t>
__device__ __forceinline__ void stage_a_update_lines(const PA& A, Slot& sm, long long ec, int l,
                                                     const LineSet<P, C>& li, bool live, const C (&divx)[NV][4],
                                                     const C (&jx)[2][NV], const C (&jy)[2][NV],
                                                     const C (&jz)[2][NV]) {
    if constexpr (sizeof(C) == 8) {
        if (A.flags & kRoundRhs) {
            // the volume terms of all directions are rounded before the lifting
            update_pass<M, 1, true, true, false>(A, sm, li, jy);
            update_pass<M, 2, false, true, false>(A, sm, li, jz);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                C r[4];
                row_line_load<0>(&sm.g[kR + v][0], li, r);
#pragma unroll
                for (int a = 0; a < 4; ++a) r[a] = (C)(float)(r[a] + divx[v][a]);
                line_terms<0, false, false, true>(A, r, jx[0][v], jx[1][v], r);
                row_line_store<0>(&sm.g[kR + v][0], li, r);
            }
            __syncwarp();
            update_pass<M, 1, false, false, true>(A, sm, li, jy);
            update_pass<M, 2, false, false, true>(A, sm, li, jz);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                C r[4];
                row_line_load<0>(&sm.g[kR + v][0], li, r);
                if (live) store_update(A, sm, li.p.x, ec, l, v, r);
            }
            return;
        }
    }
    update_pass<M, 1, true, true, true>(A, sm, li, jy);
    update_pass<M, 2, false, true, true>(A, sm, li, jz);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        C r[4], x[4];
        row_line_load<0>(&sm.g[kR + v][0], li, r);
#pragma unroll
        for (int a = 0; a < 4; ++a) x[a] = divx[v][a];
        line_terms<0, false, false, true>(A, x, jx[0][v], jx[1][v], x);
#pragma unroll
        for (int a = 0; a < 4; ++a) r[a] += x[a];
        if (live) store_update(A, sm, li.p.x, ec, l, v, r);
    }
}

// Phase A of an f64 state reads its x-lines with 256-bit loads in the kernels
// of 4 elements per block; the kernels of 2 take any 16-byte aligned state.
template <class S, int EPB>
constexpr bool kWideLoads = sizeof(S) == 8 && EPB == 4;

// One tile of phase A: EPB elements starting at A.e0 + tile * EPB, LPE
// threads each. Called by whole warps: an element's 16 threads are half of one,
// so nothing here waits for the block's other warps.
template <class M, int FLUX, int EPB, bool FEAT = false, class PA>
__device__ __forceinline__ void stage_a_tile(const PA& A, unsigned char* smem_raw, long long tile) {
    using S = typename PA::S_t;
    using P = typename PA::P_t;
    using C = typename PA::C_t;
    constexpr bool W = kWideLoads<S, EPB>;
    const int l = threadIdx.x & (LPE - 1);
    const int es = threadIdx.x / LPE;
    const int swz = (es & 1) << 3;
    const LineSet<P, C> li{line_idx<P>(l, swz), line_idx<C>(l, swz)};
    SlotFor<M, P, C>& sm = reinterpret_cast<SlotFor<M, P, C>*>(smem_raw)[es];
    const long long e = A.e0 + tile * EPB + es;
    const bool live = e < A.e1;
    const long long ec = live ? e : 0;
    const Mesh& m = A.m;
    int ex, ey, ez;
    elem_coords(m, ec, ex, ey, ez);
    const long long nxm = neighbour(m, ex, ey, ez, 0, 0), nxp = neighbour(m, ex, ey, ez, 0, 1);
    const long long nym = neighbour(m, ex, ey, ez, 1, 0), nyp = neighbour(m, ex, ey, ez, 1, 1);
    const long long nzm = neighbour(m, ex, ey, ez, 2, 0), nzp = neighbour(m, ex, ey, ez, 2, 1);

    // ---- P1: the element's x-lines -> smem (and kept for the x pass)
    P qx[NV][4];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if (live) {
            ldc4w<W, S, P>(A.u_in + v * m.npts + ec * NE + 4 * l, qx[v]);
        } else {
#pragma unroll
            for (int a = 0; a < 4; ++a) qx[v][a] = (P)1.0;
        }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) st_xline(sm.u[v], li.p.x, qx[v]);   // after every load is issued
    __syncwarp();
    if constexpr (FEAT) stage_a_features(A, sm, ec, l, swz, live, qx);

    // ---- P2-P4: face values, gradient, interface fluxes per direction
    // x neighbours of each other: the two elements of the warp
    const bool xpair = sizeof(P) == 4 && __all_sync(0xffffffffu, live && ((es & 1) ? nxm == e - 1 : nxp == e + 1));
    P tr[3][2][NV];   // own face values of this thread's lines (kept only for f32 state arithmetic)
    C jx[2][NV];      // this x-line's x-face corrections
    C jy[2][NV], jz[2][NV];   // kLineUpdate: the y- and z-line's
    C fi[3][NV];      // interface fluxes at the minus faces of this thread's lines
    line_pass<M, FLUX, 0, W>(A, sm, ec, l, li, live, nxm, nxp, xpair, tr[0][0], tr[0][1], jx, fi[0], qx);
    line_pass<M, FLUX, 1, W>(A, sm, ec, l, li, live, nym, nyp, false, tr[1][0], tr[1][1], jy, fi[1], qx);
    __syncwarp();   // the x and y gradients, read by the z faces
    line_pass<M, FLUX, 2, W>(A, sm, ec, l, li, live, nzm, nzp, false, tr[2][0], tr[2][1], jz, fi[2], qx);
    __syncwarp();

    // ---- P5: viscous face fluxes of the x and y faces, face records (the z
    // faces are done in the z pass)
    face_grad_pass<M, 0>(A, sm, ec, l, li, false, false, live, tr[0][0], tr[0][1], jx, fi[0]);
    face_grad_pass<M, 1>(A, sm, ec, l, li, nym < 0, nyp < 0, live, tr[1][0], tr[1][1], jy, fi[1]);
    __syncwarp();

    // ---- P6: pointwise fluxes of the x-line's points (own points only; the
    // point order is rotated by k so the 16 lanes of an element hit distinct
    // banks). F_y, F_z -> smem for the y / z divergences; the x-line's F_x
    // never leaves the thread: its x-divergence (with its sign, on top of the
    // forcing) is accumulated here (point i contributes column i of the x
    // derivative) and kept until P8.
    C divx[NV][4];
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int a = 0; a < 4; ++a) divx[v][a] = !M::kWideState && v == 1 ? A.forcing : (C)0;
    if constexpr (kLineUpdate<M, P, C> && sizeof(C) == 4) {
        // two points of the line at a time, in packed arithmetic (64-bit shared
        // accesses; the pair is rotated by k's high bit so that the 16 lanes
        // of an element hit distinct banks)
        const int hk = l >> 3;
#pragma unroll 1
        for (int it = 0; it < 2; ++it) {
            const int i = 2 * (it ^ hk);
            const int p = li.c.x + i;
            const VolumeFluxes2 F = volume_fluxes2<M>(
                [&](int v) { return F2(*reinterpret_cast<const float2*>(&sm.u[v][p])); },
                [&](int c) { return F2(*reinterpret_cast<const float2*>(&sm.g[c][p])); }, A.mu, A.suth);
            auto put = [&](int row, const F2& x) { *reinterpret_cast<float2*>(&sm.g[row][p]) = x.v; };
            const float2 q1 = *reinterpret_cast<const float2*>(&sm.u[1][p]);
            put(kFy1, F.m01);
            put(kFy2, F.m11);
            put(kFy3, F.m12);
            put(kFy4, F.e[1]);
            put(kFz1, F.m02);
            put(kFz3, F.m22);
            put(kFz4, F.e[2]);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const float d0 = A.sc.nd[0][a * 4 + i], d1 = A.sc.nd[0][a * 4 + i + 1];
                divx[0][a] = fma(d1, q1.y, fma(d0, q1.x, divx[0][a]));
                divx[1][a] = fma(d1, F.m00.v.y, fma(d0, F.m00.v.x, divx[1][a]));
                divx[2][a] = fma(d1, F.m01.v.y, fma(d0, F.m01.v.x, divx[2][a]));
                divx[3][a] = fma(d1, F.m02.v.y, fma(d0, F.m02.v.x, divx[3][a]));
                divx[4][a] = fma(d1, F.e[0].v.y, fma(d0, F.e[0].v.x, divx[4][a]));
            }
        }
    } else {
        const int lk = l >> 2;
#pragma unroll 1
        for (int it = 0; it < 4; ++it) {
            const int i = (it + lk) & 3;
            const int p = sw<C>(4 * l + i, swz), pp = sw<P>(4 * l + i, swz);
            C g[15];
#pragma unroll
            for (int c = 0; c < 15; ++c) g[c] = sm.g[c][p];
            P qp[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) qp[v] = sm.u[v][pp];
            const FaceState<C> s = make_face_state<M, C, P>(qp);
            C fx[NV];
            if constexpr (M::kWideState) {
                C F[3][NV];
                const C mu = viscosity<M>(A.mu, A.suth, s);
                volume_fluxes_wide<C>(s, g, mu, heat_coeff<M>(mu, A.kappa), F);
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    sm.g[v][p] = F[1][v];
                    sm.g[5 + v][p] = F[2][v];
                    fx[v] = F[0][v];
                }
            } else {
                const VolumeFluxes<C> F = volume_fluxes<C>(s, g, viscosity<M>(A.mu, A.suth, s));
                sm.g[kFy1][p] = F.m01;
                sm.g[kFy2][p] = F.m11;
                sm.g[kFy3][p] = F.m12;
                sm.g[kFy4][p] = F.e[1];
                sm.g[kFz1][p] = F.m02;
                sm.g[kFz3][p] = F.m22;
                sm.g[kFz4][p] = F.e[2];
                fx[0] = s.q[1];
                fx[1] = F.m00;
                fx[2] = F.m01;
                fx[3] = F.m02;
                fx[4] = F.e[0];
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const C d = M::kWideState ? A.sc.d[0][a * 4 + i] : A.sc.nd[0][a * 4 + i];
#pragma unroll
                for (int v = 0; v < NV; ++v) divx[v][a] = fma(d, fx[v], divx[v][a]);
            }
        }
    }
    __syncwarp();

    // ---- P7 + P8: y / z divergences, RHS, lifting, RK combination (or the
    // RHS alone for phase B)
    if constexpr (kLineUpdate<M, P, C>)
        stage_a_update_lines<M>(A, sm, ec, l, li, live, divx, jx, jy, jz);
    else if (live)
        stage_a_update<M>(A, sm, ec, l, swz, divx, jx);
}

// Blocks per SM the register budget is set for. f32 state arithmetic and
// fluxes (the all-f32 pipeline, and the reference's default of an f64 state
// with f32 arithmetic): at most 128 registers per thread, so that 8 blocks of
// 4 elements (16 of 2) fit per SM, the occupancy the shared memory allows
// (u64/c32 at 64^3: phase A 1161 us at the 5 blocks its free choice of 198
// registers allowed, 931 us at 8; its SLAU2 fast-math kernel does not spill,
// some IEEE, AUSM+ and Sutherland variants spill 8-72 bytes). Mixed precision (f64 state, f32
// fluxes): 6 blocks of 4 elements, at most 168 registers (left free, the
// compiler takes 190 and 5 blocks fit: 10% slower at 96^3; 7 blocks spill and
// are 9% slower). Slots with f64 gradients are larger; shared memory bounds
// those kernels first.
template <class S, class P, class C, int EPB>
constexpr int stage_a_min_blocks() {
    if (sizeof(P) == 4 && sizeof(C) == 4) return 32 / EPB;
    if (sizeof(S) == 8 && sizeof(P) == 8 && sizeof(C) == 4) return 24 / EPB;
    return 1;
}

template <class S, class P, class C, class M, int FLUX, int EPB, bool FEAT = false>
__global__ void __launch_bounds__(LPE * EPB, (stage_a_min_blocks<S, P, C, EPB>())) stage_a_kernel(const StageAParams<S, P, C> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // the kernel launched next may become resident on SMs this grid no longer
    // needs; it reads nothing before griddepcontrol.wait, i.e. before this grid
    // is complete (the closure network: its prologue and weight prefetch
    // overlap). The wait here is for the kernel before, when this launch is
    // its programmatic dependent.
    dependent_start();
    stage_a_tile<M, FLUX, EPB, FEAT>(A, smem_raw, blockIdx.x);
}

template <class S, class P, class C>
struct StageBParams {
    using S_t = S;
    using P_t = P;
    using C_t = C;
    S* u_out;
    const S* rhs;   // deferred RK: phase A's RHS
    const S* u_in;
    const S* u0;
    const C* fv;
    const C* fi;
    Mesh m;
    Tab<C> tc;
    C jac[3];
    P ra, rb, rc;
    int flags;
    long long e0, e1;   // element range of this launch
};

// Phase B: the neighbour-dependent part of the face corrections,
//   plus faces:  j += F_I - 1/2 Fv_nbr (the plus neighbour's minus-face record)
//   minus faces: j += -1/2 Fv_nbr (the minus neighbour's plus-face record)
// lifted with -(j g') jac (rk.cu:12-25) over the element's non-wall faces and
// added to the new state (times rc), or (deferred RK) folded into
// u_out = ra*u0 + rb*u_in + rc*(RHS + lift). 16 threads per element, each the
// x-line l = j + 4k (128-bit accesses).
// Scalar load of data written earlier by the same kernel (COH) or by an
// earlier launch; phase B reads each face record and RHS value once, so the
// latter loads are evict-first (ld.global.cs): the L2 keeps the new state for
// the next phase A instead (48^3 f32: phase B 117.6 -> 117.0 us).
template <bool COH, class T>
__device__ __forceinline__ T ldf(const T* p) {
    if constexpr (COH)
        return *p;
    else
        return __ldcs(p);
}

// 4-wide load of data read once (evict-first: the face records and the RHS
// phase B consumes, in buffers of this library: 32-byte aligned lines), or
// coherent inside a persistent kernel (COH)
template <bool COH, class S, class P>
__device__ __forceinline__ void ld4once(const S* p, P* q) {
    if constexpr (COH) {
        ldc4<S, P>(p, q);
    } else if constexpr (sizeof(S) == 8) {
        double a, b, c, d;
        asm volatile("ld.global.cs.v4.f64 {%0,%1,%2,%3}, [%4];"
                     : "=d"(a), "=d"(b), "=d"(c), "=d"(d)
                     : "l"(p)
                     : "memory");
        q[0] = (P)a; q[1] = (P)b; q[2] = (P)c; q[3] = (P)d;
    } else {
        const float4 v = __ldcs(reinterpret_cast<const float4*>(p));
        q[0] = (P)v.x; q[1] = (P)v.y; q[2] = (P)v.z; q[3] = (P)v.w;
    }
}

// One tile of phase B: EPB elements starting at B.e0 + tile * EPB. COH: the
// face buffers and the RHS were written by this same launch (a persistent
// kernel after its grid barrier), so they are read through the coherent path.
// Per-element context of phase B: the element, its x-line and its neighbours.
template <class C>
struct BCtx {
    long long e;
    int nxm, nxp, nym, nyp, nzm, nzp;   // 32-bit: each record address is one wide multiply-add
    int l, lj, lk;
    C hx, hy, hz;
};

template <class PB, class C = typename PB::C_t>
__device__ __forceinline__ BCtx<C> b_ctx(const PB& B, long long e, int l) {
    BCtx<C> x;
    const Mesh& m = B.m;
    int ex, ey, ez;
    elem_coords(m, e, ex, ey, ez);
    x.e = e;
    x.l = l;
    x.lj = l & 3;
    x.lk = l >> 2;
    x.nxm = neighbour(m, ex, ey, ez, 0, 0);
    x.nxp = neighbour(m, ex, ey, ez, 0, 1);
    x.nym = neighbour(m, ex, ey, ez, 1, 0);
    x.nyp = neighbour(m, ex, ey, ez, 1, 1);
    x.nzm = neighbour(m, ex, ey, ez, 2, 0);
    x.nzp = neighbour(m, ex, ey, ez, 2, 1);
    x.hx = (C)0.5 * B.jac[0];
    x.hy = (C)0.5 * B.jac[1];
    x.hz = (C)0.5 * B.jac[2];
    return x;
}

// Phase B of variable v on the x-line x.l of element x.e, in two halves:
// b_load gathers everything the update reads (the lifted neighbour terms
// accumulated from the face records, and the RHS / state values), b_store
// forms the new state and stores it. A thread that handles several variables
// issues all their loads before its first store.
template <class P, class C>
struct BVar {
    C acc[4];   // lifted neighbour face terms
    C r[4];     // deferred RK: phase A's RHS
    P un[4];    // deferred RK: u_in; otherwise the current u_out
    P u0[4];
};

template <bool COH, class PB, class C = typename PB::C_t, class P = typename PB::P_t>
__device__ __forceinline__ BVar<P, C> b_load(const PB& B, const BCtx<C>& x, int v) {
    using S = typename PB::S_t;
    const Mesh& m = B.m;
    const bool defer = (B.flags & kDeferRK) != 0;
    const long long e = x.e;
    const int nxm = x.nxm, nxp = x.nxp, nym = x.nym, nyp = x.nyp, nzm = x.nzm, nzp = x.nzp;
    // the records of an element, at this variable
    auto fi = [&](int nb, int dir) { return B.fi + (dir * NV + v) * NF + (size_t)(unsigned)nb * (3 * NV * NF); };
    auto fvr = [&](int nb, int dir) { return B.fv + (dir * 4 + v - 1) * NF + (size_t)(unsigned)nb * (3 * 4 * NF); };
    const int l = x.l, lj = x.lj, lk = x.lk;
    const C hx = x.hx, hy = x.hy, hz = x.hz;
    BVar<P, C> d;
#pragma unroll
    for (int i = 0; i < 4; ++i) d.acc[i] = (C)0;
    // plus faces: the plus neighbours' minus-face records F_I - 1/2 Fv
    {
        const C f0 = ldf<COH>(fi(nxp, 0) + l);
#pragma unroll
        for (int i = 0; i < 4; ++i) d.acc[i] = fma(-B.jac[0] * B.tc.gR[i], f0, d.acc[i]);
    }
    if (nyp >= 0) {
        C w[4];
        ld4once<COH, C, C>(fi(nyp, 1) + 4 * lk, w);
        const C c = -B.jac[1] * B.tc.gR[lj];
#pragma unroll
        for (int i = 0; i < 4; ++i) d.acc[i] = fma(c, w[i], d.acc[i]);
    }
    {
        C w[4];
        ld4once<COH, C, C>(fi(nzp, 2) + 4 * lj, w);
        const C c = -B.jac[2] * B.tc.gR[lk];
#pragma unroll
        for (int i = 0; i < 4; ++i) d.acc[i] = fma(c, w[i], d.acc[i]);
    }
    if (v > 0) {
        // minus faces: the minus neighbours' viscous fluxes at their plus faces
        {
            const C a0 = ldf<COH>(fvr(nxm, 0) + l);
#pragma unroll
            for (int i = 0; i < 4; ++i) d.acc[i] = fma(hx * B.tc.gL[i], a0, d.acc[i]);
        }
        if (nym >= 0) {
            C w[4];
            ld4once<COH, C, C>(fvr(nym, 1) + 4 * lk, w);
            const C c = hy * B.tc.gL[lj];
#pragma unroll
            for (int i = 0; i < 4; ++i) d.acc[i] = fma(c, w[i], d.acc[i]);
        }
        {
            C w[4];
            ld4once<COH, C, C>(fvr(nzm, 2) + 4 * lj, w);
            const C c = hz * B.tc.gL[lk];
#pragma unroll
            for (int i = 0; i < 4; ++i) d.acc[i] = fma(c, w[i], d.acc[i]);
        }
    }
    const long long off = v * m.npts + e * NE + 4 * l;
    if (defer) {
        ld4once<COH, S, C>(B.rhs + off, d.r);
        ldc4<S, P>(B.u_in + off, d.un);
        if (B.flags & kHasU0) ldc4<S, P>(B.u0 + off, d.u0);
    } else if (sizeof(S) == 8 && (B.flags & kWideOut)) {
        ld4wide(B.u_out + off, d.un);
    } else {
        ldc4<S, P>(B.u_out + off, d.un);
    }
    return d;
}

template <class PB, class C = typename PB::C_t, class P = typename PB::P_t>
__device__ __forceinline__ void b_store(const PB& B, const BCtx<C>& x, int v, const BVar<P, C>& d) {
    using S = typename PB::S_t;
    const bool defer = (B.flags & kDeferRK) != 0;
    const long long off = v * B.m.npts + x.e * NE + 4 * x.l;
    P out[4];
    if (defer) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const C rt = d.r[i] + d.acc[i];
            P o = B.rb * d.un[i] + B.rc * (P)rt;
            if (B.flags & kHasU0) o = B.ra * d.u0[i] + B.rb * d.un[i] + B.rc * (P)rt;
            out[i] = o;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) out[i] = d.un[i] + B.rc * (P)d.acc[i];
    }
    if (sizeof(S) == 8 && (B.flags & kWideOut))
        st4wide(B.u_out + off, out);
    else
        stg4<S, P>(B.u_out + off, out);
}

template <bool COH, class PB, class C = typename PB::C_t>
__device__ __forceinline__ void stage_b_var(const PB& B, const BCtx<C>& x, int v) {
    b_store(B, x, v, b_load<COH>(B, x, v));
}

// One tile of phase B: EPB elements starting at B.e0 + tile * EPB, 16
// threads (x-lines) each, all five variables per thread. COH: the face
// buffers and the RHS were written by this same launch (a persistent kernel
// after its grid barrier), so they are read through the coherent path.
template <int EPB, bool COH, class PB>
__device__ __forceinline__ void stage_b_tile(const PB& B, long long tile) {
    const int l = threadIdx.x & (LPE - 1);
    const long long e = B.e0 + tile * EPB + threadIdx.x / LPE;
    if (e >= B.e1) return;
    const auto x = b_ctx(B, e, l);
    if constexpr (COH) {
        // inside the persistent ensemble kernel (phase A's occupancy): all
        // five variables' loads first for memory-level parallelism, then the
        // stores (6.89 -> 6.05 ms per step on the 64-box ensemble)
        using P = typename PB::P_t;
        using C = typename PB::C_t;
        BVar<P, C> d[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) d[v] = b_load<COH>(B, x, v);
#pragma unroll
        for (int v = 0; v < NV; ++v) b_store(B, x, v, d[v]);
    } else {
        // a launch of its own: one variable at a time keeps the registers,
        // and with them the occupancy, low
#pragma unroll
        for (int v = 0; v < NV; ++v) stage_b_var<COH>(B, x, v);
    }
}

template <class S, class P, class C, int EPB>
__global__ void __launch_bounds__(LPE * EPB) stage_b_kernel(const StageBParams<S, P, C> B) {
    stage_b_tile<EPB, false>(B, blockIdx.x);
}

// Phase B with one thread per (element, variable, x-line): 80 threads per
// element; a warp holds two elements' lines of one variable. Blocks walk
// the elements in reverse order: phase A's last RHS and face records (the
// highest elements) are still in L2 when phase B starts, and phase B's last
// stores (the lowest elements) are what the next phase A reads first
// (48^3 f32: phase B 120.9 -> 117.5 us, phase A 263.0 -> 262.4 us).
template <class S, class P, class C, int EPB>
__global__ void __launch_bounds__(LPE * NV * EPB) stage_b_split_kernel(const StageBParams<S, P, C> B) {
    dependent_start();   // as phase A
    const int g = threadIdx.x / LPE;
    const int v = g / EPB;
    const long long e = B.e0 + (long long)(gridDim.x - 1 - blockIdx.x) * EPB + (g - v * EPB);
    if (e >= B.e1) return;
    stage_b_var<false>(B, b_ctx(B, e, threadIdx.x & (LPE - 1)), v);
}

}  // namespace od
