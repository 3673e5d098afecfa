// Templated host launcher for one precision combination; included by the
// od_inst_*.cu translation units only.
#pragma once

#include <cstdint>
#include <type_traits>

#include "od_launch.h"
#include "od_stage.cuh"

namespace od {

template <class T>
Tab<T> cast_tab(const TablesD& t) {
    Tab<T> r;
    for (int i = 0; i < 16; ++i) r.D[i] = (T)t.D[i];
    for (int i = 0; i < 4; ++i) {
        r.eL[i] = (T)t.eL[i];
        r.eR[i] = (T)t.eR[i];
        r.gL[i] = (T)t.gL[i];
        r.gR[i] = (T)t.gR[i];
    }
    return r;
}

// The kernels that also write the closure's features exist for the all-f32
// pipeline with constant viscosity at 4 elements per block (the closure's
// configuration); feat says whether this launch writes them.
template <class S, class P, class C, class M>
constexpr bool has_feat_variant() {
    return sizeof(S) == 4 && sizeof(P) == 4 && sizeof(C) == 4 && !M::kSutherland && !M::kWideState;
}

// Launches of small meshes are programmatic dependents of the kernel before
// them: their blocks are resident and past their launch latency when it ends
// (every stage kernel waits for it with griddepcontrol.wait before its first
// load). On B200, steps of n^3 elements: f32 1.33x at 4, 1.26x at 8, 1.22x at
// 16, 1.09x at 24, 1.04x at 32, 1.5% at 40, 0.7% at 48; f64 1.24x at 4, 1.11x
// at 8 to 16, 1.2% at 32, nothing at 48; but u64/c32 2% slower at 48 and 64.
constexpr long long kDependentElems = 1 << 16;
// Phase A with f32 fluxes is an ordinary launch on meshes that give an SM some
// of its places only: its blocks then spread evenly, where a dependent's fill
// the gaps that phase B's leave and pile up on some SMs. The band is in elements
// (blocks of 2 and of 4 elements behave alike). 10 steps, dependent / ordinary,
// geometric means over random meshes of the range (elements: ratio):
//   f32     384-511: 0.95  512-639: 0.97 | 640-767: 1.04  768-1023: 1.06
//           1024-1791: 1.11  1792-2047: 0.91  2048-3071: 1.07
//           3072-3399: 1.03 | 3584-4095: 0.89
//   u64/c32 256-383: 0.90 | 384-511: 1.06  512-767: 1.10  768-1791: 1.15
//           1792-2047: 0.93  2048-3071: 1.11  3072-3399: 1.06 | 3584-4095: 0.92
//   mixed   256-383: 0.96 | 384-511: 1.02  512-767: 1.14  768-1535: 1.12
//           1536-1791: 0.90  1792-2047: 1.13  2048-2559: 1.04 | 2560-3583: 0.92
// Single meshes scatter by 0.8 to 1.25 inside it. f64 fluxes gain as dependents
// nearly everywhere (0.89 to 0.97; 640-1023: 1.04).
template <class P, class C, class M>
bool dependent_a(long long nelem) {
    if (nelem > kDependentElems) return false;
    if (sizeof(C) == 8) return true;
    const long long lo = M::kWideState ? 384 : 640, hi = sizeof(P) == 8 ? 2560 : 3400;
    return nelem < lo || nelem >= hi;
}

// Phase A that writes the closure's features: from 4096 elements only. Its own
// dependent, the network, follows it into residence, and below that the
// network's blocks poll beside phase B and phase A for longer than the launch
// latency saves (20 steps with the closure, ordinary against dependent: 512
// elements 2.34 against 2.51 ms, 1728 2.45 / 2.65, 2744 2.61 / 2.73; 4096 2.88 /
// 2.82, 13824 5.04 / 4.94).
constexpr long long kDependentFeatElems = 1 << 12;

template <class S, class P, class C, class M, int FLUX, int EPB>
cudaError_t launch_a(const StageAParams<S, P, C>& A, long long nelem, cudaStream_t s, bool feat = false) {
    const unsigned grid = (unsigned)((nelem + EPB - 1) / EPB);
    if (grid == 0) return cudaSuccess;
    const size_t smem = sizeof(SlotFor<M, P, C>) * EPB;
    if constexpr (has_feat_variant<S, P, C, M>() && EPB == 4) {
        if (feat) {
            return launch_dependent(nelem >= kDependentFeatElems && nelem <= kDependentElems,
                                    stage_a_kernel<S, P, C, M, FLUX, EPB, true>, grid, LPE * EPB, smem, s, A);
        }
    }
    if (feat) return cudaErrorInvalidValue;   // no variant writes the features for this launch
    return launch_dependent(dependent_a<P, C, M>(nelem), stage_a_kernel<S, P, C, M, FLUX, EPB>, grid, LPE * EPB, smem, s,
                            A);
}

template <class S, class P, class C, class M, int FLUX>
cudaError_t launch_a_epb(const StageAParams<S, P, C>& A, long long nelem, int epb, cudaStream_t s, bool feat) {
    if (epb == 2 && !feat) return launch_a<S, P, C, M, FLUX, 2>(A, nelem, s);
    return launch_a<S, P, C, M, FLUX, 4>(A, nelem, s, feat);
}

// f32 fluxes under an f64 state: the policy that keeps their operation order
// (WIDE: such a state held in f32, launch_stage_u64c32_narrow)
template <class S, class C, class M, bool WIDE>
using MathFor = std::conditional_t<WIDE || (sizeof(S) == 8 && sizeof(C) == 4), WideState<M>, M>;

template <class S, class P, class C, class M>
cudaError_t launch_a_flux(const StageAParams<S, P, C>& A, int flux, long long nelem, int epb, cudaStream_t s,
                          bool feat) {
    // a caller's state (od_rhs_noalloc) may be less than 32-byte aligned: the
    // kernels of 2 elements use 16-byte loads (40^3 f64 step 1.59 ms with 128-bit
    // loads, 1.55 with 256-bit ones; u64/c32 1.9% faster, mixed 1.5%)
    const bool narrow = sizeof(S) == 8 && (reinterpret_cast<uintptr_t>(A.u_in) & 31) != 0;
    if (narrow) epb = 2;
    if (A.suth >= (C)0) {
        // Sutherland variant: 4 elements per block (2 only for that case), no feature writing
        if (feat) return cudaErrorInvalidValue;
        using MS = WithSutherland<M>;
        if constexpr (sizeof(S) == 8) {
            if (narrow) {
                switch (flux) {
                    case kSlau2: return launch_a<S, P, C, MS, kSlau2, 2>(A, nelem, s);
                    case kAusmPlus: return launch_a<S, P, C, MS, kAusmPlus, 2>(A, nelem, s);
                    default: return launch_a<S, P, C, MS, kRusanov, 2>(A, nelem, s);
                }
            }
        }
        switch (flux) {
            case kSlau2: return launch_a<S, P, C, MS, kSlau2, 4>(A, nelem, s);
            case kAusmPlus: return launch_a<S, P, C, MS, kAusmPlus, 4>(A, nelem, s);
            default: return launch_a<S, P, C, MS, kRusanov, 4>(A, nelem, s);
        }
    }
    switch (flux) {
        case kSlau2: return launch_a_epb<S, P, C, M, kSlau2>(A, nelem, epb, s, feat);
        case kAusmPlus: return launch_a_epb<S, P, C, M, kAusmPlus>(A, nelem, epb, s, feat);
        default: return launch_a_epb<S, P, C, M, kRusanov>(A, nelem, epb, s, feat);
    }
}

template <class S, class P, class C, int EPB>
cudaError_t launch_b(const StageBParams<S, P, C>& B, long long nelem, cudaStream_t s) {
    const unsigned grid = (unsigned)((nelem + EPB - 1) / EPB);
    if (grid == 0) return cudaSuccess;
    stage_b_kernel<S, P, C, EPB><<<grid, LPE * EPB, 0, s>>>(B);
    return cudaGetLastError();
}

template <class S, class P, class C, int EPB>
cudaError_t launch_b_split(const StageBParams<S, P, C>& B, long long nelem, cudaStream_t s) {
    const unsigned grid = (unsigned)((nelem + EPB - 1) / EPB);
    if (grid == 0) return cudaSuccess;
    return launch_dependent(nelem <= kDependentElems, stage_b_split_kernel<S, P, C, EPB>, grid, LPE * NV * EPB, 0, s, B);
}

// fast math changes only f32 arithmetic: f64-compute combinations use one variant
template <class C>
constexpr bool has_fast_variant() { return sizeof(C) == 4; }

template <class S, class P, class C, bool WIDE = false>
cudaError_t launch_stage_t(const StageLaunch& L, cudaStream_t s) {
    StageAParams<S, P, C> A{};
    A.u_in = (const S*)L.u_in;
    A.u0 = (const S*)L.u0;
    A.u_out = (S*)(L.rhs ? L.rhs : L.u_out);
    A.fv = (C*)L.fv;
    A.fi = (C*)L.fv + L.nelem * kFvWords;
    A.m.nx = L.nx;
    A.m.ny = L.ny;
    A.m.nz = L.nz;
    A.m.y_wall = L.y_wall;
    A.m.nelem = L.nelem;
    mesh_set_div(A.m);
    A.m.npts = L.nelem * NE;
    A.kappa = heat_coeff_host<C>((C)L.mu);
    A.tp = cast_tab<P>(L.tab);
    A.tc = cast_tab<C>(L.tab);
    for (int d = 0; d < 3; ++d) A.jac[d] = (C)L.jac[d];
    A.sc = scale_tab<C>(A.tc, A.jac);
    A.ra = (P)L.ra;
    A.rb = (P)L.rb;
    A.rc = (P)L.rc;
    A.mu = (C)L.mu;
    A.forcing = (C)L.forcing;
    A.suth = (C)L.suth;
    A.flux = L.flux;
    A.flags = L.flags | (L.rhs ? kDeferRK : 0);
    A.e0 = L.e0;
    A.e1 = L.e1;
    const bool feat = L.feat != nullptr;
    if (feat) A.feat = *L.feat;
    const long long count = L.e1 - L.e0;
    cudaError_t err = cudaSuccess;
    if (L.phases & 1) {
        if (L.ev[0]) cudaEventRecord(L.ev[0], s);
        if constexpr (has_fast_variant<C>()) {
            if (L.fast_math)
                err = launch_a_flux<S, P, C, MathFor<S, C, MathFast, WIDE>>(A, L.flux, count, L.epb_a, s, feat);
            else
                err = launch_a_flux<S, P, C, MathFor<S, C, MathIeee, WIDE>>(A, L.flux, count, L.epb_a, s, feat);
        } else {
            err = launch_a_flux<S, P, C, MathFor<S, C, MathIeee, WIDE>>(A, L.flux, count, L.epb_a, s, feat);
        }
        if (err != cudaSuccess) return err;
        if (L.ev[1]) cudaEventRecord(L.ev[1], s);
    }
    if (L.phases & 2) {
        StageBParams<S, P, C> B;
        B.u_out = (S*)L.u_out;
        B.rhs = (const S*)L.rhs;
        B.u_in = (const S*)L.u_in;
        B.u0 = (const S*)L.u0;
        B.fv = (const C*)L.fv;
        B.fi = A.fi;
        B.m = A.m;
        B.tc = A.tc;
        for (int d = 0; d < 3; ++d) B.jac[d] = A.jac[d];
        B.ra = A.ra;
        B.rb = A.rb;
        B.rc = A.rc;
        B.flags = A.flags;
        if (sizeof(S) == 8 && (reinterpret_cast<uintptr_t>(L.u_out) & 31) == 0) B.flags |= kWideOut;
        B.e0 = L.e0;
        B.e1 = L.e1;
        if (L.epb_b == 8)
            err = launch_b<S, P, C, 8>(B, count, s);
        else if (L.epb_b == 16)
            err = launch_b<S, P, C, 16>(B, count, s);
        else if (L.epb_b == 2)
            err = launch_b_split<S, P, C, 2>(B, count, s);
        else
            err = launch_b_split<S, P, C, 4>(B, count, s);
        if (err != cudaSuccess) return err;
        if (L.ev[2]) cudaEventRecord(L.ev[2], s);
    }
    return cudaSuccess;
}

template <class S, class P, class C, class M, int FLUX>
cudaError_t prepare_flux() {
    cudaError_t e = cudaFuncSetAttribute(stage_a_kernel<S, P, C, M, FLUX, 2>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(sizeof(SlotFor<M, P, C>) * 2));
    if (e != cudaSuccess) return e;
    if constexpr (sizeof(S) == 8) {
        e = cudaFuncSetAttribute(stage_a_kernel<S, P, C, WithSutherland<M>, FLUX, 2>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(SlotFor<M, P, C>) * 2));
        if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(stage_a_kernel<S, P, C, WithSutherland<M>, FLUX, 4>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(SlotFor<M, P, C>) * 4));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(stage_a_kernel<S, P, C, M, FLUX, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(SlotFor<M, P, C>) * 4));
}

template <class S, class P, class C, class M>
cudaError_t prepare_m() {
    cudaError_t e = prepare_flux<S, P, C, M, kSlau2>();
    if (e != cudaSuccess) return e;
    e = prepare_flux<S, P, C, M, kAusmPlus>();
    if (e != cudaSuccess) return e;
    return prepare_flux<S, P, C, M, kRusanov>();
}

template <class S, class P, class C, bool WIDE = false>
cudaError_t prepare_t() {
    cudaError_t e = prepare_m<S, P, C, MathFor<S, C, MathIeee, WIDE>>();
    if constexpr (has_fast_variant<C>()) {
        if (e == cudaSuccess) e = prepare_m<S, P, C, MathFor<S, C, MathFast, WIDE>>();
    }
    return e;
}

}  // namespace od

#define OD_INSTANTIATE(NAME, S, P, C)                                                          \
    namespace od {                                                                             \
    cudaError_t launch_stage_##NAME(const StageLaunch& L, cudaStream_t s) {                   \
        return launch_stage_t<S, P, C>(L, s);                                                  \
    }                                                                                          \
    cudaError_t prepare_kernels_##NAME() { return prepare_t<S, P, C>(); }                      \
    }
