// Learned closure: a per-element MLP (896 -> 256 -> 256 -> 256 -> 320,
// GELU) that corrects the RHS of an under-resolved coarse run.
//
// Kernels here:
//   project   L2 projection of a fine FR P=3 state (or RHS) onto the coarse
//             P=3 basis of elements `factor` times larger per axis (exact for
//             the piecewise cubic fine field: Gauss-Legendre quadrature of the
//             fine elements, the coarse mass matrix is diagonal at the GL
//             points)
//   features  64 points x (5 conserved + 9 velocity gradients) per element,
//             standardised with per-channel constants and clipped to +-8,
//             bf16 rows
//   apply     rhs += out_scale[v] * network output (between the two phases
//             of an RK stage)
//   training  loss gradient, bias gradients, gathers and Adam
// The network's matrix products run on the tcgen05 GEMM of od_mlp.cuh.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/opendynamo.h"
#include "od_launch.h"
#include "od_mlp.cuh"

namespace od {
TablesD host_fr_tables();
namespace mlp {
cudaError_t launch_gemm(const GemmArgs& g, int epi, cudaStream_t s, size_t ws_floats);
cudaError_t launch_gemm_group(GemmArgs* g, int n, float* ws, size_t ws_floats, cudaStream_t s);
}
}  // namespace od

namespace {

using bf16 = __nv_bfloat16;
constexpr int kIn = 896, kHid = 256, kOut = 320, kOutPad = 384, kChan = 14;
constexpr float kClip = 8.0f;  // standardised inputs are clipped to +-kClip (states outside the training range)

// ---------------------------------------------------------------- projection
struct ProjParams {
    int nxc, nyc, nzc;
    float P[4][32];  // P[i][a]: coarse node i from fine sample a (a < 4 f)
};

// x-contracted samples of one coarse element and variable, [b][c] float4 over
// the coarse i; rows of 4 f + 2 so that the 8 lanes of a 128-bit store phase
// (4 values of b, 2 of c) hit distinct banks.
template <int f>
struct ProjSlot {
    static constexpr int F = 4 * f, row = F + 2;
    // coarse elements per block: 16 f^2 threads each (one per fine x-line of
    // the element's cross-section), so that small factors fill a block too
    static constexpr int epb = f >= 3 ? 1 : f == 2 ? 4 : 16;
    float4 t1[5][F * row];
    float4 t2[5][F * 4];   // y-contracted: [c][j] over i
};

// VEC: the planes are 16-byte aligned (any caller's pointer is accepted)
template <bool VEC, class TS>
__device__ __forceinline__ float4 proj_load4(const TS* p) {
    if constexpr (!VEC) {
        return make_float4((float)p[0], (float)p[1], (float)p[2], (float)p[3]);
    } else if constexpr (sizeof(TS) == 4) {
        return __ldcs(reinterpret_cast<const float4*>(p));
    } else {
        const double2 a = __ldcs(reinterpret_cast<const double2*>(p));
        const double2 b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
        return make_float4((float)a.x, (float)a.y, (float)b.x, (float)b.y);
    }
}

template <bool VEC, class TD>
__device__ __forceinline__ void proj_store4(TD* p, const float4& v) {
    if constexpr (!VEC) {
        p[0] = (TD)v.x;
        p[1] = (TD)v.y;
        p[2] = (TD)v.z;
        p[3] = (TD)v.w;
    } else if constexpr (sizeof(TD) == 4) {
        *reinterpret_cast<float4*>(p) = v;
    } else {
        reinterpret_cast<double2*>(p)[0] = make_double2((double)v.x, (double)v.y);
        reinterpret_cast<double2*>(p)[1] = make_double2((double)v.z, (double)v.w);
    }
}

__device__ __forceinline__ void axpy4(float c, const float4& x, float4& y) {
    y.x += c * x.x;
    y.y += c * x.y;
    y.z += c * x.z;
    y.w += c * x.w;
}

// Sum-factorised projection, bound by reading the fine state once. A thread
// owns one (b, c) line of fine samples of its coarse element: 16 consecutive
// lanes read the 16 x-lines of a fine element (256 contiguous bytes as
// 128-bit loads) and contract x in registers over the f fine elements of the
// line, for all five variables (5 f loads in flight). y and z are contracted
// from shared memory, four coarse i per 128-bit access, one task per
// (variable, c, j) and (variable, k, j). Every sum runs over its fine samples
// in ascending order. 96^3 f32 onto 24^3 (1.13 GB read, 170 us at the copy
// rate) with the features of the result: 1421 us a call when a block gathered
// one sample a thread per variable, 224 us so.
template <class TS, class TD, int f, bool VEC>
__global__ void __launch_bounds__(16 * f * f * ProjSlot<f>::epb)
    project_kernel(const TS* __restrict__ src, TD* __restrict__ dst, const ProjParams pp) {
    constexpr int F = 4 * f, T = 16 * f * f, G = ProjSlot<f>::epb;
    extern __shared__ __align__(16) unsigned char proj_smem[];
    const int g = threadIdx.x / T, t = threadIdx.x - g * T;
    ProjSlot<f>& sm = reinterpret_cast<ProjSlot<f>*>(proj_smem)[g];
    const long long nec = (long long)pp.nxc * pp.nyc * pp.nzc;
    const long long ec = (long long)blockIdx.x * G + g;
    const bool live = ec < nec;
    const long long npc = nec * 64, npf = npc * (f * f * f);
    {
        const unsigned e = (unsigned)(live ? ec : 0);
        const unsigned r = e / (unsigned)pp.nxc, cx = e - r * (unsigned)pp.nxc;
        const unsigned cz = r / (unsigned)pp.nyc, cy = r - cz * (unsigned)pp.nyc;
        const int l = t & 15, qy = (t >> 4) % f, qz = (t >> 4) / f;
        const long long nxf = (long long)pp.nxc * f, nyf = (long long)pp.nyc * f;
        const long long fe = (long long)cx * f + nxf * ((long long)cy * f + qy + nyf * ((long long)cz * f + qz));
        const TS* p = src + fe * 64 + 4 * l;
        const int at = (4 * qy + (l & 3)) * ProjSlot<f>::row + 4 * qz + (l >> 2);
#pragma unroll(f <= 4 ? 5 : 1)
        for (int v = 0; v < 5; ++v) {
            float4 w[f];
#pragma unroll
            for (int q = 0; q < f; ++q) w[q] = proj_load4<VEC>(p + v * npf + q * 64);
            float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int q = 0; q < f; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    a[i] += pp.P[i][4 * q + 0] * w[q].x;
                    a[i] += pp.P[i][4 * q + 1] * w[q].y;
                    a[i] += pp.P[i][4 * q + 2] * w[q].z;
                    a[i] += pp.P[i][4 * q + 3] * w[q].w;
                }
            sm.t1[v][at] = make_float4(a[0], a[1], a[2], a[3]);
        }
    }
    __syncthreads();
    for (int s = t; s < 5 * 4 * F; s += T) {
        const int j = s & 3, c = (s >> 2) % F, v = (s >> 2) / F;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int b = 0; b < F; ++b) axpy4(pp.P[j][b], sm.t1[v][b * ProjSlot<f>::row + c], acc);
        sm.t2[v][c * 4 + j] = acc;
    }
    __syncthreads();
    if (!live) return;
    for (int s = t; s < 5 * 16; s += T) {
        const int j = s & 3, k = (s >> 2) & 3, v = s >> 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int c = 0; c < F; ++c) axpy4(pp.P[k][c], sm.t2[v][c * 4 + j], acc);
        proj_store4<VEC>(dst + v * npc + ec * 64 + 4 * (s & 15), acc);
    }
}

template <class TS, class TD, int f>
cudaError_t launch_project(const void* src, void* dst, const ProjParams& pp, cudaStream_t s) {
    constexpr int G = ProjSlot<f>::epb;
    const size_t sm = sizeof(ProjSlot<f>) * G;
    const long long ne = (long long)pp.nxc * pp.nyc * pp.nzc;
    // 128-bit accesses on 16-byte aligned buffers (what cudaMalloc and torch give), scalar ones on others
    const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
    auto* fn = vec ? project_kernel<TS, TD, f, true> : project_kernel<TS, TD, f, false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    fn<<<(unsigned)((ne + G - 1) / G), 16 * f * f * G, sm, s>>>((const TS*)src, (TD*)dst, pp);
    return cudaGetLastError();
}

template <class TS, class TD>
cudaError_t launch_project_f(int f, const void* src, void* dst, const ProjParams& pp, cudaStream_t s) {
    switch (f) {
        case 1: return launch_project<TS, TD, 1>(src, dst, pp, s);
        case 2: return launch_project<TS, TD, 2>(src, dst, pp, s);
        case 3: return launch_project<TS, TD, 3>(src, dst, pp, s);
        case 4: return launch_project<TS, TD, 4>(src, dst, pp, s);
        case 5: return launch_project<TS, TD, 5>(src, dst, pp, s);
        case 6: return launch_project<TS, TD, 6>(src, dst, pp, s);
        case 7: return launch_project<TS, TD, 7>(src, dst, pp, s);
        default: return launch_project<TS, TD, 8>(src, dst, pp, s);
    }
}

ProjParams proj_params(int nxc, int nyc, int nzc, int f) {
    ProjParams pp{};
    pp.nxc = nxc;
    pp.nyc = nyc;
    pp.nzc = nzc;
    const od::TablesD t = od::host_fr_tables();
    double w[4];
    for (int a = 0; a < 4; ++a) {
        const double x = t.pts[a];
        const double p4 = (35 * x * x * x * x - 30 * x * x + 3) / 8.0, p3 = (5 * x * x * x - 3 * x) / 2.0;
        const double dp4 = 4.0 * (x * p4 - p3) / (x * x - 1.0);
        w[a] = 2.0 / ((1.0 - x * x) * dp4 * dp4);
    }
    auto lag = [&](int i, double xi) {
        double r = 1.0;
        for (int m = 0; m < 4; ++m)
            if (m != i) r *= (xi - t.pts[m]) / (t.pts[i] - t.pts[m]);
        return r;
    };
    for (int i = 0; i < 4; ++i)
        for (int a = 0; a < 4 * f; ++a) {
            const int q = a / 4, jf = a % 4;
            const double xc = -1.0 + (2.0 * q + 1.0 + t.pts[jf]) / f;
            pp.P[i][a] = (float)(w[jf] * lag(i, xc) / (f * w[i]));
        }
    return pp;
}

// ---------------------------------------------------------------- features
struct FeatParams {
    int nx, ny, nz;
    float jac[3];
    float D[16];
    float mean[kChan], inv_scale[kChan];
};

// The standardised features of a point from its conserved variables c and
// their derivatives d[var][direction]: (value - mean) / scale, clipped, as
// bf16. Every rounding is pinned (no contraction is left to the compiler):
// phase A writes the same features (stage_a_features), value for value.
template <class Put>
__device__ __forceinline__ void feature_channels(const FeatParams& fp, const float* c, const float (&d)[4][3], Put put) {
    auto emit = [&](int i, float x) {   // x: the channel minus its mean
        put(i, __float2bfloat16_rn(fminf(fmaxf(__fmul_rn(x, fp.inv_scale[i]), -kClip), kClip)));
    };
    const float ir = 1.0f / c[0];
#pragma unroll
    for (int v = 0; v < 5; ++v) emit(v, __fadd_rn(c[v], -fp.mean[v]));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float nu = __fmul_rn(c[1 + a], -ir);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const int i = 5 + 3 * a + b;
            emit(i, __fmaf_rn(__fmaf_rn(nu, d[0][b], d[1 + a][b]), ir, -fp.mean[i]));
        }
    }
}

// X: row-major [element][channel * 64 + point]; a thread per point.
template <class T>
__global__ void __launch_bounds__(64) features_kernel(const T* __restrict__ u, FeatParams fp, bf16* __restrict__ X) {
    __shared__ float q[4][64];
    const long long e = blockIdx.x;
    const long long npts = (long long)fp.nx * fp.ny * fp.nz * 64;
    const int p = threadIdx.x, i = p & 3, j = (p >> 2) & 3, k = p >> 4;
    float c[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) c[v] = (float)u[v * npts + e * 64 + p];
#pragma unroll
    for (int v = 0; v < 4; ++v) q[v][p] = c[v];
    __syncthreads();
    float d[4][3];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            sx = __fmaf_rn(fp.D[i * 4 + m], q[v][m + 4 * j + 16 * k], sx);
            sy = __fmaf_rn(fp.D[j * 4 + m], q[v][i + 4 * m + 16 * k], sy);
            sz = __fmaf_rn(fp.D[k * 4 + m], q[v][i + 4 * j + 16 * m], sz);
        }
        d[v][0] = __fmul_rn(sx, fp.jac[0]);
        d[v][1] = __fmul_rn(sy, fp.jac[1]);
        d[v][2] = __fmul_rn(sz, fp.jac[2]);
    }
    bf16* row = X + e * kIn + p;
    feature_channels(fp, c, d, [&](int ch, bf16 x) { row[ch * 64] = x; });
}

// The same features for the fused inference kernel, written in its layout:
// per 128-element tile, per channel (one 64-wide K block) the 128 x 64 block
// in the shared-memory core-matrix layout, so that one bulk copy fills a
// feature stage. f32 state. 16 threads per element, 4 elements per block:
// thread l owns the x-line (j, k) = (l & 3, l >> 2) of its element, takes the
// x derivatives of its four points in registers and the y / z derivatives
// from the four x-lines of its k-plane / j-column in shared memory (128-bit
// loads), in the same operation order as features_kernel. The channels are
// staged in shared memory and stored as 16-byte chunks.
constexpr int kFeatEpb = 4;

__global__ void __launch_bounds__(16 * kFeatEpb) features_tiled_kernel(const float* __restrict__ u, FeatParams fp,
                                                                        bf16* __restrict__ X, long long nelem) {
    __shared__ __align__(16) float q[kFeatEpb][4][64];
    __shared__ __align__(16) bf16 st[kFeatEpb][kChan][64];
    // the fused inference kernel that follows may start its prologue now
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int es = threadIdx.x >> 4, l = threadIdx.x & 15, j = l & 3, k = l >> 2;
    const long long e = (long long)blockIdx.x * kFeatEpb + es;
    const bool live = e < nelem;
    const long long ec = live ? e : 0;
    const long long npts = (long long)fp.nx * fp.ny * fp.nz * 64;
    float c[5][4];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
        const float4 w = __ldg(reinterpret_cast<const float4*>(u + v * npts + ec * 64 + 4 * l));
        c[v][0] = w.x;
        c[v][1] = w.y;
        c[v][2] = w.z;
        c[v][3] = w.w;
        if (v < 4) *reinterpret_cast<float4*>(&q[es][v][4 * l]) = w;
    }
    __syncthreads();
    float d[4][4][3];   // [point of the line][var][direction]
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        float ly[4][4], lz[4][4];   // the x-lines (m, k) and (j, m), m = 0..3
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const float4 a = *reinterpret_cast<const float4*>(&q[es][v][4 * (m + 4 * k)]);
            const float4 b = *reinterpret_cast<const float4*>(&q[es][v][4 * (j + 4 * m)]);
            ly[m][0] = a.x; ly[m][1] = a.y; ly[m][2] = a.z; ly[m][3] = a.w;
            lz[m][0] = b.x; lz[m][1] = b.y; lz[m][2] = b.z; lz[m][3] = b.w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                sx = __fmaf_rn(fp.D[i * 4 + m], c[v][m], sx);
                sy = __fmaf_rn(fp.D[j * 4 + m], ly[m][i], sy);
                sz = __fmaf_rn(fp.D[k * 4 + m], lz[m][i], sz);
            }
            d[i][v][0] = __fmul_rn(sx, fp.jac[0]);
            d[i][v][1] = __fmul_rn(sy, fp.jac[1]);
            d[i][v][2] = __fmul_rn(sz, fp.jac[2]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int p = i + 4 * l;
        const float ci[5] = {c[0][i], c[1][i], c[2][i], c[3][i], c[4][i]};
        feature_channels(fp, ci, d[i], [&](int ch, bf16 x) { st[es][ch][p] = x; });
    }
    __syncthreads();
    if (!live) return;
    bf16* tile = X + (e >> 7) * (128 * kIn);
    for (int q8 = l; q8 < kChan * 8; q8 += 16) {
        const int ch_i = q8 >> 3, kc = q8 & 7;
        *reinterpret_cast<uint4*>(tile + ch_i * (128 * 64) + od::mlp::tile_off((int)(e & 127), kc) / 2) =
            *reinterpret_cast<const uint4*>(&st[es][ch_i][8 * kc]);
    }
}

FeatParams feat_params(int nx, int ny, int nz, double lx, double ly, double lz, const float* mean,
                       const float* scale) {
    FeatParams fp{};
    fp.nx = nx;
    fp.ny = ny;
    fp.nz = nz;
    fp.jac[0] = (float)(2.0 * nx / lx);
    fp.jac[1] = (float)(2.0 * ny / ly);
    fp.jac[2] = (float)(2.0 * nz / lz);
    const od::TablesD t = od::host_fr_tables();
    for (int a = 0; a < 16; ++a) fp.D[a] = (float)t.D[a];
    for (int c = 0; c < kChan; ++c) {
        fp.mean[c] = mean ? mean[c] : 0.f;
        fp.inv_scale[c] = scale ? 1.0f / scale[c] : 1.f;
    }
    return fp;
}

// rhs[v][e*64+p] += scale[v] * Y[e][v*64+p]
template <class T>
__global__ void apply_kernel(T* __restrict__ rhs, const float* __restrict__ Y, long long nelem, float s0, float s1,
                             float s2, float s3, float s4) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long npts = nelem * 64;
    if (idx >= npts * 5) return;
    const int v = (int)(idx / npts);
    const long long r = idx - v * npts;
    const long long e = r >> 6;
    const int p = (int)(r & 63);
    const float sc = v == 0 ? s0 : v == 1 ? s1 : v == 2 ? s2 : v == 3 ? s3 : s4;
    rhs[idx] = (T)((float)rhs[idx] + sc * Y[e * kOutPad + v * 64 + p]);
}

// ---------------------------------------------------------------- training kernels
// The operands of the weight-gradient products are wanted twice, row-major
// and transposed. Every kernel here that writes both goes through a tile of
// 64 columns in shared memory and writes 16-byte chunks in both orientations
// (a 2-byte store per value into the transposed copy touched a sector each:
// at a batch of 8192 the gather took 81 us and the loss gradient 129 us, both
// about 8 us of traffic; now 8 and 7).

// shared-memory position of (row r, column c) of a tile of 64 columns: the
// row's 16-byte chunks are XORed with its row group, so that whole-row writes
// and reads of eight row groups of one column both hit distinct banks
__device__ __forceinline__ int tr_at(int r, int c) { return r * 64 + (c ^ (((r >> 3) & 7) << 3)); }

__device__ __forceinline__ uint4 pack8(const bf16* v) {
    uint4 o;
    o.x = (uint32_t)__bfloat16_as_ushort(v[0]) | ((uint32_t)__bfloat16_as_ushort(v[1]) << 16);
    o.y = (uint32_t)__bfloat16_as_ushort(v[2]) | ((uint32_t)__bfloat16_as_ushort(v[3]) << 16);
    o.z = (uint32_t)__bfloat16_as_ushort(v[4]) | ((uint32_t)__bfloat16_as_ushort(v[5]) << 16);
    o.w = (uint32_t)__bfloat16_as_ushort(v[6]) | ((uint32_t)__bfloat16_as_ushort(v[7]) << 16);
    return o;
}

// rows 8 rc .. 8 rc + 7 of column c of the tile
__device__ __forceinline__ uint4 tr_column(const bf16* tile, int rc, int c) {
    bf16 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = tile[tr_at(8 * rc + i, c)];
    return pack8(v);
}

// eight values of a caller's pool; VEC: the pool is 16-byte aligned
template <bool VEC>
__device__ __forceinline__ uint4 pool8(const bf16* p) {
    if constexpr (VEC) {
        return __ldg(reinterpret_cast<const uint4*>(p));
    } else {
        bf16 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p[i];
        return pack8(v);
    }
}

// rows of the bf16 feature pool into a batch: X [M x 896] and X^T; rows past
// mv are zero. Block (x, y): 64 rows, 64 columns.
template <bool VEC>
__global__ void __launch_bounds__(256) gather_kernel(const bf16* __restrict__ Xp, const long long* __restrict__ rows,
                                                     int mv, int M, bf16* __restrict__ X, bf16* __restrict__ XT) {
    od::dependent_start();
    __shared__ __align__(16) bf16 tile[64 * 64];
    const int m0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int r = (threadIdx.x + 256 * q) >> 3, c = (threadIdx.x & 7) * 8, m = m0 + r;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (m < mv) v = pool8<VEC>(Xp + rows[m] * kIn + c0 + c);
        *reinterpret_cast<uint4*>(X + (size_t)m * kIn + c0 + c) = v;
        *reinterpret_cast<uint4*>(&tile[tr_at(r, c)]) = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int c = (threadIdx.x + 256 * q) >> 3, rc = threadIdx.x & 7;
        *reinterpret_cast<uint4*>(XT + (size_t)(c0 + c) * M + m0 + 8 * rc) = tr_column(tile, rc, c);
    }
}

// dY = g (Y - T) on the valid block (rows < mv, columns < kOut), 0 elsewhere;
// bf16 [M x 384] and its transpose; loss += sum (Y - T)^2. The targets are
// fp32 rows [M x 384], or (POOL) rows of the bf16 target pool [n x 320].
// Block (x, y): 64 rows, 64 columns.
template <bool POOL, bool VEC>
__global__ void __launch_bounds__(256) loss_grad_kernel(const float* Y, const float* T, const bf16* __restrict__ Tp,
                                                        const long long* __restrict__ rows,
                                                        int M, int mv, float g, bf16* __restrict__ dY,
                                                        bf16* __restrict__ dYT, double* loss) {
    od::dependent_start();
    __shared__ __align__(16) bf16 tile[64 * 64];
    __shared__ double red[8];
    const int m0 = blockIdx.x * 64, n0 = blockIdx.y * 64;
    double sq = 0.0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int r = (threadIdx.x + 256 * q) >> 3, c = (threadIdx.x & 7) * 8, m = m0 + r;
        uint4 o = make_uint4(0, 0, 0, 0);
        if (m < mv && n0 < kOut) {   // kOut is a multiple of 64
            const size_t at = (size_t)m * kOutPad + n0 + c;
            float y[8], t[8];
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float4*>(y + 4 * h) = reinterpret_cast<const float4*>(Y + at)[h];
            if constexpr (POOL) {
                const uint4 w = pool8<VEC>(Tp + rows[m] * kOut + n0 + c);
                const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    t[2 * i] = __uint_as_float(u[i] << 16);
                    t[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
                }
            } else {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    *reinterpret_cast<float4*>(t + 4 * h) = reinterpret_cast<const float4*>(T + at)[h];
            }
            bf16 b[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float d = y[i] - t[i];
                b[i] = __float2bfloat16_rn(g * d);
                sq += (double)(d * d);
            }
            o = pack8(b);
        }
        *reinterpret_cast<uint4*>(dY + (size_t)m * kOutPad + n0 + c) = o;
        *reinterpret_cast<uint4*>(&tile[tr_at(r, c)]) = o;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int c = (threadIdx.x + 256 * q) >> 3, rc = threadIdx.x & 7;
        *reinterpret_cast<uint4*>(dYT + (size_t)(n0 + c) * M + m0 + 8 * rc) = tr_column(tile, rc, c);
    }
    if (threadIdx.x == 0 && n0 < kOut) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += red[w];
        atomicAdd(loss, s);
    }
}

// The end of the backward pass in one launch: bias gradients out[n] = sum_m
// AT[n][m] (bf16 -> fp32) from the transposed copies, and the sums of the
// weight gradients' K ranges. Launched one by one they took 69 and 28 us at a
// batch of 8192 (2-byte loads, each waiting for its first ones alone); together
// 19 us.
//
// Row sums, a warp per row: the order is that of 256 partial sums s[t] =
// AT[n][t] + AT[n][t + 256] + ..., each 32 of them summed in a tree (t + 16,
// t + 8, ... + 1), the eight trees in sequence: Adam's first steps divide by
// the gradient's own size, so another order moves the weights. Lane l holds
// the partial sums 8 l .. 8 l + 7 and loads 16 bytes at a time (M % 8 == 0).
// K ranges: one value a thread, in ascending order, 16 loads in flight.
constexpr int kFinishThreads = 128;

struct GradFinish {
    const bf16* AT[4];      // [rows x M]
    float* bias[4];
    const float* ws[4];     // [ks x mn]
    float* w[4];
    long long mn[4];
    int ks[4];
    int first_b[5], first_w[5];   // blocks of each row-sum part, then of each K-range part
    int M;
};

__device__ __forceinline__ float row_sum(const bf16* AT, int M, int n, int lane) {
    const uint4* row = reinterpret_cast<const uint4*>(AT + (size_t)n * M);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int q = lane; q < M / 8; q += 32) {
        const uint4 w = row[q];
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            s[2 * i] += __uint_as_float(u[i] << 16);
            s[2 * i + 1] += __uint_as_float(u[i] & 0xffff0000u);
        }
    }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += __shfl_down_sync(0xffffffffu, s[i], o, 4);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) s[i] += s[i + o];
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += __shfl_sync(0xffffffffu, s[0], 4 * w);
    return t;
}

__global__ void __launch_bounds__(kFinishThreads) grad_finish_kernel(const GradFinish F) {
    od::dependent_start();
    const int b = (int)blockIdx.x;
    if (b < F.first_b[4]) {
        int l = 0;
        while (b >= F.first_b[l + 1]) ++l;
        const int n = (b - F.first_b[l]) * (kFinishThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
        const float t = row_sum(F.AT[l], F.M, n, lane);
        if (lane == 0) F.bias[l][n] = t;
        return;
    }
    int l = 0;
    while (b >= F.first_w[l + 1]) ++l;
    const long long i = (long long)(b - F.first_w[l]) * kFinishThreads + threadIdx.x, mn = F.mn[l];
    const float* p = F.ws[l] + i;
    const int ks = F.ks[l];
    float v = 0.f;
#pragma unroll 16
    for (int z = 0; z < ks; ++z) v += __ldcs(p + z * mn);
    F.w[l][i] = v;
}

struct AdamStep {
    float lr, b1, b2, eps, c1, c2;
};

// The two moments' multiply-adds are pinned: where the compiler contracts them
// depends on the code around, and an early step, which divides by the
// gradient's own size, carries the last bit of them into the weights.
__device__ __forceinline__ float adam_update(const AdamStep& p, float w, float g, float& m1, float& m2) {
    const float a = __fmaf_rn(1.f - p.b1, g, __fmul_rn(p.b1, m1));
    const float b = __fmaf_rn(__fmul_rn(1.f - p.b2, g), g, __fmul_rn(p.b2, m2));
    m1 = a;
    m2 = b;
    return w - p.lr * (a / p.c1) / (sqrtf(b / p.c2) + p.eps);
}

// the flat parameter layout of all layers and the bf16 copies made from it
struct AdamArgs {
    float *w, *m1, *m2;
    const float* g;
    long long off_w[4], off_b[4];
    int rows[4], cols[4];
    bf16 *wb[4], *wbT[4];
    bf16* wt;
    AdamStep p;
};

constexpr int kAdamRows = 32;   // rows of a weight tile (of 64 columns)

// Adam on the fp32 master weights of every layer in one launch: blocks 0..:
// weight tiles of 32 rows x 64 columns, which also write the bf16 copies W and
// W^T and the fused inference kernel's weight image; the last four blocks: the
// layers' biases. (Eight launches of one value a thread with 2-byte stores
// into W^T, and a ninth for the image, took 36 us; this one 9 us.)
__global__ void __launch_bounds__(256) adam_kernel(const AdamArgs A, int tiles) {
    od::dependent_start();
    __shared__ __align__(16) bf16 tile[kAdamRows * 64];
    int b = blockIdx.x, l = 0;
    if (b >= tiles) {
        l = b - tiles;
        const long long o = A.off_b[l];
        for (int i = threadIdx.x; i < A.rows[l]; i += 256)
            A.w[o + i] = adam_update(A.p, A.w[o + i], A.g[o + i], A.m1[o + i], A.m2[o + i]);
        return;
    }
    for (int n; b >= (n = (A.rows[l] / kAdamRows) * (A.cols[l] / 64)); ++l) b -= n;
    const int cb = A.cols[l] / 64, kb = b % cb, r0 = b / cb * kAdamRows, cols = A.cols[l], rows = A.rows[l];
    const int r = threadIdx.x >> 3, kc = threadIdx.x & 7;
    const long long at = A.off_w[l] + (long long)(r0 + r) * cols + kb * 64 + 8 * kc;
    bf16 h[8];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        float4 w = *reinterpret_cast<const float4*>(A.w + at + 4 * q);
        float4 m1 = *reinterpret_cast<const float4*>(A.m1 + at + 4 * q);
        float4 m2 = *reinterpret_cast<const float4*>(A.m2 + at + 4 * q);
        const float4 g = *reinterpret_cast<const float4*>(A.g + at + 4 * q);
        w.x = adam_update(A.p, w.x, g.x, m1.x, m2.x);
        w.y = adam_update(A.p, w.y, g.y, m1.y, m2.y);
        w.z = adam_update(A.p, w.z, g.z, m1.z, m2.z);
        w.w = adam_update(A.p, w.w, g.w, m1.w, m2.w);
        *reinterpret_cast<float4*>(A.w + at + 4 * q) = w;
        *reinterpret_cast<float4*>(A.m1 + at + 4 * q) = m1;
        *reinterpret_cast<float4*>(A.m2 + at + 4 * q) = m2;
        h[4 * q] = __float2bfloat16_rn(w.x);
        h[4 * q + 1] = __float2bfloat16_rn(w.y);
        h[4 * q + 2] = __float2bfloat16_rn(w.z);
        h[4 * q + 3] = __float2bfloat16_rn(w.w);
    }
    const uint4 o = pack8(h);
    *reinterpret_cast<uint4*>(A.wb[l] + (size_t)(r0 + r) * cols + kb * 64 + 8 * kc) = o;
    const uint32_t img = od::mlp::fused_image_off(l, r0 + r, kb, kc);
    if (img < od::mlp::kFusedWeightBytes) *reinterpret_cast<uint4*>(reinterpret_cast<char*>(A.wt) + img) = o;
    *reinterpret_cast<uint4*>(&tile[tr_at(r, 8 * kc)]) = o;
    __syncthreads();
    const int c = threadIdx.x >> 2, rc = threadIdx.x & 3;
    *reinterpret_cast<uint4*>(A.wbT[l] + (size_t)(kb * 64 + c) * rows + r0 + 8 * rc) = tr_column(tile, rc, c);
}

// bf16 copies of all layers from the fp32 master weights
__global__ void cast_weights_kernel(const float* __restrict__ w, long long n, int rows, int cols,
                                    bf16* __restrict__ wb, bf16* __restrict__ wbT) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bf16 h = __float2bfloat16_rn(w[i]);
    wb[i] = h;
    const int r = (int)(i / cols), c = (int)(i % cols);
    wbT[(long long)c * rows + r] = h;
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ a, bf16* __restrict__ b, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = __float2bfloat16_rn(a[i]);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// ------------------------------------------------------------------ network
struct od_mlp {
    int device = 0;
    int mmax = 0;                    // batch capacity (rows, multiple of 128)
    cudaStream_t stream = nullptr;
    // parameters: fp32 master, Adam moments, gradients (same flat layout)
    float *w = nullptr, *m1 = nullptr, *m2 = nullptr, *g = nullptr;
    long long nparam = 0;
    long long off_w[4], off_b[4];
    int rows[4], cols[4];
    bf16 *wb[4] = {}, *wbT[4] = {};
    // the fused inference kernel's weight image (refreshed with wb). That kernel
    // reads it and the biases in w before it waits for the kernels ahead of it on
    // its stream: whatever writes them is complete before the writing call returns
    bf16* wt = nullptr;
    // activations
    float* Z[3] = {};
    bf16 *A[3] = {}, *AT[3] = {};
    float* Y = nullptr;
    bf16 *dY = nullptr, *dYT = nullptr;
    bf16 *dZ[2] = {}, *dZT[3] = {};   // row-major: a layer and the one above; transposed: kept for the weight gradients
    bf16 *X = nullptr, *XT = nullptr;   // gathered batch (training)
    float* T = nullptr;
    long long* rows_d = nullptr;
    double* loss = nullptr;         // 16 bytes: the loss sum, then err
    int* err = nullptr;             // set by a timed-out wait
    float* ws = nullptr;            // split-K partial sums of the weight gradients
    size_t ws_floats = 0;
    long long step = 0;
    std::string msg;
    // closure attachment (features of the coarse state + output scaling)
    float mean[kChan], scale[kChan], out_scale[5];
    bool fused = true;       // inference as one kernel (mlp_fused_kernel) on an f32 state
    bf16* Xc = nullptr;      // features of the attached solver's elements
    float* Yc = nullptr;
    long long nelem_c = 0, mpad_c = 0;
    FeatParams fp{};
    bool attached_f64 = false;
};

namespace {

int mfail(od_mlp* m, int code, const std::string& s) {
    if (m) m->msg = s;
    return code;
}

cudaError_t gemm(od_mlp* m, const bf16* A, const bf16* B, int M, int N, int K, int epi, const float* bias,
                 float* of32, bf16* obf, bf16* obfT, const float* zin) {
    od::mlp::GemmArgs a{};
    a.A = A;
    a.B = B;
    a.M = M;
    a.N = N;
    a.K = K;
    a.bias = bias;
    a.out_f32 = of32;
    a.out_bf = obf;
    a.out_bfT = obfT;
    a.z_in = zin;
    a.err = m->err;
    a.ws = m->ws;
    return od::mlp::launch_gemm(a, epi, m->stream, m->ws_floats);
}

// hidden layers of M rows of X (bf16 [M x 896]); training keeps the
// pre-activations and the transposed activations
cudaError_t hidden(od_mlp* m, const bf16* X, int M, bool train) {
    cudaError_t e = cudaSuccess;
    const bf16* in = X;
    int kin = kIn;
    for (int l = 0; l < 3 && e == cudaSuccess; ++l) {
        e = gemm(m, in, m->wb[l], M, kHid, kin, od::mlp::kBiasGelu, m->w + m->off_b[l], train ? m->Z[l] : nullptr,
                 m->A[l], train ? m->AT[l] : nullptr, nullptr);
        in = m->A[l];
        kin = kHid;
    }
    return e;
}

// forward of M rows of X into Y [M x 384]
cudaError_t forward(od_mlp* m, const bf16* X, int M, float* Y, bool keep_t) {
    cudaError_t e = hidden(m, X, M, keep_t);
    if (e == cudaSuccess)
        e = gemm(m, m->A[2], m->wb[3], M, kOutPad, kHid, od::mlp::kStoreF32, m->w + m->off_b[3], Y, nullptr, nullptr,
                 nullptr);
    return e;
}

// gradients of 1/(mv*320) sum (Y - T)^2 w.r.t. all parameters into m->g
// (targets: m->T, or the gathered rows of the pool Tp)
cudaError_t backward(od_mlp* m, const bf16* XT, int M, int mv, const bf16* Tp) {
    cudaError_t e = cudaSuccess;
    const float gs = 2.0f / ((float)mv * (float)kOut);
    auto* lg = !Tp ? loss_grad_kernel<false, true>
                   : aligned16(Tp) ? loss_grad_kernel<true, true> : loss_grad_kernel<true, false>;
    e = od::launch_dependent(true, lg, dim3(M / 64, kOutPad / 64), 256, 0, m->stream, m->Y, m->T, Tp, m->rows_d, M, mv,
                             gs, m->dY, m->dYT, m->loss);
    // down the layers: dZ of the hidden layers, each with its transposed copy
    const bf16* dz = m->dY;
    for (int l = 2; l >= 0 && e == cudaSuccess; --l) {
        e = gemm(m, dz, m->wbT[l + 1], M, kHid, l == 2 ? kOutPad : kHid, od::mlp::kGeluGrad, nullptr, nullptr,
                 m->dZ[l & 1], m->dZT[l], m->Z[l]);
        dz = m->dZ[l & 1];
    }
    // every weight gradient in one launch, then the sums over K ranges and rows
    od::mlp::GemmArgs g[4] = {};
    GradFinish F{};
    F.M = M;
    int nb = 0;
    for (int l = 0; l < 4; ++l) {
        g[l].A = l == 3 ? m->dYT : m->dZT[l];
        g[l].B = l == 0 ? XT : m->AT[l - 1];
        g[l].M = m->rows[l];
        g[l].N = m->cols[l];
        g[l].K = M;
        g[l].out_f32 = m->g + m->off_w[l];
        g[l].err = m->err;
        F.AT[l] = g[l].A;
        F.bias[l] = m->g + m->off_b[l];
        F.first_b[l] = nb;
        nb += m->rows[l] / (kFinishThreads / 32);
    }
    F.first_b[4] = nb;
    if (e == cudaSuccess) e = od::mlp::launch_gemm_group(g, 4, m->ws, m->ws_floats, m->stream);
    if (e != cudaSuccess) return e;
    for (int l = 0; l < 4; ++l) {
        F.ws[l] = g[l].ws;
        F.w[l] = g[l].out_f32;
        F.ks[l] = g[l].ksplit;
        F.mn[l] = (long long)g[l].M * g[l].N;
        F.first_w[l] = nb;
        if (g[l].ksplit > 1) nb += (int)(F.mn[l] / kFinishThreads);
    }
    F.first_w[4] = nb;
    return od::launch_dependent(true, grad_finish_kernel, (unsigned)nb, kFinishThreads, 0, m->stream, F);
}

constexpr size_t kStatusBytes = 16;   // loss and err, cleared and read back together

cudaError_t clear_status(od_mlp* m) { return cudaMemsetAsync(m->loss, 0, kStatusBytes, m->stream); }

// waits for the stream; loss (may be null; left alone when that fails): the
// loss sum of the calls since clear_status over n
int read_status(od_mlp* m, double* loss, double n = 1.0) {
    struct {
        double loss;
        int err, pad;
    } h{};
    static_assert(sizeof h == kStatusBytes, "one copy");
    cudaError_t e = cudaMemcpyAsync(&h, m->loss, sizeof h, cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e != cudaSuccess) return mfail(m, OD_ERR_CUDA, cudaGetErrorString(e));
    if (loss) *loss = h.loss / n;
    if (h.err) return mfail(m, OD_ERR_CUDA, "tensor-core GEMM wait timed out");
    return OD_OK;
}

}  // namespace

extern "C" {

int od_mlp_create(int max_rows, int device, od_mlp** out) {
    if (!out || max_rows <= 0) return OD_ERR_ARG;
    *out = nullptr;
    od_mlp* m = new od_mlp();
    m->device = device;
    m->mmax = (max_rows + 127) / 128 * 128;
    const int R[4] = {kHid, kHid, kHid, kOutPad}, C[4] = {kIn, kHid, kHid, kHid};
    long long off = 0;
    for (int l = 0; l < 4; ++l) {
        m->rows[l] = R[l];
        m->cols[l] = C[l];
        m->off_w[l] = off;
        off += (long long)R[l] * C[l];
        m->off_b[l] = off;
        off += R[l];
    }
    m->nparam = off;
    for (int c = 0; c < kChan; ++c) {
        m->mean[c] = 0.f;
        m->scale[c] = 1.f;
    }
    for (int v = 0; v < 5; ++v) m->out_scale[v] = 1.f;
    *out = m;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    const size_t P = sizeof(float) * (size_t)m->nparam;
    const size_t M = (size_t)m->mmax;
    auto mal = [&](void** p, size_t n) {
        if (e == cudaSuccess) e = cudaMalloc(p, n);
        if (e == cudaSuccess) e = cudaMemset(*p, 0, n);
    };
    mal((void**)&m->w, P);
    mal((void**)&m->m1, P);
    mal((void**)&m->m2, P);
    mal((void**)&m->g, P);
    for (int l = 0; l < 4; ++l) {
        mal((void**)&m->wb[l], sizeof(bf16) * R[l] * C[l]);
        mal((void**)&m->wbT[l], sizeof(bf16) * R[l] * C[l]);
    }
    mal((void**)&m->wt, od::mlp::kFusedWeightBytes);
    for (int l = 0; l < 3; ++l) {
        mal((void**)&m->Z[l], sizeof(float) * M * kHid);
        mal((void**)&m->A[l], sizeof(bf16) * M * kHid);
        mal((void**)&m->AT[l], sizeof(bf16) * M * kHid);
    }
    mal((void**)&m->Y, sizeof(float) * M * kOutPad);
    mal((void**)&m->dY, sizeof(bf16) * M * kOutPad);
    mal((void**)&m->dYT, sizeof(bf16) * M * kOutPad);
    for (int l = 0; l < 2; ++l) mal((void**)&m->dZ[l], sizeof(bf16) * M * kHid);
    for (int l = 0; l < 3; ++l) mal((void**)&m->dZT[l], sizeof(bf16) * M * kHid);
    mal((void**)&m->X, sizeof(bf16) * M * kIn);
    mal((void**)&m->XT, sizeof(bf16) * M * kIn);
    mal((void**)&m->T, sizeof(float) * M * kOutPad);
    mal((void**)&m->rows_d, sizeof(long long) * M);
    mal((void**)&m->loss, kStatusBytes);
    m->err = reinterpret_cast<int*>(m->loss + 1);
    // partial sums of the four weight gradients together: each is split over K
    // until its tiles of 128 x 64 times its K ranges reach two CTAs per SM
    for (int l = 0; l < 4; ++l) {
        size_t tiles = (size_t)(R[l] / 128) * (C[l] / 64);
        while (tiles < 2 * 148) tiles *= 2;
        m->ws_floats += tiles * 128 * 64;
    }
    mal((void**)&m->ws, sizeof(float) * m->ws_floats);
    if (e != cudaSuccess) return mfail(m, OD_ERR_CUDA, std::string("od_mlp_create: ") + cudaGetErrorString(e));
    return OD_OK;
}

void od_mlp_destroy(od_mlp* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    void* ps[] = {m->w, m->m1, m->m2, m->g, m->wb[0], m->wb[1], m->wb[2], m->wb[3], m->wbT[0], m->wbT[1], m->wbT[2],
                  m->wbT[3], m->Z[0], m->Z[1], m->Z[2], m->A[0], m->A[1], m->A[2], m->AT[0], m->AT[1], m->AT[2],
                  m->Y, m->dY, m->dYT, m->dZ[0], m->dZ[1], m->dZT[0], m->dZT[1], m->dZT[2], m->X, m->XT, m->T, m->rows_d, m->loss,
                  m->Xc, m->Yc, m->ws, m->wt};
    for (void* p : ps)
        if (p) cudaFree(p);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
}

const char* od_mlp_last_error(const od_mlp* m) { return m ? m->msg.c_str() : ""; }

long long od_mlp_param_count(const od_mlp* m) { return m ? m->nparam : 0; }

// host fp32 parameters (flat: W1 [256x896], b1, W2, b2, W3, b3, W4 [384x256], b4 [384];
// rows 320..383 of W4 and b4 must be zero) -> device, bf16 copies, Adam reset
int od_mlp_set_params(od_mlp* m, const float* host) {
    if (!m || !host) return OD_ERR_ARG;
    cudaSetDevice(m->device);
    const size_t P = sizeof(float) * (size_t)m->nparam;
    cudaError_t e = cudaMemcpyAsync(m->w, host, P, cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->m1, 0, P, m->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->m2, 0, P, m->stream);
    for (int l = 0; l < 4 && e == cudaSuccess; ++l) {
        const long long n = (long long)m->rows[l] * m->cols[l];
        cast_weights_kernel<<<blocks(n, 256), 256, 0, m->stream>>>(m->w + m->off_w[l], n, m->rows[l], m->cols[l],
                                                                    m->wb[l], m->wbT[l]);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = od::mlp::tile_fused_weights(m->wb, m->wt, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    m->step = 0;
    if (e != cudaSuccess) return mfail(m, OD_ERR_CUDA, cudaGetErrorString(e));
    return OD_OK;
}

int od_mlp_get_params(od_mlp* m, float* host) {
    if (!m || !host) return OD_ERR_ARG;
    cudaSetDevice(m->device);
    cudaError_t e = cudaMemcpyAsync(host, m->w, sizeof(float) * (size_t)m->nparam, cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    return e == cudaSuccess ? OD_OK : mfail(m, OD_ERR_CUDA, cudaGetErrorString(e));
}

// Y [rows x 384] fp32 (device) of X [rows x 896] bf16 (device); rows % 128 == 0
int od_mlp_forward(od_mlp* m, const void* X, int rows, float* Y) {
    if (!m || !X || !Y || rows <= 0 || rows % 128 || rows > m->mmax) return OD_ERR_ARG;
    cudaSetDevice(m->device);
    cudaError_t e = clear_status(m);
    if (e == cudaSuccess) e = forward(m, (const bf16*)X, rows, Y, false);
    if (e != cudaSuccess) return mfail(m, OD_ERR_CUDA, cudaGetErrorString(e));
    return read_status(m, nullptr);
}

// Gradients (host fp32, flat layout) and loss of a batch given as device rows:
// X [rows x 896] bf16, XT its transpose [896 x rows], T [rows x 384] fp32;
// only the first `valid` rows and 320 columns count.
int od_mlp_gradients(od_mlp* m, const void* X, const void* XT, const float* T, int rows, int valid, float* grads,
                     double* loss) {
    if (!m || !X || !XT || !T || rows <= 0 || rows % 128 || rows > m->mmax || valid <= 0 || valid > rows)
        return OD_ERR_ARG;
    cudaSetDevice(m->device);
    cudaError_t e = clear_status(m);
    if (e == cudaSuccess) e = cudaMemcpyAsync(m->T, T, sizeof(float) * (size_t)rows * kOutPad, cudaMemcpyDeviceToDevice, m->stream);
    if (e == cudaSuccess) e = forward(m, (const bf16*)X, rows, m->Y, true);
    if (e == cudaSuccess) e = backward(m, (const bf16*)XT, rows, valid, nullptr);
    if (e == cudaSuccess && grads)
        e = cudaMemcpyAsync(grads, m->g, sizeof(float) * (size_t)m->nparam, cudaMemcpyDeviceToHost, m->stream);
    if (e != cudaSuccess) return mfail(m, OD_ERR_CUDA, cudaGetErrorString(e));
    return read_status(m, loss, (double)valid * kOut);
}

// One Adam step on a batch gathered from device pools: features Xpool
// [n x 896] bf16, targets Tpool [n x 320] bf16, row indices `rows_host`
// (count = batch). Returns the batch's mean squared error (before the step).
int od_mlp_train_step(od_mlp* m, const void* Xpool, const void* Tpool, const long long* rows_host, int batch,
                      float lr, double* loss) {
    if (!m || !Xpool || !Tpool || !rows_host || batch <= 0 || batch > m->mmax) return OD_ERR_ARG;
    cudaSetDevice(m->device);
    const int M = (batch + 127) / 128 * 128;
    cudaError_t e = clear_status(m);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(m->rows_d, rows_host, sizeof(long long) * batch, cudaMemcpyHostToDevice, m->stream);
    auto* gk = aligned16(Xpool) ? gather_kernel<true> : gather_kernel<false>;
    gk<<<dim3(M / 64, kIn / 64), 256, 0, m->stream>>>((const bf16*)Xpool, m->rows_d, batch, M, m->X, m->XT);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = forward(m, m->X, M, m->Y, true);
    if (e == cudaSuccess) e = backward(m, m->XT, M, batch, (const bf16*)Tpool);
    m->step++;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
    AdamArgs A{};
    A.w = m->w;
    A.m1 = m->m1;
    A.m2 = m->m2;
    A.g = m->g;
    A.wt = m->wt;
    A.p = {lr, b1, b2, eps, c1, c2};
    int tiles = 0;
    for (int l = 0; l < 4; ++l) {
        A.off_w[l] = m->off_w[l];
        A.off_b[l] = m->off_b[l];
        A.rows[l] = m->rows[l];
        A.cols[l] = m->cols[l];
        A.wb[l] = m->wb[l];
        A.wbT[l] = m->wbT[l];
        tiles += (m->rows[l] / kAdamRows) * (m->cols[l] / 64);
    }
    if (e == cudaSuccess) {
        e = od::launch_dependent(true, adam_kernel, tiles + 4, 256, 0, m->stream, A, tiles);
    }
    if (e != cudaSuccess) return mfail(m, OD_ERR_CUDA, cudaGetErrorString(e));
    return read_status(m, loss, (double)batch * kOut);
}

// Normalisation of the closure's inputs and outputs.
int od_mlp_set_fused(od_mlp* m, int on) {
    if (!m) return OD_ERR_ARG;
    m->fused = on != 0;
    return OD_OK;
}

int od_mlp_set_scaling(od_mlp* m, const float* mean14, const float* scale14, const float* out_scale5) {
    if (!m || !mean14 || !scale14 || !out_scale5) return OD_ERR_ARG;
    std::memcpy(m->mean, mean14, sizeof m->mean);
    std::memcpy(m->scale, scale14, sizeof m->scale);
    std::memcpy(m->out_scale, out_scale5, sizeof m->out_scale);
    return OD_OK;
}

// ---- data kernels on caller-owned device memory (stream-ordered) ----

int od_project(const void* src, int src_f64, int nxc, int nyc, int nzc, int factor, void* dst, int dst_f64,
               void* stream) {
    if (!src || !dst || nxc <= 0 || nyc <= 0 || nzc <= 0 || factor < 1 || factor > 8) return OD_ERR_ARG;
    const ProjParams pp = proj_params(nxc, nyc, nzc, factor);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    if (src_f64)
        e = dst_f64 ? launch_project_f<double, double>(factor, src, dst, pp, s)
                    : launch_project_f<double, float>(factor, src, dst, pp, s);
    else
        e = dst_f64 ? launch_project_f<float, double>(factor, src, dst, pp, s)
                    : launch_project_f<float, float>(factor, src, dst, pp, s);
    return e == cudaSuccess ? OD_OK : OD_ERR_CUDA;
}

int od_closure_features(const void* state, int u_f64, int nx, int ny, int nz, double lx, double ly, double lz,
                        const float* mean14, const float* scale14, void* X, void* stream) {
    if (!state || !X || nx <= 0 || ny <= 0 || nz <= 0) return OD_ERR_ARG;
    const FeatParams fp = feat_params(nx, ny, nz, lx, ly, lz, mean14, scale14);
    const long long ne = (long long)nx * ny * nz;
    cudaStream_t s = (cudaStream_t)stream;
    if (u_f64)
        features_kernel<double><<<(unsigned)ne, 64, 0, s>>>((const double*)state, fp, (bf16*)X);
    else
        features_kernel<float><<<(unsigned)ne, 64, 0, s>>>((const float*)state, fp, (bf16*)X);
    return cudaGetLastError() == cudaSuccess ? OD_OK : OD_ERR_CUDA;
}

int od_f32_to_bf16(const float* a, void* b, long long n, void* stream) {
    if (!a || !b || n < 0) return OD_ERR_ARG;
    f32_to_bf16_kernel<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(a, (bf16*)b, n);
    return cudaGetLastError() == cudaSuccess ? OD_OK : OD_ERR_CUDA;
}

}  // extern "C"

// ------------------------------------------------------------------ solver hook
// Between phase A (which leaves the RHS in the solver's RHS buffer) and
// phase B of every RK stage: features of the stage's input state, network
// forward, rhs += out_scale * output. With the fused network on an f32
// state, phase A writes the features itself (closure_stage_features) and
// closure_network_hook runs the network alone.
namespace od {
static_assert(kChan == kFeatChan && kClip == kFeatClip, "phase A writes the same features");

bool closure_stage_features(void* user, StageFeatures* out) {
    od_mlp* m = (od_mlp*)user;
    if (!m || !m->fused || m->attached_f64 || !m->Xc) return false;
    out->X = m->Xc;
    for (int d = 0; d < 3; ++d) out->jac[d] = m->fp.jac[d];
    for (int a = 0; a < 16; ++a) out->D[a] = m->fp.D[a];
    for (int c = 0; c < kChan; ++c) {
        out->mean[c] = m->fp.mean[c];
        out->inv_scale[c] = m->fp.inv_scale[c];
    }
    return true;
}

cudaError_t closure_network_hook(void* user, const void* u_in, void* rhs, cudaStream_t s) {
    (void)u_in;
    od_mlp* m = (od_mlp*)user;
    od::mlp::FusedArgs a{};
    a.X = m->Xc;
    a.Wt = m->wt;
    for (int l = 0; l < 4; ++l) a.bias[l] = m->w + m->off_b[l];
    a.rhs = (float*)rhs;
    a.rhs_npts = m->nelem_c * 64;
    a.rhs_rows = (int)m->nelem_c;
    for (int v = 0; v < 5; ++v) a.rhs_scale[v] = m->out_scale[v];
    a.err = m->err;
    return od::mlp::launch_fused(a, (int)m->mpad_c, s);
}

cudaError_t closure_stage_hook(void* user, const void* u_in, void* rhs, cudaStream_t s) {
    od_mlp* m = (od_mlp*)user;
    cudaError_t e = cudaSuccess;
    if (m->attached_f64)
        features_kernel<double><<<(unsigned)m->nelem_c, 64, 0, s>>>((const double*)u_in, m->fp, m->Xc);
    else if (m->fused)
        features_tiled_kernel<<<(unsigned)((m->nelem_c + kFeatEpb - 1) / kFeatEpb), 16 * kFeatEpb, 0, s>>>(
            (const float*)u_in, m->fp, m->Xc, (long long)m->nelem_c);
    else
        features_kernel<float><<<(unsigned)m->nelem_c, 64, 0, s>>>((const float*)u_in, m->fp, m->Xc);
    e = cudaGetLastError();
    // the network runs on the solver's stream; the last layer's epilogue adds
    // out_scale * (output) into the RHS directly (f32 state)
    cudaStream_t keep = m->stream;
    m->stream = s;
    if (e == cudaSuccess && m->fused && !m->attached_f64) {
        // the whole network per 128-element tile in one kernel, output into the RHS
        od::mlp::FusedArgs a{};
        a.X = m->Xc;
        a.Wt = m->wt;
        for (int l = 0; l < 4; ++l) {
            a.bias[l] = m->w + m->off_b[l];
        }
        a.rhs = (float*)rhs;
        a.rhs_npts = m->nelem_c * 64;
        a.rhs_rows = (int)m->nelem_c;
        for (int v = 0; v < 5; ++v) a.rhs_scale[v] = m->out_scale[v];
        a.err = m->err;
        e = od::mlp::launch_fused(a, (int)m->mpad_c, s);
        m->stream = keep;
        return e;
    }
    if (e == cudaSuccess) e = hidden(m, m->Xc, (int)m->mpad_c, false);
    if (e == cudaSuccess) {
        if (m->attached_f64) {
            e = gemm(m, m->A[2], m->wb[3], (int)m->mpad_c, kOutPad, kHid, od::mlp::kStoreF32, m->w + m->off_b[3],
                     m->Yc, nullptr, nullptr, nullptr);
            const long long n = m->nelem_c * 64 * 5;
            const float* o = m->out_scale;
            if (e == cudaSuccess)
                apply_kernel<double><<<blocks(n, 256), 256, 0, s>>>((double*)rhs, m->Yc, m->nelem_c, o[0], o[1], o[2],
                                                                    o[3], o[4]);
        } else {
            od::mlp::GemmArgs a{};
            a.A = m->A[2];
            a.B = m->wb[3];
            a.M = (int)m->mpad_c;
            a.N = kOutPad;
            a.K = kHid;
            a.bias = m->w + m->off_b[3];
            a.err = m->err;
            a.rhs = (float*)rhs;
            a.rhs_npts = m->nelem_c * 64;
            a.rhs_rows = (int)m->nelem_c;
            for (int v = 0; v < 5; ++v) a.rhs_scale[v] = m->out_scale[v];
            e = od::mlp::launch_gemm(a, od::mlp::kApplyRhs, s, 0);
        }
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    m->stream = keep;
    return e;
}

// prepares the network for a solver's mesh; returns 0 or an OD_ERR code
int closure_prepare(od_mlp* m, int nx, int ny, int nz, double lx, double ly, double lz, bool f64) {
    const long long ne = (long long)nx * ny * nz;
    const long long mp = (ne + 127) / 128 * 128;
    if (mp > m->mmax) return mfail(m, OD_ERR_SIZE, "mesh has more elements than the network's batch capacity");
    cudaSetDevice(m->device);
    if (m->Xc) cudaFree(m->Xc);
    if (m->Yc) cudaFree(m->Yc);
    m->Xc = nullptr;
    m->Yc = nullptr;
    cudaError_t e = cudaMalloc(&m->Xc, sizeof(bf16) * mp * kIn);
    if (e == cudaSuccess) e = cudaMemset(m->Xc, 0, sizeof(bf16) * mp * kIn);
    if (e == cudaSuccess) e = cudaMalloc(&m->Yc, sizeof(float) * mp * kOutPad);
    if (e != cudaSuccess) return mfail(m, OD_ERR_CUDA, cudaGetErrorString(e));
    m->nelem_c = ne;
    m->mpad_c = mp;
    m->fp = feat_params(nx, ny, nz, lx, ly, lz, m->mean, m->scale);
    m->attached_f64 = f64;
    return OD_OK;
}
}  // namespace od
