// Flow diagnostics of a state on the device: volume integrals (mass,
// x-momentum, total energy, kinetic energy, enstrophy) and x-z plane
// averages at every y row of solution points (the mean profile and the
// second moments a Reynolds-stress comparison needs).
//
// Quadrature: Gauss-Legendre weights of the solution points times the
// element Jacobian (h/2 per axis). Gradients for the vorticity are the
// element-local FR derivative D (no interface correction).
//
// Sums are formed in double. 16 threads per element, each an x-line of four
// points, two elements per warp; a warp walks the elements of one y row of
// elements and keeps its twelve sums in registers, so that the reduction over
// the block and the global atomics (37 per block) are paid once per block and
// not once per element.

#include <cuda_runtime.h>

#include "od_launch.h"

namespace od {
namespace {

struct DiagParams {
    int nx, ny, nz;
    double hx, hy, hz;   // element sizes
    double w[4];         // GL weights on [-1, 1]
    double D[16];        // D[a*4+m] = l'_m(x_a)
};

constexpr int kDiagWarps = 4;     // warps per block
constexpr int kDiagSums = 12;     // per y row of points: the 8 profile moments, rho u, E, kinetic energy, enstrophy
constexpr int kDiagBlocks = 444;  // 148 SMs x the 3 blocks that are resident (168 registers a thread)

// the x-line p[0..3] of a plane
__device__ __forceinline__ void load_line(const float* p, double* q) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
}

__device__ __forceinline__ void load_line(const double* p, double* q) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(p));
    const double2 b = __ldg(reinterpret_cast<const double2*>(p) + 1);
    q[0] = a.x; q[1] = a.y; q[2] = b.x; q[3] = b.y;
}

// r[i] = sum_m c[m] (x-line of row m)[i] over four x-lines of a shared plane,
// the lines `step` apart; a plane holds the first halves of its 16 lines,
// then the second halves (conflict-free 128-bit accesses)
__device__ __forceinline__ void rows_deriv(const double2* plane, int line0, int step, const double* c, double* r) {
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = 0.0;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const double2 a = plane[line0 + step * m], b = plane[16 + line0 + step * m];
        r[0] += c[m] * a.x;
        r[1] += c[m] * a.y;
        r[2] += c[m] * b.x;
        r[3] += c[m] * b.y;
    }
}

// Block b: chunk b % chunks of element row ey = b / chunks. Bound by f64
// arithmetic (about 90 operations a point: 35 us for 48^3 at 64 a cycle and
// SM) and the shared-memory reads of the derivatives. od_diagnostics at 48^3,
// f32: 1446 us with a block per element (38 global atomics each, six of them
// on the same addresses for every element), 104 us so.
template <class S>
__global__ void __launch_bounds__(32 * kDiagWarps, 3) diag_kernel(const S* __restrict__ u, const DiagParams P, int chunks,
                                                               double* vol, double* prof) {
    __shared__ double2 q[kDiagWarps][2][4][32];   // rho, rho u, rho v, rho w of the warp's two elements
    __shared__ double red[kDiagWarps][4][kDiagSums];
    const int ey = (int)(blockIdx.x / (unsigned)chunks), chunk = (int)(blockIdx.x - (unsigned)ey * (unsigned)chunks);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int es = lane >> 4, l = lane & 15, j = l & 3, k = l >> 2;
    const long long npts = (long long)P.nx * P.ny * P.nz * 64;
    const unsigned nx = (unsigned)P.nx, row = nx * (unsigned)P.nz, stride = 2u * (unsigned)(chunks * kDiagWarps);
    double cy[4], cz[4], wpl[4], acc[kDiagSums];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        cy[m] = P.D[j * 4 + m] * (2.0 / P.hy);
        cz[m] = P.D[k * 4 + m] * (2.0 / P.hz);
        wpl[m] = P.w[m] * P.w[k] * (0.25 * P.hx * P.hz);
    }
#pragma unroll
    for (int c = 0; c < kDiagSums; ++c) acc[c] = 0.0;
    const double jx = 2.0 / P.hx;
    // first of the warp's two elements in the row; both halves of the warp
    // make the same number of passes (the last may have one element)
    for (unsigned first = 2u * (unsigned)(chunk * kDiagWarps + warp); first < row; first += stride) {
        const unsigned idx = first + es;
        const bool live = idx < row;
        const unsigned c = live ? idx : first, ez = c / nx, ex = c - ez * nx;
        const S* p = u + ((long long)ex + (long long)nx * (ey + (long long)P.ny * ez)) * 64 + 4 * l;
        double s[5][4];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            load_line(p + v * npts, s[v]);
            // no partner: a state whose zero weight gives zero (the first
            // element's infinite or NaN values times zero would not)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[v][i] = live ? s[v][i] : (v == 0 ? 1.0 : 0.0);
        }
        __syncwarp();   // the pass before is done with the planes
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            q[warp][es][v][l] = make_double2(s[v][0], s[v][1]);
            q[warp][es][v][16 + l] = make_double2(s[v][2], s[v][3]);
        }
        __syncwarp();
        // rho times the vorticity, from the nine derivatives it needs (rho in
        // all directions, rho u in y and z, rho v in x and z, rho w in x and
        // y), one direction at a time
        double ox[4], oy[4], oz[4], ir[4];
        const double2(*pl)[32] = q[warp][es];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            double rx = 0.0, vx = 0.0, wx = 0.0;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                rx += P.D[i * 4 + m] * s[0][m];
                vx += P.D[i * 4 + m] * s[2][m];
                wx += P.D[i * 4 + m] * s[3][m];
            }
            ir[i] = 1.0 / s[0][i];
            oy[i] = -jx * (wx - s[3][i] * ir[i] * rx);
            oz[i] = jx * (vx - s[2][i] * ir[i] * rx);
        }
        {
            double r[4], d[4];
            rows_deriv(pl[0], 4 * k, 1, cy, r);
            rows_deriv(pl[3], 4 * k, 1, cy, d);
#pragma unroll
            for (int i = 0; i < 4; ++i) ox[i] = d[i] - s[3][i] * ir[i] * r[i];
            rows_deriv(pl[1], 4 * k, 1, cy, d);
#pragma unroll
            for (int i = 0; i < 4; ++i) oz[i] -= d[i] - s[1][i] * ir[i] * r[i];
            rows_deriv(pl[0], j, 4, cz, r);
            rows_deriv(pl[1], j, 4, cz, d);
#pragma unroll
            for (int i = 0; i < 4; ++i) oy[i] += d[i] - s[1][i] * ir[i] * r[i];
            rows_deriv(pl[2], j, 4, cz, d);
#pragma unroll
            for (int i = 0; i < 4; ++i) ox[i] -= d[i] - s[2][i] * ir[i] * r[i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double a = s[1][i] * ir[i], b = s[2][i] * ir[i], d = s[3][i] * ir[i];
            const double w = live ? wpl[i] : 0.0;
            const double wa = w * a, wb = w * b, wd = w * d;
            acc[0] += w * s[0][i];
            acc[1] += wa;
            acc[2] += wb;
            acc[3] += wd;
            acc[4] += wa * a;
            acc[5] += wb * b;
            acc[6] += wd * d;
            acc[7] += wa * b;
            acc[8] += w * s[1][i];
            acc[9] += w * s[4][i];
            acc[10] += wa * s[1][i] + wb * s[2][i] + wd * s[3][i];
            acc[11] += w * ir[i] * (ox[i] * ox[i] + oy[i] * oy[i] + oz[i] * oz[i]);
        }
    }
#pragma unroll
    for (int c = 0; c < kDiagSums; ++c) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
        if (lane < 4) red[warp][lane][c] = acc[c];
    }
    __syncthreads();
    if (threadIdx.x < 4 * kDiagSums) {
        const int jj = threadIdx.x & 3, c = threadIdx.x >> 2;
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kDiagWarps; ++w) t += red[w][jj][c];
        if (prof && c < 8) atomicAdd(&prof[((long long)ey * 4 + jj) * 8 + c], t);
        red[0][jj][c] = t;
    }
    __syncthreads();
    // the volume integrals: the rows' sums weighted along y (plane sums x w_j hy / 2)
    if (threadIdx.x < 5) {
        const int t = threadIdx.x, c = t == 0 ? 0 : 7 + t;   // rho, rho u, E, kinetic energy, enstrophy
        double v = 0.0;
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) v += P.w[jj] * red[0][jj][c];
        atomicAdd(vol + t, (t >= 3 ? 0.25 : 0.5) * P.hy * v);
    } else if (threadIdx.x == 5 && chunk == 0) {
        const double sw = P.w[0] + P.w[1] + P.w[2] + P.w[3];
        atomicAdd(vol + 5, (double)row * (sw * sw * sw * (0.125 * P.hx * P.hy * P.hz)));
    }
}

}  // namespace

cudaError_t launch_diag(const void* u, bool u_f64, int nx, int ny, int nz, double lx, double ly, double lz,
                        const TablesD& tab, double* d_vol6, double* d_prof, cudaStream_t s) {
    DiagParams P;
    P.nx = nx;
    P.ny = ny;
    P.nz = nz;
    P.hx = lx / nx;
    P.hy = ly / ny;
    P.hz = lz / nz;
    // GL weights from the points: w_i = 2 / ((1 - x^2) P'_4(x)^2)
    for (int a = 0; a < 4; ++a) {
        const double x = tab.pts[a];
        const double dp4 = (4.0 * (x * (35 * x * x * x * x - 30 * x * x + 3) / 8.0) -
                            4.0 * ((5 * x * x * x - 3 * x) / 2.0)) / (x * x - 1.0);
        P.w[a] = 2.0 / ((1.0 - x * x) * dp4 * dp4);
    }
    for (int a = 0; a < 16; ++a) P.D[a] = tab.D[a];
    const long long nelem = (long long)nx * ny * nz;
    if (nelem > 0x7fffffffLL) return cudaErrorInvalidValue;
    // as many chunks per element row as fill the GPU once, and no more than
    // give every warp a pair of elements
    const long long pairs = ((long long)nx * nz + 1) / 2;
    long long chunks = kDiagBlocks / ny;
    if (chunks > (pairs + kDiagWarps - 1) / kDiagWarps) chunks = (pairs + kDiagWarps - 1) / kDiagWarps;
    if (chunks < 1) chunks = 1;
    const unsigned grid = (unsigned)(ny * chunks);
    if (u_f64)
        diag_kernel<double><<<grid, 32 * kDiagWarps, 0, s>>>((const double*)u, P, (int)chunks, d_vol6, d_prof);
    else
        diag_kernel<float><<<grid, 32 * kDiagWarps, 0, s>>>((const float*)u, P, (int)chunks, d_vol6, d_prof);
    return cudaGetLastError();
}

}  // namespace od
