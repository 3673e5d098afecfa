// ParaView conversion of state files (the reference's scripts/h5_to_xdmf.py):
// the element-major planes are reordered into the global solution-point
// tensor with the derived velocity magnitude and pressure on the GPU, then
// written as a chunked point-field file and an XDMF description.

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/opendynamo.h"

namespace od {
namespace {

constexpr int kFields = 7;
constexpr int kPfWarps = 4;

// numpy.maximum: NaN if either operand is NaN
__device__ __forceinline__ float nan_max(float a, float b) { return (a != a || b != b) ? __int_as_float(0x7fc00000) : (a > b ? a : b); }

// an x-line of four points
template <class S>
__device__ __forceinline__ void load_xline(const S* p, bool vec, float* q) {
    if (!vec) {
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = (float)p[i];
    } else if constexpr (sizeof(S) == 4) {
        const float4 a = __ldcs(reinterpret_cast<const float4*>(p));
        q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
    } else {
        const double2 a = __ldcs(reinterpret_cast<const double2*>(p)), b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
        q[0] = (float)a.x; q[1] = (float)a.y; q[2] = (float)b.x; q[3] = (float)b.y;
    }
}

// Bound by memory: 20 (40 for f64 planes) bytes read and 28 written a point. A
// thread owns the 16 points of one j of one element, four lanes an element,
// and a warp takes eight elements that follow one another along z: the loads
// are whole x-lines (64 contiguous bytes an element and k), all 20 of a thread
// in flight, and a store is the four points along z of one (i, j), so that
// eight lanes write a whole 128-byte line of the tensor. Work index: (ex, ey,
// group of eight along z), the group fastest. vec: the buffers are 16-byte
// aligned (any caller's pointers are accepted). 48^3 f32 (340 MB): 91.0 us with a
// point a thread through shared memory, 75.8 with a z-line a thread (stores of
// 32-byte sectors), 60.8 so (5.6 TB/s).
template <class S>
__global__ void __launch_bounds__(32 * kPfWarps) point_fields_kernel(const S* __restrict__ u, int nx, int ny, int nz,
                                                                     long long npts, float* __restrict__ out,
                                                                     bool vec) {
    const unsigned nzg = ((unsigned)nz + 7) / 8;
    const long long w = (long long)blockIdx.x * kPfWarps + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31, j = lane >> 3;
    const unsigned col = (unsigned)(w / nzg);   // ey + ny ex
    const int ez = 8 * (int)(w - (long long)col * nzg) + (lane & 7);
    const int ex = (int)(col / (unsigned)ny), ey = (int)(col - (unsigned)ex * (unsigned)ny);
    if (ex >= nx || ez >= nz) return;
    const S* src = u + (ex + (long long)nx * (ey + (long long)ny * ez)) * 64 + 4 * j;
    float q[5][4][4];   // [variable][k][i]
#pragma unroll
    for (int v = 0; v < 5; ++v)
#pragma unroll
        for (int k = 0; k < 4; ++k) load_xline(src + v * npts + 16 * k, vec, q[v][k]);
    const long long npy = 4LL * ny, npz = 4LL * nz, ntot = 64LL * nx * ny * nz;
    float* dst = out + (4LL * ex * npy + 4LL * ey + j) * npz + 4LL * ez;
    auto put = [&](int c, int i, const float (&f)[4]) {
        float* p = dst + c * ntot + i * npy * npz;
        if (vec) {
            *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) p[k] = f[k];
        }
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float f[kFields][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            // operation order of h5_to_xdmf.py:76-79, f32, no contraction
            const float r = nan_max(q[0][k][i], 1e-30f);
            const float k2 = __fadd_rn(__fadd_rn(__fmul_rn(q[1][k][i], q[1][k][i]), __fmul_rn(q[2][k][i], q[2][k][i])),
                                       __fmul_rn(q[3][k][i], q[3][k][i]));
#pragma unroll
            for (int v = 0; v < 5; ++v) f[v][k] = q[v][k][i];
            f[5][k] = __fdiv_rn(__fsqrt_rn(k2), r);
            f[6][k] = nan_max(1e-7f, __fmul_rn(0.4f, __fsub_rn(q[4][k][i], __fdiv_rn(__fmul_rn(0.5f, k2), r))));
        }
#pragma unroll
        for (int c = 0; c < kFields; ++c) put(c, i, f[c]);
    }
}

const char* const kNames[kFields] = {"rho", "rhou", "rhov", "rhow", "E", "vel", "p"};

void put(char* err, int len, const std::string& s) {
    if (err && len > 0) std::snprintf(err, (size_t)len, "%s", s.c_str());
}

void copy_out(char* dst, size_t len, const std::string& s) {
    if (dst && len > 0) std::snprintf(dst, len, "%s", s.c_str());
}

// Path.with_suffix(suffix) of the script (h5_to_xdmf.py:81, 142)
std::string with_suffix(const std::string& path, const char* suffix) {
    const size_t slash = path.find_last_of('/');
    const size_t name0 = slash == std::string::npos ? 0 : slash + 1;
    const size_t dot = path.find_last_of('.');
    if (dot != std::string::npos && dot > name0 && dot + 1 < path.size()) return path.substr(0, dot) + suffix;
    return path + suffix;
}

std::string base_name(const std::string& path) {
    const size_t slash = path.find_last_of('/');
    return slash == std::string::npos ? path : path.substr(slash + 1);
}

std::string fmt_g(const char* f, double x) {
    char b[64];
    std::snprintf(b, sizeof b, f, x);
    return b;
}

}  // namespace
}  // namespace od

extern "C" int od_point_fields(const void* planes, int u_f64, int nx, int ny, int nz, float* out, void* stream) {
    if (!planes || !out || nx <= 0 || ny <= 0 || nz <= 0) return OD_ERR_ARG;
    const long long npts = 64LL * nx * ny * nz;
    if (ny > 65535 || (nz + 7) / 8 > 65535) return OD_ERR_ARG;   // mesh limits of this call
    const long long warps = (long long)nx * ny * ((nz + 7) / 8);
    const long long grid = (warps + od::kPfWarps - 1) / od::kPfWarps;
    if (grid > 0x7fffffffLL || (long long)nx * ny > 0xffffffffLL) return OD_ERR_ARG;
    const bool vec = ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(planes)) & 15) == 0;
    cudaStream_t s = (cudaStream_t)stream;
    if (u_f64)
        od::point_fields_kernel<double><<<(unsigned)grid, 32 * od::kPfWarps, 0, s>>>((const double*)planes, nx, ny, nz,
                                                                                      npts, out, vec);
    else
        od::point_fields_kernel<float><<<(unsigned)grid, 32 * od::kPfWarps, 0, s>>>((const float*)planes, nx, ny, nz,
                                                                                     npts, out, vec);
    return cudaGetLastError() == cudaSuccess ? OD_OK : OD_ERR_CUDA;
}

extern "C" long long od_xdmf_text(char* buf, size_t len, const char* h5_name, int npx, int npy, int npz, double lx,
                                  double ly, double lz, unsigned long long step, double t) {
    if (!h5_name || npx <= 0 || npy <= 0 || npz <= 0) return -1;
    std::string x;
    x += "<?xml version=\"1.0\" ?>\n<!DOCTYPE Xdmf SYSTEM \"Xdmf.dtd\" []>\n<Xdmf Version=\"2.0\">\n  <Domain>\n";
    x += "    <Grid Name=\"FR_Grid\" GridType=\"Uniform\" t_step=\"" + std::to_string(step) + "\" t_time=\"" +
         od::fmt_g("%.6g", t) + "\">\n";
    x += "      <Topology TopologyType=\"3DRectMesh\" Dimensions=\"" + std::to_string(npz + 1) + " " +
         std::to_string(npy + 1) + " " + std::to_string(npx + 1) + "\"/>\n";
    x += "      <Geometry GeometryType=\"VXVYVZ\">\n";
    const int n[3] = {npx, npy, npz};
    const double L[3] = {lx, ly, lz};
    for (int d = 0; d < 3; ++d) {
        x += "        <DataItem Dimensions=\"" + std::to_string(n[d] + 1) +
             "\" NumberType=\"Float\" Precision=\"8\" Format=\"XML\">\n          ";
        // numpy.linspace(0, L, n + 1): i * (L / n) + 0, the last point exactly L
        const double step_d = L[d] / n[d];
        for (int i = 0; i <= n[d]; ++i) {
            const double v = i == n[d] ? L[d] : (double)i * step_d + 0.0;
            if (i) x += " ";
            x += od::fmt_g("%.10g", v);
        }
        x += "\n        </DataItem>\n";
    }
    x += "      </Geometry>\n";
    for (int c = 0; c < od::kFields; ++c) {
        if (c) x += "\n";
        x += std::string("      <Attribute Name=\"") + od::kNames[c] + "\" AttributeType=\"Scalar\" Center=\"Cell\">\n";
        x += "        <DataItem Dimensions=\"" + std::to_string(npz) + " " + std::to_string(npy) + " " +
             std::to_string(npx) + "\" NumberType=\"Float\" Precision=\"4\" Format=\"HDF\">\n";
        x += std::string("          ") + h5_name + ":/data/" + od::kNames[c] + "\n";
        x += "        </DataItem>\n      </Attribute>";
    }
    x += "\n    </Grid>\n  </Domain>\n</Xdmf>\n";
    if (buf && len > 0) std::snprintf(buf, len, "%s", x.c_str());
    return (long long)x.size();
}

extern "C" int od_xdmf_convert(const char* src, char* out_h5, size_t out_h5_len, char* out_xmf, size_t out_xmf_len,
                               char* err, int err_len) {
    using namespace od;
    if (!src) {
        put(err, err_len, "no source file");
        return OD_ERR_ARG;
    }
    int nx = 0, ny = 0, nz = 0, fr = 0;
    unsigned long long step = 0;
    double t = 0, lx = 0, ly = 0, lz = 0;
    char ureal[4] = {0};
    if (od_state_info(src, &nx, &ny, &nz, &fr, &step, &t, &lx, &ly, &lz, ureal) != 0) {
        put(err, err_len, base_name(src) + ": " + od_state_error());
        return OD_ERR_IO;
    }
    const int f64 = std::strcmp(ureal, "f64") == 0;
    const size_t npts = (size_t)nx * ny * nz * 64;
    const size_t es = f64 ? 8 : 4;
    std::vector<unsigned char> host(5 * npts * es);
    if (od_state_load(src, host.data(), host.size(), f64, nx, ny, nz, &step, &t) != 0) {
        put(err, err_len, base_name(src) + ": " + od_state_error());
        return OD_ERR_IO;
    }
    void* d_in = nullptr;
    float* d_out = nullptr;
    std::vector<float> fields(kFields * npts);
    cudaError_t e = cudaMalloc(&d_in, host.size());
    if (e == cudaSuccess) e = cudaMalloc((void**)&d_out, fields.size() * sizeof(float));
    if (e == cudaSuccess) e = cudaMemcpy(d_in, host.data(), host.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && od_point_fields(d_in, f64, nx, ny, nz, d_out, nullptr) != OD_OK) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(fields.data(), d_out, fields.size() * sizeof(float), cudaMemcpyDeviceToHost);
    if (d_in) cudaFree(d_in);
    if (d_out) cudaFree(d_out);
    if (e != cudaSuccess) {
        put(err, err_len, std::string("CUDA: ") + cudaGetErrorString(e));
        return OD_ERR_CUDA;
    }
    const std::string h5 = with_suffix(src, ".pv.h5"), xmf = with_suffix(src, ".xmf");
    if (od_fields_save(h5.c_str(), fields.data(), kFields, kNames, 4LL * nx, 4LL * ny, 4LL * nz, 48, "gzip4") != 0) {
        put(err, err_len, od_state_error());
        return OD_ERR_IO;
    }
    const long long n = od_xdmf_text(nullptr, 0, base_name(h5).c_str(), 4 * nx, 4 * ny, 4 * nz, lx, ly, lz, step, t);
    std::vector<char> text((size_t)n + 1);
    od_xdmf_text(text.data(), text.size(), base_name(h5).c_str(), 4 * nx, 4 * ny, 4 * nz, lx, ly, lz, step, t);
    FILE* fp = std::fopen(xmf.c_str(), "wb");
    const bool ok = fp && std::fwrite(text.data(), 1, (size_t)n, fp) == (size_t)n;
    if (fp && std::fclose(fp) != 0) {
        put(err, err_len, "cannot write " + xmf);
        return OD_ERR_IO;
    }
    if (!ok) {
        put(err, err_len, "cannot write " + xmf);
        return OD_ERR_IO;
    }
    copy_out(out_h5, out_h5_len, h5);
    copy_out(out_xmf, out_xmf_len, xmf);
    return OD_OK;
}
