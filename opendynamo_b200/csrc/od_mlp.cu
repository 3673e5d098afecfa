// Closure network: launches of the tcgen05 GEMM (one product, the grouped weight
// gradients, the sums over K ranges), of the fused inference kernel and of its
// weight image; self-tests.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/opendynamo.h"
#include "od_mlp.cuh"
#include "od_mlp_fused.cuh"

namespace od {
namespace mlp {

constexpr long long kSMs = 148;  // B200

// out = sum of the ksplit partial tiles in order (+ bias), a value per thread,
// 16 loads in flight
__global__ void __launch_bounds__(128) splitk_reduce_kernel(const float* __restrict__ ws, int ks, long long mn, int N,
                                                            const float* __restrict__ bias, float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= mn) return;
    float v = 0.f;
#pragma unroll 16
    for (int z = 0; z < ks; ++z) v += __ldcs(ws + z * mn + i);
    if (bias) v += bias[i % N];
    out[i] = v;
}

template <int NT, int EPI>
cudaError_t launch_gemm_t(const GemmArgs& g, cudaStream_t s) {
    const size_t smem = gemm_smem_bytes<NT>();
    // the shared-memory limit is set once per device (a host call per launch
    // cost more than the small GEMMs themselves)
    static bool prepared[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!prepared[dev]) {
        e = cudaFuncSetAttribute(gemm_kernel<NT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        prepared[dev] = true;
    }
    const int ks = g.ksplit > 1 ? g.ksplit : 1;
    dim3 grid((unsigned)(g.M / BM), (unsigned)(g.N / NT), (unsigned)ks);
    e = launch_dependent(true, gemm_kernel<NT, EPI>, grid, kGemmThreads, smem, s, g);
    if (e == cudaSuccess && ks > 1) {
        const long long mn = (long long)g.M * g.N;
        splitk_reduce_kernel<<<(unsigned)((mn + 127) / 128), 128, 0, s>>>(g.ws, ks, mn, g.N, g.bias, g.out_f32);
        e = cudaGetLastError();
    }
    return e;
}

template <int EPI>
cudaError_t launch_nt(const GemmArgs& g, int nt, cudaStream_t s) {
    if (nt == 256) return launch_gemm_t<256, EPI>(g, s);
    if (nt == 128) return launch_gemm_t<128, EPI>(g, s);
    return launch_gemm_t<64, EPI>(g, s);
}

// K ranges of a product with few tiles: doubled until there are two CTAs per
// SM, while every range keeps two K blocks and the partial sums fit.
static int split_k(const GemmArgs& g, int nt, size_t ws_floats) {
    const long long tiles = (long long)(g.M / BM) * (g.N / nt);
    const int kblocks = g.K / BK;
    int ks = 1;
    while (tiles * ks < 2 * kSMs && kblocks % (2 * ks) == 0 && kblocks / (2 * ks) >= 2 &&
           (size_t)(2 * ks) * g.M * g.N <= ws_floats)
        ks *= 2;
    return ks;
}

__global__ void __launch_bounds__(kGemmThreads, 2) gemm_group_kernel(const GemmGroup q) {
    int i = 0;
    while (i + 1 < kGroupMax && (int)blockIdx.x >= q.first[i + 1]) ++i;
    const int t = (int)blockIdx.x - q.first[i], rows = q.g[i].M / BM, cols = q.g[i].N / 64;
    gemm_tile<64, kStoreF32>(q.g[i], t % rows, t / rows % cols, t / (rows * cols));
}

// n <= kGroupMax fp32 products (no bias) in one launch, each split over K as
// launch_gemm splits it; ksplit of each is set, and where it is above 1 its
// partial sums are left in the product's own part of ws (the caller adds
// them up). The weight gradients of the closure: four products of 8 to 28
// tiles, at a batch of 8192 89 us launched one by one before the swizzled
// layout (16 to 39 each), 41 together.
cudaError_t launch_gemm_group(GemmArgs* g, int n, float* ws, size_t ws_floats, cudaStream_t s) {
    if (n < 1 || n > kGroupMax) return cudaErrorInvalidValue;
    GemmGroup q{};
    size_t used = 0;
    int ctas = 0;
    for (int i = 0; i < n; ++i) {
        GemmArgs& a = g[i];
        if (a.M <= 0 || a.N <= 0 || a.K <= 0 || a.M % BM || a.N % 64 || a.K % BK || a.bias)
            return cudaErrorInvalidValue;
        a.ws = ws + used;
        a.ksplit = split_k(a, 64, ws_floats - used);
        if (a.ksplit > 1) used += (size_t)a.ksplit * a.M * a.N;
        q.g[i] = a;
        q.first[i] = ctas;
        ctas += (a.M / BM) * (a.N / 64) * a.ksplit;
    }
    for (int i = n; i <= kGroupMax; ++i) q.first[i] = ctas;
    const size_t smem = gemm_smem_bytes<64>();
    static bool prepared[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!prepared[dev]) {
        e = cudaFuncSetAttribute(gemm_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        prepared[dev] = true;
    }
    return launch_dependent(true, gemm_group_kernel, (unsigned)ctas, kGemmThreads, smem, s, q);
}

// C = A B^T with the epilogue `epi`; M % 128 == 0, N % 64 == 0, K % 64 == 0.
// Tile width: the widest of 256 / 128 / 64 dividing N of which there are two
// tiles per SM, else 64 (fewer and wider tiles load A less often, but leave SMs
// idle; tiles of 64 and 128 run two per SM, of 256 one). Forward pass, tiles of 64
// / of 128 / by this rule: 8192 rows 57 / 75 / 57 us, 19072 rows 107 / 94 / 94,
// 65536 rows 257 / 206 / 206 (just past two tiles of 256 per SM, at 38016 rows,
// 128 would be better: 144 against 155). kStoreF32 products with few tiles and a long K (weight gradients)
// split K when the caller passes a workspace of ksplit * M * N floats.
cudaError_t launch_gemm(const GemmArgs& g0, int epi, cudaStream_t s, size_t ws_floats) {
    if (g0.M <= 0 || g0.N <= 0 || g0.K <= 0 || g0.M % BM || g0.N % 64 || g0.K % BK) return cudaErrorInvalidValue;
    GemmArgs g = g0;
    const long long rows = g.M / BM;
    int nt = 64;
    for (int c : {256, 128}) {
        if (g.N % c == 0 && rows * (g.N / c) >= 2 * kSMs) {
            nt = c;
            break;
        }
    }
    g.ksplit = epi == kStoreF32 && g.ws ? split_k(g, nt, ws_floats) : 1;
    switch (epi) {
        case kStoreF32: return launch_nt<kStoreF32>(g, nt, s);
        case kBiasGelu: return launch_nt<kBiasGelu>(g, nt, s);
        case kGeluGrad: return launch_nt<kGeluGrad>(g, nt, s);
        case kApplyRhs: return launch_nt<kApplyRhs>(g, nt, s);
        default: return cudaErrorInvalidValue;
    }
}

__global__ void tile_fused_weights_kernel(const __nv_bfloat16* __restrict__ W0, const __nv_bfloat16* __restrict__ W1,
                                          const __nv_bfloat16* __restrict__ W2, const __nv_bfloat16* __restrict__ W3,
                                          __nv_bfloat16* __restrict__ Wt) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;   // 16-byte chunk of the image
    if (q >= kFusedWeightBytes / 16) return;
    const uint32_t byte = q * 16;
    int s;
    uint32_t within;
    if (byte < 22u * kFStageBytes) {
        s = (int)(byte / kFStageBytes);
        within = byte % kFStageBytes;
    } else {
        s = 22 + (int)((byte - 22u * kFStageBytes) / kFOutStageBytes);
        within = (byte - 22u * kFStageBytes) % kFOutStageBytes;
    }
    const FStep f = fused_step(s);
    const int r = (int)(within / 1024) * 8 + (int)(within % 128) / 16;   // inverse of tile_off
    const int kc = (int)(within % 1024) / 128;
    const int K = f.layer == 0 ? kFIn : kFHid;
    const int n0 = f.layer == 3 ? f.pass * kFPass : 0;
    const __nv_bfloat16* W = f.layer == 0 ? W0 : f.layer == 1 ? W1 : f.layer == 2 ? W2 : W3;
    *reinterpret_cast<uint4*>(reinterpret_cast<char*>(Wt) + byte) =
        *reinterpret_cast<const uint4*>(W + (size_t)(n0 + r) * K + f.kb * BK + kc * 8);
}

cudaError_t tile_fused_weights(const __nv_bfloat16* const W[4], __nv_bfloat16* Wt, cudaStream_t s) {
    constexpr unsigned n = (unsigned)(kFusedWeightBytes / 16);
    tile_fused_weights_kernel<<<(n + 255) / 256, 256, 0, s>>>(W[0], W[1], W[2], W[3], Wt);
    return cudaGetLastError();
}

cudaError_t launch_fused(const FusedArgs& a, int M, cudaStream_t s) {
    if (M <= 0 || M % BM) return cudaErrorInvalidValue;
    static bool prepared[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!prepared[dev]) {
        e = cudaFuncSetAttribute(mlp_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_smem_bytes());
        if (e != cudaSuccess) return e;
        prepared[dev] = true;
    }
    // programmatic dependent launch: the prologue and the first weight copies
    // overlap the tail of the kernel before (griddepcontrol.wait in the kernel
    // orders everything that reads its results)
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(M / BM));
    cfg.blockDim = dim3(kFThreads);
    cfg.dynamicSmemBytes = fused_smem_bytes();
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, mlp_fused_kernel, a);
}

// Self-test of the bounded mbarrier wait of the tcgen05 kernels: a barrier
// nothing arrives on must give up after `limit` polls; after one arrival the
// same wait completes. out[0] = first wait completed, out[1] = second.
__global__ void mbar_wait_selftest_kernel(long long limit, int* out) {
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x != 0) return;
    const uint32_t b = smem_addr(&bar);
    mbar_init(b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const bool first = mbar_wait(b, 0, limit);
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory");
    const bool second = mbar_wait(b, 0, limit);
    out[0] = first ? 1 : 0;
    out[1] = second ? 1 : 0;
}

}  // namespace mlp
}  // namespace od

extern "C" int od_mlp_wait_selftest(long long limit, int device, int* first_completed, int* second_completed) {
    if (limit <= 0 || !first_completed || !second_completed) return OD_ERR_ARG;
    int prev = 0;
    if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return OD_ERR_CUDA;
    int* d = nullptr;
    int h[2] = {-1, -1};
    cudaError_t e = cudaMalloc((void**)&d, 2 * sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(d, 0xff, 2 * sizeof(int));
    if (e == cudaSuccess) {
        od::mlp::mbar_wait_selftest_kernel<<<1, 32>>>(limit, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
    if (d) cudaFree(d);
    cudaSetDevice(prev);
    if (e != cudaSuccess) return OD_ERR_CUDA;
    *first_completed = h[0];
    *second_completed = h[1];
    return OD_OK;
}

extern "C" int od_gemm_bf16(int M, int N, int K, const void* dA, const void* dB, float* dC, const float* dbias,
                            void* stream) {
    if (!dA || !dB || !dC) return OD_ERR_ARG;
    if (M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 64 || K % 64) return OD_ERR_ARG;
    int* err = nullptr;
    float* ws = nullptr;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t ws_floats = (size_t)16 * M * N;
    cudaError_t e = cudaMallocAsync((void**)&err, sizeof(int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), s);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&ws, ws_floats * sizeof(float), s);
    od::mlp::GemmArgs g{};
    g.A = (const __nv_bfloat16*)dA;
    g.B = (const __nv_bfloat16*)dB;
    g.M = M;
    g.N = N;
    g.K = K;
    g.bias = dbias;
    g.out_f32 = dC;
    g.err = err;
    g.ws = ws;
    if (e == cudaSuccess) e = od::mlp::launch_gemm(g, od::mlp::kStoreF32, s, ws_floats);
    int herr = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (err) cudaFreeAsync(err, s);
    if (ws) cudaFreeAsync(ws, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return OD_ERR_CUDA;
    return herr ? OD_ERR_CUDA : OD_OK;
}
