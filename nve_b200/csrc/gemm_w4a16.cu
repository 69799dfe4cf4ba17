// Entry points of the batched W4A16 GEMM:  Y[M,N] = X[M,K] . W^T  for one to three matrices that share X.
//
// Replaces the reference's batch > 1 path, which materialises the whole weight matrix as f16 in HBM
// (cuda/nve_kernels.cu:397-433, nve_dequant_w4a16) and then runs a dense GEMM on it (src/gpu_layer.rs:220-239): 0.625 +
// 2 + 2 = 4.6 bytes of HBM traffic per weight instead of 0.625.  The kernel is in gemm_w4a16_pair.cu.  Weights are always
// dequantised to f16, the type the reference dequantises to; bf16 activations are converted to f16 by a small pre-pass
// into the caller's scratch (bf16 weights would cost 2^-8 per weight and leave no tolerance margin; tcgen05.mma
// kind::f16 takes both operands in one format).
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "gemm_w4a16.cuh"

namespace nve {

constexpr int kKBlock = 64;  // K is a multiple of this

// bf16 -> f16, eight elements per thread.  The GEMM behind it may start at once: it asks for weights until its own wait returns.
__global__ void bf16_to_f16_kernel(const uint4* in, uint4* out, long long n8) {
    pdl_wait();
    pdl_launch_dependents();
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n8) return;
    const uint4 v = in[i];
    out[i] = make_uint4(bf16x2_to_f16x2(v.x), bf16x2_to_f16x2(v.y), bf16x2_to_f16x2(v.z), bf16x2_to_f16x2(v.w));
}

static size_t x16_region_bytes(int M, int K) { return (static_cast<size_t>(M) * K * 2 + 255) & ~static_cast<size_t>(255); }

// Scratch layout: [f16 copy of bf16 activations (x16_region_bytes)][partial tiles].  bf16 activations need the first
// region; the partial tiles of split runs use what is left.
static int run_gemm_multi(const void* X, int x_dtype, const PairMat* mats, int num_mats, int y_dtype, int M, int K, void* scratch,
                          size_t scratch_bytes, cudaStream_t st) {
    unsigned char* sp = static_cast<unsigned char*>(scratch);
    const uint16_t* x = static_cast<const uint16_t*>(X);
    if (x_dtype == NVE_DT_BF16) {
        const size_t xb = x16_region_bytes(M, K);
        int status;  // few rows: converted on the way into shared memory; above kFewRows a workspace without room for the copy stays refused
        if (aligned(sp, 16) && (M <= kFewRows || scratch_bytes >= xb) &&
            gemm_rows_try(X, x_dtype, mats, num_mats, y_dtype, M, K, sp, scratch_bytes, st, PairFinish(), &status))
            return status;
        if (sp == nullptr || scratch_bytes < xb) return set_status(NVE_ERR_TOO_LARGE);
        if (!aligned(sp, 16)) return set_status(NVE_ERR_BAD_ALIGNMENT);
        const long long n8 = static_cast<long long>(M) * K / 8;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>((n8 + 255) / 256));
        cfg.blockDim = dim3(256);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        if (pdl_enabled()) {
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
        }
        const cudaError_t e = cudaLaunchKernelEx(&cfg, bf16_to_f16_kernel, static_cast<const uint4*>(X), reinterpret_cast<uint4*>(sp), n8);
        count_launch();
        if (e != cudaSuccess) return set_cuda_status(e);
        x = reinterpret_cast<const uint16_t*>(sp);
        sp += xb;
        scratch_bytes -= xb;
    }
    return gemm_pair(x, mats, num_mats, y_dtype, M, K, sp, sp != nullptr ? scratch_bytes : 0, st);
}

}  // namespace nve

using namespace nve;

extern "C" size_t nve_b200_gemm_w4a16_multi_scratch_bytes(int M, const int* Ns, int num_mats, int K) {
    if (M <= 0 || K <= 0 || (K % kKBlock) != 0 || Ns == nullptr || num_mats < 1 || num_mats > 3) return 0;
    for (int m = 0; m < num_mats; m++)
        if (Ns[m] <= 0) return 0;
    return x16_region_bytes(M, K) + gemm_partial_bytes(Ns, num_mats, M, K);
}

extern "C" size_t nve_b200_gemm_w4a16_scratch_bytes(int M, int N, int K) { return nve_b200_gemm_w4a16_multi_scratch_bytes(M, &N, 1, K); }

namespace nve {
static int check_gemm_multi(const void* X, int x_dtype, const nve_b200_w4_matrix* mats, int num_mats, int y_dtype, int K, PairMat* g) {
    if (!X || !mats) return set_status(NVE_ERR_BAD_POINTER);
    if (num_mats < 1 || num_mats > 3 || K < kKBlock || (K % kKBlock) != 0) return set_status(NVE_ERR_BAD_SHAPE);
    if (x_dtype != NVE_DT_F16 && x_dtype != NVE_DT_BF16) return set_status(NVE_ERR_BAD_DTYPE);
    if (y_dtype != x_dtype && y_dtype != NVE_DT_F32) return set_status(NVE_ERR_BAD_DTYPE);
    if (!aligned(X, 16)) return set_status(NVE_ERR_BAD_ALIGNMENT);
    long long cols = 0;
    for (int m = 0; m < num_mats; m++) {
        if (!mats[m].nibbles || !mats[m].scales || !mats[m].out) return set_status(NVE_ERR_BAD_POINTER);
        if (mats[m].residual != nullptr) return set_status(NVE_ERR_BAD_POINTER);  // no fused residual in the GEMM
        if (mats[m].N < 1) return set_status(NVE_ERR_BAD_SHAPE);
        if (!aligned(mats[m].nibbles, 16) || !aligned(mats[m].scales, 8)) return set_status(NVE_ERR_BAD_ALIGNMENT);
        g[m] = {mats[m].nibbles, mats[m].scales, mats[m].out, mats[m].N};
        cols += mats[m].N;
    }
    if (cols > 0x7FFFFFF0ll) return set_status(NVE_ERR_BAD_SHAPE);
    return NVE_OK;
}
int gemm_qkv(const uint16_t* X, const nve_b200_w4_matrix* mats, int M, int K, void* scratch, size_t scratch_bytes, PairLeft* left, cudaStream_t st) {
    PairMat g[3];
    if (M < 1) return set_status(NVE_ERR_BAD_SHAPE);
    if (int s = check_gemm_multi(X, NVE_DT_F16, mats, 3, NVE_DT_F16, K, g); s != NVE_OK) return s;
    PairFinish fin;
    fin.left = left;
    return gemm_pair(X, g, 3, NVE_DT_F16, M, K, scratch, scratch != nullptr ? scratch_bytes : 0, st, fin);
}
}  // namespace nve

extern "C" int nve_b200_gemm_w4a16_multi(const void* X, int x_dtype, const nve_b200_w4_matrix* mats, int num_mats, int y_dtype,
                                         int M, int K, void* scratch, size_t scratch_bytes, nve_stream_t stream) {
    PairMat g[3];
    if (M < 1 || M > 64) return set_status(NVE_ERR_BAD_SHAPE);
    if (int s = check_gemm_multi(X, x_dtype, mats, num_mats, y_dtype, K, g); s != NVE_OK) return s;
    return run_gemm_multi(X, x_dtype, g, num_mats, y_dtype, M, K, scratch, scratch_bytes, static_cast<cudaStream_t>(stream));
}

extern "C" int nve_b200_gemm_w4a16_wide(const void* X, int x_dtype, const nve_b200_w4_matrix* mats, int num_mats, int y_dtype,
                                        int M, int K, void* scratch, size_t scratch_bytes, nve_stream_t stream) {
    PairMat g[3];
    if (M < 1) return set_status(NVE_ERR_BAD_SHAPE);
    if (int s = check_gemm_multi(X, x_dtype, mats, num_mats, y_dtype, K, g); s != NVE_OK) return s;
    return run_gemm_multi(X, x_dtype, g, num_mats, y_dtype, M, K, scratch, scratch_bytes, static_cast<cudaStream_t>(stream));
}

extern "C" int nve_b200_gemm_w4a16(const void* X, int x_dtype, const uint8_t* nibbles, const float* scales, void* Y, int y_dtype,
                                   int M, int N, int K, void* scratch, size_t scratch_bytes, nve_stream_t stream) {
    const nve_b200_w4_matrix one = {nibbles, scales, Y, nullptr, N};
    return nve_b200_gemm_w4a16_multi(X, x_dtype, &one, 1, y_dtype, M, K, scratch, scratch_bytes, stream);
}

extern "C" int nve_b200_gemm_w4a16_add_rmsnorm(const uint16_t* X, const uint8_t* nibbles, const float* scales, const uint16_t* residual,
                                               uint16_t* Y, const uint16_t* norm_weight, uint16_t* normed, float eps, int M, int N, int K,
                                               void* scratch, size_t scratch_bytes, nve_stream_t stream) {
    const nve_b200_w4_matrix one = {nibbles, scales, Y, nullptr, N};
    PairMat g[3];
    if (!residual || !norm_weight || !normed) return set_status(NVE_ERR_BAD_POINTER);
    if (int s = check_gemm_multi(X, NVE_DT_F16, &one, 1, NVE_DT_F16, K, g); s != NVE_OK) return s;
    if (M < 1 || !pair_norm_fits(N)) return set_status(NVE_ERR_BAD_SHAPE);
    if (!aligned(residual, 16) || !aligned(Y, 16) || !aligned(norm_weight, 16) || !aligned(normed, 16)) return set_status(NVE_ERR_BAD_ALIGNMENT);
    PairFinish fin;
    fin.res = residual;
    fin.norm_w = norm_weight;
    fin.normed = normed;
    fin.eps = eps;
    return gemm_pair(X, g, 1, NVE_DT_F16, M, K, scratch, scratch != nullptr ? scratch_bytes : 0, static_cast<cudaStream_t>(stream), fin);
}

extern "C" int nve_b200_gemm_w4a16_gateup_silu(const uint16_t* X, const nve_b200_w4_matrix* gate, const nve_b200_w4_matrix* up, uint16_t* mid,
                                               int M, int K, void* scratch, size_t scratch_bytes, nve_stream_t stream) {
    if (!gate || !up || !mid) return set_status(NVE_ERR_BAD_POINTER);
    nve_b200_w4_matrix mats[2] = {*gate, *up};
    mats[0].out = mats[1].out = mid;
    PairMat g[3];
    if (int s = check_gemm_multi(X, NVE_DT_F16, mats, 2, NVE_DT_F16, K, g); s != NVE_OK) return s;
    if (M < 1 || gate->N != up->N) return set_status(NVE_ERR_BAD_SHAPE);
    PairFinish fin;
    fin.silu = true;
    return gemm_pair(X, g, 2, NVE_DT_F16, M, K, scratch, scratch != nullptr ? scratch_bytes : 0, static_cast<cudaStream_t>(stream), fin);
}

extern "C" int nve_b200_gemm_error(int reset) { return gemm_pair_error(reset != 0); }

// ---------------------------------------------------------------------------------------------------------
// Allocation-free variant of the batched GEMM.
//
// Who needs it: the reference's batch > 1 call site (GpuWeight::matmul_x) receives only the activations and the
// weight tensors -- it has no workspace to hand down -- and it can run while a CUDA graph is being recorded,
// where cudaMalloc is illegal; a serving thread that must not touch the allocator is in the same position.
// For those callers the partial tiles of split runs live in a fixed array inside the library image instead of a
// caller-provided buffer.
//
// Cost and limits: the array is kStaticScratchFloats * 4 bytes (4 MiB) of device memory on every GPU that loads
// the library, until the process exits.  A call whose partial tiles exceed it, counted
// as noalloc_partial_bytes does, is rejected with NVE_ERR_TOO_LARGE; what the kernel could use beyond it only lengthens its runs.  All calls share the one array: two such GEMMs that overlap on the same
// GPU (different streams) race on it; issue them on one stream.  The array keeps whatever the previous call
// left in it; nothing in it has to start at zero, because every partial a call reads was written by that same
// call's first kernel.
//
// The first call on each device looks up the array's device address (cudaGetSymbolAddress, with that device
// current) and caches it; make that first call before starting any stream capture.
// ---------------------------------------------------------------------------------------------------------
namespace nve {

constexpr size_t kStaticScratchFloats = static_cast<size_t>(1) << 20;  // 1 Mi floats = 4 MiB
static __device__ __align__(256) float g_gemm_static_scratch[kStaticScratchFloats];

// What counts against the limit: partial tiles of M x 128 floats, two per SM, of runs of at least two units of 256 along K that are cut
// evenly over the SMs, where K is a multiple of 256 and not (M > 32 and a whole tile for every SM).  The sizes that are taken are part of the
// interface and do not follow the tiles of the kernel behind it.
static size_t noalloc_partial_bytes(int M, int N, int K) {
    const long long tiles = (static_cast<long long>(N) + 127) / 128, sb = K / 256, sms = sm_count();
    if (K % 256 != 0 || (M > 32 && tiles >= sms)) return 0;
    const long long total = tiles * sb;
    const long long U = std::max((total + sms - 1) / sms, std::min(sb, 2ll));
    return U % sb == 0 ? 0 : static_cast<size_t>(2 * ((total + U - 1) / U) * M * 128) * sizeof(float);
}

// Device address of g_gemm_static_scratch on the current device.  In host code the symbol itself is only a
// stand-in and must never be passed to a kernel; the address comes from the runtime, once per device.
static int static_scratch_address(float** out) {
    static std::mutex mu;
    static float* cached[64] = {};
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_cuda_status(e);
    if (dev < 0 || dev >= 64) return set_status(NVE_ERR_BAD_SHAPE);
    std::lock_guard<std::mutex> lock(mu);
    if (cached[dev] == nullptr) {
        float* ptr = nullptr;
        e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_gemm_static_scratch);
        if (e != cudaSuccess) return set_cuda_status(e);
        if (ptr == nullptr) return set_status(NVE_ERR_BAD_POINTER);
        cached[dev] = ptr;
    }
    *out = cached[dev];
    return NVE_OK;
}

}  // namespace nve

extern "C" int nve_b200_gemm_w4a16_noalloc(const void* X, int x_dtype, const uint8_t* nibbles, const float* scales, void* Y,
                                           int y_dtype, int M, int N, int K, nve_stream_t stream) {
    if (!X || !nibbles || !scales || !Y) return set_status(NVE_ERR_BAD_POINTER);
    if (M < 1 || M > 64 || N < 1 || K < kKBlock || (K % kKBlock) != 0) return set_status(NVE_ERR_BAD_SHAPE);
    if (x_dtype != NVE_DT_F16 && x_dtype != NVE_DT_BF16) return set_status(NVE_ERR_BAD_DTYPE);
    if (y_dtype != x_dtype && y_dtype != NVE_DT_F32) return set_status(NVE_ERR_BAD_DTYPE);
    if (!aligned(X, 16) || !aligned(nibbles, 16) || !aligned(scales, 8)) return set_status(NVE_ERR_BAD_ALIGNMENT);
    const size_t need = (x_dtype == NVE_DT_BF16 ? x16_region_bytes(M, K) : 0) + noalloc_partial_bytes(M, N, K);
    if (need > kStaticScratchFloats * sizeof(float)) return set_status(NVE_ERR_TOO_LARGE);
    float* scratch = nullptr;
    int st = static_scratch_address(&scratch);
    if (st != NVE_OK) return st;
    const PairMat one = {nibbles, scales, Y, N};
    return run_gemm_multi(X, x_dtype, &one, 1, y_dtype, M, K, scratch, kStaticScratchFloats * sizeof(float), static_cast<cudaStream_t>(stream));
}
