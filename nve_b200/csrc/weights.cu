// Weight-side helpers: dense f16 GEMV, full dequantisation, on-device Q4 quantisation and repacking,
// and the synthetic input generator.
//
// Replaces cuda/nve_kernels.cu:273-314 (nve_matvec_f16) and :397-433 (nve_dequant_w4a16) of the reference
// project, and moves src/quantize.rs:711-731 (quantize_block_q4) and :437-463 (extract_for_gpu) onto the
// device with bit-identical results.
#include "common.cuh"

namespace nve {

// ---------------------------------------------------------------------------------------------
// Dense f16 GEMV: one warp per row, 128-bit loads when aligned.
// ---------------------------------------------------------------------------------------------
template <bool VEC> __global__ void __launch_bounds__(256) matvec_f16_kernel(const uint16_t* x, const uint16_t* W,
                                                                              uint16_t* out, int N, int K) {
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= N) return;
    const uint16_t* w = W + static_cast<long long>(row) * K;
    float acc = 0.0f;
    if constexpr (VEC) {
        for (int c = lane; c < K / 8; c += 32) {
            const uint4 wv = ld_stream_u4(w + c * 8);
            const uint4 xv = reinterpret_cast<const uint4*>(x)[c];
            const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
            const uint32_t xx[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                acc = fmaf(Act16<NVE_DT_F16>::to_f32(ww[j] & 0xFFFFu), Act16<NVE_DT_F16>::to_f32(xx[j] & 0xFFFFu), acc);
                acc = fmaf(Act16<NVE_DT_F16>::to_f32(ww[j] >> 16), Act16<NVE_DT_F16>::to_f32(xx[j] >> 16), acc);
            }
        }
    } else {
        for (int k = lane; k < K; k += 32) acc = fmaf(Act16<NVE_DT_F16>::to_f32(w[k]), Act16<NVE_DT_F16>::to_f32(x[k]), acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) out[row] = Act16<NVE_DT_F16>::from_f32(acc);
}

// ---------------------------------------------------------------------------------------------
// Dequantisation: one thread per 16-byte block -> 32 outputs (4 x 128-bit stores).
// ---------------------------------------------------------------------------------------------
template <int ODT> __global__ void __launch_bounds__(256) dequant_kernel(const uint8_t* nibbles, const float* scales,
                                                                          const float* awq, uint16_t* out,
                                                                          long long total_blocks, int nb) {
    const long long blk = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (blk >= total_blocks) return;
    const uint4 w = ld_stream_u4(nibbles + blk * 16);
    const float sc = scales[blk];
    const int b = static_cast<int>(blk % nb);
    const uint32_t wv[4] = {w.x, w.y, w.z, w.w};
    uint16_t h[32];
#pragma unroll
    for (int j = 0; j < 4; j++) {
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const int lo = static_cast<int>((wv[j] >> (8 * t)) & 0xFu) - 8;
            const int hi = static_cast<int>((wv[j] >> (8 * t + 4)) & 0xFu) - 8;
            float vlo = __fmul_rn(static_cast<float>(lo), sc);
            float vhi = __fmul_rn(static_cast<float>(hi), sc);
            if (awq != nullptr) {
                vlo = __fmul_rn(vlo, awq[b * 32 + 4 * j + t]);
                vhi = __fmul_rn(vhi, awq[b * 32 + 16 + 4 * j + t]);
            }
            h[4 * j + t] = Act16<ODT>::from_f32(vlo);
            h[16 + 4 * j + t] = Act16<ODT>::from_f32(vhi);
        }
    }
    uint4* dst = reinterpret_cast<uint4*>(out + blk * 32);
#pragma unroll
    for (int v = 0; v < 4; v++) {
        uint4 o;
        o.x = h[8 * v + 0] | (static_cast<uint32_t>(h[8 * v + 1]) << 16);
        o.y = h[8 * v + 2] | (static_cast<uint32_t>(h[8 * v + 3]) << 16);
        o.z = h[8 * v + 4] | (static_cast<uint32_t>(h[8 * v + 5]) << 16);
        o.w = h[8 * v + 6] | (static_cast<uint32_t>(h[8 * v + 7]) << 16);
        dst[v] = o;
    }
}

template <int ODT> __global__ void dequant_scalar_kernel(const uint8_t* nibbles, const float* scales, const float* awq,
                                                          uint16_t* out, long long total, int K) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long blk = i / 32;
    const int pos = static_cast<int>(i % 32);
    const uint8_t bv = nibbles[blk * 16 + (pos & 15)];
    const int nib = (pos < 16) ? (bv & 0xF) : (bv >> 4);
    float v = __fmul_rn(static_cast<float>(nib - 8), scales[blk]);
    if (awq != nullptr) v = __fmul_rn(v, awq[i % K]);
    out[i] = Act16<ODT>::from_f32(v);
}

// ---------------------------------------------------------------------------------------------
// On-device Q4 quantisation (bit-identical to the host quantizer of the reference project):
//   amax = max|v| ; scale = amax > 0 ? amax/7 : 0 ; inv = scale > 0 ? 1/scale : 0
//   q = clamp(round_half_away(v*inv), -8, 7) + 8 ; device byte j = q[j] | q[j+16] << 4
// HBM is the floor (4 bytes in, 0.625 out per weight), the instruction count what has to be kept below it: at 25 instructions
// per weight-lane and two IEEE divisions per lane and block the kernel was bound by issue, as the form with one thread per
// block (whose warp-wide loads touched 32 cache lines each) was by its loads.  So: eight lanes share a block, one 16-byte
// load each (512 contiguous bytes per warp-wide load, four in flight per thread); the four blocks of a lane group are
// reduced together, so that lane t holds the maximum of block t & 3, divides for it alone and hands the factor back.
// ---------------------------------------------------------------------------------------------
// clamp(round_half_away(v), -8, 7), NaN -> 0 as a saturating float->int8 cast gives.
__device__ __forceinline__ int round_q4(float v) {
    if (v != v) return 0;
    return static_cast<int>(fminf(fmaxf(roundf(v), -8.0f), 7.0f));
}
// Four codes q + 8, one per byte, of products p with |p| <= 7.01: floor(p + 8.5) is round-half-away(p) + 8 except where p is a
// negative tie, and adding one to the bits of a negative p (one ulp away from zero) settles those.  The sum with 2^22 + 8.5,
// rounded down, holds floor(2 * (p + 8.5)) in its low bits.
__device__ __forceinline__ uint32_t pack_q4(float p0, float p1, float p2, float p3) {
    auto low = [](float p) {
        const uint32_t b = __float_as_uint(p);
        return __float_as_uint(__fadd_rd(__uint_as_float(b + (b >> 31)), 4194312.5f));
    };
    constexpr uint32_t kBase = 0x4A800000u * 0x01010101u;  // 2^22 in each summand
    const uint32_t t = low(p0) + low(p1) * 0x100u + low(p2) * 0x10000u + low(p3) * 0x1000000u;
    return ((t - kBase) >> 1) & 0x0F0F0F0Fu;
}

constexpr int kQ4Loads = 4;  // 16-byte loads per thread = blocks per group of eight lanes
template <bool AWQ>
__global__ void __launch_bounds__(256) q4_quantize_kernel(const float* W, const float* awq_scales, uint8_t* nibbles, float* scales,
                                                          long long total_blocks, int nb) {
    pdl_wait();
    const int t = threadIdx.x & 7;  // elements 4t .. 4t + 3 of the blocks blk0 + 32 * i
    const long long blk0 = static_cast<long long>(blockIdx.x) * (32 * kQ4Loads) + (threadIdx.x >> 3);
    float v[kQ4Loads][4];
#pragma unroll
    for (int i = 0; i < kQ4Loads; i++) {
        const long long blk = blk0 + 32 * i;
        uint4 r = make_uint4(0, 0, 0, 0);
        if (blk < total_blocks) r = ld_stream_u4(W + blk * 32 + 4 * t);
        v[i][0] = __uint_as_float(r.x);
        v[i][1] = __uint_as_float(r.y);
        v[i][2] = __uint_as_float(r.z);
        v[i][3] = __uint_as_float(r.w);
    }
    if (AWQ) {
#pragma unroll
        for (int i = 0; i < kQ4Loads; i++) {
            const float* a = awq_scales + static_cast<int>((blk0 + 32 * i) % nb) * 32 + 4 * t;
#pragma unroll
            for (int e = 0; e < 4; e++) v[i][e] = __fmul_rn(v[i][e], a[e]);
        }
    }
    // maxima of the four blocks over the eight lanes: lane t ends up with block t & 3
    float m[kQ4Loads];
#pragma unroll
    for (int i = 0; i < kQ4Loads; i++) m[i] = max_nan(max_nan(fabsf(v[i][0]), fabsf(v[i][1])), max_nan(fabsf(v[i][2]), fabsf(v[i][3])));
    {
        const bool up2 = (t & 2) != 0, up1 = (t & 1) != 0;
#pragma unroll
        for (int i = 0; i < 2; i++) m[i] = max_nan(up2 ? m[i + 2] : m[i], __shfl_xor_sync(0xffffffffu, up2 ? m[i] : m[i + 2], 2));
        m[0] = max_nan(up1 ? m[1] : m[0], __shfl_xor_sync(0xffffffffu, up1 ? m[0] : m[1], 1));
        m[0] = max_nan(m[0], __shfl_xor_sync(0xffffffffu, m[0], 4));
    }
    float amax = m[0];
    // a NaN or infinity in the block, or a maximum so small that the reciprocal of its scale overflows: one by one below
    const bool plain = !__any_sync(0xffffffffu, !(amax == 0.0f || (amax >= 1e-30f && amax < INFINITY)));
    if (!plain) {
#pragma unroll
        for (int i = 0; i < kQ4Loads; i++) {
            // fmaxf: NaN never wins, matching f32::max folding from 0
            float a = fmaxf(fmaxf(fmaxf(fmaxf(0.0f, fabsf(v[i][0])), fabsf(v[i][1])), fabsf(v[i][2])), fabsf(v[i][3]));
            for (int k = 1; k < 8; k <<= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, k));
            if ((t & 3) == i) amax = a;
        }
    }
    const float scale = amax > 0.0f ? __fdiv_rn(amax, 7.0f) : 0.0f;
    const float inv = scale > 0.0f ? __fdiv_rn(1.0f, scale) : 0.0f;
    if (t < 4 && blk0 + 32 * t < total_blocks) scales[blk0 + 32 * t] = scale;
    uint32_t q[kQ4Loads];
#pragma unroll
    for (int i = 0; i < kQ4Loads; i++) {
        const float f = __shfl_sync(0xffffffffu, inv, i, 8);
        float p[4];
#pragma unroll
        for (int e = 0; e < 4; e++) p[e] = __fmul_rn(v[i][e], f);
        if (plain) {
            q[i] = pack_q4(p[0], p[1], p[2], p[3]);
        } else {
            q[i] = 0;
#pragma unroll
            for (int e = 0; e < 4; e++) q[i] |= static_cast<uint32_t>(round_q4(p[e]) + 8) << (8 * e);
        }
    }
    // byte j of a block is element j | element j + 16 << 4: lane t < 4 has the low, lane t + 4 the high halves of word t.  Of
    // every two blocks the lower lanes store the first, the upper lanes the second.
    const bool hi = (t & 4) != 0;
#pragma unroll
    for (int i = 0; i < kQ4Loads; i += 2) {
        const uint32_t own = hi ? q[i + 1] : q[i];
        const uint32_t got = __shfl_xor_sync(0xffffffffu, hi ? q[i] : q[i + 1], 4);
        const uint32_t w = hi ? got | (own << 4) : own | (got << 4);
        const long long blk = blk0 + 32 * (i + (hi ? 1 : 0));
        if (blk < total_blocks) reinterpret_cast<uint32_t*>(nibbles)[blk * 4 + (t & 3)] = w;
    }
}

// CPU block (f32 scale + 16 bytes of {2i, 2i+1}) -> device layout.
__global__ void __launch_bounds__(256) q4_repack_kernel(const uint8_t* cpu_blocks, uint8_t* nibbles, float* scales,
                                                        long long total_blocks) {
    const long long blk = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (blk >= total_blocks) return;
    const uint8_t* src = cpu_blocks + blk * 20;
    uint8_t raw[20];
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(src + 4 * i);  // blocks are 20 bytes: 4-byte aligned
        raw[4 * i] = w & 0xFF; raw[4 * i + 1] = (w >> 8) & 0xFF; raw[4 * i + 2] = (w >> 16) & 0xFF; raw[4 * i + 3] = w >> 24;
    }
    uint32_t sbits = raw[0] | (raw[1] << 8) | (raw[2] << 16) | (static_cast<uint32_t>(raw[3]) << 24);
    scales[blk] = __uint_as_float(sbits);
    uint8_t* dst = nibbles + blk * 16;
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const int h = j >> 1;
        const uint8_t ej = (j & 1) ? (raw[4 + h] >> 4) : (raw[4 + h] & 0xF);
        const uint8_t ej16 = (j & 1) ? (raw[4 + h + 8] >> 4) : (raw[4 + h + 8] & 0xF);
        dst[j] = static_cast<uint8_t>(ej | (ej16 << 4));
    }
}

// ---------------------------------------------------------------------------------------------
// Synthetic generator
// ---------------------------------------------------------------------------------------------
template <int ODT> __global__ void __launch_bounds__(256) fill_normal_kernel(void* out, long long n, unsigned long long st,
                                                                              unsigned long long first, float scale) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = __fmul_rn(gen_normal(st, first + static_cast<unsigned long long>(i)), scale);
    store_out<ODT>(out, i, v);
}

static unsigned grid_for(long long n, int block) { return static_cast<unsigned>((n + block - 1) / block); }

}  // namespace nve

using namespace nve;

extern "C" void nve_matvec_f16(const uint16_t* x, const uint16_t* W, uint16_t* out, int N, int K, nve_stream_t stream) {
    if (!x || !W || !out) { set_status(NVE_ERR_BAD_POINTER); return; }
    if (N <= 0 || K <= 0) { set_status(NVE_ERR_BAD_SHAPE); return; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool vec = (K % 8) == 0 && aligned(x, 16) && aligned(W, 16);
    const int wpb = 8;
    if (vec) matvec_f16_kernel<true><<<(N + wpb - 1) / wpb, wpb * 32, 0, st>>>(x, W, out, N, K);
    else matvec_f16_kernel<false><<<(N + wpb - 1) / wpb, wpb * 32, 0, st>>>(x, W, out, N, K);
    count_launch();
    check_launch();
}

extern "C" int nve_b200_dequant_w4a16(const uint8_t* nibbles, const float* scales, const float* awq, void* out, int N,
                                      int K, int out_dtype, nve_stream_t stream) {
    if (!nibbles || !scales || !out) return set_status(NVE_ERR_BAD_POINTER);
    if (N <= 0 || K <= 0 || (K % 32) != 0) return set_status(NVE_ERR_BAD_SHAPE);
    if (out_dtype != NVE_DT_F16 && out_dtype != NVE_DT_BF16) return set_status(NVE_ERR_BAD_DTYPE);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long blocks = static_cast<long long>(N) * (K / 32);
    uint16_t* o = static_cast<uint16_t*>(out);
    if (aligned(nibbles, 16) && aligned(out, 16)) {
        if (out_dtype == NVE_DT_F16) dequant_kernel<NVE_DT_F16><<<grid_for(blocks, 256), 256, 0, st>>>(nibbles, scales, awq, o, blocks, K / 32);
        else dequant_kernel<NVE_DT_BF16><<<grid_for(blocks, 256), 256, 0, st>>>(nibbles, scales, awq, o, blocks, K / 32);
    } else {
        const long long total = blocks * 32;
        if (out_dtype == NVE_DT_F16) dequant_scalar_kernel<NVE_DT_F16><<<grid_for(total, 256), 256, 0, st>>>(nibbles, scales, awq, o, total, K);
        else dequant_scalar_kernel<NVE_DT_BF16><<<grid_for(total, 256), 256, 0, st>>>(nibbles, scales, awq, o, total, K);
    }
    count_launch();
    return check_launch();
}

extern "C" void nve_dequant_w4a16(const uint8_t* nibbles, const float* scales, const float* awq, uint16_t* out, int N,
                                  int K, nve_stream_t stream) {
    nve_b200_dequant_w4a16(nibbles, scales, awq, out, N, K, NVE_DT_F16, stream);
}

extern "C" int nve_b200_q4_quantize(const float* W, const float* awq_scales, uint8_t* nibbles, float* scales, int N, int K,
                                    nve_stream_t stream) {
    if (!W || !nibbles || !scales) return set_status(NVE_ERR_BAD_POINTER);
    if (N <= 0 || K <= 0 || (K % 32) != 0) return set_status(NVE_ERR_BAD_SHAPE);
    if (!aligned(W, 16) || !aligned(nibbles, 16)) return set_status(NVE_ERR_BAD_ALIGNMENT);
    const long long blocks = static_cast<long long>(N) * (K / 32);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid_for(blocks, 32 * kQ4Loads));
    cfg.blockDim = dim3(256);
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    if (pdl_enabled()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    const cudaError_t e = awq_scales != nullptr ? cudaLaunchKernelEx(&cfg, q4_quantize_kernel<true>, W, awq_scales, nibbles, scales, blocks, K / 32)
                                                : cudaLaunchKernelEx(&cfg, q4_quantize_kernel<false>, W, awq_scales, nibbles, scales, blocks, K / 32);
    count_launch();
    return set_cuda_status(e);
}

extern "C" int nve_b200_q4_repack_blocks(const uint8_t* cpu_blocks, uint8_t* nibbles, float* scales, int N, int K,
                                         nve_stream_t stream) {
    if (!cpu_blocks || !nibbles || !scales) return set_status(NVE_ERR_BAD_POINTER);
    if (N <= 0 || K <= 0 || (K % 32) != 0) return set_status(NVE_ERR_BAD_SHAPE);
    if (!aligned(cpu_blocks, 4)) return set_status(NVE_ERR_BAD_ALIGNMENT);
    const long long blocks = static_cast<long long>(N) * (K / 32);
    q4_repack_kernel<<<grid_for(blocks, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(cpu_blocks, nibbles, scales, blocks);
    count_launch();
    return check_launch();
}

extern "C" int nve_b200_fill_normal(float* out, long long n, unsigned long long seed, unsigned long long stream_id,
                                    unsigned long long first, float scale, nve_stream_t stream) {
    if (!out) return set_status(NVE_ERR_BAD_POINTER);
    if (n <= 0) return set_status(NVE_ERR_BAD_SHAPE);
    fill_normal_kernel<NVE_DT_F32><<<grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        out, n, gen_state(seed, stream_id), first, scale);
    count_launch();
    return check_launch();
}

extern "C" int nve_b200_fill_normal_16(void* out, long long n, unsigned long long seed, unsigned long long stream_id,
                                       unsigned long long first, float scale, int dtype, nve_stream_t stream) {
    if (!out) return set_status(NVE_ERR_BAD_POINTER);
    if (n <= 0) return set_status(NVE_ERR_BAD_SHAPE);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned long long s = gen_state(seed, stream_id);
    if (dtype == NVE_DT_F16) fill_normal_kernel<NVE_DT_F16><<<grid_for(n, 256), 256, 0, st>>>(out, n, s, first, scale);
    else if (dtype == NVE_DT_BF16) fill_normal_kernel<NVE_DT_BF16><<<grid_for(n, 256), 256, 0, st>>>(out, n, s, first, scale);
    else return set_status(NVE_ERR_BAD_DTYPE);
    count_launch();
    return check_launch();
}
