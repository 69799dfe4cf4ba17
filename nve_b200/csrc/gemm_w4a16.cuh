// The batched W4A16 GEMM: nibble dequantisation and the interface between its entry points (gemm_w4a16.cu) and its
// kernel (gemm_w4a16_pair.cu).
#pragma once

#include "common.cuh"

namespace nve {

__device__ __forceinline__ uint32_t s_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// bf16 -> f16 of two elements.  Exact for 6.1e-5 <= |x| <= 65504 (every bf16 significand fits f16); larger magnitudes saturate to
// +-65504, smaller ones round into the f16 subnormal range.
__device__ __forceinline__ uint32_t bf16x2_to_f16x2(uint32_t w) {
    const float lo = fminf(fmaxf(__uint_as_float(w << 16), -65504.0f), 65504.0f);
    const float hi = fminf(fmaxf(__uint_as_float(w & 0xFFFF0000u), -65504.0f), 65504.0f);
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Dequantisation of two nibbles.  0x6400 is 1024.0 in f16 with one ulp = 1, so OR-ing a nibble into mantissa bits
// 0-3 gives 1024 + q exactly; 0x5400 is 64.0 with one ulp = 1/16, so a nibble left in place at bits 4-7 gives
// 64 + q exactly (no shift needed).  Subtracting 1032 (72) gives q - 8 exactly, and one multiply by the f16 scale
// rounds once.  (A single-FMA form needs 1.5 * scale to be exact, which costs two bits of scale precision --
// measured at 9e-3 of the output RMS, too close to the tolerance -- so it is not used.)
struct DequantScale {
    uint32_t mul2;  // half2(s, s)
};
__device__ __forceinline__ DequantScale make_dequant_scale(float scale) {
    const __half2 m = __float2half2_rn(scale);
    DequantScale d;
    d.mul2 = *reinterpret_cast<const uint32_t*>(&m);
    return d;
}
// Masks, magic numbers and offsets live in registers that the optimiser cannot see through: with literal
// constants the compiler emitted two LOP3 per pair (one immediate per instruction); (w & mask) | magic is a
// single LOP3 when all three operands are registers.
struct DequantConsts {
    uint32_t mask_lo, magic_lo, off_lo, mask_hi, magic_hi, off_hi;
};
__device__ __forceinline__ DequantConsts make_dequant_consts() {
    DequantConsts c;
    asm volatile("mov.b32 %0, 0x000F000F;" : "=r"(c.mask_lo));
    asm volatile("mov.b32 %0, 0x64006400;" : "=r"(c.magic_lo));
    asm volatile("mov.b32 %0, 0x64086408;" : "=r"(c.off_lo));   // 1032
    asm volatile("mov.b32 %0, 0x00F000F0;" : "=r"(c.mask_hi));
    asm volatile("mov.b32 %0, 0x54005400;" : "=r"(c.magic_hi));
    asm volatile("mov.b32 %0, 0x54805480;" : "=r"(c.off_hi));   // 72
    return c;
}
template <bool HIGH> __device__ __forceinline__ uint32_t dequant_pair(uint32_t w, const DequantScale& d, const DequantConsts& c) {
    uint32_t bits;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(bits) : "r"(w), "r"(HIGH ? c.mask_hi : c.mask_lo), "r"(HIGH ? c.magic_hi : c.magic_lo));
    const uint32_t off = HIGH ? c.off_hi : c.off_lo;
    __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&bits), *reinterpret_cast<const __half2*>(&off));
    v = __hmul2(v, *reinterpret_cast<const __half2*>(&d.mul2));
    return *reinterpret_cast<const uint32_t*>(&v);
}

// One raw word (4 bytes = elements j..j+3 in the low nibbles, j+16..j+19 in the high nibbles) -> pairs in natural
// order: lo0 = (e_j, e_j+1), lo1 = (e_j+2, e_j+3), hi0 = (e_j+16, e_j+17), hi1 = (e_j+18, e_j+19).  One byte
// permute per word ([b0,b2,b1,b3]) puts the two elements of every pair 16 bits apart, where a half2 wants them.
__device__ __forceinline__ void dequant_word(uint32_t w, const DequantScale& d, const DequantConsts& c, uint32_t& lo0,
                                             uint32_t& lo1, uint32_t& hi0, uint32_t& hi1) {
    const uint32_t u = __byte_perm(w, 0, 0x3120);
    const uint32_t t = u >> 8;
    lo0 = dequant_pair<false>(u, d, c);  // b0 low nibble, b1 low nibble
    hi0 = dequant_pair<true>(u, d, c);   // b0 high, b1 high
    lo1 = dequant_pair<false>(t, d, c);  // b2 low, b3 low
    hi1 = dequant_pair<true>(t, d, c);   // b2 high, b3 high
}

// Rows of X that fill one mma column.  Up to here the kernel for few rows takes every call whose partial tiles the workspace holds, and bf16
// rows need no room for an f16 copy; from 9 to 16 it leaves some to the two-SM kernel.
constexpr int kFewRows = 8;

// The two-SM tcgen05 kernel (gemm_w4a16_pair.cu): any number of rows of X (f16), up to three matrices side by side.
struct PairMat {
    const uint8_t* nib;
    const float* sc;
    void* Y;
    int N;
};
struct PairPlan {
    int NB, XT, SB;        // rows of X per tile, X tiles, units (256 elements of K) per tile
    long long tiles, U, grid_pairs;
    size_t partial_bytes;  // workspace for partial tiles, 0 when every run consists of whole tiles
};
// Rotary embedding of the products of q and k (in place / into the cache), v into the cache; row s of X is position start_pos + s
struct PairRope {
    uint16_t *k_cache, *v_cache;
    const uint16_t *cos_t, *sin_t;
    int start_pos, hd, max_seq;
};
// Where a product that was left unfinished lies (rows of X in one tile): of tiles that were cut the f32 sums of their segments, of others Y.
struct PairLeft {
    const float* partial = nullptr;  // nullptr: everything is in Y
    int part_rows = 0, SB = 0, U = 0, by_tile = 0;
    int tile0[3] = {0, 0, 0};        // first tile of a matrix
};
// What becomes of the product (f16 outputs only; nothing set: Y = X . W^T)
struct PairFinish {
    const uint16_t* res = nullptr;     // one matrix: Y = res + round16(product)
    const uint16_t* norm_w = nullptr;  // with res: also normed = RMSNorm(Y) with this weight (pair_norm_fits)
    uint16_t* normed = nullptr;
    float eps = 0.0f;
    const PairRope* rope = nullptr;    // three matrices q, k, v of whole heads; the cache is written, the outputs of k and v are scratch
    PairLeft* left = nullptr;          // no finishing launch: the caller's next kernel sums the segments (PairFeatures)
    bool silu = false;                 // two matrices of the same N: Y of the first = silu(first product) * second product
};
PairPlan pair_plan(const int* Ns, int num_mats, int M, int K, bool have_scratch, size_t avail, bool silu = false);
// Workspace that a call of these sizes can use, whichever kernel takes it
size_t rows_partial_bytes(const int* Ns, int num_mats, int M, int K, bool silu);
inline size_t gemm_partial_bytes(const int* Ns, int num_mats, int M, int K, bool silu = false) {
    const size_t a = pair_plan(Ns, num_mats, M, K, true, ~static_cast<size_t>(0), silu).partial_bytes, b = rows_partial_bytes(Ns, num_mats, M, K, silu);
    return a > b ? a : b;
}
int gemm_pair(const uint16_t* X, const PairMat* mats, int num_mats, int y_dtype, int M, int K, void* partial, size_t avail, cudaStream_t st,
              const PairFinish& fin = PairFinish());
// The kernel for few rows (gemm_w4a16_rows.cuh), X in f16 or bf16; false: not its sizes, or a workspace too small, and nothing was
// launched.  gemm_pair asks it first.
bool gemm_rows_try(const void* X, int x_dtype, const PairMat* mats, int num_mats, int y_dtype, int M, int K, void* partial, size_t avail,
                   cudaStream_t st, const PairFinish& fin, int* status);
// q, k and v of `M` rows of X (f16), left unfinished where `left` is given and the rows are one tile; the entry point's checks
int gemm_qkv(const uint16_t* X, const nve_b200_w4_matrix* mats, int M, int K, void* scratch, size_t scratch_bytes, PairLeft* left, cudaStream_t st);
bool pair_norm_fits(int N);
#ifdef __CUDACC__
// E features of row m of a product that was left unfinished, rounded to f16: element e is feature n of the matrix whose tiles begin at
// tile0 and whose finished values are at y.  Found before the grid dependency; the segments of all E are then under way together, eight at a
// time, and added in ascending K order like the finishing kernel does; behind() runs when the first are under way.
template <int E> struct PairFeatures {
    const float* src[E];  // segment i of count[e] is `delta` further than i - 1; where `late` has bit e, the first is one slot further
    int count[E];         // 0: finished
    unsigned late = 0;
    int most = 0;
    long long delta, slot;
    __device__ __forceinline__ void find(const PairLeft& L, int m, const int (&tile0)[E], const int (&n)[E]) {
        slot = static_cast<long long>(L.part_rows) * 256;
        delta = L.by_tile ? slot : 2 * slot;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int tile = tile0[e] + (n[e] >> 8), first = tile * L.SB / L.U;
            count[e] = ((tile + 1) * L.SB - 1) / L.U - first + 1;
            if (count[e] == 1 && !L.by_tile) count[e] = 0;
            most = max(most, count[e]);
            src[e] = L.partial + static_cast<long long>(L.by_tile ? first + tile : 2 * first) * slot + static_cast<long long>(m) * 256 + (n[e] & 255);
            if (!L.by_tile && first * L.U < tile * L.SB) late |= 1u << e;
        }
    }
    template <class F> __device__ __forceinline__ void sum(const uint16_t* const (&y)[E], uint16_t (&out)[E], F behind) {
        constexpr int kFly = E > 8 ? 4 : 8;  // registers (64 sequences of 300, 56 over 8 heads of 128: 75.2 -> 73.7 us a layer)
        float total[E];
        for (int c0 = 0; c0 == 0 || c0 < most; c0 += kFly) {
            float v[kFly][E];
#pragma unroll
            for (int i = 0; i < kFly; i++)
#pragma unroll
                for (int e = 0; e < E; e++)
                    if (c0 + i < count[e]) v[i][e] = __ldcg(src[e] + (c0 + i) * delta + (i == 0 && c0 == 0 && (late >> e & 1) ? slot : 0));
            if (c0 == 0) {
#pragma unroll
                for (int e = 0; e < E; e++)
                    if (count[e] == 0) out[e] = *y[e];
                behind();
            }
#pragma unroll
            for (int i = 0; i < kFly; i++)
#pragma unroll
                for (int e = 0; e < E; e++)
                    if (c0 + i < count[e]) total[e] = c0 + i == 0 ? v[i][e] : __fadd_rn(total[e], v[i][e]);
        }
#pragma unroll
        for (int e = 0; e < E; e++)
            if (count[e] > 0) out[e] = Act16<NVE_DT_F16>::from_f32(total[e]);
    }
};
#endif
int gemm_pair_error(bool reset);

}  // namespace nve
