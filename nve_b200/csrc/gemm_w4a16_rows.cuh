// W4A16 GEMM for up to eight rows of X: weights straight from HBM into registers.  Included by gemm_w4a16_pair.cu, whose
// finishing kernels it shares.
//
// With so few rows the two-SM kernel's fixed costs (cluster start, TMEM, operand rings, the drain of a tile) are a large part of
// a call.  Here a warp streams 16 weight rows like a decode GEMV does -- 16 bytes (a block of 32) per lane and row, kRowsDepth
// units ahead, the first of them before the grid dependency resolves -- and multiplies them by mma.sync (m16n8k16).  The four
// GEMMs of a layer with 7 rows, us: 1B 41.4 -> 36, 3B 50.0 -> 44.7, 8B 69.3 -> 66 (not the largest matrices: 8B gate/up and down take
// 27.3 and 16.6 here with 8 rows, 24.2 and 15.2 there with 16); with more rows than fill one mma (15: 74 against
// 70) the multiplications no longer hide behind the weights.  What is left is the dequantisation (two thirds of the issue
// slots), the weights' latency and the two launches.  Taken back: two CTAs per SM (small matrices 1 to 2 us slower), more units
// in flight with them (slower still).
//
//   unit  = 128 elements of K x 256 weight rows, 16 rows per warp; tile = SB units
//   run   = U consecutive units of the (tile, unit) sequence, one per CTA (one CTA per SM), inside at most two tiles
//
// A contraction may take K in any order that both operands share: lane 4g + c holds the whole block c of the unit for rows g and
// g + 8, so that step i of four multiplies the elements {4i .. 4i+3} and {16+4i .. 16+4i+3} of four different blocks, one raw
// word per row.  X is staged once per run in the order in which the lanes read it: 16 bytes per lane and step, no bank conflicts.
//
// Every segment of a run goes to the workspace in f32; the finishing kernel sums the segments of a tile in ascending K order.
#pragma once

#include "gemm_w4a16.cuh"

namespace nve {

constexpr int kRowsMax = 8;           // rows of X
constexpr int kRowsThreads = 512;
constexpr int kRowsDepth = 4;         // units of weights in flight per warp
constexpr int kRowsSmemMax = 200 * 1024;
constexpr int kRowsSlab = 2048;       // bytes of X per unit

__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int XDT, bool SILU>
__global__ void __launch_bounds__(kRowsThreads, 1) gemm_w4a16_rows_kernel(const PairParams p, const uint16_t* X) {
    extern __shared__ __align__(16) unsigned char rows_x[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int half_k = p.K / 2;
    const int u0 = static_cast<int>(blockIdx.x) * p.U;
    const int n_units = min(p.U, p.total - u0);
    const int tile0 = u0 / p.SB, k0 = u0 - tile0 * p.SB;
    const int n_first = min(n_units, p.SB - k0);  // units in the first of at most two tiles

    // ---- weights of this lane: rows g and g + 8 of the warp's sixteen, in one tile and then the next
    const uint8_t *nib_a, *nib_b;
    const float *sc_a, *sc_b;
    auto set_tile = [&](int tile) {
        const PairTile t = pair_locate<SILU ? kPairSilu : kPairPlain>(p, tile);
        // SILU: columns 0-63 and 128-191 of a tile are gate rows, the others the up rows of the same indices
        const int mi = SILU ? (warp >> 2) & 1 : t.mi;
        const int row = t.n0 + (SILU ? (warp >> 3) * 64 + (warp & 3) * 16 : warp * 16) + g, last = p.Nm[mi] - 1;
        const int ra = min(row, last), rb = min(row + 8, last);  // rows past the end repeat the last one; nobody reads their sums
        nib_a = p.nib[mi] + static_cast<long long>(ra) * half_k + c * 16;
        nib_b = p.nib[mi] + static_cast<long long>(rb) * half_k + c * 16;
        sc_a = p.sc[mi] + static_cast<long long>(ra) * p.nb + c;
        sc_b = p.sc[mi] + static_cast<long long>(rb) * p.nb + c;
    };
    uint4 wa[kRowsDepth], wb[kRowsDepth];
    float sa[kRowsDepth], sb[kRowsDepth];
    int lj = 0, lk = k0;  // next unit to load: index in the run and in its tile
    auto load = [&](uint4& a, uint4& b, float& xa, float& xb) {
        if (lj < n_units) {
            if (4 * lk + c < p.nb) {
                a = ld_stream_u4(nib_a + static_cast<long long>(lk) * 64);
                b = ld_stream_u4(nib_b + static_cast<long long>(lk) * 64);
                xa = __ldg(sc_a + 4 * lk);
                xb = __ldg(sc_b + 4 * lk);  // cached: a line holds the scales of eight units
            } else {  // past the end of K (a multiple of 64)
                a = b = make_uint4(0, 0, 0, 0);
                xa = xb = 0.0f;
            }
            lj++;
            if (++lk == p.SB) {
                lk = 0;
                if (lj < n_units) set_tile(tile0 + 1);
            }
        }
    };
    set_tile(tile0);
#pragma unroll
    for (int d = 0; d < kRowsDepth; d++) load(wa[d], wb[d], sa[d], sb[d]);

    // ---- X of the run's units (unit j of the run in slab j): [unit][step i][lane][16 bytes]
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t sx = s_addr(rows_x);
    constexpr int kPieces = 128;  // 16-byte chunks of X per unit: 8 rows x 16
    const int pieces = n_units * kPieces;
#pragma unroll 4
    for (int i = tid; i < pieces; i += kRowsThreads) {
        const int j = i / kPieces, q = i - j * kPieces;
        const int m = q >> 4, ch = q & 15;  // row of X, chunk: elements 8 ch .. 8 ch + 7 of the unit
        int ku = k0 + j;
        if (ku >= p.SB) ku -= p.SB;
        const int e = ku * 128 + ch * 8;
        const bool in = m < p.M && e < p.K;
        const uint16_t* src = X + (in ? static_cast<long long>(m) * p.K + e : 0);
        // chunk ch = block ch >> 2, quarter ch & 3: elements 4i .. 4i + 7 of the low (quarters 0, 1) or high half of the block
        const uint32_t dst = sx + static_cast<uint32_t>(j * kRowsSlab + (ch & 1) * 2 * 512 + (m * 4 + (ch >> 2)) * 16 + ((ch >> 1) & 1) * 8);
        if constexpr (XDT == NVE_DT_F16) {
            const int have = in ? 8 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(have) : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + 512), "l"(src + 4), "r"(have) : "memory");
        } else {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (in) v = *reinterpret_cast<const uint4*>(src);
            asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(dst), "r"(bf16x2_to_f16x2(v.x)), "r"(bf16x2_to_f16x2(v.y)) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(dst + 512), "r"(bf16x2_to_f16x2(v.z)), "r"(bf16x2_to_f16x2(v.w)) : "memory");
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // ---- units
    const DequantConsts dc = make_dequant_consts();
    float acc[4] = {};
    int done = 0;  // units multiplied
    auto flush = [&](int tile) {
        float* part = p.partial + static_cast<long long>(static_cast<int>(blockIdx.x) + tile) * p.part_rows * kPairTile + warp * 16 + g;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int m = 2 * c + (e & 1);
            if (m < p.M) part[m * kPairTile + (e >> 1) * 8] = acc[e];
            acc[e] = 0.0f;
        }
    };
    auto unit = [&](const uint4& a, const uint4& b, float xa, float xb) {
        const DequantScale da = make_dequant_scale(xa), db = make_dequant_scale(xb);
        const uint32_t xs = sx + static_cast<uint32_t>(done * kRowsSlab + lane * 16);
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t al0, al1, ah0, ah1, bl0, bl1, bh0, bh1;
            dequant_word(aw[i], da, dc, al0, al1, ah0, ah1);
            dequant_word(bw[i], db, dc, bl0, bl1, bh0, bh1);
            uint4 x;
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(xs + i * 512));
            mma_f16(acc, al0, bl0, al1, bl1, x.x, x.y);
            mma_f16(acc, ah0, bh0, ah1, bh1, x.z, x.w);
        }
        if (++done == n_first) flush(tile0);
    };
    for (int j = 0; j < n_units; j += kRowsDepth) {
#pragma unroll
        for (int d = 0; d < kRowsDepth; d++) {
            if (j + d < n_units) {
                const uint4 a = wa[d], b = wb[d];
                const float xa = sa[d], xb = sb[d];
                load(wa[d], wb[d], sa[d], sb[d]);
                unit(a, b, xa, xb);
            }
        }
    }
    if (done > n_first) flush(tile0 + 1);
}

// How a call is cut: equal runs, one per SM, of at least two units, inside at most two tiles; grid == 0 when this kernel is not
// the one to take: too many rows, so many weight rows that a CTA has whole tiles, or X of a run larger than shared memory.
struct RowsPlan {
    int grid = 0, SB = 0, U = 0, total = 0, tiles = 0;
    size_t smem = 0, partial_bytes = 0;
};
static RowsPlan rows_plan(const int* Ns, int num_mats, int M, int K, bool silu) {
    RowsPlan r;
    if (M > kRowsMax) return r;
    long long tiles = 0;
    if (silu) tiles = (Ns[0] + kPairTile / 2 - 1) / (kPairTile / 2);
    else
        for (int i = 0; i < num_mats; i++) tiles += (Ns[i] + kPairTile - 1) / kPairTile;
    r.SB = (K + 127) / 128;
    const long long total = tiles * r.SB;
    const int sm = max(1, sm_count());
    long long U = (total + sm - 1) / sm;
    if (U < 2) U = r.SB < 2 ? r.SB : 2;
    if (U > r.SB) return r;
    r.smem = static_cast<size_t>(U) * kRowsSlab;
    if (r.smem > static_cast<size_t>(kRowsSmemMax)) return r;
    r.U = static_cast<int>(U);
    r.total = static_cast<int>(total);
    r.tiles = static_cast<int>(tiles);
    r.grid = static_cast<int>((total + U - 1) / U);
    // segment (CTA, tile) has number CTA + tile: no two segments of the sequence share it
    r.partial_bytes = static_cast<size_t>(r.grid + r.tiles - 1) * M * kPairTile * sizeof(float);
    return r;
}

template <int XDT, bool SILU> static int launch_rows(const PairParams& p, const RowsPlan& r, const uint16_t* X, cudaStream_t st) {
    auto kern = gemm_w4a16_rows_kernel<XDT, SILU>;
    if (int s = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kRowsSmemMax); s != NVE_OK) return s;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(r.grid));
    cfg.blockDim = dim3(kRowsThreads);
    cfg.dynamicSmemBytes = r.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (pdl_enabled()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p, X);
    count_launch();
    return set_cuda_status(e);
}
}  // namespace nve
