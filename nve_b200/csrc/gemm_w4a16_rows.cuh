// W4A16 GEMM for up to sixteen rows of X: weights through a ring of shared memory per warp, mma.sync.  Included by
// gemm_w4a16_pair.cu, whose finishing kernels it shares.
//
// With so few rows the two-SM kernel's fixed costs (cluster start, TMEM, operand rings, the drain of a tile) are a large part of
// a call.  Here a warp streams sixteen weight rows and multiplies them by mma.sync (m16n8k16), one mma per eight rows of X.
//
// What bounds it: how the weights come in, then their dequantisation.  A 28672 x 4096 matrix (HBM floor 11.2 us) without launch, X and
// the rest of the kernel: 16-byte loads straight into registers, eight rows x 64 bytes and eight x 16 bytes of scales per
// instruction, the former form: 19.8 us with nothing else, 24.4 with dequantisation and mma (more loads in flight change nothing: the SM takes
// the 32 short pieces one by one).  The same through cp.async, whole 128-byte lines: 11.8 and 14.4 us; arithmetic alone 11.8.  32-byte
// loads into registers 14.2 and 19.  cp.async.bulk takes some 55 cycles per copy: only pieces of 2 KB and more keep up with HBM.
// Two units of a ring ahead are enough; a third costs shared memory that X needs (and a ring with more stages than the run has units, time).
//
// The four GEMMs of a layer in turn, us (before: weights into registers up to 8 rows, the two-SM kernel above): 8B 59.6 -> 46.6 with 2 rows,
// 61.1 -> 48.4 with 8, 61.6 -> 57.6 with 16; 3B 36.4 -> 34.0 with 8, 42.9 -> 39.1 with 16; 1B 27.5 -> 26.3 and 35.9 -> 30.2.  Matrices with
// more tiles than SMs: 40000 x 4096 30.3 -> 23.7 with one row, 31.0 -> 29.7 with 16; 128256 x 4096 82 -> 61 and 87.5 -> 78.9; 57344 x 8192 72 ->
// 57 and 73.3 -> 74.0.  Sixteen rows are the most: with 24 the mma rate (an SM takes
// three cycles for one) is what bounds it, 66.3 against 63.3 in the two-SM kernel (8B), 47.3 against 43.8 (3B).
//
//   unit  = 256 elements of K x 256 weight rows, 16 rows per warp; tile = SB units
//   run   = U consecutive units of the (tile, unit) sequence, one per CTA (one CTA per SM)
//
// A contraction may take K in any order that both operands share: lane 4g + c holds the blocks 2c and 2c + 1 of the unit for rows g
// and g + 8, so that a step multiplies the elements {4i .. 4i+3} and {16+4i .. 16+4i+3} of four different blocks, one raw word per row.
// X is staged once per run in the order in which the lanes read it: 16 bytes per lane and step, no bank conflicts.
//
// Sums: an MMA rounds its accumulator towards zero, so that the error of a sum grows with the length of its chain.  A chain is eight MMAs long
// and added to the sum with a rounding to nearest: sums are 1.7e-7 to 2.5e-7 of the result off (against 64 bits).  One chain for a whole
// run: 3.3e-7 at 512 x 2048, 6.4e-7 at 4096 x 4096, 2.1e-6 at 4096 x 14336, where the two-SM kernel with its shorter ones has
// 2.7e-7, 4.5e-7 and 1.3e-6 (16 rows).  It costs 1 to 2 %.
//
// Every segment of a run goes to the workspace in f32; the finishing kernel sums the segments of a tile in ascending K order.
#pragma once

#include "gemm_w4a16.cuh"

namespace nve {

constexpr int kRowsMax = 16;                       // rows of X
constexpr int kRowsThreads = 512;
constexpr int kRowsStage = 16 * (128 + 32);        // a unit of a warp: 16 rows x (256 nibbles, 8 scales)
constexpr int kRowsSlab = 4096;                    // bytes of X per unit and eight rows
constexpr int kRowsSmemMax = 226 * 1024;

__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the first of a chain
__device__ __forceinline__ void mma_f16_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}

// NT: eights of rows of X, D: units in a warp's ring, all but one of them requested ahead (D = 1: a run of one unit)
template <int XDT, bool SILU, int NT, int D>
__global__ void __launch_bounds__(kRowsThreads, 1) gemm_w4a16_rows_kernel(const PairParams p, const uint16_t* X) {
    extern __shared__ __align__(128) unsigned char rows_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int u0 = static_cast<int>(blockIdx.x) * p.U;
    const int n_units = min(p.U, p.total - u0);
    const int tile0 = u0 / p.SB, k0 = u0 - tile0 * p.SB;
    const uint32_t ring = s_addr(rows_smem) + static_cast<uint32_t>(warp * D * kRowsStage), sx = s_addr(rows_smem) + 16 * D * kRowsStage;

    // ---- weights: a lane copies 16-byte chunk lane & 7 of the rows (lane >> 3) + 4 i, and half of the scales of row lane >> 1
    const uint8_t* np[4];
    const float* sp;
    int lj = 0, lk = k0, lt = tile0;  // next unit to load: index in the run, in its tile, tile
    auto set_tile = [&]() {
        const PairTile t = pair_locate<SILU ? kPairSilu : kPairPlain>(p, lt);
        // SILU: columns 0-63 and 128-191 of a tile are gate rows, the others the up rows of the same indices
        const int mi = SILU ? (warp >> 2) & 1 : t.mi;
        const int row0 = t.n0 + (SILU ? (warp >> 3) * 64 + (warp & 3) * 16 : warp * 16), last = p.Nm[mi] - 1;
        // rows past the end repeat the last one; nobody reads their sums
#pragma unroll
        for (int i = 0; i < 4; i++)
            np[i] = p.nib[mi] + static_cast<long long>(min(row0 + (lane >> 3) + 4 * i, last)) * (p.K / 2) + (lane & 7) * 16;
        sp = p.sc[mi] + static_cast<long long>(min(row0 + (lane >> 1), last)) * p.nb + (lane & 1) * 4;
    };
    // odd rows have neighbouring chunks swapped: two rows that are read together then fall into different banks
    const uint32_t nd = static_cast<uint32_t>((lane >> 3) * 128 + (((lane & 7) ^ ((lane >> 3) & 1)) << 4)), sd = 2048 + lane * 16;
    auto load = [&](int slot) {
        if (lj < n_units) {
            const uint32_t dst = ring + static_cast<uint32_t>(slot * kRowsStage);
            const bool in = 8 * lk + (lane & 7) < p.nb;  // past the end of K (a multiple of 64): zeros
#pragma unroll
            for (int i = 0; i < 4; i++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + nd + i * 512), "l"(np[i] + (in ? lk * 128 : 0)), "r"(in ? 16 : 0) : "memory");
            const int left = p.nb - 8 * lk - (lane & 1) * 4;
            const float* sc = sp + 8 * lk;
            if (p.sc16) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + sd), "l"(left > 0 ? sc : sp), "r"(left > 0 ? 16 : 0) : "memory");
            } else {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + sd), "l"(left > 0 ? sc : sp), "r"(left > 0 ? 8 : 0) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + sd + 8), "l"(left > 2 ? sc + 2 : sp), "r"(left > 2 ? 8 : 0) : "memory");
            }
            lj++;
            if (++lk == p.SB) {
                lk = 0;
                lt++;
                if (lj < n_units) set_tile();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    set_tile();
#pragma unroll
    for (int d = 0; d < (D == 1 ? 1 : D - 1); d++) load(d);

    // ---- X of the run's units (a run longer than a tile comes back to the same ones): [unit][step][eight rows][lane][16 bytes]; of lane
    // (row, c) and step 4 h + i the elements 4i .. 4i + 3 and 16 + 4i .. of block 2c + h, both in the order 0 2 1 3 in which the
    // nibbles of a word come out
    pdl_wait();
    pdl_launch_dependents();
    {
        // A thread keeps its chunk of 16 bytes and its row from one unit to the next.  Two loads on their way at a time: eight made calls of
        // a unit or two 3 to 5 % slower (their code is fetched by every launch), one the long ones 3 %.
        constexpr int kStep = kRowsThreads / (NT * 256), kFly = 2;
        const int q = tid & 31, r = (tid >> 5) & 7, nt = NT == 1 ? 0 : (tid >> 8) & 1, m = nt * 8 + r;
        const int n = min(n_units, p.SB), left = m < p.M ? p.K - q * 8 : 0;  // elements of the row from this chunk of unit 0 on
        const uint16_t* src = X + static_cast<long long>(m) * p.K + q * 8;
        // block q >> 2, quarter q & 3
        const uint32_t dst = sx + static_cast<uint32_t>(((((q >> 2) & 1) * 4 + (q & 1) * 2) * NT + nt) * 512 + (r * 4 + (q >> 3)) * 16 + ((q >> 1) & 1) * 8);
        for (int u = NT == 1 ? tid >> 8 : 0; u < n; u += kFly * kStep) {
            uint4 v[kFly];
#pragma unroll
            for (int j = 0; j < kFly; j++) {
                const int ul = u + j * kStep, ku = k0 + ul - (k0 + ul >= p.SB ? p.SB : 0);
                v[j] = make_uint4(0, 0, 0, 0);
                if (ul < n && ku * 256 < left) v[j] = *reinterpret_cast<const uint4*>(src + ku * 256);
            }
#pragma unroll
            for (int j = 0; j < kFly; j++) {
                const int ul = u + j * kStep;
                if (ul >= n) break;
                uint4 w = v[j];
                if (XDT == NVE_DT_BF16) w = make_uint4(bf16x2_to_f16x2(w.x), bf16x2_to_f16x2(w.y), bf16x2_to_f16x2(w.z), bf16x2_to_f16x2(w.w));
                const uint32_t d = dst + static_cast<uint32_t>(ul) * (kRowsSlab * NT);
                asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(d), "r"(__byte_perm(w.x, w.y, 0x5410)), "r"(__byte_perm(w.x, w.y, 0x7632)) : "memory");
                asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(d + NT * 512), "r"(__byte_perm(w.z, w.w, 0x5410)), "r"(__byte_perm(w.z, w.w, 0x7632)) : "memory");
            }
        }
    }
    __syncthreads();

    // ---- units
    const DequantConsts dc = make_dequant_consts();
    float acc[NT][4] = {};
    int slot = 0, slab = 0, tile = tile0, k = k0;
    for (int j = 0; j < n_units; j++) {
        if (D > 1) load(slot == 0 ? D - 1 : slot - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
        __syncwarp();
        const uint32_t st = ring + static_cast<uint32_t>(slot * kRowsStage), xs = sx + static_cast<uint32_t>(slab * (kRowsSlab * NT) + lane * 16);
        float2 s[2];
#pragma unroll
        for (int r = 0; r < 2; r++) asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(s[r].x), "=f"(s[r].y) : "r"(st + 2048 + (g + 8 * r) * 32 + c * 8));
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint4 w[2];
#pragma unroll
            for (int r = 0; r < 2; r++)
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[r].x), "=r"(w[r].y), "=r"(w[r].z), "=r"(w[r].w) : "r"(st + (g + 8 * r) * 128 + (((2 * c + h) ^ (g & 1)) << 4)));
            const DequantScale da = make_dequant_scale(h ? s[0].y : s[0].x), db = make_dequant_scale(h ? s[1].y : s[1].x);
            const uint32_t aw[4] = {w[0].x, w[0].y, w[0].z, w[0].w}, bw[4] = {w[1].x, w[1].y, w[1].z, w[1].w};
            float chain[NT][4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t va = aw[i] >> 8, vb = bw[i] >> 8;
                const uint32_t l0 = dequant_pair<false>(aw[i], da, dc), l1 = dequant_pair<false>(bw[i], db, dc), l2 = dequant_pair<false>(va, da, dc),
                               l3 = dequant_pair<false>(vb, db, dc);
                const uint32_t h0 = dequant_pair<true>(aw[i], da, dc), h1 = dequant_pair<true>(bw[i], db, dc), h2 = dequant_pair<true>(va, da, dc),
                               h3 = dequant_pair<true>(vb, db, dc);
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    uint4 x;
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(xs + ((h * 4 + i) * NT + nt) * 512));
                    if (i == 0) mma_f16_zero(chain[nt], l0, l1, l2, l3, x.x, x.y);
                    else mma_f16(chain[nt], l0, l1, l2, l3, x.x, x.y);
                    mma_f16(chain[nt], h0, h1, h2, h3, x.z, x.w);
                }
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[nt][e] = __fadd_rn(acc[nt][e], chain[nt][e]);
        }
        __syncwarp();  // the stage is free
        if (++slot == D) slot = 0;
        if (++slab == p.SB) slab = 0;
        if (++k == p.SB || j + 1 == n_units) {  // end of the segment
            float* part = p.partial + static_cast<long long>(static_cast<int>(blockIdx.x) + tile) * p.part_rows * kPairTile + warp * 16 + g;
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int m = nt * 8 + 2 * c + (e & 1);
                    if (m < p.M) part[m * kPairTile + (e >> 1) * 8] = acc[nt][e];
                    acc[nt][e] = 0.0f;
                }
            k = 0;
            tile++;
        }
    }
}

// How a call is cut: equal runs, at most one per SM; grid == 0 when this kernel is not the one to take: too many rows, or X of a run larger
// than shared memory.
struct RowsPlan {
    int grid = 0, SB = 0, U = 0, total = 0, tiles = 0, nt = 0, depth = 0;
    size_t smem = 0, partial_bytes = 0;
};
static RowsPlan rows_plan(const int* Ns, int num_mats, int M, int K, bool silu) {
    RowsPlan r;
    if (M > kRowsMax) return r;
    long long tiles = 0;
    if (silu) tiles = (Ns[0] + kPairTile / 2 - 1) / (kPairTile / 2);
    else
        for (int i = 0; i < num_mats; i++) tiles += (Ns[i] + kPairTile - 1) / kPairTile;
    r.SB = (K + 255) / 256;
    const long long total = tiles * r.SB;
    if (total > 0x3FFFFFFFll) return r;
    const int sm = max(1, sm_count());
    // A tile in many segments costs the finish more than a second unit costs the run: 512 x 14336 (56 units a tile), 8 rows, 9.0 us in runs of one,
    // 7.7 of two, 16 rows 9.4 and 8.2; 28 units 6.2 and 6.1; 16 units 4.9 and 5.4.
    const long long U = std::max((total + sm - 1) / sm, r.SB >= 28 ? 2ll : 1ll);
    r.nt = (M + kFewRows - 1) / kFewRows;
    const size_t x = static_cast<size_t>(std::min<long long>(U, r.SB)) * r.nt * kRowsSlab;
    // No more stages than units: 37888 x 512 (runs of two units, 8 rows) 7.3 us with three stages, 6.9 with two; 3072 x 3072 (one unit) 6.9
    // with two, 5.6 with one.
    const int most = static_cast<int>(std::min<long long>(U, 3)), least = std::min(most, 2);
    for (r.depth = most; r.depth >= least; r.depth--) {
        r.smem = x + static_cast<size_t>(16) * r.depth * kRowsStage;
        if (r.smem <= static_cast<size_t>(kRowsSmemMax)) break;
    }
    if (r.depth < least) return r;
    r.U = static_cast<int>(U);
    r.total = static_cast<int>(total);
    r.tiles = static_cast<int>(tiles);
    r.grid = static_cast<int>((total + U - 1) / U);
    // segment (CTA, tile) has number CTA + tile: no two segments of the sequence share it
    r.partial_bytes = static_cast<size_t>(r.grid + r.tiles - 1) * M * kPairTile * sizeof(float);
    return r;
}

template <int XDT, bool SILU, int NT, int D> static int launch_rows_as(const PairParams& p, const RowsPlan& r, const uint16_t* X, cudaStream_t st) {
    auto kern = gemm_w4a16_rows_kernel<XDT, SILU, NT, D>;
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
template <int XDT, bool SILU> static int launch_rows(const PairParams& p, const RowsPlan& r, const uint16_t* X, cudaStream_t st) {
    using Launch = int (*)(const PairParams&, const RowsPlan&, const uint16_t*, cudaStream_t);
    static constexpr Launch by_depth[2][3] = {{launch_rows_as<XDT, SILU, 1, 1>, launch_rows_as<XDT, SILU, 1, 2>, launch_rows_as<XDT, SILU, 1, 3>},
                                              {launch_rows_as<XDT, SILU, 2, 1>, launch_rows_as<XDT, SILU, 2, 2>, launch_rows_as<XDT, SILU, 2, 3>}};
    return by_depth[r.nt - 1][r.depth - 1](p, r, X, st);
}
}  // namespace nve
