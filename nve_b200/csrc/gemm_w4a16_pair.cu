// W4A16 GEMM on the 5th-generation tensor cores, two SMs per tile:  Y[M,N] = X[M,K] . W^T.
//
// A pair of CTAs (cluster of two, tcgen05 cta_group::2) computes tiles of 256 weight rows x NB rows of X.  The packed
// weights are read once per X tile, dequantised to f16 in registers, written into tensor memory and consumed from
// there (A operand); the rows of X come by TMA into shared memory (B operand), HALF of them into each CTA: what one SM
// loads per 128 x 128 weights is 10 KB of weights and NB / 2 x 256 bytes of X, so that neither L2 nor shared memory
// is the limit at NB = 64, and at NB = 256 the tensor pipe is.
//
//   step  = 128 elements of K: A slot of 64 TMEM columns, X slot of NB / 2 rows x 256 bytes, one phase of the "full"
//           (A and X) and "empty" barriers, eight tcgen05.mma (M = 256, N = NB, K = 16).  The X ring is deeper than
//           the A ring: a slot that waits for a TMA load from L2 (about a microsecond) would set the pace otherwise.
//   unit  = 2 steps = 256 elements of K: one raw stage (128 rows x 128 nibble bytes and 8 scales, by cp.async)
//   tile  = SB units;  the sequence of all (tile, unit) is dealt out in equal contiguous runs, one per pair
//
// Roles (768 threads per CTA):
//   warps 0-2    issue the MMAs (leader, cluster rank 0, only): warp w < W the steps w, w + W, ... of a segment into
//                accumulator set w
//   warp 3       X loader: TMA of this CTA's half of the X rows, bytes counted on the leader's full barrier
//   warps 4-7    raw loaders: run ahead by the depth of the raw ring; start before the grid dependency resolves
//   warps 8-23   dequantisers: four groups of four warps (thread = weight row = TMEM lane), group s % 4 takes step s.
//                Waits for the raw stage and for the A slot, 4 blocks of 32 weights per thread: LDS, (q - 8) * scale,
//                tcgen05.st; one arrival per warp on the LEADER's full barrier.  The same warps are the epilogue.
// TMEM: W accumulator sets of NB columns, then the A slots.  X is loaded without multicast.
//
// Ring discipline: a parity wait is only meaningful when the waiter knows the barrier's previous phase to be complete.
// full / empty barriers are indexed by the step modulo kBarRing = 24 (a multiple of the number of dequantiser groups
// and of issuing warps), raw barriers by the unit modulo an even ring: consecutive phases of a barrier are always
// awaited by the same threads, in order.  Every wait is bounded in time; an expired one latches an error code
// (nve_b200_gemm_error) and both CTAs leave through the normal path.
#include <cuda.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "act_ops.cuh"
#include "gemm_w4a16.cuh"

namespace nve {

constexpr int kPairRows = 128;           // weight rows per CTA
constexpr int kPairTile = 256;           // per pair
constexpr int kPairStepCols = 64;        // TMEM columns of an A slot (128 f16 per row)
constexpr int kPairIssueWarp = 0;        // first of up to three issuing warps
constexpr int kPairRawWarp = 4, kPairRawWarps = 4;
constexpr int kPairDeqWarp = 8, kPairDeqWarps = 16;
constexpr int kPairXWarp = 3;
constexpr int kPairThreads = 24 * 32;
constexpr int kBarRing = 24;
constexpr int kMaxRaw = 8;
constexpr int kRawNib = kPairRows * 128, kRawSc = kPairRows * 32, kRawBytes = kRawNib + kRawSc;
constexpr int kPairSiluBytes = 4 * 2 * 128 * 16;
constexpr int kPairSmemMax = 226 * 1024;  // dynamic; the barriers take the first (static) kilobyte
constexpr unsigned long long kPairWaitLimitNs = 50ull * 1000 * 1000;  // a legitimate wait lasts microseconds

struct PairParams {
    const uint8_t* nib[3];
    const float* sc[3];
    void* Y[3];
    int Nm[3];
    int wt_end[3];   // cumulative 256-row tiles of the matrices
    float* partial;  // [2 * pairs][part_rows][256] f32: slot 2c = first, 2c + 1 = last cut segment of pair c
    int M, K, nb;
    int part_rows;   // rows of X that a partial tile holds: min(M, NB)
    int NB;          // rows of X per tile (multiple of 32, <= 256)
    int XT;          // X tiles
    int W;           // accumulator sets = issuing warps
    int slots;       // A slots (TMEM)
    int xslots;      // X slots (shared memory), at most kBarRing
    int raw;         // raw stages (even)
    int SB;          // units per tile
    int U;           // units per pair
    int total;       // units
    int sc16;        // 1: rows of scales are 16-byte aligned
    short y2;        // 1: an output is not 4-byte aligned
    short y8;        // 1: the 16-bit outputs, what is added to them, and their rows are 8-byte aligned
    int by_tile;     // 1: every segment is in the workspace, that of (run, tile) in slot run + tile (the kernel for few rows)
    const uint16_t* res;  // kPairAdd: [M, N] f16, added to the rounded product
};
// What happens to the product on its way out
constexpr int kPairPlain = 0;  // Y = X . W^T
constexpr int kPairAdd = 1;    // Y = res + round16(X . W^T), f16, one matrix
constexpr int kPairSilu = 2;   // Y = silu(round16(X . G^T)) * round16(X . U^T), f16: a tile is 128 rows of G and the 128 rows of U
                               // of the same indices, each CTA has 64 of both (TMEM lanes 0-63 and 64-127)

// ---- mbarrier / TMA / tcgen05 wrappers
__device__ __forceinline__ void pg_init(uint32_t bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void pg_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void pg_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void pg_expect(uint32_t bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t pg_map(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ bool pg_try(uint32_t bar, unsigned parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Wait of a whole, converged warp; the answer is the same for all its lanes (the tcgen05 instructions that follow need
// the whole warp).
__device__ __noinline__ bool pg_wait_slow(uint32_t bar, unsigned parity) {
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    bool late;
    do {
        for (int i = 0; i < 64; i++)
            if (__all_sync(0xffffffffu, pg_try(bar, parity))) return true;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        late = __any_sync(0xffffffffu, t - t0 >= kPairWaitLimitNs);
    } while (!late);
    return false;
}
__device__ __forceinline__ bool pg_wait(uint32_t bar, unsigned parity) {
    if (__all_sync(0xffffffffu, pg_try(bar, parity))) return true;
    return pg_wait_slow(bar, parity);
}
// tile load into this CTA's shared memory, bytes counted on a barrier of either CTA of the pair
__device__ __forceinline__ void pg_tma_pair(uint32_t dst, const CUtensorMap* map, int row, int kblock, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(0), "r"(row), "r"(kblock), "r"(cluster_bar)
        : "memory");
}
__device__ __forceinline__ bool pg_elect() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void pg_mma(bool issuer, uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(static_cast<uint32_t>(issuer))
        : "memory");
}
// arrives on the barrier at this offset in both CTAs when the thread's MMAs so far are complete
__device__ __forceinline__ void pg_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}
__device__ __forceinline__ void pg_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void pg_tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
__device__ __forceinline__ void pg_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void pg_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// K-major SWIZZLE_128B descriptor: 1024 bytes between 8-row groups, descriptor version 1, layout type 2
__device__ __forceinline__ uint64_t pg_desc(uint32_t smem_addr) {
    uint64_t d = static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

static __device__ int g_pair_error = 0;

struct PairTile {
    int mi, n0, xt;  // matrix, first weight row of the pair's tile inside it, X tile
};
template <int MODE> __device__ __forceinline__ PairTile pair_locate(const PairParams& p, int tile) {
    PairTile t;
    const int wt = tile / p.XT;
    t.xt = tile - wt * p.XT;
    t.mi = wt < p.wt_end[0] ? 0 : (wt < p.wt_end[1] ? 1 : 2);
    t.n0 = (wt - (t.mi == 0 ? 0 : p.wt_end[t.mi - 1])) * (MODE == kPairSilu ? kPairTile / 2 : kPairTile);
    return t;
}

// R rows of X (rows m, m + 1, ... of Y) x this lane's feature n.  16-bit types: lanes 2i and 2i + 1 exchange values
// so that every lane stores two neighbouring features of every second row in one 4-byte store.
template <int ODT, int MODE, int R>
__device__ __forceinline__ void pair_store(void* Y, const uint16_t* res, bool narrow, int Nloc, int n, int lane, int m, int rows, const float (&y)[R]) {
    constexpr int DT16 = ODT == NVE_DT_BF16 ? NVE_DT_BF16 : NVE_DT_F16;
    auto add = [](uint16_t a, uint16_t b) { return Act16<DT16>::from_f32(__fadd_rn(Act16<DT16>::to_f32(a), Act16<DT16>::to_f32(b))); };
    if (ODT == NVE_DT_F32 || narrow || (Nloc & 1)) {
#pragma unroll
        for (int e = 0; e < R; e++)
            if (e < rows && n < Nloc) {
                const long long o = static_cast<long long>(m + e) * Nloc + n;
                if (MODE == kPairAdd) static_cast<uint16_t*>(Y)[o] = add(Act16<DT16>::from_f32(y[e]), res[o]);
                else store_out<ODT>(Y, o, y[e]);
            }
    } else {
        const int odd = lane & 1;
        const long long o = static_cast<long long>(m + odd) * Nloc + (n - odd);
        uint16_t* dst = static_cast<uint16_t*>(Y) + o;
        const uint16_t* src = MODE == kPairAdd ? res + o : nullptr;
#pragma unroll
        for (int e = 0; e < R; e += 2) {
            const uint32_t own = static_cast<uint32_t>(Act16<DT16>::from_f32(y[e])) | (static_cast<uint32_t>(Act16<DT16>::from_f32(y[e + 1])) << 16);
            const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
            // even lane: row e of (n, n + 1); odd lane: row e + 1 of (n - 1, n)
            uint32_t v = odd ? __byte_perm(other, own, 0x7632) : __byte_perm(own, other, 0x5410);
            if (e + odd < rows && n < Nloc) {
                if (MODE == kPairAdd) {
                    const uint32_t r = *reinterpret_cast<const uint32_t*>(src);
                    v = static_cast<uint32_t>(add(static_cast<uint16_t>(v), static_cast<uint16_t>(r))) |
                        (static_cast<uint32_t>(add(static_cast<uint16_t>(v >> 16), static_cast<uint16_t>(r >> 16))) << 16);
                }
                *reinterpret_cast<uint32_t*>(dst) = v;
            }
            dst += 2 * static_cast<long long>(Nloc);
            if (MODE == kPairAdd) src += 2 * static_cast<long long>(Nloc);
        }
    }
}

template <int ODT, int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
    gemm_w4a16_pair_kernel(const PairParams p, const __grid_constant__ CUtensorMap xmap) {
    extern __shared__ __align__(1024) unsigned char pg_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kBarRing + 2 * kMaxRaw + 2 + 4];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t smem = (s_addr(pg_raw) + 1023u) & ~1023u;
    const uint32_t bslot_bytes = static_cast<uint32_t>(p.NB) * 128;  // NB / 2 rows x 256 bytes
    const uint32_t sB = smem, sRaw = smem + p.xslots * bslot_bytes;
    const uint32_t sX = sRaw + p.raw * kRawBytes;  // kPairSilu: exchange between the halves of a tile, [4 groups][2][128 rows][16 B]
    const uint32_t full = s_addr(bars), empty = full + 8 * kBarRing, rawf = empty + 8 * kBarRing, rawe = rawf + 8 * kMaxRaw;
    const uint32_t accum = rawe + 8 * kMaxRaw, accfree = accum + 8, swap = accfree + 8;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int pair = blockIdx.x >> 1;
    const int u0 = pair * p.U;
    const int n_units = min(p.U, p.total - u0);
    const int n_steps = 2 * n_units;

    if (tid < kBarRing) {
        pg_init(full + 8 * tid, 9);   // leader: four dequantiser warps of each CTA + expect_tx of both halves of the X rows
        pg_init(empty + 8 * tid, 1);  // tcgen05.commit
        if (tid < p.raw) {
            pg_init(rawf + 8 * tid, 32 * kPairRawWarps);  // the copies of every loader lane
            pg_init(rawe + 8 * tid, 8);                   // the eight warps that read the stage
        }
        if (MODE == kPairSilu && tid < 4) pg_init(swap + 8 * tid, 4);  // the four warps of a dequantiser group
        if (tid == 0) {
            pg_init(accum, p.W);
            pg_init(accfree, 2 * kPairDeqWarps);  // leader: every dequantiser (= epilogue) warp of both CTAs
            abort_flag = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pg_cluster_arrive();  // matched below: nothing reaches into the other CTA before its barriers are set up
    bool ok = true;
    auto fail = [&](int code) {
        atomicCAS(&g_pair_error, 0, code);
        *reinterpret_cast<volatile int*>(&abort_flag) = 1;
        ok = false;
    };

    if (warp >= kPairRawWarp && warp < kPairRawWarp + kPairRawWarps) {
        // ------------------------------------------------------------------ raw loaders (weights: no dependency wait)
        // Plain asynchronous copies, not TMA: the TMA unit needs about four cycles per 128-byte row, and 256 rows of
        // nibbles and scales per unit next to the rows of X made it the slowest part of the kernel.
        const int lw = warp - kPairRawWarp;
        const int nr = lw * 32 + (lane >> 3), nc = lane & 7;  // nibbles: rows nr, nr + 4, ..., nr + 28, 16-byte chunk nc
        const int half_k = p.K / 2;
        int tile = u0 / p.SB, sbi = u0 - (u0 / p.SB) * p.SB;
        PairTile tl = pair_locate<MODE>(p, tile);
        int st = 0;
        unsigned par = 1;
        for (int j = 0; j < n_units; j++) {
            if (j >= p.raw) {
                if (!pg_wait(rawe + 8 * st, par)) {
                    fail(3);
                    break;
                }
            }
            // row 0 of the warp's 32: rows of one matrix, or (gate / up) rows 0-63 of the one and 64-127 of the other
            const int mi = MODE == kPairSilu ? lw >> 1 : tl.mi;
            const int row0 = MODE == kPairSilu ? tl.n0 + static_cast<int>(rank) * 64 - (lw >> 1) * 64 : tl.n0 + static_cast<int>(rank) * kPairRows;
            const int nlast = p.Nm[mi] - 1;
            const uint32_t dst = sRaw + st * kRawBytes;
            {
                // chunks past the end of K read as zero, rows past the end repeat the last one
                const int kb = sbi * 128 + nc * 16;
                const uint8_t* src = p.nib[mi] + (kb < half_k ? kb : 0);
                const int have = kb < half_k ? 16 : 0;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int r = nr + 4 * i;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * 128 + ((nc ^ (r & 7)) << 4)),
                                 "l"(src + static_cast<long long>(min(row0 + r, nlast)) * half_k), "r"(have)
                                 : "memory");
                }
            }
            const float* sc = p.sc[mi];
            const int b0 = sbi * 8;
            if (p.sc16) {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int r = lw * 32 + (lane >> 1) + 16 * i, c = lane & 1;
                    const int have = min(16, max(0, (p.nb - b0 - 4 * c) * 4));
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + kRawNib + r * 32 + c * 16),
                                 "l"(sc + static_cast<long long>(min(row0 + r, nlast)) * p.nb + (have > 0 ? b0 + 4 * c : 0)), "r"(have)
                                 : "memory");
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = lw * 32 + (lane >> 2) + 8 * i, c = lane & 3;
                    const int have = min(8, max(0, (p.nb - b0 - 2 * c) * 4));
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + kRawNib + r * 32 + c * 8),
                                 "l"(sc + static_cast<long long>(min(row0 + r, nlast)) * p.nb + (have > 0 ? b0 + 2 * c : 0)), "r"(have)
                                 : "memory");
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(rawf + 8 * st) : "memory");
            if (++st == p.raw) {
                st = 0;
                par ^= 1;
            }
            if (++sbi == p.SB) {
                sbi = 0;
                tile++;
                if (j + 1 < n_units) tl = pair_locate<MODE>(p, tile);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        // not before the kernel in front is complete: what starts then may read what was written two launches ahead of it
        pdl_wait();
        pdl_launch_dependents();
        pg_cluster_wait();
    } else {
        if (warp == kPairIssueWarp) {  // TMEM allocation is warp-wide, one warp of each CTA of the pair
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_addr(&tmem_slot)), "r"(512) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(kPairThreads - 32 * kPairRawWarps) : "memory");  // everyone but the raw loaders
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        pg_cluster_wait();
        const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
        const uint32_t acols = p.W * p.NB;

        if (warp >= kPairDeqWarp && warp < kPairDeqWarp + kPairDeqWarps) {
            // -------------------------------------------------------------- dequantisers
            const int grp = (warp - kPairDeqWarp) >> 2;                       // takes steps grp, grp + 4, ...
            const int r = (warp & 3) * 32 + lane;            // weight row of the CTA = TMEM lane
            const uint32_t tmem_lane = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + acols;
            const uint32_t lfull = pg_map(full, 0);
            uint32_t roff[4];  // chunk (4 * half + q) of the 128-byte swizzled row
#pragma unroll
            for (int q = 0; q < 4; q++) roff[q] = r * 128 + (((4 * (grp & 1) + q) ^ (r & 7)) << 4);
            const uint32_t soff = kRawNib + r * 32 + (grp & 1) * 16;
            const DequantConsts dc = make_dequant_consts();
            // The epilogue of a segment is shared by all sixteen warps: a quarter of the columns per group.  A group takes one
            // step of the next segment first (the segment's last MMAs run meanwhile) and comes back here; the accumulators are handed
            // back as soon as they are in registers.  With every operand slot filled first and the accumulators handed back at the end
            // the MMAs stood still for 8100 of 36000 cycles (8B gate/up, 61 rows; four GEMMs of a layer 70.7 us, 68.0 as it is; 69.3
            // with as many steps ahead as there are slots).
            const uint32_t lfree = pg_map(accfree, 0);
            int xb = 0;  // kPairSilu: half of the exchange buffer, and parity of its barrier
            int ej = 0, eseg = 0, etile = u0 / p.SB, esbi = u0 - (u0 / p.SB) * p.SB;  // first segment without its epilogue
            int eunits = min(p.SB - esbi, n_units);
            int lim = min(n_steps, 2 * eunits + 4);  // the group's steps from here on wait for the epilogue: one step of the next segment each
            auto epilogue = [&]() -> bool {
                if (eseg == 0) pdl_wait();  // the stores below must not overtake the previous kernel's reads
                if (!pg_wait(accum, static_cast<unsigned>(eseg) & 1u)) {
                    fail(5);
                    return false;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const PairTile tl = pair_locate<MODE>(p, etile);
                const int Nloc = p.Nm[tl.mi];
                const bool whole = eunits == p.SB;
                const int col = static_cast<int>(rank) * kPairRows + r;
                // this thread's output feature (kPairSilu: lanes 64 and up hold the second factor of the same features)
                const int n = MODE == kPairSilu ? tl.n0 + static_cast<int>(rank) * 64 + (r & 63) : tl.n0 + col;
                const int m0 = tl.xt * p.NB;
                const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
                float* part = p.partial + static_cast<long long>(2 * pair + (eseg > 0 ? 1 : 0)) * p.part_rows * kPairTile + col;
                const int mrows = min(p.NB, p.M - m0);
                // the accumulators are read: the next segment's products may come in while this one's are finished and stored
                auto release = [&]() {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) pg_arrive_cluster(lfree);
                };
                if (16 * grp >= mrows) release();
                for (int cb = 16 * grp; cb < mrows; cb += 64) {
                    float y[16];
                    uint32_t v[16];
                    pg_tmem_ld16(taddr + cb, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 16; e++) y[e] = __uint_as_float(v[e]);
                    for (int a = 1; a < min(p.W, 2 * eunits); a++) {
                        pg_tmem_ld16(taddr + a * p.NB + cb, v);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int e = 0; e < 16; e++) y[e] = __fadd_rn(y[e], __uint_as_float(v[e]));
                    }
                    if (cb + 64 >= mrows) release();
                    if (!whole) {
#pragma unroll
                        for (int e = 0; e < 16; e++)
                            if (cb + e < mrows) part[(cb + e) * kPairTile] = y[e];
                    } else {
                        if constexpr (MODE == kPairSilu) {
                            // the lower warps have sixteen values of the one factor, the upper ones of the other; rounded to f16 like a
                            // stored product, each half hands eight over and finishes eight rows of X
                            const bool up = r >= 64;
                            const uint32_t buf = sX + static_cast<uint32_t>((grp * 2 + xb) * 2048);
                            uint32_t h[4];
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                const __half2 v2 = up ? __floats2half2_rn(y[2 * e], y[2 * e + 1]) : __floats2half2_rn(y[8 + 2 * e], y[9 + 2 * e]);
                                h[e] = *reinterpret_cast<const uint32_t*>(&v2);
                            }
                            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(buf + r * 16), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
                            __syncwarp();
                            if (lane == 0) pg_arrive(swap + 8 * grp);
                            if (!pg_wait(swap + 8 * grp, static_cast<unsigned>(xb))) {  // a warp of the group has given up
                                fail(6);
                                return false;
                            }
                            xb ^= 1;  // the other half next time: one barrier per exchange is enough
                            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]) : "r"(buf + (r ^ 64) * 16) : "memory");
                            float z[8];
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                const float own = Act16<NVE_DT_F16>::to_f32(Act16<NVE_DT_F16>::from_f32(up ? y[8 + e] : y[e]));
                                const float other = Act16<NVE_DT_F16>::to_f32(static_cast<uint16_t>(h[e >> 1] >> (16 * (e & 1))));
                                z[e] = silu_mul_f32(up ? other : own, up ? own : other);
                            }
                            const int from = cb + (up ? 8 : 0);
                            pair_store<ODT, MODE>(p.Y[0], nullptr, p.y2 != 0, Nloc, n, lane, m0 + from, min(8, mrows - from), z);
                        } else {
                            pair_store<ODT, MODE>(p.Y[tl.mi], p.res, p.y2 != 0, Nloc, n, lane, m0 + cb, min(16, mrows - cb), y);
                        }
                    }
                }
                ej += eunits;
                esbi += eunits;
                if (esbi == p.SB) {
                    esbi = 0;
                    etile++;
                }
                eunits = min(p.SB - esbi, n_units - ej);
                eseg++;
                lim = min(n_steps, 2 * (ej + eunits) + 4);
                return true;
            };
            const uint32_t col_end = tmem_lane + p.slots * kPairStepCols;
            uint32_t col = tmem_lane + grp * kPairStepCols;                            // A slot (there are at least four)
            uint32_t rsrc = sRaw + (grp >> 1) * kRawBytes, rbar = 8 * (grp >> 1);      // raw stage
            unsigned rpar = 0, epar = 1;
            int fb = 8 * grp;                                                          // full barrier of the step
            int eb = 8 * (grp - p.slots + kBarRing);                                   // empty barrier of the step p.slots before
            for (int s = grp;;) {
                if (s >= lim) {
                    if (ej == n_units) break;
                    if (!epilogue()) break;
                    continue;
                }
                if (!pg_wait(rawf + rbar, rpar)) {
                    fail(1);
                    break;
                }
                uint4 raw[4];
                float4 scv;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(raw[q].x), "=r"(raw[q].y), "=r"(raw[q].z), "=r"(raw[q].w)
                                 : "r"(rsrc + roff[q])
                                 : "memory");
                asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                             : "=f"(scv.x), "=f"(scv.y), "=f"(scv.z), "=f"(scv.w)
                             : "r"(rsrc + soff)
                             : "memory");
                if (s >= p.slots) {  // the step that used this slot last has been multiplied
                    if (!pg_wait(empty + eb, epar)) {
                        fail(1);
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                const float scq[4] = {scv.x, scv.y, scv.z, scv.w};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const DequantScale ds = make_dequant_scale(scq[q]);
                    uint32_t v[16];  // v[c] = elements (2c, 2c+1) of the block
                    dequant_word(raw[q].x, ds, dc, v[0], v[1], v[8], v[9]);
                    dequant_word(raw[q].y, ds, dc, v[2], v[3], v[10], v[11]);
                    dequant_word(raw[q].z, ds, dc, v[4], v[5], v[12], v[13]);
                    dequant_word(raw[q].w, ds, dc, v[6], v[7], v[14], v[15]);
                    pg_tmem_st16(col + 16 * q, v);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    pg_arrive_cluster(lfull + fb);
                    pg_arrive(rawe + rbar);
                }
                s += 4;
                col += 4 * kPairStepCols;
                if (col >= col_end) col -= p.slots * kPairStepCols;
                rsrc += 2 * kRawBytes;
                rbar += 16;
                if (rbar >= static_cast<uint32_t>(8 * p.raw)) {
                    rbar -= 8 * p.raw;
                    rsrc -= p.raw * kRawBytes;
                    rpar ^= 1u;
                }
                fb += 32;
                if (fb >= 8 * kBarRing) fb -= 8 * kBarRing;
                eb += 32;
                if (eb >= 8 * kBarRing) {
                    eb -= 8 * kBarRing;
                    epar ^= 1u;
                }
            }
        } else if (warp == kPairXWarp) {
            // -------------------------------------------------------------- X loader
            // the whole warp runs the loop, one lane issues (operands in uniform registers)
            const bool issuer = pg_elect();
            if (issuer) asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
            pdl_wait();  // activations come from the previous kernel
            const uint32_t lfull = pg_map(full, 0);
            int tile = u0 / p.SB, ts = 2 * (u0 - (u0 / p.SB) * p.SB);
            int xrow = (tile % p.XT) * p.NB + static_cast<int>(rank) * (p.NB / 2);
            int slot = 0, bi = 0, eb = 0;  // X slot; full barrier of the step; empty barrier of the step that used the slot last
            unsigned epar = 0;
            for (int s = 0; s < n_steps; s++) {
                if (s >= p.xslots) {
                    if (!pg_wait(empty + 8 * eb, epar)) {
                        fail(4);
                        break;
                    }
                    if (++eb == kBarRing) {
                        eb = 0;
                        epar ^= 1u;
                    }
                }
                if (issuer) {
                    if (rank == 0) pg_expect(full + 8 * bi, 2 * bslot_bytes);
                    pg_tma_pair(sB + slot * bslot_bytes, &xmap, xrow, 2 * ts, lfull + 8 * bi);
                }
                __syncwarp();
                if (++slot == p.xslots) slot = 0;
                if (++bi == kBarRing) bi = 0;
                if (++ts == 2 * p.SB) {
                    ts = 0;
                    tile++;
                    xrow = (tile % p.XT) * p.NB + static_cast<int>(rank) * (p.NB / 2);
                }
            }
        } else if (rank == 0 && warp < kPairIssueWarp + p.W) {
            // -------------------------------------------------------------- MMA issue
            // The whole warp runs this loop and one lane of it issues: operands then live in uniform registers.  Warp w
            // takes the steps w, w + W, ... of a segment into accumulator set w.
            const int w = warp - kPairIssueWarp;
            const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(p.NB >> 3) << 17) | (static_cast<uint32_t>(kPairTile >> 4) << 24);
            const bool issuer = pg_elect();
            int j = 0, seg = 0;
            int tile = u0 / p.SB, sbi = u0 - (u0 / p.SB) * p.SB;
            while (j < n_units) {
                const int seg_units = min(p.SB - sbi, n_units - j);
                const int seg_steps = 2 * seg_units;
                if (seg > 0 && !pg_wait(accfree, static_cast<unsigned>(seg - 1) & 1u)) fail(2);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                int s = 2 * j + w;
                int bi = s % kBarRing, slot = s % p.slots, xslot = s % p.xslots;
                unsigned par = static_cast<unsigned>(s / kBarRing) & 1u;
                uint32_t acc = 0;
                for (int q = w; q < seg_steps; q += p.W) {
                    if (!pg_wait(full + 8 * bi, par)) {
                        fail(2);
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a = tmem + acols + slot * kPairStepCols;
                    const uint32_t xs = sB + xslot * bslot_bytes;
                    const uint64_t bd0 = pg_desc(xs), bd1 = pg_desc(xs + bslot_bytes / 2);
                    pg_mma(issuer, tmem + w * p.NB, a, bd0, idesc, acc);
#pragma unroll
                    for (int kk = 1; kk < 8; kk++)  // 16 elements along K: 8 TMEM columns of A, 32 bytes of B
                        pg_mma(issuer, tmem + w * p.NB, a + 8 * kk, (kk < 4 ? bd0 : bd1) + 2 * (kk & 3), idesc, 1u);
                    acc = 1;
                    if (issuer) pg_commit(empty + 8 * bi);
                    __syncwarp();
                    bi += p.W;
                    if (bi >= kBarRing) {
                        bi -= kBarRing;
                        par ^= 1u;
                    }
                    slot += p.W;
                    if (slot >= p.slots) slot -= p.slots;
                    xslot += p.W;
                    if (xslot >= p.xslots) xslot -= p.xslots;
                }
                if (!ok) break;
                if (issuer) pg_commit(accum);  // a warp without a step in the segment arrives at once
                __syncwarp();
                j += seg_units;
                sbi += seg_units;
                if (sbi == p.SB) {
                    sbi = 0;
                    tile++;
                }
                seg++;
            }
        }
    }
    // ---- teardown.  After an expired wait copies may still be in flight into this CTA: give them time to land.
    if (*reinterpret_cast<volatile int*>(&abort_flag)) {
        for (int i = 0; i < 100; i++) __nanosleep(10000);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pg_cluster_arrive();
    pg_cluster_wait();  // neither CTA leaves, or frees its TMEM, while the other may still reach into it
    if (warp == kPairIssueWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// Sums of four consecutive columns of row mm of a tile, from col, col + step, ..., over the pairs that worked on it, in ascending K order.
// Eight loads on their way at a time: one after the other each cost an L2 round trip, and that was most of the call for a row or two of
// tiles cut into a dozen segments.  So did a second group of columns behind the first (layers, us, one group after the other / together: 8B
// 20 rows 70.7 / 69.4, 61 rows 76.4 / 74.9, 300 rows 155.6 / 152.4, 3B 300 rows at 700 116.9 / 113.6).
template <int C> __device__ __forceinline__ void pair_sums4(const PairParams& p, int tile, int first, int last, int mm, int col, int step, float4 (&y)[C]) {
    auto part = [&](int c, int g) {
        // by pair: its first segment when its run starts inside this tile
        const int slot = p.by_tile ? c + tile : 2 * c + (c * p.U >= tile * p.SB ? 0 : 1);
        return __ldcg(reinterpret_cast<const float4*>(p.partial + (static_cast<long long>(slot) * p.part_rows + mm) * kPairTile + col + g * step));
    };
    constexpr int kFly = 8 / C;
#pragma unroll
    for (int g = 0; g < C; g++) y[g] = part(first, g);
    for (int c = first + 1; c <= last; c += kFly) {
        float4 v[kFly][C];
#pragma unroll
        for (int i = 0; i < kFly; i++)
            if (c + i <= last)
#pragma unroll
                for (int g = 0; g < C; g++) v[i][g] = part(c + i, g);
#pragma unroll
        for (int i = 0; i < kFly; i++)
            if (c + i <= last)
#pragma unroll
                for (int g = 0; g < C; g++) {
                    y[g].x = __fadd_rn(y[g].x, v[i][g].x);
                    y[g].y = __fadd_rn(y[g].y, v[i][g].y);
                    y[g].z = __fadd_rn(y[g].z, v[i][g].z);
                    y[g].w = __fadd_rn(y[g].w, v[i][g].w);
                }
    }
}
__device__ __forceinline__ float4 pair_sum4(const PairParams& p, int tile, int first, int last, int mm, int col) {
    float4 y[1];
    pair_sums4<1>(p, tile, first, last, mm, col, 0, y);
    return y[0];
}

// Tiles that more than one pair worked on: sum their partial tiles, finish as the epilogue would and store.  One block
// per (tile, four rows of X), a thread takes four consecutive features.  Where runs are at least a tile long, a boundary of two runs stands for
// the tile that it cuts: most tiles of a wide call are whole (8B gate/up, 1777 rows: 73 of 784), and blocks that found that out and left
// took most of the launch; 16-bit values move four at a time (8B layer, 1777 rows, the two finishes of the FFN: 53 us less; four rows a
// thread instead of one: 128 rows 92.5 -> 100, 1777 rows no change).
// CUT: a block per boundary (a branch instead costs a call of a few rows another division).
template <int ODT, int MODE, bool CUT> __global__ void __launch_bounds__(256) gemm_pair_reduce_kernel(const PairParams p) {
    pdl_wait();
    pdl_launch_dependents();
    const int tile = CUT ? (static_cast<int>(blockIdx.x) + 1) * p.U / p.SB : static_cast<int>(blockIdx.x);
    const int first = (tile * p.SB) / p.U, last = ((tile + 1) * p.SB - 1) / p.U;
    if (first == last && !p.by_tile) return;
    const PairTile tl = pair_locate<MODE>(p, tile);
    const int Nloc = p.Nm[tl.mi];
    const int c4 = static_cast<int>(threadIdx.x) * 4, n = tl.n0 + c4;
    const int mm = static_cast<int>(blockIdx.y * blockDim.y + threadIdx.y), m = tl.xt * p.NB + mm;
    if (n >= Nloc || mm >= p.NB || m >= p.M) return;
    const long long o = static_cast<long long>(m) * Nloc + n;
    // kPairSilu: feature c4 of the tile is column (c4 & 63) of CTA c4 / 64, its second factor 64 columns further
    const int col = MODE == kPairSilu ? (c4 >> 6) * kPairRows + (c4 & 63) : c4;
    const bool four = p.y8 && n + 4 <= Nloc;
    uint2 res = make_uint2(0, 0);
    if (MODE == kPairAdd && four) res = *reinterpret_cast<const uint2*>(p.res + o);
    float4 sums[MODE == kPairSilu ? 2 : 1];
    pair_sums4(p, tile, first, last, mm, col, 64, sums);
    float yy[4] = {sums[0].x, sums[0].y, sums[0].z, sums[0].w};
    using A = Act16<NVE_DT_F16>;
    if constexpr (MODE == kPairSilu) {
        const float4 u = sums[1];
        const float uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; e++) yy[e] = silu_mul_f32(A::to_f32(A::from_f32(yy[e])), A::to_f32(A::from_f32(uu[e])));
    }
    if constexpr (MODE == kPairAdd) {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (n + e < Nloc)
                yy[e] = __fadd_rn(A::to_f32(A::from_f32(yy[e])), A::to_f32(four ? static_cast<uint16_t>((e < 2 ? res.x : res.y) >> (16 * (e & 1))) : p.res[o + e]));
    }
    if (ODT != NVE_DT_F32 && four) {
        using O = Act16<ODT == NVE_DT_BF16 ? NVE_DT_BF16 : NVE_DT_F16>;
        auto two = [](float a, float b) { return static_cast<uint32_t>(O::from_f32(a)) | (static_cast<uint32_t>(O::from_f32(b)) << 16); };
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p.Y[tl.mi]) + o) = make_uint2(two(yy[0], yy[1]), two(yy[2], yy[3]));
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (n + e < Nloc) store_out<ODT>(p.Y[tl.mi], o + e, yy[e]);
    }
}

// The same for q, k and v of a prompt block, and what follows them: the rotary embedding, with the arithmetic and the rounding of the
// stand-alone kernel, and the K/V write.  Every tile goes through here; those that one pair covered are in Y already.  A thread
// takes four element pairs (i, i + hd / 2) of a head, 32 threads a row of the tile.  As launches of their own the finish and the embedding
// cost two grid dependencies (1.85 us each) and read q, k and v once more.
__global__ void __launch_bounds__(256) gemm_pair_reduce_rope_kernel(const PairParams p, const PairRope ro) {
    const int tile = blockIdx.x;
    const int first = (tile * p.SB) / p.U, last = ((tile + 1) * p.SB - 1) / p.U;
    const PairTile tl = pair_locate<kPairPlain>(p, tile);
    const int Nloc = p.Nm[tl.mi], half = ro.hd / 2, per = half / 4;
    const int head = static_cast<int>(threadIdx.x) / per, i = (static_cast<int>(threadIdx.x) - head * per) * 4, col = head * ro.hd + i;
    const int mm = static_cast<int>(blockIdx.y * blockDim.y + threadIdx.y), m = tl.xt * p.NB + mm, n = tl.n0 + col;
    const bool have = n < Nloc && mm < p.NB && m < p.M;
    using A = Act16<NVE_DT_F16>;
    uint16_t* y = static_cast<uint16_t*>(p.Y[tl.mi]) + static_cast<long long>(m) * Nloc + n;
    const int pos = ro.start_pos + m;
    uint2 cw = make_uint2(0, 0), sw = cw;  // static, like all up to here: 61 rows 74.7 -> 74.1 us a layer (the other finishes: few rows slower)
    if (have && tl.mi < 2) {
        cw = *reinterpret_cast<const uint2*>(ro.cos_t + static_cast<long long>(pos) * half + i);
        sw = *reinterpret_cast<const uint2*>(ro.sin_t + static_cast<long long>(pos) * half + i);
    }
    pdl_wait();
    pdl_launch_dependents();
    if (!have) return;
    uint2 a, b;
    if (first == last && !p.by_tile) {
        a = __ldcg(reinterpret_cast<const uint2*>(y));
        b = __ldcg(reinterpret_cast<const uint2*>(y + half));
    } else {
        float4 fg[2];
        pair_sums4<2>(p, tile, first, last, mm, col, half, fg);
        const float4 f = fg[0], g = fg[1];
        auto two = [](float u, float v) { return static_cast<uint32_t>(A::from_f32(u)) | (static_cast<uint32_t>(A::from_f32(v)) << 16); };
        a = make_uint2(two(f.x, f.y), two(f.z, f.w));
        b = make_uint2(two(g.x, g.y), two(g.z, g.w));
    }
    if (tl.mi < 2) {
        auto turn = [](uint32_t& x, uint32_t& z, uint32_t co2, uint32_t si2) {
            uint32_t r0 = 0, r1 = 0;
#pragma unroll
            for (int e = 0; e < 2; e++) {
                auto pick = [&](uint32_t w) { return A::to_f32(static_cast<uint16_t>(w >> (16 * e))); };
                const float x0 = pick(x), x1 = pick(z), co = pick(co2), si = pick(si2);
                r0 |= static_cast<uint32_t>(A::from_f32(__fsub_rn(__fmul_rn(x0, co), __fmul_rn(x1, si)))) << (16 * e);
                r1 |= static_cast<uint32_t>(A::from_f32(__fadd_rn(__fmul_rn(x0, si), __fmul_rn(x1, co)))) << (16 * e);
            }
            x = r0;
            z = r1;
        };
        turn(a.x, b.x, cw.x, sw.x);
        turn(a.y, b.y, cw.y, sw.y);
    }
    if (tl.mi > 0) y = (tl.mi == 1 ? ro.k_cache : ro.v_cache) + (static_cast<long long>(n / ro.hd) * ro.max_seq + pos) * ro.hd + i;
    *reinterpret_cast<uint2*>(y) = a;
    *reinterpret_cast<uint2*>(y + half) = b;
}

// The same for one matrix whose product goes through the residual add and an RMSNorm: one block per row of X finishes
// the row -- Y = res + round16(product), normed = RMSNorm(Y) -- with the arithmetic and the summation order of the separate
// kernels (of 256 threads, thread t takes the 8-element chunks t, t + 256, ...).  Tiles that one pair covered are in Y already.
// The sums over segments are spread over all threads, four columns each: with few rows of X (at most one block per SM) they are
// a chain of L2 round trips.
constexpr int kPairNormChunks = 4;  // 8-element chunks per thread: N <= 8192
constexpr int kPairNormThreads = 1024;
__global__ void __launch_bounds__(kPairNormThreads) gemm_pair_reduce_norm_kernel(const PairParams p, const uint16_t* norm_w, uint16_t* normed, float eps) {
    __shared__ float warp_part[8];
    __shared__ uint2 row16[8 * 256 * kPairNormChunks / 4];  // Y of the row
    const int m = blockIdx.x, N = p.Nm[0], chunks = N >> 3;
    const int xt = m / p.NB, mm = m - xt * p.NB;
    const long long row = static_cast<long long>(m) * N;
    const int tid = static_cast<int>(threadIdx.x);
    uint4 w[kPairNormChunks];
    if (tid < 256) {
#pragma unroll
        for (int j = 0; j < kPairNormChunks; j++) {
            const int c = j * 256 + tid;
            if (c < chunks) w[j] = reinterpret_cast<const uint4*>(norm_w)[c];  // static, unlike what follows
        }
    }
    pdl_wait();
    pdl_launch_dependents();
    uint16_t* y16 = static_cast<uint16_t*>(p.Y[0]);
    for (int q = tid; q < (N >> 2); q += kPairNormThreads) {
        const int wt = q >> 6, col = (q & 63) * 4, tile = wt * p.XT + xt;
        const int first = (tile * p.SB) / p.U, last = ((tile + 1) * p.SB - 1) / p.U;
        const uint2 r2 = reinterpret_cast<const uint2*>(p.res + row)[q];
        uint2 y2;
        if (first == last && !p.by_tile) {
            y2 = __ldcg(reinterpret_cast<const uint2*>(y16 + row) + q);
        } else {
            const float4 f = pair_sum4(p, tile, first, last, mm, col);
            y2.x = static_cast<uint32_t>(Act16<NVE_DT_F16>::from_f32(f.x)) | (static_cast<uint32_t>(Act16<NVE_DT_F16>::from_f32(f.y)) << 16);
            y2.y = static_cast<uint32_t>(Act16<NVE_DT_F16>::from_f32(f.z)) | (static_cast<uint32_t>(Act16<NVE_DT_F16>::from_f32(f.w)) << 16);
        }
        auto add = [](uint32_t a, uint32_t b) {
            auto one = [](uint16_t u, uint16_t v) { return Act16<NVE_DT_F16>::from_f32(__fadd_rn(Act16<NVE_DT_F16>::to_f32(u), Act16<NVE_DT_F16>::to_f32(v))); };
            return static_cast<uint32_t>(one(static_cast<uint16_t>(a), static_cast<uint16_t>(b))) |
                   (static_cast<uint32_t>(one(static_cast<uint16_t>(a >> 16), static_cast<uint16_t>(b >> 16))) << 16);
        };
        y2 = make_uint2(add(y2.x, r2.x), add(y2.y, r2.y));
        reinterpret_cast<uint2*>(y16 + row)[q] = y2;
        row16[q] = y2;
    }
    __syncthreads();
    uint4 h[kPairNormChunks];
    if (tid < 256) {
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < kPairNormChunks; j++) {
            const int c = j * 256 + tid;
            if (c < chunks) {
                const uint2 lo = row16[2 * c], hi = row16[2 * c + 1];
                h[j] = make_uint4(lo.x, lo.y, hi.x, hi.y);
                uint16_t a[8];
                unpack8(h[j], a);
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const float v = Act16<NVE_DT_F16>::to_f32(a[e]);
                    acc = __fmaf_rn(v, v, acc);
                }
            }
        }
        acc = warp_sum(acc);
        if ((tid & 31) == 0) warp_part[tid >> 5] = acc;
    }
    __syncthreads();
    if (tid >= 256) return;
    float total = warp_part[0];
#pragma unroll
    for (int i = 1; i < 8; i++) total = __fadd_rn(total, warp_part[i]);
    const float r = __frcp_rn(__fsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(N)), eps)));
#pragma unroll
    for (int j = 0; j < kPairNormChunks; j++) {
        const int c = j * 256 + tid;
        if (c < chunks) {
            uint16_t a[8], b[8];
            unpack8(h[j], a);
            unpack8(w[j], b);
#pragma unroll
            for (int e = 0; e < 8; e++)
                a[e] = Act16<NVE_DT_F16>::from_f32(__fmul_rn(__fmul_rn(Act16<NVE_DT_F16>::to_f32(a[e]), r), Act16<NVE_DT_F16>::to_f32(b[e])));
            reinterpret_cast<uint4*>(normed + row)[c] = pack8(a);
        }
    }
}

// More rows of X than SMs: the blocks hide each other's latency and a thread keeps its chunks of the row in registers, all of
// their loads under way together (o projection with its finish, 8B, 1777 rows: 78.7 us with the form above, 73.4 with this one; 300
// rows 25.6 and 23.5; at 147 and 149 rows, each with its own form, 15.5 and 16.5).
__global__ void __launch_bounds__(256) gemm_pair_reduce_norm_rows_kernel(const PairParams p, const uint16_t* norm_w, uint16_t* normed, float eps) {
    __shared__ float warp_part[8];
    const int m = blockIdx.x, N = p.Nm[0], chunks = N >> 3;
    const int xt = m / p.NB, mm = m - xt * p.NB;
    const long long row = static_cast<long long>(m) * N;
    uint4 w[kPairNormChunks], rs[kPairNormChunks], h[kPairNormChunks];
#pragma unroll
    for (int j = 0; j < kPairNormChunks; j++) {
        const int c = j * 256 + static_cast<int>(threadIdx.x);
        if (c < chunks) w[j] = reinterpret_cast<const uint4*>(norm_w)[c];  // static, unlike what follows
    }
    pdl_wait();
    pdl_launch_dependents();
    uint16_t* y16 = static_cast<uint16_t*>(p.Y[0]);
#pragma unroll
    for (int j = 0; j < kPairNormChunks; j++) {
        const int c = j * 256 + static_cast<int>(threadIdx.x);
        if (c < chunks) rs[j] = reinterpret_cast<const uint4*>(p.res + row)[c];
    }
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < kPairNormChunks; j++) {
        const int c = j * 256 + static_cast<int>(threadIdx.x);
        if (c < chunks) {
            const int wt = c >> 5, col = (c & 31) * 8, tile = wt * p.XT + xt;
            const int first = (tile * p.SB) / p.U, last = ((tile + 1) * p.SB - 1) / p.U;
            uint16_t a[8], b[8];
            if (first == last && !p.by_tile) {
                unpack8(__ldcg(reinterpret_cast<const uint4*>(y16 + row) + c), a);
            } else {
                float4 eight[2];
                pair_sums4<2>(p, tile, first, last, mm, col, 4, eight);
                const float f[8] = {eight[0].x, eight[0].y, eight[0].z, eight[0].w, eight[1].x, eight[1].y, eight[1].z, eight[1].w};
#pragma unroll
                for (int e = 0; e < 8; e++) a[e] = Act16<NVE_DT_F16>::from_f32(f[e]);
            }
            unpack8(rs[j], b);
#pragma unroll
            for (int e = 0; e < 8; e++) {
                a[e] = Act16<NVE_DT_F16>::from_f32(__fadd_rn(Act16<NVE_DT_F16>::to_f32(a[e]), Act16<NVE_DT_F16>::to_f32(b[e])));
                const float v = Act16<NVE_DT_F16>::to_f32(a[e]);
                acc = __fmaf_rn(v, v, acc);
            }
            h[j] = pack8(a);
            reinterpret_cast<uint4*>(y16 + row)[c] = h[j];
        }
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = acc;
    __syncthreads();
    float total = warp_part[0];
#pragma unroll
    for (int i = 1; i < 8; i++) total = __fadd_rn(total, warp_part[i]);
    const float r = __frcp_rn(__fsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(N)), eps)));
#pragma unroll
    for (int j = 0; j < kPairNormChunks; j++) {
        const int c = j * 256 + static_cast<int>(threadIdx.x);
        if (c < chunks) {
            uint16_t a[8], b[8];
            unpack8(h[j], a);
            unpack8(w[j], b);
#pragma unroll
            for (int e = 0; e < 8; e++)
                a[e] = Act16<NVE_DT_F16>::from_f32(__fmul_rn(__fmul_rn(Act16<NVE_DT_F16>::to_f32(a[e]), r), Act16<NVE_DT_F16>::to_f32(b[e])));
            reinterpret_cast<uint4*>(normed + row)[c] = pack8(a);
        }
    }
}

}  // namespace nve
#include "gemm_w4a16_rows.cuh"
namespace nve {

using PairEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (a pure host-side encoder, legal in capture)
static PairEncodeFn pair_encode_fn() {
    static PairEncodeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<PairEncodeFn>(f);
    }();
    return fn;
}
// X [M, K] f16 seen as [K / 64][M][64]: one box = two K blocks x box_rows rows x 64 elements (128 bytes, 128-byte
// swizzle), i.e. all X rows of a step in one instruction; zeros outside.
static bool pair_x_map(CUtensorMap* map, const uint16_t* X, int K, int M, int box_rows) {
    PairEncodeFn fn = pair_encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(M), static_cast<cuuint64_t>(K / 64)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(K) * 2, 128};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), 2};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<uint16_t*>(X), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// How the (tile, unit) sequence is cut into one contiguous run per pair.  With a workspace the runs are equal (total /
// pairs, rounded up; at least two units = 512 weights per row): few tiles are split over K so that every SM works, and
// a tile count that is not a multiple of the pair count costs total / pairs instead of a whole extra wave.  Without a
// workspace a pair takes exactly one tile.
PairPlan pair_plan(const int* Ns, int num_mats, int M, int K, bool have_scratch, size_t avail, bool silu) {
    PairPlan g;
    g.XT = (M + 255) / 256;
    g.NB = ((M + g.XT - 1) / g.XT + 31) / 32 * 32;
    g.XT = (M + g.NB - 1) / g.NB;
    g.SB = (K + 255) / 256;
    long long wt = 0;
    if (silu) wt = (Ns[0] + kPairTile / 2 - 1) / (kPairTile / 2);
    else
        for (int i = 0; i < num_mats; i++) wt += (Ns[i] + kPairTile - 1) / kPairTile;
    g.tiles = wt * g.XT;
    const long long total = g.tiles * g.SB;
    const int pairs = max(1, sm_count() / 2);
    const long long rows = M < g.NB ? M : g.NB;
    long long U = g.SB;
    auto bytes = [&](long long u) -> size_t {
        return u % g.SB == 0 ? 0 : static_cast<size_t>(2 * ((total + u - 1) / u) * rows * kPairTile) * sizeof(float);
    };
    if (have_scratch) {
        U = (total + pairs - 1) / pairs;
        if (U < 2) U = g.SB < 2 ? g.SB : 2;
        while (bytes(U) > avail) U++;  // a workspace too small for the partial tiles: longer runs; whole tiles need none
    }
    g.U = U;
    g.grid_pairs = (total + U - 1) / U;
    g.partial_bytes = bytes(U);
    return g;
}

// What a GEMM kernel left to be finished: tiles in several segments, a row that goes through a norm, q, k and v on their way to the cache.
template <int ODT, int MODE> static int launch_finish(const PairParams& p, unsigned tiles, const PairFinish& fin, cudaStream_t st) {
    if (fin.left != nullptr && p.XT == 1) {
        *fin.left = PairLeft();
        fin.left->partial = p.by_tile || p.U % p.SB != 0 ? p.partial : nullptr;
        fin.left->part_rows = p.part_rows;
        fin.left->SB = p.SB;
        fin.left->U = p.U;
        fin.left->by_tile = p.by_tile;
        for (int i = 1; i < 3; i++) fin.left->tile0[i] = p.wt_end[i - 1];
        return set_status(NVE_OK);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (pdl_enabled()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    cudaError_t e = cudaSuccess;
    if (fin.rope != nullptr) {
        cfg.gridDim = dim3(tiles, static_cast<unsigned>((p.part_rows + 7) / 8));
        cfg.blockDim = dim3(kPairTile / 8, 8);
        e = cudaLaunchKernelEx(&cfg, gemm_pair_reduce_rope_kernel, p, *fin.rope);
        count_launch();
    } else if (fin.norm_w != nullptr) {
        cfg.gridDim = dim3(static_cast<unsigned>(p.M));
        const bool wide = p.M <= sm_count();
        cfg.blockDim = dim3(wide ? kPairNormThreads : 256);
        e = cudaLaunchKernelEx(&cfg, wide ? gemm_pair_reduce_norm_kernel : gemm_pair_reduce_norm_rows_kernel, p, fin.norm_w, fin.normed, fin.eps);
        count_launch();
    } else if (p.by_tile || p.U % p.SB != 0) {
        const unsigned cuts = static_cast<unsigned>((p.total - 1) / p.U);  // boundaries of two runs; no tile has more than one
        const bool cut = !p.by_tile && p.U >= p.SB && cuts > 0;
        cfg.gridDim = dim3(cut ? cuts : tiles, static_cast<unsigned>((p.part_rows + 3) / 4));
        cfg.blockDim = dim3(MODE == kPairSilu ? kPairTile / 8 : kPairTile / 4, MODE == kPairSilu ? 8 : 4);
        if (MODE == kPairSilu) cfg.gridDim.y = static_cast<unsigned>((p.part_rows + 7) / 8);
        e = cudaLaunchKernelEx(&cfg, cut ? gemm_pair_reduce_kernel<ODT, MODE, true> : gemm_pair_reduce_kernel<ODT, MODE, false>, p);
        count_launch();
    }
    return set_cuda_status(e);
}

template <int ODT, int MODE>
static int launch_pair(const PairParams& p, const PairPlan& g, const CUtensorMap& xmap, int smem, const PairFinish& fin, cudaStream_t st) {
    auto kern = gemm_w4a16_pair_kernel<ODT, MODE>;
    if (int s = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kPairSmemMax); s != NVE_OK) return s;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(2 * g.grid_pairs));
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (pdl_enabled()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p, xmap);
    count_launch();
    if (e != cudaSuccess) return set_cuda_status(e);
    return launch_finish<ODT, MODE>(p, static_cast<unsigned>(g.tiles), fin, st);
}

// Outputs and matrices of a call, common to the kernels
static void set_matrices(PairParams& p, const PairMat* mats, int num_mats, int M, int K, void* partial, const PairFinish& fin) {
    int wt = 0;
    p.sc16 = (K % 128) == 0;
    const int rows = fin.silu ? kPairTile / 2 : kPairTile;
    for (int i = 0; i < 3; i++) {
        const PairMat& m = mats[i < num_mats ? i : 0];
        p.nib[i] = m.nib;
        p.sc[i] = m.sc;
        p.Y[i] = m.Y;
        p.Nm[i] = i < num_mats ? m.N : 0;
        if (i < (fin.silu ? 1 : num_mats)) wt += (m.N + rows - 1) / rows;
        p.wt_end[i] = wt;
        if (!aligned(m.sc, 16)) p.sc16 = 0;
        if (!aligned(m.Y, 4)) p.y2 = 1;
    }
    p.res = fin.res;
    if (!aligned(fin.res, 4)) p.y2 = 1;
    p.y8 = aligned(fin.res, 8);
    for (int i = 0; i < num_mats; i++)
        if (!aligned(mats[i].Y, 8) || (mats[i].N & 3) != 0) p.y8 = 0;
    p.partial = static_cast<float*>(partial);
    p.M = M;
    p.K = K;
    p.nb = K / 32;
}
// f(ODT, MODE) of a call
template <typename F> static int by_finish(const PairFinish& fin, int y_dtype, F f) {
    using std::integral_constant;
    const integral_constant<int, kPairPlain> plain;
    if (fin.silu) return f(integral_constant<int, NVE_DT_F16>(), integral_constant<int, kPairSilu>());
    if (fin.norm_w != nullptr) return f(integral_constant<int, NVE_DT_F16>(), plain);  // the add is in the second kernel
    if (fin.res != nullptr) return f(integral_constant<int, NVE_DT_F16>(), integral_constant<int, kPairAdd>());
    if (y_dtype == NVE_DT_F32) return f(integral_constant<int, NVE_DT_F32>(), plain);
    if (y_dtype == NVE_DT_F16) return f(integral_constant<int, NVE_DT_F16>(), plain);
    return f(integral_constant<int, NVE_DT_BF16>(), plain);
}

size_t rows_partial_bytes(const int* Ns, int num_mats, int M, int K, bool silu) { return rows_plan(Ns, num_mats, M, K, silu).partial_bytes; }

bool gemm_rows_try(const void* X, int x_dtype, const PairMat* mats, int num_mats, int y_dtype, int M, int K, void* partial, size_t avail,
                   cudaStream_t st, const PairFinish& fin, int* status) {
    int Ns[3] = {0, 0, 0};
    for (int i = 0; i < num_mats; i++) Ns[i] = mats[i].N;
    const RowsPlan r = rows_plan(Ns, num_mats, M, K, fin.silu);
    if (r.grid == 0 || partial == nullptr || r.partial_bytes > avail) return false;
    PairParams p = {};
    set_matrices(p, mats, num_mats, M, K, partial, fin);
    p.NB = p.part_rows = M;
    p.XT = 1;
    p.SB = r.SB;
    p.U = r.U;
    p.total = r.total;
    p.by_tile = 1;
    const uint16_t* x = static_cast<const uint16_t*>(X);
    int s;
    if (fin.silu) s = launch_rows<NVE_DT_F16, true>(p, r, x, st);
    else s = x_dtype == NVE_DT_F16 ? launch_rows<NVE_DT_F16, false>(p, r, x, st) : launch_rows<NVE_DT_BF16, false>(p, r, x, st);
    if (s == NVE_OK)
        s = by_finish(fin, y_dtype, [&](auto odt, auto mode) { return launch_finish<odt.value, mode.value>(p, static_cast<unsigned>(r.tiles), fin, st); });
    *status = s;
    return true;
}

int gemm_pair(const uint16_t* X, const PairMat* mats, int num_mats, int y_dtype, int M, int K, void* partial, size_t avail, cudaStream_t st,
              const PairFinish& fin) {
    // partial tiles are read four floats at a time: of a workspace that is not aligned to that, the part from the first boundary on
    if (const size_t over = reinterpret_cast<uintptr_t>(partial) % 16; over != 0) {
        partial = static_cast<unsigned char*>(partial) + (16 - over);
        avail -= std::min(avail, 16 - over);
    }
    int Ns[3] = {0, 0, 0};
    for (int i = 0; i < num_mats; i++) Ns[i] = mats[i].N;
    const PairPlan g = pair_plan(Ns, num_mats, M, K, partial != nullptr, avail, fin.silu);
    // More than kFewRows rows on one tile per pair of SMs, with nothing that needs a finishing launch anyway, stay here: one launch against two
    // (16 rows, us: 2000 x 512 3.6 here, 4.4 in the kernel for few rows, 16384 x 1024 6.7 and 7.3, 18944 x 4096 15.5 and 16.9; where the
    // runs cut tiles, 17000 x 4096 17.6 and 16.6).
    const bool one_launch = M > kFewRows && g.U == g.SB && fin.norm_w == nullptr && fin.rope == nullptr;
    int status;
    if (!one_launch && gemm_rows_try(X, NVE_DT_F16, mats, num_mats, y_dtype, M, K, partial, avail, st, fin, &status)) return status;
    PairParams p = {};
    if (g.tiles * g.SB > 0x3FFFFFFFll) return set_status(NVE_ERR_BAD_SHAPE);
    CUtensorMap xmap;
    if (!pair_x_map(&xmap, X, K, M, g.NB / 2)) return set_status(NVE_ERR_CUDA);
    set_matrices(p, mats, num_mats, M, K, partial, fin);
    p.NB = g.NB;
    p.part_rows = M < g.NB ? M : g.NB;
    p.XT = g.XT;
    p.SB = g.SB;
    p.U = static_cast<int>(g.U);
    p.total = static_cast<int>(g.tiles * g.SB);
    // Accumulator sets = issuing warps: a step costs an issuing warp about a thousand cycles of waiting and issuing, the
    // MMAs themselves 8 * NB / 2.  The sets of a step follow its index in the segment.
    // Up to 64 rows the third set is there for the sums: an MMA rounds its accumulator towards zero, so that the error of a sum grows with the
    // length of its chain (4096 x 4096, 24 rows, against 64 bits: 4.6e-7 of the result, 6.4e-7 with two sets).  It takes an operand
    // slot's columns (8B layer, us, one / two / three sets: 24 rows 67.2 / 61.5 / 61.4, 61 rows 72.9 / 67.6 / 68.6).
    p.W = g.NB <= 64 ? 3 : (g.NB <= 128 ? 2 : 1);
    p.slots = min(7, (512 - p.W * p.NB) / kPairStepCols);
    // shared memory: the X rows of a step take NB * 128 bytes per CTA; at 256 rows five of them and two raw units
    // (four steps), for narrow tiles up to twelve steps of X and eight raw units, which is what hides HBM latency
    const int extra = fin.silu ? kPairSiluBytes : 0;
    p.raw = g.NB > 192 ? 2 : (g.NB > 96 ? 4 : (g.NB > 32 ? 6 : 8));
    p.xslots = min(12, (kPairSmemMax - 1024 - extra - p.raw * kRawBytes) / (p.NB * 128));
    const int smem = 1024 + p.xslots * p.NB * 128 + p.raw * kRawBytes + extra;
    return by_finish(fin, y_dtype, [&](auto odt, auto mode) { return launch_pair<odt.value, mode.value>(p, g, xmap, smem, fin, st); });
}

bool pair_norm_fits(int N) { return (N & 7) == 0 && N <= 8 * 256 * kPairNormChunks; }

int gemm_pair_error(bool reset) {
    int v = 0;
    if (cudaError_t e = cudaMemcpyFromSymbol(&v, g_pair_error, sizeof(int)); e != cudaSuccess) {
        set_cuda_status(e);
        return -1;
    }
    if (reset && v != 0) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_pair_error, &zero, sizeof(int));
    }
    return v;
}

}  // namespace nve
