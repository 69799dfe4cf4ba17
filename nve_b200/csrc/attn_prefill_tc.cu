// Causal attention of a block of new positions on the 5th-generation tensor cores: the form of attn_prefill_mma.cu's work for
// blocks that fill the SMs with tiles of 128 query rows.
//
// One CTA per SM takes one or two tiles of 128 query rows of one KV head (rows as there: (position, head) pairs, all heads of the group
// share the staged K/V) and walks the cached positions in steps of 128.  Both products are tcgen05.mma (cta_group::1, M = 128):
//   S = Q . K^T    operands in shared memory (TMA, 128-byte swizzle), S in tensor memory
//   O += P . V     P in f16 in tensor memory, over the columns of S; V in shared memory as it lies in the cache (rows of dims:
//                  the "MN-major" form of the B operand); O stays in tensor memory
// Two threads share a row, each with half of its columns in registers: no shuffles, one number exchanged per step.
//
// Roles (608 threads): warps 0-7 and 8-15 softmax, rescaling and epilogue of tile 0 and 1, warps 16 and 17 issue their MMAs, warp 18 the
// TMA loads.  TMEM: S0 | S1 | O0 | O1, 128 columns each.  Every wait is bounded in time; an expired one makes NaN of the CTA's rows.
//
// A commit behind S of step j covers every product issued before it, that of P of step j - 1 among them: whoever sees that S may
// overwrite it and may rescale O.
//
// What bounds it: the chain of a step.  8B, 1777 rows: 0.28 of the tensor pipe's cycles; from S to P 2900
// cycles (exponentials 2000: both tiles compute them at the same time), the two products with their waits 2000, start and end of a CTA
// 6000.  Against tiles of 64 rows on mma.sync (us): 1777 rows 107 -> 41, 600 rows 21.4 -> 13.8, 300 rows 11.9 -> 9.4, behind 1000 positions
// 39.5 -> 24.7; 24 heads over 8, 300 rows at 700 26.2 -> 23.2.  Tried, where this form took 46 with 1777 rows (a row sum that had to convert P
// back): one thread per row (54.8: its chain is twice as long), one warp issuing for both tiles (50.9), the second tile half a step behind the first
// (41.5 against 40.5), positions split over a cluster of two
// or four (300 rows at 700 21 to 22, but the merge through distributed shared memory makes everything shorter slower, and its code all).
// Error against 64 bits (2-norm over six random inputs, tiles of 64 / this): 300 rows 2.433e-4 / 2.442e-4, 600 2.474e-4 / 2.484e-4, 1777 2.532e-4 /
// 2.542e-4, 1000 at 500 2.776e-4 / 2.785e-4; 24 over 8 heads, 300 at 700 2.073e-4 both; heads of 64, 700 rows 2.478e-4 / 2.488e-4, 300 at 400 2.751e-4 /
// 2.765e-4.  Both round p to f16 for the product (3, 5, 6 and 7 heads: two numbers) and sum it in f32; which p the running maximum makes exact
// differs with the length of a step.  A sum of the rounded p has 0.45 % less here and up to ten times as much where one key dominates thousands of equal ones.
#include <cuda.h>

#include "attn_mma.cuh"
#include "attn_params.cuh"

namespace nve {

constexpr int kTcKeys = 128;     // cached positions per step
constexpr int kTcSoftmax = 512;  // threads: two per query row
constexpr int kTcThreads = kTcSoftmax + 96;
constexpr int kTcMmaWarp = 16, kTcLoadWarp = 18;  // an MMA warp per tile
constexpr unsigned long long kTcWaitLimitNs = 50ull * 1000 * 1000;  // a legitimate wait lasts microseconds

struct TcBars {
    uint64_t qfull[2], kfull[2], kempty[2], vfull[2], vempty[2], s[2], p[2], o[2];
};
struct TcShared {
    TcBars bars[2];  // of the first pass and of a second one: the last commits to kempty and vempty, which nobody waits for, may arrive late
    float pass[2][2][128];  // between the two threads of a row: [tile][half][row]
    uint32_t tmem;
    int abort, bad;
};

__device__ __forceinline__ uint32_t tc_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void tc_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void tc_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_addr(bar)) : "memory");
}
__device__ __forceinline__ void tc_expect(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_addr(bar)), "r"(bytes) : "memory");
}
// Wait of a whole, converged warp; the answer is the same for all its lanes.
__device__ __forceinline__ bool tc_wait(uint64_t* bar, unsigned parity, volatile int* abort) {
    const uint32_t a = tc_addr(bar);
    unsigned long long t0 = 0, t;
    for (unsigned spin = 0;; spin++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (__all_sync(0xffffffffu, done != 0)) return true;
        if ((spin & 63) == 63) {
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            if (__any_sync(0xffffffffu, t - t0 >= kTcWaitLimitNs || *abort != 0)) {
                *abort = 1;
                return false;
            }
        }
    }
}
__device__ __forceinline__ bool tc_elect() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void tc_load3(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(z), "r"(tc_addr(bar))
                 : "memory");
}
// Shared-memory operand with 128-byte swizzle.  K-major (Q, K): 1024 bytes between groups of eight rows (sbo), lbo unused.  MN-major (V: rows
// of 64 dims): sbo between groups of eight positions, lbo to the next 64 dims.
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(lbo >> 4) << 16;
    d |= static_cast<uint64_t>(sbo >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}
__device__ __forceinline__ void tc_mma_ss(bool issuer, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(static_cast<uint32_t>(issuer))
        : "memory");
}
__device__ __forceinline__ void tc_mma_ts(bool issuer, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(static_cast<uint32_t>(issuer))
        : "memory");
}
__device__ __forceinline__ void tc_commit(bool issuer, uint64_t* bar) {
    if (issuer) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_addr(bar)) : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float* v) {
    uint32_t* u = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]),
          "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]),
          "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t* u) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(u[0]),
                 "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]),
                 "r"(u[13]), "r"(u[14]), "r"(u[15])
                 : "memory");
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ float tc_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tc_softmax_barrier() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ void tc_tile_barrier(int t) { asm volatile("bar.sync %0, 256;" ::"r"(10 + t) : "memory"); }
// the two warps that share 32 rows of a tile
__device__ __forceinline__ void tc_rows_barrier(int rows) { asm volatile("bar.sync %0, 64;" ::"r"(2 + rows) : "memory"); }
// d = a * b + c on two numbers
__device__ __forceinline__ float2 tc_fma2(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(*reinterpret_cast<const uint64_t*>(&a)), "l"(*reinterpret_cast<const uint64_t*>(&b)), "l"(*reinterpret_cast<const uint64_t*>(&c)));
    return *reinterpret_cast<const float2*>(&d);
}
__device__ __forceinline__ float2 tc_add2(float2 a, float2 b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<const uint64_t*>(&a)), "l"(*reinterpret_cast<const uint64_t*>(&b)));
    return *reinterpret_cast<const float2*>(&d);
}

struct TcMaps {
    CUtensorMap q, k, v, out;
};
// Which rows and how many steps: the same for every thread
struct TcTiles {
    int groups, inv, PT;     // heads per KV head, ceil(65536 / groups), positions per tile
    int kvh, start;          // KV head, position of block row 0
    int pos0[2], npos[2], steps[2];  // first block row, rows (positions), steps
};

// What a CTA computes.  CAREFUL: a position that some rows do not see yet may hold an infinity or a NaN in v, which their zero
// probability would turn into NaN.  In the steps that are cut by the diagonal such elements are added by the threads of the rows that see them and
// are zeros in the product; everything else keeps its bits.
template <int HD, bool SPLIT, bool CAREFUL>
__device__ __forceinline__ void tc_block(const AttnParams& p, const TcMaps& maps, const TcTiles& tl, TcShared& sh, uint32_t base) {
    constexpr uint32_t kHalf = 128 * 128;             // 128 rows of 64 elements
    constexpr uint32_t kTile = kHalf * (HD / 64);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sq = base, sk = sq + 2 * kTile, sv = sk + 2 * kTile;
    const int n = max(tl.steps[0], tl.steps[1]);
    volatile int* abort = &sh.abort;
    TcBars& bars = sh.bars[CAREFUL ? 1 : 0];
    const uint32_t tmem = sh.tmem;

    if (warp < kTcMmaWarp) {
        // ------------------------------- softmax: row of the tile = TMEM lane; two threads a row, each half of the columns of S and of O
        const int t = warp >> 3, half = (warp >> 2) & 1, r = (warp & 3) * 32 + lane, rows_id = t * 4 + (warp & 3);
        const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t ts = tmem + lanes + t * 128, to = tmem + lanes + 256 + t * 128 + half * (HD / 2);
        float* mine = &sh.pass[t][half][r];
        const float* other = &sh.pass[t][half ^ 1][r];
        const int pos0 = t == 0 ? tl.pos0[0] : tl.pos0[1], steps = t == 0 ? tl.steps[0] : tl.steps[1];
        const bool valid = r < (t == 0 ? tl.npos[0] : tl.npos[1]) * tl.groups;
        const int lim = tl.start + pos0 + ((r * tl.inv) >> 16) + 1;  // positions that the row sees
        const int lim_min = tl.start + pos0 + 1;                     // ... the first row of the tile
        const int cut_from = tl.start + tl.pos0[0] + 1;              // ... of the CTA
        const float sl2 = p.scale * 1.4426950408889634f;    // exponentials in base 2
        float m = -1e30f, l = 0.0f;
        float extra[CAREFUL ? HD : 1];
        if (CAREFUL)
            for (int d = 0; d < HD; d++) extra[d] = 0.0f;
        bool ok = true;
        for (int j = 0; j < steps; j++) {
            if (ok && !tc_wait(&bars.s[t], j & 1, abort)) ok = false;  // (the steps go on: the warps of a row meet at barriers)
            tc_fence_after();
            float s[64];
            tc_ld32(ts + half * 64, s);
            tc_ld32(ts + half * 64 + 32, s + 32);
            tc_ld_wait();
            if ((j + 1) * kTcKeys > lim_min) {  // some row does not see the whole step
                const int seen = lim - j * kTcKeys - half * 64;
#pragma unroll
                for (int i = 0; i < 64; i++)
                    if (i >= seen) s[i] = -INFINITY;
            }
            float mx[4];
#pragma unroll
            for (int i = 0; i < 4; i++) mx[i] = fmaxf(s[i], s[i + 4]);
#pragma unroll
            for (int i = 8; i < 64; i += 8)
#pragma unroll
                for (int c = 0; c < 4; c++) mx[c] = fmaxf(fmaxf(mx[c], s[i + c]), s[i + 4 + c]);
            mx[0] = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            *mine = mx[0];
            tc_rows_barrier(rows_id);  // S is in registers: P may come over it
            const float mn = fmaxf(m, fmaxf(mx[0], *other) * sl2);  // finite: the masked value is below -1e30
            const float f = tc_exp2(m - mn);
            m = mn;
            l *= f;
            const bool grown = j > 0 && __any_sync(0xffffffffu, f != 1.0f);
            if (CAREFUL)
                for (int d = 0; d < HD; d++) extra[d] *= f;
            const float shift = SPLIT ? kAmSplitLog2 - m : -m;
            float2 sum[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
            for (int c = 0; c < 2; c++) {
                float* v = s + 32 * c;
                uint32_t hi[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    float2 e = tc_fma2(make_float2(v[2 * i], v[2 * i + 1]), make_float2(sl2, sl2), make_float2(shift, shift));
                    e.x = tc_exp2(e.x);
                    e.y = tc_exp2(e.y);
                    hi[i] = pack_f16x2(e.x, e.y);
                    sum[i & 1] = tc_add2(sum[i & 1], e);  // as they are, not as they are multiplied: f16 ends at 2^-24, and many equal small ones round the same way
                    if (SPLIT || CAREFUL) {
                        v[2 * i] = e.x;
                        v[2 * i + 1] = e.y;
                    }
                }
                tc_st16(ts + (SPLIT ? 64 * half + 32 * c : 32 * half + 16 * c), hi);
                if (SPLIT) {
#pragma unroll
                    for (int i = 0; i < 16; i++) hi[i] = pack_f16x2_rest(v[2 * i], v[2 * i + 1], hi[i]);
                    tc_st16(ts + 64 * half + 32 * c + 16, hi);
                }
                if (c == 0 && grown) {  // this thread's part of O; here half of S has left the registers
#pragma unroll
                    for (int d = 0; d < HD / 2; d += 32) {
                        float o[32];
                        tc_ld32(to + d, o);
                        tc_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] *= f;
                        tc_st16(to + d, reinterpret_cast<const uint32_t*>(o));
                        tc_st16(to + d + 16, reinterpret_cast<const uint32_t*>(o) + 16);
                    }
                }
            }
            l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
            if (CAREFUL && (j + 1) * kTcKeys > cut_from) {  // the same for both tiles
                if (ok && !tc_wait(&bars.vfull[j & 1], (j >> 1) & 1, abort)) ok = false;
                const uint32_t vb = sv + static_cast<uint32_t>(j & 1) * kTile;
                float ps[64];
                for (int i = 0; i < 64; i++) ps[i] = s[i];
                for (int i = 0; i < 64; i++) {
                    const int row = half * 64 + i;
                    if (j * kTcKeys + row >= lim) break;
                    for (int d = 0; d < HD; d += 2) {
                        uint32_t w;
                        const uint32_t o = vb + (d >> 6) * kHalf + row * 128 + ((((d & 63) >> 3) ^ (row & 7)) << 4) + (d & 7) * 2;
                        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(o) : "memory");
                        for (int b = 0; b < 2; b++)
                            if (((w >> (16 * b)) & 0x7C00u) == 0x7C00u)
                                extra[d + b] = fmaf(ps[i], Act16<NVE_DT_F16>::to_f32(static_cast<uint16_t>(w >> (16 * b))), extra[d + b]);
                    }
                }
                tc_softmax_barrier();
                for (uint32_t i = tid; i < kTile / 4; i += kTcSoftmax) {
                    uint32_t w;
                    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(vb + i * 4) : "memory");
                    if ((w & 0x7C00u) == 0x7C00u) w &= 0xFFFF0000u;
                    if ((w & 0x7C000000u) == 0x7C000000u) w &= 0xFFFFu;
                    asm volatile("st.shared.b32 [%0], %1;" ::"r"(vb + i * 4), "r"(w) : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_softmax_barrier();
            }
            tc_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) tc_arrive(&bars.p[t]);
        }
        // ---- epilogue: the commit behind the last product of the tile is one more phase of its S barrier.  The rows go to the
        // tile's Q, which nobody needs any more.
        if (steps > 0) {
            if (ok && !tc_wait(&bars.s[t], steps & 1, abort)) ok = false;
            tc_fence_after();
            tc_rows_barrier(rows_id);  // the last maxima have been read
            *mine = l;
            tc_rows_barrier(rows_id);
            l = half == 0 ? l + *other : *other + l;
            if (CAREFUL) {  // each of the two threads has the positions of its half: the sums change hands
                float* swap = reinterpret_cast<float*>(__cvta_shared_to_generic(sq + t * kTile)) + r * (HD / 2);
                for (int from = 0; from < 2; from++) {
                    if (half == from)
                        for (int d = 0; d < HD / 2; d++) swap[d] = extra[(from ^ 1) * (HD / 2) + d];
                    tc_rows_barrier(rows_id);
                    if (half != from)
                        for (int d = 0; d < HD / 2; d++) extra[half * (HD / 2) + d] += swap[d];
                    tc_rows_barrier(rows_id);
                }
                tc_tile_barrier(t);
            }
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            float probe[4] = {};
#pragma unroll
            for (int c = 0; c < HD / 2; c += 32) {
                float o[32];
                tc_ld32(to + c, o);
                tc_ld_wait();
                if (CAREFUL)
                    for (int d = 0; d < 32; d++) o[d] += extra[half * (HD / 2) + c + d];
#pragma unroll
                for (int d = 0; d < 32; d++) probe[d & 3] += o[d];
#pragma unroll
                for (int d = 0; d < 32; d += 8) {
                    const int dim = half * (HD / 2) + c + d;
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) w[i] = ok ? pack_f16x2(o[d + 2 * i] * inv, o[d + 2 * i + 1] * inv) : 0x7E007E00u;  // an expired wait is visible
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(sq + t * kTile + (dim >> 6) * kHalf + r * 128 + ((((dim & 63) >> 3) ^ (r & 7)) << 4)),
                                 "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                                 : "memory");
                }
            }
            if (!CAREFUL && valid && !(fabsf((probe[0] + probe[1]) + (probe[2] + probe[3])) <= 3.0e38f)) sh.bad = 1;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // for the store behind the CTA's next barrier
        }
    } else if (warp < kTcLoadWarp) {
        // -------------------------------------------------------------- MMA issue: the whole warp runs the loop, one lane issues
        const int t = warp - kTcMmaWarp, steps = t == 0 ? tl.steps[0] : tl.steps[1];
        const bool issuer = tc_elect();
        constexpr uint32_t kIdesc = (1u << 4) | ((128u >> 4) << 24);  // f32 accumulator, f16 operands, M = 128
        constexpr uint32_t kIdescS = kIdesc | ((128u >> 3) << 17), kIdescO = kIdesc | (1u << 16) | ((static_cast<uint32_t>(HD) >> 3) << 17);
        const uint32_t ds = tmem + t * 128, dst = tmem + 256 + t * 128;
        auto product_s = [&](int j) {
            const uint32_t a = sq + t * kTile, b = sk + static_cast<uint32_t>(j & 1) * kTile;
#pragma unroll
            for (int kk = 0; kk < HD / 16; kk++) {  // 16 dims: 32 bytes of the 128-byte rows
                const uint32_t o = (kk >> 2) * kHalf + (kk & 3) * 32;
                tc_mma_ss(issuer, ds, tc_desc(a + o, 16, 1024), tc_desc(b + o, 16, 1024), kIdescS, kk > 0);
            }
            tc_commit(issuer, &bars.s[t]);
            tc_commit(issuer, &bars.kempty[j & 1]);
            __syncwarp();
        };
        if (steps > 0 && tc_wait(&bars.qfull[t], 0, abort) && tc_wait(&bars.kfull[0], 0, abort)) {
            tc_fence_after();
            product_s(0);
            for (int j = 0; j < steps; j++) {
                if (!tc_wait(&bars.vfull[j & 1], (j >> 1) & 1, abort) || !tc_wait(&bars.p[t], j & 1, abort)) break;
                tc_fence_after();
                const uint32_t b = sv + static_cast<uint32_t>(j & 1) * kTile;
#pragma unroll
                for (int part = 0; part < (SPLIT ? 2 : 1); part++)
#pragma unroll
                    for (int kk = 0; kk < 8; kk++)  // 16 positions: two groups of eight rows
                        tc_mma_ts(issuer, dst, ds + (SPLIT ? 32 * (kk >> 1) + 8 * (kk & 1) + 16 * part : 8 * kk), tc_desc(b + kk * 2048, kHalf, 1024), kIdescO,
                                  j > 0 || kk > 0 || part > 0);
                tc_commit(issuer, j + 1 == steps ? &bars.s[t] : &bars.o[t]);
                tc_commit(issuer, &bars.vempty[j & 1]);
                __syncwarp();
                if (j + 1 == steps) break;
                // S of the next step comes over P: not before the product above is complete
                if (!tc_wait(&bars.kfull[(j + 1) & 1], ((j + 1) >> 1) & 1, abort) || !tc_wait(&bars.o[t], j & 1, abort)) break;
                tc_fence_after();
                product_s(j + 1);
            }
        }
    } else {
        // -------------------------------------------------------------- loads
        const bool issuer = tc_elect();
        bool ok = true;
        for (int j = 0; ok && j < n; j++) {
            const int b = j & 1;
            for (int kv = 0; ok && kv < 2; kv++) {
                uint64_t* full = kv == 0 ? &bars.kfull[b] : &bars.vfull[b];
                if (j >= 2) ok = tc_wait(kv == 0 ? &bars.kempty[b] : &bars.vempty[b], ((j >> 1) - 1) & 1, abort);
                if (ok && issuer) {
                    tc_expect(full, kTile);
                    for (int c = 0; c < HD / 64; c++)
                        tc_load3((kv == 0 ? sk : sv) + b * kTile + c * kHalf, kv == 0 ? &maps.k : &maps.v, 64 * c, j * kTcKeys, tl.kvh, full);
                    if (j == 0 && kv == 0)
                        for (int t = 0; t < 2; t++)
                            if (tl.npos[t] > 0) {
                                tc_expect(&bars.qfull[t], tl.PT * tl.groups * 128 * (HD / 64));  // (a box counts whole, also past the end of the block)
                                for (int c = 0; c < HD / 64; c++)
                                    tc_load3(sq + t * kTile + c * kHalf, &maps.q, 64 * c, tl.kvh * tl.groups, tl.pos0[t], &bars.qfull[t]);
                            } else if (CAREFUL) {
                                tc_arrive(&bars.qfull[t]);
                            }
                }
                __syncwarp();
            }
        }
    }
}
template <int HD, bool SPLIT>
__device__ __noinline__ void tc_block_careful(const AttnParams& p, const TcMaps& maps, const TcTiles& tl, TcShared& sh, uint32_t base) {
    tc_block<HD, SPLIT, true>(p, maps, tl, sh, base);
}

template <int HD, bool SPLIT>
__global__ void __launch_bounds__(kTcThreads, 1)
    attn_prefill_tc_kernel(const __grid_constant__ AttnParams p, const __grid_constant__ TcMaps maps, int groups, int PT, int inv, int per_cta) {
    extern __shared__ __align__(1024) unsigned char tc_raw[];
    __shared__ TcShared sh;
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t base = (tc_addr(tc_raw) + 1023u) & ~1023u;
    TcTiles tl;
    tl.groups = groups;
    tl.inv = inv;
    tl.PT = PT;
    tl.kvh = blockIdx.x;
    tl.start = p.seq_len - 1;
    const int tile2 = static_cast<int>(gridDim.y - 1 - blockIdx.y);  // the longest prefixes first
#pragma unroll
    for (int i = 0; i < 2; i++) {
        tl.pos0[i] = (per_cta * tile2 + i) * PT;
        tl.npos[i] = i < per_cta ? max(0, min(PT, p.rows - tl.pos0[i])) : 0;
        tl.steps[i] = tl.npos[i] > 0 ? (tl.start + tl.pos0[i] + tl.npos[i] + kTcKeys - 1) / kTcKeys : 0;
    }
    auto init = [&](TcBars& bars, int both) {  // tiles with steps; one may have one step less than the other, but the last ones are not waited for
        for (int i = 0; i < 2; i++) {
            tc_init(&bars.qfull[i], 1);
            tc_init(&bars.kfull[i], 1);
            tc_init(&bars.kempty[i], both);
            tc_init(&bars.vfull[i], 1);
            tc_init(&bars.vempty[i], both);
            tc_init(&bars.s[i], 1);
            tc_init(&bars.p[i], 8);  // the tile's warps
            tc_init(&bars.o[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    };
    if (tid == 0) {
        init(sh.bars[0], tl.steps[1] > 0 ? 2 : 1);
        sh.abort = sh.bad = 0;
    }
    if (warp == kTcMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_addr(&sh.tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp == kTcLoadWarp && (tid & 31) < 4)
        asm volatile("prefetch.tensormap [%0];" ::"l"((tid & 31) == 0 ? &maps.q : ((tid & 31) == 1 ? &maps.k : ((tid & 31) == 2 ? &maps.v : &maps.out))) : "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    pdl_launch_dependents();
    tc_block<HD, SPLIT, false>(p, maps, tl, sh, base);
    __syncthreads();
    if (sh.bad && !sh.abort) {  // every product and every load has been waited for, nothing has been stored: q is as it was, also where out is the same memory
        TcTiles all = tl;
        all.steps[0] = all.steps[1] = max(tl.steps[0], tl.steps[1]);  // (a step that no row of a tile sees adds zeros)
        if (tid == 0) init(sh.bars[1], 2);
        __syncthreads();
        tc_block_careful<HD, SPLIT>(p, maps, all, sh, base);
        __syncthreads();
    }
    // By TMA: sixteen bytes per lane straight to 32 different rows took 4000 cycles.  Rows behind the block's last are outside the map.
    const int t = warp >> 3;
    if (warp < kTcMmaWarp && (tid & 255) == 0 && (t == 0 ? tl.npos[0] : tl.npos[1]) > 0) {
        constexpr uint32_t kHalf = 128 * 128;
        for (int c = 0; c < HD / 64; c++)
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(&maps.out),
                         "r"(base + t * (kHalf * (HD / 64)) + c * kHalf), "r"(64 * c), "r"(tl.kvh * groups), "r"(t == 0 ? tl.pos0[0] : tl.pos0[1])
                         : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    if (*static_cast<volatile int*>(&sh.abort)) {  // copies and products may still be under way: give them time
        for (int i = 0; i < 100; i++) __nanosleep(10000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kTcMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem), "r"(512) : "memory");
    }
}

using TcEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static TcEncodeFn tc_encode_fn() {
    static TcEncodeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<TcEncodeFn>(f);
    }();
    return fn;
}
// f16 [z][y][x], 64 elements of x per box, 128-byte swizzle, zeros outside
static bool tc_map(CUtensorMap* map, const uint16_t* ptr, long long x, long long y, long long z, long long sy, long long sz, int by, int bz) {
    TcEncodeFn fn = tc_encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(x), static_cast<cuuint64_t>(y), static_cast<cuuint64_t>(z)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(sy) * 2, static_cast<cuuint64_t>(sz) * 2};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(by), static_cast<cuuint32_t>(bz)}, estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<uint16_t*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int HD, bool SPLIT> static bool launch_tc(const AttnParams& p, int per_cta, cudaStream_t st, cudaError_t& err) {
    const int groups = p.num_heads / p.num_kv_heads, PT = 2 * (64 / groups);
    const int tiles = (p.rows + per_cta * PT - 1) / (per_cta * PT), inv = (65536 + groups - 1) / groups;  // r * inv >> 16 = r / groups below 128
    const long long end = p.seq_len - 1 + p.rows;  // positions behind the block are never read
    TcMaps maps;
    if (!tc_map(&maps.q, p.q, HD, p.num_heads, p.rows, HD, p.row_stride, groups, PT) ||
        !tc_map(&maps.k, p.k_cache, HD, end, p.num_kv_heads, HD, static_cast<long long>(p.kv_stride) * HD, kTcKeys, 1) ||
        !tc_map(&maps.out, p.out, HD, p.num_heads, p.rows, HD, p.row_stride, groups, PT) ||
        !tc_map(&maps.v, p.v_cache, HD, end, p.num_kv_heads, HD, static_cast<long long>(p.kv_stride) * HD, kTcKeys, 1))
        return false;
    constexpr int smem = 6 * 128 * HD * 2 + 1024;
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(attn_prefill_tc_kernel<HD, SPLIT>), smem) != NVE_OK) {
        err = cudaErrorInvalidValue;
        return true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.dynamicSmemBytes = smem;
    cfg.gridDim = dim3(p.num_kv_heads, tiles);
    cfg.blockDim = dim3(kTcThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (pdl_enabled()) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    err = cudaLaunchKernelEx(&cfg, attn_prefill_tc_kernel<HD, SPLIT>, p, maps, groups, PT, inv, per_cta);
    return true;
}

bool attn_prefill_tc_try(const AttnParams& p, int head_dim, cudaStream_t st, cudaError_t& err) {
    const int groups = p.num_heads / p.num_kv_heads;
    if (groups > 64 || (head_dim != 64 && head_dim != 128)) return false;
    if (!aligned(p.q, 16) || !aligned(p.k_cache, 16) || !aligned(p.v_cache, 16) || !aligned(p.out, 16) || (p.row_stride & 7) != 0) return false;
    const bool split = am_split(groups);
    // Where tiles of 128 rows take seven tenths of the SMs they are always the faster ones (us, tiles of 64 / this, 32 over 8 heads of 128 where nothing else
    // is said: 385 rows 14.9 / 10.6, heads of 64 9.6 / 8.5).  With fewer it depends on whether the other form has more tiles than SMs
    // (tiles64 > sm): if not, it gives each to two CTAs from 449 positions on.
    //  - It has: this form from 257 positions on (289 rows 11.8 / 9.4).  Heads of 64: from 513 on (310 rows at 203 11.6 / 10.5) and where its tiles share most
    //    SMs or are of similar length (16 over 4 heads, 152 tiles, 608 rows at 0 9.9 / 10.6, at 192 12.8 / 13.4, at 592 19.3 / 17.9).
    //  - It has not: while dealing the positions out saves it little and this form has three eighths of the SMs, heads of 64 three sevenths
    //    (224 rows at 216 11.2 / 11.6, at 225 13.5 / 11.4, at 976 24.1 / 22.7, at 2276 41.9 / 41.1, at 4108 66.8 / 67.1; heads of 64, 193 rows at 1007
    //    15.1 / 18.0, 225 rows at 215 7.7 / 9.4, at 375 12.2 / 10.8, at 975 19.0 / 18.0).
    const long long PT = 2 * (64 / groups), ctas = (p.rows + PT - 1) / PT * p.num_kv_heads, sm = sm_count();
    const long long tiles64 = (p.rows + PT / 2 - 1) / (PT / 2) * p.num_kv_heads;
    const int positions = p.seq_len - 1 + p.rows, steps = (positions + kTcKeys - 1) / kTcKeys;
    if (ctas * 10 < sm * 7) {
        if (head_dim == 128 ? (tiles64 > sm ? positions <= 256 : ctas * 8 < sm * 3 || positions <= 448 || positions > 2560)
                            : positions <= 512 || (tiles64 * 25 < sm * 27 &&
                                                   (tiles64 > sm ? 2 * p.rows > positions : ctas * 7 < sm * 3 || positions > 2560)))
            return false;
    }
    // Two tiles in a CTA take 1.3 to 1.45 times as long as one: from two waves of single tiles on, or where a second wave would be as long as
    // the first (us, one / two: 1000 rows 23.1 / 25.4, at 500 38.2 / 36.4, at 1000 53.0 / 46.1; 1300 rows 35.8 / 31.0; 1777 rows 56.5 / 40.9; 24 over 8 heads,
    // whose steps are longer, 1000 rows at 1000 58.0 / 58.3, 1300 rows 32.0 / 39.0, 1777 rows 56.5 / 51.8).
    const int per_cta = ctas > 2 * sm || (ctas > sm && steps >= 12 && !split) ? 2 : 1;
    if (head_dim == 128) return split ? launch_tc<128, true>(p, per_cta, st, err) : launch_tc<128, false>(p, per_cta, st, err);
    return split ? launch_tc<64, true>(p, per_cta, st, err) : launch_tc<64, false>(p, per_cta, st, err);
}

}  // namespace nve
