// Decode attention that streams: RoPE + K/V write + single-query GQA attention (+ optional int8 codes of the output) where
// there is more K/V to read than the latency kernel (attn_decode_mma.cu) keeps in flight -- many sequences, or one with a
// long context -- and the plain flash-decode form of the same arithmetic.
//
// What bounds it is HBM: 2 * nkv * hd * 2 bytes per cached position, a few instructions per 8 KB.  The former kernel for many
// sequences loaded a tile of 16 positions per warp into registers, multiplied it and only then asked for the next: 4.3 TB/s
// at 64 sequences, and one sequence per CTA whatever its length; a long single sequence ran on 64 of the 148 SMs.  Here
//   * a CTA of NW = 4 or 8 warps serves one (sequence, KV head) with all its query heads (rows of mma.sync.m16n8k16; G <= 8),
//     each warp with a private ring of NS 16-position tiles filled by cp.async: two to three tiles (16 - 24 KB) per warp are
//     always under way, eight warps per SM, 130 KB or more per SM;
//   * the positions of a unit are split over a cluster of 1 .. 8 CTAs (distributed-shared-memory merge in rank 0, as in the
//     latency kernel), chosen so that the grid fills the GPU whatever the batch; the slices follow the sequence's own length;
//   * the position words are read before the grid dependency resolves, for the slices and the RoPE row, and again after it (both
//     are redone in the rare case that they changed); the first tiles are requested then.
// Tile layout in shared memory: rows of HD f16, 16-byte chunks XORed with the row, so that ldmatrix reads eight rows of a
// chunk from eight bank groups; K as the B operand of q.K^T as it is, V through ldmatrix.trans for p.V.
#include <cooperative_groups.h>

#include <atomic>
#include <cstddef>

#include "attn_mma.cuh"
#include "attn_params.cuh"

namespace cg = cooperative_groups;

namespace nve {

constexpr int kAsMaxCluster = 8;
constexpr unsigned long long kAsWaitLimitNs = 20ull * 1000 * 1000;  // a legitimate wait lasts microseconds

template <int HD> __device__ __forceinline__ uint32_t as_off(int r, int c) {
    return static_cast<uint32_t>(r * (HD * 2) + ((c ^ (r & 7)) << 4));
}
__device__ __forceinline__ uint32_t as_smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void as_cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void as_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void as_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
template <bool TRANS> __device__ __forceinline__ void as_ldm4(uint32_t addr, uint32_t (&r)[4]) {
    if constexpr (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr)
                     : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr)
                     : "memory");
}
__device__ __forceinline__ float as_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <int HD, int G, int NW, int NS> struct AsSmem {
    __align__(16) unsigned char ring[NW][NS][2][16 * HD * 2];  // tiles of K and V; after the loop a warp's partial
    __align__(16) uint16_t q[8][HD];                                        // rotated q, rows g >= G zero
    __align__(16) uint16_t knew[HD], vnew[HD];
    float wm[NW][G], wl[NW][G];
    __align__(8) unsigned long long pbar;
    AdCtaPartial<HD, G> parts[1];  // rank 0 of a cluster: one per rank (the launch adds the room for the others)
};

// Fused: blockIdx.y is one of `rows` independent sequences (one sequence: rows <= 1).  Else: one of `rows` query rows over one
// cache, row r attends to seq_len + r positions.  blockIdx.x = KV head * csize + rank.
// LEFT (fused): q, k and v are a product whose segments are not summed yet; with heads of 64 as many CTAs as otherwise still fit an SM (us a layer, hidden
// 2048, 64 sequences of 300, finished / LEFT with three CTAs of four warps / with four: one head per KV head 49.3 / 50.1 / 47.9, four 51.7 / 51.3 / 49.7; of
// 1000 59.9 / 58.0 / 57.9 and 61.7 / 59.2 / 59.8).
template <int HD, int G, int NW, int NS, bool FUSED, bool LEFT>
__global__ void __launch_bounds__(32 * NW, LEFT && HD == 64 ? 16 / NW : 8 / NW) attn_stream_mma_kernel(const AttnParams pin, int csize) {
    AttnParams p = pin;
    int seq_len_row = p.seq_len;
    const long long b = blockIdx.y;
    if constexpr (FUSED) {
        p.q += b * (static_cast<long long>(p.num_heads) * HD);
        p.out += b * (static_cast<long long>(p.num_heads) * HD);
        p.k_new += b * (static_cast<long long>(p.num_kv_heads) * HD);
        p.v_new += b * (static_cast<long long>(p.num_kv_heads) * HD);
        p.k_cache += b * p.cache_stride;
        p.v_cache += b * p.cache_stride;
        p.d_pos += b;
        p.d_seq_len += b;
    } else {
        p.q += b * p.row_stride;
        p.out += b * p.row_stride;
        seq_len_row += static_cast<int>(b);
    }
    constexpr int HALF = HD / 2, DC = HD / 8, NT = HD / 8;
    constexpr bool SPLIT = am_split(G);
    static_assert((HD == 64 || HD == 128) && G >= 1 && G <= 8, "head_dim 64 or 128, up to 8 query heads per KV head");
    static_assert(HD <= (32 * NW) && G * (HD + 8) * 4 <= NS * 2 * 16 * HD * 2, "one element of v per thread; a partial fits its ring");
    extern __shared__ __align__(16) unsigned char as_raw[];
    AsSmem<HD, G, NW, NS>& sm = *reinterpret_cast<AsSmem<HD, G, NW, NS>*>(as_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int kvh = static_cast<int>(blockIdx.x) / csize, rank = static_cast<int>(blockIdx.x) - kvh * csize;
    const int h0 = kvh * G;
    constexpr uint32_t kPartBytes = (G * HD + 2 * G) * 4;
    if (csize > 1) {
        if (rank == 0 && tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(as_smem(&sm.pbar)));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(as_smem(&sm.pbar)), "r"((csize - 1) * kPartBytes) : "memory");
        }
        cg::this_cluster().barrier_arrive();  // matched in front of the push: rank 0 runs and its mbarrier is set up
    }
    const uint16_t* kh = p.k_cache + static_cast<long long>(kvh) * p.kv_stride * HD;
    const uint16_t* vh = p.v_cache + static_cast<long long>(kvh) * p.kv_stride * HD;

    // ---- this warp's tiles: t_begin + 16 * (warp + NW * i) of the CTA's slice (whole tiles but for the last)
    int seq_len = max(0, min(p.d_seq_len != nullptr ? *p.d_seq_len : seq_len_row, p.kv_stride));
    int pos = FUSED ? *p.d_pos : -1;
    int t_begin, t_end;
    auto slice = [&]() {
        const int chunk = ((seq_len + csize - 1) / csize + 15) & ~15;
        t_begin = min(seq_len, rank * chunk);
        t_end = min(seq_len, t_begin + chunk);
    };
    const uint32_t ring = as_smem(sm.ring[warp]);
    const int lr = lane / DC, lc = lane % DC;  // row and chunk of this lane's first copy; 32 / DC rows per pass
    auto load = [&](int p0, int st) {
        if (p0 < t_end) {
            const uint32_t dst = ring + st * (2 * 16 * HD * 2);
#pragma unroll
            for (int i = 0; i < DC / 2; i++) {
                const int r = lr + i * (32 / DC);
                const long long src = static_cast<long long>(min(p0 + r, t_end - 1)) * HD + lc * 8;  // rows past the end repeat the last: masked
                as_cp16(dst + as_off<HD>(r, lc), kh + src);
                as_cp16(dst + 16 * HD * 2 + as_off<HD>(r, lc), vh + src);
            }
        }
        as_commit();
    };
    slice();
    const int qe = tid % HALF, qh = tid / HALF;  // this thread's element pairs (qe, qe + HALF) of the heads qh, qh + HPP, ...
    constexpr int HPP = (32 * NW) / HALF, QI = (G + HPP - 1) / HPP;
    uint16_t c16 = 0, s16 = 0;
    auto rope_row = [&]() {
        const long long row = pos >= 0 && pos < p.kv_stride ? pos : 0;
        c16 = p.cos_tab[row * HALF + qe];
        s16 = p.sin_tab[row * HALF + qe];
    };
    if constexpr (FUSED) rope_row();
    for (int i = tid; i < (8 - G) * HALF; i += (32 * NW)) reinterpret_cast<uint32_t*>(sm.q[G])[i] = 0;
    constexpr int E = LEFT ? 2 * QI + 3 : 1;
    const uint16_t* y[E];
    PairFeatures<E> features;
    if constexpr (LEFT) {
        int tile0[E], n[E];
#pragma unroll
        for (int j = 0; j < QI; j++) {
            const int h = qh + j * HPP;
            tile0[2 * j] = tile0[2 * j + 1] = p.left.tile0[0];
            n[2 * j] = (h0 + (h < G ? h : 0)) * HD + qe;
            n[2 * j + 1] = n[2 * j] + HALF;
            y[2 * j] = p.q + n[2 * j];
            y[2 * j + 1] = p.q + n[2 * j + 1];
        }
        tile0[E - 3] = tile0[E - 2] = p.left.tile0[1];
        tile0[E - 1] = p.left.tile0[2];
        n[E - 3] = kvh * HD + qe;
        n[E - 2] = n[E - 3] + HALF;
        n[E - 1] = kvh * HD + (tid < HD ? tid : 0);
        y[E - 3] = p.k_new + n[E - 3];
        y[E - 2] = p.k_new + n[E - 2];
        y[E - 1] = p.v_new + n[E - 1];
        features.find(p.left, static_cast<int>(b), tile0, n);
    }
    pdl_wait();
    uint16_t x0[QI], x1[QI], k0 = 0, k1 = 0, vv = 0;
    auto positions = [&]() {
        const int now = max(0, min(p.d_seq_len != nullptr ? *reinterpret_cast<const volatile int*>(p.d_seq_len) : seq_len_row, p.kv_stride));
        const int now_pos = FUSED ? *reinterpret_cast<const volatile int*>(p.d_pos) : -1;
        if (FUSED && now_pos != pos) {
            pos = now_pos;
            rope_row();
        }
        if (now != seq_len) {  // uniform over the CTA
            seq_len = now;
            slice();
        }
    };
    // Nothing of the cache before the wait: the launch in front may be writing it, and it may let its dependents start before it
    // has stored.  Behind q, k and v, which everything waits for: tiles requested before the wait hold them up where there is much
    // K/V (us per token with early tiles and so: 8B at 16384 positions 1772 and 1725; 3B, 7 sequences 1492 and 1459; 8B, 64
    // sequences 3314 and 3305; tiles right after the wait, in front of q: 1776, 1504 and 3344).  Only attention launches right behind one another
    // were shorter with early tiles: 7 sequences of 500 - 2000 8.9 us, 10.8 so.
    auto request = [&]() {
#pragma unroll
        for (int i = 0; i < NS; i++) load(t_begin + 16 * (warp + NW * i), i);
    };
    if constexpr (LEFT) {
        // No finishing launch of the GEMM in between: 3B, 7 sequences of up to 2000 positions 1308 -> 1254 us per step, 8B, 64 of up to 1024
        // 3242 -> 3195.  What counts is the order: the segments are found before the wait and requested first, K/V behind them and in front of
        // the sums (sums first: 1320), and the positions are read ahead all the same (1312 without).
        uint16_t x[E];
        features.sum(y, x, [&]() {
            positions();
            request();
        });
#pragma unroll
        for (int j = 0; j < QI; j++) {
            x0[j] = x[2 * j];
            x1[j] = x[2 * j + 1];
        }
        k0 = x[E - 3];
        k1 = x[E - 2];
        vv = x[E - 1];
    } else {
#pragma unroll
        for (int j = 0; j < QI; j++) {
            const int h = qh + j * HPP;
            const uint16_t* qp = p.q + static_cast<long long>(h0 + (h < G ? h : 0)) * HD;
            x0[j] = qp[qe];
            x1[j] = qp[qe + HALF];
        }
        if constexpr (FUSED) {
            const uint16_t* kp = p.k_new + static_cast<long long>(kvh) * HD;
            if (tid < HALF) {
                k0 = kp[qe];
                k1 = kp[qe + HALF];
            }
            if (tid < HD) vv = p.v_new[static_cast<long long>(kvh) * HD + tid];
        }
        positions();
        request();
    }
    const bool pos_ok = FUSED && pos >= 0 && pos < p.kv_stride;
    {
        // the rotation of the stand-alone RoPE kernel: same IEEE operations, same 16-bit rounding
        const float c = Act16<NVE_DT_F16>::to_f32(c16), sn = Act16<NVE_DT_F16>::to_f32(s16);
        auto rot = [&](uint16_t a, uint16_t bb, uint16_t& r0, uint16_t& r1) {
            const float f0 = Act16<NVE_DT_F16>::to_f32(a), f1 = Act16<NVE_DT_F16>::to_f32(bb);
            r0 = Act16<NVE_DT_F16>::from_f32(__fsub_rn(__fmul_rn(f0, c), __fmul_rn(f1, sn)));
            r1 = Act16<NVE_DT_F16>::from_f32(__fadd_rn(__fmul_rn(f0, sn), __fmul_rn(f1, c)));
        };
#pragma unroll
        for (int j = 0; j < QI; j++) {
            const int h = qh + j * HPP;
            if (h < G) {
                uint16_t r0 = x0[j], r1 = x1[j];
                if constexpr (FUSED) rot(x0[j], x1[j], r0, r1);
                sm.q[h][qe] = r0;
                sm.q[h][qe + HALF] = r1;
            }
        }
        if constexpr (FUSED) {
            if (tid < HALF) rot(k0, k1, sm.knew[qe], sm.knew[qe + HALF]);
            if (tid < HD) sm.vnew[tid] = vv;
        }
    }
    __syncthreads();
    pdl_launch_dependents();
    // one CTA per KV head stores the new row; the tile that covers `pos` takes it from shared memory
    if (FUSED && pos_ok && rank == 0 && tid < 2 * DC) {
        const int which = tid / DC, d = tid % DC;
        uint16_t* dst = (which == 0 ? p.k_cache : p.v_cache) + (static_cast<long long>(kvh) * p.kv_stride + pos) * HD;
        reinterpret_cast<uint4*>(dst)[d] = reinterpret_cast<const uint4*>(which == 0 ? sm.knew : sm.vnew)[d];
    }
    uint32_t qa[HD / 16][2];
#pragma unroll
    for (int kk = 0; kk < HD / 16; kk++) {
        qa[kk][0] = *reinterpret_cast<const uint32_t*>(&sm.q[g][16 * kk + 2 * t]);
        qa[kk][1] = *reinterpret_cast<const uint32_t*>(&sm.q[g][16 * kk + 2 * t + 8]);
    }
    const float sl2 = p.scale * 1.4426950408889634f;  // exponentials in base 2
    float m = -1e30f, l = 0.0f;                         // running maximum of row g, this lane's share of its sum
    float o[NT][2];
#pragma unroll
    for (int j = 0; j < NT; j++) o[j][0] = o[j][1] = 0.0f;

    int st = 0;
    for (int p0 = t_begin + 16 * warp; p0 < t_end; p0 += 16 * NW) {
        as_wait<NS - 1>();
        __syncwarp();
        const uint32_t kt = ring + st * (2 * 16 * HD * 2), vt = kt + 16 * HD * 2;
        if (pos_ok && pos >= p0 && pos < p0 + 16) {
            if (lane < 2 * DC) {
                const int which = lane / DC, d = lane % DC;
                const uint4 x = reinterpret_cast<const uint4*>(which == 0 ? sm.knew : sm.vnew)[d];
                // the rows past the end repeat the last one, which may be this one
                const int r1 = pos == t_end - 1 ? 16 : pos - p0 + 1;
                for (int r = pos - p0; r < r1; r++)
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"((which == 0 ? kt : vt) + as_off<HD>(r, d)), "r"(x.x), "r"(x.y),
                                 "r"(x.z), "r"(x.w)
                                 : "memory");
            }
            __syncwarp();
        }
        float s0[4] = {0, 0, 0, 0}, s1[4] = {0, 0, 0, 0}, s2[4] = {0, 0, 0, 0}, s3[4] = {0, 0, 0, 0};  // two chains per half tile
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
            uint32_t kb[4];  // positions 0-7 (kb[0], kb[1]) and 8-15 (kb[2], kb[3]), dims 16 kk .. + 15
            as_ldm4<false>(kt + as_off<HD>((lane & 7) + ((lane >> 4) << 3), 2 * kk + ((lane >> 3) & 1)), kb);
            const uint32_t a[4] = {qa[kk][0], 0, qa[kk][1], 0};
            mma_f16_16816((kk & 1) ? s2 : s0, a, kb[0], kb[1]);
            mma_f16_16816((kk & 1) ? s3 : s1, a, kb[2], kb[3]);
        }
        // this lane's four scores of row g: positions p0 + 2t, + 1, + 8, + 9
        float sc[4] = {(s0[0] + s2[0]) * sl2, (s0[1] + s2[1]) * sl2, (s1[0] + s3[0]) * sl2, (s1[1] + s3[1]) * sl2};
        if (p0 + 16 > t_end) {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (p0 + 2 * t + (e & 1) + 8 * (e >> 1) >= t_end) sc[e] = -INFINITY;
        }
        float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mn = fmaxf(m, mx);
        const float corr = as_exp2(m - mn);
        m = mn;
#pragma unroll
        for (int e = 0; e < 4; e++) sc[e] = as_exp2(SPLIT ? sc[e] - (mn - kAmSplitLog2) : sc[e] - mn);
        l = l * corr + ((sc[0] + sc[1]) + (sc[2] + sc[3]));
        uint32_t pa[4] = {pack_f16x2(sc[0], sc[1]), 0, pack_f16x2(sc[2], sc[3]), 0};
        if (SPLIT) {  // the rests in rows g + 8
            pa[1] = pack_f16x2_rest(sc[0], sc[1], pa[0]);
            pa[3] = pack_f16x2_rest(sc[2], sc[3], pa[2]);
        }
#pragma unroll
        for (int j = 0; j < NT; j += 2) {
            uint32_t vb[4];  // dims 8j .. + 7 (vb[0], vb[1]) and the next eight (vb[2], vb[3]) of the sixteen positions
            as_ldm4<true>(vt + as_off<HD>(lane & 15, j + (lane >> 4)), vb);
            float d0[4] = {o[j][0] * corr, o[j][1] * corr, 0, 0}, d1[4] = {o[j + 1][0] * corr, o[j + 1][1] * corr, 0, 0};
            mma_f16_16816(d0, pa, vb[0], vb[1]);
            mma_f16_16816(d1, pa, vb[2], vb[3]);
            o[j][0] = SPLIT ? d0[0] + d0[2] : d0[0];
            o[j][1] = SPLIT ? d0[1] + d0[3] : d0[1];
            o[j + 1][0] = SPLIT ? d1[0] + d1[2] : d1[0];
            o[j + 1][1] = SPLIT ? d1[1] + d1[3] : d1[1];
        }
        __syncwarp();  // every lane has read the tile
        load(p0 + 16 * NW * NS, st);
        st = st + 1 == NS ? 0 : st + 1;
    }

    // ---- level 1: the warps' partials meet in shared memory (each in its warp's own ring); level 2: rank 0 of the cluster
    as_wait<0>();
    __syncwarp();
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    constexpr int WR = HD + 8;  // floats per partial row
    if (g < G) {
        if (t == 0) {
            sm.wm[warp][g] = m;
            sm.wl[warp][g] = l;
        }
        float* wo = reinterpret_cast<float*>(sm.ring[warp]) + g * WR;
#pragma unroll
        for (int j = 0; j < NT; j++) *reinterpret_cast<float2*>(wo + 8 * j + 2 * t) = make_float2(o[j][0], o[j][1]);
    }
    __syncthreads();
    if (csize > 1) cg::this_cluster().barrier_wait();  // all CTAs of the cluster run
    AdCtaPartial<HD, G>* parts = sm.parts;
    auto finish = [&](int i, float a, float ss, bool arrived) {
        const uint16_t o16 = arrived ? Act16<NVE_DT_F16>::from_f32(ss == 0.0f ? 0.0f : a / ss) : static_cast<uint16_t>(0x7E00);  // NaN
        const long long oi = static_cast<long long>(h0) * HD + i;
        p.out[oi] = o16;
        if (p.out_q != nullptr) {
            // i advances by whole warps and HD is a multiple of 32: the 32 lanes of a warp hold one group
            float scale;
            const int qv = attn_quantize_lane(o16, scale);
            p.out_q[oi] = static_cast<int8_t>(qv);
            if (lane == 0) p.out_scales[oi >> 5] = scale;
        }
    };
    uint32_t remote = 0, remote_bar = 0;
    if (rank > 0) {
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(as_smem(&parts[rank])), "r"(0));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote_bar) : "r"(as_smem(&sm.pbar)), "r"(0));
    }
    auto post = [&](size_t off, float x) {
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(remote + static_cast<uint32_t>(off)),
                     "r"(__float_as_uint(x)), "r"(remote_bar)
                     : "memory");
    };
    using Part = AdCtaPartial<HD, G>;
#pragma unroll
    for (int i = tid; i < G * HD; i += (32 * NW)) {
        const int h = i / HD, d = i % HD;
        float mm = -1e30f, ss = 0.0f, a = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; w++) mm = fmaxf(mm, sm.wm[w][h]);
#pragma unroll
        for (int w = 0; w < NW; w++) {  // warps in ascending order
            const float c = as_exp2(sm.wm[w][h] - mm);
            ss = fmaf(sm.wl[w][h], c, ss);
            a = fmaf(reinterpret_cast<const float*>(sm.ring[w])[h * WR + d], c, a);
        }
        if (csize == 1) {
            finish(i, a, ss, true);
        } else if (rank == 0) {
            parts[0].acc[h][d] = a;
            if (d == 0) {
                parts[0].m[h] = mm;
                parts[0].s[h] = ss;
            }
        } else {
            post(offsetof(Part, acc) + (h * HD + d) * 4, a);
            if (d == 0) {
                post(offsetof(Part, m) + h * 4, mm);
                post(offsetof(Part, s) + h * 4, ss);
            }
        }
    }
    if (csize == 1 || rank != 0) return;
    __syncthreads();  // rank 0's own partial
    bool arrived = false;
    {
        const uint32_t bar = as_smem(&sm.pbar);
        unsigned long long t0 = 0, tn = 0;
        for (int spin = 0; !arrived; spin++) {
            uint32_t done;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar)
                : "memory");
            arrived = done != 0;
            if (!arrived && (spin & 63) == 63) {  // bounded in time: a partial that never arrives poisons the output
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tn));
                if (t0 == 0) t0 = tn;
                else if (tn - t0 > kAsWaitLimitNs) break;
            }
        }
    }
#pragma unroll
    for (int i = tid; i < G * HD; i += (32 * NW)) {
        const int h = i / HD, d = i % HD;
        float mm = -1e30f, ss = 0.0f, a = 0.0f;
        for (int r = 0; r < csize; r++) mm = fmaxf(mm, parts[r].m[h]);
        for (int r = 0; r < csize; r++) {  // ranks in ascending order
            const float c = as_exp2(parts[r].m[h] - mm);
            ss = fmaf(parts[r].s[h], c, ss);
            a = fmaf(parts[r].acc[h][d], c, a);
        }
        finish(i, a, ss, arrived);
    }
}

template <int HD, int G, int NW, int NS> constexpr int as_smem_bytes(int csize) {
    return static_cast<int>(sizeof(AsSmem<HD, G, NW, NS>) + (csize - 1) * sizeof(AdCtaPartial<HD, G>));
}
// A CTA of eight warps takes most of an SM: three stages where they fit next to the partials of eight ranks.
template <int HD, int G> constexpr int as_wide_stages() { return as_smem_bytes<HD, G, 8, 3>(8) <= 227 * 1024 ? 3 : 2; }

template <int HD, int G, int NW, int NS, bool FUSED, bool LEFT> struct AsLaunch {
    static void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, const AttnParams& p, int rows, int csize, cudaStream_t st) {
        cfg = {};
        cfg.dynamicSmemBytes = as_smem_bytes<HD, G, NW, NS>(csize);
        cfg.gridDim = dim3(p.num_kv_heads * csize, rows);
        cfg.blockDim = dim3(32 * NW);
        cfg.stream = st;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = csize;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    static int prepare() {
        return ensure_dynamic_smem(reinterpret_cast<const void*>(attn_stream_mma_kernel<HD, G, NW, NS, FUSED, LEFT>), as_smem_bytes<HD, G, NW, NS>(kAsMaxCluster));
    }
    // How many clusters of `csize` CTAs the current device holds at a time (clusters do not straddle the SM groups of the chip, so this
    // is less than SMs / csize: 15 clusters of 8 on 148 SMs); asked once per device.
    static int active(const AttnParams& p, int csize) {
        constexpr int kDevices = 64;
        static std::atomic<int> known[kDevices][kAsMaxCluster + 1];
        int dev = 0;
        const bool keep = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kDevices;
        int n = keep ? known[dev][csize].load(std::memory_order_relaxed) : 0;
        if (n == 0) {
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute attr[2];
            config(cfg, attr, p, 1, csize, nullptr);
            if (cudaOccupancyMaxActiveClusters(&n, attn_stream_mma_kernel<HD, G, NW, NS, FUSED, LEFT>, &cfg) != cudaSuccess || n < 1) n = 1;
            if (keep) known[dev][csize].store(n, std::memory_order_relaxed);
        }
        return n;
    }
    static cudaError_t launch(const AttnParams& p, int rows, int csize, cudaStream_t st) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        config(cfg, attr, p, rows, csize, st);
        if (pdl_enabled()) {
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.numAttrs = 2;
        }
        return cudaLaunchKernelEx(&cfg, attn_stream_mma_kernel<HD, G, NW, NS, FUSED, LEFT>, p, csize);
    }
};

// The split.  us per launch on B200 (HD 128, 4 heads per KV head; 4 warps x 3 stages, two CTAs per SM / 8 warps, one CTA per SM), as
// measured when it was chosen; back to back the chosen forms take 28.7, 27.6, 10.8, 14.7 and 14.7 now:
//   512 units of 256 - 1024 positions   one CTA per unit 30.7 / 40.1, clusters of two 48.9 / 59.5 (HBM floor 25.6)
//   160 units of 750 - 3000             34.8 / 28.8, clusters of two 30.2 / 35.6 (23.5)
//   56 units of 500 - 2000              clusters of four 10.7 / of two 10.7, one CTA per unit 18.5 / 15.0 (5.5)
//   24 units of 2000 - 8000             clusters of six 19.8 / 14.9 (9.4);   8 units of 16384   clusters of eight 21.8 / 17.4 (10.2)
// Launching a cluster costs about 0.1 us of the whole device, so: up to one and a half units per SM slot eight warps each, the
// largest cluster (no more than eight CTAs: seven of 16 fit) of which all units run at a time and whose warps all get a tile;
// beyond that four warps per unit.
template <int HD, int G, bool FUSED, bool LEFT> static cudaError_t launch_as_with(const AttnParams& p, cudaStream_t st) {
    using Wide = AsLaunch<HD, G, 8, as_wide_stages<HD, G>(), FUSED, LEFT>;
    using Narrow = AsLaunch<HD, G, 4, 3, FUSED, LEFT>;
    using Split = AsLaunch<HD, G, 8, as_wide_stages<HD, G>(), FUSED, false>;  // the same split, and so the same values, whatever registers LEFT takes
    const int rows = p.rows > 1 ? p.rows : 1;
    const long long units = static_cast<long long>(p.num_kv_heads) * rows;
    if (Split::prepare() != NVE_OK || Wide::prepare() != NVE_OK || Narrow::prepare() != NVE_OK) return cudaErrorInvalidValue;
    if (2 * units > 3ll * Split::active(p, 1)) return Narrow::launch(p, rows, 1, st);
    int csize = kAsMaxCluster;
    while (csize > 1 && (units > Split::active(p, csize) || p.kv_stride <= 128 * (csize - 1))) csize--;
    return Wide::launch(p, rows, csize, st);
}
template <int HD, int G, bool FUSED> static cudaError_t launch_as(const AttnParams& p, cudaStream_t st) {
    if constexpr (FUSED) {
        if (p.left.partial != nullptr) return launch_as_with<HD, G, true, true>(p, st);
    }
    return launch_as_with<HD, G, FUSED, false>(p, st);
}
template <int HD, bool FUSED> static bool launch_as_groups(const AttnParams& p, cudaStream_t st, cudaError_t& err) {
    switch (p.num_heads / p.num_kv_heads) {
        case 1: err = launch_as<HD, 1, FUSED>(p, st); return true;
        case 2: err = launch_as<HD, 2, FUSED>(p, st); return true;
        case 3: err = launch_as<HD, 3, FUSED>(p, st); return true;
        case 4: err = launch_as<HD, 4, FUSED>(p, st); return true;
        case 5: err = launch_as<HD, 5, FUSED>(p, st); return true;
        case 6: err = launch_as<HD, 6, FUSED>(p, st); return true;
        case 7: err = launch_as<HD, 7, FUSED>(p, st); return true;
        case 8: err = launch_as<HD, 8, FUSED>(p, st); return true;
        default: return false;
    }
}

bool attn_stream_mma_try(const AttnParams& p, int head_dim, cudaStream_t st, cudaError_t& err, bool fused) {
    if (head_dim == 128) return fused ? launch_as_groups<128, true>(p, st, err) : launch_as_groups<128, false>(p, st, err);
    if (head_dim == 64) return fused ? launch_as_groups<64, true>(p, st, err) : launch_as_groups<64, false>(p, st, err);
    return false;
}

}  // namespace nve
