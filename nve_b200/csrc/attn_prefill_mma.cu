// Causal attention of a block of new positions (prefill) on the tensor cores: tiles of 64 query rows against tiles
// of 64 cached positions, online softmax, K/V staged in shared memory once per tile and used by all its rows.  Blocks that fill the
// SMs with tiles of 128 rows go to attn_prefill_tc.cu (1777 rows 107 -> 41 us); this form is the one for shorter ones.
//
// What bounds it: with one CTA per (row, KV head) every row read the whole K/V prefix through L2 by itself (1777 rows
// of an 8B model: 1.58 M (row, position) pairs x 512 bytes x 8 KV heads = 6.5 GB per layer); a tile of 64 rows reads
// it 64 / G times less often and the kernel is bound by the mma.sync rate (about 1000 multiply-adds per cycle and SM) and by
// what stands between the two products of a step.  Tiles of 64 rows, not 128: twice the CTAs where the block is short, half the
// registers of a step, and faster at every size (8B, us: 61 rows 7.8 -> 4.7, 300 rows 25.5 -> 12.0, 600 rows 36.8 -> 20.8,
// 1777 rows 126 -> 107).  The queries stay in shared memory: in registers they leave room for a third CTA per SM, and all
// of it was slower (1777 rows 122, 3B 300 rows at 700 21.5 -> 29.7).
//
// A query row of a tile is a (position, head) pair of ONE KV head: row r of a tile is position t * PT + r / G, head
// h0 + r % G with PT = 64 / G positions per tile.  All G heads of the group share the staged K/V, and a short block
// fills its tiles; any group size up to 64 works.  Four warps take 16 rows each.
//
// Few tiles (a short block behind a long prefix) would leave most SMs idle: a cluster of 2, 4 or 8 CTAs then splits
// the positions of one tile, leaves unnormalised partials in shared memory and every CTA merges 64 / C of the rows
// through distributed shared memory.
#include <cooperative_groups.h>

#include "attn_mma.cuh"
#include "attn_params.cuh"

namespace cg = cooperative_groups;

namespace nve {

constexpr int kApRows = 64;      // query rows per tile
constexpr int kApKeys = 64;      // cached positions per step
constexpr int kApThreads = 128;  // four warps of 16 rows

__device__ __forceinline__ uint32_t ap_smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ap_cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ap_ldm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void ap_ldm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ float ap_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// byte offset of 16-byte chunk c of row r in a tile of HD f16 per row; chunks XORed with the row so that the eight
// rows of an 8x8 matrix lie in eight different bank groups
template <int HD> __device__ __forceinline__ uint32_t ap_off(int r, int c) {
    return static_cast<uint32_t>(r * (HD * 2) + ((c ^ (r & 7)) << 4));
}

// bits 15 and 31: which half of a word is an infinity or a NaN (all exponent bits set)
__device__ __forceinline__ uint32_t ap_not_finite(uint32_t w) { return ((w & 0x7C007C00u) + 0x04000400u) & 0x80008000u; }

template <int HD> constexpr int ap_smem_bytes() {
    constexpr int stage = kApRows * HD * 2 + 4 * kApKeys * HD * 2;  // Q, two K and two V tiles
    constexpr int part = kApRows * (HD + 4) * 4 + kApRows * 8 + kApRows * 32;  // f32 partials of a split tile + their m, l + weights
    return stage > part ? stage : part;
}

// One CTA's work.  A position that some rows of the tile do not see yet may hold an infinity or a NaN in v, which their zero probability
// would turn into NaN.  So a CTA that finds an output that is not finite stores nothing and says false, and the tile is computed once more,
// CAREFUL: in the steps that are cut such elements go to the rows that see them one by one and are zeros in the product.  (In line, as a
// branch of the steps, this cost 0.7 to 3 us per launch in a prefill of 61 rows, 8B; so 0.3.)
template <int HD, bool SPLIT, bool CAREFUL>
__device__ __forceinline__ bool ap_tile(const AttnParams& p, int groups, int tiles) {
    extern __shared__ __align__(128) unsigned char ap_raw[];
    constexpr int CH = HD / 8;  // 16-byte chunks per row
    constexpr int KVB = kApKeys * HD * 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    cg::cluster_group cluster = cg::this_cluster();
    const int csize = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
    const int tile = tiles - 1 - static_cast<int>(blockIdx.x) / csize;  // the tiles with the longest prefix first
    const int kvh = blockIdx.y;
    const int h0 = kvh * groups;
    const int PT = kApRows / groups;
    const int pos0 = tile * PT;                    // first block row of the tile
    const int npos = min(PT, p.rows - pos0);
    const int nrows = npos * groups;               // valid query rows
    const int start = p.seq_len - 1;               // position of block row 0
    const uint16_t* kh = p.k_cache + static_cast<long long>(kvh) * p.kv_stride * HD;
    const uint16_t* vh = p.v_cache + static_cast<long long>(kvh) * p.kv_stride * HD;
    const uint32_t sq = ap_smem(ap_raw), sk = sq + kApRows * HD * 2, sv = sk + 2 * KVB;

    const int kend = start + pos0 + npos;          // positions that the last row of the tile sees
    const int nkt = (kend + kApKeys - 1) / kApKeys;
    const int per = (nkt + csize - 1) / csize;
    const int kt0 = rank * per, kt1 = min(nkt, kt0 + per);

    if (!CAREFUL) {
        pdl_wait();
        pdl_launch_dependents();
    }
    auto load_kv = [&](int kt, int buf) {
#pragma unroll
        for (int i = 0; i < kApKeys * CH / kApThreads; i++) {
            const int id = tid + i * kApThreads;
            const int r = id / CH, c = id % CH;
            // rows past the end repeat the last one: finite values, masked below
            const long long src = static_cast<long long>(min(kt * kApKeys + r, kend - 1)) * HD + c * 8;
            ap_cp16(sk + buf * KVB + ap_off<HD>(r, c), kh + src);
            ap_cp16(sv + buf * KVB + ap_off<HD>(r, c), vh + src);
        }
    };
    for (int id = tid; id < kApRows * CH; id += kApThreads) {
        const int r = min(id / CH, nrows - 1), c = id % CH;
        const int pr = r / groups, h = r - pr * groups;
        ap_cp16(sq + ap_off<HD>(id / CH, c), p.q + static_cast<long long>(pos0 + pr) * p.row_stride + (h0 + h) * HD + c * 8);
    }
    if (kt0 < kt1) load_kv(kt0, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");

    // this thread's two query rows: g and g + 8 of the warp's sixteen; lim = positions the row may see
    int lim[2];
#pragma unroll
    for (int hh = 0; hh < 2; hh++) lim[hh] = start + pos0 + min(warp * 16 + hh * 8 + g, nrows - 1) / groups + 1;
    const int lim_min = start + pos0 + 1;
    const float sl2 = p.scale * 1.4426950408889634f;  // exponentials in base 2
    float m[2] = {-1e30f, -1e30f}, l[2] = {0.0f, 0.0f};
    float o[CH][4];
#pragma unroll
    for (int j = 0; j < CH; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.0f;

    for (int kt = kt0; kt < kt1; kt++) {
        const int buf = (kt - kt0) & 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the tile is there, and everyone is done with the other buffer
        if (kt + 1 < kt1) load_kv(kt + 1, buf ^ 1);
        asm volatile("cp.async.commit_group;" ::: "memory");

        float s[8][4];
#pragma unroll
        for (int n = 0; n < 8; n++) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.0f;
        const uint32_t kb = sk + buf * KVB, vb = sv + buf * KVB;
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
            uint32_t qa[4];
            ap_ldm4(sq + ap_off<HD>(warp * 16 + (lane & 15), 2 * kk + (lane >> 4)), qa);
#pragma unroll
            for (int np = 0; np < 4; np++) {
                uint32_t b[4];  // positions np*16 .. +7 (b0, b1) and +8 .. +15 (b2, b3)
                ap_ldm4(kb + ap_off<HD>(np * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * kk + ((lane >> 3) & 1)), b);
                mma_f16_16816(s[2 * np], qa, b[0], b[1]);
                mma_f16_16816(s[2 * np + 1], qa, b[2], b[3]);
            }
        }
        const bool cut = (kt + 1) * kApKeys > lim_min;  // some row does not see the whole tile
        if (cut) {
#pragma unroll
            for (int n = 0; n < 8; n++)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (kt * kApKeys + n * 8 + 2 * t + (e & 1) >= lim[e >> 1]) s[n][e] = -INFINITY;
        }
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
            float mx = s[0][2 * hh];
#pragma unroll
            for (int n = 0; n < 8; n++) mx = fmaxf(mx, fmaxf(s[n][2 * hh], s[n][2 * hh + 1]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float mn = fmaxf(m[hh], mx * sl2);  // stays finite: the masked value is below -1e30
            const float corr = ap_exp2(m[hh] - mn), shift = SPLIT ? kAmSplitLog2 - mn : -mn;
            m[hh] = mn;
            float sum = 0.0f;
#pragma unroll
            for (int n = 0; n < 8; n++) {
                s[n][2 * hh] = ap_exp2(fmaf(s[n][2 * hh], sl2, shift));
                s[n][2 * hh + 1] = ap_exp2(fmaf(s[n][2 * hh + 1], sl2, shift));
                sum += s[n][2 * hh] + s[n][2 * hh + 1];
            }
            l[hh] = l[hh] * corr + sum;
#pragma unroll
            for (int j = 0; j < CH; j++) {
                o[j][2 * hh] *= corr;
                o[j][2 * hh + 1] *= corr;
            }
        }
        if (CAREFUL && cut) {
            float ps[32];
#pragma unroll
            for (int i = 0; i < 32; i++) ps[i] = s[i >> 2][i & 3];
#pragma unroll 1
            for (int r = 0; r < kApKeys; r++) {
                const int i = (r >> 3) * 4 + (r & 1), from = (lane & ~3) | ((r & 7) >> 1), col = kt * kApKeys + r;
                const float p0 = __shfl_sync(0xffffffffu, ps[i], from), p1 = __shfl_sync(0xffffffffu, ps[i + 2], from);
#pragma unroll
                for (int j = 0; j < CH; j++) {
                    uint32_t w;
                    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(vb + ap_off<HD>(r, j) + 4 * t) : "memory");
#pragma unroll
                    for (int d = 0; d < 2; d++)
                        if (ap_not_finite(w) & (d == 0 ? 0x8000u : 0x80000000u)) {
                            const float v = Act16<NVE_DT_F16>::to_f32(static_cast<uint16_t>(w >> (16 * d)));
                            if (col < lim[0]) o[j][d] = fmaf(p0, v, o[j][d]);
                            if (col < lim[1]) o[j][2 + d] = fmaf(p1, v, o[j][2 + d]);
                        }
                }
            }
            __syncthreads();
#pragma unroll 1
            for (int i = tid; i < kApKeys * (HD / 2); i += kApThreads) {
                uint32_t w;
                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(vb + i * 4) : "memory");
                const uint32_t bad = ap_not_finite(w), keep = ((bad & 0x8000u) ? 0u : 0xFFFFu) | ((bad & 0x80000000u) ? 0u : 0xFFFF0000u);
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(vb + i * 4), "r"(w & keep) : "memory");
            }
            __syncthreads();
        }
        uint32_t pa[4][4], pb[4][4];
#pragma unroll
        for (int kp = 0; kp < 4; kp++)  // probabilities of 16 positions as the A operand of the second product
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float p0 = s[2 * kp + (i >> 1)][2 * (i & 1)], p1 = s[2 * kp + (i >> 1)][2 * (i & 1) + 1];
                pa[kp][i] = pack_f16x2(p0, p1);
                pb[kp][i] = SPLIT ? pack_f16x2_rest(p0, p1, pa[kp][i]) : 0;
            }
#pragma unroll
        for (int kp = 0; kp < 4; kp++)
#pragma unroll
            for (int dp = 0; dp < HD / 16; dp++) {
                uint32_t b[4];  // dims dp*16 .. +7 (b0, b1) and +8 .. +15 (b2, b3) of positions kp*16 .. +15
                ap_ldm4t(vb + ap_off<HD>(kp * 16 + (lane & 15), 2 * dp + (lane >> 4)), b);
                mma_f16_16816(o[2 * dp], pa[kp], b[0], b[1]);
                mma_f16_16816(o[2 * dp + 1], pa[kp], b[2], b[3]);
                if (SPLIT) {
                    mma_f16_16816(o[2 * dp], pb[kp], b[0], b[1]);
                    mma_f16_16816(o[2 * dp + 1], pb[kp], b[2], b[3]);
                }
            }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
        l[hh] += __shfl_xor_sync(0xffffffffu, l[hh], 1);
        l[hh] += __shfl_xor_sync(0xffffffffu, l[hh], 2);
    }
    // barrier: the staged tiles are no longer read, the buffers are free
    if (CAREFUL) {
        __syncthreads();
    } else {
        float probe[4] = {};
#pragma unroll
        for (int j = 0; j < CH; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) probe[e] += o[j][e];
        if (__syncthreads_or(!(fabsf((probe[0] + probe[1]) + (probe[2] + probe[3])) <= 3.0e38f))) return false;
    }

    if (csize == 1) {
        // rows through shared memory (each warp its own 16) so that they leave in 16-byte pieces
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
            const int r = warp * 16 + hh * 8 + g;
            const float inv = l[hh] > 0.0f ? 1.0f / l[hh] : 0.0f;
#pragma unroll
            for (int j = 0; j < CH; j++)
                *reinterpret_cast<uint32_t*>(ap_raw + ap_off<HD>(r, j) + 4 * t) = pack_f16x2(o[j][2 * hh] * inv, o[j][2 * hh + 1] * inv);
        }
        __syncwarp();
        for (int id = lane; id < 16 * CH; id += 32) {
            const int r = warp * 16 + id / CH, c = id % CH;
            if (r < nrows) {
                const int pr = r / groups, h = r - pr * groups;
                *reinterpret_cast<uint4*>(p.out + static_cast<long long>(pos0 + pr) * p.row_stride + (h0 + h) * HD + c * 8) =
                    *reinterpret_cast<const uint4*>(ap_raw + ap_off<HD>(r, c));
            }
        }
        return true;
    }
    // ---- split tile: unnormalised partials in shared memory, merged across the cluster
    constexpr int PR = HD + 4;  // floats per partial row
    float* part = reinterpret_cast<float*>(ap_raw);
    float* pm = part + kApRows * PR;
    float* pl = pm + kApRows;
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
        const int r = warp * 16 + hh * 8 + g;
        if (t == 0) {
            pm[r] = m[hh];
            pl[r] = l[hh];
        }
#pragma unroll
        for (int j = 0; j < CH; j++)
            *reinterpret_cast<float2*>(part + r * PR + j * 8 + 2 * t) = make_float2(o[j][2 * hh], o[j][2 * hh + 1]);
    }
    cluster.sync();
    // This CTA's share of the rows: first the weights of the ranks' partials, then the sums with the loads of all ranks and of
    // several pieces on their way together.  One dependent remote load after the other, this took 10 us.
    float* pw = pl + kApRows;  // [8][kApRows]
    const int rows_per = kApRows / csize, r0 = rank * rows_per;
    const int rows_here = min(rows_per, nrows - r0);
    for (int r = r0 + tid; r < r0 + rows_here; r += kApThreads) {
        float mk[8], lk[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k < csize) {
                mk[k] = cluster.map_shared_rank(pm, k)[r];
                lk[k] = cluster.map_shared_rank(pl, k)[r];
            }
        float mm = -1e30f, ss = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k < csize) mm = fmaxf(mm, mk[k]);
#pragma unroll
        for (int k = 0; k < 8; k++)  // ranks in ascending order
            if (k < csize) {
                mk[k] = ap_exp2(mk[k] - mm);
                ss = fmaf(lk[k], mk[k], ss);
            }
        const float inv = ss > 0.0f ? 1.0f / ss : 0.0f;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k < csize) pw[k * kApRows + r] = mk[k] * inv;
    }
    __syncthreads();
    constexpr int kFly = 2;  // pieces of four dims a thread has under way
    for (int id0 = tid; id0 < rows_here * (HD / 4); id0 += kFly * kApThreads) {
        float4 v[kFly][8];
#pragma unroll
        for (int f = 0; f < kFly; f++) {
            const int id = id0 + f * kApThreads, r = r0 + id / (HD / 4), c = id % (HD / 4);
            if (id < rows_here * (HD / 4)) {
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k < csize) v[f][k] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(part, k) + r * PR + c * 4);
            }
        }
#pragma unroll
        for (int f = 0; f < kFly; f++) {
            const int id = id0 + f * kApThreads, r = r0 + id / (HD / 4), c = id % (HD / 4);
            if (id < rows_here * (HD / 4)) {
                float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (int k = 0; k < 8; k++)  // ranks in ascending order
                    if (k < csize) {
                        const float w = pw[k * kApRows + r];
                        a.x = fmaf(v[f][k].x, w, a.x);
                        a.y = fmaf(v[f][k].y, w, a.y);
                        a.z = fmaf(v[f][k].z, w, a.z);
                        a.w = fmaf(v[f][k].w, w, a.w);
                    }
                const int pr = r / groups, h = r - pr * groups;
                *reinterpret_cast<uint2*>(p.out + static_cast<long long>(pos0 + pr) * p.row_stride + (h0 + h) * HD + c * 4) =
                    make_uint2(pack_f16x2(a.x, a.y), pack_f16x2(a.z, a.w));
            }
        }
    }
    cluster.sync();  // nobody leaves while its shared memory is read
    return true;
}

template <int HD, bool SPLIT> __device__ __noinline__ void ap_tile_careful(const AttnParams& p, int groups, int tiles) {
    ap_tile<HD, SPLIT, true>(p, groups, tiles);
}

template <int HD, bool SPLIT>
__global__ void __launch_bounds__(kApThreads, 2) attn_prefill_mma_kernel(const __grid_constant__ AttnParams p, int groups, int tiles) {
    if (!ap_tile<HD, SPLIT, false>(p, groups, tiles)) ap_tile_careful<HD, SPLIT>(p, groups, tiles);
}

template <int HD, bool SPLIT> static cudaError_t launch_ap(const AttnParams& p, cudaStream_t st) {
    constexpr int smem = ap_smem_bytes<HD>();
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(attn_prefill_mma_kernel<HD, SPLIT>), smem) != NVE_OK) return cudaErrorInvalidValue;
    const int groups = p.num_heads / p.num_kv_heads;
    const int PT = kApRows / groups;
    const int tiles = (p.rows + PT - 1) / PT;
    const int nkt = (p.seq_len - 1 + p.rows + kApKeys - 1) / kApKeys;
    // Split the positions of a tile while the larger grid still fits two CTAs per SM and it pays: a step of 64 positions takes
    // about 1.2 us, merging two to four CTAs 2.5 us, eight another one or two.
    int csize = 1;
    while (csize < 8 && static_cast<long long>(tiles) * p.num_kv_heads * csize * 2 <= 2 * sm_count() && nkt >= max(8, 4 * csize)) csize *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.dynamicSmemBytes = smem;
    cfg.gridDim = dim3(tiles * csize, p.num_kv_heads);
    cfg.blockDim = dim3(kApThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (pdl_enabled()) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    return cudaLaunchKernelEx(&cfg, attn_prefill_mma_kernel<HD, SPLIT>, p, groups, tiles);
}

bool attn_prefill_mma_try(const AttnParams& p, int head_dim, cudaStream_t st, cudaError_t& err) {
    if (p.num_heads / p.num_kv_heads > kApRows || p.num_kv_heads > 65535) return false;
    if (attn_prefill_tc_try(p, head_dim, st, err)) return true;
    const bool split = am_split(p.num_heads / p.num_kv_heads);
    if (head_dim == 128) err = split ? launch_ap<128, true>(p, st) : launch_ap<128, false>(p, st);
    else if (head_dim == 64) err = split ? launch_ap<64, true>(p, st) : launch_ap<64, false>(p, st);
    else return false;
    return true;
}

}  // namespace nve
