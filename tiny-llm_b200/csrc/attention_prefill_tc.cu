// Paged causal FlashAttention prefill on the 5th-generation tensor cores (tcgen05 + TMEM + TMA),
// bf16, head_dim 128, L > 8; and the same arithmetic for a few new tokens (L <= 8) further down.
//
// Replaces paged_attention_mma_bf16_d128 (src/extensions_ref/src/
// paged_attention.metal:250-506): same arithmetic - fp32 scores in base 2 (:414 scale_log2),
// bottom-right causal limit key <= row + (context - L) (:411), fp32 running max / sum, the
// probabilities rounded to bf16 before P V (:439-444), output = O / sum (0 when nothing is visible).
//
// One CTA = one (request, KV head, block of RH query positions): its 128 MMA rows are the G = Hq/Hkv
// query heads of the KV head x RH = 128/G consecutive query positions, so every K/V tile the CTA
// fetches is shared by all the query heads that need it, and the causal frontier is almost the same
// for every row (RH <= 128 positions apart).  Per 64-key tile:
//
//   warp 4 (one lane)  TMA producer: Q once (3-D map [D, L, B*Hq], box 64 x RH x G, 128-byte
//                      swizzle = the K-major UMMA layout), then K and V tiles - a (page, kv head)
//                      slab is one contiguous [page x 128] bf16 block, fetched as 4-D boxes
//                      [64 d x 64 keys] keyed by block_table (invalid page ids land outside the
//                      tensor and are zero-filled by the TMA unit) - through a 2-stage ring;
//   warp 5 (one lane)  MMA issuer: S = Q K^T  (tcgen05.mma kind::f16, M128 N64 K16 x 8, K tile =
//                      K-major B operand), then O += P V (M128 N128 K16 x 4, V tile = MN-major B
//                      operand straight from the page layout), accumulators S and O in TMEM;
//   warps 0-3          softmax: thread = MMA row = TMEM lane.  tcgen05.ld the 64 scores of its row,
//                      scale, mask, running max (no shuffles: a thread owns the row), exp2, row sum,
//                      bf16 probabilities -> back over the scores in tensor memory (A operand of P V;
//                      TL_FA_P_TMEM=0: through shared memory, a control).  O is rescaled IN TMEM (tcgen05.ld / st) only when a row's maximum
//                      grows by more than 2^8 since the last rescale: P and the row sum always use
//                      the same (possibly stale) maximum, so the result is exact.
//                      Epilogue: O / sum -> bf16 -> global.
//
// 256 TMEM columns and 112 KB of shared memory per CTA: two CTAs per SM, so one CTA's softmax
// overlaps the other's MMAs without an intra-CTA ping-pong.
//
// paged_decode_tc_kernel and decode_merge_tc_kernel (a few new tokens) have a comment of their own.
#include <stdlib.h>
#include <math_constants.h>

#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "kernels.h"
#include "per_device.h"
#include "tc_wait.cuh"

namespace tl {

typedef __nv_bfloat16 bf16;

constexpr int TC_D = 128;         // head dim
constexpr int TC_BM = 128;        // MMA rows per CTA (G heads x RH query positions)
constexpr int TC_BN = 64;         // keys per tile
constexpr int TC_STAGES = 2;
constexpr int TC_THREADS = 6 * 32;
constexpr int TC_Q_BYTES = TC_BM * TC_D * 2;        // 32 KiB: two 64-column halves of [128 rows x 128 B]
constexpr int TC_KV_TILE = TC_BN * TC_D * 2;        // 16 KiB: two 64-column halves of [64 rows x 128 B]
constexpr int TC_P_BYTES = TC_BM * TC_BN * 2;       // 16 KiB: [128 rows x 128 B]
constexpr int TC_Q_OFF = 0;
constexpr int TC_P_OFF = TC_Q_OFF + TC_Q_BYTES;
constexpr int TC_K_OFF = TC_P_OFF + TC_P_BYTES;
constexpr int TC_V_OFF = TC_K_OFF + TC_STAGES * TC_KV_TILE;
constexpr int TC_BAR_OFF = TC_V_OFF + TC_STAGES * TC_KV_TILE;
constexpr int TC_SMEM_BYTES = TC_BAR_OFF + 256;
constexpr int TC_TMEM_COLS = 256;  // S (two buffers): columns [0, 64) and [64, 128), O: columns [128, 256)
constexpr int TC_TMEM_O = 128;
constexpr float TC_LOG2E = 1.44269504089f;
constexpr float TC_RESCALE_THRESHOLD = 8.0f;  // log2: rescale O when a row maximum grew by more than 2^8

// kind::f16 instruction descriptor: bf16 x bf16 -> f32, A K-major; b_mn: B operand MN-major.
__host__ __device__ constexpr uint32_t tc_instr_desc(int n, bool b_mn) {
    return (1u << 4)                                // c_format = f32
           | (1u << 7)                              // a_format = bf16
           | (1u << 10)                             // b_format = bf16
           | (0u << 15)                             // a_major = K
           | ((b_mn ? 1u : 0u) << 16)               // b_major
           | (static_cast<uint32_t>(n >> 3) << 17)  // n_dim
           | (static_cast<uint32_t>(TC_BM >> 4) << 24);
}

// ex2.approx.ftz: the hardware approximation without the denormal range that exp2f() keeps (ncu of the first version: issue
// slots 54 % busy with the tensor pipe at 40 %).  Relative error
// 2^-22; the reference kernel uses fast::exp2 (paged_attention.metal:428-436).
__device__ __forceinline__ float tc_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct TcArgs {
    const int32_t *block_table, *context_lens;
    bf16 *out;
    int L, Hq, Hkv, G, RH;       // RH = query positions per CTA: 128 / G, or L where that is fewer
    int page_size, max_pages, num_pages;
    int tiles_per_page;          // page_size / 64
    float scale_log2;
    int is_causal;
    int out_token_major;  // out[(b, l, head), :] instead of [(b, head, l), :] (the layout the o-projection takes)
};

// PT: the probabilities of a tile stay in TENSOR memory - P_j (bf16 pairs, 32 columns) overwrites the first half of the
// score buffer S_j it was computed from, and P V reads its A operand from there (the TS form of tcgen05.mma).  The
// shared-memory form kept ONE P tile, so the exponentials of tile j could not start before P V of tile j-1 had finished
// reading it; now the exponentials overlap it and nothing waits for it but the rare rescale of O, and the eight 16-byte stores +
// proxy fence per row become one tcgen05.st.  Buffer reuse needs no barrier: S_{j+2} is issued behind P V_j in the same MMA queue.
// S_j complete implies P V_{j-2} complete (the tensor core takes them in order), and nothing about P V_{j-1} or any load.
template <bool PT>
__global__ void __launch_bounds__(TC_THREADS, 2)
paged_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                        const __grid_constant__ CUtensorMap tmap_v, const TcArgs a) {
    extern __shared__ __align__(1024) unsigned char tsm[];
    griddep_launch();  // programmatic dependent launch (common.cuh): the successor may set itself up under this grid
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qb = static_cast<int>((gridDim.x - 1 - blockIdx.x) / a.Hkv);  // long (late) query blocks of all heads first
    const int kvh = blockIdx.x % a.Hkv, b = blockIdx.z;
    const int q0 = qb * a.RH;
    const int ctx = min(a.context_lens[b], a.max_pages * a.page_size);
    // keys any row of this CTA may see: [0, key_end)
    const int last_row = min(q0 + a.RH, a.L) - 1;
    const int key_end = ctx <= 0 ? 0 : (a.is_causal ? min(ctx, max(ctx - a.L + last_row + 1, 0)) : ctx);
    const int n_tiles = (key_end + TC_BN - 1) / TC_BN;
    // MMA rows in use: row = head of the group x RH + position (side by side: warps without rows leave at once)
    const int rows = a.RH * a.G;

    const uint32_t q_base = g_smem_u32(tsm + TC_Q_OFF), p_base = g_smem_u32(tsm + TC_P_OFF);
    const uint32_t k_base = g_smem_u32(tsm + TC_K_OFF), v_base = g_smem_u32(tsm + TC_V_OFF);
    const uint32_t bar = g_smem_u32(tsm + TC_BAR_OFF);
    const uint32_t q_full = bar, s_full = bar + 8 /* two: one per S buffer */, p_full = bar + 24, pv_done = bar + 40 /* two of each, by the tile's parity */;
    const uint32_t k_full = bar + 56, k_empty = k_full + 8 * TC_STAGES, v_full = k_full + 16 * TC_STAGES, v_empty = k_full + 24 * TC_STAGES;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tsm + TC_BAR_OFF + 56 + 32 * TC_STAGES);

    if (warp == 4 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_q) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_v) : "memory");
    }
    if (warp == 5 && lane == 0) {
        g_mbar_init(q_full, 1);
        g_mbar_init(s_full, 1);
        g_mbar_init(s_full + 8, 1);
        for (int i = 0; i < 2; ++i) g_mbar_init(p_full + 8 * i, (rows + 31) / 32), g_mbar_init(pv_done + 8 * i, 1);  // one arrival per softmax warp that has rows
        for (int i = 0; i < TC_STAGES; ++i) {
            g_mbar_init(k_full + 8 * i, 1);
            g_mbar_init(k_empty + 8 * i, 1);
            g_mbar_init(v_full + 8 * i, 1);
            g_mbar_init(v_empty + 8 * i, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem_u32(tmem_slot)), "n"(TC_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    g_tc_fence_before();
    __syncthreads();
    g_tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // q and the newest K/V rows are the predecessor's output, and this grid overwrites buffers (output, split partials)
    // the predecessor may still read; block tables and context lengths are step inputs uploaded before the chain.
    griddep_wait();

    if (warp == 4) {
        // ------------------------------------------------------------ TMA producer
        if (n_tiles > 0) {  // whole warp, one elected lane issues (see the MMA warp)
            const int head0 = b * a.Hq + kvh * a.G;
            if (g_elect_one()) {
                g_mbar_expect_tx(q_full, rows * TC_D * 2);
                g_tma_load_3d(q_base, &tmap_q, 0, q0, head0, q_full);
                g_tma_load_3d(q_base + TC_Q_BYTES / 2, &tmap_q, 64, q0, head0, q_full);
            }
            __syncwarp();
            const int32_t *table = a.block_table + static_cast<size_t>(b) * a.max_pages;
            int s = 0;
            uint32_t ph = 1;  // producer side: first pass through the ring does not wait
            for (int j = 0; j < n_tiles; ++j) {
                const int lp = j / a.tiles_per_page;
                int pid = table[lp];
                if (pid < 0 || pid >= a.num_pages) pid = a.num_pages;  // outside the tensor: the TMA unit writes zeros
                const int slot0 = (j - lp * a.tiles_per_page) * TC_BN;
                g_mbar_wait(k_empty + 8 * s, ph);
                if (g_elect_one()) {
                    g_mbar_expect_tx(k_full + 8 * s, TC_KV_TILE);
                    g_tma_load_4d(k_base + s * TC_KV_TILE, &tmap_k, 0, slot0, kvh, pid, k_full + 8 * s);
                    g_tma_load_4d(k_base + s * TC_KV_TILE + TC_KV_TILE / 2, &tmap_k, 64, slot0, kvh, pid, k_full + 8 * s);
                }
                __syncwarp();
                g_mbar_wait(v_empty + 8 * s, ph);
                if (g_elect_one()) {
                    g_mbar_expect_tx(v_full + 8 * s, TC_KV_TILE);
                    g_tma_load_4d(v_base + s * TC_KV_TILE, &tmap_v, 0, slot0, kvh, pid, v_full + 8 * s);
                    g_tma_load_4d(v_base + s * TC_KV_TILE + TC_KV_TILE / 2, &tmap_v, 64, slot0, kvh, pid, v_full + 8 * s);
                }
                __syncwarp();
                if (++s == TC_STAGES) s = 0, ph ^= 1u;
            }
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------ MMA issuer
        // Order: S_0, then per tile j: S_{j+1} (second score buffer) | wait P_j | O += P_j V_j.  The tensor core works
        // on the next tile's scores while the softmax warps are busy with this tile's.
        // The whole warp walks the loop (uniform control flow, running stage / phase counters, descriptors derived by
        // adding to three base descriptors), one elected lane issues (tc05.cuh: g_elect_one - behind `if (lane == 0)`
        // the issue latency of a tile, by the cycle trace, was of the order of its 512 cycles of tensor work).
        if (n_tiles > 0) {
            constexpr uint32_t idesc_s = tc_instr_desc(TC_BN, false);
            constexpr uint32_t idesc_o = tc_instr_desc(TC_D, true);
            const uint64_t qdesc0 = g_smem_desc_sw128(q_base, 0, 1024), pdesc0 = g_smem_desc_sw128(p_base, 0, 1024);
            const uint64_t kdesc0 = g_smem_desc_sw128(k_base, 0, 1024);
            // V: 16 keys = 2 groups of 8 rows (SBO 1024 B); the two 64-wide d blocks are TC_KV_TILE/2 apart (LBO)
            const uint64_t vdesc0 = g_smem_desc_sw128(v_base, TC_KV_TILE / 2, 1024);
            g_mbar_wait(q_full, 0);
            int ks = 0, vs = 0;
            uint32_t kph = 0, vph = 0;
            auto issue_scores = [&](int j) {  // S_j = Q K_j^T: both operands K-major, two 64-wide halves of the head dimension
                g_mbar_wait(k_full + 8 * ks, kph);
                g_tc_fence_after();
                if (g_elect_one()) {
                    const uint64_t kd = kdesc0 + static_cast<uint64_t>(ks * (TC_KV_TILE >> 4));
#pragma unroll
                    for (int k = 0; k < TC_D / 16; ++k) {
                        const uint32_t half = (k >> 2), kk = (k & 3);
                        g_tc_mma(tmem + (j & 1) * TC_BN, qdesc0 + half * (TC_Q_BYTES / 2 >> 4) + 2 * kk, kd + half * (TC_KV_TILE / 2 >> 4) + 2 * kk,
                                 idesc_s, k > 0 ? 1u : 0u);
                    }
                    g_tc_commit(k_empty + 8 * ks);       // K stage reusable once these MMAs have read it
                    g_tc_commit(s_full + 8 * (j & 1));   // ... and the scores of tile j are complete
                }
                __syncwarp();
                if (++ks == TC_STAGES) ks = 0, kph ^= 1u;
            };
            issue_scores(0);
            for (int j = 0; j < n_tiles; ++j) {
                // score buffer (j+1)&1 was last read for tile j-1, whose P has been waited for below
                if (j + 1 < n_tiles) issue_scores(j + 1);
                // ---- O += P V: P K-major [128 x 64 keys], V MN-major [64 keys x 128 d] as loaded from the page
                g_mbar_wait(p_full + 8 * (j & 1), (j >> 1) & 1);
                g_mbar_wait(v_full + 8 * vs, vph);
                g_tc_fence_after();
                if (g_elect_one()) {
                    const uint64_t vd = vdesc0 + static_cast<uint64_t>(vs * (TC_KV_TILE >> 4));
#pragma unroll
                    for (int k = 0; k < TC_BN / 16; ++k) {
                        if constexpr (PT)  // 16 keys = 8 columns of bf16 pairs per K step
                            g_tc_mma_ts(tmem + TC_TMEM_O, tmem + (j & 1) * TC_BN + 8 * k, vd + k * (2048 >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
                        else
                            g_tc_mma(tmem + TC_TMEM_O, pdesc0 + 2 * k, vd + k * (2048 >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
                    }
                    g_tc_commit(v_empty + 8 * vs);
                    g_tc_commit(pv_done + 8 * (j & 1));  // O holds tiles 0..j and the P buffer is free again
                }
                __syncwarp();
                if (++vs == TC_STAGES) vs = 0, vph ^= 1u;
            }
        }
    } else if (warp * 32 < rows) {
        // ------------------------------------------------------------ softmax warps (thread = row = TMEM lane)
        const int r = threadIdx.x;                 // 0..127
        const int g = r / a.RH, lq = r - g * a.RH;  // query head of the KV group, position inside the block
        const int l = q0 + lq;
        const bool stored = r < rows && l < a.L;
        const bool row_valid = stored && ctx > 0;
        // last key this row may see (bottom-right causal alignment, paged_attention.metal:411)
        const int limit = !row_valid ? -1 : (a.is_causal ? min(ctx - 1, l + (ctx - a.L)) : ctx - 1);
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        float m_used = -CUDART_INF_F, l_sum = 0.f;
        const int32_t *table = a.block_table + static_cast<size_t>(b) * a.max_pages;
        for (int j = 0; j < n_tiles; ++j) {
            const int lp = j / a.tiles_per_page;
            const int pid = table[lp];
            const bool page_ok = pid >= 0 && pid < a.num_pages;
            g_mbar_wait(s_full + 8 * (j & 1), (j >> 1) & 1);
            g_tc_fence_after();
            uint32_t sv[2][32];
            g_tmem_ld32_nowait(tmem + lane_base + (j & 1) * TC_BN, sv[0]);
            g_tmem_ld32_nowait(tmem + lane_base + (j & 1) * TC_BN + 32, sv[1]);
            g_tmem_ld_wait();
            const int key0 = j * TC_BN;
            const int visible = page_ok ? min(limit - key0 + 1, TC_BN) : 0;  // keys [0, visible) of the tile
            // raw maximum (the scale is positive, so it commutes with max); masking only on boundary tiles
            float raw_max = -CUDART_INF_F;
            if (visible >= TC_BN) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int c = 0; c < 32; ++c) raw_max = fmaxf(raw_max, __uint_as_float(sv[h][c]));
            } else {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        if ((h * 32 + c) >= visible) sv[h][c] = 0xff800000u;  // -inf: exp2 gives exactly 0
                        raw_max = fmaxf(raw_max, __uint_as_float(sv[h][c]));
                    }
            }
            const float tile_max = raw_max * a.scale_log2;  // -inf stays -inf
            if constexpr (!PT)
                if (j > 0) g_mbar_wait(pv_done + 8 * ((j - 1) & 1), ((j - 1) >> 1) & 1);  // P V of tile j-1 complete: O is stable, the P buffer is free
            // lazy rescale: keep the stale maximum unless this tile exceeds it by more than 2^8
            const bool grow = tile_max > m_used + TC_RESCALE_THRESHOLD || (m_used == -CUDART_INF_F && tile_max != -CUDART_INF_F);
            if (__any_sync(0xffffffffu, grow) && j > 0) {
                if constexpr (PT) g_mbar_wait(pv_done + 8 * ((j - 1) & 1), ((j - 1) >> 1) & 1);  // O must be stable while it is rescaled
                g_tc_fence_after();
                const float m_new = grow ? tile_max : m_used;
                const float alpha = (grow && m_used != -CUDART_INF_F) ? exp2f(m_used - m_new) : (grow ? 0.f : 1.f);
                l_sum *= alpha;
#pragma unroll
                for (int cb = 0; cb < TC_D / 32; ++cb) {
                    uint32_t ov[32];
                    g_tmem_ld32(tmem + lane_base + TC_TMEM_O + cb * 32, ov);
#pragma unroll
                    for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * alpha);
                    g_tmem_st32(tmem + lane_base + TC_TMEM_O + cb * 32, ov);
                }
                g_tmem_st_wait();
                m_used = m_new;
            } else if (grow) {
                m_used = tile_max;  // first tile: nothing accumulated yet
            }
            const float m_eff = m_used == -CUDART_INF_F ? 0.f : m_used;
            float tile_sum = 0.f;
            uint32_t pk[32];  // 64 bf16 probabilities
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    const float p0 = tc_ex2(fmaf(__uint_as_float(sv[h][c]), a.scale_log2, -m_eff));
                    const float p1 = tc_ex2(fmaf(__uint_as_float(sv[h][c + 1]), a.scale_log2, -m_eff));
                    tile_sum += p0 + p1;
                    pk[h * 16 + c / 2] = pack2<bf16>(p0, p1);
                }
            l_sum += tile_sum;
            if constexpr (PT) {
                // lane = row, column c = keys (2c, 2c + 1) of the tile: over the first 32 columns of the score buffer just read
                g_tmem_st32(tmem + lane_base + (j & 1) * TC_BN, pk);
                g_tmem_st_wait();
                // p_full is two barriers, by the tile's parity: a warp arrives for tile j without waiting for P V of tile j-1 (220 of 1750 cycles a
                // tile), and cannot arrive for j+2 on the same barrier before all have for j, since S_{j+2} is issued behind P V_j.
            } else {
                // P row r: 128 bytes = 8 chunks of 16 B, chunk c at (c ^ (r & 7)) - the 128-byte swizzle of a K-major tile
                unsigned char *prow = tsm + TC_P_OFF + r * 128;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<uint4 *>(prow + ((c ^ (r & 7)) << 4)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
                g_fence_proxy_async();  // generic-proxy stores -> visible to the tensor core's async proxy
            }
            g_tc_fence_before();    // orders this thread's tcgen05.ld / st before the MMAs released by the arrive
            __syncwarp();           // one arrival per warp: 128 arrivals on one mbarrier are 128 serialised shared-memory atomics
            if (lane == 0) g_mbar_arrive(p_full + 8 * (j & 1));
        }
        // ---- epilogue: O / sum -> bf16 -> out[(b*Hq + head) * L + l, :]
        if (n_tiles > 0) {
            g_mbar_wait(pv_done + 8 * ((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1);
            g_tc_fence_after();
        }
        const size_t out_row = static_cast<size_t>(b * a.Hq + kvh * a.G + g) * a.L + l;
        const float inv = (l_sum == 0.f || !row_valid) ? 0.f : 1.0f / l_sum;
        bf16 *dst = a.out + (a.out_token_major ? (static_cast<size_t>(b) * a.L + l) * a.Hq + (kvh * a.G + g) : out_row) * TC_D;
#pragma unroll
        for (int cb = 0; cb < TC_D / 32; ++cb) {
            uint32_t ov[32];
            if (n_tiles > 0) {
                g_tmem_ld32(tmem + lane_base + TC_TMEM_O + cb * 32, ov);
            } else {
#pragma unroll
                for (int c = 0; c < 32; ++c) ov[c] = 0u;
            }
            if (stored) {
#pragma unroll
                for (int c = 0; c < 32; c += 8) {
                    uint4 o;
                    o.x = pack2<bf16>(__uint_as_float(ov[c]) * inv, __uint_as_float(ov[c + 1]) * inv);
                    o.y = pack2<bf16>(__uint_as_float(ov[c + 2]) * inv, __uint_as_float(ov[c + 3]) * inv);
                    o.z = pack2<bf16>(__uint_as_float(ov[c + 4]) * inv, __uint_as_float(ov[c + 5]) * inv);
                    o.w = pack2<bf16>(__uint_as_float(ov[c + 6]) * inv, __uint_as_float(ov[c + 7]) * inv);
                    *reinterpret_cast<uint4 *>(dst + cb * 32 + c) = o;
                }
            }
        }
    }
    g_tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        g_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TC_TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------- a few new tokens --
// Decode (G heads x L tokens of a key/value head in at most 128 rows): the launch is as many CTAs as the GPU holds at a time, and
// the key tiles of ALL requests and key/value heads, one after another, are dealt to them in equal shares.  A share may end in the
// middle of a (request, head) and go on with the next; a (request, head) in one share is finished there, one in several leaves a
// partial result per share for decode_merge_tc_kernel.  What is dealt out are the requests' real lengths, read on the device, so a
// captured launch follows them.  (Before, every (request, head) had its own CTAs, as many for all as suited a full block table: requests
// of very different lengths waited for the longest, which alone on its SM takes 1.3 us a tile, and more than one wave of CTAs
// waited for a last, emptier one.  A few short requests are cut into single tiles: one of 900 tokens 7.0 us, in shares of at least two,
// three and four tiles 8.2, 8.6 and 10.5.  One new token, 32 heads over 8: 32 requests of 200 to 7200 tokens 124 -> 72 us, 64 of 100 to 4100
// 123 -> 96, 8 of 300 to 7300 39 -> 28, one of 8000 beside 31 of 200 134 -> 18.)
// The query rows sit side by side (row = head of the group x L + token), so that only the softmax warps that have rows
// run; up to 32 rows there is one, and room for two query stages and a third key and value stage.
// Of 24 requests' steps 11.65 ms without, 11.50 with two tiles, 11.60 with four, 11.73 with sixteen (then the requests are in one another's way);
// 32 requests of 200 to 7200 tokens, launches back to back, 74.2 -> 73.2 us.
constexpr int TC_AHEAD = 2;
struct DecodeTcArgs {
    const int32_t *block_table, *context_lens;
    bf16 *out;
    int L, Hq, Hkv, G, requests;
    int page_size, max_pages, num_pages, tiles_per_page;
    float scale_log2;
    int is_causal;
    int slots, max_pieces;  // CTAs the GPU holds at a time; pieces of a (request, head) that the workspace has room for (>= 2)
    float *ws_o, *ws_m, *ws_l;
};

__device__ __forceinline__ void tc_prefetch_4d(const CUtensorMap *map, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ int dc_context(const DecodeTcArgs &a, int r) { return min(max(a.context_lens[r], 0), a.max_pages * a.page_size); }
__device__ __forceinline__ int dc_tiles(const DecodeTcArgs &a, int r) { return (dc_context(a, r) + TC_BN - 1) / TC_BN; }

// The tiles of all heads of all requests, those before `request` and the tiles of a share; called by whole warps.  Where every
// (request, head) can have a CTA and the longest is within a quarter of an equal share, per is 0 and each keeps to its own: the launch is
// bound by HBM then, and cutting only adds partial results (32 requests of 2000 tokens, 8 heads: 49 us cut, 45 whole; of 7200: 151 and 143).
// Nothing here depends on how many requests of length 0 the launch has, so a step over more idle slots cuts the same way, to the bit.
struct DecodeDeal {
    int total, before, per;
};
__device__ __forceinline__ DecodeDeal dc_deal(const DecodeTcArgs &a, int request) {
    int total = 0, before = 0, longest = 0, live = 0;
    for (int r = threadIdx.x & 31; r < a.requests; r += 32) {
        const int n = dc_tiles(a, r);
        total += n, longest = max(longest, n), live += n > 0;
        if (r < request) before += n;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        total += __shfl_xor_sync(0xffffffffu, total, o);
        before += __shfl_xor_sync(0xffffffffu, before, o);
        longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
        live += __shfl_xor_sync(0xffffffffu, live, o);
    }
    total *= a.Hkv, before *= a.Hkv;
    // n tiles touch at most ceil(n / per) + 1 shares
    if (static_cast<long long>(live) * a.Hkv <= a.slots && static_cast<long long>(longest) * 4 * a.slots <= 5LL * total) return {total, before, 0};
    return {total, before, max((total + a.slots - 1) / a.slots, (longest + a.max_pieces - 2) / (a.max_pieces - 1))};
}

// The rank-th request that has keys, -1 past the last; whole warps.
__device__ __forceinline__ int dc_live(const DecodeTcArgs &a, int rank) {
    for (int r0 = 0; r0 < a.requests; r0 += 32) {
        const int r = r0 + (threadIdx.x & 31);
        const unsigned live = __ballot_sync(0xffffffffu, r < a.requests && dc_tiles(a, r) > 0);
        if (rank < __popc(live)) return r0 + static_cast<int>(__fns(live, 0, rank + 1));
        rank -= __popc(live);
    }
    return -1;
}

// A share's walk over the (request, key/value head) pairs it touches.  Every role of the CTA walks it by itself.
struct DecodeWalk {
    int pos, end;       // of the share, in tiles over all requests and heads
    int b, tiles, base; // the request, its tiles a head, where its tiles begin
    int kvh, t0, n;     // this stretch: the head, its first tile and how many
    __device__ __forceinline__ void stretch() {
        const int off = pos - base;
        kvh = off / tiles, t0 = off - kvh * tiles, n = min(tiles - t0, end - pos);
    }
    __device__ __forceinline__ void start(const DecodeTcArgs &a, int begin, int stop) {  // whole warps; begin < stop <= total
        pos = begin, end = stop;
        const int lane = threadIdx.x & 31;
        int run = 0;
        for (int r0 = 0; r0 < a.requests; r0 += 32) {
            const int mine = r0 + lane < a.requests ? dc_tiles(a, r0 + lane) : 0;
            int upto = mine * a.Hkv;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += below;
            }
            const unsigned past = __ballot_sync(0xffffffffu, pos < run + upto);
            if (past) {
                const int src = __ffs(past) - 1;
                b = r0 + src, tiles = __shfl_sync(0xffffffffu, mine, src), base = run + __shfl_sync(0xffffffffu, upto, src) - tiles * a.Hkv;
                break;
            }
            run += __shfl_sync(0xffffffffu, upto, 31);
        }
        stretch();
    }
    __device__ __forceinline__ void own(int request, int head, int all) {
        pos = 0, end = all, b = request, tiles = all, base = 0, kvh = head, t0 = 0, n = all;
    }
    __device__ __forceinline__ bool next(const DecodeTcArgs &a) {
        pos += n;
        if (pos >= end) return false;
        if (pos == base + tiles * a.Hkv) {
            base = pos;
            do tiles = dc_tiles(a, ++b);
            while (tiles == 0);
        }
        stretch();
        return true;
    }
};

template <int SW>  // softmax warps: rows / 32
struct DecodeTcShape {
    static constexpr int q_half = SW * 32 * 128, q_stages = SW == 1 ? 2 : 1, stages = SW == 1 ? 3 : 2;
    static constexpr int k_off = q_stages * 2 * q_half, v_off = k_off + stages * TC_KV_TILE, bar_off = v_off + stages * TC_KV_TILE;
    static constexpr int smem = bar_off + 256, threads = 32 * (SW + 2);
    // the score product reads 128 rows from every query half, whatever they hold
    static_assert((q_stages * 2 - 1) * q_half + 128 * 128 <= bar_off, "rows past the queries lie in shared memory");
};

template <int SW>
__global__ void __launch_bounds__(DecodeTcShape<SW>::threads, 2)
paged_decode_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                       const DecodeTcArgs a) {
    using Z = DecodeTcShape<SW>;
    extern __shared__ __align__(1024) unsigned char tsm[];
    griddep_launch();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // context lengths and block tables are step inputs uploaded before the chain
    const DecodeDeal deal = dc_deal(a, 0);
    DecodeWalk w;
    const bool own = deal.per == 0;
    const int request = own ? dc_live(a, blockIdx.x / a.Hkv) : 0;
    if (own ? request < 0 : static_cast<long long>(blockIdx.x) * deal.per >= deal.total) {
        griddep_wait();  // also without work: what follows relies on this launch ending after the one before it
        return;
    }
    if (own) w.own(request, blockIdx.x % a.Hkv, dc_tiles(a, request));
    else w.start(a, blockIdx.x * deal.per, min((blockIdx.x + 1) * deal.per, deal.total));
    const int share = w.end - w.pos;
    const int rows = a.G * a.L;

    const uint32_t q_base = g_smem_u32(tsm), k_base = g_smem_u32(tsm + Z::k_off), v_base = g_smem_u32(tsm + Z::v_off);
    const uint32_t bar = g_smem_u32(tsm + Z::bar_off);
    const uint32_t s_full = bar /* two: one per score buffer */, p_full = bar + 16, pv_done = bar + 32 /* two of each, by the tile's parity */, q_full = bar + 48, q_empty = bar + 64;
    const uint32_t k_full = bar + 80, k_empty = k_full + 24, v_full = k_full + 48, v_empty = k_full + 72;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tsm + Z::bar_off + 80 + 96);
    volatile int *dead = reinterpret_cast<volatile int *>(tsm + Z::bar_off + 80 + 100);

    if (warp == SW && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_q) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_v) : "memory");
    }
    if (warp == SW + 1 && lane == 0) {
        *dead = 0;
        g_mbar_init(s_full, 1);
        g_mbar_init(s_full + 8, 1);
        for (int i = 0; i < 2; ++i) g_mbar_init(p_full + 8 * i, (rows + 31) / 32), g_mbar_init(pv_done + 8 * i, 1);  // one arrival per softmax warp that has rows
        for (int i = 0; i < Z::q_stages; ++i) g_mbar_init(q_full + 8 * i, 1), g_mbar_init(q_empty + 8 * i, 1);
        for (int i = 0; i < Z::stages; ++i) {
            g_mbar_init(k_full + 8 * i, 1), g_mbar_init(k_empty + 8 * i, 1);
            g_mbar_init(v_full + 8 * i, 1), g_mbar_init(v_empty + 8 * i, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem_u32(tmem_slot)), "n"(TC_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    g_tc_fence_before();
    __syncthreads();
    g_tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (warp == SW) {
        // The first tiles of the share are asked into L2 while the predecessor still runs: HBM is idle under it.  (Into L2 alone, where whatever the
        // predecessor writes to these rows arrives too; a copy into shared memory could miss it.)
        DecodeWalk early = w;
        int left = TC_AHEAD;
        do {
            const int32_t *table = a.block_table + static_cast<size_t>(early.b) * a.max_pages;
            for (int t = early.t0; t < early.t0 + early.n && left > 0; ++t, --left) {
                const int lp = t / a.tiles_per_page, slot0 = (t - lp * a.tiles_per_page) * TC_BN, pid = table[lp];
                if (pid >= 0 && pid < a.num_pages && g_elect_one())
#pragma unroll
                    for (int h = 0; h < TC_D; h += 64) {
                        tc_prefetch_4d(&tmap_k, h, slot0, early.kvh, pid);
                        tc_prefetch_4d(&tmap_v, h, slot0, early.kvh, pid);
                    }
                __syncwarp();
            }
        } while (left > 0 && early.next(a));
    }
    // q and the newest K/V rows are the predecessor's output, and this grid overwrites buffers (output, partials) that the
    // predecessor may still read
    griddep_wait();

    if (warp == SW) {
        // ------------------------------------------------------------ TMA producer (whole warp, one elected lane issues)
        int s = 0, qs = 0;
        uint32_t ph = 1, qph = 1;  // producer side: the first pass through a ring does not wait
        do {
            if (!tc_wait(q_empty + 8 * qs, qph, dead)) goto out;
            if (g_elect_one()) {
                const int head0 = w.b * a.Hq + w.kvh * a.G;
                const uint32_t q_at = q_base + qs * 2 * Z::q_half;
                g_mbar_expect_tx(q_full + 8 * qs, rows * TC_D * 2);
                g_tma_load_3d(q_at, &tmap_q, 0, 0, head0, q_full + 8 * qs);
                g_tma_load_3d(q_at + Z::q_half, &tmap_q, 64, 0, head0, q_full + 8 * qs);
            }
            __syncwarp();
            if (++qs == Z::q_stages) qs = 0, qph ^= 1u;
            const int32_t *table = a.block_table + static_cast<size_t>(w.b) * a.max_pages;
            for (int t = w.t0; t < w.t0 + w.n; ++t) {
                const int lp = t / a.tiles_per_page, slot0 = (t - lp * a.tiles_per_page) * TC_BN;
                int pid = table[lp];
                if (pid < 0 || pid >= a.num_pages) pid = a.num_pages;  // outside the tensor: the TMA unit writes zeros
                if (!tc_wait(k_empty + 8 * s, ph, dead)) goto out;
                if (g_elect_one()) {
                    g_mbar_expect_tx(k_full + 8 * s, TC_KV_TILE);
                    g_tma_load_4d(k_base + s * TC_KV_TILE, &tmap_k, 0, slot0, w.kvh, pid, k_full + 8 * s);
                    g_tma_load_4d(k_base + s * TC_KV_TILE + TC_KV_TILE / 2, &tmap_k, 64, slot0, w.kvh, pid, k_full + 8 * s);
                }
                __syncwarp();
                if (!tc_wait(v_empty + 8 * s, ph, dead)) goto out;
                if (g_elect_one()) {
                    g_mbar_expect_tx(v_full + 8 * s, TC_KV_TILE);
                    g_tma_load_4d(v_base + s * TC_KV_TILE, &tmap_v, 0, slot0, w.kvh, pid, v_full + 8 * s);
                    g_tma_load_4d(v_base + s * TC_KV_TILE + TC_KV_TILE / 2, &tmap_v, 64, slot0, w.kvh, pid, v_full + 8 * s);
                }
                __syncwarp();
                if (++s == Z::stages) s = 0, ph ^= 1u;
            }
        } while (w.next(a));
    } else if (warp == SW + 1) {
        // ------------------------------------------------------------ MMA issuer: scores one tile ahead, across stretches too
        constexpr uint32_t idesc_s = tc_instr_desc(TC_BN, false), idesc_o = tc_instr_desc(TC_D, true);
        const uint64_t qdesc0 = g_smem_desc_sw128(q_base, 0, 1024), kdesc0 = g_smem_desc_sw128(k_base, 0, 1024);
        const uint64_t vdesc0 = g_smem_desc_sw128(v_base, TC_KV_TILE / 2, 1024);
        DecodeWalk ahead = w;
        int ks = 0, vs = 0, qs = 0, left = ahead.n, value = 0;  // left: tiles of the stretch whose scores are still to come; value: this stretch's tile
        uint32_t kph = 0, vph = 0, qph = 0;
        bool fresh = true, more = true;
        auto issue_scores = [&](int j) {
            if (fresh && !tc_wait(q_full + 8 * qs, qph, dead)) return false;
            fresh = false;
            if (!tc_wait(k_full + 8 * ks, kph, dead)) return false;
            g_tc_fence_after();
            const bool last = --left == 0;
            if (g_elect_one()) {
                const uint64_t kd = kdesc0 + static_cast<uint64_t>(ks * (TC_KV_TILE >> 4)), qd = qdesc0 + static_cast<uint64_t>(qs * (2 * Z::q_half >> 4));
#pragma unroll
                for (int k = 0; k < TC_D / 16; ++k) {
                    const uint32_t half = (k >> 2), kk = (k & 3);
                    g_tc_mma(tmem + (j & 1) * TC_BN, qd + half * (Z::q_half >> 4) + 2 * kk, kd + half * (TC_KV_TILE / 2 >> 4) + 2 * kk, idesc_s, k > 0 ? 1u : 0u);
                }
                g_tc_commit(k_empty + 8 * ks);
                if (last) g_tc_commit(q_empty + 8 * qs);
                g_tc_commit(s_full + 8 * (j & 1));
            }
            __syncwarp();
            if (++ks == Z::stages) ks = 0, kph ^= 1u;
            if (last) {
                if (++qs == Z::q_stages) qs = 0, qph ^= 1u;
                more = ahead.next(a), left = ahead.n, fresh = true;
            }
            return true;
        };
        if (!issue_scores(0)) goto out;
        for (int j = 0; j < share; ++j) {
            // score buffer (j+1)&1 was last read for tile j-1, whose P has been waited for below
            if (more && !issue_scores(j + 1)) goto out;
            // a new stretch's first product overwrites O: the softmax warps arrive for it after they have read the old one
            if (!tc_wait(p_full + 8 * (j & 1), (j >> 1) & 1, dead) || !tc_wait(v_full + 8 * vs, vph, dead)) goto out;
            g_tc_fence_after();
            if (g_elect_one()) {
                const uint64_t vd = vdesc0 + static_cast<uint64_t>(vs * (TC_KV_TILE >> 4));
#pragma unroll
                for (int k = 0; k < TC_BN / 16; ++k)  // 16 keys = 8 columns of bf16 pairs per K step
                    g_tc_mma_ts(tmem + TC_TMEM_O, tmem + (j & 1) * TC_BN + 8 * k, vd + k * (2048 >> 4), idesc_o, (value > 0 || k > 0) ? 1u : 0u);
                g_tc_commit(v_empty + 8 * vs);
                g_tc_commit(pv_done + 8 * (j & 1));
            }
            __syncwarp();
            if (++vs == Z::stages) vs = 0, vph ^= 1u;
            if (++value == w.n) value = 0, w.next(a);
        }
    } else if (warp * 32 < rows) {
        // ------------------------------------------------------------ softmax warps (thread = row = TMEM lane)
        const int r = threadIdx.x, g = r / a.L, l = r - g * a.L;
        const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
        int j = 0;  // tile of the share
        do {
            const int ctx = dc_context(a, w.b);
            const int limit = r >= rows ? -1 : (a.is_causal ? min(ctx - 1, l + (ctx - a.L)) : ctx - 1);  // the last key this row may see
            const int32_t *table = a.block_table + static_cast<size_t>(w.b) * a.max_pages;
            float m_used = -CUDART_INF_F, l_sum = 0.f;
            bool ok = true;
            for (int i = 0; i < w.n; ++i, ++j) {
                const int pid = table[(w.t0 + i) / a.tiles_per_page];
                const int visible = pid >= 0 && pid < a.num_pages ? min(limit - (w.t0 + i) * TC_BN + 1, TC_BN) : 0;  // keys [0, visible) of the tile
                if (!(ok = tc_wait(s_full + 8 * (j & 1), (j >> 1) & 1, dead))) break;
                g_tc_fence_after();
                uint32_t sv[2][32];
                g_tmem_ld32_nowait(tmem + lane_base + (j & 1) * TC_BN, sv[0]);
                g_tmem_ld32_nowait(tmem + lane_base + (j & 1) * TC_BN + 32, sv[1]);
                g_tmem_ld_wait();
                float raw_max = -CUDART_INF_F;  // the scale is positive, so it commutes with max
                if (visible < TC_BN)
#pragma unroll
                    for (int c = 0; c < TC_BN; ++c)
                        if (c >= visible) sv[c >> 5][c & 31] = 0xff800000u;  // -inf: exp2 gives exactly 0
#pragma unroll
                for (int c = 0; c < TC_BN; ++c) raw_max = fmaxf(raw_max, __uint_as_float(sv[c >> 5][c & 31]));
                const float tile_max = raw_max * a.scale_log2;
                // The maximum is taken anew for every tile.  (Kept until it had grown by 2^8, as for prompts, it left the largest weights inexact:
                // error against 64 bits .00234 instead of .00225 at 32 requests of 2000, where the many short pieces of an earlier cut
                // had hidden that.  With few rows it seldom grows: 32 x 7200 140.5 -> 141.2 us, 32 of 200 to 7200 72 -> 75.)
                const bool grow = tile_max > m_used;
                if (__any_sync(0xffffffffu, grow) && i > 0) {
                    if (!(ok = tc_wait(pv_done + 8 * ((j - 1) & 1), ((j - 1) >> 1) & 1, dead))) break;  // O must be stable while it is rescaled
                    g_tc_fence_after();
                    const float m_new = grow ? tile_max : m_used;
                    const float alpha = (grow && m_used != -CUDART_INF_F) ? exp2f(m_used - m_new) : (grow ? 0.f : 1.f);
                    l_sum *= alpha;
#pragma unroll
                    for (int cb = 0; cb < TC_D / 32; ++cb) {
                        uint32_t ov[32];
                        g_tmem_ld32(tmem + lane_base + TC_TMEM_O + cb * 32, ov);
#pragma unroll
                        for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * alpha);
                        g_tmem_st32(tmem + lane_base + TC_TMEM_O + cb * 32, ov);
                    }
                    g_tmem_st_wait();
                    m_used = m_new;
                } else if (grow) {
                    m_used = tile_max;  // first tile: nothing accumulated yet
                }
                const float m_eff = m_used == -CUDART_INF_F ? 0.f : m_used;
                float tile_sum = 0.f;
                uint32_t pk[32];  // 64 bf16 probabilities, over the first 32 columns of the score buffer just read
#pragma unroll
                for (int c = 0; c < TC_BN; c += 2) {
                    const float p0 = tc_ex2(fmaf(__uint_as_float(sv[c >> 5][c & 31]), a.scale_log2, -m_eff));
                    const float p1 = tc_ex2(fmaf(__uint_as_float(sv[c >> 5][(c & 31) + 1]), a.scale_log2, -m_eff));
                    tile_sum += p0 + p1;
                    pk[c / 2] = pack2<bf16>(p0, p1);
                }
                l_sum += tile_sum;
                g_tmem_st32(tmem + lane_base + (j & 1) * TC_BN, pk);
                g_tmem_st_wait();
                g_tc_fence_before();
                __syncwarp();
                if (lane == 0) g_mbar_arrive(p_full + 8 * (j & 1));
            }
            ok = ok && tc_wait(pv_done + 8 * ((j - 1) & 1), ((j - 1) >> 1) & 1, dead);
            g_tc_fence_after();
            const size_t out_row = static_cast<size_t>(w.b * a.Hq + w.kvh * a.G + g) * a.L + l;
            const bool whole = w.n == w.tiles;
            const float inv = whole ? (l_sum == 0.f ? 0.f : 1.0f / l_sum) : 1.f, bad = tc_verdict(ok, dead);
            const size_t slot = out_row * a.max_pieces + (whole ? 0 : blockIdx.x - (w.base + w.kvh * w.tiles) / deal.per);
#pragma unroll
            for (int cb = 0; cb < TC_D / 32; ++cb) {
                uint32_t ov[32];
                g_tmem_ld32(tmem + lane_base + TC_TMEM_O + cb * 32, ov);
                if (r >= rows) continue;
                if (whole) {
                    bf16 *dst = a.out + out_row * TC_D + cb * 32;
#pragma unroll
                    for (int c = 0; c < 32; c += 8) {
                        uint32_t o[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            o[e] = pack2<bf16>(__uint_as_float(ov[c + 2 * e]) * inv * bad, __uint_as_float(ov[c + 2 * e + 1]) * inv * bad);
                        *reinterpret_cast<uint4 *>(dst + c) = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                } else {
                    float *po = a.ws_o + slot * TC_D + cb * 32;
#pragma unroll
                    for (int c = 0; c < 32; c += 4) *reinterpret_cast<uint4 *>(po + c) = make_uint4(ov[c], ov[c + 1], ov[c + 2], ov[c + 3]);
                }
            }
            if (!whole && r < rows) a.ws_m[slot] = m_used == -CUDART_INF_F ? -1e30f : m_used, a.ws_l[slot] = l_sum * bad;
        } while (w.next(a));
    }
out:  // also from a role whose wait gave up
    g_tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_settle(dead);
        g_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TC_TMEM_COLS) : "memory");
    }
}

// One CTA per row: the pieces' sums brought to their common maximum and divided, in the pieces' order.  Rows that one CTA finished are
// left alone, rows of a request without keys are zero.
__global__ void __launch_bounds__(TC_D) decode_merge_tc_kernel(const DecodeTcArgs a) {
    griddep_launch();
    const int row = blockIdx.x, d = threadIdx.x, lane = d & 31;
    const int b = row / (a.Hq * a.L), kvh = (row - b * a.Hq * a.L) / (a.G * a.L);
    const DecodeDeal deal = dc_deal(a, b);
    const int tiles = dc_tiles(a, b), u0 = deal.before + kvh * tiles;
    const int pieces = tiles == 0 ? 0 : deal.per == 0 ? 1 : (u0 + tiles - 1) / deal.per - u0 / deal.per + 1;
    griddep_wait();
    if (pieces == 1) return;
    const float *pm = a.ws_m + static_cast<size_t>(row) * a.max_pieces, *pl = a.ws_l + static_cast<size_t>(row) * a.max_pieces;
    const float *po = a.ws_o + static_cast<size_t>(row) * a.max_pieces * TC_D + d;
    float v[8];  // the first columns go out beside the weights (the workspace is rewritten by every layer: read through L2)
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = j < pieces ? __ldcg(po + static_cast<size_t>(j) * TC_D) : 0.f;
    const float m = lane < pieces ? __ldcg(pm + lane) : -1e30f, s = lane < pieces ? __ldcg(pl + lane) : 0.f;  // at most 32 pieces
    const float gm = warp_max(m), f = exp2f(m - gm), gl = warp_sum(s * f);
    float o = 0.f;
    for (int s0 = 0; s0 < pieces; s0 += 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float fj = __shfl_sync(0xffffffffu, f, (s0 + j) & 31);
            if (s0 + j < pieces) o += v[j] * fj;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (s0 + 8 + j < pieces) v[j] = __ldcg(po + static_cast<size_t>(s0 + 8 + j) * TC_D);
    }
    a.out[static_cast<size_t>(row) * TC_D + d] = __float2bfloat16_rn(gl == 0.f ? 0.f : o / gl);
}

// ---------------------------------------------------------------- host side --
// Tensor maps are cached per (base pointer, shape): a prefill of 36 layers x N chunks re-uses a
// handful of distinct operands.  (An encoding takes 0.05 us; a look-up costs no more.)
struct MapKey {
    const void *ptr;
    unsigned long long d0, d1, d2, d3;
    unsigned b1, b2;
    bool operator==(const MapKey &o) const { return ptr == o.ptr && d0 == o.d0 && d1 == o.d1 && d2 == o.d2 && d3 == o.d3 && b1 == o.b1 && b2 == o.b2; }
};
struct MapKeyHash {
    size_t operator()(const MapKey &k) const {
        size_t h = reinterpret_cast<size_t>(k.ptr);
        for (unsigned long long v : {k.d0, k.d1, k.d2, k.d3, static_cast<unsigned long long>(k.b1), static_cast<unsigned long long>(k.b2)})
            h = h * 1000003u ^ static_cast<size_t>(v);
        return h;
    }
};
static int cached_map(CUtensorMap *out, const void *ptr, int rank, const cuuint64_t *dims, const cuuint32_t *box) {
    static std::mutex mu;
    static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
    MapKey key{ptr, dims[0], dims[1], dims[2], rank > 3 ? dims[3] : 0, box[1], box[2]};
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
        *out = it->second;
        return TL_OK;
    }
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (encode == nullptr) return fail(TL_ECUDA, "paged_attention: cuTensorMapEncodeTiled is unavailable");
    cuuint64_t strides[3];
    cuuint64_t acc = 2;
    for (int i = 0; i + 1 < rank; ++i) {
        acc *= dims[i];
        strides[i] = acc;
    }
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUtensorMap map;
    CUresult r = encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(ptr), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TL_ECUDA, "paged_attention: cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
    if (cache.size() > 4096) cache.clear();
    cache.emplace(key, map);
    *out = map;
    return TL_OK;
}

long long decode_tc_gave_up() { return read_gave_up(); }

bool paged_prefill_tc_supported(int L, int num_pages, int page_size, int num_kv_heads, int num_heads) {
    static const bool off = [] { const char *e = getenv("TL_PREFILL_TC"); return e != nullptr && e[0] == '0'; }();
    if (off || num_kv_heads < 1 || num_heads % num_kv_heads != 0) return false;
    const int G = num_heads / num_kv_heads;
    if (G < 1 || G > TC_BM || (TC_BM % G) != 0) return false;
    return L > 0 && num_pages > 0 && page_size >= TC_BN && page_size % TC_BN == 0;
}

// A chained launch with `smem` bytes of dynamic shared memory, the limit raised once per device and kernel.
template <auto KERNEL, typename Args>
static int attention_launch(dim3 grid, int threads, size_t smem, cudaStream_t st, const CUtensorMap &mq, const CUtensorMap &mk, const CUtensorMap &mv, const Args &a) {
    static PerDevice ready;
    int device = -1;
    cudaGetDevice(&device);
    const bool raised = ready(device, [&] {
        return cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) == cudaSuccess &&
               cudaFuncSetAttribute(KERNEL, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) == cudaSuccess;
    });
    if (!raised) {
        cudaGetLastError();
        return fail(TL_ECUDA, "paged_attention: cannot raise shared memory limit");
    }
    const cudaError_t e = launch_chained(KERNEL, grid, dim3(threads), smem, st, mq, mk, mv, a);
    return e == cudaSuccess ? TL_OK : fail(TL_ECUDA, "paged_attention: launch failed: %s", cudaGetErrorString(e));
}

// Tensor maps of the queries (boxes of RH positions x G heads) and of the pages (boxes of one tile).
static int attention_maps(CUtensorMap *mq, CUtensorMap *mk, CUtensorMap *mv, const void *q, const void *kp, const void *vp, int rows, int L, int RH, int G, int num_pages,
                          int page_size, int num_kv_heads) {
    const cuuint64_t qdims[3] = {TC_D, static_cast<cuuint64_t>(L), static_cast<cuuint64_t>(rows)};
    const cuuint32_t qbox[3] = {64, static_cast<cuuint32_t>(RH), static_cast<cuuint32_t>(G)};
    if (int e = cached_map(mq, q, 3, qdims, qbox)) return e;
    const cuuint64_t dims[4] = {TC_D, static_cast<cuuint64_t>(page_size), static_cast<cuuint64_t>(num_kv_heads), static_cast<cuuint64_t>(num_pages)};
    const cuuint32_t box[4] = {64, TC_BN, 1, 1};
    if (int e = cached_map(mk, kp, 4, dims, box)) return e;
    return cached_map(mv, vp, 4, dims, box);
}

int launch_paged_prefill_tc(const void *q, const void *kp, const void *vp, const int32_t *bt, const int32_t *cl, void *out, int rows,
                            int L, int num_pages, int page_size, int max_pages, float scale, int is_causal, int num_kv_heads,
                            int num_heads, cudaStream_t st, bool out_token_major) {
    const int G = num_heads / num_kv_heads;
    const int B = rows / num_heads;
    TcArgs a{};
    a.block_table = bt, a.context_lens = cl, a.out = static_cast<bf16 *>(out);
    a.L = L, a.Hq = num_heads, a.Hkv = num_kv_heads, a.G = G, a.RH = std::min(TC_BM / G, L);
    a.page_size = page_size, a.max_pages = max_pages, a.num_pages = num_pages;
    a.tiles_per_page = page_size / TC_BN;
    a.scale_log2 = scale * TC_LOG2E;
    a.is_causal = is_causal;
    CUtensorMap mq, mk, mv;
    if (int e = attention_maps(&mq, &mk, &mv, q, kp, vp, rows, L, a.RH, G, num_pages, page_size, num_kv_heads)) return e;
    const int q_blocks = (L + a.RH - 1) / a.RH;
    a.out_token_major = out_token_major ? 1 : 0;
    // Key/value heads vary fastest, so that a request's longest blocks start first in all heads and its shortest come last: with a head's blocks together
    // the last head's longest ones started last (32 heads over 8, 2048 tokens of 3500: 104 -> 84 us; of 2048: 60 -> 41; 4096 of 4096: 157 -> 131).
    dim3 grid(static_cast<unsigned>(q_blocks) * num_kv_heads, 1, B);
    if (num_kv_heads > 65535 || grid.z > 65535 || static_cast<long long>(q_blocks) * num_kv_heads > 0x7fffffffLL) return fail(TL_EINVAL, "paged_attention: too many heads / requests for one launch");
    static const bool p_tmem = [] { const char *e = getenv("TL_FA_P_TMEM"); return e == nullptr || e[0] != '0'; }();  // 0: P through shared memory (control)
    if (int e = p_tmem ? attention_launch<paged_prefill_tc_kernel<true>>(grid, TC_THREADS, TC_SMEM_BYTES, st, mq, mk, mv, a)
                       : attention_launch<paged_prefill_tc_kernel<false>>(grid, TC_THREADS, TC_SMEM_BYTES, st, mq, mk, mv, a))
        return e;
    TL_LAUNCH_CHECK("paged_prefill_tc");
    return TL_OK;
}

int launch_paged_decode_tc(const void *q, const void *kp, const void *vp, const int32_t *bt, const int32_t *cl, void *out, int rows, int L,
                           int num_pages, int page_size, int max_pages, float scale, int is_causal, int num_kv_heads, int num_heads, void *ws,
                           size_t ws_bytes, cudaStream_t st) {
    const size_t rows_total = static_cast<size_t>(rows) * L;
    const long long pieces = ws == nullptr ? 0 : std::min<long long>(32, ws_bytes / (rows_total * (TC_D + 2) * sizeof(float)));
    const long long most = (static_cast<long long>(max_pages) * page_size + TC_BN - 1) / TC_BN * num_kv_heads * (rows / num_heads);
    if (pieces < 2 || most > (1LL << 30))  // no room for partial results, or more tiles than an int counts: a CTA per (request, head)
        return launch_paged_prefill_tc(q, kp, vp, bt, cl, out, rows, L, num_pages, page_size, max_pages, scale, is_causal, num_kv_heads, num_heads, st);
    if (num_kv_heads > 65535 || rows / num_heads > 65535) return fail(TL_EINVAL, "paged_attention: too many heads / requests for one launch");
    DecodeTcArgs a{};
    a.block_table = bt, a.context_lens = cl, a.out = static_cast<bf16 *>(out);
    a.L = L, a.Hq = num_heads, a.Hkv = num_kv_heads, a.G = num_heads / num_kv_heads, a.requests = rows / num_heads;
    a.page_size = page_size, a.max_pages = max_pages, a.num_pages = num_pages, a.tiles_per_page = page_size / TC_BN;
    a.scale_log2 = scale * TC_LOG2E, a.is_causal = is_causal;
    a.slots = 2 * sm_count();
    const unsigned ctas = static_cast<unsigned>(std::max(1LL, std::min<long long>(a.slots, most)));  // shares of one tile at least
    a.max_pieces = static_cast<int>(pieces);
    a.ws_o = static_cast<float *>(ws), a.ws_m = a.ws_o + rows_total * pieces * TC_D, a.ws_l = a.ws_m + rows_total * pieces;
    CUtensorMap mq, mk, mv;
    if (int e = attention_maps(&mq, &mk, &mv, q, kp, vp, rows, L, L, a.G, num_pages, page_size, num_kv_heads)) return e;
    const bool narrow = a.G * L <= 32;
    if (int e = narrow ? attention_launch<paged_decode_tc_kernel<1>>(dim3(ctas), DecodeTcShape<1>::threads, DecodeTcShape<1>::smem, st, mq, mk, mv, a)
                       : attention_launch<paged_decode_tc_kernel<4>>(dim3(ctas), DecodeTcShape<4>::threads, DecodeTcShape<4>::smem, st, mq, mk, mv, a))
        return e;
    TL_LAUNCH_CHECK("paged_decode_tc");
    const cudaError_t le = launch_chained(decode_merge_tc_kernel, dim3(static_cast<unsigned>(rows_total)), dim3(TC_D), 0, st, a);
    if (le != cudaSuccess) return fail(TL_ECUDA, "paged_attention: launch failed: %s", cudaGetErrorString(le));
    TL_LAUNCH_CHECK("decode_merge_tc");
    return TL_OK;
}

}  // namespace tl
