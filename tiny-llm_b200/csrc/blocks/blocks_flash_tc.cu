// Attention of prompt portions over paged keys and values on the 5th-generation tensor cores (tcgen05 + TMEM + TMA): the same
// masks, weights, sinks and gates as blocks_paged_attention_flash.cu, for bf16 caches.
//
// One CTA = one run of consecutive tokens of a sequence x the query heads of one key/value head, as 128 MMA rows (= tensor-memory
// lanes), so every key and value tile is fetched once for all of them.  Which run a CTA takes it finds in seq_info itself; there
// is no work list.  Per 64-key tile:
//   warp 4     TMA: the queries once (boxes 64 columns x heads x tokens), then key and value tiles, addressed through the block
//              table; boxes end at a head's last column and at the last page, what lies beyond reads as zeros, and so does a
//              tile whose table entry is bad.  The keys may come from two places (k_first 64-column blocks of one matrix per head,
//              the rest from a matrix shared by all heads): a latent layer's up-projected keys and its rotated part.
//   warp 5     tcgen05.mma, one elected lane: S = Q K^T into one of two score buffers, O += P V; the next tile's scores are
//              issued ahead of this tile's values
//   warps 0-3  softmax, thread = row: scores from tensor memory, maximum, 2^x, P as bf16 back over its own score buffer (the
//              value product reads its left operand from tensor memory).  The maximum is taken anew for every tile, and O is
//              rescaled in tensor memory in a tile where one of the warp's rows has a new one; sums are of the rounded P.  (A
//              maximum kept until it had grown by 2^8 saves 1 to 4 % of a layer's time, but a row's largest weights are
//              exact against its own maximum only, where they are 1: the layer's error against 64 bits was up to 2.8 % above
//              that of the register kernel, now it is the same.)
// 256 columns of tensor memory and at most 113 KB of shared memory (head sizes up to 192 + 128) let two CTAs share an SM: one's
// exponentials run beside the other's products, both of which take about 512 cycles a tile at 128 + 128 (64 x 128 exponentials
// at 16 a cycle).  With 192 key columns that leaves room for one value stage.
// Tiles are 64-aligned in absolute positions and taken in ascending order.  Rows of values past the newest key are cleared in
// shared memory, so that what an earlier owner of the page left there cannot reach a sum through a zero weight.
#include "blocks_tc.cuh"

namespace tlb {

using tl::g_tma_load_3d;
using tl::g_tmem_ld32;
using tl::g_tmem_ld32_nowait;
using tl::g_tmem_ld_wait;
using tl::g_tmem_st32;
using tl::g_tmem_st_wait;

constexpr int kXKeys = 64;
constexpr int kXThreads = 6 * 32;
constexpr int kXBars = 256;
constexpr float kXLog2e = 1.4426950408889634f;

struct FlashTcArgs {
    const int32_t *seq_info;  // 4 numbers a sequence: first token, tokens, position of the first, -
    int num_seqs, run /* tokens per CTA */, group;
    const int32_t *block_table;
    int max_pages, num_pages, page_size;
    int k_steps /* 16-column steps of the scores */, k_first /* key blocks from the first map */, dv;
    int mask, mask_size, keep_first, sink, weights;
    float scale, softcap;
    const float *head_bias;
    const bf16 *gate;
    long long g_token;
    int gate_wide;
    bf16 *out;
    long long o_token, o_head;
    int o_wide /* 16-byte stores */;
};

__device__ __forceinline__ float x_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float x_tanh(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// KB, VB: 64-column blocks of keys and values; VST: value stages.
template <int KB, int VB, int VST>
struct FlashTcShape {
    static constexpr int q_block = 128 * 128, kv_block = kXKeys * 128;
    static constexpr int k_off = KB * q_block, v_off = k_off + 2 * KB * kv_block, bar_off = v_off + VST * VB * kv_block;
    static constexpr int smem = bar_off + kXBars;
    static constexpr int tmem_cols = VB <= 2 ? 256 : 512;
};

template <int KB, int VB, int VST>
__global__ void __launch_bounds__(kXThreads, FlashTcShape<KB, VB, VST>::smem <= 115 * 1024 && VB <= 2 ? 2 : 1)
flash_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k0, const __grid_constant__ CUtensorMap map_k1,
                const __grid_constant__ CUtensorMap map_v, const FlashTcArgs a) {
    using Z = FlashTcShape<KB, VB, VST>;
    constexpr uint32_t O = 128;  // columns: scores [0, 64) and [64, 128), then the output
    extern __shared__ __align__(1024) unsigned char flash_tc_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // the CTA's run of tokens: the (gridDim.x - 1 - blockIdx.x)-th over all sequences, late ones first (they see most keys)
    int seq = -1, first = 0, count = 0, pos0 = 0;
    {
        int left = (int)gridDim.x - 1 - (int)blockIdx.x;
        for (int s0 = 0; s0 < a.num_seqs && seq < 0; s0 += 32) {
            int3 info = make_int3(0, 0, 0);
            if (s0 + lane < a.num_seqs) {
                const int32_t *i = a.seq_info + 4 * (s0 + lane);
                info = make_int3(i[0], i[1], i[2]);
            }
            const int runs = (info.y + a.run - 1) / a.run;
            int sum = runs;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += below;
            }
            const int all = __shfl_sync(0xffffffffu, sum, 31);
            if (left < all) {
                const int at = __ffs(__ballot_sync(0xffffffffu, sum > left)) - 1;
                const int skip = (left - __shfl_sync(0xffffffffu, sum - runs, at)) * a.run;
                seq = s0 + at;
                first = __shfl_sync(0xffffffffu, info.x, at) + skip;
                count = min(a.run, __shfl_sync(0xffffffffu, info.y, at) - skip);
                pos0 = __shfl_sync(0xffffffffu, info.z, at) + skip;
            }
            left -= all;
        }
    }
    if (seq < 0) return;  // the grid is an upper bound

    const int g = blockIdx.y, head0 = g * a.group;
    // the key tiles: kept first positions that the window does not reach, then from `lo` to the newest key
    const int hi = pos0 + count - 1;
    int lo = 0;
    if (a.mask == 1) lo = max(0, pos0 - a.mask_size + 1);
    if (a.mask == 2) lo = pos0 / a.mask_size * a.mask_size;
    lo = lo / kXKeys * kXKeys;
    const int kept_tiles = a.mask == 1 ? min(lo, (a.keep_first + kXKeys - 1) / kXKeys * kXKeys) / kXKeys : 0;
    const int n_tiles = kept_tiles + (hi - lo) / kXKeys + 1;
    auto tile_key = [&](int t) { return t < kept_tiles ? t * kXKeys : lo + (t - kept_tiles) * kXKeys; };

    const uint32_t base = g_smem_u32(flash_tc_smem), k_at = base + Z::k_off, v_at = base + Z::v_off, bar = base + Z::bar_off;
    const uint32_t q_full = bar, s_full = bar + 8, p_full = bar + 24, pv_done = bar + 40, k_full = bar + 56, k_empty = bar + 72, v_full = bar + 88, v_empty = bar + 104;
    volatile int *dead = reinterpret_cast<volatile int *>(flash_tc_smem + Z::bar_off + 120);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(flash_tc_smem + Z::bar_off + 124);
    if (warp == 5 && lane == 0) {
        g_mbar_init(q_full, 1);
        // two of each, by the tile's parity: a warp hands its weights over without waiting for the last tile's product.  A wait by
        // parity passes at once while its barrier is still in the phase BEFORE the one waited for, so a wait that is not made for
        // every phase needs another reason why that phase is over.  S_t complete means that the products before it, P_(t-2) V_(t-2)
        // among them, are (the tensor core takes them in order, and a commit covers all before it): enough for pv_done of tile
        // t - 1, whose phase before is tile t - 3, not for v_full of a single stage (below).
        for (int i = 0; i < 2; ++i) g_mbar_init(p_full + 8 * i, 4), g_mbar_init(pv_done + 8 * i, 1);
        for (int i = 0; i < 2; ++i) g_mbar_init(s_full + 8 * i, 1), g_mbar_init(k_full + 8 * i, 1), g_mbar_init(k_empty + 8 * i, 1);
        for (int i = 0; i < VST; ++i) g_mbar_init(v_full + 8 * i, 1), g_mbar_init(v_empty + 8 * i, 1);
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k0) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem_u32(tmem_slot)), "n"(Z::tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    g_tc_fence_before();
    __syncthreads();
    g_tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int32_t *table = a.block_table + (size_t)seq * a.max_pages;

    if (warp == 4) {  // ---- TMA
        if (g_elect_one()) {
            g_mbar_expect_tx(q_full, KB * a.run * a.group * 128);
#pragma unroll
            for (int b = 0; b < KB; ++b) g_tma_load_3d(base + b * Z::q_block, &map_q, b * 64, head0, first, q_full);
        }
        __syncwarp();
        int ks = 0, vs = 0;
        uint32_t kph = 1, vph = 1;
        for (int t = 0; t < n_tiles; ++t) {
            const int key = tile_key(t), page = table[key / a.page_size];
            const int row = (page >= 0 && page < a.num_pages ? page : a.num_pages) * a.page_size + key % a.page_size;  // past the last page: zeros
            if (!tc_wait(k_empty + 8 * ks, kph, dead)) break;
            if (g_elect_one()) {
                g_mbar_expect_tx(k_full + 8 * ks, KB * Z::kv_block);
#pragma unroll
                for (int b = 0; b < KB; ++b) {
                    const uint32_t to = k_at + (ks * KB + b) * Z::kv_block;
                    if (b < a.k_first) g_tma_load_3d(to, &map_k0, b * 64, g, row, k_full + 8 * ks);
                    else g_tma_load_3d(to, &map_k1, (b - a.k_first) * 64, 0, row, k_full + 8 * ks);
                }
            }
            __syncwarp();
            if (++ks == 2) ks = 0, kph ^= 1u;
            if (!tc_wait(v_empty + 8 * vs, vph, dead)) break;
            if (g_elect_one()) {
                g_mbar_expect_tx(v_full + 8 * vs, VB * Z::kv_block);
#pragma unroll
                for (int b = 0; b < VB; ++b) g_tma_load_3d(v_at + (vs * VB + b) * Z::kv_block, &map_v, b * 64, g, row, v_full + 8 * vs);
            }
            __syncwarp();
            if (++vs == VST) vs = 0, vph ^= 1u;
        }
    } else if (warp == 5) {  // ---- MMA: S_0, then per tile S_(t+1), P_t V_t
        constexpr uint32_t idesc_s = tc_idesc(kXKeys), idesc_o = tc_idesc(64 * VB, true);
        const uint64_t qd = g_smem_desc_sw128(base, 0, 1024), kd0 = g_smem_desc_sw128(k_at, 0, 1024), vd0 = g_smem_desc_sw128(v_at, Z::kv_block, 1024);
        int ks = 0, vs = 0;
        uint32_t kph = 0, vph = 0;
        auto scores = [&](int t) {
            if (!tc_wait(k_full + 8 * ks, kph, dead)) return false;
            g_tc_fence_after();
            if (g_elect_one()) {
                const uint64_t kd = kd0 + (uint64_t)(ks * KB * (Z::kv_block >> 4));
#pragma unroll
                for (int k = 0; k < KB * 4; ++k)
                    if (k < a.k_steps)
                        g_tc_mma(tmem + (t & 1) * kXKeys, qd + (k >> 2) * (Z::q_block >> 4) + 2 * (k & 3), kd + (k >> 2) * (Z::kv_block >> 4) + 2 * (k & 3), idesc_s, k > 0);
                g_tc_commit(k_empty + 8 * ks);
                g_tc_commit(s_full + 8 * (t & 1));
            }
            __syncwarp();
            if (++ks == 2) ks = 0, kph ^= 1u;
            return true;
        };
        const bool begun = tc_wait(q_full, 0, dead) && scores(0);
        for (int t = 0; begun && t < n_tiles; ++t) {
            if (t + 1 < n_tiles && !scores(t + 1)) break;  // its buffer held P_(t-1), read by a product already queued ahead of this one
            if (!tc_wait(p_full + 8 * (t & 1), (t >> 1) & 1, dead) || !tc_wait(v_full + 8 * vs, vph, dead)) break;
            g_tc_fence_after();
            if (g_elect_one()) {
                const uint64_t vd = vd0 + (uint64_t)(vs * VB * (Z::kv_block >> 4));
#pragma unroll
                for (int k = 0; k < kXKeys / 16; ++k) g_tc_mma_ts(tmem + O, tmem + (t & 1) * kXKeys + 8 * k, vd + k * (2048 >> 4), idesc_o, t > 0 || k > 0);
                g_tc_commit(v_empty + 8 * vs);
                g_tc_commit(pv_done + 8 * (t & 1));
            }
            __syncwarp();
            if (++vs == VST) vs = 0, vph ^= 1u;
        }
    } else {  // ---- softmax: thread = row
        const int r = threadIdx.x, tq = r / a.group, hh = r - tq * a.group;
        const bool live = tq < count;
        const int p = pos0 + tq;
        const int see_hi = live ? p : -1;
        const int see_lo = !live ? 0x7fffffff : a.mask == 1 ? max(0, p - a.mask_size + 1) : a.mask == 2 ? p / a.mask_size * a.mask_size : 0;
        const int first_kept = a.mask == 1 ? a.keep_first : 0;
        const uint32_t lanes = static_cast<uint32_t>(warp * 32) << 16;
        const float bias = a.head_bias && live ? a.head_bias[head0 + hh] * kXLog2e : 0.f;
        // scores enter the exponential in base 2; where the scale is positive and there is no cap, the maximum is taken over the
        // products as they are
        const float scale2 = a.scale * kXLog2e, cap_in = a.softcap > 0.f ? a.scale / a.softcap : 0.f, cap_out = a.softcap * kXLog2e;
        const bool raw = a.softcap <= 0.f && a.scale > 0.f && a.weights == 0;
        const float mult = raw ? scale2 : 1.f;
        float m = a.weights == 1 ? 0.f : a.sink ? bias : -INFINITY;       // the maximum P and the sums refer to, in base 2
        float sum = a.sink || a.weights == 1 ? 1.f : 0.f;                 // the sink's term (m is its score), or the sigmoid form's constant
        int vs = 0;
        uint32_t vph = 0;
        bool ok = true;
        for (int t = 0; t < n_tiles; ++t) {
            const int key0 = tile_key(t);
            if (!(ok = tc_wait(s_full + 8 * (t & 1), (t >> 1) & 1, dead))) break;
            g_tc_fence_after();
            uint32_t s[2][32];
            g_tmem_ld32_nowait(tmem + lanes + (t & 1) * kXKeys, s[0]);
            g_tmem_ld32_nowait(tmem + lanes + (t & 1) * kXKeys + 32, s[1]);
            g_tmem_ld_wait();
            if (a.softcap > 0.f) {
#pragma unroll
                for (int c = 0; c < kXKeys; ++c) s[c >> 5][c & 31] = __float_as_uint(cap_out * x_tanh(__uint_as_float(s[c >> 5][c & 31]) * cap_in));
            } else if (!raw) {
#pragma unroll
                for (int c = 0; c < kXKeys; ++c) s[c >> 5][c & 31] = __float_as_uint(__uint_as_float(s[c >> 5][c & 31]) * scale2);
            }
            const bool cut = key0 + kXKeys - 1 > see_hi || (key0 < see_lo && key0 + kXKeys > first_kept);
            if (__any_sync(0xffffffffu, cut)) {
#pragma unroll
                for (int c = 0; c < kXKeys; ++c) {
                    const int key = key0 + c;
                    if (key > see_hi || (key < see_lo && key >= first_kept)) s[c >> 5][c & 31] = 0xff800000u;
                }
            }
            uint32_t pk[32];
            if (a.weights == 1) {  // every visible key by itself: no maximum, no sum, nothing to rescale
#pragma unroll
                for (int c = 0; c < kXKeys; c += 2) {
                    const float x = __uint_as_float(s[c >> 5][c & 31]), y = __uint_as_float(s[c >> 5][(c & 31) + 1]);
                    pk[c / 2] = tl::pack2<bf16>(x == -INFINITY ? 0.f : 1.0f / (1.0f + x_ex2(-(x + bias))), y == -INFINITY ? 0.f : 1.0f / (1.0f + x_ex2(-(y + bias))));
                }
            } else {
                float top = -INFINITY;
#pragma unroll
                for (int c = 0; c < kXKeys; ++c) top = fmaxf(top, __uint_as_float(s[c >> 5][c & 31]));
                top *= mult;
                const bool grow = top > m;
                if (__any_sync(0xffffffffu, grow) && t > 0) {
                    if (!(ok = tc_wait(pv_done + 8 * ((t - 1) & 1), ((t - 1) >> 1) & 1, dead))) break;  // O has to be still while it is rescaled
                    g_tc_fence_after();
                    const float to = grow ? top : m;
                    const float alpha = !grow ? 1.f : m == -INFINITY ? 0.f : x_ex2(m - to);
                    sum *= alpha;
#pragma unroll
                    for (int b = 0; b < 2 * VB; ++b) {
                        uint32_t o[32];
                        g_tmem_ld32(tmem + lanes + O + b * 32, o);
#pragma unroll
                        for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * alpha);
                        g_tmem_st32(tmem + lanes + O + b * 32, o);
                    }
                    g_tmem_st_wait();
                    m = to;
                } else if (grow) {
                    sum *= m == -INFINITY ? 0.f : x_ex2(m - top);  // first tile: only the sink's term so far
                    m = top;
                }
                const float at = m == -INFINITY ? 0.f : m;
                float s0 = 0.f, s1 = 0.f;
#pragma unroll
                for (int c = 0; c < kXKeys; c += 2) {
                    const uint32_t u = tl::pack2<bf16>(x_ex2(fmaf(__uint_as_float(s[c >> 5][c & 31]), mult, -at)), x_ex2(fmaf(__uint_as_float(s[c >> 5][(c & 31) + 1]), mult, -at)));
                    pk[c / 2] = u;
                    s0 += __uint_as_float(u << 16), s1 += __uint_as_float(u & 0xffff0000u);  // numerator and denominator see the same rounded weights
                }
                sum += s0 + s1;
            }
            g_tmem_st32(tmem + lanes + (t & 1) * kXKeys, pk);  // column c = keys 2 c and 2 c + 1
            g_tmem_st_wait();
            if (key0 + kXKeys - 1 > hi) {  // values past the newest key: cleared before the product may read them
                // These warps wait on v_full here only, and a parity says nothing unless the phase before it is known to be over: with
                // one stage that is V_(t-1), which may still be on its way when S_t is complete (nothing orders its load before K_t's).
                // Its product is the proof that it landed and was read.  With two stages it is V_(t-2), whose product S_t follows.
                if constexpr (VST == 1)
                    if (t > 0 && !(ok = tc_wait(pv_done + 8 * ((t - 1) & 1), ((t - 1) >> 1) & 1, dead))) break;
                if (!(ok = tc_wait(v_full + 8 * vs, vph, dead))) break;
                if (r < kXKeys && key0 + r > hi) {
#pragma unroll
                    for (int i = 0; i < VB * 8; ++i)
                        *reinterpret_cast<uint4 *>(flash_tc_smem + Z::v_off + (vs * VB + i / 8) * Z::kv_block + r * 128 + (i % 8) * 16) = make_uint4(0, 0, 0, 0);
                }
                tl::g_fence_proxy_async();
            }
            if (++vs == VST) vs = 0, vph ^= 1u;
            g_tc_fence_before();
            __syncwarp();
            if (lane == 0) g_mbar_arrive(p_full + 8 * (t & 1));
        }
        ok = ok && tc_wait(pv_done + 8 * ((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1, dead);
        g_tc_fence_after();
        float inv = (sum > 0.f ? 1.0f / sum : 0.f) * tc_verdict(ok, dead);
        if (live && a.gate && !a.gate_wide) inv *= sigmoid(__bfloat162float(a.gate[(size_t)(first + tq) * a.g_token + head0 + hh]));
        bf16 *out = a.out + (size_t)(first + tq) * a.o_token + (size_t)(head0 + hh) * a.o_head;
        const bf16 *wide = a.gate_wide ? a.gate + (size_t)(first + tq) * a.g_token + (size_t)(head0 + hh) * a.dv : nullptr;
#pragma unroll
        for (int b = 0; b < 2 * VB; ++b) {
            uint32_t o[32];
            g_tmem_ld32(tmem + lanes + O + b * 32, o);
            if (!live) continue;
            if (a.o_wide && !wide) {
#pragma unroll
                for (int c = 0; c < 32; c += 8) {
                    if (b * 32 + c >= a.dv) break;
                    uint4 u;
                    u.x = tl::pack2<bf16>(__uint_as_float(o[c]) * inv, __uint_as_float(o[c + 1]) * inv);
                    u.y = tl::pack2<bf16>(__uint_as_float(o[c + 2]) * inv, __uint_as_float(o[c + 3]) * inv);
                    u.z = tl::pack2<bf16>(__uint_as_float(o[c + 4]) * inv, __uint_as_float(o[c + 5]) * inv);
                    u.w = tl::pack2<bf16>(__uint_as_float(o[c + 6]) * inv, __uint_as_float(o[c + 7]) * inv);
                    *reinterpret_cast<uint4 *>(out + b * 32 + c) = u;
                }
            } else {
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    const int col = b * 32 + c;
                    if (col < a.dv) out[col] = __float2bfloat16_rn(__uint_as_float(o[c]) * inv * (wide ? sigmoid(__bfloat162float(wide[col])) : 1.f));
                }
            }
        }
    }
    g_tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_settle(dead);
        g_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(Z::tmem_cols) : "memory");
    }
}

// What a launch needs beside FlashTcArgs: where queries, keys and values lie (elements; unit stride within a head).
struct FlashTcOperands {
    const void *q, *k0, *k1, *v;
    long long q_token, q_head, k0_head, k0_row, k1_row, v_head, v_row;
    int tokens, heads, kv_heads, dk, dk0 /* of which from k0 */, runs;
    long long rows;
};

template <int KB, int VB, int VST>
static int flash_tc_run(const FlashTcOperands &x, const FlashTcArgs &a, cudaStream_t st) {
    using Z = FlashTcShape<KB, VB, VST>;
    CUtensorMap mq, m0, m1, mv;
    if (int e = tc_map_3d(&mq, x.q, x.dk, x.heads, x.tokens, x.q_head, x.q_token, a.group, a.run)) return e;
    if (int e = tc_map_3d(&m0, x.k0, x.dk0, x.kv_heads, x.rows, x.k0_head, x.k0_row, 1, kXKeys)) return e;
    m1 = m0;
    if (x.k1)
        if (int e = tc_map_3d(&m1, x.k1, x.dk - x.dk0, 1, x.rows, x.k1_row, x.k1_row, 1, kXKeys)) return e;
    if (int e = tc_map_3d(&mv, x.v, a.dv, x.kv_heads, x.rows, x.v_head, x.v_row, 1, kXKeys)) return e;
    auto kernel = flash_tc_kernel<KB, VB, VST>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Z::smem) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess) {
        cudaGetLastError();
        return tl::fail(TL_ECUDA, "flash_tc: no shared memory");
    }
    kernel<<<dim3(x.runs, x.kv_heads), kXThreads, Z::smem, st>>>(mq, m0, m1, mv, a);
    return TL_OK;
}

static int flash_tc_launch(const FlashTcOperands &x, const FlashTcArgs &a, cudaStream_t st) {
    const int kb = ceil_div(x.dk0, 64) + (x.k1 ? ceil_div(x.dk - x.dk0, 64) : 0), vb = ceil_div(a.dv, 64);
    int rc;
#define TLB_X(K, V, S) rc = flash_tc_run<K, V, S>(x, a, st)
    switch (kb) {
        case 1: if (vb == 1) TLB_X(1, 1, 2); else if (vb == 2) TLB_X(1, 2, 2); else TLB_X(1, 4, 2); break;
        case 2: if (vb == 1) TLB_X(2, 1, 2); else if (vb == 2) TLB_X(2, 2, 2); else TLB_X(2, 4, 2); break;
        case 3: if (vb == 1) TLB_X(3, 1, 2); else if (vb == 2) TLB_X(3, 2, 1); else TLB_X(3, 4, 2); break;
        default: if (vb == 1) TLB_X(4, 1, 2); else if (vb == 2) TLB_X(4, 2, 2); else TLB_X(4, 4, 2); break;
    }
#undef TLB_X
    if (rc != TL_OK) return rc;
    TL_LAUNCH_CHECK("flash_tc");
    return TL_OK;
}

// A latent layer's cached rows of every sequence that a query of the step may see (window > 0: from the tile of the first query's first
// visible key on), one after the other from whole 64-row pages on, and the block table that finds them there: what the up projections of
// keys and values read.  Rows past a sequence's newest token are zeros.  `seen` [num_seqs, 4], or NULL: seq_info with positions counted
// from the first row kept; that is a whole tile, so the attention takes the same tiles as over all rows.
constexpr int kRowParts = 4;
__global__ void __launch_bounds__(256)
latent_rows_kernel(const bf16 *__restrict__ slab, int num_pages, int page_size, int width, const int32_t *__restrict__ seq_info, int num_seqs,
                   const int32_t *__restrict__ block_table, int max_pages, int window, bf16 *__restrict__ rows, int32_t *__restrict__ table, int table_pages, int total_pages,
                   int32_t *__restrict__ seen) {
    constexpr int ROWS = kXKeys / kRowParts;  // of a page a CTA
    const int s = blockIdx.y, p = blockIdx.x / kRowParts, row0 = blockIdx.x % kRowParts * ROWS, lane = threadIdx.x & 31;
    auto skipped = [&](int i) { return window > 0 ? max(0, seq_info[4 * i + 2] - window + 1) / kXKeys * kXKeys : 0; };
    auto context = [&](int i) { return seq_info[4 * i + 1] + seq_info[4 * i + 2] - skipped(i); };
    const int skip = skipped(s), ctx = context(s);
    if (seen && blockIdx.x == 0 && threadIdx.x < 4) seen[4 * s + threadIdx.x] = seq_info[4 * s + threadIdx.x] - (threadIdx.x == 2 ? skip : 0);
    if (p * kXKeys >= ctx) return;
    int before = 0;
    for (int i = lane; i < s; i += 32) before += (context(i) + kXKeys - 1) / kXKeys;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (before + p >= total_pages || p >= table_pages) return;
    if (threadIdx.x == 0 && row0 == 0) table[(size_t)s * table_pages + p] = before + p;
    const int pieces = width / 8;
    for (int i = threadIdx.x; i < ROWS * pieces; i += 256) {
        const int j = row0 + i / pieces, piece = i % pieces, key = skip + p * kXKeys + j;
        const int page = key < skip + ctx && key / page_size < max_pages ? block_table[(size_t)s * max_pages + key / page_size] : -1;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (page >= 0 && page < num_pages) v = *reinterpret_cast<const uint4 *>(slab + ((size_t)page * page_size + key % page_size) * width + piece * 8);
        *reinterpret_cast<uint4 *>(rows + ((size_t)(before + p) * kXKeys + j) * width + piece * 8) = v;
    }
}

long long flash_tc_gave_up() { return tl::read_gave_up(); }

static bool map_ok(const void *p, long long s0, long long s1) { return tl::aligned16(p) && s0 % 8 == 0 && s1 % 8 == 0; }

}  // namespace tlb

using namespace tlb;

extern "C" {

int tlb_flash_tc_run_tokens(int heads, int kv_heads) {
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || heads / kv_heads > 128) return 0;
    return 128 / (heads / kv_heads);
}

int tlb_flash_tc_supported(int dk, int dv, int heads, int kv_heads, int page_size) {
    return dk > 0 && dv > 0 && dk % 8 == 0 && dv % 8 == 0 && dk <= 256 && dv <= 256 && page_size > 0 && page_size % kXKeys == 0 && tlb_flash_tc_run_tokens(heads, kv_heads) > 0;
}

int tlb_paged_attention_tc(const void *q, long long q_token, long long q_head, int tokens, const void *slab, int num_pages, int page_size, int dk, int dv, int heads,
                           int kv_heads, const int32_t *block_table, int max_pages, const int32_t *seq_info, int num_seqs, int runs, int mask, int mask_size,
                           int keep_first, float scale, float softcap, int sink, const void *gate, long long g_token, int gate_wide, void *out, long long o_token,
                           long long o_head, const float *head_bias, int weights, void *stream) {
    if (runs <= 0 || tokens <= 0) return TL_OK;
    if (!q || !slab || !block_table || !seq_info || !out || max_pages <= 0 || num_pages <= 0 || num_seqs <= 0)
        return tl::fail(TL_EINVAL, "paged_attention_tc: bad argument");
    if (weights < 0 || weights > 1 || (weights == 1 && (sink || softcap > 0.f))) return tl::fail(TL_EINVAL, "paged_attention_tc: bad weights mode");
    if (!tlb_flash_tc_supported(dk, dv, heads, kv_heads, page_size) || !map_ok(q, q_token, q_head) || !tl::aligned16(slab) || kv_heads > 65535)
        return tl::fail(TL_EINVAL, "paged_attention_tc: unsupported sizes or alignment");
    if (mask < 0 || mask > 2 || (mask != 0 && mask_size <= 0) || keep_first < 0 || keep_first > (1 << 30) || (keep_first > 0 && mask != 1))
        return tl::fail(TL_EINVAL, "paged_attention_tc: bad mask");
    const long long row = (long long)kv_heads * (dk + dv);
    FlashTcOperands x = {q, slab, nullptr, (const bf16 *)slab + (size_t)kv_heads * dk, q_token, q_head, dk, row, 0, dv, row, tokens, heads, kv_heads, dk, dk, runs,
                         (long long)num_pages * page_size};
    FlashTcArgs a = {};
    a.seq_info = seq_info, a.num_seqs = num_seqs, a.run = tlb_flash_tc_run_tokens(heads, kv_heads), a.group = heads / kv_heads;
    a.block_table = block_table, a.max_pages = max_pages, a.num_pages = num_pages, a.page_size = page_size;
    a.k_steps = ceil_div(dk, 16), a.k_first = 4, a.dv = dv;
    a.mask = mask, a.mask_size = mask_size, a.keep_first = keep_first, a.sink = sink, a.weights = weights, a.scale = scale, a.softcap = softcap, a.head_bias = head_bias;
    a.gate = (const bf16 *)gate, a.g_token = g_token, a.gate_wide = gate && gate_wide;
    a.out = (bf16 *)out, a.o_token = o_token, a.o_head = o_head, a.o_wide = map_ok(out, o_token, o_head);
    return flash_tc_launch(x, a, as_stream(stream));
}

int tlb_latent_rows(const void *slab, int num_pages, int page_size, int width, const int32_t *seq_info, int num_seqs, const int32_t *block_table, int max_pages, void *rows,
                    int window, int32_t *table, int table_pages, int total_pages, int32_t *seen, void *stream) {
    if (num_seqs <= 0 || total_pages <= 0) return TL_OK;
    if (!slab || !seq_info || !block_table || !rows || !table || num_pages <= 0 || page_size <= 0 || max_pages <= 0 || table_pages <= 0 || width <= 0 || width % 8 || window < 0 ||
        !tl::aligned16(slab) || !tl::aligned16(rows) || num_seqs > 65535)
        return tl::fail(TL_EINVAL, "latent_rows: bad argument");
    latent_rows_kernel<<<dim3(table_pages * kRowParts, num_seqs), 256, 0, as_stream(stream)>>>((const bf16 *)slab, num_pages, page_size, width, seq_info, num_seqs,
                                                                                   block_table, max_pages, window, (bf16 *)rows, table, table_pages, total_pages, seen);
    TL_LAUNCH_CHECK("latent_rows");
    return TL_OK;
}

int tlb_latent_attention_heads(const void *q, long long q_token, long long q_head, int tokens, const void *k, long long k_row, const void *v, long long v_head,
                               long long v_row, const void *k_rot, long long k_rot_row, int dim, int rot, int dv, int heads, long long rows, const int32_t *table,
                               int table_pages, const int32_t *seq_info, int num_seqs, int runs, int window, float scale, void *out, long long o_token,
                               long long o_head, const float *sink, void *stream) {
    if (runs <= 0 || tokens <= 0) return TL_OK;
    if (!q || !k || !v || (rot > 0 && !k_rot) || !table || !seq_info || !out || heads <= 0 || heads > 65535 || num_seqs <= 0 || table_pages <= 0 || rows <= 0 ||
        rows % kXKeys)
        return tl::fail(TL_EINVAL, "latent_attention_heads: bad argument");
    if (dim <= 0 || dim % 64 || rot < 0 || rot % 8 || dim + rot > 256 || rot > 64 || dv <= 0 || dv % 8 || dv > 256 || !map_ok(q, q_token, q_head) || !map_ok(k, dim, k_row) ||
        !map_ok(v, v_head, v_row) || (rot > 0 && !map_ok(k_rot, k_rot_row, 0)))
        return tl::fail(TL_EINVAL, "latent_attention_heads: unsupported sizes or alignment");
    FlashTcOperands x = {q, k, rot > 0 ? k_rot : nullptr, v, q_token, q_head, dim, k_row, k_rot_row, v_head, v_row, tokens, heads, heads, dim + rot, dim, runs, rows};
    FlashTcArgs a = {};
    a.seq_info = seq_info, a.num_seqs = num_seqs, a.run = 128, a.group = 1;
    a.block_table = table, a.max_pages = table_pages, a.num_pages = (int)(rows / kXKeys), a.page_size = kXKeys;
    a.k_steps = ceil_div(dim + rot, 16), a.k_first = dim / 64, a.dv = dv;
    a.mask = window > 0 ? 1 : 0, a.mask_size = window, a.sink = sink != nullptr, a.head_bias = sink, a.scale = scale;
    a.out = (bf16 *)out, a.o_token = o_token, a.o_head = o_head, a.o_wide = map_ok(out, o_token, o_head);
    return flash_tc_launch(x, a, as_stream(stream));
}

}  // extern "C"
