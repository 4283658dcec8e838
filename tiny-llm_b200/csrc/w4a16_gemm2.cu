// W4A16 prefill GEMM on CTA PAIRS (tcgen05 cta_group::2): the large-M form of w4a16_gemm.cu.
//
//   out[m, n] = sum_k a[m, k] * T(code[n, k] * scale[n, k/128] + bias[n, k/128])       (m = token, n = feature)
//
// Why pairs: with cta_group::2 one MMA spans 256 token rows (128 per CTA) x 256 weight rows, each CTA dequantises HALF of the weight tile into its own
// shared memory and the tensor cores of both SMs read both halves.  Per CTA and 64-wide block that is 32 KB of activations (two 256-token MMA
// tiles) and one dequantised tile for 1024 cycles of tensor work.  The one-CTA kernel needs 68 KB from L2 for the same (about 42 bytes a cycle and
// SM is what the chip gives), and 208 KB through its shared memory (operands read, tiles written), 1640 cycles at 128 bytes a cycle;
// here it is 112 KB.
//
// Persistent: one pair of CTAs per two SMs takes tiles in turn, so that the next tile's activations and weights arrive, and are unpacked, while the last
// one's results are read out by warps of their own and leave by TMA.  (With a CTA pair a tile, its dequantisers reading the results out in 16-byte
// stores of 32 rows each, a tile cost 24 us beside its blocks.)
//
// Roles per CTA (640 threads): warp 0 TMA producer (its 128 token rows of each MMA tile), warp 1 MMA issuer in the
// leader CTA (rank 0) / readiness forwarder in the peer, warp 2 TMEM allocation (cta_group::2, all 512 columns: two
// accumulators of 256 features), warps 4-11 dequantisers, warps 12-19 epilogue (lane = token row).
// Barriers live at the same offsets in both CTAs: full (own TMA + own dequantisers; in the leader also the peer's
// "my tiles of this stage are complete"), empty and acc_full (arrived in BOTH CTAs by the leader's multicast commit), acc_empty (the leader's: both CTAs'
// epilogue warps).  Every wait is bounded (tc_wait.cuh); a CTA whose wait gave up stores NaN.
// Replaces quantized_matmul_simdgroup_w4a16_g128 (src/extensions_ref/src/quantized_matmul.metal:96-249)
// for larger M; same rounding points as w4a16_gemm.cu (weights rounded to the activation dtype, fp32 accumulation).
//
// Measured (bf16; before: a pair of CTAs a tile): 2048 rows of 2560 -> 19456 230 -> 139 us (1464 TF/s, 90 % of the measured burst), 4096 rows 442 -> 264
// (1546 TF/s), 2560 -> 9728 131 -> 77; gate and up projection with their activation in one launch, 2048 rows of 2560 -> 9728: 244 (two
// launches of the one-CTA kernel and one of the activation) -> 155 us, fp16 243 -> 173; 129 rows 50 -> 43 and 51 -> 48.
#include <cuda.h>
#include <stdlib.h>
#include <cudaTypedefs.h>

#include "common.cuh"
#include "kernels.h"
#include "per_device.h"
#include "tc_wait.cuh"
#include "trace.cuh"

namespace tl {

constexpr int P_TOK = 128;        // token rows per CTA and MMA tile (the pair's MMA spans 256)
constexpr int P_ROWS = 128;       // weight rows dequantised per CTA (the pair's MMA spans 256)
constexpr int P_KB = 64;          // reduction elements per stage (one 128-byte swizzle atom)
constexpr int P_MT = 2;           // 256-token MMA tiles per pair: 2 x 256 accumulator columns = all of TMEM
constexpr int P_STAGES = 4;
constexpr int P_TILE = P_TOK * P_KB * 2;          // 16 KiB, activation and weight tiles alike
constexpr int P_A_STAGE = P_MT * P_TILE;
constexpr int P_STAGE = P_A_STAGE + P_TILE;       // 48 KiB
constexpr int P_DEQ_WARPS = 8, P_EPI_WARPS = 8;
constexpr int P_OUT_OFF = P_STAGES * P_STAGE;     // 192 KiB; then 32 token rows x 64 features of results per epilogue warp
constexpr int P_OUT_BYTES = 32 * 128;
constexpr int P_BAR_OFF = P_OUT_OFF + P_EPI_WARPS * P_OUT_BYTES;
constexpr int P_SMEM = P_BAR_OFF + 256;
constexpr int P_THREADS = 32 * (4 + P_DEQ_WARPS + P_EPI_WARPS);
constexpr int P_TMEM_COLS = 512;

// ---- cluster / pair primitives ------------------------------------------------
__device__ __forceinline__ uint32_t p_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void p_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// An arrival on the barrier at this shared-memory offset in the leader.  What it reports (tiles in, or accumulators out of, the arriving CTA's own
// memory) is read and written by that CTA's own SM and has been ordered there by a barrier or a proxy fence; a release at cluster
// scope, which was here before, waits for all of the SM's memory traffic: 2000 cycles a stage under load (512 tokens of 2560 -> 18944:
// 60 -> 45 us without it).
__device__ __forceinline__ void p_mbar_arrive_leader(uint32_t bar) {
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, 0;\n\tmbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void p_tc_mma2(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// completion of all MMAs issued so far -> one arrival on the barrier at this offset in BOTH CTAs of the pair
__device__ __forceinline__ void p_tc_commit2(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(static_cast<unsigned short>(3))
                 : "memory");
}

__device__ __forceinline__ void p_tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {  // without the wait
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
          "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

template <typename T>
__host__ __device__ constexpr uint32_t p_instr_desc() {
    const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;  // 0 = f16, 1 = bf16
    return (1u << 4) | (fmt << 7) | (fmt << 10) | (0u << 15) | (0u << 16) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
}

template <typename T>
struct PDeq;
template <>
struct PDeq<__nv_bfloat16> {
    using V2 = __nv_bfloat162;
    static constexpr uint32_t MAGIC = 0x43004300u;  // (128, 128)
};
template <>
struct PDeq<__half> {
    using V2 = __half2;
    static constexpr uint32_t MAGIC = 0x64006400u;  // (1024, 1024)
};

// What a pair works on: n_tiles feature tiles x groups of two 256-token tiles, dealt to the pairs in turn.  The first `full` of them go out whole; the
// rest, which would fill less than half of a last round, in single 256-token tiles.
struct PairPlan {
    int n_tiles, m_tiles, full, items;
};
struct PairItem {
    int n_tile, m0, mt;  // feature tile, first 256-token tile, how many (0: nothing, a short group's second half)
};
__host__ __device__ __forceinline__ PairItem pair_item(const PairPlan &p, int i) {
    int tile = i, m0 = 0, most = P_MT;
    if (i >= p.full) tile = p.full + (i - p.full) / P_MT, m0 = (i - p.full) % P_MT, most = 1;
    m0 += tile / p.n_tiles * P_MT;
    const int left = p.m_tiles - m0;
    return {tile % p.n_tiles, m0, left < most ? (left < 0 ? 0 : left) : most};
}

template <typename T>
struct PairWeights {
    const T *scales, *biases;
    const uint32_t *b;
};

// GATED: out = silu(a gate^T) * (a up^T), both rounded to T first.  The leader brings 128 rows of the gate, the peer the same 128 of the up projection, so
// that both halves of a feature's pair lie in the same lane of tensor memory, 128 columns apart.
template <typename T, bool GATED>
__global__ void __launch_bounds__(P_THREADS, 1)
w4a16_gemm2_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_out, const PairWeights<T> w0, const PairWeights<T> w1,
                   T *__restrict__ out, int M, int N, int K, int tma_store, const PairPlan plan) {
    extern __shared__ __align__(1024) unsigned char psm[];
#if TL_TRACE
    // per-block cycle stamps of the leader CTA's first tile (tools/gemm_blocks.py): role 0 = MMA warp (k: stage complete in both
    // CTAs, -, MMAs issued), role 1 = first dequantiser warp (k: loop top, math done, stage free, handed over)
    __shared__ unsigned int trc[2][40][4];  // (of 64 bits it would not fit beside the stages)
#define P_TRC(role, item, i, k)                                                                                              \
    do {                                                                                                                     \
        if (blockIdx.x == 0 && (item) == 0 && (threadIdx.x & 31) == 0 && (i) < 40) trc[role][i][k] = static_cast<unsigned int>(clock64()); \
    } while (0)
#else
#define P_TRC(role, item, i, k) do { } while (0)
#endif
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = static_cast<int>(p_cta_rank());       // 0 = leader (issues the MMAs)
    const int unit = blockIdx.x >> 1, units = gridDim.x >> 1;
    const int num_kb = N / P_KB;
    const int G = N / 128;
    constexpr int FEATURES = GATED ? P_ROWS : 2 * P_ROWS;  // of a tile

    const uint32_t smem0 = g_smem_u32(psm);
    const uint32_t bar = smem0 + P_BAR_OFF;
    // ONE "full" barrier per stage and CTA: own TMA (expect_tx arrival + bytes) + own eight dequantiser warps; in the
    // leader one more arrival, sent by the peer when ITS barrier of the stage has completed.  The MMA warp pays a single
    // try_wait per block: what it executes between two blocks' MMAs is time the tensor cores idle.
    const uint32_t full = bar, empty = full + 8 * P_STAGES, acc_full = empty + 8 * P_STAGES, acc_empty = acc_full + 8 * P_MT;
    volatile int *dead = reinterpret_cast<volatile int *>(psm + P_BAR_OFF + 16 * P_STAGES + 16 * P_MT);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(const_cast<int *>(dead)) + 1;

    if (warp == 1 && lane == 0) {
        for (int i = 0; i < P_STAGES; ++i) {
            g_mbar_init(full + 8 * i, 1 + P_DEQ_WARPS + (rank == 0 ? 1 : 0));
            g_mbar_init(empty + 8 * i, 1);
        }
        for (int i = 0; i < P_MT; ++i) {
            g_mbar_init(acc_full + 8 * i, 1);
            g_mbar_init(acc_empty + 8 * i, 2 * P_EPI_WARPS);  // both CTAs' (the leader's barrier is the one that is used)
        }
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_out) : "memory");
    }
    if (warp == 2) {  // both CTAs of the pair issue the paired allocation (same shared-memory slot offset)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem_u32(tmem_slot)), "n"(P_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    g_tc_fence_before();
    p_cluster_sync();  // barriers of both CTAs are initialised before anyone arrives remotely; also a CTA barrier
    g_tc_fence_after();
    const uint32_t tmem_d = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------ TMA producer: this CTA's 128 token rows of each MMA tile
        int s = 0;
        uint32_t ph = 1;
        for (int it = unit; it < plan.items; it += units) {
            const PairItem item = pair_item(plan, it);
            for (int kb = 0; item.mt > 0 && kb < num_kb; ++kb) {
                if (!tc_wait(empty + 8 * s, ph, dead)) goto done;
                if (g_elect_one()) {
                    g_mbar_expect_tx(full + 8 * s, item.mt * P_TILE);
#pragma unroll
                    for (int i = 0; i < P_MT; ++i)  // token rows beyond M are zero-filled by the TMA unit
                        if (i < item.mt)
                            g_tma_load_2d(smem0 + s * P_STAGE + i * P_TILE, &tmap_a, kb * P_KB, (item.m0 + i) * 256 + rank * P_TOK, full + 8 * s);
                }
                __syncwarp();
                if (++s == P_STAGES) s = 0, ph ^= 1u;
            }
        }
    } else if (warp == 1 && rank == 0) {
        // ------------------------------------------------ MMA issuer (leader): 256 x 256 x 16 a time
        constexpr uint32_t idesc = p_instr_desc<T>();
        const uint64_t adesc0 = g_smem_desc_sw128(smem0, 0, 1024), bdesc0 = g_smem_desc_sw128(smem0 + P_A_STAGE, 0, 1024);
        int s = 0;
        uint32_t ph = 0, e_ph[P_MT] = {1, 1};
        auto products = [&](int stage, int i, int kb) {  // one lane: a block's four steps of one token tile
            const uint64_t at = static_cast<uint64_t>(stage * (P_STAGE >> 4));
#pragma unroll
            for (int k = 0; k < P_KB / 16; ++k)  // +32 bytes along K per step: +2 in the (addr >> 4) field
                p_tc_mma2(tmem_d + i * 256, adesc0 + at + i * (P_TILE >> 4) + 2 * k, bdesc0 + at + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        };
        for (int it = unit; it < plan.items; it += units) {
            const PairItem item = pair_item(plan, it);
            if (item.mt == 0) continue;
            // The first blocks, as many as there are stages, for the first token tile, then for the second: its accumulator is still being read
            // out for the tile before, meanwhile.
            const int head = min(P_STAGES, num_kb), s0 = s;
            if (!tc_wait(acc_empty, e_ph[0], dead)) goto done;
            e_ph[0] ^= 1u;
            for (int kb = 0; kb < head; ++kb) {
                if (!tc_wait(full + 8 * s, ph, dead)) goto done;
                P_TRC(0, it, kb, 0);
                P_TRC(0, it, kb, 1);
                g_tc_fence_after();
                if (g_elect_one()) {
                    products(s, 0, kb);
                    if (item.mt == 1) p_tc_commit2(empty + 8 * s);
                }
                __syncwarp();
                P_TRC(0, it, kb, 2);
                if (++s == P_STAGES) s = 0, ph ^= 1u;
            }
            if (item.mt > 1) {
                if (!tc_wait(acc_empty + 8, e_ph[1], dead)) goto done;
                e_ph[1] ^= 1u;
                g_tc_fence_after();
                if (g_elect_one())
                    for (int kb = 0; kb < head; ++kb) {
                        const int at = (s0 + kb) % P_STAGES;
                        products(at, 1, kb);
                        p_tc_commit2(empty + 8 * at);  // both CTAs may refill the stage once these MMAs have read it
                    }
                __syncwarp();
            }
            for (int kb = head; kb < num_kb; ++kb) {
                if (!tc_wait(full + 8 * s, ph, dead)) goto done;
                P_TRC(0, it, kb, 0);
                P_TRC(0, it, kb, 1);
                g_tc_fence_after();
                if (g_elect_one()) {
                    products(s, 0, kb);
                    if (kb == num_kb - 1) p_tc_commit2(acc_full);
                    if (item.mt > 1) products(s, 1, kb);
                    p_tc_commit2(empty + 8 * s);
                }
                __syncwarp();
                P_TRC(0, it, kb, 2);
                if (++s == P_STAGES) s = 0, ph ^= 1u;
            }
            if (g_elect_one()) {
                if (head == num_kb) p_tc_commit2(acc_full);
                if (item.mt > 1) p_tc_commit2(acc_full + 8);
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        // ------------------------------------------------ peer: tell the leader when this CTA's tiles of a stage are complete
        int s = 0;
        uint32_t ph = 0;
        for (int it = unit; it < plan.items; it += units)
            for (int kb = 0; pair_item(plan, it).mt > 0 && kb < num_kb; ++kb) {
                if (!tc_wait(full + 8 * s, ph, dead)) goto done;
                if (lane == 0) p_mbar_arrive_leader(full + 8 * s);
                __syncwarp();
                if (++s == P_STAGES) s = 0, ph ^= 1u;
            }
    } else if (warp >= 4 && warp < 4 + P_DEQ_WARPS) {
        // ------------------------------------------------ dequantisers: this CTA's 128 weight rows, thread = (row, 32-element half)
        const int dt = threadIdx.x - 128;
        const int row = dt >> 1, half = dt & 1;  // adjacent lanes = the two 16-byte halves of one weight row
        const PairWeights<T> &w = GATED && rank ? w1 : w0;
        using V2 = typename PDeq<T>::V2;
        const uint32_t magic = PDeq<T>::MAGIC;
        const V2 offset2 = *reinterpret_cast<const V2 *>(&magic);
        auto first_row = [&](int it) { return min(pair_item(plan, it).n_tile * FEATURES + (GATED ? 0 : rank * P_ROWS) + row, K - 1); };
        auto next_item = [&](int it) {
            do it += units;
            while (it < plan.items && pair_item(plan, it).mt == 0);
            return it;
        };
        int s = 0;
        uint32_t ph = 1;
        int it = next_item(unit - units), n = it < plan.items ? first_row(it) : 0, g = 0;  // the group that is fetched next
        uint4 next[2];
        T next_sc, next_bi;
        auto fetch = [&]() {  // a quantisation group, two blocks, ahead of its use
            const uint32_t *at = w.b + static_cast<size_t>(n) * (N / 8) + g * 16 + half * 4;
            next[0] = *reinterpret_cast<const uint4 *>(at), next[1] = *reinterpret_cast<const uint4 *>(at + 8);
            next_sc = w.scales[static_cast<size_t>(n) * G + g], next_bi = w.biases[static_cast<size_t>(n) * G + g];
            if (++g == G) {
                g = 0, it = next_item(it);
                if (it < plan.items) n = first_row(it);
            }
        };
        if (it < plan.items) fetch();
        for (int mine = next_item(unit - units); mine < plan.items; mine = next_item(mine))
            for (int group = 0; group < G; ++group) {
                const uint4 cur[2] = {next[0], next[1]};
                V2 s2, b2;
                s2.x = s2.y = next_sc, b2.x = b2.y = next_bi;
                if (it < plan.items) fetch();
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (warp == 4) P_TRC(1, mine, 2 * group + u, 0);
                    uint32_t outw[16];
                    const uint32_t wv[4] = {cur[u].x, cur[u].y, cur[u].z, cur[u].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t up4 = wv[j] >> 4;  // the pair of column q: code 2q beside code 2q + 1, by a permute of w and w >> 4
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t bits;  // (128 + code_2q, 128 + code_2q+1) in one LOP3
                            asm("lop3.b32 %0, %1, 0x000F000F, %2, 0xEA;" : "=r"(bits) : "r"(__byte_perm(wv[j], up4, 0x4400 + 0x1111 * q)), "r"(magic));
                            const V2 code = __hsub2(*reinterpret_cast<V2 *>(&bits), offset2);  // exact codes
                            const V2 v = __hfma2(code, s2, b2);                                // q*scale+bias, one rounding
                            outw[4 * j + q] = *reinterpret_cast<const uint32_t *>(&v);
                        }
                    }
                    if (warp == 4) P_TRC(1, mine, 2 * group + u, 1);
                    if (!tc_wait(empty + 8 * s, ph, dead)) goto done;
                    if (warp == 4) P_TRC(1, mine, 2 * group + u, 2);
                    unsigned char *tile = psm + s * P_STAGE + P_A_STAGE + row * 128;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int chunk = half * 4 + j;  // 16-byte chunk (8 elements) along K
                        *reinterpret_cast<uint4 *>(tile + ((chunk ^ (row & 7)) << 4)) = make_uint4(outw[4 * j], outw[4 * j + 1], outw[4 * j + 2], outw[4 * j + 3]);
                    }
                    g_fence_proxy_async();  // generic-proxy stores -> visible to the tensor cores' async proxy (of both SMs)
                    __syncwarp();
                    if (lane == 0) g_mbar_arrive(full + 8 * s);
                    if (warp == 4) P_TRC(1, mine, 2 * group + u, 3);
                    if (++s == P_STAGES) s = 0, ph ^= 1u;
                }
            }
    } else if (warp >= 4 + P_DEQ_WARPS) {
        // ------------------------------------------------ epilogue: TMEM lane = token row of THIS CTA, a warp 32 rows of half of the columns
        const int q = warp & 3, side = (warp - 4 - P_DEQ_WARPS) >> 2;
        unsigned char *stage = psm + P_OUT_OFF + (warp - 4 - P_DEQ_WARPS) * P_OUT_BYTES;
        uint32_t f_ph[P_MT] = {0, 0};
        for (int it = unit; it < plan.items; it += units) {
            const PairItem item = pair_item(plan, it);
            for (int i = 0; i < item.mt; ++i) {
                const bool ok = tc_wait(acc_full + 8 * i, f_ph[i], dead);
                const float bad = tc_verdict(ok, dead);  // of a marked CTA this tile and all that follow are stored as NaN
                f_ph[i] ^= 1u;
                g_tc_fence_after();
                const uint32_t d = tmem_d + (static_cast<uint32_t>(q * 32) << 16) + i * 256;
                const int m0 = (item.m0 + i) * 256 + rank * P_TOK + q * 32;  // this warp's first token
                constexpr int BOXES = GATED ? 1 : 2;                           // of 64 features
#pragma unroll 1
                for (int box = 0; box < BOXES; ++box) {
                    const int col0 = (GATED ? side : side * 2 + box) * 64, n0 = item.n_tile * FEATURES + col0;
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // lane 0's store of the box before has left the staging rows
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 64; c += 16) {
                        uint32_t v[16], u[16];
                        p_tmem_ld16(d + col0 + c, v);
                        if constexpr (GATED) p_tmem_ld16(d + 128 + col0 + c, u);
                        g_tmem_ld_wait();
                        float y[16];
                        if constexpr (GATED) {  // both factors rounded as if they had been stored
                            float gate[16], up[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j) gate[j] = to_f(from_f<T>(__uint_as_float(v[j]) * bad)), up[j] = to_f(from_f<T>(__uint_as_float(u[j])));
                            // silu(gate) * up as swiglu's kernel gives it, to the bit
                            quotient_times<T>(gate, [](float g) { return 1.0f + expf(-g); }, up, y, m0 + lane < M ? K - n0 - c : 0);
                            __syncwarp();
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j) y[j] = __uint_as_float(v[j]) * bad;
                        }
                        uint32_t packed[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) packed[j] = pack2<T>(y[2 * j], y[2 * j + 1]);
#pragma unroll
                        for (int j = 0; j < 2; ++j)
                            *reinterpret_cast<uint4 *>(stage + lane * 128 + (((c >> 3) + j) ^ (lane & 7)) * 16) =
                                make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
                    }
                    if (box == BOXES - 1) {  // all of this accumulator's columns are read
                        g_tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            if (rank == 0) g_mbar_arrive(acc_empty + 8 * i);
                            else p_mbar_arrive_leader(acc_empty + 8 * i);
                        }
                    }
                    if (tma_store) {
                        g_fence_proxy_async();
                        __syncwarp();
                        if (lane == 0 && m0 < M && n0 < K) {  // rows and features past the end are not written
                            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&tmap_out), "r"(n0), "r"(m0),
                                         "r"(g_smem_u32(stage))
                                         : "memory");
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        }
                    } else {  // rows that TMA cannot address: one at a time, lanes along the features
                        __syncwarp();
                        for (int r = 0; r < 32 && m0 + r < M; ++r)
                            for (int f = lane; f < 64 && n0 + f < K; f += 32)
                                out[static_cast<size_t>(m0 + r) * K + n0 + f] = *reinterpret_cast<const T *>(stage + r * 128 + (((f >> 3) ^ (r & 7)) << 4) + (f & 7) * 2);
                        __syncwarp();
                    }
                }
            }
        }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
done:  // also from a role whose wait gave up
    g_tc_fence_before();
    __syncthreads();
    if (warp == 2) tc_settle(dead);
    p_cluster_sync();  // neither CTA frees tensor memory (or exits) while the other may still depend on it
    if (warp == 2) {
        g_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "n"(P_TMEM_COLS) : "memory");
    }
#if TL_TRACE
    if (blockIdx.x == 0 && g_trace_buf != nullptr) {  // tag = 20000 + role * 1000 + block * 4 + k (as w4a16_gemm.cu)
        for (int e = threadIdx.x; e < 2 * 40 * 4; e += P_THREADS) {
            const int role = e / 160, rest = e - role * 160;
            if (rest / 4 < num_kb && (role == 1 || (rest & 3) != 3)) {
                const unsigned at = atomicAdd(g_trace_n, 1u);
                if (at < g_trace_cap) g_trace_buf[2 * at] = 20000 + role * 1000 + rest, g_trace_buf[2 * at + 1] = trc[role][rest / 4][rest & 3];
            }
        }
    }
#endif
}

#if TL_TRACE
void trace_bind_gemm2(unsigned long long *buf, unsigned int *n, unsigned int cap) { trace_bind(buf, n, cap); }
#endif

// ---------------------------------------------------------------- host side --
// Mode: 0 = never, 1 = where they take less time (default), 2 = every M > 256 (tests, A/B runs).  TL_GEMM2 sets
// the initial value, tl_set_gemm_pairs() changes it.
static int pairs_default() {
    const char *e = getenv("TL_GEMM2");
    return e == nullptr ? 1 : atoi(e);
}
static int g_pairs_mode = pairs_default();
void set_gemm_pairs(int mode) { g_pairs_mode = mode; }

static PairPlan pair_plan(int M, int K, int features, int units) {
    PairPlan p;
    p.n_tiles = ceil_div(K, features), p.m_tiles = ceil_div(M, 256);
    const int tiles = p.n_tiles * ceil_div(p.m_tiles, P_MT), left = tiles % units;
    p.full = left * P_MT <= units ? tiles - left : tiles;
    p.items = p.full + (tiles - p.full) * P_MT;
    return p;
}

// The pairs where their rounds of tiles cost less than the one-CTA kernel's waves, in that kernel's unit (w4a16_gemm.cu).  A round of whole tiles is 1100 a
// block, of single ones 700; of reductions above 4096 a whole round takes 1500 (0.69 us a block of 9728, 0.73 of 12288), above 16384 a single one
// 1100 (0.52 us).  Measured over 260 sizes (13 matrices, 260 to 8192 rows) the choice is 0.3 % from the better one in the mean and 7 % at most; us, one-CTA kernel /
// pairs: 2560 -> 9728 300 rows 39 / 31, 2048 103 / 75, 4096 208 / 135; 9728 -> 2560 700 rows 66 / 68, 3000 167 / 105, 4096 181 / 186, 6144 296 / 215;
// 18944 -> 3584 800 rows 142 / 151, 2048 340 / 195, 4096 537 / 397.
bool w4a16_gemm2_supported(int M, int N, int K, int dtype) {
    if (g_pairs_mode <= 0 || !(dtype == TL_BF16 || dtype == TL_F16) || M <= 256 || K <= 0 || N % 128 != 0) return false;
    if (g_pairs_mode >= 2) return true;
    const int units = sm_count() / 2;
    const PairPlan p = pair_plan(M, K, 2 * P_ROWS, units);
    const long long whole = ceil_div(p.full, units), single = ceil_div(p.items - p.full, units);
    return whole * (N > 4096 ? 1500 : 1100) + single * (N > 16384 ? 1100 : 700) < w4a16_gemm_cost(M, N, K);
}

template <typename T>
static int pair_map(CUtensorMap *map, const void *p, uint64_t cols, uint64_t rows, uint32_t box_rows) {
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (encode == nullptr) return fail(TL_ECUDA, "quantized_matmul: cuTensorMapEncodeTiled is unavailable");
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2};
    const cuuint32_t box[2] = {P_KB, box_rows}, estr[2] = {1, 1};
    const CUtensorMapDataType dt = std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUresult r = encode(map, dt, 2, const_cast<void *>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TL_OK : fail(TL_ECUDA, "quantized_matmul: cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
}

template <typename T, bool GATED>
static int gemm2_t(const PairWeights<T> &w0, const PairWeights<T> &w1, const void *a, void *out, int M, int N, int K, cudaStream_t st) {
    if (!aligned16(a) || !aligned16(w0.b) || !aligned16(w1.b)) return fail(TL_EINVAL, "quantized_matmul: a and b must be 16-byte aligned");
    const int tma_store = K % 8 == 0 && aligned16(out) ? 1 : 0;
    CUtensorMap map_a, map_out;
    if (int e = pair_map<T>(&map_a, a, N, M, P_TOK)) return e;
    if (!tma_store) map_out = map_a;  // not used
    else if (int e = pair_map<T>(&map_out, out, K, M, 32)) return e;
    static PerDevice configured;
    int device = 0;
    cudaGetDevice(&device);
    if (!configured(device, [] { return cudaFuncSetAttribute(w4a16_gemm2_kernel<T, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM) == cudaSuccess; })) {
        cudaGetLastError();
        return fail(TL_ECUDA, "quantized_matmul: cannot raise shared memory limit");
    }
    const int units = sm_count() / 2;
    const PairPlan plan = pair_plan(M, K, GATED ? P_ROWS : 2 * P_ROWS, units);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * (plan.items < units ? plan.items : units));
    cfg.blockDim = dim3(P_THREADS);
    cfg.dynamicSmemBytes = P_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, w4a16_gemm2_kernel<T, GATED>, map_a, map_out, w0, w1, static_cast<T *>(out), M, N, K, tma_store, plan);
    if (e != cudaSuccess) return fail(TL_ECUDA, "w4a16_gemm2: launch failed: %s", cudaGetErrorString(e));
    TL_LAUNCH_CHECK("w4a16_gemm2");
    return TL_OK;
}

template <typename T>
static PairWeights<T> pair_weights(const void *scales, const void *biases, const void *b) {
    return {static_cast<const T *>(scales), static_cast<const T *>(biases), static_cast<const uint32_t *>(b)};
}

int launch_w4a16_gemm2(const void *scales, const void *biases, const void *a, const void *b, void *out, int M, int N, int K, int dtype,
                       cudaStream_t st) {
    if (M == 0 || K == 0) return TL_OK;
    if (dtype == TL_BF16) {
        const auto w = pair_weights<__nv_bfloat16>(scales, biases, b);
        return gemm2_t<__nv_bfloat16, false>(w, w, a, out, M, N, K, st);
    }
    if (dtype == TL_F16) {
        const auto w = pair_weights<__half>(scales, biases, b);
        return gemm2_t<__half, false>(w, w, a, out, M, N, K, st);
    }
    return fail(TL_EDTYPE, "quantized_matmul: scales must be float16 or bfloat16");
}

// No comparison here: one launch of pairs took less time than two products and their activation at all of 210 sizes (129 to 4096 rows, 7 matrices, both types);
// the least, fp16 of 129 rows of 2560 -> 9728 51 -> 48 us and bf16 of 2048 rows of 9728 -> 2560 192 -> 173, the most, 129 rows of 3072 -> 1024 48 -> 26.
bool launch_w4a16_gemm2_gated(const tl_packed_matrix &gate, const tl_packed_matrix &up, const void *a, void *out, int M, int N, int K, int dtype, cudaStream_t st, int *rc) {
    if (g_pairs_mode <= 0 || M <= 128 || !(dtype == TL_BF16 || dtype == TL_F16) || N % 128 != 0) return false;
    if (dtype == TL_BF16)
        *rc = gemm2_t<__nv_bfloat16, true>(pair_weights<__nv_bfloat16>(gate.scales, gate.biases, gate.weight), pair_weights<__nv_bfloat16>(up.scales, up.biases, up.weight), a, out, M, N,
                                           K, st);
    else
        *rc = gemm2_t<__half, true>(pair_weights<__half>(gate.scales, gate.biases, gate.weight), pair_weights<__half>(up.scales, up.biases, up.weight), a, out, M, N, K, st);
    return true;
}

long long gemm2_gave_up() { return read_gave_up(); }

}  // namespace tl
