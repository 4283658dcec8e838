// The experts' grouped products on the 5th-generation tensor cores (bf16, fp32 accumulation): tcgen05.mma fed by TMA.
//
// Swapped operands: the M side of a product is the expert's WEIGHTS (128 rows of them, one tensor-memory lane each), the N side
// the tokens that chose it, in a chunk of up to 192 rounded up to 16 - so an expert with 5 tokens pays for 16 columns and one
// with 190 for 192, and the same kernel serves a decoding batch (weights streamed once, bound by HBM) and a prompt portion.
// A tile takes two 128-row blocks of weights over one chunk: the gate rows and the up rows of the same 128 features (their
// product is formed in the epilogue from two accumulators of the same lane), or 256 rows of the other products.  Two blocks per
// chunk because the operands come through L2 at about 64 bytes a cycle and SM: with 192 tokens 57 KB feed 768 cycles of tensor
// work, with one block 41 KB would feed 384.
//
// One persistent CTA per SM takes tiles in order, the feature blocks of a chunk side by side, so an expert's rows are fetched
// from HBM once even when its tokens make several chunks.  16 warps:
//   warp 0      TMA of the weight blocks (boxes 64 x 128 rows, 128-byte swizzle) and the stage's byte count
//   warp 1      tcgen05.mma, one elected lane; chunks of up to 128 tokens alternate between two halves of tensor memory
//   warp 2      second product: TMA of the chunk's consecutive rows of the intermediate (boxes of 16 rows)
//   warps 4-11  epilogue: tensor memory -> activation -> bf16 intermediate, or fp32 rows in pair order
//   warps 12-15 first product: the chunk's rows, gathered through the sorted list by 16-byte cp.async straight into the swizzled
//               layout.  (tile::gather4 TMA, four rows an instruction, fed 512 bytes per ~70 ns and SM: 422 us instead of 230 for
//               gate and up of 2048 tokens.)
// Columns past a chunk's tokens hold zeros or stale rows: columns do not mix, and they are not stored.
//
// Measured (64 experts of 2048 x 1408, 6 choices a token): 2048 tokens gate and up 226 -> 187 us (755 TF/s; 180 with quotients
// 2 ulp off throughout, which gives other bits; the weights alone are 113 us of HBM time),
// down 104 us; 1024 tokens 154 -> 140 and 80 -> 74; 16 tokens 89 and 49 us, 6.5 and 5.9 TB/s of weights.  What that step changed: the epilogue without
// branches, chunks of at most 192 rows (four stages in place of three: 203 us with 256, 208 with 128, where every weight block is
// fetched for fewer columns), tiles dealt largest first (the slowest CTA had worked 380,000 cycles, the fastest 259,000).  Tried
// and taken back: pairs of CTAs sharing a chunk's columns (cta_group::2; 199 and 100 us where this form then took 191 and 103, at 512 tokens 134
// against 129), the next blocks' weights asked into L2 ahead of the copies (235 us with four blocks, 286 with sixteen: more requests
// than HBM takes), a ring of its own for the rows (no faster).
#include "blocks_moe.cuh"
#include "blocks_tc.cuh"

namespace tlb {

constexpr int kTcThreads = 16 * 32;
constexpr int kTcGatherWarps = 4;
constexpr int kTcEpilogueWarps = 8;
constexpr int kTcBlockBytes = 128 * 128;      // 128 weight rows x 64 columns
constexpr int kTcBars = 256;                  // barriers and flags at the end of shared memory
constexpr int kTcMaxStages = 8;

enum { kEpiGated = 0, kEpiAct = 1, kEpiPairs = 2 };

struct MoeTcArgs {
    const bf16 *x;             // the gathered operand, rows K apart
    const int32_t *sorted_pair;
    const int4 *chunks;        // (expert, first row of the sorted list, tokens, -)
    const int32_t *counters;   // [2]: number of chunks
    int epilogue, gather, top;
    int K, k_blocks, n /* weight rows per expert */, m_blocks, act;
    float limit, slope;
    bf16 *inter;
    float *pair_out;
    int stages, stage_bytes;
    int turning;  // 1: tiles of different sizes: dealt forth and back
    int second;   // 1: the launch before this one is the first product of the same lists, which are older than both
};

// A warp's part of a finished tile: 32 weight rows, tokens begin .. end - 1 of the chunk that starts at row0 of the sorted list, eight
// at a time.  Neither the activation (a template argument) nor, as a rule, the division (quotient_times) has a branch, so that the eight chains overlap: with an exact division
// and a switch an element a tile of 192 tokens took 18,000 cycles, in which the tensor cores stand still, as such a tile has all of
// tensor memory.  (The next eight read out of tensor memory ahead: no faster, and registers spilled.)
constexpr int kStorePairs = 8, kStoreAct = 9;  // MODE: these, or the activation of a gated pair
template <int MODE>
__device__ __forceinline__ void epilogue(const MoeTcArgs &a, uint32_t d0, uint32_t d1, int row0, int begin, int end, int f0, int f1, float bad) {
    for (int col = begin; col < end; col += 8) {
        const int here = end - col, row = row0 + col;
        uint32_t u[8], v[8];
        tc_ld8(d0 + col, u);
        tc_ld8(d1 + col, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if constexpr (MODE == kStorePairs) {
            int pair[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) pair[i] = i < here ? a.sorted_pair[row + i] : 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float *o = a.pair_out + (size_t)pair[i] * a.n;
                if (i < here) {
                    if (f0 < a.n) o[f0] = __uint_as_float(u[i]) * bad;
                    if (f1 < a.n) o[f1] = __uint_as_float(v[i]) * bad;
                }
            }
        } else {
            bf16 *o = a.inter + (size_t)row * a.n + f0;
            bf16 x[8];
            float p[8], q[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) p[i] = __uint_as_float(u[i]), q[i] = __uint_as_float(v[i]);
            if constexpr (MODE == kStoreAct) {
                auto act = [&](float z) { return a.act == 2 ? (z > 0.f ? z * z : 0.f) : act_apply(z, a.act); };
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    x[i] = __float2bfloat16_rn(act(p[i]) * bad);
                    if (i < here && f1 < a.n) o[(size_t)i * a.n + 128] = __float2bfloat16_rn(act(q[i]) * bad);
                }
            } else {
                float y[8];
                gated_pairs<bf16, MODE>(p, q, a.limit, a.slope, y, here);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = __float2bfloat16_rn(y[i] * bad);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i, o += a.n)
                if (i < here && f0 < a.n) *o = x[i];
        }
    }
}

__global__ void __launch_bounds__(kTcThreads, 1)
moe_tc_kernel(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_x, const MoeTcArgs a) {
    extern __shared__ __align__(1024) unsigned char moe_tc_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = g_smem_u32(moe_tc_smem);
    const uint32_t bars = base + a.stages * a.stage_bytes;
    const uint32_t full = bars, empty = full + 8 * kTcMaxStages, acc_full = empty + 8 * kTcMaxStages, acc_empty = acc_full + 16;
    volatile int *dead = reinterpret_cast<volatile int *>(moe_tc_smem + a.stages * a.stage_bytes + 16 * kTcMaxStages + 32);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(const_cast<int *>(dead)) + 1;
    const bool gathers = a.gather != kGatherSorted;

    if (warp == 0 && lane == 0) {
        for (int i = 0; i < a.stages; ++i) g_mbar_init(full + 8 * i, gathers ? 1 + kTcGatherWarps : 1), g_mbar_init(empty + 8 * i, 1);
        for (int i = 0; i < 2; ++i) g_mbar_init(acc_full + 8 * i, 1), g_mbar_init(acc_empty + 8 * i, kTcEpilogueWarps);
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w0) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w1) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(g_smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    g_tc_fence_before();
    __syncthreads();
    g_tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (!a.second) {
        tl::griddep_wait();
        tl::griddep_launch();  // the lists are complete: see moe_launch
    }
    const int tiles = a.counters[2] * a.m_blocks;
    const bool gated = a.epilogue == kEpiGated;
    // Tiles come largest first (moe_sort_kernel), dealt forth and back, so that the CTAs' sums differ by little more than the smallest tile.  (Tiles of one
    // size always forth: of 16 tokens, where weights from HBM are all there is, the way back cost 2 %.)
    auto tile_of = [&](int turn) { return turn * (int)gridDim.x + (int)(a.turning & turn ? gridDim.x - 1 - blockIdx.x : blockIdx.x); };

    if (warp == 0) {  // ---- weights
        int s = 0;
        uint32_t ph = 1;
        for (int turn = 0, tile; (tile = tile_of(turn)) < tiles; ++turn) {
            const int4 c = a.chunks[tile / a.m_blocks];
            const int mb = tile % a.m_blocks, cols = (c.z + 15) & ~15;
            const int r0 = c.x * a.n + mb * (gated ? 128 : 256), r1 = gated ? r0 : r0 + 128;
            for (int kb = 0; kb < a.k_blocks; ++kb) {
                if (!tc_wait(empty + 8 * s, ph, dead)) goto out;
                if (g_elect_one()) {
                    const uint32_t at = base + s * a.stage_bytes;
                    g_mbar_expect_tx(full + 8 * s, 2 * kTcBlockBytes + (gathers ? 0 : cols * 128));
                    g_tma_load_2d(at, &map_w0, kb * 64, r0, full + 8 * s);
                    g_tma_load_2d(at + kTcBlockBytes, &map_w1, kb * 64, r1, full + 8 * s);
                }
                __syncwarp();
                if (++s == a.stages) s = 0, ph ^= 1u;
            }
        }
    } else if (warp == 2) {  // ---- consecutive rows of the second operand
        int s = 0;
        uint32_t ph = 1;
        if (a.second) tl::griddep_wait();
        for (int turn = 0, tile; !gathers && (tile = tile_of(turn)) < tiles; ++turn) {
            const int4 c = a.chunks[tile / a.m_blocks];
            for (int kb = 0; kb < a.k_blocks; ++kb) {
                if (!tc_wait(empty + 8 * s, ph, dead)) goto out;
                if (lane * 16 < c.z) g_tma_load_2d(base + s * a.stage_bytes + 2 * kTcBlockBytes + lane * 16 * 128, &map_x, kb * 64, c.y + lane * 16, full + 8 * s);
                __syncwarp();
                if (++s == a.stages) s = 0, ph ^= 1u;
            }
        }
    } else if (warp >= 12) {  // ---- gathered rows: a thread copies piece t % 8 of rows t / 8 + 16 j
        const int t = threadIdx.x - 12 * 32, piece = t & 7, r0 = t >> 3;
        const uint32_t to = 2 * kTcBlockBytes + r0 * 128 + ((piece ^ (r0 & 7)) << 4);
        int s = 0, before = -1;  // the stage whose copies this thread has issued and not yet reported
        uint32_t ph = 1;
        if (a.second) tl::griddep_wait();
        auto report = [&](int stage) {  // landed: visible to the tensor core's proxy, then one arrival per warp
            tl::g_fence_proxy_async();
            __syncwarp();
            if (lane == 0) g_mbar_arrive(full + 8 * stage);
        };
        for (int turn = 0, tile; gathers && (tile = tile_of(turn)) < tiles; ++turn) {
            const int4 c = a.chunks[tile / a.m_blocks];
            const int groups = (c.z + 15) >> 4;
            int src[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) src[j] = r0 + 16 * j < c.z ? moe_src_row(a.sorted_pair[c.y + r0 + 16 * j], 0, a.top, a.gather) : -1;
            for (int kb = 0; kb < a.k_blocks; ++kb) {
                if (!tc_wait(empty + 8 * s, ph, dead)) goto out;
                const uint32_t at = base + s * a.stage_bytes + to;
                const int k = kb * 64 + piece * 8;
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (j < groups) {
                        const bool ok = src[j] >= 0 && k < a.K;
                        const int bytes = ok ? 16 : 0;  // 0: the 16 bytes are zero-filled
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + j * 2048), "l"(a.x + (ok ? (size_t)src[j] * a.K + k : 0)), "r"(bytes) : "memory");
                    }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (before >= 0) {
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                    report(before);
                }
                before = s;
                if (++s == a.stages) s = 0, ph ^= 1u;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (before >= 0) report(before);
    } else if (warp == 1) {  // ---- the products
        int s = 0, buf = 0;
        uint32_t ph = 0, acc_ph[2] = {1, 1};
        for (int turn = 0, tile; (tile = tile_of(turn)) < tiles; ++turn) {
            const int cols = (a.chunks[tile / a.m_blocks].z + 15) & ~15;
            const bool whole = cols > 128;  // both halves of tensor memory
            if (whole) buf = 0;
            const uint32_t d0 = tmem + buf * 256, d1 = d0 + (whole ? 256 : 128), idesc = tc_idesc(cols);
            if (!tc_wait(acc_empty + 8 * buf, acc_ph[buf], dead)) goto out;
            acc_ph[buf] ^= 1u;
            if (whole) {
                if (!tc_wait(acc_empty + 8, acc_ph[1], dead)) goto out;
                acc_ph[1] ^= 1u;
            }
            g_tc_fence_after();
            for (int kb = 0; kb < a.k_blocks; ++kb) {
                if (!tc_wait(full + 8 * s, ph, dead)) goto out;
                g_tc_fence_after();
                if (g_elect_one()) {
                    const uint32_t at = base + s * a.stage_bytes;
                    const uint64_t w0 = g_smem_desc_sw128(at, 0, 1024), w1 = g_smem_desc_sw128(at + kTcBlockBytes, 0, 1024),
                                   x = g_smem_desc_sw128(at + 2 * kTcBlockBytes, 0, 1024);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t accumulate = kb > 0 || k > 0;
                        g_tc_mma(d0, w0 + 2 * k, x + 2 * k, idesc, accumulate);
                        g_tc_mma(d1, w1 + 2 * k, x + 2 * k, idesc, accumulate);
                    }
                    g_tc_commit(empty + 8 * s);
                    if (kb == a.k_blocks - 1) g_tc_commit(acc_full + 8 * buf);
                }
                __syncwarp();
                if (++s == a.stages) s = 0, ph ^= 1u;
            }
            buf = whole ? 0 : buf ^ 1;
        }
    } else if (warp >= 4 && warp < 12) {  // ---- epilogue: lane = weight row, column = token
        const int quarter = warp & 3, half = (warp - 4) >> 2;
        const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
        int buf = 0;
        uint32_t acc_ph[2] = {0, 0};
        for (int turn = 0, tile; (tile = tile_of(turn)) < tiles; ++turn) {
            const int4 c = a.chunks[tile / a.m_blocks];
            const int mb = tile % a.m_blocks, cols = (c.z + 15) & ~15;
            const bool whole = cols > 128;
            if (whole) buf = 0;
            const uint32_t d0 = tmem + lanes + buf * 256, d1 = d0 + (whole ? 256 : 128);
            const int f0 = mb * (gated ? 128 : 256) + quarter * 32 + lane, f1 = f0 + 128;
            const bool ok = tc_wait(acc_full + 8 * buf, acc_ph[buf], dead);
            const float bad = tc_verdict(ok, dead);  // of a marked CTA this tile and all that follow are stored as NaN
            acc_ph[buf] ^= 1u;
            g_tc_fence_after();
            const int begin = half * (cols / 2), end = min(begin + cols / 2, c.z);
            if (gated) {
                if (a.act == 0) epilogue<0>(a, d0, d1, c.y, begin, end, f0, f1, bad);
                else if (a.act == 3) epilogue<3>(a, d0, d1, c.y, begin, end, f0, f1, bad);
                else epilogue<1>(a, d0, d1, c.y, begin, end, f0, f1, bad);
            } else if (a.epilogue == kEpiPairs) {
                epilogue<kStorePairs>(a, d0, d1, c.y, begin, end, f0, f1, bad);
            } else {
                epilogue<kStoreAct>(a, d0, d1, c.y, begin, end, f0, f1, bad);
            }
            g_tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                g_mbar_arrive(acc_empty + 8 * buf);
                if (whole) g_mbar_arrive(acc_empty + 8);
            }
            buf = whole ? 0 : buf ^ 1;
        }
    }
out:  // also from a role whose wait gave up
    asm volatile("cp.async.wait_all;" ::: "memory");
    g_tc_fence_before();
    __syncthreads();
    if (warp == 3) {
        tc_settle(dead);
        g_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

bool moe_tc_ok(int dtype, int K, const void *x, const void *w0, const void *w1) {
    return dtype == TL_BF16 && K % 8 == 0 && tl::aligned16(x) && tl::aligned16(w0) && (!w1 || tl::aligned16(w1));
}

int moe_tc_product(const MoeProduct &p, cudaStream_t st) {
    MoeTcArgs a;
    a.sorted_pair = p.lists.sorted_pair, a.chunks = p.lists.chunks, a.counters = p.lists.counters;
    a.epilogue = p.w1 ? kEpiGated : p.inter ? kEpiAct : kEpiPairs;
    a.x = (const bf16 *)p.x, a.gather = p.gather, a.top = p.top, a.K = p.K, a.n = p.N, a.act = p.act, a.limit = p.limit, a.slope = p.slope;
    a.inter = (bf16 *)p.inter, a.pair_out = p.pair_out;
    CUtensorMap m0, m1, mx;
    if (int e = tc_map_2d(&m0, p.w0, p.K, (uint64_t)p.experts * p.N, p.K, 128)) return e;
    if (int e = tc_map_2d(&m1, p.w1 ? p.w1 : p.w0, p.K, (uint64_t)p.experts * p.N, p.K, 128)) return e;
    if (p.gather != kGatherSorted) mx = m0;  // not read
    else if (int e = tc_map_2d(&mx, p.x, p.K, tlb_moe_max_rows(p.tokens, p.top, p.experts), p.K, 16)) return e;
    a.k_blocks = ceil_div(p.K, 64);
    a.stage_bytes = 2 * kTcBlockBytes + moe_chunk_rows(p.tokens) * 128;
    a.stages = std::min(kTcMaxStages, (227 * 1024 - kTcBars) / a.stage_bytes);
    a.turning = moe_chunk_rows(p.tokens) > 16;
    a.second = p.second;
    a.m_blocks = ceil_div(p.N, a.epilogue == kEpiGated ? 128 : 256);
    // the largest that any call asks for; on every call, because the attribute belongs to the device that is current
    if (cudaFuncSetAttribute(moe_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) {
        cudaGetLastError();
        return tl::fail(TL_ECUDA, "moe_tc: no shared memory");
    }
    const long long most = moe_max_chunks(p.tokens, p.top, p.experts) * a.m_blocks;  // tiles there can be
    moe_launch(moe_tc_kernel, (unsigned)std::min<long long>(sm_count(), most), kTcThreads, a.stages * a.stage_bytes + kTcBars, st, m0, m1, mx, a);
    return TL_OK;
}

// One CTA: count the pairs of every expert, lay the experts' segments out in whole 32-row tiles (the general products read
// those), cut them into chunks for the tensor cores, and scatter the pairs.  A pair's place among its expert's is the value its
// counting atomic returned, kept in a register.  2048 tokens of 6 choices: 25 -> 13 us, 16 tokens: 13 -> 7 us (one thread walked
// the experts before).
constexpr int kSortThreads = 1024, kSortKeep = 16;
__global__ void __launch_bounds__(kSortThreads)
moe_sort_kernel(const int32_t *__restrict__ idx, int pairs, int experts, int most /* rows of a chunk */, MoeLists out) {
    int32_t *sorted_pair = out.sorted_pair, *tile_expert = out.tile_expert;
    extern __shared__ int sm[];
    int *count = sm, *start = sm + experts, *first_chunk = sm + 2 * experts;  // [experts] each
    __shared__ int carry[2], part[2][32];
    __shared__ int size_at[16];  // chunks by their size in groups of 16 rows
    const int sizes = most / 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < experts; e += kSortThreads) count[e] = 0;
    if (threadIdx.x < 2) carry[threadIdx.x] = 0;
    tl::griddep_wait();
    __syncthreads();
    // chunks of an expert's n rows: of equal length, in whole groups of 16 rows
    auto chunk_rows = [&](int n) {
        const int parts = (n + most - 1) / most;
        return ((n + parts - 1) / parts + 15) / 16 * 16;
    };
    auto chunk_count = [&](int n) { return n == 0 ? 0 : (n + chunk_rows(n) - 1) / chunk_rows(n); };
    int expert[kSortKeep], rank[kSortKeep];
#pragma unroll
    for (int i = 0; i < kSortKeep; ++i) {
        const int p = threadIdx.x + i * kSortThreads;
        const int e = p < pairs ? tl::ld_cg(idx + p) : -1;
        expert[i] = e >= 0 && e < experts ? e : -1;
    }
#pragma unroll
    for (int i = 0; i < kSortKeep; ++i) rank[i] = expert[i] >= 0 ? atomicAdd(&count[expert[i]], 1) : 0;
    __syncthreads();  // the kept ones take an expert's first places
    for (int p = threadIdx.x + kSortKeep * kSortThreads; p < pairs; p += kSortThreads) {
        const int e = tl::ld_cg(idx + p);
        if (e >= 0 && e < experts) atomicAdd(&count[e], 1);
    }
    __syncthreads();
    for (int e0 = 0; e0 < experts; e0 += kSortThreads) {  // running sums over the experts: rows (whole tiles) and chunks
        const int e = e0 + threadIdx.x, n = e < experts ? count[e] : 0;
        const int rows = (n + 31) / 32 * 32, cut = chunk_count(n);
        int r = rows, c = cut;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int r1 = __shfl_up_sync(0xffffffffu, r, o), c1 = __shfl_up_sync(0xffffffffu, c, o);
            if (lane >= o) r += r1, c += c1;
        }
        if (lane == 31) part[0][warp] = r, part[1][warp] = c;
        __syncthreads();
        int r_before = carry[0], c_before = carry[1];
        for (int w = 0; w < warp; ++w) r_before += part[0][w], c_before += part[1][w];
        // first_chunk: by expert, or, until the chunks are ordered by size below, the size and the number of the expert's chunks
        if (e < experts) start[e] = r_before + r - rows, first_chunk[e] = sizes == 1 ? c_before + c - cut : n > 0 ? chunk_rows(n) / 16 << 27 | cut : 0;
        __syncthreads();
        if (threadIdx.x == kSortThreads - 1) carry[0] = r_before + r, carry[1] = c_before + c;
        __syncthreads();
    }
    if (threadIdx.x == 0) out.counters[0] = carry[0] / 32, out.counters[1] = carry[0], out.counters[2] = carry[1];
    if (sizes == 1) {
        if (threadIdx.x == 0) size_at[0] = 0;
    } else if (warp < sizes) {  // the largest chunks first (the products' CTAs take tiles in this order), those of one size by expert: a warp a size
        int at = 0;
        for (int e0 = 0; e0 < experts; e0 += 32) {
            // an entry is written by the warp of its size alone; to the others it is of no size before and after
            volatile int *entry = first_chunk + e0 + lane;
            const int has = e0 + lane < experts ? *entry : 0;
            const int cut = has >> 27 == warp + 1 ? has & ((1 << 27) - 1) : 0;
            int c = cut;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int c1 = __shfl_up_sync(0xffffffffu, c, o);
                if (lane >= o) c += c1;
            }
            if (cut) *entry = at + c - cut;
            at += __shfl_sync(0xffffffffu, c, 31);
        }
        if (lane == 0) size_at[warp] = at;
    }
    __syncthreads();
    if (sizes > 1) {
        if (threadIdx.x == 0)
            for (int i = sizes - 1, at = 0; i >= 0; --i) {
                const int n = size_at[i];
                size_at[i] = at, at += n;
            }
        __syncthreads();
    }
    for (int e = warp; e < experts; e += kSortThreads / 32) {
        const int n = count[e], row0 = start[e], cut = chunk_count(n);
        for (int i = lane; i < (n + 31) / 32; i += 32) tile_expert[row0 / 32 + i] = e;
        if (n % 32 && lane >= n % 32) sorted_pair[row0 + n / 32 * 32 + lane] = -1;  // the last tile's rows without a pair
        for (int i = lane; i < cut; i += 32) {
            const int size = chunk_rows(n);
            out.chunks[size_at[size / 16 - 1] + first_chunk[e] + i] = make_int4(e, row0 + i * size, min(size, n - i * size), 0);
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortKeep; ++i)
        if (expert[i] >= 0) sorted_pair[start[expert[i]] + rank[i]] = threadIdx.x + i * kSortThreads;
    if (pairs > kSortKeep * kSortThreads) {  // more pairs than a thread keeps: the rest in a second count, from where the kept ones end
        for (int e = threadIdx.x; e < experts; e += kSortThreads) count[e] = 0;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSortKeep; ++i)
            if (expert[i] >= 0) atomicAdd(&count[expert[i]], 1);
        __syncthreads();
        for (int p = threadIdx.x + kSortKeep * kSortThreads; p < pairs; p += kSortThreads) {
            const int e = tl::ld_cg(idx + p);
            if (e >= 0 && e < experts) sorted_pair[start[e] + atomicAdd(&count[e], 1)] = p;
        }
    }
}

}  // namespace tlb

using namespace tlb;

extern "C" {

long long tlb_moe_max_rows(int tokens, int top, int experts) {
    const long long pairs = (long long)tokens * top, groups = std::min<long long>(pairs, experts);  // at most that many segments carry padding
    return (pairs + groups * 31 + 31) / 32 * 32;
}

long long tlb_moe_lists_ints(int tokens, int top, int experts) {
    return 4 + 4 * moe_max_chunks(tokens, top, experts) + tlb_moe_max_rows(tokens, top, experts) / 32 + tlb_moe_max_rows(tokens, top, experts);
}

int tlb_moe_sort(const int32_t *idx, int tokens, int top, int experts, int32_t *lists, void *stream) {
    if (tokens <= 0) return TL_OK;
    if (!idx || !lists || top <= 0 || experts <= 0 || !tl::aligned16(lists)) return tl::fail(TL_EINVAL, "moe_sort: bad argument");
    const size_t smem = (size_t)3 * experts * sizeof(int);
    if (smem > 48 * 1024) return tl::fail(TL_EINVAL, "moe_sort: %d experts do not fit", experts);
    if (smem > 40 * 1024 && cudaFuncSetAttribute(moe_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024) != cudaSuccess) {
        cudaGetLastError();
        return tl::fail(TL_ECUDA, "moe_sort: no shared memory");
    }
    moe_launch(moe_sort_kernel, 1, kSortThreads, smem, as_stream(stream), idx, tokens * top, experts, moe_chunk_rows(tokens), moe_lists(lists, tokens, top, experts));
    TL_LAUNCH_CHECK("moe_sort");
    return TL_OK;
}

long long tlb_tc_gave_up(void) {
    const long long experts = tl::read_gave_up(), attention = flash_tc_gave_up();
    return experts < 0 || attention < 0 ? -1 : experts + attention;
}

}  // extern "C"
