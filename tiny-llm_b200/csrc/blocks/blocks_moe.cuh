// The lists of (token, choice) pairs grouped by expert, and the grouped products that read them.
#pragma once

#include <algorithm>

#include "blocks_common.cuh"

namespace tlb {

// The experts' launches follow one another closely: sort, gate|up, down and sum may each become resident while the one before is ending, and wait
// (griddep_wait, in every CTA, before anything of it is read or overwritten).  Only gate|up lets its successor in early, behind its own wait for the sort: a
// down product that says that it follows one (tlb_moe_down_next) reads the lists ahead of its wait and fills its ring with weights on every SM whose gate|up
// CTA is done, and waits for the rows alone.  Any other waits before it reads the lists, which may be the launch before's.  16 tokens, 6 of 64 experts of 1408 x 2048: 189 -> 178 us the call; 2048 tokens 472 -> 469.
template <typename... P, typename... A>
static inline cudaError_t moe_launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A &&...a) {
    return tl::launch_chained(kernel, grid, dim3(threads), smem, st, static_cast<P>(a)...);
}

// Which rows of its operand a tile's rows read: the sorted rows themselves (the second product), the token of the pair, or the pair.
constexpr int kGatherSorted = 0, kGatherToken = 1, kGatherPair = 2;
__device__ __forceinline__ int moe_src_row(int pair, int sorted_row, int top, int gather) {
    if (pair < 0) return -1;
    return gather == kGatherSorted ? sorted_row : gather == kGatherToken ? pair / top : pair;
}

// One int32 block of memory: counters [4] = {32-row tiles in use, rows in use, chunks in use, -}; chunks (expert, first row, rows,
// -), the tensor cores' work list; tile_expert, the expert of every 32-row tile; sorted_pair, the pair of every row or -1.
struct MoeLists {
    int32_t *counters;
    int4 *chunks;
    int32_t *tile_expert, *sorted_pair;
};

// The most rows of a chunk: one tensor-core tile's columns, fewer where no expert can get that many (a token names an expert once).  192: four
// stages of two weight blocks and the rows fit in shared memory (blocks_moe_tc.cu).
static inline int moe_chunk_rows(int tokens) { return std::min(192, (tokens + 15) / 16 * 16); }
// An expert's rows make one chunk, and one more for every moe_chunk_rows of them.
static inline long long moe_max_chunks(int tokens, int top, int experts) {
    const long long pairs = (long long)tokens * top;
    return pairs / moe_chunk_rows(tokens) + std::min<long long>(pairs, experts);
}
static inline MoeLists moe_lists(int32_t *p, int tokens, int top, int experts) {
    MoeLists l;
    l.counters = p;
    l.chunks = reinterpret_cast<int4 *>(p + 4);
    l.tile_expert = p + 4 + 4 * moe_max_chunks(tokens, top, experts);
    l.sorted_pair = l.tile_expert + tlb_moe_max_rows(tokens, top, experts) / 32;
    return l;
}

// One grouped product: w0 (and, gated, w1) [experts, N, K] times rows of x.  inter: activation applied, sorted rows; else pair_out.
struct MoeProduct {
    const void *x, *w0, *w1;
    MoeLists lists;
    int tokens, top, experts, K, N, act, gather;
    float limit, slope;
    void *inter;
    float *pair_out;
    bool second = false;  // the launch before is the first product of these lists, which let this one in only once they were whole
};

bool moe_tc_ok(int dtype, int K, const void *x, const void *w0, const void *w1);
int moe_tc_product(const MoeProduct &p, cudaStream_t st);

}  // namespace tlb
