// What the tcgen05 kernels of the blocks library share beside tc05.cuh and tc_wait.cuh: tensor maps, descriptors.
#pragma once

#include "../tc_wait.cuh"
#include "blocks_common.cuh"

namespace tlb {

using tl::g_elect_one;
using tl::g_mbar_arrive;
using tl::g_mbar_expect_tx;
using tl::g_mbar_init;
using tl::g_smem_desc_sw128;
using tl::g_smem_u32;
using tl::g_tc_commit;
using tl::g_tc_fence_after;
using tl::g_tc_fence_before;
using tl::g_tc_mma;
using tl::g_tc_mma_ts;
using tl::g_tma_load_2d;

using tl::tc_settle;
using tl::tc_verdict;
using tl::tc_wait;

long long flash_tc_gave_up();  // of the attention kernels

// kind::f16 instruction descriptor: bf16 x bf16 -> f32, 128 rows, n columns; A K-major, B K-major or (b_mn) MN-major.
__host__ __device__ __forceinline__ constexpr uint32_t tc_idesc(int n, bool b_mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | (static_cast<uint32_t>(n >> 3) << 17) | (8u << 24);
}

// 8 consecutive 32-bit columns of the warp's 32 lanes, without the wait.
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}

// A bf16 matrix [rows, cols] with `stride` elements from row to row, in boxes of box_rows x 64 columns (128-byte swizzle).
int tc_map_2d(CUtensorMap *map, const void *ptr, uint64_t cols, uint64_t rows, uint64_t stride, uint32_t box_rows);
// A bf16 tensor [rows, heads, cols] with `head` and `row` elements between heads and rows, in boxes of box_rows x box_heads x 64.
int tc_map_3d(CUtensorMap *map, const void *ptr, uint64_t cols, uint64_t heads, uint64_t rows, uint64_t head, uint64_t row, uint32_t box_heads, uint32_t box_rows);

}  // namespace tlb
