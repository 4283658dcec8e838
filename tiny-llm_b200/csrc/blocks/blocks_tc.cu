// Tensor maps for the TMA-fed kernels.  Encoded anew for every launch (0.05 us each): operands move from call to call.
#include "blocks_tc.cuh"

namespace tlb {

static int tc_encode(CUtensorMap *map, const void *ptr, uint32_t rank, const cuuint64_t *dims, const cuuint64_t *strides, const cuuint32_t *box) {
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    if (!encode) return tl::fail(TL_ECUDA, "cuTensorMapEncodeTiled is unavailable");
    const cuuint32_t step[3] = {1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(ptr), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TL_OK : tl::fail(TL_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
}

int tc_map_2d(CUtensorMap *map, const void *ptr, uint64_t cols, uint64_t rows, uint64_t stride, uint32_t box_rows) {
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {stride * 2};
    const cuuint32_t box[2] = {64, box_rows};
    return tc_encode(map, ptr, 2, dims, strides, box);
}

int tc_map_3d(CUtensorMap *map, const void *ptr, uint64_t cols, uint64_t heads, uint64_t rows, uint64_t head, uint64_t row, uint32_t box_heads, uint32_t box_rows) {
    const cuuint64_t dims[3] = {cols, heads, rows}, strides[2] = {head * 2, row * 2};
    const cuuint32_t box[3] = {64, box_heads, box_rows};
    return tc_encode(map, ptr, 3, dims, strides, box);
}

}  // namespace tlb
