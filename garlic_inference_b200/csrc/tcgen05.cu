// Tensor maps for the kernels that include tcgen05.cuh.
#include "tcgen05.cuh"

typedef CUresult (*t5_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static t5_encode_fn t5_find_encoder() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
        return (t5_encode_fn)p;
    return nullptr;
}

int t5_make_map(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, const void* base, long long rows, long long cols, long long stride,
                int box_rows, int box_cols, CUtensorMapSwizzle swizzle, const char* who, int planes) {
    static const t5_encode_fn enc = t5_find_encoder();
    GI_REQUIRE(enc != nullptr, "%s: the driver does not offer cuTensorMapEncodeTiled", who);
    GI_REQUIRE((uintptr_t)base % 16 == 0 && stride % 16 == 0 && box_cols * elem_bytes % 16 == 0, "%s: rows that do not start on 16 bytes", who);
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)stride, (cuuint64_t)(stride * rows)};
    const cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, (cuuint32_t)planes};
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult r = enc(map, type, planes ? 3 : 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    GI_REQUIRE(r == CUDA_SUCCESS, "%s: cuTensorMapEncodeTiled failed with code %d", who, (int)r);
    return 0;
}
