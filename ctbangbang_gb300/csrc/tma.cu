// tma.cu -- host side of tma.cuh.
#include "tma.cuh"

namespace ctbb {

int tensor_map_f32(CUtensorMap *map, const float *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
                   const cuuint32_t *box)
{
    using EncodeTiled = decltype(&cuTensorMapEncodeTiled);
    static EncodeTiled encode = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<EncodeTiled>(f);
    }();
    if (!encode) {
        set_error("cuTensorMapEncodeTiled not available");
        return CTBB_ERR_CUDA;
    }
    const cuuint32_t step[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<float *>(base), dims,
                              strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
        return CTBB_ERR_CUDA;
    }
    return CTBB_OK;
}

int CopyError::ensure()
{
    if (word) return CTBB_OK;
    void *v = nullptr;
    const cudaError_t e = cudaHostAlloc(&v, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("no pinned memory for the kernels' error word: %s", cudaGetErrorString(e));
        return CTBB_ERR_ALLOC;
    }
    word = static_cast<int *>(v);
    *word = 0;
    return CTBB_OK;
}

void CopyError::release()
{
    if (word) cudaFreeHost(word);
    word = nullptr;
}

}  // namespace ctbb
