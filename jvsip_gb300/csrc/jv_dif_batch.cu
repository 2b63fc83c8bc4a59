// jv_dif_batch.cu -- the batching form's instances of the in-place mixed-radix
// kernel (jv_dif.cuh).
#include "jv_dif.cuh"

namespace jv {

template <bool COLS>
static bool go(const DifArgs<float> *calls, const DifTile *q, int ntiles, int nthr, size_t smem, cudaStream_t st) {
    static std::atomic<bool> attr{false};  // set once; concurrent first calls both set it
    if (!attr) {
        if (!cuda_ok(cudaFuncSetAttribute(k_dif_batch<COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)(device()->smem_optin - kStaticArgs)),
                     "cudaFuncSetAttribute"))
            return false;
        attr = true;
    }
    k_dif_batch<COLS><<<(unsigned)ntiles, (unsigned)nthr, smem, st>>>(calls, q);
    count_launch();
    return cuda_ok(cudaGetLastError(), "k_dif_batch launch");
}

bool dif_batch_go(bool cols, const DifArgs<float> *calls, const DifTile *q, int ntiles, int nthr, size_t smem,
                  cudaStream_t st) {
    return cols ? go<true>(calls, q, ntiles, nthr, smem, st) : go<false>(calls, q, ntiles, nthr, smem, st);
}

}  // namespace jv
