// jv_dif_komega.cu -- the k-omega pipeline's instances of the in-place
// mixed-radix kernel (jv_dif.cuh).
#include "jv_dif.cuh"

namespace jv {
bool dif_komega_go(int kind, const DifArgs<float> &a, int nthr, size_t smem, cudaStream_t st) {
    if (kind == DIF_R2CT) return dif_launch<float, DIF_R2CT, false>(a, nthr, smem, st);
    return dif_launch<float, DIF_POWER, false>(a, nthr, smem, st);
}
}  // namespace jv
