// jv_dif_step.cu -- the long transforms' steps on the in-place mixed-radix
// kernel (jv_dif.cuh): column tiles with groups along the grid's y and the
// first step's output twiddle; the passes over a single long vector.
#include "jv_dif.cuh"

namespace jv {
bool dif_step_go(const DifArgs<float> &a, int nthr, size_t smem, cudaStream_t st, unsigned groups) {
    return dif_launch<float, DIF_STEP, true>(a, nthr, smem, st, groups);
}
bool dif_vec_go(int kind, const DifArgs<float> &a, int nthr, size_t smem, cudaStream_t st, unsigned groups) {
    if (kind == DIF_VEC1) return dif_launch<float, DIF_VEC1, true>(a, nthr, smem, st, groups);
    if (kind == DIF_VEC2) return dif_launch<float, DIF_VEC2, true>(a, nthr, smem, st, groups);
    return dif_launch<float, DIF_VECR, false>(a, nthr, smem, st, groups);
}
}  // namespace jv
