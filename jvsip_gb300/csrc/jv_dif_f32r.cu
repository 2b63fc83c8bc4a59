// jv_dif_f32r.cu -- single-precision real rows instances of the in-place mixed-radix kernel (jv_dif.cuh).
#include "jv_dif.cuh"

namespace jv {
JV_DIF_INSTANCE(float, DIF_R2C, false)
JV_DIF_INSTANCE(float, DIF_C2R, false)
}  // namespace jv
