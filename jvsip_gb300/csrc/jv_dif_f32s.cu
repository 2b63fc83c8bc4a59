// jv_dif_f32s.cu -- single-precision split complex instances of the in-place mixed-radix kernel (jv_dif.cuh).
#include "jv_dif.cuh"

namespace jv {
JV_DIF_INSTANCE(float, DIF_SPLIT, false)
JV_DIF_INSTANCE(float, DIF_SPLIT, true)
}  // namespace jv
