// jv_dif_f64.cu -- double-precision c2c instances of the in-place mixed-radix
// kernel (jv_dif.cuh).
#include "jv_dif.cuh"

namespace jv {
JV_DIF_INSTANCE(double, DIF_C2C, false)
JV_DIF_INSTANCE(double, DIF_C2C, true)
}  // namespace jv
