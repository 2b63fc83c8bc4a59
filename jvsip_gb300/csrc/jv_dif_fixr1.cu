// jv_dif_fixr1.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// R2C rows, half lengths up to 1000.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_r2c_1(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_real<DIF_R2C, __VA_ARGS__>());
    JV_DIF_R2C_1(X)
#undef X
}
}  // namespace jv
