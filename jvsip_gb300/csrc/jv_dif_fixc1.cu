// jv_dif_fixc1.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// C2R rows, half lengths up to 1000.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_c2r_1(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_real<DIF_C2R, __VA_ARGS__>());
    JV_DIF_C2R_1(X)
#undef X
}
}  // namespace jv
