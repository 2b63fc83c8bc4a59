// jv_dif_fixc2.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// C2R rows, longer ones.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_c2r_2(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_real<DIF_C2R, __VA_ARGS__>());
    JV_DIF_C2R_2(X)
#undef X
}
}  // namespace jv
