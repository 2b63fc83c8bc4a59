// jv_dif_fixp.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// the k-omega pipeline's power rows.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_power_1(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_power<__VA_ARGS__>());
    JV_DIF_LENGTHS_1(X)
    JV_DIF_LENGTHS_2(X)
    JV_DIF_LENGTHS_3(X)
#undef X
}
}  // namespace jv
