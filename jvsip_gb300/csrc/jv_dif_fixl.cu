// jv_dif_fixl.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// the steps and passes of long transforms.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_long_1(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_long<__VA_ARGS__>());
    JV_DIF_LENGTHS_1(X)
#undef X
}
}  // namespace jv
