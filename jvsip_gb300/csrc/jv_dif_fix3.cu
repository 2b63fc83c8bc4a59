// jv_dif_fix3.cu -- compiled-in schedules of the in-place mixed-radix kernel:
// c2c rows beyond 3000 points.
#include "jv_dif_fix.cuh"

namespace jv {
void dif_fix_c2c_3(std::vector<DifFixEntry> &out) {
#define X(...) out.push_back(dif_fix_c2c<__VA_ARGS__>());
    JV_DIF_LENGTHS_3(X)
#undef X
}
}  // namespace jv
