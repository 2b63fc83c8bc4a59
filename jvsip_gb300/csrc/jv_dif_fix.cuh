// jv_dif_fix.cuh -- launchers of the in-place mixed-radix kernel with schedules
// known at compile time (jv_dif_table.h); included by the translation units
// that instantiate a part of the table each.
#pragma once

#include "jv_dif.cuh"
#include "jv_dif_table.h"

namespace jv {

template <class F, int KIND, bool COLS, int NT>
static bool dif_fix_go(const DifArgs<float> &a, size_t smem, cudaStream_t st, unsigned groups) {
    constexpr int MB = 1024 / NT;  // 64 registers
    static std::atomic<bool> attr{false};  // set once; concurrent first calls both set it
    if (!attr) {
        if (!cuda_ok(cudaFuncSetAttribute(k_dif_fix<F, float, KIND, COLS, NT, MB>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)device()->smem_optin),
                     "cudaFuncSetAttribute"))
            return false;
        attr = true;
    }
    const long grid = (a.nvec + a.vpb - 1) / a.vpb;
    if (grid > 0x7fffffffL) return false;
    k_dif_fix<F, float, KIND, COLS, NT, MB><<<dim3((unsigned)grid, groups), NT, smem, st>>>(a);
    count_launch();
    return cuda_ok(cudaGetLastError(), "k_dif_fix launch");
}

// Lengths of one part of the table: c2c rows and column tiles ...
template <int N, int P1, int T, int VPB, int VC, int TC, int TV, int TL, int... R> static DifFixEntry dif_fix_c2c() {
    static_assert((R * ...) == N, "radices give the length");
    DifFixEntry e;
    e.N = N;
    e.P1 = P1;
    e.vpb = VPB;
    e.nthr = T;
    e.vcol = VC;
    e.radix = {R...};
    e.rows = dif_fix_go<DifFix<1, P1, R...>, DIF_C2C, false, T>;
    if constexpr (VC > 0) e.cols = dif_fix_go<DifFix<VC, P1, R...>, DIF_C2C, true, TC>;
    if constexpr (TL > 0) e.cols4 = dif_fix_go<DifFix<4, P1, R...>, DIF_C2C, true, TL>;
    return e;
}
// ... tiles of 16 for the steps and passes of long transforms ...
template <int N, int P1, int T, int VPB, int VC, int TC, int TV, int TL, int... R> static DifFixEntry dif_fix_long() {
    DifFixEntry e;
    e.N = N;
    if constexpr (TV > 0) {
        e.step = dif_fix_go<DifFix<16, P1, R...>, DIF_STEP, true, TV>;
        e.vec[0] = dif_fix_go<DifFix<16, P1, R...>, DIF_VEC1, true, TV>;
        e.vec[1] = dif_fix_go<DifFix<16, P1, R...>, DIF_VEC2, true, TV>;
        e.vec[2] = dif_fix_go<DifFix<16, P1, R...>, DIF_VECR, false, TV>;
    }
    return e;
}
// ... the k-omega pipeline's tapered R2C tiles (about 64 KB) and power rows ...
constexpr int dif_taper_rows(int N) { return N <= 512 ? 16 : N <= 1024 ? 8 : 4; }
template <int N, int P1, int T, int VPB, int... R> static DifFixEntry dif_fix_taper() {
    DifFixEntry e;
    e.N = N;
    if constexpr (N <= 4096) {
        constexpr int V = dif_taper_rows(N), W = (V * N / 16 + 31) / 32 * 32, NT = W < 96 ? 96 : W < 512 ? W : 512;
        e.vtaper = V;
        e.taper = dif_fix_go<DifFix<V, P1, R...>, DIF_R2CT, false, NT>;
    }
    return e;
}
template <int N, int P1, int T, int VPB, int VC, int TC, int TV, int TL, int... R> static DifFixEntry dif_fix_power() {
    DifFixEntry e;
    e.N = N;
    if constexpr (N <= 4096) e.power = dif_fix_go<DifFix<1, P1, R...>, DIF_POWER, false, T>;
    return e;
}
// ... and real rows, and the rows-only lengths.
template <int KIND, int N, int P1, int T, int VPB, int... R> static DifFixEntry dif_fix_real() {
    static_assert((R * ...) == N, "radices give the length");
    DifFixEntry e;
    e.N = N;
    e.P1 = P1;
    e.vpb = VPB;
    e.nthr = T;
    e.radix = {R...};
    e.rows = dif_fix_go<DifFix<1, P1, R...>, KIND, false, T>;
    return e;
}

}  // namespace jv
