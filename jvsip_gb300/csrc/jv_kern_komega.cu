// jv_kern_komega.cu -- the k-omega pipeline's instances of the shared-memory
// kernel (single precision): R2C rows whose first pass tapers the real pairs
// it loads (and writes them back), and c2c columns whose last pass stores the
// power and accumulates it into the gram.  The in-place mixed-radix kernel's
// instances go first (a column-major spectrum), then the register-resident
// kernel's.  4096 sensors x 4096 samples: 102 us (159 with both launches on the
// register-resident kernel, whose R2C stores its spectrum one 8-byte element
// per 32 KB column); 2500 x 3000: 57 us (137 on the shared-memory kernel).
#include "jv_launch.cuh"

namespace jv {
// Few sensors: the register-resident kernel's R2C rows first, at lengths where a
// tile's chain there is the shorter one (us, that and the in-place kernel: 2 x 4096
// 6.1 and 9.9, 8 x 256 4.9 and 6.5, 32 x 2048 8.2 and 9.7, 4 x 512 5.0 and 5.2; the
// other way 48 x 2048 9.1 and 7.9, 16 x 512 7.1 and 5.9, 8 x 1536 7.9 and 6.4).
static bool few_sensors(const Job &j) {
    return (j.nvec <= 40 && (j.N == 128 || j.N >= 1000)) || (j.nvec <= 4 && (j.N == 256 || j.N == 512));
}
bool launch_komega_r2c_f32(const Job &j, cudaStream_t s) {
    if (j.kind != K_R2C || !j.taper_n || !j.taper_t) {
        set_error(E_ARG, "tapered R2C without tapers");
        return false;
    }
    const int e0 = jvsip_gpu_last_error();
    if (few_sensors(j) && launch_fast_komega_r2c_f32(j, s)) return true;
    if (jvsip_gpu_last_error() != e0) return false;
    if (launch_dif_komega_r2c_f32(j, s)) return true;
    if (jvsip_gpu_last_error() != e0) return false;
    if (launch_fast_komega_r2c_f32(j, s)) return true;
    if (jvsip_gpu_last_error() != e0) return false;
    return launch_smem_t<float, KX_R2C_TAPER>(j, s);
}
bool launch_komega_power_f32(const Job &j, cudaStream_t s) {
    if (j.kind != K_C2C || !j.gram) {
        set_error(E_ARG, "power columns without a gram");
        return false;
    }
    const int e0 = jvsip_gpu_last_error();
    if (launch_dif_komega_power_f32(j, s)) return true;
    if (jvsip_gpu_last_error() != e0) return false;
    if (launch_fast_komega_power_f32(j, s)) return true;
    if (jvsip_gpu_last_error() != e0) return false;
    return launch_smem_t<float, KX_C2C_POWER>(j, s);
}
}  // namespace jv
