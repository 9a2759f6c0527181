// Instances of the cluster-resident multigrid cycles (k_mgl.cuh), FP64 form.
#include "k_mgl.cuh"

namespace lg {

MglKernel mgl_kernel_fp64(int r) {
    switch (r) {
    case 2: return k_mgl_modes<2, false>;
    case 3: return k_mgl_modes<3, false>;
    case 4: return k_mgl_modes<4, false>;
    case 6: return k_mgl_modes<6, false>;
    case 8: return k_mgl_modes<8, false>;
    case 12: return k_mgl_modes<12, false>;
    default: return k_mgl_modes<16, false>;
    }
}

}  // namespace lg
