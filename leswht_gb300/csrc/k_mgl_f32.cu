// Instances of the cluster-resident multigrid cycles (k_mgl.cuh), mixed form.
#include "k_mgl.cuh"

namespace lg {

MglKernel mgl_kernel_mixed(int r) {
    switch (r) {
    case 2: return k_mgl_modes<2, true>;
    case 3: return k_mgl_modes<3, true>;
    case 4: return k_mgl_modes<4, true>;
    case 6: return k_mgl_modes<6, true>;
    case 8: return k_mgl_modes<8, true>;
    case 12: return k_mgl_modes<12, true>;
    default: return k_mgl_modes<16, true>;
    }
}

}  // namespace lg
