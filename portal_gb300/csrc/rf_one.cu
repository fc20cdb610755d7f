// The single-model radiation-field kernel: one slot of 32 channels (and the remainder)
// (compiled apart so that the instantiations build in parallel).
#include "rf_kernel.cuh"

namespace portal {
const void *rf_kernel_one(int nlg, bool split) {
    switch (nlg) {
    case 1: return split ? (const void *)k_radiation_field<1, false, false, 1, true>
                          : (const void *)k_radiation_field<1, false, false, 1, false>;
    case 2: return split ? (const void *)k_radiation_field<2, false, false, 1, true>
                          : (const void *)k_radiation_field<2, false, false, 1, false>;
    case 3: return split ? (const void *)k_radiation_field<3, false, false, 1, true>
                          : (const void *)k_radiation_field<3, false, false, 1, false>;
    case 4: return split ? (const void *)k_radiation_field<4, false, false, 1, true>
                          : (const void *)k_radiation_field<4, false, false, 1, false>;
    case 5: return split ? (const void *)k_radiation_field<5, false, false, 1, true>
                          : (const void *)k_radiation_field<5, false, false, 1, false>;
    case 6: return split ? (const void *)k_radiation_field<6, false, false, 1, true>
                          : (const void *)k_radiation_field<6, false, false, 1, false>;
    case 7: return split ? (const void *)k_radiation_field<7, false, false, 1, true>
                          : (const void *)k_radiation_field<7, false, false, 1, false>;
    case 8: return split ? (const void *)k_radiation_field<8, false, false, 1, true>
                          : (const void *)k_radiation_field<8, false, false, 1, false>;
    case 9: return split ? (const void *)k_radiation_field<9, false, false, 1, true>
                          : (const void *)k_radiation_field<9, false, false, 1, false>;
    default: return split ? (const void *)k_radiation_field<10, false, false, 1, true>
                          : (const void *)k_radiation_field<10, false, false, 1, false>;
    }
}
}  // namespace portal
