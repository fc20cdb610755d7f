// The single-model radiation-field kernel: one slot of 32 channels (and the remainder)
// (compiled apart so that the instantiations build in parallel).
#include "rf_kernel.cuh"

#ifndef RF_FLAT
#define RF_FLAT false
#endif

namespace portal {
template <>
const void *rf_kernel_one<RF_FLAT>(int nlg, bool split) {
    switch (nlg) {
    case 1: return split ? (const void *)k_radiation_field<1, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<1, false, false, 1, false, RF_FLAT>;
    case 2: return split ? (const void *)k_radiation_field<2, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<2, false, false, 1, false, RF_FLAT>;
    case 3: return split ? (const void *)k_radiation_field<3, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<3, false, false, 1, false, RF_FLAT>;
    case 4: return split ? (const void *)k_radiation_field<4, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<4, false, false, 1, false, RF_FLAT>;
    case 5: return split ? (const void *)k_radiation_field<5, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<5, false, false, 1, false, RF_FLAT>;
    case 6: return split ? (const void *)k_radiation_field<6, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<6, false, false, 1, false, RF_FLAT>;
    case 7: return split ? (const void *)k_radiation_field<7, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<7, false, false, 1, false, RF_FLAT>;
    case 8: return split ? (const void *)k_radiation_field<8, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<8, false, false, 1, false, RF_FLAT>;
    case 9: return split ? (const void *)k_radiation_field<9, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<9, false, false, 1, false, RF_FLAT>;
    default: return split ? (const void *)k_radiation_field<10, false, false, 1, true, RF_FLAT>
                          : (const void *)k_radiation_field<10, false, false, 1, false, RF_FLAT>;
    }
}
}  // namespace portal
