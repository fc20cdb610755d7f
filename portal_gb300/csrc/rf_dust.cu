// The single-model radiation-field kernel: with dust, groups of 1 to 5 lines
// (compiled apart so that the instantiations build in parallel).
#include "rf_kernel.cuh"

#ifndef RF_FLAT
#define RF_FLAT false
#endif

namespace portal {
template <>
const void *rf_kernel_dust<RF_FLAT>(int nlg, int slots) {
    switch (nlg) {
    case 1: return slots == 1   ? (const void *)k_radiation_field<1, true, false, 1, true, RF_FLAT>
                   : slots == 2 ? (const void *)k_radiation_field<1, true, false, 2, true, RF_FLAT>
                                : (const void *)k_radiation_field<1, true, false, 0, true, RF_FLAT>;
    case 2: return slots == 1   ? (const void *)k_radiation_field<2, true, false, 1, true, RF_FLAT>
                   : slots == 2 ? (const void *)k_radiation_field<2, true, false, 2, true, RF_FLAT>
                                : (const void *)k_radiation_field<2, true, false, 0, true, RF_FLAT>;
    case 3: return slots == 1   ? (const void *)k_radiation_field<3, true, false, 1, true, RF_FLAT>
                   : slots == 2 ? (const void *)k_radiation_field<3, true, false, 2, true, RF_FLAT>
                                : (const void *)k_radiation_field<3, true, false, 0, true, RF_FLAT>;
    case 4: return slots == 1   ? (const void *)k_radiation_field<4, true, false, 1, true, RF_FLAT>
                   : slots == 2 ? (const void *)k_radiation_field<4, true, false, 2, true, RF_FLAT>
                                : (const void *)k_radiation_field<4, true, false, 0, true, RF_FLAT>;
    default: return slots == 1   ? (const void *)k_radiation_field<5, true, false, 1, true, RF_FLAT>
                   : slots == 2 ? (const void *)k_radiation_field<5, true, false, 2, true, RF_FLAT>
                                : (const void *)k_radiation_field<5, true, false, 0, true, RF_FLAT>;
    }
}
}  // namespace portal
