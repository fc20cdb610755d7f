// The single-model radiation-field kernel without dust, groups of 6 to 10
// lines.
#include "rf_kernel.cuh"

namespace portal {
const void *rf_kernel_wide(int nlg) {
    switch (nlg) {
    case 6: return (const void *)k_radiation_field<6, false, false>;
    case 7: return (const void *)k_radiation_field<7, false, false>;
    case 8: return (const void *)k_radiation_field<8, false, false>;
    case 9: return (const void *)k_radiation_field<9, false, false>;
    default: return (const void *)k_radiation_field<10, false, false>;
    }
}
}  // namespace portal
