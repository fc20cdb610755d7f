// The single-model radiation-field kernel with dust, groups of 1 to 5 lines.
#include "rf_kernel.cuh"

namespace portal {
const void *rf_kernel_dust(int nlg) {
    switch (nlg) {
    case 1: return (const void *)k_radiation_field<1, true, false>;
    case 2: return (const void *)k_radiation_field<2, true, false>;
    case 3: return (const void *)k_radiation_field<3, true, false>;
    case 4: return (const void *)k_radiation_field<4, true, false>;
    default: return (const void *)k_radiation_field<5, true, false>;
    }
}
}  // namespace portal
