// The single-model radiation-field kernel without dust, groups of 1 to 5
// lines (compiled apart from the wider ones so that the instantiations build
// in parallel).
#include "rf_kernel.cuh"

namespace portal {
const void *rf_kernel_narrow(int nlg) {
    switch (nlg) {
    case 1: return (const void *)k_radiation_field<1, false, false>;
    case 2: return (const void *)k_radiation_field<2, false, false>;
    case 3: return (const void *)k_radiation_field<3, false, false>;
    case 4: return (const void *)k_radiation_field<4, false, false>;
    default: return (const void *)k_radiation_field<5, false, false>;
    }
}
}  // namespace portal
