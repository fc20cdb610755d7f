// The batched radiation-field kernel: one slot, any number of slots, dust, the
// split field.
#include "rf_kernel.cuh"

namespace portal {
const void *rf_batch_any(bool dust, bool one_slot, bool split) {
    if (dust) return (const void *)k_radiation_field<0, true, true, 0, true>;
    if (split) return (const void *)k_radiation_field<0, false, true, 0, true>;
    return one_slot ? (const void *)k_radiation_field<0, false, true, 1, false>
                    : (const void *)k_radiation_field<0, false, true, 0, false>;
}
}  // namespace portal
