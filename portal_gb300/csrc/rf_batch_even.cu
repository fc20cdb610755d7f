// The batched radiation-field kernel: no dust, an even number of slots.
#include "rf_kernel.cuh"

namespace portal {
const void *rf_batch_even() { return (const void *)k_radiation_field<0, false, true, 2, false>; }
}  // namespace portal
