// The single-model radiation-field kernel: one slot of 32 channels (and the remainder);
// items of consecutive rays
#define RF_FLAT true
#include "rf_one.cu"
