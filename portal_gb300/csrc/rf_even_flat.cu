// The single-model radiation-field kernel: an even number of slots;
// items of consecutive rays
#define RF_FLAT true
#include "rf_even.cu"
