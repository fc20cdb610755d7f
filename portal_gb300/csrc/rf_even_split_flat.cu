// The single-model radiation-field kernel: an even number of slots, with the split field;
// items of consecutive rays
#define RF_FLAT true
#include "rf_even_split.cu"
