// The single-model radiation-field kernel: any number of slots, with or without the split field;
// items of consecutive rays
#define RF_FLAT true
#include "rf_any.cu"
