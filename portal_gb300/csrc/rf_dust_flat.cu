// The single-model radiation-field kernel: with dust, groups of 1 to 5 lines;
// items of consecutive rays
#define RF_FLAT true
#include "rf_dust.cu"
