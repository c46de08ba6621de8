// pass-1 register-FFT kernels for transform length 324
#define NSIZE 324
#include "pass1_fast.inc"
