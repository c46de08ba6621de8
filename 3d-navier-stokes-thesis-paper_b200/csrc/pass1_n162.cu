// pass-1 register-FFT kernels for transform length 162
#define NSIZE 162
#include "pass1_fast.inc"
