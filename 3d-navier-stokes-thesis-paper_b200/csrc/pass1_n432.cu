// pass-1 register-FFT kernels for transform length 432
#define NSIZE 432
#include "pass1_fast.inc"
