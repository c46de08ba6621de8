// pass-1 register-FFT kernels for transform length 108
#define NSIZE 108
#include "pass1_fast.inc"
