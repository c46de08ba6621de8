// pass-1 register-FFT kernels for transform length 36
#define NSIZE 36
#include "pass1_fast.inc"
