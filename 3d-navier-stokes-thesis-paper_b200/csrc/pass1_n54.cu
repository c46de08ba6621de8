// pass-1 register-FFT kernels for transform length 54
#define NSIZE 54
#include "pass1_fast.inc"
