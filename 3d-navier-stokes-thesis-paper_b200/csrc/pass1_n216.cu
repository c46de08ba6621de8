// pass-1 register-FFT kernels for transform length 216
#define NSIZE 216
#include "pass1_fast.inc"
