// The passes for axes of any length in complex128 (mmx_gen.cu compiles the complex64 ones beside it).
#define MMX_GEN_DOUBLE
#include "mmx_gen.cu"
