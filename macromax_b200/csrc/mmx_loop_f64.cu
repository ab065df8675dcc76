// The chunks in one launch in complex128 (mmx_loop.cu compiles the complex64 ones beside it).
#define MMX_GEN_DOUBLE
#include "mmx_loop.cu"
