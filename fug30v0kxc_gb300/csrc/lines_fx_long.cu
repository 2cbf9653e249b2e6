// lines_fx_long.cu -- the FP64 line kernels for more than 512 points: those of lines_fx.cu
// without the halvings that the bound on their values does not need, and with the others
// rounded without a bias (fx.cuh), which shorter lines need not pay for.
#define FX_LONG 1
#include "lines_fx.cu"
