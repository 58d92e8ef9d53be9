// FP64 instantiation of the step kernels (built with -fmad=false so that
// every product and sum is rounded as in the serial reference).
#define GF_FP64_UNIT
#include "gf_kernels_impl.cuh"

template struct GfKernels<double>;
