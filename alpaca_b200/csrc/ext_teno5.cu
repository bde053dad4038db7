// Kernels of the run-time selected schemes with the TENO5 stencil.
#include "ext_kernels.cuh"

template struct alp::ExtKernels<alp::ST_TENO5>;
