// Kernels of the run-time selected schemes with the FIRST_ORDER stencil.
#include "ext_kernels.cuh"

template struct alp::ExtKernels<alp::ST_FIRST_ORDER>;
