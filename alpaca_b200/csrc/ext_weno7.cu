// Kernels of the run-time selected schemes with the WENO7 stencil.
#include "ext_kernels.cuh"

template struct alp::ExtKernels<alp::ST_WENO7>;
