// Kernels of the run-time selected schemes with the WENO5Z stencil.
#include "ext_kernels.cuh"

template struct alp::ExtKernels<alp::ST_WENO5Z>;
