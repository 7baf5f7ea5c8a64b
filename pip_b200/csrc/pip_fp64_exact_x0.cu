// Stage kernels of pip_fp64_exact.cu without extra physics (X = 0).
#define PIP_FLAVOUR exact
#define PIP_RCP 0
#define PIP_FAST 0
#define PIP_STAGE_X 0
#include "pip_step_impl.cuh"
