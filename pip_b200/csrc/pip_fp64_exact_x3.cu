// Stage kernels of pip_fp64_exact.cu with both extra physics (X = 3).
#define PIP_FLAVOUR exact
#define PIP_RCP 0
#define PIP_FAST 0
#define PIP_STAGE_X 3
#include "pip_step_impl.cuh"
