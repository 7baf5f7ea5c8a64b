// Stage kernels of pip_fp64_fast.cu with both extra physics (X = 3).
#define PIP_FLAVOUR fast
#define PIP_RCP 1
#define PIP_FAST 1
#define PIP_STAGE_X 3
#include "pip_step_impl.cuh"
