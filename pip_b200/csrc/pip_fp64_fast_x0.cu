// Stage kernels of pip_fp64_fast.cu without extra physics (X = 0).
#define PIP_FLAVOUR fast
#define PIP_RCP 1
#define PIP_FAST 1
#define PIP_STAGE_X 0
#include "pip_step_impl.cuh"
