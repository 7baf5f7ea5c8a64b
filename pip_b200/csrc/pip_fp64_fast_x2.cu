// Stage kernels of pip_fp64_fast.cu with resistivity (X = 2).
#define PIP_FLAVOUR fast
#define PIP_RCP 1
#define PIP_FAST 1
#define PIP_STAGE_X 2
#include "pip_step_impl.cuh"
