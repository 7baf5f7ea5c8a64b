// Stage kernels of pip_fp64_fast.cu with set_coefficients at every stage (X = 1).
#define PIP_FLAVOUR fast
#define PIP_RCP 1
#define PIP_FAST 1
#define PIP_STAGE_X 1
#include "pip_step_impl.cuh"
