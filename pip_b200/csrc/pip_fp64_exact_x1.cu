// Stage kernels of pip_fp64_exact.cu with set_coefficients at every stage (X = 1).
#define PIP_FLAVOUR exact
#define PIP_RCP 0
#define PIP_FAST 0
#define PIP_STAGE_X 1
#include "pip_step_impl.cuh"
