// FP64 kernels with FMA contraction and the reciprocal forms of pip_physics.cuh instead of
// pip_fp64_forms.cuh, for runs with a result that hangs on every rounding (launchers_of):
//
// * Implicit conduction (2D, no resistivity).  BiCGstab stops by a residual (1e-10): with the
//   other forms, whose fluxes agree to 1e-15, the solves of a 2048x1024 shear layer stop after
//   other iteration counts, the temperatures differ by 1e-10, and the HLLD states' jumps carry
//   single cells to 6e-8 within ten steps.
// * The parameter blocks that the adjoint takes.  A gradient follows the branch that minmod and
//   the solvers take at every face, and where their operands differ by rounding only the
//   trajectory's last bits choose it: with the other forms (states equal to 2e-15) the gradient
//   moved in every shock tube (1 % of its norm, in the feet of the waves), beside open ends and
//   walls (1e-4), and in 18 of 120 runs from a uniform start (single entries by 8e-3).  The
//   adjoint's forward is pip_run bit for bit, so pip_run takes these forms for such blocks too:
//   1D 1024 cells 11.2 us a step (8.0 with the other forms, 26.1 before the small tiles).
#define PIP_FLAVOUR rcp
#define PIP_RCP 1
#define PIP_FAST 0
#define PIP_RCP_ONLY 1
#define PIP_LAUNCHERS launchers_rcp
#include "pip_step_impl.cuh"
