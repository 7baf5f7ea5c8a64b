// FP64 kernels with FMA contraction for contexts with implicit conduction (2D, no
// resistivity): the reciprocal forms of pip_physics.cuh instead of pip_fp64_forms.cuh.
//
// BiCGstab runs to a relative residual (1e-10) and its path depends on every rounding: with
// the forms of pip_fp64_forms.cuh, whose fluxes agree to 1e-15, the solves of a 2048x1024
// shear layer stop after other iteration counts, the temperatures differ by 1e-10, and the
// HLLD states' jumps carry single cells of the field to 6e-8 within ten steps.  These
// kernels keep the trajectories of conduction runs bit for bit; the stages are a quarter of
// such a step (about 1 of 3.9 ms), so the faster forms would give it 6 %.
#define PIP_FLAVOUR heat
#define PIP_RCP 1
#define PIP_FAST 0
#define PIP_HEAT_ONLY 1
#define PIP_LAUNCHERS launchers_heat
#include "pip_step_impl.cuh"
