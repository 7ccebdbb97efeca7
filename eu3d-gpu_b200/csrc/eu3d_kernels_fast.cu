// Fast-arithmetic kernels: FMA contraction, the division-light flux
// reconstruction and the fast FP64 forms of the rates (one exponential per
// species' Gibbs energy and per rate constant). The state recovery keeps the
// reference's operand order: a uniform gas's pressure noise then follows the
// reference's, and a near-zero velocity that feels it stays within the 1e-9 of
// its plane over 100 steps (the mixture-polynomial recovery: 1.3e-9).
#define EU_EXACT_THERMO 1
#define EU_EXACT_FLUX 0
#define EU3D_NS fast
#include "eu3d_kernels_impl.cuh"
