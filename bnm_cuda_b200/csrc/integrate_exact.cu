// Reference-order integrators, compiled with -fmad=false (no FMA contraction)
// so their arithmetic is the reference CPU build's: FP64 (default u_real) and
// FP32 in the reference's USE_FLOATS operand types.  These are the parity
// kernels of the oracle-noise mode; see integrate_generic.cuh.
#include "kernels.h"
#define BNM_GENERIC_NS exact
#include "integrate_generic.cuh"

cudaError_t bnm_launch_integrate_exact(const bnm::SimArgs& a, int fp64, int num_sms, cudaStream_t st) {
    using namespace bnm;
    return fp64 ? exact::launch_generic<double>(a, num_sms, st) : exact::launch_generic<float>(a, num_sms, st);
}
