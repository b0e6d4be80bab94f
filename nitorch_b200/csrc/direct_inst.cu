// One (storage type, dimension, mode) slice of the direct kernels.  Compiled
// several times by the Makefile with
//   -DPD_STYPE=<float|__nv_bfloat16> -DPD_SNAME=<f32|bf16> -DPD_DIM=<2|3> -DPD_MODE=<0..5>
// and exports  pp_direct_<sname>_d<dim>_m<mode>(order, args, stream).
#include "pp_direct.cuh"

#define PD_CAT2(a, b) a##b
#define PD_CAT(a, b) PD_CAT2(a, b)
#define PD_NAME PD_CAT(PD_CAT(PD_CAT(PD_CAT(PD_CAT(pp_direct_, PD_SNAME), _d), PD_DIM), _m), PD_MODE)

cudaError_t PD_NAME(int ord, const ppk::PPArgs& a, cudaStream_t st) {
  if (ord == 1) return ppk::launch_direct_cb<PD_DIM, 1, PD_STYPE, PD_MODE>(a, st);
  if (ord == 2) return ppk::launch_direct_cb<PD_DIM, 2, PD_STYPE, PD_MODE>(a, st);
#if PD_DIM == 2
  if (ord == 3) return ppk::launch_direct_cb<PD_DIM, 3, PD_STYPE, PD_MODE>(a, st);
#endif
  return cudaErrorInvalidValue;
}
