// One (storage type, mode) slice of the brick kernels.  Compiled several
// times by the Makefile with
//   -DPK_STYPE=<float|__nv_bfloat16> -DPK_SNAME=<f32|bf16> -DPK_MODE=<0..5>
// and exports  pp_brick_<sname>_m<mode>(order, args, stream).
#include "pp_brick.cuh"

#define PK_CAT2(a, b) a##b
#define PK_CAT(a, b) PK_CAT2(a, b)
#define PK_NAME PK_CAT(PK_CAT(PK_CAT(pp_brick_, PK_SNAME), _m), PK_MODE)

cudaError_t PK_NAME(int ord, const ppk::PPArgs& a, cudaStream_t st) {
  if (ord == 2) return ppk::launch_brick_cb<2, PK_STYPE, PK_MODE>(a, st);
  if (ord == 3) return ppk::launch_brick_cb<3, PK_STYPE, PK_MODE>(a, st);
  return cudaErrorInvalidValue;
}
