// Instantiation of the generic functor stage for AUSM+ (FP64; this
// translation unit is compiled with -fmad=false).
#include "fv_schemes.cuh"

namespace dn {

cudaError_t launch_ausm_functor_stage(const dn_stage_launch* L, const WallBC& wall)
{
  SchemeFlux<AusmPlusScheme> op{AusmPlusScheme{}, wall};
  return launch_functor_stage(L, op);
}

} // namespace dn
