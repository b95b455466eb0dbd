// Entry points whose Lanczos phase keeps the problem on chip
// (fab_resident.cuh): the Lanczos group and the fused solve, both precisions.
// One block per SM, so every phase compiles for 128 registers.
#include "fab_kernel.cuh"

namespace gm {
template <class Pol, int R>
static void* resident_ptr(bool fused) {
  return fused ? (void*)fab_kernel<Pol, R, KG_LANCZOS | KG_SOLVE | KG_APPLY | PH_RESIDENT>
               : (void*)fab_kernel<Pol, R, KG_LANCZOS | PH_RESIDENT>;
}
void* kernel_resident(bool fp64, int R, bool fused) {
  if (fp64) return R == 1 ? resident_ptr<PolFP64, 1>(fused) : R == 2 ? resident_ptr<PolFP64, 2>(fused)
                                                                     : resident_ptr<PolFP64, 4>(fused);
  return R == 1 ? resident_ptr<PolMixed, 1>(fused) : R == 2 ? resident_ptr<PolMixed, 2>(fused)
                                                            : resident_ptr<PolMixed, 4>(fused);
}
}  // namespace gm
