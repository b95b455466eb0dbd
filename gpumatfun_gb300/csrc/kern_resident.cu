// Entry points whose Lanczos phase keeps the problem on chip
// (fab_resident.cuh): the Lanczos group and the fused solve, both precisions.
// One block of up to 640 threads per SM: the phases have up to 96 registers
// (they take 80 to 96, without spills).
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
