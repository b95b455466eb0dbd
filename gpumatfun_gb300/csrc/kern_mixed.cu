// Mixed-precision instantiations of the engine's phase-group kernels.
#include "fab_kernel.cuh"

namespace gm {
template <class Pol, int R>
static void* group_ptr(int group) {
  switch (group) {
    case 0: return (void*)fab_kernel<Pol, R, KG_LANCZOS>;
    case 1: return (void*)k_solve<Pol, R>;
    case 2: return (void*)fab_kernel<Pol, R, KG_APPLY>;
    case 3: return (void*)fab_kernel<Pol, R, KG_DEFLATE>;
    case 4: return (void*)fab_kernel<Pol, R, KG_LANCZOS | PH_MPK>;
    case 5: return (void*)fab_kernel<Pol, R, KG_LANCZOS | PH_REORTH>;
    case 8: return (void*)k_lift<Pol, R>;
  }
  return nullptr;
}
void* kernel_mixed(int R, int group) {
  if (R == 1) return group_ptr<PolMixed, 1>(group);
  if (R == 2) return group_ptr<PolMixed, 2>(group);
  if (R == 4) return group_ptr<PolMixed, 4>(group);
  return nullptr;
}
}  // namespace gm
