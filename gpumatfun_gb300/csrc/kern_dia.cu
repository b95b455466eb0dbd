// Entry points for matrices whose slices are mostly diagonals (PolFP64Dia and
// its mixed counterparts), at the residency of the ordinary entry points: the
// SpMV phase groups without matrix-powers passes.
#include "fab_kernel.cuh"

namespace gm {
template <class Pol, int R>
static void* dia_ptr(int group) {
  switch (group) {
    case 0: return (void*)fab_kernel<Pol, R, KG_LANCZOS>;
    case 2: return (void*)fab_kernel<Pol, R, KG_APPLY>;
    case 5:
      if constexpr (!Pol::kL2) return (void*)fab_kernel<Pol, R, KG_LANCZOS | PH_REORTH>;
  }
  return nullptr;
}
void* kernel_dia(bool fp64, int R, int group, bool l2) {
  if (!fp64 && l2 && R == 1 && group != 5) return dia_ptr<PolMixedL2Dia, 1>(group);
  if (fp64) return R == 1 ? dia_ptr<PolFP64Dia, 1>(group) : R == 2 ? dia_ptr<PolFP64Dia, 2>(group)
                                                                   : dia_ptr<PolFP64Dia, 4>(group);
  return R == 1 ? dia_ptr<PolMixedDia, 1>(group) : R == 2 ? dia_ptr<PolMixedDia, 2>(group)
                                                          : dia_ptr<PolMixedDia, 4>(group);
}
}  // namespace gm
