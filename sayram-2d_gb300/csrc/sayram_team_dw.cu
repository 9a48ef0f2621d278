// sayram_team_dw.cu -- k_team for one precision mode (see sayram_team.cuh).
#include "sayram_team.cuh"

namespace sg {

cudaError_t team_launch_dw(const TeamLaunch& l, const Common& cm, const Geo& geo, const Fields& fl,
                           const Coef<float>& co, const Kry<float>& kr, const TeamArgs& ta) {
  return l.chip ? team_launch<float, float, DWA, 4>(l, cm, geo, fl, co, co, kr, ta)
                : team_launch<float, float, DWA, 0>(l, cm, geo, fl, co, co, kr, ta);
}
size_t team_smem_limit_dw(bool chip) {
  return chip ? team_limit<float, float, DWA, 4>() : team_limit<float, float, DWA, 0>();
}

}  // namespace sg
