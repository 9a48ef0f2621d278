// sayram_team_mixed.cu -- k_team for one precision mode (see sayram_team.cuh).
#include "sayram_team.cuh"

namespace sg {

cudaError_t team_launch_mixed(const TeamLaunch& l, const Common& cm, const Geo& geo, const Fields& fl,
                           const Coef<float>& co, const Kry<float>& kr, const TeamArgs& ta) {
  return l.chip ? team_launch<float, float, F64A, 4>(l, cm, geo, fl, co, co, kr, ta)
                : team_launch<float, float, F64A, 0>(l, cm, geo, fl, co, co, kr, ta);
}
size_t team_smem_limit_mixed(bool chip) {
  return chip ? team_limit<float, float, F64A, 4>() : team_limit<float, float, F64A, 0>();
}

}  // namespace sg
