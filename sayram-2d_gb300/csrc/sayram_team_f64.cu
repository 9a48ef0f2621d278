// sayram_team_f64.cu -- k_team for one precision mode (see sayram_team.cuh).
#include "sayram_team.cuh"

namespace sg {

cudaError_t team_launch_f64(const TeamLaunch& l, const Common& cm, const Geo& geo, const Fields& fl,
                           const Coef<double>& co, const Kry<double>& kr, const TeamArgs& ta) {
  return l.chip ? team_launch<double, double, F64A, 2>(l, cm, geo, fl, co, co, kr, ta)
                : team_launch<double, double, F64A, 0>(l, cm, geo, fl, co, co, kr, ta);
}
size_t team_smem_limit_f64(bool chip) {
  return chip ? team_limit<double, double, F64A, 2>() : team_limit<double, double, F64A, 0>();
}

}  // namespace sg
