// sayram_team.h -- whole backward-Euler steps of a small batch in one cooperative launch: the
// interface between the host runtime and the kernels in sayram_team.cuh.
#pragma once

#include "sayram_ops.cuh"

namespace sg {

constexpr int kTeamThreads = 512;
constexpr int kTeamParts = 4;  // tiles a block assembles at once, by a quarter of its threads each

// One block's share of one instance: reduction segments [s0, s1), none for a block that only helps
// with the assembly. The nb blocks of an instance (its team) are neighbours in the grid, rank 0 first.
struct TeamShare {
  int inst, rank, nb;
  int s0, s1;
  int ty;  // rows of the assembly tiles of this instance
};

enum { TEAM_ASSEMBLE = 1, TEAM_SOLVE = 2, TEAM_POLISH = 4, TEAM_STEP = 7 };

enum { TEAM_GAVE_UP = 0, TEAM_NEGATIVE = 1, TEAM_NOT_CONVERGED = 2, TEAM_FLAGS = 3 };

struct TeamArgs {
  const TeamShare* share;
  const int* first;    // block k has shares [first[k], first[k + 1]), more than one only of teams of one;
                       // null: share k
  unsigned* bar;       // kTeamBarStride counters per instance: arrivals, departures
  float* tmax;         // per block: max of the right-hand side over its tiles
  volatile int* stat;  // TEAM_* flags in mapped host memory: what the launch's last step ended with
  double tol, inner_tol;
  int max_refine, max_iters;
  int nsteps, phases;
  int polls;           // most polls of one barrier (kTeamPolls; 0: the first barrier gives up)
  int report;          // 1: set the flags of the last step
  int own_cap;         // cells of the largest share, rounded up to whole segments
  int pmax;            // widest row pitch
};
constexpr int kTeamPolls = 1 << 20;  // ~0.7 us each; blocks of a launch run together, milliseconds apart at most
constexpr int kTeamBarStride = 16;  // 64 bytes: one team's counters do not share a line with another's

// Bytes of dynamic shared memory (sayram_team.cuh lays it out). chip: the Krylov vectors of a share
// stay in shared memory; otherwise x, t, v and the shadow residual stay in global memory.
inline size_t team_smem(size_t tsize, bool chip, long long own_cap, long long pmax, size_t tile_bytes) {
  const size_t ext = (size_t)(own_cap + 2 * pmax), halo = (size_t)(2 * pmax);
  // r, p, v, x with both halos, t and r^ / r, the staged 8-byte solution (p, and in FP32 v), the halos of
  // x and in FP64 v
  size_t n = chip ? 4 * ext * tsize + 2 * (size_t)own_cap * tsize
                  : ext * tsize + ext * 8 + (tsize == 4 ? 1 : 2) * halo * tsize;
  if (n < kTeamParts * tile_bytes) n = kTeamParts * tile_bytes;
  return n + (size_t)kPartQ * (own_cap / 128) * 8 + 16;
}

// cells of a share the on-chip form holds the coefficients of in registers
inline long long team_chip_cells(size_t tsize) { return 4LL * kTeamThreads * (tsize == 4 ? 4 : 2); }

struct TeamLaunch {
  int grid;
  size_t smem;
  bool chip;
  cudaStream_t stream;
};
// One launcher per precision mode, each in a translation unit of its own.
cudaError_t team_launch_f64(const TeamLaunch& l, const Common& cm, const Geo& geo, const Fields& fl,
                            const Coef<double>& co, const Kry<double>& kr, const TeamArgs& ta);
cudaError_t team_launch_mixed(const TeamLaunch& l, const Common& cm, const Geo& geo, const Fields& fl,
                              const Coef<float>& co, const Kry<float>& kr, const TeamArgs& ta);
cudaError_t team_launch_dw(const TeamLaunch& l, const Common& cm, const Geo& geo, const Fields& fl,
                           const Coef<float>& co, const Kry<float>& kr, const TeamArgs& ta);
// largest dynamic shared memory a block of the kernels may use on this device (0: not usable)
size_t team_smem_limit_f64(bool chip);
size_t team_smem_limit_mixed(bool chip);
size_t team_smem_limit_dw(bool chip);

}  // namespace sg
