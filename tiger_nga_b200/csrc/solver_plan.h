// The launch shape of the implicit solve: which kernel, how many warps, matrix areas and blocks. A rule on
// sizes only: what depends on the compiled kernels comes from a query, so that it can be tested without a GPU.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace tng {

// warps per block; SOLVER_8X2 has launch bounds for two blocks per SM (128 registers), SOLVER_POOLED shares
// the block's matrix areas between kPoolWarps warps and keeps the factors in global memory
enum SolverKernelId { SOLVER_2, SOLVER_4, SOLVER_8, SOLVER_8X2, SOLVER_POOLED };
constexpr int kPoolWarps = 12;

struct SolverSizes {  // bytes
  size_t own, area;   // a warp's workspace, a matrix area
  size_t hot, cold;   // the staged tables, the Jacobian's term lists
  size_t optin;       // shared memory of a block at most
  size_t factors;     // the factors of a warp of the pooled kernel; 0: the mechanism has none
};

struct SolverShape {
  int kernel = -1, warps = 0, stages = 0, cold = 0, per_sm = 0;  // cold: term lists in shared memory
  size_t smem = 0, factors = 0;                                  // factors: of all the grid's warps
  int from = 0;  // fewer cells than this have another shape by default (0: all have this one)
};

// the range of cell counts that share a shape
inline int solver_size_class(int64_t ncells, int sm_count) {
  return ncells <= 8LL * sm_count ? 0 : ncells <= 10LL * sm_count ? 1 : 2;
}

// warps / occupancy as configured (tng_cfg; 0 picks the default of the mechanism's size and the number of
// cells); scratch: whether the caller has memory for the factors. resident(kernel, threads, smem): the
// blocks that an SM holds, or a negative value that is returned.
template <class Resident>
int solver_shape(const SolverSizes& z, int warps, int occupancy, int64_t ncells, int sm_count, bool scratch,
                 Resident&& resident, SolverShape* shape) {
  constexpr size_t kStatic = 1024;  // the staged BDF coefficients and the pool's words
  const int cls = solver_size_class(ncells, sm_count);
  const bool pick = warps == 0 && occupancy == 0;
  SolverShape s;
  if (z.factors && scratch && (warps == kPoolWarps || (pick && cls == 2))) {
    // As many matrix areas as fit (a warp holds one for about a third of its time). The line is where
    // the time for 12 warps crosses that for 8, pooled / 8 warps in ms: GRI 1,201 cells 6.25 / 6.02,
    // 1,500 6.65 / 7.35, 3,000 10.4 / 11.3, 24,273 58.9 / 65.2; DME 1,201 15.2 / 14.5, 1,500 16.2 /
    // 16.2, 3,000 23.0 / 24.8, 12,000 69.2 / 77.0. Below it eight warps hold every cell, or all but a few.
    const size_t fixed = z.hot + z.cold + kPoolWarps * z.own + kStatic;
    const int fit = fixed < z.optin ? (int)((z.optin - fixed) / z.area) : 0;
    if (fit >= kPoolWarps / 3) {
      s.kernel = SOLVER_POOLED;
      s.warps = kPoolWarps;
      s.stages = fit < kPoolWarps ? fit : kPoolWarps;
      s.cold = 1;
      s.smem = z.hot + z.cold + kPoolWarps * z.own + s.stages * z.area;
    }
  }
  auto own_areas = [&](int occ) {  // the kernels with a matrix area per warp
    s.warps = (warps == 2 || warps == 4) ? warps : 8;
    s.kernel = s.warps == 2 ? SOLVER_2 : s.warps == 4 ? SOLVER_4 : occ == 2 ? SOLVER_8X2 : SOLVER_8;
    s.stages = s.warps;
    s.smem = z.hot + s.warps * (z.own + z.area);
    // the Jacobian's term tables go to shared memory whenever the blocks still fit
    s.cold = (s.smem + z.cold + kStatic) * occ <= z.optin ? 1 : 0;
    if (s.cold) s.smem += z.cold;
  };
  // A small matrix leaves shared memory for 16 warps per SM: worth their 128 registers once there are cells
  // for them (32,768 hydrogen cells: 14.7 ms, 21.5 ms with 8; 64 registers and 32 warps gain nothing). With
  // one block resident the kernel would spill for nothing: 8 warps with the registers they ask for then.
  const bool two = s.kernel < 0 && pick && !z.factors && cls > 0;
  if (s.kernel < 0) own_areas(two || (warps != 2 && warps != 4 && occupancy == 2) ? 2 : 1);
  s.per_sm = resident(s.kernel, 32 * s.warps, s.smem);
  if (two && s.per_sm >= 0 && s.per_sm < 2) {
    own_areas(1);
    s.per_sm = resident(s.kernel, 32 * s.warps, s.smem);
  }
  if (s.per_sm < 0) return s.per_sm;
  if (pick && s.kernel == SOLVER_POOLED) s.from = 10 * sm_count + 1;
  if (pick && s.kernel == SOLVER_8X2) s.from = 8 * sm_count + 1;
  if (s.kernel == SOLVER_POOLED) s.factors = z.factors * s.warps * (size_t)s.per_sm * sm_count;
  *shape = s;
  return 0;
}

}  // namespace tng
