// fsph_mixed_pairs.cu -- the mixed-precision pair passes of
// fsph_mixed_kernels.cuh for one viscosity and lane split.  The build compiles
// this file four times, with FSPH_PAIRS_CULLEN and FSPH_PAIRS_SPLIT of 0 or 1.
#include <cuda_runtime.h>

#include "fsph_internal.cuh"
#include "fsph_mixed_kernels.cuh"

#if FSPH_PAIRS_CULLEN && FSPH_PAIRS_SPLIT
#define PAIRS(fn) fn##_mixed_cullen_split
#elif FSPH_PAIRS_CULLEN
#define PAIRS(fn) fn##_mixed_cullen
#elif FSPH_PAIRS_SPLIT
#define PAIRS(fn) fn##_mixed_split
#else
#define PAIRS(fn) fn##_mixed
#endif

namespace fsph {

constexpr bool CULLEN = FSPH_PAIRS_CULLEN != 0, LANES4 = FSPH_PAIRS_SPLIT != 0;

void PAIRS(run_density)(const Launch & L, const Particles & P, const PhysParams & pp,
  const Lists & Ls, const Packed & K, double * cs_new, DevStatus * st, const DevTime * tm) {
  run_density_pass<CULLEN, LANES4>(L, P, pp, Ls, K, cs_new, st, tm);
}

void PAIRS(run_accel)(const Launch & L, const Particles & P, const PhysParams & pp,
  const Lists & Ls, const Packed & K, int kick, const DevTime * t, int fused_vsig) {
  run_accel_pass<CULLEN, LANES4>(L, P, pp, Ls, K, kick, t, fused_vsig);
}

void PAIRS(run_dudt)(const Launch & L, const Particles & P, const PhysParams & pp,
  const Lists & Ls, const Packed & K, const DevTime * t, int then_op) {
  run_dudt_pass<CULLEN, LANES4>(L, P, pp, Ls, K, t, then_op);
}

void PAIRS(run_dedt)(const Launch & L, const Particles & P, const PhysParams & pp,
  const Lists & Ls, const Packed & K, int then_op, const DevTime * t, DevStatus * st,
  int use_ahyd) {
  run_dedt_pass<CULLEN, LANES4>(L, P, pp, Ls, K, then_op, t, st, use_ahyd);
}

}  // namespace fsph
