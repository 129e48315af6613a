// fsph_mixed.cu -- the mixed-precision path: packing of the FP32 records,
// the signal-speed pass, and the launchers of the pair kernels of
// fsph_mixed_kernels.cuh (instances: fsph_mixed_pairs.cu).
#include <cuda_runtime.h>

#include "fsph_internal.cuh"
#include "fsph_mixed_kernels.cuh"

namespace fsph {

static_assert(SPLIT_MAX <= LIST_STAT_MAX, "the walk keeps the statistics the passes read");

// ------------------------------------------------------------- packing --
// PACK_VHM: {v_half, m} and m alone (the FP32 passes, the alpha pass);
// PACK_VEL: {v, c_s before the density pass} (the signal speed);
// PACK_AV_IN: {c_s, sign(div v)} for the Cullen & Dehnen alpha pass;
// PACK_AV: {alpha, 0} for the pair passes that weight the viscosity by it;
// PACK_DEDT: the FP32 de/dt pass's {v, P/rho^2} and {rho, c_s} records;
// PACK_FV: v_half's high and low words with rho and c_s (the float-float
// acceleration pass, the energy passes); PACK_FDV: {v - v_half, m} (the
// energy passes); PACK_VEL_V: v alone into the PACK_VEL record, its c_s
// slot left as the density pass found it (the alpha pass, between the
// density pass and the acceleration pass that reads that slot).  Each pass
// packs only what its kernels read.
enum { PACK_VHM = 1, PACK_VEL = 2, PACK_THERMO = 4, PACK_AV_IN = 8, PACK_AV = 16,
       PACK_DEDT = 32, PACK_FV = 64, PACK_FDV = 128, PACK_VEL_V = 256 };

// Refresh the packed records a pass reads from the FP64 state, so every
// pass sees the current v_half, v, rho, P and c_s whatever the caller did
// in between (separate kicks, repeated pressure updates).
__global__ void k_pack_state(Particles P, int dim, Packed K, int what) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= P.n)
    return;
  // FP32 high word and low word of an FP64 velocity component
  auto hl = [&](int f, float & h, float & l) {
    const double v = P.f[f][i];
    h = to_f32(v);
    l = to_f32(v - to_f64(h));
  };
  if(what & (PACK_VHM | PACK_FV)) {
    float h[3] = {0.f, 0.f, 0.f}, l[3] = {0.f, 0.f, 0.f};
    for(int d = 0; d < dim; ++d)
      hl(F_VHX + d, h[d], l[d]);
    if(what & PACK_VHM) {
      const float m = to_f32(P.f[F_M][i]);
      K.vhm[i] = make_float4(h[0], h[1], h[2], m);
      K.mass[i] = m;
    }
    if(what & PACK_FV) {
      // rho and c_s as the state holds them: after the density pass, the
      // new c_s
      K.fv1[i] = make_float4(h[0], h[1], h[2], to_f32(P.f[F_RHO][i]));
      K.fv2[i] = make_float4(l[0], l[1], l[2], to_f32(P.f[F_CS][i]));
    }
  }
  if(what & PACK_VEL)
    K.vel[i] = make_float4(to_f32(P.f[F_VX][i]), to_f32(P.f[F_VY][i]),
      dim == 3 ? to_f32(P.f[F_VZ][i]) : 0.f, to_f32(P.f[F_CS][i]));
  if(what & PACK_VEL_V) {
    float * v = (float *)&K.vel[i];
    v[0] = to_f32(P.f[F_VX][i]);
    v[1] = to_f32(P.f[F_VY][i]);
    v[2] = dim == 3 ? to_f32(P.f[F_VZ][i]) : 0.f;
  }
  if(what & PACK_THERMO) {
    const double rho = P.f[F_RHO][i], cs = P.f[F_CS][i];
    const double A = P.f[F_P][i] / (rho * rho);
    K.thermo[i] = make_float4((float)rho, (float)A, (float)cs, (float)cs);
    const float Ah = (float)A;
    ((float2 *)K.fmA)[2 * i + 1] = make_float2(Ah, (float)(A - (double)Ah));
  }
  if(what & PACK_AV_IN) {
    // signnum_c of the reference (viscosity.h:63-67), taken in FP64
    const double dv = P.f[F_DIVV][i];
    const float sgn = dv > 0.0 ? 1.f : (dv < 0.0 ? -1.f : (float)dv);
    K.visc[i] = make_float2(to_f32(P.f[F_CS][i]), sgn);
  }
  if(what & PACK_AV)
    K.visc[i] = make_float2(to_f32(P.f[F_ALPHA][i]), 0.f);
  if(what & PACK_DEDT) {
    const double rho = P.f[F_RHO][i];
    K.velp[i] = make_float4(to_f32(P.f[F_VX][i]), to_f32(P.f[F_VY][i]),
      dim == 3 ? to_f32(P.f[F_VZ][i]) : 0.f, (float)(P.f[F_P][i] / (rho * rho)));
    K.rc[i] = make_float2((float)rho, to_f32(P.f[F_CS][i]));
  }
  if(what & PACK_FDV) {
    float dv[3] = {0.f, 0.f, 0.f};
    for(int d = 0; d < dim; ++d)
      dv[d] = (float)(P.f[F_VX + d][i] - P.f[F_VHX + d][i]);
    K.fdv[i] = make_float4(dv[0], dv[1], dv[2], to_f32(P.f[F_M][i]));
  }
}

// -------------------------------------------------------- signal speed --
// Same visiting-order rule as the FP64 pass: neighbours with a higher
// sorted index contribute their new sound speed (thermo.z), the others the
// previous one (thermo.w).
template<int D, bool AUTO>
__global__ void __launch_bounds__(MIX_THREADS) k_vsig_mixed(Particles P, Lists Ls,
  Packed Kp) {
  chain_begin();
  const bool split = four_lanes<AUTO>(Ls);
  const int a = pass_particle<MIX_THREADS>(split);
  if(a >= P.n)
    return;
  const float s0 = Kp.qscale[0], s1 = Kp.qscale[1], s2 = D == 3 ? Kp.qscale[2] : 0.f;
  const int4 qa = Kp.qpos[a];
  const float4 va = Kp.vel[a];
  const float ca = Kp.thermo[a].z;
  const int cnt = Ls.cnt[a];
  const int * lp = Ls.idx + list_slot(a, 0, Ls.maxnb);
  float vsig = 0.f;
  auto pair = [&](int b) {
    const PairGeom g = geom<D>(qa, Kp.qpos[b], s0, s1, s2);
    const float4 vb = Kp.vel[b];
    const float4 tb = Kp.thermo[b];
    const float dotv = ((va.x - vb.x) * g.dx + (va.y - vb.y) * g.dy +
                         (va.z - vb.z) * g.dz) * rsqrtf(g.r2);
    const float cb = b > a ? tb.z : tb.w;
    // the self pair and coincident pairs are NaN in the reference and drop out
    const float cand = fmaxf(ca, cb) - fminf(dotv, 0.f);
    vsig = fmaxf(vsig, (b != a && g.r2 > 0.f) ? cand : 0.f);
  };
  if(split) {
    QuadChunks qc(lp);
    for(int j0 = 0; j0 < cnt; j0 += 4)
      pair(qc.next(j0, cnt));
    vsig = fmaxf(vsig, __shfl_xor_sync(qc.mask, vsig, 1));
    vsig = fmaxf(vsig, __shfl_xor_sync(qc.mask, vsig, 2));
    if((threadIdx.x & 3) != 0)
      return;
  }
  else {
    ListChunks lc(lp);
    for(int j0 = 0; j0 < cnt; j0 += 4) {
      // four slots per 16-byte load; padding slots hold a itself
      const int4 q4 = lc.next(j0, cnt);
      pair(q4.x);
      pair(q4.y);
      pair(q4.z);
      pair(q4.w);
    }
  }
  P.f[F_VSIG][a] = (double)vsig;
}

// a pair pass with the configured viscosity, with the choice of four lanes per
// particle up to SPLIT_MAX particles
#define PAIR_PASS(fn, ...)                                                     \
  do {                                                                         \
    if(pp.cullen)                                                              \
      (P.n <= SPLIT_MAX ? fn##_mixed_cullen_split : fn##_mixed_cullen)(__VA_ARGS__); \
    else                                                                       \
      (P.n <= SPLIT_MAX ? fn##_mixed_split : fn##_mixed)(__VA_ARGS__);         \
  } while(0)

cudaError_t launch_density_mixed(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const Packed & K, double * cs_new,
  DevStatus * st, const DevTime * tm, int vel_current) {
  // velocities of this step for the signal speed (unless the permute of
  // update_iteration wrote them); masses for the FP32 density pass (the
  // float-float one reads them from the position packing)
  const int what = wendland_kernel(pp.kernel) ? (vel_current ? 0 : PACK_VEL)
                                              : PACK_VHM | PACK_VEL;
  if(what) {
    chain(L, k_pack_state, (P.n + PACK_THREADS - 1) / PACK_THREADS, PACK_THREADS, 0, P, pp.dim, K, what);
    *L.counter += 1;
  }
  PAIR_PASS(run_density, L, P, pp, Ls, K, cs_new, st, tm);
  return cudaGetLastError();
}

cudaError_t launch_alpha_mixed(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const Packed & K, const DevTime * t) {
  // current velocities and masses; sound speeds and div v signs of the
  // neighbours
  chain(L, k_pack_state, (P.n + PACK_THREADS - 1) / PACK_THREADS, PACK_THREADS, 0, P, pp.dim, K,
    PACK_VHM | PACK_VEL_V | PACK_AV_IN);
  *L.counter += 1;
  run_alpha_mixed(L, P, pp, Ls, K, t);
  return cudaGetLastError();
}

cudaError_t launch_vsig_mixed(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const Packed & K) {
  const int nb = (P.n + MIX_THREADS - 1) / MIX_THREADS;
  const int ns = (P.n + MIX_THREADS / 4 - 1) / (MIX_THREADS / 4);
  if(P.n <= SPLIT_MAX) {
    if(pp.dim == 3)
      chain(L, k_vsig_mixed<3, true>, ns, MIX_THREADS, 0, P, Ls, K);
    else
      chain(L, k_vsig_mixed<2, true>, ns, MIX_THREADS, 0, P, Ls, K);
  }
  else if(pp.dim == 3)
    chain(L, k_vsig_mixed<3, false>, nb, MIX_THREADS, 0, P, Ls, K);
  else
    chain(L, k_vsig_mixed<2, false>, nb, MIX_THREADS, 0, P, Ls, K);
  *L.counter += 1;
  return cudaGetLastError();
}

cudaError_t launch_accel_mixed(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const Packed & K, int kick,
  const DevTime * t, int fused_vsig, int fv_current) {
  // v_half of this step (set by the caller's save_velocityhalf); the thermo
  // records are refreshed unless they come straight from the density pass
  // (fused signal speed needs their previous-sound-speed slot)
  const int av = pp.cullen ? PACK_AV : 0;
  const int vh = wendland_kernel(pp.kernel) ? (fv_current ? 0 : PACK_FV) : PACK_VHM;
  const int what = (fused_vsig ? vh : (vh | PACK_THERMO)) | av;
  if(what) {
    chain(L, k_pack_state, (P.n + PACK_THREADS - 1) / PACK_THREADS, PACK_THREADS, 0, P, pp.dim, K, what);
    *L.counter += 1;
  }
  PAIR_PASS(run_accel, L, P, pp, Ls, K, kick, t, fused_vsig);
  return cudaGetLastError();
}

cudaError_t launch_dudt_mixed(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const Packed & K, const DevTime * t,
  int then_op, int fv_current, int fdv_current) {
  const int what = (fv_current ? 0 : PACK_FV) | (fdv_current ? 0 : PACK_FDV) |
                   (pp.cullen ? PACK_AV : 0);
  if(what) {
    chain(L, k_pack_state, (P.n + PACK_THREADS - 1) / PACK_THREADS, PACK_THREADS, 0, P, pp.dim, K, what);
    *L.counter += 1;
  }
  PAIR_PASS(run_dudt, L, P, pp, Ls, K, t, then_op);
  return cudaGetLastError();
}

cudaError_t launch_dedt_mixed(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const Packed & K, int then_op,
  const DevTime * t, DevStatus * st, int use_ahyd, int fdv_current) {
  // through a^P, v_half, rho and c_s are those the acceleration pass packed
  // (the caller's flag says so): only v - v_half is new, and not even that
  // when the acceleration pass's kick wrote it
  const int what = (use_ahyd && wendland_kernel(pp.kernel)
                      ? (fdv_current ? 0 : PACK_FDV) : PACK_VHM | PACK_DEDT) |
                   (pp.cullen ? PACK_AV : 0);
  if(what) {
    chain(L, k_pack_state, (P.n + PACK_THREADS - 1) / PACK_THREADS, PACK_THREADS, 0, P, pp.dim, K, what);
    *L.counter += 1;
  }
  PAIR_PASS(run_dedt, L, P, pp, Ls, K, then_op, t, st, use_ahyd);
  return cudaGetLastError();
}

}  // namespace fsph
