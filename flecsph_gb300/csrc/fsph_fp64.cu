// fsph_fp64.cu -- the plain-FP64 neighbour-pair kernels (density/EOS,
// signal speed, acceleration, du/dt, de/dt).
//
// One thread per particle walks its neighbour list (interleaved layout, so
// a warp reads 32 consecutive slots per step).  Compiled with -fmad=false and
// evaluated in the reference's operand order: with lists in the reference's
// order the results are those of the reference on the CPU, but for the last
// bits in which libm's pow and cbrt differ from CUDA's, in which quotients and
// roots from a reciprocal may (fsph_pair64.cuh: none has been seen to), in which
// the order of three products in some kernels' gradients shows (there too), and
// in the fused signal speed pairs whose v . x and v . (x / r) round to different
// signs.
#include <cuda_runtime.h>

#include "fsph_pair64.cuh"
#include "fsph_sphmath.cuh"

namespace fsph {

// Blocks of 64: the passes are bound by the FP64 pipe (two FMAs a clock and
// SM), which two warps already fill, so what counts is an even share of warps
// per SM.  Blocks of 256 left 121 of 152 SMs idle at 8k particles and a third
// of the last wave at 91k.
#define PAIR_THREADS 64

// The loops below read a list's slots four at a time; the slots past its end
// hold the particle itself, at distance zero.
__device__ __forceinline__ int slot4(const int4 & q, int u) {
  return u == 0 ? q.x : u == 1 ? q.y : u == 2 ? q.z : q.w;
}

// compute_density + recover_internal_energy + eos (default_physics.h:193-228,
// 126-145, 309-316), and with visc_cullen compute_divv (:273-299) from the same
// traversal.  The new sound speed goes to cs_new: the signal speed still needs
// the old one (see k_vsig).  prho2 receives P / rho^2, which every pair of the
// force and energy passes reads of its neighbour (a division per particle
// instead of one per pair).
template<int D, int K, bool CULL>
__global__ void __launch_bounds__(PAIR_THREADS) k_density(Particles P,
  PhysParams pp, Lists Ls, double * cs_new, double * prho2, DevStatus * st,
  const DevTime * tm) {
  chain_begin();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if(a >= P.n)
    return;
  const double * X = P.f[F_X];
  const double * Y = P.f[F_Y];
  const double * Z = P.f[F_Z];
  const double * H = P.f[F_H];
  const double * M = P.f[F_M];
  const double pa0 = X[a], pa1 = Y[a], pa2 = D == 3 ? Z[a] : 0.0;
  const double h_a = H[a];
  double va[3] = {0.0, 0.0, 0.0};
  if(CULL)
    for(int d = 0; d < D; ++d)
      va[d] = P.f[F_VX + d][a];
  const int cnt = Ls.cnt[a];
  const int * lp = Ls.idx + list_slot(a, 0, Ls.maxnb);
  double rho_a = 0.0, div_v = 0.0;
  PairH<D, K> ph;
  ph.init();
  for(int j0 = 0; j0 < cnt; j0 += 4) {
    const int4 q4 = *(const int4 *)(lp + (j0 << 5));
#pragma unroll
    for(int u = 0; u < 4; ++u) {
      const int b = slot4(q4, u);
      const double d0 = pa0 - X[b], d1 = pa1 - Y[b];
      double r2 = d0 * d0 + d1 * d1, d2 = 0.0;
      if(D == 3) {
        d2 = pa2 - Z[b];
        r2 += d2 * d2;
      }
      const PairR r = pair_r(r2);
      ph.template set<true, CULL>(h_a, H[b], pp);
      const double mb = M[b];
      const double w = mb * pair_w<D, K>(r.r, ph, pp);
      if(j0 + u < cnt)
        rho_a += w;
      if(CULL) {
        const double f = pair_g<D, K>(r, ph, pp);
        double dot = va[0] * (d0 * f) + va[1] * (d1 * f);
        if(D == 3)
          dot += va[2] * (d2 * f);
        div_v += mb * dot;  // the padding slots' terms are zero
      }
    }
  }
  if(!(rho_a > 0))
    raise_status(st, FSPH_ERR_NEG_DENSITY, a);
  P.f[F_RHO][a] = rho_a;
  double u = P.f[F_U][a];
  if(pp.evolve_u && pp.thermokinetic) {
    double vv = 0;
    for(int d = 0; d < D; ++d)
      vv += P.f[F_VX + d][a] * P.f[F_VX + d][a];
    double ekin = .5 * vv;
    const double pos_a[3] = {pa0, pa1, pa2};
    double eint = P.f[F_E][a] - ekin - ext_potential<D>(pp, pos_a);
    if(!(eint > 0))
      raise_status(st, FSPH_ERR_NEG_ENERGY, a);
    u = eint;
    P.f[F_U][a] = u;
  }
  double Pa, cs;
  eos_p_cs(pp, rho_a, u, P.f[F_K][a], P.f[F_YE][a], P.f[F_P][a], P.f[F_CS][a], Pa,
    cs);
  P.f[F_P][a] = Pa;
  cs_new[a] = cs;
  prho2[a] = kept_prho2(pp, Pa, rho_a, cs, P.f[F_ALPHA][a]);
  if(CULL) {
    div_v /= rho_a;
    const double div_v_p = P.f[F_DIVV][a];
    P.f[F_DDIVVDT][a] = (div_v - div_v_p) / tm->dt;
    P.f[F_DIVV][a] = div_v;
  }
}

// P / rho^2 of every particle where the density pass's is out of date (a
// caller changed P, rho, c_s or alpha in between).
__global__ void __launch_bounds__(256) k_prho2(Particles P, PhysParams pp,
  double * prho2) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i < P.n)
    prho2[i] = kept_prho2(pp, P.f[F_P][i], P.f[F_RHO][i], P.f[F_CS][i], P.f[F_ALPHA][i]);
}

// viscosity::compute_alpha with A_trigger and compute_xi (viscosity.h:
// 185-363): Cullen & Dehnen's adaptive alpha from the velocity divergence,
// its rate and the traceless shear, in the reference's operand order.  prho2 is
// written anew, with the new alpha.
template<int D, int K>
__global__ void __launch_bounds__(PAIR_THREADS) k_alpha_cullen(Particles P,
  PhysParams pp, Lists Ls, const DevTime * tm, double * prho2) {
  chain_begin();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if(a >= P.n)
    return;
  const double * X = P.f[F_X];
  const double * Y = P.f[F_Y];
  const double * Z = P.f[F_Z];
  const double * H = P.f[F_H];
  const double * M = P.f[F_M];
  const double * CS = P.f[F_CS];
  const double * DV = P.f[F_DIVV];
  const double * V[3] = {P.f[F_VX], P.f[F_VY], P.f[F_VZ]};
  const double c_a = CS[a], h_a = H[a], alpha_a = P.f[F_ALPHA][a];
  const double rho_a = P.f[F_RHO][a];
  const double pa[3] = {X[a], Y[a], D == 3 ? Z[a] : 0.0};
  double va[3] = {0, 0, 0};
  for(int d = 0; d < D; ++d)
    va[d] = V[d][a];
  const int cnt = Ls.cnt[a];
  // signal speed of this pass: all sound speeds are the new ones here
  double vsig = 0.0;
  // compute_xi accumulations
  double R_a = 0.0;
  double gradV[D * D];
  for(int k = 0; k < D * D; ++k)
    gradV[k] = 0.0;
  const int * lp = Ls.idx + list_slot(a, 0, Ls.maxnb);
  PairH<D, K> ph;
  ph.init();
  for(int j = 0; j < cnt; ++j) {
    const int b = lp[slot_off(j)];
    const double pb[3] = {X[b], Y[b], D == 3 ? Z[b] : 0.0};
    double pos_ab[3] = {0, 0, 0}, vab[3] = {0, 0, 0};
    double dist2 = 0.0;
    for(int d = 0; d < D; ++d) {
      pos_ab[d] = pa[d] - pb[d];
      vab[d] = va[d] - V[d][b];
      dist2 += pos_ab[d] * pos_ab[d];
    }
    const PairR r = pair_r(dist2);
    // vsig = max(vsig, max(c_a, c_b) - min(v_ab . n_ab, 0)); the self pair
    // (0/0) is a NaN that std::max drops
    if(nonzero(dist2)) {
      const double cmax = c_a < CS[b] ? CS[b] : c_a;
      const double cand = cmax - approach<D>(vab, pos_ab, r);
      vsig = vsig < cand ? cand : vsig;      // std::max(vsig, cand)
    }
    ph.template set<true, true>(h_a, H[b], pp);
    const double f = pair_g<D, K>(r, ph, pp);
    const double Wab = pair_w<D, K>(r.r, ph, pp);
    const double dvb = DV[b];
    const double sgn = dvb > 0.0 ? 1.0 : (dvb < 0.0 ? -1.0 : dvb);
    R_a += sgn * M[b] * Wab;
    for(int k = 0; k < D; ++k) {
      const double DiW = pos_ab[k] * f;
      for(int i = 0; i < D; ++i)
        gradV[D * i + k] += M[b] * (-vab[i]) * DiW;
    }
  }
  R_a /= rho_a;
  for(int k = 0; k < D * D; ++k)
    gradV[k] /= rho_a;
  const double divV_a = DV[a];
  double traceSS = 0.0;
  for(int i = 0; i < D; ++i) {
    double row[3];
    for(int k = 0; k < D; ++k)
      row[k] = 0.5 * (gradV[D * i + k] + gradV[D * k + i]);
    row[i] -= divV_a / D;
    for(int k = 0; k < D; ++k)
      traceSS += row[k] * row[k];
  }
  const double om = 1.0 - R_a;
  const double q4 = om * om * om * om;
  const double t = 2.0 * q4 * divV_a;
  const double res = t * t;
  const double xi = (res < 1e-16) ? 0.0 : res / (res + traceSS);
  const double ddv = P.f[F_DDIVVDT][a];
  const double trig = -ddv < 0.0 ? 0.0 : -ddv;   // std::max(-dDivVdt, 0.0)
  const double Atrig = xi * trig;
  const double vh = vsig / h_a;
  const double alpha_loc = pp.alpha_max * Atrig / (pp.visc_delta * (vh * vh) + Atrig);
  double alpha;
  if(alpha_a <= alpha_loc)
    alpha = alpha_loc;
  else {
    const double decayt = h_a / (2.0 * pp.visc_l * vsig);
    const double dalphadt = (alpha_a - alpha_loc) / decayt;
    alpha = alpha_a * exp(-dalphadt * tm->dt);
  }
  P.f[F_ALPHA][a] = alpha;
  prho2[a] = kept_prho2(pp, P.f[F_P][a], rho_a, c_a, alpha);
}

// compute_signalspeed (default_physics.h:236-265).  The reference visits
// particles in descending key order and sets each particle's sound speed
// just before its signal speed (tree_topology.h:220-235,401-408;
// default_physics.h:309-317), so a neighbour with a higher sorted index
// (visited earlier) contributes its new sound speed, any other its old one.
template<int D>
__global__ void __launch_bounds__(PAIR_THREADS) k_vsig(Particles P, Lists Ls,
  const double * cs_new) {
  chain_begin();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if(a >= P.n)
    return;
  const double * X = P.f[F_X];
  const double * Y = P.f[F_Y];
  const double * Z = P.f[F_Z];
  const double * VX = P.f[F_VX];
  const double * VY = P.f[F_VY];
  const double * VZ = P.f[F_VZ];
  const double * CS = P.f[F_CS];
  const double pa0 = X[a], pa1 = Y[a], pa2 = D == 3 ? Z[a] : 0.0;
  const double va0 = VX[a], va1 = VY[a], va2 = D == 3 ? VZ[a] : 0.0;
  const double c_a = cs_new[a];
  const double va[3] = {va0, va1, va2};
  const int cnt = Ls.cnt[a];
  const int * lp = Ls.idx + list_slot(a, 0, Ls.maxnb);
  double vsig = 0.0;
  for(int j = 0; j < cnt; ++j) {
    const int b = lp[slot_off(j)];
    const double x[3] = {pa0 - X[b], pa1 - Y[b], D == 3 ? pa2 - Z[b] : 0.0};
    double dist2 = x[0] * x[0] + x[1] * x[1];
    if(D == 3)
      dist2 += x[2] * x[2];
    if(!nonzero(dist2))
      continue;  // the self pair's 0/0 drops out of the reference's maximum
    double v[3] = {va[0] - VX[b], va[1] - VY[b], D == 3 ? va[2] - VZ[b] : 0.0};
    const double c_b = b >= a ? cs_new[b] : CS[b];
    const double cab = c_a < c_b ? c_b : c_a;
    const double cand = cab - approach<D>(v, x, pair_r(dist2));
    vsig = vsig < cand ? cand : vsig;
  }
  P.f[F_VSIG][a] = vsig;
}

// compute_acceleration (default_physics.h:348-408); optionally followed by
// leapfrog_kick_v (integration.h:65-70) for the same particle: the pass
// reads only v_half of neighbours, never v.
//
// With VSIG the signal speed of k_vsig rides along: the caller says that v
// equals v_half everywhere (true in a driver iteration, where both are saved
// together), so the pair's velocity difference, distance and its reciprocal
// are at hand; cs_old is the sound speed before the density pass.
//
// The pass leaves {grad W factor, Pi} of every pair in `pair` (16 bytes, slot
// j of particle a at [a >> 5][j][a & 31]) for the energy pass, which needs the
// same two values: read back from HBM they cost a fraction of the ~60 FP64
// operations that recompute them.
//
// Bound by the FP64 pipe.  Per pair of a uniform-h run 3D: ~60 operations, and
// ~35 more in the branch of approaching pairs, which holds what only the
// viscosity needs (its two divisions among them); recomputing every division
// per pair (six and a root) took 130 and more.
template<int D, int K, bool VSIG>
__global__ void __launch_bounds__(PAIR_THREADS) k_accel(Particles P,
  PhysParams pp, Lists Ls, int kick, const DevTime * tm, const double * prho2,
  const double * cs_old, double2 * pair) {
  chain_begin();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if(a >= P.n)
    return;
  const double * X = P.f[F_X];
  const double * Y = P.f[F_Y];
  const double * Z = P.f[F_Z];
  const double * H = P.f[F_H];
  const double * M = P.f[F_M];
  const double * RHO = P.f[F_RHO];
  const double * CS = P.f[F_CS];
  const double * VH[3] = {P.f[F_VHX], P.f[F_VHY], P.f[F_VHZ]};
  const double h_a = H[a], rho_a = RHO[a], c_a = CS[a];
  double pa[3] = {X[a], Y[a], D == 3 ? Z[a] : 0.0};
  double v12a[3];
  for(int d = 0; d < D; ++d)
    v12a[d] = VH[d][a];
  const double Prho2_a = prho2[a];
  double acc[3] = {0, 0, 0};
  double vsig = 0.0;
  const int cnt = Ls.cnt[a];
  const int * lp = Ls.idx + list_slot(a, 0, Ls.maxnb);
  double2 * pw = pair ? pair + pair_slot(a, 0, Ls.maxnb) : nullptr;
  PairH<D, K> ph;
  ph.init();
  for(int j0 = 0; j0 < cnt; j0 += 4) {
    const int4 q4 = *(const int4 *)(lp + (j0 << 5));
#pragma unroll
    for(int u = 0; u < 4; ++u) {
      const int b = slot4(q4, u);
      double pos_ab[3] = {0, 0, 0}, v12_ab[3] = {0, 0, 0};
      pos_ab[0] = pa[0] - X[b];
      pos_ab[1] = pa[1] - Y[b];
      double dist2 = pos_ab[0] * pos_ab[0] + pos_ab[1] * pos_ab[1];
      if(D == 3) {
        pos_ab[2] = pa[2] - Z[b];
        dist2 += pos_ab[2] * pos_ab[2];
      }
      for(int d = 0; d < D; ++d)
        v12_ab[d] = v12a[d] - VH[d][b];
      double dotp = v12_ab[0] * pos_ab[0] + v12_ab[1] * pos_ab[1];
      if(D == 3)
        dotp += v12_ab[2] * pos_ab[2];
      ph.template set<false, true>(h_a, H[b], pp);
      const PairR r = pair_r(dist2);
      const double f = pair_g<D, K>(r, ph, pp);
      // mu and Pi are zero unless the pair approaches (viscosity.h:81-93)
      const double Prho2_b = prho2[b];
      double Pi = pi_apart(Prho2_a, Prho2_b, dotp);
      double appr = nan64(dotp) ? dotp : 0.0;  // (drops out of the maximum)
      if(dotp < 0.0) {
        Pi = pair_pi<D>(pp, P.f[F_ALPHA], a, b, .5 * (rho_a + RHO[b]),
          .5 * (c_a + CS[b]), ph.h, dotp, dist2);
        if(VSIG)
          appr = approach<D>(v12_ab, pos_ab, r);
      }
      if(VSIG && nonzero(dist2)) {
        const double c_b = b >= a ? CS[b] : cs_old[b];
        const double cand = (c_a < c_b ? c_b : c_a) - appr;
        vsig = vsig < cand ? cand : vsig;
      }
      // the self pair, coincident pairs and padding slots have x_ab = 0 and
      // f = 0: their terms vanish, as the reference's m_b = 0 makes them
      const double s = -M[b] * (Prho2_a + Prho2_b + Pi);
      for(int d = 0; d < D; ++d)
        acc[d] += pos_ab[d] * f * s;
      if(pw)
        pw[(size_t)(j0 + u) * 32] = make_double2(f, Pi);
    }
  }
  // acc_a += external_force::acceleration(particle) (:404)
  double ext[3] = {0.0, 0.0, 0.0};
  if(pp.has_eacc)
    ext_acceleration<D>(pp, pa, ext);
  const double half_dt = kick ? 0.5 * tm->dt : 0.0;
  for(int d = 0; d < D; ++d) {
    const double ad = acc[d] + ext[d];
    P.f[F_AX + d][a] = ad;
    P.f[F_GAX + d][a] = 0.0;
    if(kick)
      P.f[F_VX + d][a] = P.f[F_VX + d][a] + (ad + 0.0) * half_dt;
  }
  P.f[F_GPOT][a] = 0.0;
  if(VSIG)
    P.f[F_VSIG][a] = vsig;
}

// The gradient factor and Pi of one pair: read from the acceleration pass's
// `pair` (KEPT) or evaluated.
template<int D, int K, bool KEPT>
__device__ __forceinline__ double2 pair_terms(const Particles & P, const PhysParams & pp,
  PairH<D, K> & ph, const double2 * pr, int j, int a, int b, const double * pos_ab,
  const double * v12a, double h_a, double rho_a, double c_a, const double * prho2) {
  if(KEPT)
    return pr[(size_t)j * 32];
  double dist2 = 0.0, dotp = 0.0;
  for(int d = 0; d < D; ++d) {
    dist2 += pos_ab[d] * pos_ab[d];
    dotp += (v12a[d] - P.f[F_VHX + d][b]) * pos_ab[d];
  }
  ph.template set<false, true>(h_a, P.f[F_H][b], pp);
  double2 t = make_double2(pair_g<D, K>(pair_r(dist2), ph, pp),
    pi_apart(prho2[a], prho2[b], dotp));
  if(dotp < 0.0)
    t.y = pair_pi<D>(pp, P.f[F_ALPHA], a, b, .5 * (rho_a + P.f[F_RHO][b]),
      .5 * (c_a + P.f[F_CS][b]), ph.h, dotp, dist2);
  return t;
}

// compute_dudt (default_physics.h:421-487).  KEPT: the pair terms of the
// acceleration pass are still those of the state.
template<int D, int K, bool KEPT>
__global__ void __launch_bounds__(PAIR_THREADS) k_dudt(Particles P,
  PhysParams pp, Lists Ls, const DevTime * tm, const double * prho2,
  const double2 * pair) {
  chain_begin();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if(a >= P.n)
    return;
  // no internal energy change while relaxing (:423-427)
  if(tm->iteration < pp.relax_steps) {
    P.f[F_DUDT][a] = 0.0;
    return;
  }
  const double h_a = P.f[F_H][a], rho_a = P.f[F_RHO][a], c_a = P.f[F_CS][a];
  double pa[3] = {0, 0, 0}, va[3] = {0, 0, 0}, v12a[3] = {0, 0, 0};
  for(int d = 0; d < D; ++d) {
    pa[d] = P.f[F_X + d][a];
    va[d] = P.f[F_VX + d][a];
    v12a[d] = P.f[F_VHX + d][a];
  }
  double dp = 0.0, dv = 0.0;
  const int cnt = Ls.cnt[a];
  const int * lp = Ls.idx + list_slot(a, 0, Ls.maxnb);
  const double2 * pr = KEPT ? pair + pair_slot(a, 0, Ls.maxnb) : nullptr;
  PairH<D, K> ph;
  ph.init();
  for(int j0 = 0; j0 < cnt; j0 += 4) {
    const int4 q4 = *(const int4 *)(lp + (j0 << 5));
#pragma unroll
    for(int u = 0; u < 4; ++u) {
      const int b = slot4(q4, u);
      double pos_ab[3] = {0, 0, 0};
      for(int d = 0; d < D; ++d)
        pos_ab[d] = pa[d] - P.f[F_X + d][b];
      const double2 t = pair_terms<D, K, KEPT>(P, pp, ph, pr, j0 + u, a, b, pos_ab, v12a,
        h_a, rho_a, c_a, prho2);
      double vdw = 0;
      for(int d = 0; d < D; ++d)
        vdw += (va[d] - P.f[F_VX + d][b]) * (pos_ab[d] * t.x);
      const double mvdw = P.f[F_M][b] * vdw;
      dp += mvdw;
      dv += mvdw * t.y;
    }
  }
  P.f[F_DUDT][a] = prho2[a] * dp + .5 * dv;
}

// compute_dedt (default_physics.h:502-566).  KEPT: as in k_dudt.
template<int D, int K, bool KEPT>
__global__ void __launch_bounds__(PAIR_THREADS) k_dedt(Particles P,
  PhysParams pp, Lists Ls, const double * prho2, const double2 * pair) {
  chain_begin();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if(a >= P.n)
    return;
  const double h_a = P.f[F_H][a], rho_a = P.f[F_RHO][a], c_a = P.f[F_CS][a];
  double pa[3] = {0, 0, 0}, va[3] = {0, 0, 0}, v12a[3] = {0, 0, 0};
  double gv = 0;
  for(int d = 0; d < D; ++d) {
    pa[d] = P.f[F_X + d][a];
    va[d] = P.f[F_VX + d][a];
    v12a[d] = P.f[F_VHX + d][a];
    gv += P.f[F_GAX + d][a] * va[d];
  }
  const double Prho2_a = prho2[a];
  double dedt = 0;
  const int cnt = Ls.cnt[a];
  const int * lp = Ls.idx + list_slot(a, 0, Ls.maxnb);
  const double2 * pr = KEPT ? pair + pair_slot(a, 0, Ls.maxnb) : nullptr;
  PairH<D, K> ph;
  ph.init();
  for(int j0 = 0; j0 < cnt; j0 += 4) {
    const int4 q4 = *(const int4 *)(lp + (j0 << 5));
#pragma unroll
    for(int u = 0; u < 4; ++u) {
      const int b = slot4(q4, u);
      double pos_ab[3] = {0, 0, 0};
      for(int d = 0; d < D; ++d)
        pos_ab[d] = pa[d] - P.f[F_X + d][b];
      const double2 t = pair_terms<D, K, KEPT>(P, pp, ph, pr, j0 + u, a, b, pos_ab, v12a,
        h_a, rho_a, c_a, prho2);
      double vad = 0, vbd = 0;
      for(int d = 0; d < D; ++d) {
        const double DiW = pos_ab[d] * t.x;
        vad += va[d] * DiW;
        vbd += P.f[F_VX + d][b] * DiW;
      }
      dedt -= P.f[F_M][b] * (Prho2_a * vbd + vad * prho2[b] + .5 * t.y * (vbd + vad));
    }
  }
  dedt += gv;
  P.f[F_DEDT][a] = dedt;
}

// ------------------------------------------------------------ dispatch --
#define DISPATCH_DK(KERNEL_T, TA, ...)                                             \
  do {                                                                         \
    const int nb_ = (P.n + PAIR_THREADS - 1) / PAIR_THREADS;                   \
    if(pp.dim == 3) {                                                          \
      switch(pp.kernel) {                                                      \
        case FSPH_KERNEL_CUBIC_SPLINE:                                         \
          chain(L, KERNEL_T<3, FSPH_KERNEL_CUBIC_SPLINE TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_QUINTIC_SPLINE:                                       \
          chain(L, KERNEL_T<3, FSPH_KERNEL_QUINTIC_SPLINE TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_GAUSSIAN:                                             \
          chain(L, KERNEL_T<3, FSPH_KERNEL_GAUSSIAN TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_SUPER_GAUSSIAN:                                       \
          chain(L, KERNEL_T<3, FSPH_KERNEL_SUPER_GAUSSIAN TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_SINC:                                                 \
          chain(L, KERNEL_T<3, FSPH_KERNEL_SINC TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_WENDLAND_C2:                                          \
          chain(L, KERNEL_T<3, FSPH_KERNEL_WENDLAND_C2 TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_WENDLAND_C4:                                          \
          chain(L, KERNEL_T<3, FSPH_KERNEL_WENDLAND_C4 TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        default:                                                               \
          chain(L, KERNEL_T<3, FSPH_KERNEL_WENDLAND_C6 TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
      }                                                                        \
    }                                                                          \
    else {                                                                     \
      switch(pp.kernel) {                                                      \
        case FSPH_KERNEL_CUBIC_SPLINE:                                         \
          chain(L, KERNEL_T<2, FSPH_KERNEL_CUBIC_SPLINE TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_QUINTIC_SPLINE:                                       \
          chain(L, KERNEL_T<2, FSPH_KERNEL_QUINTIC_SPLINE TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_GAUSSIAN:                                             \
          chain(L, KERNEL_T<2, FSPH_KERNEL_GAUSSIAN TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_SUPER_GAUSSIAN:                                       \
          chain(L, KERNEL_T<2, FSPH_KERNEL_SUPER_GAUSSIAN TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_SINC:                                                 \
          chain(L, KERNEL_T<2, FSPH_KERNEL_SINC TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_WENDLAND_C2:                                          \
          chain(L, KERNEL_T<2, FSPH_KERNEL_WENDLAND_C2 TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        case FSPH_KERNEL_WENDLAND_C4:                                          \
          chain(L, KERNEL_T<2, FSPH_KERNEL_WENDLAND_C4 TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
        default:                                                               \
          chain(L, KERNEL_T<2, FSPH_KERNEL_WENDLAND_C6 TA>, nb_, PAIR_THREADS, 0, __VA_ARGS__); break; \
      }                                                                        \
    }                                                                          \
    *L.counter += 1;                                                           \
  } while(0)

#define TARG(X) , X

cudaError_t launch_density_fp64(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, double * cs_new, double * prho2,
  DevStatus * st, const DevTime * t) {
  if(pp.cullen)
    DISPATCH_DK(k_density, TARG(true), P, pp, Ls, cs_new, prho2, st, t);
  else
    DISPATCH_DK(k_density, TARG(false), P, pp, Ls, cs_new, prho2, st, t);
  return cudaGetLastError();
}

cudaError_t launch_prho2(const Launch & L, const Particles & P, const PhysParams & pp,
  double * prho2) {
  chain(L, k_prho2, (P.n + 255) / 256, 256, 0, P, pp, prho2);
  *L.counter += 1;
  return cudaGetLastError();
}

cudaError_t launch_alpha_cullen(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const DevTime * t, double * prho2) {
  DISPATCH_DK(k_alpha_cullen, , P, pp, Ls, t, prho2);
  return cudaGetLastError();
}

// add_short_range_repulsion (default_physics.h:723-753): neighbours other
// than the particle itself (by id) within relaxation_repulsion_radius of
// h_ab push it away with m_b x_ab / r_ab^3, scaled by
// relaxation_repulsion_gamma.  FP64 on both precision paths (it runs in
// relaxation iterations only).
template<int D>
__global__ void __launch_bounds__(PAIR_THREADS) k_repulsion(Particles P,
  PhysParams pp, Lists Ls) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if(a >= P.n)
    return;
  const double * H = P.f[F_H];
  const double * M = P.f[F_M];
  const double h_a = H[a];
  const long long id_a = P.id[a];
  double pa[3] = {0.0, 0.0, 0.0}, acc_r[3] = {0.0, 0.0, 0.0};
  for(int d = 0; d < D; ++d)
    pa[d] = P.f[F_X + d][a];
  const int cnt = Ls.cnt[a];
  for(int j = 0; j < cnt; ++j) {
    const int b = Ls.idx[list_slot(a, j, Ls.maxnb)];
    if(P.id[b] == id_a)
      continue;
    double dx[3] = {0.0, 0.0, 0.0};
    double r2 = 0.0;
    for(int d = 0; d < D; ++d) {
      dx[d] = pa[d] - P.f[F_X + d][b];
      r2 += dx[d] * dx[d];
    }
    const double h_ab = .5 * (h_a + H[b]);
    const double r_ab = sqrt(r2);
    if(r_ab > h_ab * pp.rep_radius)
      continue;
    const double m_b = M[b];
    const double r3 = r_ab * r_ab * r_ab;
    for(int d = 0; d < D; ++d)
      acc_r[d] += m_b * dx[d] / r3;
  }
  for(int d = 0; d < D; ++d)
    P.f[F_AX + d][a] = P.f[F_AX + d][a] + acc_r[d] * pp.rep_gamma;
}

cudaError_t launch_repulsion(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls) {
  const int nb = (P.n + PAIR_THREADS - 1) / PAIR_THREADS;
  if(pp.dim == 3)
    k_repulsion<3><<<nb, PAIR_THREADS, 0, L.stream>>>(P, pp, Ls);
  else
    k_repulsion<2><<<nb, PAIR_THREADS, 0, L.stream>>>(P, pp, Ls);
  *L.counter += 1;
  return cudaGetLastError();
}

cudaError_t launch_vsig_fp64(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const double * cs_new) {
  const int nb = (P.n + PAIR_THREADS - 1) / PAIR_THREADS;
  if(pp.dim == 3)
    chain(L, k_vsig<3>, nb, PAIR_THREADS, 0, P, Ls, cs_new);
  else
    chain(L, k_vsig<2>, nb, PAIR_THREADS, 0, P, Ls, cs_new);
  *L.counter += 1;
  return cudaGetLastError();
}

cudaError_t launch_accel_fp64(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, int kick, const DevTime * t,
  const double * prho2, const double * cs_old, double2 * pair) {
  if(cs_old)
    DISPATCH_DK(k_accel, TARG(true), P, pp, Ls, kick, t, prho2, cs_old, pair);
  else
    DISPATCH_DK(k_accel, TARG(false), P, pp, Ls, kick, t, prho2, cs_old, pair);
  return cudaGetLastError();
}

cudaError_t launch_dudt_fp64(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const DevTime * t, const double * prho2,
  const double2 * pair) {
  if(pair)
    DISPATCH_DK(k_dudt, TARG(true), P, pp, Ls, t, prho2, pair);
  else
    DISPATCH_DK(k_dudt, TARG(false), P, pp, Ls, t, prho2, pair);
  return cudaGetLastError();
}

cudaError_t launch_dedt_fp64(const Launch & L, const Particles & P,
  const PhysParams & pp, const Lists & Ls, const double * prho2,
  const double2 * pair) {
  if(pair)
    DISPATCH_DK(k_dedt, TARG(true), P, pp, Ls, prho2, pair);
  else
    DISPATCH_DK(k_dedt, TARG(false), P, pp, Ls, prho2, pair);
  return cudaGetLastError();
}

}  // namespace fsph
