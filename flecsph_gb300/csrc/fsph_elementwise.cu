// fsph_elementwise.cu -- per-particle (apply_all / get_all) kernels, the
// timestep reduction and the scalar time bookkeeping, all FP64 and
// compiled with -fmad=false so they round like the reference.
#include <cuda_runtime.h>

#include "fsph_range.cuh"
#include "fsph_sphmath.cuh"

namespace fsph {

#define ELEM_THREADS 256

__device__ __forceinline__ double dmin_(double a, double b) { return b < a ? b : a; }

// recover_internal_energy (default_physics.h:126-145)
template<int D>
__device__ __forceinline__ double recover_u(const Particles & P,
  const PhysParams & pp, int i, DevStatus * st) {
  double vv = 0;
  for(int d = 0; d < D; ++d)
    vv += P.f[F_VX + d][i] * P.f[F_VX + d][i];
  double ekin = .5 * vv;
  double eint = P.f[F_E][i] - ekin - ext_potential_of<D>(pp, P.f, i);
  if(!(eint > 0))
    raise_status(st, FSPH_ERR_NEG_ENERGY, i);
  return eint;
}

template<int D>
__global__ void __launch_bounds__(ELEM_THREADS) k_elem(Particles P,
  PhysParams pp, int op, const DevTime * tm, DevStatus * st) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= P.n)
    return;
  double ** f = P.f;
  const double dt = tm->dt;
  switch(op) {
    case OP_EOS_INIT:  // eos_t<>::init (eos.h:67-92, 157-159, 240-243, 345-364)
      if(pp.eos == FSPH_EOS_WD)
        f[F_U][i] = wd_internal_energy(f[F_RHO][i], f[F_YE][i]);
      else if(pp.eos == FSPH_EOS_PPT) {
        const double rho = f[F_RHO][i], P_ = f[F_P][i], thr = pp.rho_thr;
        double K1 = 0.0;
        if(rho < thr)
          K1 = P_ / pow(rho, pp.gamma);
        else {
          double K2 = P_ / pow(rho, pp.gamma2);
          K1 = K2 * pow(thr, pp.gamma2 - pp.gamma);
        }
        f[F_K][i] = K1;
      }
      else if(pp.eos != FSPH_EOS_NO_EOS)
        f[F_K][i] = f[F_P][i] / pow(f[F_RHO][i], pp.gamma);
      break;
    case OP_SET_TOTAL_ENERGY: {  // default_physics.h:327-335
      double vv = 0;
      for(int d = 0; d < D; ++d)
        vv += f[F_VX + d][i] * f[F_VX + d][i];
      double ekin = .5 * vv;
      f[F_E][i] = ekin + f[F_U][i] + ext_potential_of<D>(pp, f, i);
      break;
    }
    case OP_SAVE_VHALF:  // integration.h:52-55
      for(int d = 0; d < D; ++d)
        f[F_VHX + d][i] = f[F_VX + d][i];
      break;
    case OP_KICK_V: {  // integration.h:65-70
      const double s = 0.5 * dt;
      for(int d = 0; d < D; ++d)
        f[F_VX + d][i] = f[F_VX + d][i] + (f[F_AX + d][i] + f[F_GAX + d][i]) * s;
      break;
    }
    case OP_KICK_U:  // integration.h:80-84
      f[F_U][i] = f[F_U][i] + 0.5 * dt * f[F_DUDT][i];
      break;
    case OP_KICK_E:  // integration.h:94-98
      f[F_E][i] = f[F_E][i] + 0.5 * dt * f[F_DEDT][i];
      break;
    case OP_DRIFT:  // integration.h:106-110
      for(int d = 0; d < D; ++d)
        f[F_X + d][i] = f[F_X + d][i] + f[F_VX + d][i] * dt;
      break;
    case OP_RECOMPUTE:
    case OP_RECOMPUTE_KICK_U: {  // default_physics.h:153-161 (+ kick_u)
      double uint = f[F_U][i];
      double P_, cs;
      eos_p_cs(pp, f[F_RHO][i], uint + 0.5 * dt * f[F_DUDT][i], f[F_K][i],
        f[F_YE][i], f[F_P][i], f[F_CS][i], P_, cs);
      f[F_P][i] = P_;
      f[F_CS][i] = cs;
      if(op == OP_RECOMPUTE_KICK_U)
        f[F_U][i] = uint + 0.5 * dt * f[F_DUDT][i];
      break;
    }
    case OP_RECOMPUTE_THERMO:
    case OP_RECOMPUTE_KICK_E: {  // default_physics.h:169-182 (+ kick_e)
      double eint = recover_u<D>(P, pp, i, st);
      f[F_U][i] = eint;
      double vda = 0;
      for(int d = 0; d < D; ++d)
        vda += f[F_VX + d][i] * f[F_AX + d][i];
      double P_, cs;
      eos_p_cs(pp, f[F_RHO][i], eint + 0.5 * dt * (f[F_DEDT][i] - vda),
        f[F_K][i], f[F_YE][i], f[F_P][i], f[F_CS][i], P_, cs);
      f[F_P][i] = P_;
      f[F_CS][i] = cs;
      if(op == OP_RECOMPUTE_KICK_E)
        f[F_E][i] = f[F_E][i] + 0.5 * dt * f[F_DEDT][i];
      break;
    }
    case OP_SMOOTHING_LENGTH: {  // default_physics.h:825-848
      double q = f[F_M][i] / f[F_RHO][i];
      double r = D == 3 ? cbrt(q) : sqrt(q);
      f[F_H][i] = r * pp.eta * pp.kw;
      break;
    }
    case OP_INIT_ALPHA:  // viscosity::initialize_alpha (viscosity.h:171-177)
      f[F_ALPHA][i] = pp.cullen ? 0.0 : pp.alpha;
      break;
    case OP_DRAG_ACC:    // add_drag_acceleration (default_physics.h:699-708)
    case OP_DRAG_DEDT:   // add_drag_dedt (:571-579)
    case OP_DRAG_DUDT: { // add_drag_dudt (:586-594)
      double vel[3] = {0.0, 0.0, 0.0}, drag[3];
      for(int d = 0; d < D; ++d)
        vel[d] = f[F_VX + d][i];
      drag_acceleration<D>(pp, vel, drag);
      if(op == OP_DRAG_ACC) {
        for(int d = 0; d < D; ++d)
          f[F_AX + d][i] = f[F_AX + d][i] + drag[d];
      }
      else {
        double v_dot_a = 0.0;
        for(int d = 0; d < D; ++d)
          v_dot_a += vel[d] * drag[d];
        const int F = op == OP_DRAG_DEDT ? F_DEDT : F_DUDT;
        f[F][i] = f[F][i] + v_dot_a;
      }
      break;
    }
    case OP_SET_H:  // second half of compute_average_smoothinglength
      f[F_H][i] = 1. / (double)P.n * tm->hsum;
      break;
    case OP_CHECK_NANS: {  // default_physics.h:918-945
      bool bad = false;
      for(int d = 0; d < D; ++d) {
        double q[5] = {f[F_X + d][i], f[F_VX + d][i], f[F_VHX + d][i],
          f[F_AX + d][i], f[F_GAX + d][i]};
        for(int k = 0; k < 5; ++k)
          bad |= q[k] != q[k];
      }
      const int sc[] = {F_M, F_GPOT, F_RHO, F_P, F_E, F_DEDT, F_DUDT, F_K, F_VSIG};
      for(int k = 0; k < 9; ++k)
        bad |= f[sc[k]][i] != f[sc[k]][i];
      if(pp.evolve_u)
        bad |= f[F_U][i] != f[F_U][i];
      if(bad)
        raise_status(st, FSPH_ERR_NAN, i);
      break;
    }
    case OP_CHECK_NEGATIVITY:  // default_physics.h:953-979
      if(f[F_RHO][i] < 0 || f[F_P][i] < 0 || (pp.evolve_u && f[F_U][i] < 0))
        raise_status(st, FSPH_ERR_NEGATIVITY, i);
      break;
  }
}

cudaError_t launch_elementwise(const Launch & L, const Particles & P,
  const PhysParams & pp, int op, DevTime * t, DevStatus * st) {
  const int nb = (P.n + ELEM_THREADS - 1) / ELEM_THREADS;
  if(pp.dim == 3)
    chain(L, k_elem<3>, nb, ELEM_THREADS, 0, P, pp, op, t, st);
  else
    chain(L, k_elem<2>, nb, ELEM_THREADS, 0, P, pp, op, t, st);
  *L.counter += 1;
  return cudaGetLastError();
}

// The start of a leapfrog step, hydro/main_driver.cc:176-188: kick e (or u),
// kick v, save v_half, drift; with RANGE the range of the drifted positions is
// gathered on the way, which a pass of its own would read them again for.
template<int D, int OP, bool RANGE>
__global__ void __launch_bounds__(ELEM_THREADS) k_kick_drift(Particles P,
  const DevTime * tm, unsigned long long * range, unsigned long long * part) {
  chain_begin();
  double ** f = P.f;
  const double dt = tm->dt, s = 0.5 * dt;
  RangeAcc<D> r;
  if(RANGE)
    r.init(f[F_H][0]);
  auto drift = [&](int i, int d, double & v) {
    // (a + 0 is a but for a = -0, whose sum with v is v all the same)
    const double g = f[F_GAX + d][i];
    double a = f[F_AX + d][i];
    if((__double_as_longlong(g) << 1) != 0)
      a = add_rare(a, g);
    v = f[F_VX + d][i] + a * s;
    return f[F_X + d][i] + v * dt;
  };
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n;
      i += gridDim.x * blockDim.x) {
    if(OP == OP_KICK_DRIFT_E)
      f[F_E][i] = f[F_E][i] + 0.5 * dt * f[F_DEDT][i];
    else if(OP == OP_KICK_DRIFT_U)
      f[F_U][i] = f[F_U][i] + 0.5 * dt * f[F_DUDT][i];
    double x[3] = {0.0, 0.0, 0.0};
    for(int d = 0; d < D; ++d) {
      double v;
      x[d] = drift(i, d, v);
      f[F_VX + d][i] = v;
      f[F_VHX + d][i] = v;
      f[F_X + d][i] = x[d];
    }
    if(RANGE)
      r.add(x, f[F_H][i]);
  }
  if(RANGE) {
    // (the last particle lies in its own [x - h, x + h]: the reference's start
    // from its coordinates changes nothing, and another block may hold it)
    r.finish(range, part, nullptr);
  }
}

cudaError_t launch_kick_drift(const Launch & L, const Particles & P, const PhysParams & pp,
  int op, const DevTime * t, unsigned long long * range, unsigned long long * range_part) {
  int nb = (P.n + ELEM_THREADS - 1) / ELEM_THREADS;
  if(range && nb > RANGE_BLOCKS)
    nb = RANGE_BLOCKS;
#define KD_LAUNCH(D, OP)                                                       \
  do {                                                                         \
    if(range)                                                                  \
      chain(L, k_kick_drift<D, OP, true>, nb, ELEM_THREADS, 0, P, t, range, range_part); \
    else                                                                       \
      chain(L, k_kick_drift<D, OP, false>, nb, ELEM_THREADS, 0, P, t, nullptr, nullptr); \
  } while(0)
#define KD_OP(D)                                                               \
  do {                                                                         \
    if(op == OP_KICK_DRIFT_E)                                                  \
      KD_LAUNCH(D, OP_KICK_DRIFT_E);                                           \
    else if(op == OP_KICK_DRIFT_U)                                             \
      KD_LAUNCH(D, OP_KICK_DRIFT_U);                                           \
    else                                                                       \
      KD_LAUNCH(D, OP_KICK_DRIFT_NONE);                                        \
  } while(0)
  if(pp.dim == 3)
    KD_OP(3);
  else
    KD_OP(2);
#undef KD_OP
#undef KD_LAUNCH
  *L.counter += 1;
  return cudaGetLastError();
}

// compute_dt (default_physics.h:602-695) per particle, then the minimum.
// FP32 constants of the single-precision estimate
struct DtConst {
  float eta_kw, cfl, sig;  // eta times the kernel width, cfl, 1 + 0.6 alpha
};

// NaN / negativity from the bit pattern: integer instructions instead of
// FP64 compares, which run on this part's narrow FP64 pipe.
__device__ __forceinline__ bool bits_nan(double x) {
  return ((unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull) >
         0x7ff0000000000000ull;
}
__device__ __forceinline__ bool bits_negative(double x) {  // x < 0, not -0, not NaN
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) && (b & 0x7fffffffffffffffull) != 0 &&
         (b & 0x7fffffffffffffffull) <= 0x7ff0000000000000ull;
}

__device__ __forceinline__ bool bits_positive(double x) {  // x > 0
  const long long b = __double_as_longlong(x);
  return b > 0 && b <= 0x7ff0000000000000ll;
}

// set_adaptive_timestep (default_physics.h:761-823)
__device__ __forceinline__ void set_adaptive(const PhysParams & pp, DevTime * t) {
  double dtmin = ord_dec(t->dtmin_bits);
  double dt = t->dt;
  if(dtmin < dt)
    dt = dmin_(dtmin, dt / 2.0);
  if(dtmin > 2.0 * dt)
    dt = dt * 2.0;
  double tt = t->totaltime;
  double next = tt + dt;
  if(pp.out_screen_dt > 0) {
    if(tt == t->t_screen) {
      if(t->dt_saved > 0) dt = t->dt_saved;
      t->t_screen += pp.out_screen_dt;
    }
    if(tt + dt > t->t_screen - 0.1 * pp.out_screen_dt) {
      t->dt_saved = dt;
      next = t->t_screen;
    }
  }
  if(pp.out_scalar_dt > 0) {
    if(tt == t->t_scalar) {
      if(t->dt_saved > 0) dt = t->dt_saved;
      t->t_scalar += pp.out_scalar_dt;
    }
    if(tt + dt > t->t_scalar - 0.1 * pp.out_scalar_dt) {
      t->dt_saved = dt;
      next = dmin_(next, t->t_scalar);
    }
  }
  if(pp.out_h5data_dt > 0) {
    if(tt == t->t_h5) {
      if(t->dt_saved > 0) dt = t->dt_saved;
      t->t_h5 += pp.out_h5data_dt;
    }
    if(tt + dt > t->t_h5 - 0.1 * pp.out_h5data_dt) {
      t->dt_saved = dt;
      next = dmin_(next, t->t_h5);
    }
  }
  t->totaltime_next = next;
  t->dt = next - tt;
}

// advance_time (default_physics.h:853-860)
__device__ __forceinline__ void advance(const PhysParams & pp, DevTime * t) {
  t->iteration++;
  if(pp.adaptive)
    t->totaltime = t->totaltime_next;
  else
    t->totaltime = t->totaltime + t->dt;
}

// compute_dt's last rule: dt shrinks until the potential energy the particle
// can take up in it stays below half of its internal energy.
template<int D>
__device__ __noinline__ double limit_dt(const PhysParams & pp, double * const * f, int i,
  double eint, double dtp, DevStatus * st) {
  double gdv = 0;
  for(int d = 0; d < D; ++d)
    gdv += f[F_VX + d][i] * f[F_GAX + d][i];
  if(!(gdv != 0.0 || pp.n_eforce > 0))
    return dtp;
  const double pos[3] = {f[F_X][i], f[F_Y][i], D == 3 ? f[F_Z][i] : 0.0};
  const double epot = ext_potential<D>(pp, pos);
  int it;
  for(it = 0; it < 20; ++it) {
    double p1[3] = {0.0, 0.0, 0.0};
    for(int d = 0; d < D; ++d)
      p1[d] = pos[d] + dtp * f[F_VX + d][i];
    double delta_epot = ext_potential<D>(pp, p1) - epot;
    double delta_egrv = -dtp * gdv;
    if(delta_epot + delta_egrv < eint * 0.5)
      break;
    dtp *= 0.25;
  }
  if(it >= 20)
    raise_status(st, FSPH_ERR_DT, i);
  return dtp;
}

// CHECKS folds check_nans and check_negativity (default_physics.h:918-979)
// into the same pass, as the driver runs them back to back before dt.
// F32 evaluates the per-particle estimate of compute_dt in single precision
// (mixed-precision runs); the global minimum and the adaptive rule stay FP64.
// FINISH: the last block to arrive also runs set_adaptive_timestep and
// advance_time, which follow it in the driver's iteration.
//
// Tests against zero run on the bit patterns, and what gravity adds is left
// out where g is zero: the FP64 pipe, not HBM, bounded this pass (30
// operations a particle, 163 us at 2M particles; 101 now, HBM 52).
template<int D, bool CHECKS, bool F32, bool FINISH>
__global__ void __launch_bounds__(ELEM_THREADS) k_compute_dt(Particles P,
  PhysParams pp, DtConst c32, DevTime * tm, DevStatus * st) {
  chain_begin();
  // grid-stride: one atomic per block of a grid sized to the machine
  unsigned long long dtmin = TIME_DT_MAX;  // ordered encoding
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n;
      i += gridDim.x * blockDim.x) {
    double ** f = P.f;
    double dtp = 1e24;
    double v[3] = {0.0, 0.0, 0.0}, g[3] = {0.0, 0.0, 0.0}, acc3[3] = {0.0, 0.0, 0.0};
    bool still = true;  // g = 0, v finite: v . g = 0 and a + g = a
    for(int d = 0; d < D; ++d) {
      v[d] = f[F_VX + d][i];
      g[d] = f[F_GAX + d][i];
      acc3[d] = f[F_AX + d][i];
      still = still && (__double_as_longlong(g[d]) << 1) == 0 &&
              ((unsigned)__double2hiint(v[d]) & 0x7ff00000u) != 0x7ff00000u;
    }
    if(!still)
      for(int d = 0; d < D; ++d)
        acc3[d] = add_rare(acc3[d], g[d]);
    if(CHECKS) {
      bool bad = false;
      for(int d = 0; d < D; ++d)
        bad |= bits_nan(f[F_X + d][i]) | bits_nan(v[d]) | bits_nan(f[F_VHX + d][i]) |
               bits_nan(f[F_AX + d][i]) | bits_nan(g[d]);
      const int sc[] = {F_M, F_GPOT, F_RHO, F_P, F_E, F_DEDT, F_DUDT, F_K, F_VSIG};
      for(int k = 0; k < 9; ++k)
        bad |= bits_nan(f[sc[k]][i]);
      if(pp.evolve_u)
        bad |= bits_nan(f[F_U][i]);
      if(bad)
        raise_status(st, FSPH_ERR_NAN, i);
      if(bits_negative(f[F_RHO][i]) || bits_negative(f[F_P][i]) ||
         (pp.evolve_u && bits_negative(f[F_U][i])))
        raise_status(st, FSPH_ERR_NEGATIVITY, i);
    }
    if(F32) {
      const float tiny = 1e-24f;
      const float dx = to_f32(f[F_H][i]) / c32.eta_kw;
      float vn = 0.f, acc = 0.f;
      for(int d = 0; d < D; ++d) {
        const float vf = to_f32(v[d]), af = to_f32(acc3[d]);
        vn += vf * vf;
        acc += af * af;
      }
      const float dt_v = dx / (sqrtf(vn) + tiny);
      const float dt_a = sqrtf(dx / (sqrtf(acc) + tiny));
      const float dt_c = dx / (tiny + to_f32(f[F_VSIG][i]) * c32.sig);
      dtp = to_f64(c32.cfl * fminf(fminf(dt_v, dt_a), dt_c));
    }
    else {
      const double tiny = 1e-24, mc = 0.6;
      const double dx = f[F_H][i] / (pp.eta * pp.kw);
      double vn = 0;
      for(int d = 0; d < D; ++d)
        vn += v[d] * v[d];
      vn = sqrt(vn);
      const double dt_v = dx / (vn + tiny);
      double acc = 0;
      for(int d = 0; d < D; ++d)
        acc += acc3[d] * acc3[d];
      acc = sqrt(acc);
      const double dt_a = sqrt(dx / (acc + tiny));
      const double dt_c = dx / (tiny + f[F_VSIG][i] * (1 + mc * pp.alpha));
      dtp = pp.cfl * dmin_(dmin_(dt_v, dt_a), dt_c);
    }
    if(pp.evolve_u && pp.thermokinetic) {
      const double eint = f[F_U][i];
      if(!bits_positive(eint))
        raise_status(st, FSPH_ERR_NEG_ENERGY, i);
      // with no external potential and v . g = 0, the first test passes
      if(!still || pp.n_eforce > 0)
        dtp = limit_dt<D>(pp, f, i, eint, dtp, st);
    }
    f[F_DT][i] = dtp;
    if(!bits_nan(dtp))  // (as dmin_ would drop it)
      dtmin = umin64(dtmin, ord_enc(dtp));
  }
  // block minimum first, then one atomic per block; the last block publishes
  __shared__ unsigned long long wmin[ELEM_THREADS / 32];
  for(int o = 16; o; o >>= 1)
    dtmin = umin64(dtmin, __shfl_xor_sync(0xffffffffu, dtmin, o));
  if((threadIdx.x & 31) == 0)
    wmin[threadIdx.x >> 5] = dtmin;
  __syncthreads();
  if(threadIdx.x == 0) {
    unsigned long long m = wmin[0];
    for(int k = 1; k < ELEM_THREADS / 32; ++k)
      m = umin64(m, wmin[k]);
    atomicMin(&tm->dtmin_acc, m);
    __threadfence();
    if(atomicAdd(&tm->ticket, 1u) == gridDim.x - 1) {
      __threadfence();
      tm->dtmin_bits = atomicExch(&tm->dtmin_acc, TIME_DT_MAX);
      tm->ticket = 0u;
      if(FINISH) {
        set_adaptive(pp, tm);
        advance(pp, tm);
      }
    }
  }
}

cudaError_t launch_compute_dt(const Launch & L, const Particles & P,
  const PhysParams & pp, DevTime * t, DevStatus * st, int with_checks,
  int f32, int finish) {
  // a few blocks per SM: the per-block minima meet in one atomic each
  int nb = (P.n + ELEM_THREADS - 1) / ELEM_THREADS;
  if(nb > 152 * 8)
    nb = 152 * 8;
  const DtConst c32 = {(float)(pp.eta * pp.kw), (float)pp.cfl,
    1.f + 0.6f * (float)pp.alpha};
#define DT_LAUNCH(D, C, F, E) \
  chain(L, k_compute_dt<D, C, F, E>, nb, ELEM_THREADS, 0, P, pp, c32, t, st)
#define DT_PICK(D)                                                             \
  do {                                                                         \
    if(with_checks && finish) {                                                \
      if(f32) DT_LAUNCH(D, true, true, true); else DT_LAUNCH(D, true, false, true); \
    }                                                                          \
    else if(with_checks) {                                                     \
      if(f32) DT_LAUNCH(D, true, true, false); else DT_LAUNCH(D, true, false, false); \
    }                                                                          \
    else {                                                                     \
      if(f32) DT_LAUNCH(D, false, true, false); else DT_LAUNCH(D, false, false, false); \
    }                                                                          \
  } while(0)
  if(pp.dim == 3)
    DT_PICK(3);
  else
    DT_PICK(2);
#undef DT_PICK
#undef DT_LAUNCH
  *L.counter += 1;
  return cudaGetLastError();
}

__global__ void k_set_adaptive(PhysParams pp, DevTime * t) {
  chain_begin();
  set_adaptive(pp, t);
}

cudaError_t launch_set_adaptive_timestep(const Launch & L,
  const PhysParams & pp, DevTime * t) {
  chain(L, k_set_adaptive, 1, 1, 0, pp, t);
  *L.counter += 1;
  return cudaGetLastError();
}

__global__ void k_advance(PhysParams pp, DevTime * t) {
  chain_begin();
  advance(pp, t);
}

cudaError_t launch_advance_time(const Launch & L, const PhysParams & pp,
  DevTime * t) {
  chain(L, k_advance, 1, 1, 0, pp, t);
  *L.counter += 1;
  return cudaGetLastError();
}

// The device-side upload and download: the arrays along y, 2048 words of one
// per block.  Memory-bound for large n; for small n it stands in for a copy or
// a clear per array (34 for an upload), each a command of 2 to 5 us.  Upload,
// ten iterations and download, copies per array -> this: 2k particles 2.29 ->
// 2.10 ms, 32k 2.04 -> 1.78, 50k 2.65 -> 2.40, 2M 26.20 -> 25.85, 17M with two
// iterations 137.1 -> 136.3; 32 members' downloads and eight steps 15.5 -> 11.9.
#define MOVE_THREADS 256
#define MOVE_WORDS (MOVE_THREADS * 8)
__global__ void __launch_bounds__(MOVE_THREADS) k_move(Moves m, int n,
  const DevStatus * status, DevTime * time, DevTime t0, DevStatus * clear) {
  chain_begin();
  if(status && status->code)
    return;
  const int t = threadIdx.x;
  if(time && blockIdx.x == 0 && blockIdx.y == 0 && t == 0) {
    *time = t0;
    *clear = DevStatus{};
  }
  typedef unsigned long long word;
  const word * src = (const word *)m.src[blockIdx.y];
  word * dst = (word *)m.dst[blockIdx.y];
  const int i0 = blockIdx.x * MOVE_WORDS;
  if((((size_t)src | (size_t)dst) & 15) == 0) {
    ulonglong2 v[4];
#pragma unroll
    for(int k = 0; k < 4; ++k) {
      const int i = i0 + 2 * (k * MOVE_THREADS + t);
      v[k] = make_ulonglong2(0, 0);
      if(src && i + 1 < n)
        v[k] = *(const ulonglong2 *)(src + i);
      else if(src && i < n)
        v[k].x = src[i];
    }
#pragma unroll
    for(int k = 0; k < 4; ++k) {
      const int i = i0 + 2 * (k * MOVE_THREADS + t);
      if(i + 1 < n)
        *(ulonglong2 *)(dst + i) = v[k];
      else if(i < n)
        dst[i] = v[k].x;
    }
  }
  else {
    word v[8];
#pragma unroll
    for(int k = 0; k < 8; ++k) {
      const int i = i0 + k * MOVE_THREADS + t;
      v[k] = src && i < n ? src[i] : 0;
    }
#pragma unroll
    for(int k = 0; k < 8; ++k) {
      const int i = i0 + k * MOVE_THREADS + t;
      if(i < n)
        dst[i] = v[k];
    }
  }
}

cudaError_t launch_move(const Launch & L, const Moves & m, int n, const DevStatus * status,
  DevTime * time, const DevTime & t0, DevStatus * clear) {
  if(m.count == 0 || n <= 0)
    return cudaSuccess;
  chain(L, k_move, dim3((n - 1) / MOVE_WORDS + 1, m.count), MOVE_THREADS, 0, m, n, status,
    time, t0, clear);
  *L.counter += 1;
  return cudaGetLastError();
}

// Deterministic sum of h (fixed two-level order) for the averaged h.
__global__ void __launch_bounds__(1024) k_hsum(Particles P, DevTime * t) {
  __shared__ double part[1024];
  double s = 0;
  for(int i = threadIdx.x; i < P.n; i += 1024)
    s += P.f[F_H][i];
  part[threadIdx.x] = s;
  __syncthreads();
  for(int o = 512; o; o >>= 1) {
    if(threadIdx.x < o)
      part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  if(threadIdx.x == 0)
    t->hsum = part[0];
}

cudaError_t launch_hsum(const Launch & L, const Particles & P, DevTime * t) {
  k_hsum<<<1, 1024, 0, L.stream>>>(P, t);
  *L.counter += 1;
  return cudaGetLastError();
}

// Conserved totals (analysis.h:56-214): mass, energy, momentum (3),
// angular momentum (3).  Two passes in a fixed order (deterministic):
// CONS_BLOCKS block partials, then one block adds them up.
__global__ void __launch_bounds__(256) k_conserved_part(Particles P,
  PhysParams pp, double * part_out, long long nreal) {
  __shared__ double part[8][256];
  double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int D = pp.dim;
  for(int i = blockIdx.x * 256 + threadIdx.x; i < P.n; i += gridDim.x * 256) {
    if(P.id[i] >= nreal)  // periodic copies (WALL) are not counted
      continue;
    double m = P.f[F_M][i];
    double x[3] = {P.f[F_X][i], P.f[F_Y][i], D == 3 ? P.f[F_Z][i] : 0.0};
    double v[3] = {P.f[F_VX][i], P.f[F_VY][i], D == 3 ? P.f[F_VZ][i] : 0.0};
    s[0] += m;
    if(pp.thermokinetic)
      s[1] += m * P.f[F_E][i];
    else {
      const double epot = D == 3 ? ext_potential<3>(pp, x) : ext_potential<2>(pp, x);
      s[1] += m * (.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) + P.f[F_U][i] + epot);
    }
    s[1] += .5 * m * P.f[F_GPOT][i];
    for(int d = 0; d < 3; ++d)
      s[2 + d] += m * v[d];
    s[5] += m * (x[1] * v[2] - x[2] * v[1]);
    s[6] += m * (x[2] * v[0] - x[0] * v[2]);
    s[7] += m * (x[0] * v[1] - x[1] * v[0]);
  }
  for(int k = 0; k < 8; ++k)
    part[k][threadIdx.x] = s[k];
  __syncthreads();
  for(int o = 128; o; o >>= 1) {
    if(threadIdx.x < o)
      for(int k = 0; k < 8; ++k)
        part[k][threadIdx.x] += part[k][threadIdx.x + o];
    __syncthreads();
  }
  if(threadIdx.x < 8)
    part_out[8 + 8 * blockIdx.x + threadIdx.x] = part[threadIdx.x][0];
}

__global__ void __launch_bounds__(256) k_conserved_final(double * buf, int nb) {
  __shared__ double part[8][256];
  double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for(int b = threadIdx.x; b < nb; b += 256)
    for(int k = 0; k < 8; ++k)
      s[k] += buf[8 + 8 * b + k];
  for(int k = 0; k < 8; ++k)
    part[k][threadIdx.x] = s[k];
  __syncthreads();
  for(int o = 128; o; o >>= 1) {
    if(threadIdx.x < o)
      for(int k = 0; k < 8; ++k)
        part[k][threadIdx.x] += part[k][threadIdx.x + o];
    __syncthreads();
  }
  if(threadIdx.x < 8)
    buf[threadIdx.x] = part[threadIdx.x][0];
}

cudaError_t launch_conserved(const Launch & L, const Particles & P,
  const PhysParams & pp, double * out8, long long nreal) {
  // out8 holds 8 totals followed by 8 * CONS_BLOCKS partials
  const int nb = P.n < 256 * CONS_BLOCKS ? (P.n + 255) / 256 : CONS_BLOCKS;
  k_conserved_part<<<nb > 0 ? nb : 1, 256, 0, L.stream>>>(P, pp, out8, nreal);
  k_conserved_final<<<1, 256, 0, L.stream>>>(out8, nb > 0 ? nb : 1);
  *L.counter += 2;
  return cudaGetLastError();
}

}  // namespace fsph
