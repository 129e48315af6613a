// fsph_sphmath.cuh -- FP64 device restatement of the reference's SPH
// kernels, viscosity and EOS.  Every expression keeps the reference's
// operand order; the including translation units are compiled with
// -fmad=false, so each operation rounds exactly as the reference's does.
#pragma once

#include "fsph_internal.cuh"
#include "fsph_eforce.cuh"

namespace fsph {

// kernels::TINY (include/physics/kernels.h:64) and viscosity::TINY
// (include/physics/viscosity.h:36): 1e10 * DBL_MIN.
#define FSPH_TINY (1e10 * 2.2250738585072014e-308)
#define FSPH_PI 3.14159265358979323846

// Normalisations sigma[D-1] (kernels.h:40-46)
__device__ __forceinline__ double cubic_sigma(int D) {
  return D == 1 ? 4. / 3. : (D == 2 ? 40. / (7. * FSPH_PI) : 8. / FSPH_PI);
}
__device__ __forceinline__ double wc2_sigma(int D) {
  return D == 1 ? 1.25 : (D == 2 ? 7. / FSPH_PI : 21. / (2. * FSPH_PI));
}
__device__ __forceinline__ double wc4_sigma(int D) {
  return D == 1 ? 1.5 : (D == 2 ? 9. / FSPH_PI : 495. / (32. * FSPH_PI));
}
__device__ __forceinline__ double wc6_sigma(int D) {
  return D == 1 ? 55. / 32.
                : (D == 2 ? 78. / (7. * FSPH_PI) : 1365. / (64. * FSPH_PI));
}
__device__ __forceinline__ double quintic_sigma(int D) {
  return D == 1 ? 1. / 40.
                : (D == 2 ? 63. / (478. * FSPH_PI) : 81. / (359. * FSPH_PI));
}
// kernels.h:47-55 gives these as long-double literals; the doubles they
// round to, exactly
__device__ __forceinline__ double gaussian_sigma(int D) {
  return D == 1 ? 0x1.b14ea2d5440dap+0
                : (D == 2 ? 0x1.6ebcfdd1ce67cp+1 : 0x1.36768dfdddb6bp+2);
}
__device__ __forceinline__ double super_gaussian_sigma(int D) {
  return D == 1 ? 0x1.b13778577c0efp+0
                : (D == 2 ? 0x1.6e54d13f8aff2p+1 : 0x1.354cb7a91e8ccp+2);
}

// viscosity_function<visc_constant> (viscosity.h:128-137)
__device__ __forceinline__ double visc_pi(double alpha, double beta,
  double rho_ab, double c_ab, double mu_ab) {
  return (-alpha * c_ab + beta * mu_ab) * mu_ab / rho_ab;
}

// sph_artificial_viscosity for the configured viscosity: visc_constant
// ignores alpha_ab (viscosity.h:128-137); visc_cullen is
// viscosity_function<visc_cullen> (viscosity.h:150-158) with
// alpha_ab = (alpha_a + alpha_b) / 2 (default_physics.h:388).
__device__ __forceinline__ double visc_pi_pp(const PhysParams & pp,
  const double * ALPHA, int a, int b, double rho_ab, double c_ab, double mu_ab) {
  if(pp.cullen) {
    const double alpha_ab = .5 * (ALPHA[a] + ALPHA[b]);
    return -alpha_ab * (c_ab - 2.0 * mu_ab) * mu_ab / rho_ab;
  }
  return visc_pi(pp.alpha, pp.beta, rho_ab, c_ab, mu_ab);
}

// eos_t<wd> (eos/eos.h:225-315): pressure function constants and the
// pressure, sound speed and internal energy of cold degenerate matter
#define FSPH_WD_A 6.00233181e22       // [dynes/cm^2]
#define FSPH_WD_B 9.73932099e5        // [moles/cm^3]
#define FSPH_C_LIGHT_CGS 2.99792458e10

__device__ __forceinline__ double wd_internal_energy(double rho, double Ye) {
  const double x = cbrt(rho * Ye / FSPH_WD_B), x2 = x * x, x3 = x * x * x;
  return FSPH_WD_A / rho * (8. * x3 * (sqrt(x2 + 1.) - 1.) -
                            (x * (2. * x2 - 3.) * sqrt(x2 + 1.) + 3. * asinh(x)));
}

// eos_t<>::compute_pressure + compute_soundspeed for every eos_type
// (eos/eos.h:102-119 polytropic, 166-183 ideal, 262-289 wd, 362-392 ppt,
// 425-431 no_eos).  P_old and cs_old are returned by eos_no_eos.
__device__ __forceinline__ void eos_p_cs(const PhysParams & pp, double rho,
  double u, double K, double Ye, double P_old, double cs_old, double & P,
  double & cs) {
  // The sound speed of a polytrope, sqrt(K gamma rho^(gamma - 1)), is taken
  // as sqrt(gamma P / rho): one FP64 pow per particle instead of two (pow
  // is long on this part's FP64 pipe), equal to rounding.
  const double g = pp.gamma;
  if(pp.eos == FSPH_EOS_POLYTROPIC) {
    P = K * pow(rho, g);
    cs = sqrt(g * P / rho);
  }
  else if(pp.eos == FSPH_EOS_WD) {
    // both from one x = (rho Ye / B)^(1/3)
    const double x = cbrt(rho * Ye / FSPH_WD_B), x2 = x * x;
    P = FSPH_WD_A * (x * (2. * x2 - 3.) * sqrt(x2 + 1.) + 3. * asinh(x));
    const double numer = (1. + x2) * (6. * x2 - 3.) + 3. + x2 * (2. * x2 - 3.);
    const double denom = (1. + x2) * (6. * x2 + 1.) - 1. + x2 * (2. * x2 + 1.);
    cs = sqrt(numer / (3. * denom)) * FSPH_C_LIGHT_CGS;
  }
  else if(pp.eos == FSPH_EOS_PPT) {
    // K2 = K1 rho_thr^(gamma - gamma2): the power is a constant of the run
    if(rho < pp.rho_thr) {
      P = K * pow(rho, g);
      cs = sqrt(g * P / rho);
    }
    else {
      P = K * pp.ppt_k2 * pow(rho, pp.gamma2);
      cs = sqrt(pp.gamma2 * P / rho);
    }
  }
  else if(pp.eos == FSPH_EOS_NO_EOS) {
    P = P_old;
    cs = cs_old;
  }
  else {
    P = (g - 1.) * rho * u;
    cs = sqrt(g * (g - 1.) * u);
  }
}

__device__ __forceinline__ void raise_status(DevStatus * st, int code,
  long long index) {
  if(atomicCAS(&st->code, 0, code) == 0)
    st->index = index;
}

}  // namespace fsph
