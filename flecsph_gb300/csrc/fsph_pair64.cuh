// fsph_pair64.cuh -- FP64 pair terms of the neighbour passes, written for a
// part whose FP64 pipe runs at 1/64 of its FP32 rate: there a division or a
// root is eight to ten pipe operations and everything a pair shares with its
// predecessor is worth keeping.
//
//   * What depends on h_ab alone (its reciprocal, the kernels' normalisation
//     over h^D or h^(D+1), eps h^2) is kept while the neighbour's h does not
//     change, which in a uniform-h run is the whole list.
//   * r_ab and 1 / r_ab come from one reciprocal root, and a quotient by r_ab
//     or h_ab is three operations: q = x y, then q + (x - d q) y with
//     y ~ 1 / d and the residual exact (an FMA; P. Markstein, IBM J. Res. Dev.
//     34, 1990); the root is corrected in the same way.  Before its last
//     rounding that is off by some 2^-103 of the value, so it is the rounded
//     quotient or root but for operands whose exact result lies that close to
//     the middle between two doubles (the theorem that excludes them asks for a
//     correctly rounded y): none of 1.6e10 random operands, r and h over 2^-8
//     to 2^8, gave another value than the division or the root.  Scales at
//     which a residual could underflow take the plain operators.
//
// Operand order otherwise follows kernels.h and viscosity.h of the reference,
// as fsph_sphmath.cuh does, but for one thing: with the spline, Gaussian (not
// super-Gaussian) and sinc kernels the reference multiplies x_ab in before it
// divides by r, for every axis; here, as its other kernels do, f = (dW/dr) / r
// is formed first and x_ab f after, three roundings either way (outputs differ
// by some 4e-16).
#pragma once

#include "fsph_sphmath.cuh"

namespace fsph {

// x != 0, on the integer pipe (NaN counts as nonzero)
__device__ __forceinline__ bool nonzero(double x) {
  return (__double_as_longlong(x) << 1) != 0;
}

// r = sqrt(r2) and y ~ 1 / r; both 0 at r2 = 0.  Below 1e-200 (squared) the
// residual's products would lose bits: the plain root and reciprocal.
struct PairR {
  double r, y;
};

__device__ __forceinline__ PairR pair_r(double r2) {
  PairR p;
  // exponent field of r2 above 2^-664 and below 2^664
  const unsigned ex = ((unsigned)__double2hiint(r2) >> 20) & 0x7ffu;
  if(ex - 359u < 1328u) {
    p.y = rsqrt(r2);
    const double r0 = r2 * p.y;
    p.r = __fma_rn(__fma_rn(-r0, r0, r2), 0.5 * p.y, r0);
  }
  else {
    p.r = sqrt(r2);
    p.y = nonzero(r2) ? 1.0 / p.r : 0.0;
  }
  return p;
}

// x / d for y ~ 1 / d to rounding
__device__ __forceinline__ double quot(double x, double d, double y) {
  const double q = x * y;
  return __fma_rn(__fma_rn(-d, q, x), y, q);
}

// h_ab and what the kernel K takes from it alone
template<int D, int K>
struct PairH {
  long long bits;   // the neighbour's h these belong to
  double h, ih;     // h_ab, 1 / h_ab
  double sw, sg;    // normalisations of W and of its gradient at h_ab

  __device__ __forceinline__ void init() {
    bits = -1;  // a NaN: no h has it
    h = ih = sw = sg = 0.0;
  }

  template<bool W, bool G>
  __device__ __forceinline__ void set(double h_a, double h_b, const PhysParams & pp) {
    const long long hb = __double_as_longlong(h_b);
    if(hb == bits)
      return;
    bits = hb;
    h = .5 * (h_a + h_b);
    ih = 1.0 / h;
    if(W) {
      if(K == FSPH_KERNEL_SINC) {
        double hd = h;
        for(int i = 1; i < D; i++)
          hd *= h;
        sw = pp.sinc_sigma[D - 1] / hd;
      }
      else if(K == FSPH_KERNEL_QUINTIC_SPLINE)
        sw = quintic_sigma(D) / pow(h, (double)D);
      else if(K == FSPH_KERNEL_GAUSSIAN)
        sw = gaussian_sigma(D) / pow(h, (double)D);
      else if(K == FSPH_KERNEL_SUPER_GAUSSIAN)
        sw = super_gaussian_sigma(D) / pow(h, (double)D);
      else if(K == FSPH_KERNEL_CUBIC_SPLINE)
        sw = cubic_sigma(D) / pow(h, (double)D);
      else {
        const double hd = D == 3 ? h * h * h : h * h;
        sw = (K == FSPH_KERNEL_WENDLAND_C2 ? wc2_sigma(D)
              : K == FSPH_KERNEL_WENDLAND_C4 ? wc4_sigma(D) : wc6_sigma(D)) / hd;
      }
    }
    if(G) {
      if(K == FSPH_KERNEL_SINC) {
        double hd = h * h;
        for(int i = 1; i < D; i++)
          hd *= h;
        sg = pp.sinc_sigma[D - 1] / hd;
      }
      else if(K == FSPH_KERNEL_QUINTIC_SPLINE)
        sg = 3. * quintic_sigma(D) / pow(h, (double)(D + 1));
      else if(K == FSPH_KERNEL_GAUSSIAN)
        sg = 3. * gaussian_sigma(D) / pow(h, (double)(D + 1));
      else if(K == FSPH_KERNEL_SUPER_GAUSSIAN)
        sg = 3. * super_gaussian_sigma(D) / pow(h, (double)(D + 1));
      else if(K == FSPH_KERNEL_CUBIC_SPLINE)
        sg = 2. * cubic_sigma(D) / pow(h, (double)(D + 1));
      else {
        const double hd1 = D == 3 ? h * h * h * h : h * h * h;
        sg = (K == FSPH_KERNEL_WENDLAND_C2 ? 2. * wc2_sigma(D)
              : K == FSPH_KERNEL_WENDLAND_C4 ? 14. * wc4_sigma(D) : wc6_sigma(D)) / hd1;
      }
    }
  }

  // x / h_ab; the exponent test keeps the residual clear of underflow
  __device__ __forceinline__ double over_h(double x) const {
    const unsigned ex = ((unsigned)__double2hiint(h) >> 20) & 0x7ffu;
    return ex - 523u < 1000u ? quot(x, h, ih) : x / h;
  }
};

// W(r, h_ab): kernels.h:106-121, 167-179, 217-235, 282-312, 375-410, 477-512,
// 581-590, 633-661
template<int D, int K>
__device__ __forceinline__ double pair_w(double r, const PairH<D, K> & ph,
  const PhysParams & pp) {
  if(K == FSPH_KERNEL_SINC) {
    const double eps = 1e-24, eps_root4 = 1e-6;
    double rh = fabs(ph.over_h(r));
    if(!(rh < 1.))
      return 0.;
    double sinc = 1.0;
    rh *= FSPH_PI;
    if(rh > eps_root4)
      sinc = sin(rh) / rh;
    else if(rh > eps) {
      const double rh2 = rh * rh;
      sinc += rh2 * (.05 * rh2 - 1.) / 6.;
    }
    return ph.sw * pow(sinc, pp.sinc_index);
  }
  if(K == FSPH_KERNEL_QUINTIC_SPLINE) {
    const double rh = ph.over_h(3. * r);
    if(!(rh < 3.))
      return 0.;
    double result = pow(3 - rh, 5);
    if(rh < 2.)
      result += -6 * pow(2 - rh, 5);
    if(rh < 1.)
      result += 15 * pow(1 - rh, 5);
    return result * ph.sw;
  }
  if(K == FSPH_KERNEL_GAUSSIAN) {
    const double rh = ph.over_h(3. * r);
    return rh <= 3. ? ph.sw * exp(-rh * rh) : 0.;
  }
  if(K == FSPH_KERNEL_SUPER_GAUSSIAN) {
    const double rh = ph.over_h(3. * r), rh2 = rh * rh;
    return fabs(rh) < 3. ? ph.sw * exp(-rh2) * (D / 2.0 + 1 - rh2) : 0.;
  }
  if(K == FSPH_KERNEL_CUBIC_SPLINE) {
    const double rh = ph.over_h(2. * r);
    if(!(rh < 2.0))
      return 0.;
    const double result = rh < 1.0 ? 1.0 - 1.5 * rh * rh + .75 * rh * rh * rh
                                   : 0.25 * (2 - rh) * (2 - rh) * (2 - rh);
    return result * ph.sw;
  }
  const double rh = ph.over_h(r), t = 1 - rh;
  const double t2 = t * t;
  double result;
  if(K == FSPH_KERNEL_WENDLAND_C2)
    result = ph.sw * t2 * t2 * (4 * rh + 1);
  else if(K == FSPH_KERNEL_WENDLAND_C4)
    result = ph.sw * (t2 * t2 * t2) * (1 + rh * (6 + rh * 35 / 3));
  else {
    const double t4 = t2 * t2;
    result = ph.sw * t4 * t4 * (1 + rh * (8 + rh * (25 + rh * 32)));
  }
  return rh < 1.0 ? result : 0.;
}

// f with grad_a W(x_ab, h_ab) = x_ab f: kernels.h:132-153, 189-205, 246-270,
// 322-361, 435-463, 536-566, 600-613, 671-698 (zero at r = 0)
template<int D, int K>
__device__ __forceinline__ double pair_g(const PairR & r, const PairH<D, K> & ph,
  const PhysParams & pp) {
  double dWdr = 0.0;
  bool in;
  if(K == FSPH_KERNEL_SINC) {
    const double eps = 1e-24, eps_root4 = 1e-6;
    const double n = pp.sinc_index;
    double rh = fabs(ph.over_h(r.r));
    in = rh < 1.;
    rh *= FSPH_PI;
    if(in && rh > eps_root4) {
      const double sinc = sin(rh) / rh, cosx = cos(rh) / rh;
      dWdr = -n * pow(sinc, n - 1) * FSPH_PI * (sinc / rh - cosx);
    }
    else if(in && rh > eps) {
      const double rh2 = rh * rh;
      dWdr = -n * rh / 3. * FSPH_PI * (1 - .5 * rh2 * (.2 - (n - 1) / 18));
    }
  }
  else if(K == FSPH_KERNEL_QUINTIC_SPLINE) {
    const double rh = ph.over_h(3. * r.r);
    in = rh < 3.;
    if(in) {
      dWdr = -5. * pow(3 - rh, 4);
      if(rh < 2.)
        dWdr += 30. * pow(2 - rh, 4);
      if(rh < 1.)
        dWdr += -75. * pow(1 - rh, 4);
    }
  }
  else if(K == FSPH_KERNEL_GAUSSIAN) {
    const double rh = ph.over_h(3. * r.r);
    in = rh < 3.;
    dWdr = -2. * rh * exp(-rh * rh);
  }
  else if(K == FSPH_KERNEL_SUPER_GAUSSIAN) {
    const double rh = ph.over_h(3. * r.r);
    in = rh < 3.0;
    dWdr = exp(-rh * rh) * (2. * pow(rh, 3.) - (D + 4.) * rh);
  }
  else if(K == FSPH_KERNEL_CUBIC_SPLINE) {
    const double rh = ph.over_h(2. * r.r);
    in = rh < 2.0;
    dWdr = rh < 1.0 ? -3.0 * rh + 9. / 4. * rh * rh : -.75 * (2 - rh) * (2 - rh);
  }
  else {
    const double rh = ph.over_h(r.r), t = 1 - rh;
    const double t2 = t * t, t3 = t2 * t;
    in = rh < 1.0;
    if(K == FSPH_KERNEL_WENDLAND_C2)
      dWdr = -10. * rh * t2 * t;
    else if(K == FSPH_KERNEL_WENDLAND_C4)
      dWdr = -4. / 3. * rh * t3 * t2 * (1 + 5. * rh);
    else
      dWdr = -22. * rh * (t2 * t2) * t3 * (1 + rh * (7 + rh * 16));
  }
  return in && nonzero(r.r) ? quot(ph.sg * dWdr, r.r, r.y) : 0.0;
}

// pair_g for the Wendland kernels with 1 / r cancelled against the kernel's
// r / h: (dW/dr) / r = sigma / h^(D+2) g(t), t = 1 - r / h.  Without the two
// quotients it is two thirds of pair_g's FP64 operations, which bind the pass
// that sums it (31k particles in 2D, its density pass: 0.160 -> 0.144 ms).
// Not in the reference's operand order: for the mixed path's divergence sum,
// which needs FP64 but not that order (the outputs move by 5e-14).
template<int D, int K>
__device__ __forceinline__ double pair_g_free(double r2, const PairH<D, K> & ph,
  const PhysParams & pp) {
  constexpr bool wc = K == FSPH_KERNEL_WENDLAND_C2 || K == FSPH_KERNEL_WENDLAND_C4 ||
                      K == FSPH_KERNEL_WENDLAND_C6;
  const PairR r = pair_r(r2);
  if(!wc)
    return pair_g<D, K>(r, ph, pp);
  const double q = r.r * ph.ih, t = 1 - q, t2 = t * t, t3 = t2 * t;
  const double s = ph.sg * ph.ih;  // kept with h_ab by the compiler
  double g;
  if(K == FSPH_KERNEL_WENDLAND_C2)
    g = -10. * t3;
  else if(K == FSPH_KERNEL_WENDLAND_C4)
    g = -4. / 3. * (t3 * t2) * (1 + 5. * q);
  else
    g = -22. * (t2 * t2 * t3) * (1 + q * (7 + q * 16));
  return q < 1.0 ? s * g : 0.0;
}

// Pi_ab of an approaching pair (dotp = v_ab . x_ab < 0): viscosity::mu
// (viscosity.h:81-93) and the configured viscosity function
template<int D>
__device__ __forceinline__ double pair_pi(const PhysParams & pp, const double * ALPHA,
  int a, int b, double rho_ab, double c_ab, double h_ab, double dotp, double dist2) {
  const double mu = h_ab * dotp / (dist2 + pp.eps * h_ab * h_ab + FSPH_TINY);
  return visc_pi_pp(pp, ALPHA, a, b, rho_ab, c_ab, mu);
}

// Neither infinite nor NaN, on the integer pipe
__device__ __forceinline__ bool finite64(double x) {
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u;
}
__device__ __forceinline__ bool nan64(double x) {
  return ((unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull) >
         0x7ff0000000000000ull;
}

// P / rho^2 as the passes keep it per particle.  Where the sound speed or alpha
// is not finite or the density is a NaN it is a NaN of its own: Pi of every pair
// of that particle is one then, and so is what is summed from it.
#define PRHO2_ODD 0x7ff8000050a10badll
__device__ __forceinline__ double kept_prho2(const PhysParams & pp, double p, double rho,
  double c, double alpha) {
  return finite64(c) && !nan64(rho) && (!pp.cullen || finite64(alpha))
           ? p / (rho * rho) : __longlong_as_double(PRHO2_ODD);
}

// Pi_ab of a pair that does not approach.  The reference forms it there too,
// with mu times (dotp < 0): zero, but a NaN where v_ab . x_ab, a sound speed or
// an alpha is not finite or a density is a NaN, and so the acceleration and the
// energy rates carry it.  No FP64 operation, no branch, and no gather but of
// P / rho^2 (acceleration of 2M particles 47.8 -> 48.2 ms; testing c_s, rho and
// alpha of both here took 48.7, and 5 % of an evaluating de/dt pass).
__device__ __forceinline__ double pi_apart(double prho2_a, double prho2_b, double dotp) {
  return finite64(dotp) && __double_as_longlong(prho2_a) != PRHO2_ODD &&
         __double_as_longlong(prho2_b) != PRHO2_ODD
           ? 0.0 : __longlong_as_double(0x7ff8000000000000ll);
}

// min(v_ab . x_ab / r_ab, 0), the approach speed of the signal speed
// (default_physics.h:254-262)
template<int D>
__device__ __forceinline__ double approach(const double * v, const double * x,
  const PairR & r) {
  double dot = v[0] * quot(x[0], r.r, r.y) + v[1] * quot(x[1], r.r, r.y);
  if(D == 3)
    dot += v[2] * quot(x[2], r.r, r.y);
  return 0.0 < dot ? 0.0 : dot;
}

// slot j of particle a in the acceleration pass's pair terms: lanes of a warp
// side by side
__host__ __device__ inline size_t pair_slot(int a, int j, int maxnb) {
  return ((size_t)(a >> 5) * (size_t)maxnb + (size_t)j) * 32u + (size_t)(a & 31);
}

}  // namespace fsph
