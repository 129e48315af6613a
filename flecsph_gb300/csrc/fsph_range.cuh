// fsph_range.cuh -- the bounding range of a particle set, as a block-wise
// accumulation that any pass over the positions can carry.
#pragma once

#include "fsph_internal.cuh"

namespace fsph {

// ordered integer encoding of a double, and back
__device__ __forceinline__ unsigned long long ord_enc(double x) {
  long long b = __double_as_longlong(x);
  return b < 0 ? ~(unsigned long long)b
               : ((unsigned long long)b | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord_dec(unsigned long long u) {
  return (u & 0x8000000000000000ull)
           ? __longlong_as_double((long long)(u & 0x7fffffffffffffffull))
           : __longlong_as_double((long long)~u);
}

__device__ __forceinline__ unsigned long long umin64(unsigned long long a,
  unsigned long long b) {
  return b < a ? b : a;
}

// body_system::mpi_compute_range (mpisph/bodies_system.h:231-268): the
// bounding box of [x - h, x + h] over all particles, initialised from the
// last particle's coordinates.  min/max are exact in any order.
//
// The comparisons run on the ordered encodings (the integer pipe).  Particles
// whose h is that of particle 0 only enter the extremes of x: x - h is
// monotonic in x under rounding, so h is subtracted from the extremes at the
// end; the others are widened one by one.  In an equal-h run no particle then
// costs the FP64 pipe anything (six additions per particle, 20 us of the
// 2M-particle pass, before).
template<int dim>
struct RangeAcc {
  double h0;
  // minima: x of particles with h0 [0..2], h [6], widened lo [8..10]; the
  // complements of the maxima beside them in [3..5], [7], [11..13]
  unsigned long long v[14];

  __device__ __forceinline__ void init(double h_first) {
    h0 = h_first;
    for(int k = 0; k < 14; ++k)
      v[k] = ~0ull;
  }
  __device__ __forceinline__ void add(const double * x, double h) {
    const unsigned long long eh = ord_enc(h);
    v[6] = umin64(v[6], eh);
    v[7] = umin64(v[7], ~eh);
    if(__double_as_longlong(h) == __double_as_longlong(h0))
      for(int d = 0; d < dim; ++d) {
        const unsigned long long e = ord_enc(x[d]);
        v[d] = umin64(v[d], e);
        v[3 + d] = umin64(v[3 + d], ~e);
      }
    else
      for(int d = 0; d < dim; ++d) {
        const double2 w = widen_rare(x[d], h);
        v[8 + d] = umin64(v[8 + d], ord_enc(w.x));
        v[11 + d] = umin64(v[11 + d], ~ord_enc(w.y));
      }
  }

  // All threads of a 256-thread block: the block's extremes to `part`, and by
  // the last block to arrive those of all blocks to range[0..7].  `last`: the
  // last particle's coordinates, or null.
  __device__ __forceinline__ void finish(unsigned long long * range,
    unsigned long long * part, const double * last) {
    __shared__ unsigned long long red[8][14];
    __shared__ bool s_final;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    for(int k = 0; k < 14; ++k)
      for(int o = 16; o; o >>= 1)
        v[k] = umin64(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    if(lane == 0)
      for(int k = 0; k < 14; ++k)
        red[w][k] = v[k];
    __syncthreads();
    unsigned long long m = ~0ull;
    if(t < 14) {
      m = red[0][t];
      for(int q = 1; q < (int)(blockDim.x >> 5); ++q)
        m = umin64(m, red[q][t]);
    }
    __syncthreads();
    if(t < 14)
      red[0][t] = m;
    __syncthreads();
    if(t < 8) {
      // slot t: lo[0..2], the complements of hi[3..5], h[6..7]; the extremes of
      // x widen by their common h here
      unsigned long long x = m;
      if(t < 6) {
        x = red[0][8 + t];
        if(m != ~0ull)
          x = umin64(x, t < 3 ? ord_enc(ord_dec(m) - h0) : ~ord_enc(ord_dec(~m) + h0));
      }
      __stcg(part + 8 * blockIdx.x + t, x);
      __threadfence();
    }
    __syncthreads();
    if(t == 0)
      s_final = atomicAdd((unsigned *)(range + RANGE_TICKET), 1u) == gridDim.x - 1;
    __syncthreads();
    if(!s_final)
      return;
    __threadfence();
    // slot t & 7 over the blocks, 32 threads each
    unsigned long long x = ~0ull;
    for(unsigned b = t >> 3; b < gridDim.x; b += blockDim.x >> 3)
      x = umin64(x, __ldcg(part + 8 * b + (t & 7)));
    x = umin64(x, __shfl_xor_sync(0xffffffffu, x, 8));
    x = umin64(x, __shfl_xor_sync(0xffffffffu, x, 16));
    if(lane < 8)
      red[w][lane] = x;
    __syncthreads();
    if(t < 8) {
      x = red[0][t];
      for(int q = 1; q < (int)(blockDim.x >> 5); ++q)
        x = umin64(x, red[q][t]);
      const int d = t < 3 ? t : t - 3;
      if(last && t < 6 && d < dim) {
        const unsigned long long e = ord_enc(last[d]);
        x = umin64(x, t < 3 ? e : ~e);
      }
      if(t >= 6 || d < dim)
        range[t] = (t < 3 || t == 6) ? x : ~x;
    }
    if(t == 0)
      *(unsigned *)(range + RANGE_TICKET) = 0u;
  }
};

}  // namespace fsph
