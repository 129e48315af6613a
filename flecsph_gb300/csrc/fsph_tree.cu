// fsph_tree.cu -- range, Morton keys, radix sort, permutation, binary radix
// tree, particle groups and neighbour lists.
//
// Compiled with -fmad=false: the range, the key quantisation and the
// neighbour predicate must round exactly like the reference's FP64 code
// (no fused multiply-add), so keys, sort order and neighbour sets are
// bit-identical to the CPU reference.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "fsph_internal.cuh"
#include "fsph_range.cuh"

namespace fsph {

namespace cg = cooperative_groups;

#define FULL 0xffffffffu

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// ---------------------------------------------------------------- range --
template<int dim>
__global__ void __launch_bounds__(256) k_range(Particles P, unsigned long long * range,
  unsigned long long * part) {
  chain_begin();
  const double * H = P.f[F_H];
  RangeAcc<dim> r;
  r.init(H[0]);
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n;
      i += gridDim.x * blockDim.x) {
    double x[3] = {0.0, 0.0, 0.0};
    for(int d = 0; d < dim; ++d)
      x[d] = P.f[F_X + d][i];
    r.add(x, H[i]);
  }
  double last[3] = {0.0, 0.0, 0.0};
  for(int d = 0; d < dim; ++d)
    last[d] = P.f[F_X + d][P.n - 1];
  r.finish(range, part, last);
}

// Morton key, morton_curve_u(range, p) (filling_curve.h:503-525): bit i of
// the quantised coordinate j goes to bit D*i + j, above them the depth
// marker bit at D*max_depth.
__device__ __forceinline__ unsigned long long spread3(unsigned long long x) {
  x &= 0x1fffffull;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}
__device__ __forceinline__ unsigned long long spread2(unsigned long long x) {
  x &= 0x7fffffffull;
  x = (x | x << 16) & 0x0000ffff0000ffffull;
  x = (x | x << 8) & 0x00ff00ff00ff00ffull;
  x = (x | x << 4) & 0x0f0f0f0f0f0f0f0full;
  x = (x | x << 2) & 0x3333333333333333ull;
  x = (x | x << 1) & 0x5555555555555555ull;
  return x;
}

// The reference quantises fl(t / scale) * 2^md, t = x - min.  t times the
// reciprocal, scaled by a further 2^20, gives that value in fixed point to a
// few units of its 20 fraction bits; only a fraction within KEY_MARGIN of an
// integer leaves the integer part open, and there the correctly rounded
// division decides.  Three FP64 operations an axis (subtract, multiply,
// convert): the FP64 pipe bounds this kernel on this part.
#define KEY_MARGIN 16u
template<int dim>
__global__ void __launch_bounds__(256) k_keys(Particles P, const unsigned long long * bits,
  unsigned long long * keys, int * idx) {
  chain_begin();
  // the range and its scaled reciprocal, once per block
  __shared__ double s_mn[3], s_scale[3], s_rs[3];
  constexpr int md = 63 / dim;
  const double mult = (double)(1ull << md);
  if(threadIdx.x < dim) {
    const int d = threadIdx.x;
    const double mn = ord_dec(bits[d]);
    const double scale = ord_dec(bits[3 + d]) - mn;
    s_mn[d] = mn;
    s_scale[d] = scale;
    s_rs[d] = (1.0 / scale) * (mult * 1048576.0);
  }
  __syncthreads();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= P.n)
    return;
  constexpr unsigned long long maxv = (1ull << md) - 1;
  unsigned long long c[3] = {0, 0, 0};
  for(int d = 0; d < dim; ++d) {
    const double t = P.f[F_X + d][i] - s_mn[d];
    // saturates at 0 below and far above maxv
    const unsigned long long F = __double2ull_rz(t * s_rs[d]);
    unsigned long long u = F >> 20;
    const unsigned frac = (unsigned)F & 0xfffffu;
    if(frac - KEY_MARGIN > 0xfffffu - 2u * KEY_MARGIN) {
      const double q = t / s_scale[d] * mult;
      u = q > 0.0 ? __double2ull_rz(q) : 0ull;
    }
    c[d] = u < maxv ? u : maxv;
  }
  unsigned long long k;
  if(dim == 3)
    k = (1ull << 63) | spread3(c[0]) | (spread3(c[1]) << 1) | (spread3(c[2]) << 2);
  else
    k = (1ull << 62) | spread2(c[0]) | (spread2(c[1]) << 1);
  keys[i] = k;
  idx[i] = i;
}

cudaError_t launch_range(const Launch & L, const Particles & P, const PhysParams & pp,
  unsigned long long * range, unsigned long long * range_part) {
  int nb = (P.n + 255) / 256;
  if(nb > RANGE_BLOCKS)
    nb = RANGE_BLOCKS;
  if(pp.dim == 3)
    chain(L, k_range<3>, nb, 256, 0, P, range, range_part);
  else
    chain(L, k_range<2>, nb, 256, 0, P, range, range_part);
  *L.counter += 1;
  return cudaGetLastError();
}

cudaError_t launch_keys(const Launch & L, const Particles & P, const PhysParams & pp,
  const unsigned long long * range, unsigned long long * keys_out, int * idx_out) {
  const int nb = (P.n + 255) / 256;
  if(pp.dim == 3)
    chain(L, k_keys<3>, nb, 256, 0, P, range, keys_out, idx_out);
  else
    chain(L, k_keys<2>, nb, 256, 0, P, range, keys_out, idx_out);
  *L.counter += 1;
  return cudaGetLastError();
}

// ---------------------------------------------------------- radix sort --
// LSD radix sort of (key, value) pairs, 8-bit digits.  Tiles of 4608 keys:
// histogram per tile, one exclusive scan over [digit][tile], then a stable
// scatter in which each tile ranks its keys with warp match/ballot.
//
// A pass reads and writes every pair through HBM, so the passes cover the top
// data bits only: at least 32 prefixes per key, in whole pairs of digits (32
// bits up to 2^27 keys: four passes for eight).  k_prefix_runs then puts the few
// keys that share a prefix in order; a run of more than RS_RUN_MAX of them
// (particles crowded into a small part of the range) marks the sort, and the
// eight passes over all bits follow, which return at once without the mark.
// Such sets stay so from step to step, and four passes in vain are half a sort:
// SORT_CROWDED keeps the mark for the next build, which then makes the eight
// passes only, until no long run is left (k_crowded).  The word chooses between
// two ways to the same order, so whatever set it belongs to does no harm.
// A lattice with one particle 39 times its size away, sort and permute, every
// build trying the prefix first -> this (ms): 132k (one cluster) 0.188 -> 0.136,
// 2M 0.60 -> 0.50; beside one 3,000 times away 216k 0.190 -> 0.16, 1M 0.342 ->
// 0.308, 2M 0.515 -> 0.47.
// Sort with the permute, all bits -> prefix (ms): 216k 0.140 -> 0.103, 552k 0.178
// -> 0.150, 1M 0.278 -> 0.228, 2M 0.480 -> 0.327, 4M star 0.884 -> 0.664, 19.7M
// 3.59 -> 2.67.
#define RS_THREADS 256
#ifndef RS_ITEMS
#define RS_ITEMS 18
#endif
#define RS_TILE (RS_THREADS * RS_ITEMS)
// resident scatter blocks per SM (each holds its tile, 12 B a key, in
// shared memory)
#ifndef RS_SCATTER_BLOCKS
#define RS_SCATTER_BLOCKS 3
#endif

#define RS_RUN_MAX 24

// The sort's two state words: [0] the passes over all bits are due in this sort
// (set anew by each), [1] the last sort's keys were crowded.  The passes' part
// in it: over the prefix or over all bits, and the first of each, which sets up
// the words.
#define SORT_CROWDED 1
enum { SORT_PREFIX = 0, SORT_FULL = 1, SORT_FIRST = 2 };

__device__ __forceinline__ bool sort_due(const unsigned * state, int part) {
  return (part & SORT_FULL) ? state[0] != 0u : state[SORT_CROWDED] == 0u;
}

size_t radix_hist_entries(int n) {
  size_t nb = ((size_t)n + RS_TILE - 1) / RS_TILE;
  return 256 * nb + 256;  // [digit][tile] counts, then the 256 digit totals
}

__global__ void __launch_bounds__(RS_THREADS) k_radix_hist(
  const unsigned long long * keys, int n, int shift, unsigned * hist,
  unsigned * state, int part) {
  chain_begin();
  const bool setup = (part & SORT_FIRST) && blockIdx.x == 0 && threadIdx.x == 0;
  if(setup && !(part & SORT_FULL))
    state[0] = state[SORT_CROWDED];
  if(!sort_due(state, part))
    return;
  if(setup && (part & SORT_FULL))
    state[SORT_CROWDED] = 0u;
  __shared__ unsigned sh[256];
  sh[threadIdx.x] = 0;
  __syncthreads();
  int base = blockIdx.x * RS_TILE;
  unsigned long long kreg[RS_ITEMS];
#pragma unroll
  for(int r = 0; r < RS_ITEMS; ++r) {
    const int i = base + r * RS_THREADS + threadIdx.x;
    kreg[r] = i < n ? keys[i] : 0ull;
  }
#pragma unroll
  for(int r = 0; r < RS_ITEMS; ++r) {
    const int i = base + r * RS_THREADS + threadIdx.x;
    if(i < n)
      atomicAdd(&sh[(kreg[r] >> shift) & 255], 1u);
  }
  __syncthreads();
  hist[threadIdx.x * gridDim.x + blockIdx.x] = sh[threadIdx.x];
}

// Per digit: exclusive scan of its row of tile counts (coalesced, one
// block per digit) and the row total in tot[digit].
__global__ void __launch_bounds__(1024) k_scan_rows(unsigned * hist, int nb,
  unsigned * tot, const unsigned * state, int part) {
  chain_begin();
  if(!sort_due(state, part))
    return;
  __shared__ unsigned wsum[32];
  const int d = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
  unsigned * row = hist + (size_t)d * nb;
  unsigned run = 0;
  for(int base = 0; base < nb; base += 1024) {
    const int i = base + t;
    const unsigned v = i < nb ? row[i] : 0u;
    unsigned x = v;
    for(int o = 1; o < 32; o <<= 1) {
      unsigned y = __shfl_up_sync(FULL, x, o);
      if(lane >= o)
        x += y;
    }
    if(lane == 31)
      wsum[w] = x;
    __syncthreads();
    if(w == 0) {
      unsigned s2 = wsum[lane];
      for(int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(FULL, s2, o);
        if(lane >= o)
          s2 += y;
      }
      wsum[lane] = s2;
    }
    __syncthreads();
    const unsigned excl = run + (w ? wsum[w - 1] : 0u) + x - v;
    if(i < nb)
      row[i] = excl;
    run += wsum[31];
    __syncthreads();
  }
  if(t == 0)
    tot[d] = run;
}

// Stable scatter of one tile.  Warp w owns the tile's items
// [w * 32 * RS_ITEMS, (w + 1) * 32 * RS_ITEMS) and ranks them within their
// digits with a warp-private count per digit (match/ballot per round of 32
// keys, no block barrier); one scan per digit over the warps then gives
// every key its place in the tile sorted by digit (tile order kept), the
// tile is placed there in shared memory and written out in that order, so
// the keys of one digit leave the tile as one run of consecutive addresses.
#define RS_DYN_SMEM ((size_t)RS_TILE * 12)
__global__ void __launch_bounds__(RS_THREADS, RS_SCATTER_BLOCKS) k_radix_scatter(
  const unsigned long long * kin, const int * vin, unsigned long long * kout,
  int * vout, int n, int shift, const unsigned * offs, const unsigned * state, int part) {
  chain_begin();
  if(!sort_due(state, part))
    return;
  extern __shared__ __align__(16) unsigned char rs_dyn[];
  unsigned long long * skey = (unsigned long long *)rs_dyn;
  int * sval = (int *)(rs_dyn + (size_t)RS_TILE * 8);
  __shared__ unsigned base[256];   // where the tile's run of each digit goes
  __shared__ unsigned toff[256];   // where each digit starts in the sorted tile
  __shared__ unsigned wcnt[RS_THREADS / 32][256];
  __shared__ unsigned wtot[RS_THREADS / 32];
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  // exclusive block scan of one value per thread (256 threads)
  auto block_scan = [&](unsigned v) {
    unsigned x = v;
    for(int o = 1; o < 32; o <<= 1) {
      unsigned y = __shfl_up_sync(FULL, x, o);
      if(lane >= o)
        x += y;
    }
    if(lane == 31)
      wtot[w] = x;
    __syncthreads();
    unsigned pre = 0;
    for(int k = 0; k < w; ++k)
      pre += wtot[k];
    __syncthreads();
    return pre + x - v;
  };
  // digit base = sum of the totals of smaller digits + this tile's offset
  // within its digit row
  base[t] = block_scan(offs[256 * gridDim.x + t]) + offs[t * gridDim.x + blockIdx.x];
  for(int k = 0; k < RS_THREADS / 32; ++k)
    wcnt[k][t] = 0;
  // this warp's keys into registers first: all loads in flight (the
  // values follow when the keys are placed)
  const int tile = blockIdx.x * RS_TILE;
  const int wbase = tile + w * 32 * RS_ITEMS;
  unsigned long long kreg[RS_ITEMS];
#pragma unroll
  for(int r = 0; r < RS_ITEMS; ++r) {
    const int i = wbase + r * 32 + lane;
    kreg[r] = i < n ? kin[i] : 0ull;
  }
  __syncthreads();
  const unsigned lt = lanemask_lt();
  unsigned * cnt = wcnt[w];
  unsigned rk[RS_ITEMS];  // digit << 16 | rank within the digit in this warp
#pragma unroll
  for(int r = 0; r < RS_ITEMS; ++r) {
    const bool valid = wbase + r * 32 + lane < n;
    const int digit = valid ? (int)((kreg[r] >> shift) & 255) : 256;
    const unsigned mask = __match_any_sync(FULL, digit);
    const unsigned before = valid ? cnt[digit] : 0u;
    __syncwarp();
    if(valid && (__ffs(mask) - 1) == lane)
      cnt[digit] = before + __popc(mask);
    __syncwarp();
    rk[r] = ((unsigned)(valid ? digit : 0) << 16) | (before + __popc(mask & lt));
  }
  __syncthreads();
  // per digit (thread t): exclusive prefix over the warps, then the start of
  // the digit in the sorted tile
  unsigned run = 0;
  for(int k = 0; k < RS_THREADS / 32; ++k) {
    const unsigned c = wcnt[k][t];
    wcnt[k][t] = run;
    run += c;
  }
  toff[t] = block_scan(run);
  __syncthreads();
#pragma unroll
  for(int r = 0; r < RS_ITEMS; ++r) {
    const int i = wbase + r * 32 + lane;
    if(i < n) {
      const unsigned d = rk[r] >> 16;
      const unsigned l = toff[d] + cnt[d] + (rk[r] & 0xffffu);
      skey[l] = kreg[r];
      sval[l] = vin[i];
    }
  }
  __syncthreads();
  const int ntile = n - tile < RS_TILE ? n - tile : RS_TILE;
  for(int l = t; l < ntile; l += RS_THREADS) {
    const unsigned long long key = skey[l];
    const int d = (int)((key >> shift) & 255);
    const unsigned pos = base[d] + ((unsigned)l - toff[d]);
    kout[pos] = key;
    vout[pos] = sval[l];
  }
}

// The keys are in order of key >> low: the first thread of each run that shares
// a prefix orders it in place, ties as they are (the others see the same
// prefixes meanwhile).  One read of the keys where there are no runs.
__global__ void __launch_bounds__(256) k_prefix_runs(unsigned long long * keys, int * vals,
  int n, int low, unsigned * state) {
  chain_begin();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if(i + 1 >= n || !sort_due(state, SORT_PREFIX))
    return;
  const unsigned long long p = keys[i] >> low;
  if(keys[i + 1] >> low != p || (i > 0 && keys[i - 1] >> low == p))
    return;
  int len = 2;
  while(i + len < n && keys[i + len] >> low == p)
    if(++len > RS_RUN_MAX) {
      state[0] = 1u;
      return;
    }
  for(int j = i + 1; j < i + len; ++j) {
    const unsigned long long k = keys[j];
    const int v = vals[j];
    int m = j;
    for(; m > i && keys[m - 1] > k; --m) {
      keys[m] = keys[m - 1];
      vals[m] = vals[m - 1];
    }
    if(m < j) {
      keys[m] = k;
      vals[m] = v;
    }
  }
}

// After the passes over all bits: are the keys still crowded, that is, would the
// passes over the prefix leave a run that k_prefix_runs does not take?
__global__ void __launch_bounds__(256) k_crowded(const unsigned long long * keys, int n,
  int low, unsigned * state) {
  chain_begin();
  if(!sort_due(state, SORT_FULL))
    return;
  int found = 0;
  for(int i = blockIdx.x * 256 + threadIdx.x; i + RS_RUN_MAX < n && !found;
      i += gridDim.x * 256)
    found = keys[i] >> low == keys[i + RS_RUN_MAX] >> low;
  // few blocks, one store each: of 8,192 blocks the stores to one word alone
  // took 0.1 ms
  if(__syncthreads_or(found) && threadIdx.x == 0)
    state[SORT_CROWDED] = 1u;
}

// ---- one-cluster sort --------------------------------------------------
// Up to SC_MAX keys one launch sorts everything: a cluster of up to 16 blocks,
// each with an equal share of the places.  A digit pass ranks a block's keys as
// k_radix_scatter does, the blocks exchange their digit counts through
// distributed shared memory, and the keys, put in digit order in shared memory
// first so that they leave in runs of consecutive addresses, go to their
// places through L2 (stores to the owner's shared memory instead moved 6 bytes
// a clock and SM, three times slower).  Two cluster barriers a pass (and one
// that has to be passed before a block first stores to another); no launch
// between passes.  Eight passes of three launches each (below), whose tiles
// fill a few SMs at these sizes, lost to it: range, keys and sort of 2,250 / 31,000 /
// 132,651 keys take 33 / 44 / 76 us this way, 160 / 175 / 189 that way (at
// 139,264 keys 78 against 188; beyond it a block's registers are full).
// Latency bounds it: a pass of 8,300 keys a block is 33,000 cycles, 8,000 of
// them the ballots, 5,000 the scatter.
//
// The passes cover the top data bits of the keys only, as many as tell n
// particles spread over the range apart (the prefix has at least 32 values per
// particle); keys that share a prefix are adjacent then, in input order, and
// the thread of the first sorts them by insertion.  A run longer than SC_RUN
// (a clump in a wide range) makes the cluster go on with all eight passes, and
// start with them in the next sort (SORT_CROWDED, as below, until no such run
// is left).
#define SC_THREADS 512
#define SC_WARPS (SC_THREADS / 32)
#define SC_ITEMS 17
#define SC_BLOCKS 16
#define SC_MAX (SC_BLOCKS * SC_THREADS * SC_ITEMS)
#define SC_RUN 12

// Shared memory of one block with `per` places: keys and values in digit order
// (at the end: in place order, with the places a run may reach into), digit
// counts per warp and per block of the cluster (16 bits: at most
// SC_THREADS * SC_ITEMS).
__host__ __device__ constexpr size_t sc_smem(int per) {
  return (size_t)(per + SC_RUN + 4) * 12 + SC_WARPS * 256 * 2 + SC_BLOCKS * 256 * 2 +
         2 * 256 * 4 + 64 * 4;
}

__global__ void __launch_bounds__(SC_THREADS, 1) k_sort_cluster(
  unsigned long long * keys, int * vals, unsigned long long * keys_tmp, int * vals_tmp,
  int n, int per, int bits, int prefix_bits, unsigned * state) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char sc_dyn[];
  unsigned long long * okey = (unsigned long long *)sc_dyn;
  int * oval = (int *)(okey + per + SC_RUN + 4);
  unsigned short * wcnt = (unsigned short *)(oval + per + SC_RUN + 4);
  unsigned short * ccnt = wcnt + SC_WARPS * 256;
  unsigned * base = (unsigned *)(ccnt + SC_BLOCKS * 256);  // where a digit's keys go
  unsigned * toff = base + 256;  // where they start in digit order here
  unsigned * aux = toff + 256;   // [0..15] scans, [16] long-run flag
  cg::cluster_group cl = cg::this_cluster();
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const unsigned me = cl.block_rank(), nc = cl.num_blocks();
  const int g0 = (int)me * per;                       // first place
  const int mine = max(0, min(per, n - g0));          // places of this block
  const int rounds = (per + SC_THREADS - 1) / SC_THREADS;
  const unsigned lt = lanemask_lt();
  unsigned long long *kin = keys, *kout = keys_tmp;
  int *vin = vals, *vout = vals_tmp;
  if(t == 0)
    aux[16] = 0;
  // A block's shared memory may be touched by the others once it has started:
  // every block arrives here, and waits before the first pass's exchange of
  // counts, which the loads and ballots before it leave time for.
  cl.barrier_arrive();
  bool all_started = false;
  const int low = bits - prefix_bits;
  // (every block has read the word before any passes the barrier after which
  // it is written)
  const bool crowded = state[SORT_CROWDED] != 0u;
  int first_shift = crowded ? 0 : low;
  if(crowded)
    bits = 64;
  while(true) {
    for(int shift = first_shift; shift < bits; shift += 8) {
      // warp w owns the places [w * 32 * rounds, ...) of the block
      unsigned long long kreg[SC_ITEMS];
      int vreg[SC_ITEMS];
      unsigned rk[SC_ITEMS];  // lanes with the same digit, then the rank among the warp's
      unsigned short * cnt = wcnt + w * 256;
#pragma unroll
      for(int r = 0; r < SC_ITEMS; ++r) {
        const int i = (w * rounds + r) * 32 + lane;
        const bool in = r < rounds && i < mine;
        // (the other blocks wrote these: past the L1)
        kreg[r] = in ? __ldcg(kin + g0 + i) : 0ull;
        vreg[r] = in ? __ldcg(vin + g0 + i) : 0;
      }
      for(int i = lane; i < 128; i += 32)
        ((unsigned *)cnt)[i] = 0;
      __syncwarp();
      // the lanes of a round that share a digit, by one ballot per bit (a
      // match instruction takes ~1,000 cycles on 32 different digits here):
      // independent between rounds, so they overlap; only the counts chain
#pragma unroll
      for(int r = 0; r < SC_ITEMS; ++r) {
        if(r < rounds) {
          const bool valid = (w * rounds + r) * 32 + lane < mine;
          const unsigned digit = (unsigned)(kreg[r] >> shift) & 255u;
          unsigned mask = __ballot_sync(FULL, valid);
#pragma unroll
          for(int bit = 0; bit < 8; ++bit) {
            const bool on = (digit >> bit) & 1u;
            const unsigned bal = __ballot_sync(FULL, on);
            mask &= on ? bal : ~bal;
          }
          rk[r] = valid ? mask : 0u;
        }
      }
#pragma unroll
      for(int r = 0; r < SC_ITEMS; ++r) {
        if(r < rounds) {
          const unsigned mask = rk[r];
          const unsigned digit = (unsigned)(kreg[r] >> shift) & 255u;
          const unsigned before = mask ? cnt[digit] : 0u;
          __syncwarp();
          if(mask && (__ffs(mask) - 1) == lane)
            cnt[digit] = (unsigned short)(before + __popc(mask));
          __syncwarp();
          rk[r] = before + __popc(mask & lt);
        }
      }
      __syncthreads();
      // per digit: prefix over the warps (two threads a digit, half the warps
      // each); the digit's total goes to every block of the cluster
      if(!all_started) {
        cl.barrier_wait();
        all_started = true;
      }
      {
        const int d = t >> 1, part = t & 1;
        unsigned c[SC_WARPS / 2], sum = 0;
#pragma unroll
        for(int k = 0; k < SC_WARPS / 2; ++k) {
          c[k] = sum;
          sum += wcnt[(part * (SC_WARPS / 2) + k) * 256 + d];
        }
        const unsigned other = __shfl_xor_sync(FULL, sum, 1);
#pragma unroll
        for(int k = 0; k < SC_WARPS / 2; ++k)
          wcnt[(part * (SC_WARPS / 2) + k) * 256 + d] =
            (unsigned short)((part ? other : 0u) + c[k]);
        for(unsigned b = part; b < nc; b += 2)
          cl.map_shared_rank(ccnt, b)[me * 256 + d] = (unsigned short)(sum + other);
      }
      cl.sync();
      // first place of each digit's keys of this block, in the cluster and in
      // the block: two scans over the digits
      unsigned tot = 0, pre = 0, own = 0, x = 0, y = 0;
      if(t < 256) {
        for(unsigned b = 0; b < nc; ++b) {
          const unsigned c = ccnt[b * 256 + t];
          pre += b < me ? c : 0u;
          tot += c;
        }
        own = ccnt[me * 256 + t];
        x = tot;
        y = own;
        for(int o = 1; o < 32; o <<= 1) {
          const unsigned xo = __shfl_up_sync(FULL, x, o), yo = __shfl_up_sync(FULL, y, o);
          if(lane >= o) {
            x += xo;
            y += yo;
          }
        }
        if(lane == 31) {
          aux[w] = x;
          aux[8 + w] = y;
        }
      }
      __syncthreads();
      if(t < 256) {
        unsigned loc = 0;
        for(int k = 0; k < w; ++k) {
          pre += aux[k];
          loc += aux[8 + k];
        }
        base[t] = pre + x - tot;
        toff[t] = loc + y - own;
      }
      __syncthreads();
#pragma unroll
      for(int r = 0; r < SC_ITEMS; ++r) {
        const int i = (w * rounds + r) * 32 + lane;
        if(r < rounds && i < mine) {
          const unsigned d = (unsigned)(kreg[r] >> shift) & 255u;
          const unsigned l = toff[d] + cnt[d] + rk[r];
          okey[l] = kreg[r];
          oval[l] = vreg[r];
        }
      }
      __syncthreads();
#pragma unroll 4
      for(int l = t; l < mine; l += SC_THREADS) {
        const unsigned long long key = okey[l];
        const unsigned d = (unsigned)(key >> shift) & 255u;
        const unsigned pos = base[d] + ((unsigned)l - toff[d]);
        __stcg(kout + pos, key);
        __stcg(vout + pos, oval[l]);
      }
      // the keys are in place, and nobody writes where somebody still reads:
      // a pass reads one pair of buffers and writes the other
      cl.sync();
      unsigned long long * tk = kin;
      kin = kout;
      kout = tk;
      int * tv = vin;
      vin = vout;
      vout = tv;
    }
    if(first_shift == 0)
      break;
    // Runs of equal prefixes: this block's places, the ones a run may reach
    // into and the prefix before them.
    const int ext = max(0, min(mine + SC_RUN + 1, n - g0));
    for(int i = t; i < ext; i += SC_THREADS) {
      okey[i] = __ldcg(kin + g0 + i);
      oval[i] = __ldcg(vin + g0 + i);
    }
    const unsigned long long kprev = g0 > 0 && mine > 0 ? __ldcg(kin + g0 - 1) : 0ull;
    __syncthreads();
    auto prefix = [&](int i) { return (i < 0 ? kprev : okey[i]) >> first_shift; };
    auto in_run = [&](int i) { return g0 + i > 0 && prefix(i - 1) == prefix(i); };
    for(int i = t; i < mine; i += SC_THREADS)
      if(i + SC_RUN < ext && prefix(i) == prefix(i + SC_RUN)) {
        for(unsigned b = 0; b < nc; ++b)
          cl.map_shared_rank(aux, b)[16] = 1;
      }
    cl.sync();
    if(aux[16] && me == 0 && t == 0)
      state[SORT_CROWDED] = 1u;
    if(!aux[16]) {
      // the first of a run puts it in order, the keys that begin no run and
      // belong to none are in place
      for(int i = t; i < mine; i += SC_THREADS) {
        if(in_run(i))
          continue;
        int len = 1;
        while(i + len < ext && prefix(i + len) == prefix(i)) {
          const unsigned long long kv = okey[i + len];
          const int vv = oval[i + len];
          int z = i + len;
          while(z > i && okey[z - 1] > kv) {
            okey[z] = okey[z - 1];
            oval[z] = oval[z - 1];
            --z;
          }
          okey[z] = kv;
          oval[z] = vv;
          ++len;
        }
        for(int q = 0; q < len; ++q) {
          keys[g0 + i + q] = okey[i + q];
          vals[g0 + i + q] = oval[i + q];
        }
      }
      return;
    }
    // go on from here with every digit: equal keys are still in input order
    first_shift = 0;
    bits = 64;
  }
  if(kin != keys)
    for(int i = t; i < mine; i += SC_THREADS) {
      keys[g0 + i] = __ldcg(kin + g0 + i);
      vals[g0 + i] = __ldcg(vin + g0 + i);
    }
  if(crowded) {
    // still so?
    int found = 0;
    for(int i = t; i < mine && g0 + i + SC_RUN < n && !found; i += SC_THREADS)
      found = __ldcg(kin + g0 + i) >> low == __ldcg(kin + g0 + i + SC_RUN) >> low;
    if(__syncthreads_or(found) && t == 0)
      cl.map_shared_rank(aux, 0)[16] = 1;
    cl.sync();
    if(me == 0 && t == 0)
      state[SORT_CROWDED] = aux[16];
  }
}

// Blocks of the cluster for n keys, 0 where the sort takes several launches:
// a key per thread (one round of ranking), twice the blocks with twice the keys,
// until the cluster is full.
// A cluster of 16 is beyond the portable 8: asked of the device once.
static int sc_blocks(int n) {
  static std::atomic<unsigned long long> ready{0}, wide{0};
  if(n > SC_MAX)
    return 0;
  int dev = 0;
  if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return 0;
  const cudaError_t e = once_per_device(&ready, [&]() {
    const size_t most = sc_smem(SC_THREADS * SC_ITEMS);
    cudaError_t r = cudaFuncSetAttribute(k_sort_cluster,
      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if(r == cudaSuccess)
      r = cudaFuncSetAttribute(k_sort_cluster,
        cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if(r != cudaSuccess)
      return r;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {SC_BLOCKS, 1, 1};
    cfg.gridDim = dim3(SC_BLOCKS);
    cfg.blockDim = dim3(SC_THREADS);
    cfg.dynamicSmemBytes = most;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fit = 0;
    if(cudaOccupancyMaxActiveClusters(&fit, k_sort_cluster, &cfg) == cudaSuccess && fit > 0)
      wide.fetch_or(1ull << dev, std::memory_order_release);
    else
      cudaGetLastError();
    return cudaSuccess;
  });
  if(e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  const bool w16 = (wide.load(std::memory_order_acquire) >> dev) & 1ull;
  int c = 1;
  while(c < (w16 ? SC_BLOCKS : 8) && n > c * SC_THREADS)
    c <<= 1;
  return n <= c * SC_THREADS * SC_ITEMS ? c : 0;
}

cudaError_t radix_sort_pairs(const Launch & L, unsigned long long * keys,
  int * vals, unsigned long long * keys_tmp, int * vals_tmp, int n,
  unsigned * hist, int bits, unsigned * state) {
  if(const int c = sc_blocks(n)) {
    const int per = ((n + c - 1) / c + 3) & ~3;
    // prefix bits: at least 32 prefixes per key, in whole digits
    int lg = 0;
    while((1 << lg) < n)
      ++lg;
    const int pb = (lg + 5 + 7) / 8 * 8;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)c, 1, 1};
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(SC_THREADS);
    cfg.dynamicSmemBytes = sc_smem(per);
    cfg.stream = L.stream;
    cfg.attrs = at;
    cfg.numAttrs = L.overlap() ? 2 : 1;
    *L.counter += 1;
    return cudaLaunchKernelEx(&cfg, k_sort_cluster, keys, vals, keys_tmp, vals_tmp, n, per,
      bits, pb, state);
  }
  static std::atomic<unsigned long long> attr_devices{0};
  cudaError_t ae = once_per_device(&attr_devices, []() {
    return cudaFuncSetAttribute(k_radix_scatter,
      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RS_DYN_SMEM);
  });
  if(ae != cudaSuccess)
    return ae;
  int nb = (n + RS_TILE - 1) / RS_TILE;
  unsigned long long *ka = keys, *kb = keys_tmp;
  int *va = vals, *vb = vals_tmp;
  // an even number of passes: the result is back in (keys, vals)
  auto passes = [&](int from, int to, int part) {
    for(int shift = from; shift < to; shift += 8) {
      const int p = shift == from ? part | SORT_FIRST : part;
      chain(L, k_radix_hist, nb, RS_THREADS, 0, ka, n, shift, hist, state, p);
      chain(L, k_scan_rows, 256, 1024, 0, hist, nb, hist + (size_t)256 * nb, state, p);
      chain(L, k_radix_scatter, nb, RS_THREADS, RS_DYN_SMEM, ka, va, kb, vb, n,
        shift, hist, state, p);
      *L.counter += 3;
      unsigned long long * tk = ka;
      ka = kb;
      kb = tk;
      int * tv = va;
      va = vb;
      vb = tv;
    }
  };
  int lg = 0;
  while((1ll << lg) < n)
    ++lg;
  const int low = bits - (lg + 5 + 15) / 16 * 16;
  passes(low, bits, SORT_PREFIX);
  chain(L, k_prefix_runs, (n + 255) / 256, 256, 0, keys, vals, n, low, state);
  passes(0, 64, SORT_FULL);
  chain(L, k_crowded, 152 * 2, 256, 0, keys, n, low, state);
  *L.counter += 2;
  return cudaGetLastError();
}

// Fields whose bit is set in `skip` are left behind: the caller overwrites
// them before anything reads them.  With `vel`, the mixed path's
// {v, c_s} record of the new order is written on the way (what the density
// pass would otherwise pack).
//
// The gather is bound by HBM; the position records of the tree, the walk and
// the float-float passes, whose arithmetic is FP64 and which a pass of their
// own would read five fields for again, come out of it too.  Every position is
// one 48-bit fixed-point word per axis,
//   F = round((x - lo) / E * 2^48),  E = the largest range extent
//   enlarged by 2^-19 (so F < 2^48 - 2^28),
// from which both packed forms follow by integer operations:
//   float-float X = 1 + F / 2^48 in [1, 2): the high word takes F's top
//     23 bits (exactly), the low word the other 25 (rounded to 24 bits);
//   the walk's 31-bit fixed point q = F / 2^17 rounded to nearest, one
//     step = E / 2^31 on every axis.
template<int dim>
__global__ void __launch_bounds__(256) k_permute(Particles src, Particles dst,
  const int * perm, const unsigned long long * keys, unsigned skip,
  const unsigned long long * rbits, Packed K, int * ngroups, unsigned * list_stat,
  float4 * vel) {
  chain_begin();
  __shared__ double s_lo[3], s_sc, s_iE;
  if(dim > 0 && threadIdx.x < dim)
    s_lo[threadIdx.x] = ord_dec(rbits[threadIdx.x]);
  if(dim > 0 && threadIdx.x == 0) {
    double E = 0.0;
    for(int d = 0; d < dim; ++d)
      E = fmax(E, ord_dec(rbits[3 + d]) - ord_dec(rbits[d]));
    E *= 1.0 + 0x1p-19;
    s_iE = 1.0 / E;
    s_sc = s_iE * 0x1p48;
    if(blockIdx.x == 0) {
      *ngroups = 0;
      list_stat[0] = list_stat[1] = 0u;
      K.fscale[0] = E;
      K.fscale[1] = s_iE;
      // h_min == h_max: the pair passes take h_ab = h_a throughout
      K.fscale[2] = rbits[6] == rbits[7] ? 1.0 : 0.0;
      for(int d = 0; d < 3; ++d)
        K.qscale[d] = d < dim ? (float)(E * 0x1p-31) : 0.f;
    }
  }
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= src.n)
    return;
  const int p = perm[i];
#pragma unroll
  for(int k = 0; k < NF; ++k)
    if(!((skip >> k) & 1u))
      dst.f[k][i] = src.f[k][p];
  dst.id[i] = src.id[p];
  dst.key[i] = keys[i];
  if(dim == 0)  // a plain gather
    return;
  if(vel)
    vel[i] = make_float4(to_f32(src.f[F_VX][p]), to_f32(src.f[F_VY][p]),
      dim == 3 ? to_f32(src.f[F_VZ][p]) : 0.f, to_f32(src.f[F_CS][p]));
  const long long fmax48 = (1LL << 48) - (1LL << 28);
  int q[3] = {0, 0, 0};
  float xh[4] = {1.f, 1.f, 1.f, 0.f}, xl[4] = {0.f, 0.f, 0.f, 0.f};
  for(int d = 0; d < dim; ++d) {
    long long F = __double2ll_rn((src.f[F_X + d][p] - s_lo[d]) * s_sc);
    F = F < 0 ? 0 : F > fmax48 ? fmax48 : F;
    q[d] = (int)((F + (1LL << 16)) >> 17);
    xh[d] = __int_as_float(0x3f800000 | (int)(F >> 25));
    xl[d] = (float)(int)(F & ((1LL << 25) - 1)) * 0x1p-48f;
  }
  const double h = src.f[F_H][p];
  const double hX = h * s_iE;
  xh[3] = to_f32(hX);
  xl[3] = to_f32(hX - to_f64(xh[3]));
  K.qpos[i] = make_int4(q[0], q[1], q[2], __float_as_int(to_f32(h)));
  K.fph[i] = make_float4(xh[0], xh[1], xh[2], xh[3]);
  K.fpl[i] = make_float4(xl[0], xl[1], xl[2], xl[3]);
  const double m = src.f[F_M][p];
  const float mh = to_f32(m);
  ((float2 *)K.fmA)[2 * i] = make_float2(mh, to_f32(m - to_f64(mh)));
}

cudaError_t launch_gather(const Launch & L, const Particles & src, const Particles & dst,
  const int * perm, const unsigned long long * keys, unsigned skip) {
  chain(L, k_permute<0>, (src.n + 255) / 256, 256, 0, src, dst, perm, keys, skip,
    nullptr, Packed{}, nullptr, nullptr, nullptr);
  *L.counter += 1;
  return cudaGetLastError();
}

cudaError_t launch_permute(const Launch & L, const Particles & src,
  const Particles & dst, const int * perm, const unsigned long long * keys,
  unsigned skip, const unsigned long long * rbits, const Packed & K, int * ngroups,
  unsigned * list_stat, float4 * vel, int dim) {
  const int nb = (src.n + 255) / 256;
  if(dim == 3)
    chain(L, k_permute<3>, nb, 256, 0, src, dst, perm, keys, skip, rbits, K, ngroups,
      list_stat, vel);
  else
    chain(L, k_permute<2>, nb, 256, 0, src, dst, perm, keys, skip, rbits, K, ngroups,
      list_stat, vel);
  *L.counter += 1;
  return cudaGetLastError();
}

// ------------------------------------------------------- radix tree -----
// Binary radix tree over the sorted keys.  Equal keys (reported as
// FSPH_ERR_DUPLICATE_KEY) are ordered by index, so the tree stays a valid
// binary tree and every walk over it terminates.
// One launch builds the tree bottom up: a thread per leaf climbs, and of the
// two children of a node the thread that arrives second forms it, so topology,
// node data and walk groups come out of one climb (a top-down construction
// first and a second climb for the groups read the node arrays three more
// times, one dependent load after the other on every level).
//
// Where a node goes follows from its two ends alone: with D(i) the number of
// bits the keys of i and i + 1 share (kdelta), a node [l, r] is the left child
// of the node split at r if D(r) > D(l - 1), else the right child of the node
// split at l - 1; as a left child its index is r, as a right child l, so the
// children of a node split at s are always s and s + 1 (leaves or nodes).
//
// The thread that arrives first at split s leaves the far end of its child
// and the D beyond it, the one that arrives second takes them.  A node whose
// keys all lie in this block's leaves (told from the two keys around them)
// meets in shared memory, child data included; above that, a 64-bit
// device-scope exchange releases the first child's data, which the second
// thread reads through L2, and leaves the slot empty for the next build.
//
// Node data: the fixed-point position box and the largest h of every node
// (what the neighbour walk prunes with); ALL (varying h, the ordered mode, or
// gravity) adds the reference's FP64 box of x -/+ h/2 (compute_cofm,
// default_physics.h:79-82,90-93) with its outward FP32 copy, and with gravity
// the raw mass moments (ten FP64 sums; left child first, so the sums do not
// depend on who combined them).  The boxes combine on the integer pipe: FP64
// comparisons at every node would bind the climb on this part.  The outward
// FP32 copies combine among themselves, rounding being monotonic.
//
// Latency bounds it: about 150 ns a level in shared memory, 0.8 us above.
// Leaves per block, measured (the tree phase, ms; 2k 2D and 2M 3D with one h,
// 50k and 4M star with gravity):
//   one h    256: 0.029, 0.196   512: 0.032, 0.202   1024: 0.034, 0.210
//   ALL      128: 0.069, 1.73    256: 0.071, 1.88     512: 0.071, 2.16
// A block waits for its longest climb; with the 368 bytes that a leaf's two
// slots take in ALL, 128 leaves let four blocks share an SM instead of two.
constexpr int TREE_UNI_THREADS = 256, TREE_ALL_THREADS = 128;
template<bool ALL>
__host__ __device__ constexpr int tree_threads() {
  return ALL ? TREE_ALL_THREADS : TREE_UNI_THREADS;
}
#define TREE_EMPTY 0xffffffffffffffffull

// smaller and larger of two finite doubles by their bits
__device__ __forceinline__ bool less_bits(double a, double b) {
  long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  x ^= (long long)((unsigned long long)(x >> 63) >> 1);
  y ^= (long long)((unsigned long long)(y >> 63) >> 1);
  return x < y;
}

template<bool ALL>
struct TreeData {
  int4 lo, hi;        // lo.w: float bits of h_max; hi.w: the children's code
};
template<>
struct TreeData<true> {
  int4 lo, hi;
  double b[6];        // x - h/2 minima, x + h/2 maxima
  float f[6];         // the same relative to the range's corner, outwards
  double g[10];       // moments
};

template<bool ALL>
__host__ __device__ constexpr size_t tree_smem() {
  return 2 * tree_threads<ALL>() * (ALL ? 32 + 48 + 24 + 80 : 32);
}

// (1: shared-memory deposit of a child, slot q of two per thread, as
// structure of arrays)
template<bool ALL, bool STORE>
__device__ __forceinline__ void tree_slot(unsigned char * sm, int q, TreeData<ALL> & d,
  bool boxes, bool mom) {
  constexpr int N = 2 * tree_threads<ALL>();
  int4 * s4 = (int4 *)sm;
  if(STORE) {
    s4[q] = d.lo;
    s4[N + q] = d.hi;
  }
  else {
    d.lo = s4[q];
    d.hi = s4[N + q];
  }
  if constexpr(ALL) {
    double * sb = (double *)(sm + (size_t)N * 32);
    double * sg = sb + 6 * N;
    float * sf = (float *)(sg + 10 * N);
    if(boxes)
      for(int k = 0; k < 6; ++k) {
        if(STORE) {
          sb[k * N + q] = d.b[k];
          sf[k * N + q] = d.f[k];
        }
        else {
          d.b[k] = sb[k * N + q];
          d.f[k] = sf[k * N + q];
        }
      }
    if(mom)
      for(int k = 0; k < 10; ++k) {
        if(STORE)
          sg[k * N + q] = d.g[k];
        else
          d.g[k] = sg[k * N + q];
      }
  }
}

template<int dim, bool ALL>
__device__ __forceinline__ void tree_leaf(const Particles & P, const int4 * qpos, int j,
  bool boxes, bool mom, const double * rc, const double * r0, TreeData<ALL> & d) {
  const int4 q = qpos[j];
  d.lo = q;
  d.hi = make_int4(q.x, q.y, q.z, 0);
  if constexpr(ALL) {
    double x[3] = {0.0, 0.0, 0.0};
    for(int k = 0; k < dim; ++k)
      x[k] = P.f[F_X + k][j];
    if(boxes) {
      const double hh = P.f[F_H][j] / 2.;
      for(int k = 0; k < 3; ++k) {
        d.b[k] = k < dim ? x[k] - hh : 0.0;
        d.b[3 + k] = k < dim ? x[k] + hh : 0.0;
        d.f[k] = k < dim ? __double2float_rd(d.b[k] - r0[k]) : 0.f;
        d.f[3 + k] = k < dim ? __double2float_ru(d.b[3 + k] - r0[k]) : 0.f;
      }
    }
    if(mom) {
      const double m = P.f[F_M][j];
      double y[3] = {0.0, 0.0, 0.0};
      for(int k = 0; k < dim; ++k)
        y[k] = x[k] - rc[k];
      const double my[3] = {m * y[0], m * y[1], m * y[2]};
      d.g[0] = m;
      d.g[1] = my[0];
      d.g[2] = my[1];
      d.g[3] = my[2];
      d.g[4] = my[0] * y[0];
      d.g[5] = my[1] * y[1];
      d.g[6] = my[2] * y[2];
      d.g[7] = my[0] * y[1];
      d.g[8] = my[0] * y[2];
      d.g[9] = my[1] * y[2];
    }
  }
}

// node p's data to (STORE) or from device memory (through L2)
template<bool ALL, bool STORE>
__device__ __forceinline__ void tree_node_mem(const Tree & T, int p, TreeData<ALL> & d,
  bool boxes, bool mom) {
  if(STORE) {
    T.qbox[2 * p] = d.lo;
    T.qbox[2 * p + 1] = d.hi;
  }
  else {
    d.lo = __ldcg(&T.qbox[2 * p]);
    d.hi = __ldcg(&T.qbox[2 * p + 1]);
  }
  if constexpr(ALL) {
    if(boxes) {
      // NodeBox: lo xyz, hmax (0), hi xyz, pad (0)
      double2 * bx = (double2 *)&T.box2[p];
      float4 * fx = T.fbox2 + 2 * (size_t)p;
      if(STORE) {
        bx[0] = make_double2(d.b[0], d.b[1]);
        bx[1] = make_double2(d.b[2], 0.0);
        bx[2] = make_double2(d.b[3], d.b[4]);
        bx[3] = make_double2(d.b[5], 0.0);
        fx[0] = make_float4(d.f[0], d.f[1], d.f[2], 0.f);
        fx[1] = make_float4(d.f[3], d.f[4], d.f[5], 0.f);
      }
      else {
        const double2 b0 = __ldcg(bx), b1 = __ldcg(bx + 1), b2 = __ldcg(bx + 2),
                      b3 = __ldcg(bx + 3);
        const float4 f0 = __ldcg(fx), f1 = __ldcg(fx + 1);
        d.b[0] = b0.x; d.b[1] = b0.y; d.b[2] = b1.x;
        d.b[3] = b2.x; d.b[4] = b2.y; d.b[5] = b3.x;
        d.f[0] = f0.x; d.f[1] = f0.y; d.f[2] = f0.z;
        d.f[3] = f1.x; d.f[4] = f1.y; d.f[5] = f1.z;
      }
    }
    if(mom) {
      double2 * gm = (double2 *)(T.gmom + 10 * (size_t)p);
      for(int k = 0; k < 5; ++k) {
        if(STORE)
          gm[k] = make_double2(d.g[2 * k], d.g[2 * k + 1]);
        else {
          const double2 v = __ldcg(gm + k);
          d.g[2 * k] = v.x;
          d.g[2 * k + 1] = v.y;
        }
      }
    }
  }
}

// d: one child on entry, the node of both on return
template<bool ALL>
__device__ __forceinline__ void tree_merge(TreeData<ALL> & d, const TreeData<ALL> & e,
  bool boxes, bool mom) {
  d.lo.x = min(d.lo.x, e.lo.x);
  d.lo.y = min(d.lo.y, e.lo.y);
  d.lo.z = min(d.lo.z, e.lo.z);
  d.hi.x = max(d.hi.x, e.hi.x);
  d.hi.y = max(d.hi.y, e.hi.y);
  d.hi.z = max(d.hi.z, e.hi.z);
  d.lo.w = __float_as_int(fmaxf(__int_as_float(d.lo.w), __int_as_float(e.lo.w)));
  if constexpr(ALL) {
    if(boxes)
      for(int k = 0; k < 3; ++k) {
        d.b[k] = less_bits(e.b[k], d.b[k]) ? e.b[k] : d.b[k];
        d.b[3 + k] = less_bits(d.b[3 + k], e.b[3 + k]) ? e.b[3 + k] : d.b[3 + k];
        d.f[k] = fminf(d.f[k], e.f[k]);
        d.f[3 + k] = fmaxf(d.f[3 + k], e.f[3 + k]);
      }
    if(mom)
      for(int k = 0; k < 10; ++k)
        d.g[k] = d.g[k] + e.g[k];
  }
}

// ALL or not: both are launched, and the one the device's range words do not
// select returns at once.  lead: the key bits above the data.  Two particles
// with one full key would make the reference's build_tree loop run past depth
// 0 (tree_topology.h:957-971): reported.
template<int dim, bool ALL>
__global__ void __launch_bounds__(tree_threads<ALL>()) k_tree(const unsigned long long * K,
  Particles P, Tree T, const int4 * qpos, const unsigned long long * rbits, int ordered,
  int gmax, DevStatus * st) {
  chain_begin();
  const bool boxes = ordered || rbits[6] != rbits[7], mom = T.gmom != nullptr;
  if(ALL != (boxes || mom))
    return;
  constexpr int TREE_THREADS = tree_threads<ALL>();
  extern __shared__ __align__(16) unsigned char tsm[];
  __shared__ unsigned long long skey[TREE_THREADS + 2];  // keys b0 - 1 .. b1 + 1
  __shared__ unsigned sx[TREE_THREADS];  // far end - b0 | (D + 1) << 16
  const int n = P.n, t = threadIdx.x;
  const int b0 = blockIdx.x * TREE_THREADS;
  const int b1 = min(b0 + TREE_THREADS, n) - 1;
  const int i = b0 + t;
  if(i <= b1)
    skey[t + 1] = K[i];
  if(t == 0)
    skey[0] = b0 > 0 ? K[b0 - 1] : 0ull;
  if(t == 1 || b1 == b0)
    skey[b1 - b0 + 2] = b1 + 1 < n ? K[b1 + 1] : 0ull;
  sx[t] = 0xffffffffu;
  __syncthreads();
  if(i > b1)
    return;
  // bits the keys of two particles share, equal keys told apart by index
  auto shared_bits = [&](unsigned long long x, int a, unsigned long long y, int b) {
    x ^= y;
    return x ? __clzll(x) : 64 + __clz((unsigned)(a ^ b));
  };
  auto D = [&](int a) {  // of a and a + 1, both in the block or next to it
    return a < 0 || a + 1 >= n ? -1 : shared_bits(skey[a - b0 + 1], a, skey[a - b0 + 2], a + 1);
  };
  double rc[3] = {0.0, 0.0, 0.0}, r0[3] = {0.0, 0.0, 0.0};
  if(ALL)
    for(int d = 0; d < dim; ++d) {
      r0[d] = ord_dec(rbits[d]);
      rc[d] = 0.5 * (r0[d] + ord_dec(rbits[3 + d]));
    }
  int l = i, r = i, split = -1;
  int dl = D(i - 1), dr = D(i);
  if(dr >= 64) {
    if(atomicCAS(&st->code, 0, (int)FSPH_ERR_DUPLICATE_KEY) == 0)
      st->index = i;
  }
  if(ordered) {
    // depth in the reference's octree: one level below the deepest prefix
    // shared with a key neighbour (tree_topology.h:957-986)
    const int lead = 64 - (63 / dim) * dim;
    int best = 0;
    if(i > 0)
      best = max(best, (min(dl, 64) - lead) / dim);
    if(i + 1 < n)
      best = max(best, (min(dr, 64) - lead) / dim);
    T.edepth[i] = (unsigned char)(best + 1);
  }
  TreeData<ALL> d;
  tree_leaf<dim, ALL>(P, qpos, i, boxes, mom, rc, r0, d);
  while(true) {
    const bool left = dr > dl;   // the left child of the node split at r
    const int idx = left ? r : l;
    if(split >= 0) {
      d.hi.w = (split << 2) | ((l == split) << 1) | (r == split + 1);
      T.first[idx] = l;
      T.last[idx] = r;
      if(l == split)
        T.leaf_parent[split] = idx;
      else
        T.parent[split] = idx;
      if(r == split + 1)
        T.leaf_parent[split + 1] = idx;
      else
        T.parent[split + 1] = idx;
      tree_node_mem<ALL, true>(T, idx, d, boxes, mom);
      if(l == 0 && r == n - 1) {
        T.parent[0] = -1;
        if(n <= gmax) {
          const int slot = atomicAdd(T.ngroups, 1);
          T.group_first[slot] = 0;
          T.group_last[slot] = r;
          T.group_node[slot] = 0;
        }
        return;
      }
    }
    const int s = left ? r : l - 1;
    const int far = left ? l : r, outer = left ? dl : dr;
    // the parent holds the keys that share at least D(s) bits with that of s:
    // inside the block if neither key around the block does
    bool local = s >= b0 && s < b1;
    if(local) {
      const unsigned long long ks = skey[s - b0 + 1];
      const int ds = left ? dr : dl;
      local = (b0 == 0 || shared_bits(skey[0], b0 - 1, ks, s) < ds) &&
              (b1 == n - 1 || shared_bits(skey[b1 - b0 + 2], b1 + 1, ks, s) < ds);
    }
    int sib_far, sib_outer;
    TreeData<ALL> e;
    if(local) {
      const int q = s - b0;
      tree_slot<ALL, true>(tsm, q + (left ? 0 : TREE_THREADS), d, boxes, mom);
      // the fences order the deposit before the exchange and the sibling's
      // deposit, read below, after it
      __threadfence_block();
      const unsigned prior =
        atomicExch(&sx[q], (unsigned)(far - b0) | ((unsigned)(outer + 1) << 16));
      if(prior == 0xffffffffu)
        return;
      __threadfence_block();
      sib_far = b0 + (int)(prior & 0xffffu);
      sib_outer = (int)(prior >> 16) - 1;
      tree_slot<ALL, false>(tsm, q + (left ? TREE_THREADS : 0), e, boxes, mom);
    }
    else {
      unsigned long long prior;
      const unsigned long long mine =
        (unsigned long long)(unsigned)far | ((unsigned long long)(outer + 1) << 32);
      // releases this child's data, written above, and acquires the sibling's
      asm volatile("atom.acq_rel.gpu.exch.b64 %0, [%1], %2;"
                   : "=l"(prior) : "l"(T.xchg + s), "l"(mine) : "memory");
      if(prior == TREE_EMPTY)
        return;
      T.xchg[s] = TREE_EMPTY;  // for the next build
      sib_far = (int)(unsigned)prior;
      sib_outer = (int)(prior >> 32) - 1;
      const int sib = left ? s + 1 : s;
      if(sib_far == sib)
        tree_leaf<dim, ALL>(P, qpos, sib, boxes, mom, rc, r0, e);
      else
        tree_node_mem<ALL, false>(T, sib, e, boxes, mom);
    }
    tree_merge<ALL>(d, e, boxes, mom);
    if(left) {
      r = sib_far;
      dr = sib_outer;
    }
    else {
      l = sib_far;
      dl = sib_outer;
    }
    split = s;
    // walk groups: maximal subtrees of at most gmax particles
    if(r - l + 1 > gmax) {
      for(int c = 0; c < 2; ++c) {
        const int f = c ? s + 1 : l, e_ = c ? r : s;
        if(e_ - f + 1 <= gmax) {
          const int slot = atomicAdd(T.ngroups, 1);
          T.group_first[slot] = f;
          T.group_last[slot] = e_;
          T.group_node[slot] = f == e_ ? -1 : s + c;
        }
      }
    }
  }
}

// Level of a binary node in the reference's octree: the number of whole
// D-bit digits its keys share.
__device__ __forceinline__ int node_level(const unsigned long long * K,
  const Tree & T, int v, int dim, int lead) {
  return (__clzll(K[T.first[v]] ^ K[T.last[v]]) - lead) / dim;
}

// For each particle: the binary node whose range is its octree parent in
// the reference tree (the topmost binary ancestor of the same level), and
// the reference traversal group containing it -- the octree child of the
// first octree ancestor holding more than 128 particles
// (tree_topology.h:220-235, sub_entities_ = 128 at :2121).
__global__ void k_refgroups(const unsigned long long * K, int n, int dim,
  Tree T, const unsigned long long * rbits, int refboxes) {
  chain_begin();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  // read only when h varies, or for ties in the ordered mode
  if(i >= n || (!refboxes && rbits[6] == rbits[7]))
    return;
  const int lead = 64 - (63 / dim) * dim;
  int p = T.leaf_parent[i];
  int lp = node_level(K, T, p, dim, lead);
  int q = p;
  while(T.parent[q] >= 0 && node_level(K, T, T.parent[q], dim, lead) == lp)
    q = T.parent[q];
  T.opar[i] = q;
  int g = ~i;
  int u = p;
  while(u >= 0) {
    int up = T.parent[u];
    bool octree = up < 0 || node_level(K, T, u, dim, lead) > node_level(K, T, up, dim, lead);
    if(octree) {
      if(T.last[u] - T.first[u] + 1 > 128)
        break;
      g = u;
    }
    u = up;
  }
  T.gref[i] = g;
}

// The node a group's mixed walk starts from: the lowest ancestor whose
// fixed-point box, less one step on every side, holds the group's box grown
// by the largest reach (max h, with the walk's 1e-5 slack and two steps for
// the quantisation).  A radix-tree node holds every particle whose key
// shares its prefix, so its particles' box lies in that Morton cell; a
// particle within reach lies in the grown box, hence a step inside the
// node's box, hence in the cell and in the subtree: the walk below that
// node finds every candidate the walk from the root finds.  (A one-particle
// group, node -1, walks from the root.)
__device__ __forceinline__ int walk_start(const Tree & T, int g, const int4 & glo,
  const int4 & ghi, float hmax, float qs0, float qs1, float qs2, int dim) {
  if(g < 0)
    return 0;
  const float R = hmax * 1.00001f;
  const int rx = (int)ceilf(R / qs0) + 2, ry = (int)ceilf(R / qs1) + 2;
  const int rz = dim == 3 ? (int)ceilf(R / qs2) + 2 : 0;
  int v = T.parent[g];
  while(v > 0) {
    const int4 a = T.qbox[2 * v], b = T.qbox[2 * v + 1];
    bool in = a.x + 1 <= glo.x - rx && b.x - 1 >= ghi.x + rx && a.y + 1 <= glo.y - ry &&
              b.y - 1 >= ghi.y + ry;
    if(dim == 3)
      in = in && a.z + 1 <= glo.z - rz && b.z - 1 >= ghi.z + rz;
    if(in)
      break;
    v = T.parent[v];
  }
  return v < 0 ? 0 : v;
}

// walk_start of every group by a launch of its own, where there are many: in
// the walk its chain of dependent loads (two a level) holds a whole warp, 40 us
// of the Sedov 128^3 walk more than this launch; at 2,250 to 132,651 particles
// the launch costs 3 to 9 us that it does not save.
#define WALK_START_LAUNCH (1 << 18)
__global__ void __launch_bounds__(256) k_walk_start(Tree T, int dim, const float * qscale,
  const unsigned long long * rbits) {
  chain_begin();
  const int ng = *T.ngroups;
  const float hmax = (float)ord_dec(rbits[7]);
  const float qs0 = qscale[0], qs1 = qscale[1], qs2 = dim == 3 ? qscale[2] : 0.f;
  for(int g = blockIdx.x * 256 + threadIdx.x; g < ng; g += gridDim.x * 256) {
    const int v = T.group_node[g];
    T.group_node[g] = v < 0 ? 0
      : walk_start(T, v, T.qbox[2 * v], T.qbox[2 * v + 1], hmax, qs0, qs1, qs2, dim);
  }
}

cudaError_t launch_build_tree(const Launch & L, const Particles & P,
  const PhysParams & pp, Tree & T, int group_max,
  const unsigned long long * rbits, const int4 * qpos, const float * qscale, int ordered,
  DevStatus * st) {
  static std::atomic<unsigned long long> attr_devices{0};
  cudaError_t ae = once_per_device(&attr_devices, []() {
    cudaError_t e = cudaFuncSetAttribute(k_tree<3, true>,
      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tree_smem<true>());
    if(e == cudaSuccess)
      e = cudaFuncSetAttribute(k_tree<2, true>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tree_smem<true>());
    return e;
  });
  if(ae != cudaSuccess)
    return ae;
  const int n = P.n;
#define TREE_LAUNCH(DIM, ALL)                                                \
  chain(L, k_tree<DIM, ALL>, (n + tree_threads<ALL>() - 1) / tree_threads<ALL>(),      \
    tree_threads<ALL>(), tree_smem<ALL>(), P.key, P, T, qpos, \
    rbits, ordered, group_max, st)
  // in the ordered mode and with gravity every run is ALL; else the range
  // words on the device tell
  const bool full_only = ordered || T.gmom;
  if(pp.dim == 3) {
    if(!full_only)
      TREE_LAUNCH(3, false);
    TREE_LAUNCH(3, true);
  }
  else {
    if(!full_only)
      TREE_LAUNCH(2, false);
    TREE_LAUNCH(2, true);
  }
#undef TREE_LAUNCH
  chain(L, k_refgroups, (n + 255) / 256, 256, 0, P.key, n, pp.dim, T, rbits,
    ordered);
  *L.counter += full_only ? 2 : 3;
  if(!ordered && n >= WALK_START_LAUNCH) {
    const int most = (n + 255) / 256;
    chain(L, k_walk_start, most < 152 * 8 ? most : 152 * 8, 256, 0, T, pp.dim, qscale,
      rbits);
    *L.counter += 1;
  }
  return cudaGetLastError();
}

// ---------------------------------------------------- neighbour lists --
// One warp per group (<= 32 particles, lane = member).  The warp walks the
// radix tree with a shared-memory stack, up to 32 nodes per round (one per
// lane), pruning a node when its position box lies farther from the group's
// box than max(h_max(group), h_max(node)) -- a conservative bound, so no
// pair with d <= max(h_a, h_b) is lost.  Surviving particles are staged as
// candidates in shared memory, sorted by (reference octree depth, index)
// and then filtered by every member with the reference predicate
// (tree_geometry.h:265-276, as applied at tree_topology.h:372-379):
//     (dx*dx + dy*dy) + dz*dz <= max(h_a, h_b)^2   in FP64, no FMA.
// The candidate order makes each list come out in the order in which the
// reference's breadth-first walk appends neighbours (by depth, then key).
// Launch shape: one-warp blocks, 20 resident per SM (96 registers, a few
// bytes of spills; 9 KB of shared memory each: 256 candidates and a
// 1,024-entry stack).  Two eight-warp blocks at 122 registers hold 16 warps
// per SM; the 20 here hide more of the walk's fixed-latency stalls and run
// the Sedov 128^3 walk 11 % faster.  At 80 registers (24 warps) the spills
// make it slower.  The FP64 (ordered) walk keeps its larger candidate buffer
// and runs eight blocks per SM.
#ifndef NB_WARPS
#define NB_WARPS 1
#endif
#ifndef NB_STACK
#define NB_STACK 1024
#endif
#define NB_CAND_ORDERED 2048
#ifndef NB_CAND
#define NB_CAND 256
#endif
#ifndef NB_BLOCKS_PER_SM
#define NB_BLOCKS_PER_SM 20
#endif
#define NB_ORDERED_BLOCKS_PER_SM 8
// The mixed walk comes in two variants, one for runs in which every h is
// equal and one for varying h; both are launched and each returns at once
// unless the device's range words select it.  The equal-h variant keeps
// none of the reference node-test state (FP64 group box, reference group,
// FP32 centre) and no candidate h, so it fits more warps per SM.
#ifndef NB_UNI_BLOCKS_PER_SM
#define NB_UNI_BLOCKS_PER_SM 24
#endif
#ifndef NB_UNI_CAND
#define NB_UNI_CAND 256
#endif
enum { NB_MODE_UNI = 0, NB_MODE_VAR = 1, NB_MODE_ORDERED = 2 };

__device__ __forceinline__ void warp_bitonic(unsigned long long * a, int m,
  int lane) {
  int S = 32;
  while(S < m)
    S <<= 1;
  for(int i = m + lane; i < S; i += 32)
    a[i] = ~0ull;
  __syncwarp();
  for(int k = 2; k <= S; k <<= 1)
    for(int j = k >> 1; j > 0; j >>= 1) {
      for(int i = lane; i < S; i += 32) {
        int l = i ^ j;
        if(l > i) {
          unsigned long long x = a[i], y = a[l];
          bool up = (i & k) == 0;
          if((x > y) == up) {
            a[i] = y;
            a[l] = x;
          }
        }
      }
      __syncwarp();
    }
}

// intersects_sphere_box (tree_geometry.h:329-341 in 3D, :219-227 in 2D)
__device__ __forceinline__ bool sphere_box(const double * b2, double c0,
  double c1, double c2, double r, int dim) {
  if(dim == 3) {
    double x0 = c0 < b2[4] ? c0 : b2[4];
    double x1 = c1 < b2[5] ? c1 : b2[5];
    double x2 = c2 < b2[6] ? c2 : b2[6];
    x0 = x0 < b2[0] ? b2[0] : x0;
    x1 = x1 < b2[1] ? b2[1] : x1;
    x2 = x2 < b2[2] ? b2[2] : x2;
    double dist = (x0 - c0) * (x0 - c0) + (x1 - c1) * (x1 - c1) +
                  (x2 - c2) * (x2 - c2);
    return dist <= r * r;
  }
  double y0 = b2[4] < c0 ? b2[4] : c0;
  double y1 = b2[5] < c1 ? b2[5] : c1;
  double x0 = b2[0] < y0 ? y0 : b2[0];
  double x1 = b2[1] < y1 ? y1 : b2[1];
  double sum = 0;
  sum += (x0 - c0) * (x0 - c0);
  sum += (x1 - c1) * (x1 - c1);
  return sqrt(sum) - r <= 2.220446049250313e-16 * 10.;
}

// intersects_box_box (tree_geometry.h:306-314, :201-207)
__device__ __forceinline__ bool box_box(const double * a, const double * b,
  int dim) {
  bool sep = a[4] < b[0] || a[5] < b[1] || b[4] < a[0] || b[5] < a[1];
  if(dim == 3)
    sep = sep || a[6] < b[2] || b[6] < a[2];
  return !sep;
}

// FP32 versions of the two node tests, for answers that are certain.  Boxes
// are the outward-rounded FP32 copies (fbox2) relative to the range's lower
// corner and points are FP32 roundings of the same relative coordinates, so
// every FP32 box face and point lies within `tol` (a few FP32 ulps of the
// range's extent) of its FP64 value; an answer that a perturbation of that
// size could flip returns -1 and the caller runs the FP64 test.
__device__ __forceinline__ int box_box_f(const float4 & alo, const float4 & ahi,
  const float4 & blo, const float4 & bhi, int dim, float tol) {
  float g = fmaxf(fmaxf(blo.x - ahi.x, alo.x - bhi.x),
    fmaxf(blo.y - ahi.y, alo.y - bhi.y));
  if(dim == 3)
    g = fmaxf(g, fmaxf(blo.z - ahi.z, alo.z - bhi.z));
  if(g > 0.f)  // outer boxes apart: the exact boxes are apart
    return 0;
  if(g < -2.f * tol)  // overlap by more than both roundings on every axis
    return 1;
  return -1;
}

__device__ __forceinline__ int sphere_box_f(const float4 & lo,
  const float4 & hi, float cx, float cy, float cz, float r, int dim,
  float tol) {
  const float dx = fmaxf(0.f, fmaxf(lo.x - cx, cx - hi.x));
  const float dy = fmaxf(0.f, fmaxf(lo.y - cy, cy - hi.y));
  const float dz = dim == 3 ? fmaxf(0.f, fmaxf(lo.z - cz, cz - hi.z)) : 0.f;
  const float d = sqrtf(dx * dx + dy * dy + dz * dz);
  // box faces and the point each within tol per axis; 1e-6 relative covers
  // the FP32 rounding of the distance and of r
  const float slack = 3.5f * tol + 1e-6f * (d + r) + 3e-15f;
  if(d + slack < r)
    return 1;
  if(d - slack > r)
    return 0;
  return -1;
}

// With varying h the reference's walk drops a candidate b of particle a
// unless the box of b's octree parent passes both node tests against a's
// traversal group G (tree_topology.h:323-355): box-box with G's box when G
// is a node, and sphere-box with at least one member of G.  When every h
// is equal only the box-box test can fail, and only for a pair whose
// separation along an axis ties with h to rounding.  Each
// test is decided in FP32 first and in FP64 (box_box, sphere_box) only when
// the FP32 answer is not certain, so the answers are the FP64 ones.
//
// The box-box half depends on G and b's octree parent alone: the walk asks it
// once per candidate and traversal group, a lane per candidate.
__device__ __forceinline__ bool ref_box_test(const Tree & T, int dim, int ob, int gnode,
  const float4 & glo, const float4 & ghi, float tol) {
  const int r = box_box_f(T.fbox2[2 * ob], T.fbox2[2 * ob + 1], glo, ghi, dim, tol);
  if(r >= 0)
    return r != 0;
  const double * b2 = (const double *)&T.box2[ob];
  const double * g2 = (const double *)&T.box2[gnode];
  double bb[8], gg[8];
  for(int k = 0; k < 8; ++k) {
    bb[k] = b2[k];
    gg[k] = g2[k];
  }
  return box_box(bb, gg, dim);
}

// The sphere-box half for the pair (a, b).  Particle a's own sphere passes
// whenever d(a, b) <= max(h_a, h_b) and h_b <= 2 h_a: the parent's box holds
// the cube of half-width h_b / 2 about b, hence the ball of that radius, so it
// is no farther from a than d - h_b / 2 <= max(h_a - h_b / 2, h_b / 2).  The
// caller skips the test for h_b <= 1.99 h_a, which leaves rounding its room.
__device__ bool ref_sphere_test(const Tree & T, const double * X, const double * Y,
  const double * Z, const double * H, int dim, int b, int a, int gnode, const double * rlo,
  float tol) {
  const int ob = T.opar[b];
  const float4 blo = T.fbox2[2 * ob], bhi = T.fbox2[2 * ob + 1];
  const double * b2 = (const double *)&T.box2[ob];
  const int first = gnode < 0 ? a : T.first[gnode], last = gnode < 0 ? a : T.last[gnode];
  // a first: the likeliest, and the only one where G is a single particle
  for(int j = first - 1; j <= last; ++j) {
    const int k = j < first ? a : j;
    if(j >= first && k == a)
      continue;
    const double xk = X[k], yk = Y[k], zk = dim == 3 ? Z[k] : 0.0, hk = H[k];
    const int t = sphere_box_f(blo, bhi, (float)(xk - rlo[0]), (float)(yk - rlo[1]),
      dim == 3 ? (float)(zk - rlo[2]) : 0.f, (float)hk, dim, tol);
    if(t == 1)
      return true;
    if(t < 0) {
      double bb[8];
      for(int q = 0; q < 8; ++q)
        bb[q] = b2[q];
      if(sphere_box(bb, xk, yk, zk, hk, dim))
        return true;
    }
  }
  return false;
}

// both halves (equal-h ties in the ordered mode, groups of many classes)
__device__ bool ref_node_tests(const Tree & T, const double * X, const double * Y,
  const double * Z, const double * H, int dim, int b, int a, int gnode, const double * rlo,
  float tol) {
  if(gnode >= 0 && !ref_box_test(T, dim, T.opar[b], gnode, T.fbox2[2 * gnode],
                     T.fbox2[2 * gnode + 1], tol))
    return false;
  return ref_sphere_test(T, X, Y, Z, H, dim, b, a, gnode, rlo, tol);
}

// Conservative pruning test in the fixed-point space: the separation of
// two boxes per axis, less one quantisation step (each coordinate is
// within half a step of the true one), against max(h) with 1e-5 slack.
__device__ __forceinline__ bool box_near(int4 glo, int4 ghi, float hg,
  int4 lo, int4 hi, float hn, float s0, float s1, float s2) {
  int sx = max(0, max(lo.x - ghi.x, glo.x - hi.x) - 1);
  int sy = max(0, max(lo.y - ghi.y, glo.y - hi.y) - 1);
  int sz = max(0, max(lo.z - ghi.z, glo.z - hi.z) - 1);
  float fx = (float)sx * s0, fy = (float)sy * s1, fz = (float)sz * s2;
  float R = fmaxf(hg, hn);
  return fx * fx + fy * fy + fz * fz <= R * R * 1.00001f;
}

// One warp per group (<= 32 particles, lane = member).  The warp walks the
// radix tree with a shared-memory stack, up to 32 nodes per round (one per
// lane), pruning a node when its box lies farther from the group's box than
// max(h_max(group), h_max(node)) -- conservative, so no pair with
// d <= max(h_a, h_b) is lost.  Surviving particles are staged as candidates
// in shared memory and filtered by every member with the reference
// predicate (tree_geometry.h:265-276, as applied at tree_topology.h:372-379),
//     (dx*dx + dy*dy) + dz*dz <= max(h_a, h_b)^2   in FP64, no FMA,
// decided first in FP32 from the fixed-point positions with a margin well
// above that estimate's error; only pairs inside the margin pay the FP64
// test.  ORDERED (the FP64 path) sorts the candidates by (reference octree
// depth, index) before filtering, so each list comes out in the order in
// which the reference's breadth-first walk appends neighbours; when the
// candidates of a group did not fit one chunk, every member's list is
// sorted by the same key at the end.
template<int MODE>
__global__ void __launch_bounds__(NB_WARPS * 32,
  MODE == NB_MODE_ORDERED ? NB_ORDERED_BLOCKS_PER_SM
  : MODE == NB_MODE_UNI ? NB_UNI_BLOCKS_PER_SM : NB_BLOCKS_PER_SM) k_neighbors(
  Particles P, Tree T, Lists Ls, DevStatus * st, int dim,
  const unsigned long long * rbits, Packed K) {
  chain_begin();
  constexpr bool ORDERED = MODE == NB_MODE_ORDERED;
  constexpr bool UNI = MODE == NB_MODE_UNI;
  if(!ORDERED && UNI != (rbits[6] == rbits[7]))
    return;  // the other variant's run
  extern __shared__ __align__(16) unsigned char smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int CAND = ORDERED ? NB_CAND_ORDERED : UNI ? NB_UNI_CAND : NB_CAND;
  const int cap = CAND;
  unsigned long long * ckey = nullptr;
  float * cxs = nullptr;  // candidates as SoA: minus their position relative
  float * cys = nullptr;  // to the group box corner, h and particle index,
  float * czs = nullptr;  // so the filter reads consecutive pairs as float2
  float * chs = nullptr;  // (h squared)
  int * cidx = nullptr;
  unsigned char * cflag = nullptr;  // bit k: passes class k's box-box test (varying h)
  int * stack;
  if(ORDERED) {
    ckey = (unsigned long long *)smem + (size_t)w * NB_CAND_ORDERED;
    stack = (int *)(smem + (size_t)NB_WARPS * NB_CAND_ORDERED * 8) + w * NB_STACK;
    cflag = smem + (size_t)NB_WARPS * (NB_CAND_ORDERED * 8 + NB_STACK * 4) +
            (size_t)w * NB_CAND_ORDERED;
  }
  else {
    constexpr int NA = UNI ? 4 : 5;  // arrays per candidate (no h with UNI)
    float * base = (float *)smem + (size_t)w * NA * CAND;
    cxs = base;
    cys = base + CAND;
    czs = base + 2 * CAND;
    chs = UNI ? nullptr : base + 3 * CAND;
    cidx = (int *)(base + (NA - 1) * CAND);
    stack = (int *)(smem + (size_t)NB_WARPS * CAND * NA * 4) + w * NB_STACK;
    if(!UNI)
      cflag = smem + (size_t)NB_WARPS * (CAND * NA * 4 + NB_STACK * 4) + (size_t)w * CAND;
  }
  const unsigned lt = lanemask_lt();
  const double * X = P.f[F_X];
  const double * Y = P.f[F_Y];
  const double * Z = P.f[F_Z];
  const double * H = P.f[F_H];
  const int ngroups = *T.ngroups;
  const int maxnb = Ls.maxnb;
  const bool nonuni = !UNI && rbits[6] != rbits[7];
  const float qs0 = K.qscale[0], qs1 = K.qscale[1], qs2 = dim == 3 ? K.qscale[2] : 0.f;
  const float qmax = fmaxf(qs0, fmaxf(qs1, qs2));
  const float hglob = (float)ord_dec(rbits[7]);
  double rlo[3] = {0.0, 0.0, 0.0};
  float ext = 0.f;
  for(int d = 0; d < dim; ++d) {
    rlo[d] = ord_dec(rbits[d]);
    ext = fmaxf(ext, (float)(ord_dec(rbits[3 + d]) - rlo[d]));
  }
  // FP32 boxes and points lie within a few ulps of the range's extent of
  // their FP64 values (outward rounding of the boxes, nearest of points)
  const float ftol = 4e-7f * ext;
  for(int g = blockIdx.x * NB_WARPS + w; g < ngroups;
      g += gridDim.x * NB_WARPS) {
    const int gf = T.group_first[g], gl = T.group_last[g];
    const bool mem = lane <= gl - gf;
    const int a = gf + lane;
    int4 qa = make_int4(0, 0, 0, 0);
    if(mem)
      qa = K.qpos[a];
    const float haf = __int_as_float(qa.w);
    // the members' traversal groups (they exist with varying h, and in the
    // ordered mode: k_tree, k_refgroups), told apart as up to eight classes:
    // lane k holds class k's node, every member its class
    int gnode = -1, cls = 0, cnode = -1, ncls = 0;
    if(!UNI && (nonuni || ORDERED)) {
      if(mem)
        gnode = max(T.gref[a], -1);
      unsigned left = nonuni ? __ballot_sync(FULL, mem) : 0u;
      while(left) {
        const int node = __shfl_sync(FULL, gnode, __ffs(left) - 1);
        const unsigned same = __ballot_sync(FULL, mem && gnode == node) & left;
        if((same >> lane) & 1u)
          cls = ncls;
        if(lane == ncls)
          cnode = node;
        left &= ~same;
        ++ncls;
      }
    }
    int4 glo = mem ? qa : make_int4(0x7fffffff, 0x7fffffff, 0x7fffffff, 0);
    int4 ghi = mem ? qa : make_int4(-1, -1, -1, 0);
    float hg = haf;
    for(int o = 16; o; o >>= 1) {
      glo.x = min(glo.x, __shfl_xor_sync(FULL, glo.x, o));
      glo.y = min(glo.y, __shfl_xor_sync(FULL, glo.y, o));
      glo.z = min(glo.z, __shfl_xor_sync(FULL, glo.z, o));
      ghi.x = max(ghi.x, __shfl_xor_sync(FULL, ghi.x, o));
      ghi.y = max(ghi.y, __shfl_xor_sync(FULL, ghi.y, o));
      ghi.z = max(ghi.z, __shfl_xor_sync(FULL, ghi.z, o));
      hg = fmaxf(hg, __shfl_xor_sync(FULL, hg, o));
    }
    int cnt = 0;
    int sp = 1;
    int ncand = 0;
    bool chunked = false;
    int start = 0;
    if(!ORDERED) {
      start = T.group_node[g];
      if(P.n < WALK_START_LAUNCH)
        start = walk_start(T, start, glo, ghi, hglob, qs0, qs1, qs2, dim);
    }
    if(lane == 0)
      stack[0] = ORDERED ? 0 : T.qbox[2 * start + 1].w;
    __syncwarp();
    while(sp > 0) {
      const int k = sp < 32 ? sp : 32;
      const bool act = lane < k;
      int node = act ? stack[sp - 1 - lane] : 0;
      __syncwarp();
      sp -= k;
      if(!ORDERED) {
        // The stack holds the split codes of accepted nodes (split << 2 |
        // left leaf << 1 | right leaf, as qbox's .w keeps them); a round
        // tests both children of each -- nodes split and split + 1, whose
        // boxes are adjacent in qbox, or a leaf's position -- pushes the
        // accepted inner children's codes and stages the accepted leaves, so
        // every level of the descent costs one round instead of two.
        int4 cl[2], chh[2];
        bool lf[2] = {false, false}, ca[2] = {false, false};
        int split = 0;
        if(act) {
          const int code = node;
          split = code >> 2;
          lf[0] = (code & 2) != 0;
          lf[1] = (code & 1) != 0;
          for(int c = 0; c < 2; ++c) {
            if(lf[c]) {
              cl[c] = chh[c] = K.qpos[split + c];
            }
            else {
              cl[c] = T.qbox[2 * (split + c)];
              chh[c] = T.qbox[2 * (split + c) + 1];
            }
          }
          for(int c = 0; c < 2; ++c)
            ca[c] = box_near(glo, ghi, hg, cl[c], chh[c], __int_as_float(cl[c].w), qs0,
              qs1, qs2);
        }
        const int cc[2] = {lf[0] ? ~split : chh[0].w, lf[1] ? ~(split + 1) : chh[1].w};
        const unsigned bi0 = __ballot_sync(FULL, ca[0] && !lf[0]);
        const unsigned bi1 = __ballot_sync(FULL, ca[1] && !lf[1]);
        const unsigned bl0 = __ballot_sync(FULL, ca[0] && lf[0]);
        const unsigned bl1 = __ballot_sync(FULL, ca[1] && lf[1]);
        const int npush = __popc(bi0) + __popc(bi1);
        if(sp + npush > NB_STACK) {
          if(lane == 0 && atomicCAS(&st->code, 0, (int)FSPH_ERR_STACK_OVERFLOW) == 0)
            st->index = gf;
          break;
        }
        if(ca[0] && !lf[0])
          stack[sp + __popc(bi0 & lt)] = cc[0];
        if(ca[1] && !lf[1])
          stack[sp + __popc(bi0) + __popc(bi1 & lt)] = cc[1];
        sp += npush;
        // a node's two leaves go side by side (lane order, left first): the
        // lists keep the tree's index order, which the pair passes' gathers
        // share between the lanes of a group
        const int lfirst = ncand + __popc(bl0 & lt) + __popc(bl1 & lt);
        for(int c = 0; c < 2; ++c) {
          if(ca[c] && lf[c]) {
            const int pos = lfirst + (c && ca[0] && lf[0] ? 1 : 0);
            const int4 ql = cl[c];
            // minus the position relative to the group box corner, in FP32
            cxs[pos] = -((float)(ql.x - glo.x) * qs0);
            cys[pos] = -((float)(ql.y - glo.y) * qs1);
            czs[pos] = -((float)(ql.z - glo.z) * qs2);
            if(!UNI)
              chs[pos] = __int_as_float(ql.w) * __int_as_float(ql.w);
            cidx[pos] = ~cc[c];
          }
        }
        ncand += __popc(bl0) + __popc(bl1);
      }
      else {
      bool acc = false;
      const bool leaf = node < 0;
      int4 ql = make_int4(0, 0, 0, 0);
      int code = 0;
      if(act) {
        if(!leaf) {
          const int4 lo = T.qbox[2 * node], hi = T.qbox[2 * node + 1];
          code = hi.w;
          acc = box_near(glo, ghi, hg, lo, hi, __int_as_float(lo.w), qs0, qs1, qs2);
        }
        else {
          ql = K.qpos[~node];
          acc = box_near(glo, ghi, hg, ql, ql, __int_as_float(ql.w), qs0, qs1, qs2);
        }
      }
      const unsigned bi = __ballot_sync(FULL, acc && !leaf);
      const unsigned bl = __ballot_sync(FULL, acc && leaf);
      const int npush = 2 * __popc(bi);
      if(sp + npush > NB_STACK) {
        if(lane == 0 && atomicCAS(&st->code, 0, (int)FSPH_ERR_STACK_OVERFLOW) == 0)
          st->index = gf;
        break;
      }
      if(acc && !leaf) {
        const int pos = sp + 2 * __popc(bi & lt);
        const int split = code >> 2;
        stack[pos] = (code & 1) ? ~(split + 1) : split + 1;
        stack[pos + 1] = (code & 2) ? ~split : split;
      }
      sp += npush;
      if(acc && leaf) {
        const int j = ~node;
        const int pos = ncand + __popc(bl & lt);
        ckey[pos] = ((unsigned long long)T.edepth[j] << 32) | (unsigned)j;
      }
      ncand += __popc(bl);
      }
      __syncwarp();
      const bool last = (sp == 0);
      if(ncand > cap - (ORDERED ? 33 : 65) || (last && ncand > 0)) {
        if(!last)
          chunked = true;
        if(ORDERED)
          warp_bitonic(ckey, ncand, lane);
        float rc = hg;  // varying h: the largest h among members and candidates
        if(!ORDERED) {
          // an even count (UNI) or whole batches of 32, with candidates that
          // can never pass
          const int full = UNI ? (ncand + 1) & ~1 : (ncand + 31) & ~31;
          for(int c = ncand + lane; c < full; c += 32) {
            cxs[c] = 1e30f;
            cys[c] = 1e30f;
            czs[c] = 1e30f;
            if(!UNI)
              chs[c] = 0.f;
            cidx[c] = -1;
          }
        }
        if(!UNI && nonuni) {
          if(!ORDERED) {
            float hc = 0.f;
            for(int c = lane; c < ncand; c += 32)
              hc = fmaxf(hc, chs[c]);
            for(int o = 16; o; o >>= 1)
              hc = fmaxf(hc, __shfl_xor_sync(FULL, hc, o));
            rc = fmaxf(rc, sqrtf(hc) * 1.000001f);
          }
          // the reference's box-box test, a lane per candidate, for every class
          // of members (the classes beyond the eighth test their own pairs)
          for(int k = 0; k < ncls && k < 8; ++k) {
            const int node = __shfl_sync(FULL, cnode, k);
            float4 nlo = make_float4(0.f, 0.f, 0.f, 0.f), nhi = nlo;
            if(node >= 0) {
              nlo = T.fbox2[2 * node];
              nhi = T.fbox2[2 * node + 1];
            }
            for(int c = lane; c < ncand; c += 32) {
              const int bc = ORDERED ? (int)(ckey[c] & 0xffffffffu) : cidx[c];
              const bool ok =
                node < 0 || ref_box_test(T, dim, T.opar[bc], node, nlo, nhi, ftol);
              cflag[c] = (unsigned char)((k ? cflag[c] : 0u) | ((unsigned)ok << k));
            }
          }
          __syncwarp();
        }
        __syncwarp();
        if(mem) {
          const double xa = X[a], ya = Y[a], za = dim == 3 ? Z[a] : 0.0, ha = H[a];
          int * out = Ls.idx + list_slot(a, 0, maxnb);
          // this member relative to the same corner
          const float ax = (float)(qa.x - glo.x) * qs0;
          const float ay = (float)(qa.y - glo.y) * qs1;
          const float az = (float)(qa.z - glo.z) * qs2;
          // largest extent of the group box: with the walk radius it bounds
          // the magnitude of every relative coordinate below
          const float lg = fmaxf((float)(ghi.x - glo.x) * qs0,
            fmaxf((float)(ghi.y - glo.y) * qs1, (float)(ghi.z - glo.z) * qs2));
          // The FP32 estimate t = d^2 - r^2 decides a pair only when |t|
          // exceeds a margin well above its error bound: fixed-point
          // quantisation (one step per axis), two roundings of each relative
          // coordinate (|value| <= lg + max h, as the walk accepted the
          // candidate), the squares and the sum (~2e-6 r^2).  Inside the
          // margin the exact FP64 predicate decides.
          const float kq = 16.f * qmax + 4e-6f * (lg + fmaxf(hg, hglob));
          auto decide = [&](float t, float mg, int b) -> bool {
            if(fabsf(t) > mg)
              return t < 0.f;
            const double xb = X[b], yb = Y[b], hbd = H[b];
            const double zb = dim == 3 ? Z[b] : 0.0;
            double dx = xa - xb, dy = ya - yb, dz = za - zb;
            double d2 = dx * dx + dy * dy;
            if(dim == 3)
              d2 = d2 + dz * dz;
            double r = ha < hbd ? hbd : ha;
            return d2 <= r * r;
          };
          // what the reference's node tests keep of the pairs within reach
          // (varying h): class flag, and the sphere test where h_b is far
          // above h_a or h is so small beside the range that rounding counts
          const bool hsmall = haf < 1e-6f * ext;
          auto refok = [&](int c, int b, float hb) {
            if(cls >= 8)
              return ref_node_tests(T, X, Y, Z, H, dim, b, a, gnode, rlo, ftol);
            if(!((cflag[c] >> cls) & 1u))
              return false;
            return (!hsmall && hb <= 1.99f * haf) ||
                   ref_sphere_test(T, X, Y, Z, H, dim, b, a, gnode, rlo, ftol);
          };
          // Equal h: the node tests can only drop a pair whose separation
          // along some axis ties with h, where the rounding of x +- h/2 in
          // the boxes decides (box-box, tree_topology.h:326-330).  In the
          // ordered mode such pairs (none off a lattice) take the tests,
          // decided exactly; the mixed path keeps them (W(h) = 0 for the
          // compactly supported kernels).
          auto tie = [&](float fx, float fy, float fz, float rf) {
            return fmaxf(fabsf(fx), fmaxf(fabsf(fy), fabsf(fz))) >= rf - kq;
          };
          auto append = [&](int b) {
            if(cnt < maxnb)
              out[slot_off(cnt)] = b;
            ++cnt;
          };
          if(ORDERED) {
            for(int c = 0; c < ncand; ++c) {
              const int b = (int)(ckey[c] & 0xffffffffu);
              const int4 qb = K.qpos[b];
              const float fx = (float)(qa.x - qb.x) * qs0;
              const float fy = (float)(qa.y - qb.y) * qs1;
              const float fz = (float)(qa.z - qb.z) * qs2;
              const float d2f = fx * fx + fy * fy + fz * fz;
              const float rf = fmaxf(haf, __int_as_float(qb.w));
              const float t = d2f - rf * rf;
              const float mg = rf * (4e-5f * rf + kq);
              if(decide(t, mg, b) &&
                 (nonuni ? refok(c, b, __int_as_float(qb.w))
                         : !tie(fx, fy, fz, rf) ||
                             ref_node_tests(T, X, Y, Z, H, dim, b, a, gnode, rlo, ftol)))
                append(b);
            }
          }
          else if(UNI) {
            // every h is equal: r and the margin are constants of the group
            // and the predicate decides (ties included, see tie); two
            // candidates per step in packed FP32x2.  Collecting the accepted
            // ones of 32 candidates in a mask first measured the same at Sedov
            // 128^3 (1.47 ms) and slower on small sets (52 against 34 us at
            // 2,250 particles in 2D): a batch of neighbours in space is hit
            // as a whole, so its append loop is as long as the batch.
            const float2 ax2 = make_float2(ax, ax), ay2 = make_float2(ay, ay);
            const float2 az2 = make_float2(az, az);
            const float r2 = haf * haf;
            const float2 nr2 = make_float2(-r2, -r2);
            const float mg = haf * (4e-5f * haf + kq);
            for(int c = 0; c < ncand; c += 2) {
              const float2 nx = *(const float2 *)&cxs[c];
              const float2 ny = *(const float2 *)&cys[c];
              const float2 nz = *(const float2 *)&czs[c];
              const int2 id = *(const int2 *)&cidx[c];
              const float2 dx = __fadd2_rn(ax2, nx);
              const float2 dy = __fadd2_rn(ay2, ny);
              const float2 dz = __fadd2_rn(az2, nz);
              float2 d2 = __fmul2_rn(dx, dx);
              d2 = __ffma2_rn(dy, dy, d2);
              d2 = __ffma2_rn(dz, dz, d2);
              const float2 t = __fadd2_rn(d2, nr2);
              bool in0 = t.x < 0.f, in1 = t.y < 0.f;
              if(fabsf(t.x) <= mg)
                in0 = decide(t.x, mg, id.x);
              if(fabsf(t.y) <= mg && id.y >= 0)
                in1 = decide(t.y, mg, id.y);
              if(in0)
                append(id.x);
              if(in1)
                append(id.y);
            }
          }
          else {
            // Batches of 32 candidates: the sign bits of t = d^2 -
            // max(h_a, h_b)^2 make a mask (a funnel shift per candidate), the
            // smallest |t| beyond its margin tells whether a pair of the batch
            // needs the exact predicate, and the set bits are appended.  Here
            // an accepted pair has more to do (the class flag, h_b), so taking
            // only those through the append loop pays: 5.1 against 7.4 ms
            // candidate by candidate on the 4M star.
            const float2 ax2 = make_float2(ax, ax), ay2 = make_float2(ay, ay);
            const float2 az2 = make_float2(az, az);
            const float r2 = haf * haf, mgc = kq * rc;
            for(int c0 = 0; c0 < ncand; c0 += 32) {
              unsigned mask = 0u;
              float slack = 1e38f;
#pragma unroll 2
              for(int c = c0; c < c0 + 32; c += 4) {
                const float4 nx = *(const float4 *)&cxs[c];
                const float4 ny = *(const float4 *)&cys[c];
                const float4 nz = *(const float4 *)&czs[c];
                const float4 hb2 = *(const float4 *)&chs[c];
                const float hh[4] = {hb2.x, hb2.y, hb2.z, hb2.w};
                float t[4];
                for(int q = 0; q < 2; ++q) {
                  const float2 dx = __fadd2_rn(ax2, q ? make_float2(nx.z, nx.w)
                                                      : make_float2(nx.x, nx.y));
                  const float2 dy = __fadd2_rn(ay2, q ? make_float2(ny.z, ny.w)
                                                      : make_float2(ny.x, ny.y));
                  const float2 dz = __fadd2_rn(az2, q ? make_float2(nz.z, nz.w)
                                                      : make_float2(nz.x, nz.y));
                  float2 d2 = __fmul2_rn(dx, dx);
                  d2 = __ffma2_rn(dy, dy, d2);
                  d2 = __ffma2_rn(dz, dz, d2);
                  t[2 * q] = d2.x;
                  t[2 * q + 1] = d2.y;
                }
                for(int q = 0; q < 4; ++q) {
                  // margin 4e-5 r^2 + kq r, r at most rc
                  const float rr = fmaxf(r2, hh[q]);
                  t[q] -= rr;
                  slack = fminf(slack, __fmaf_rn(-4e-5f, rr, fabsf(t[q])));
                  mask = __funnelshift_l(__float_as_uint(t[q]), mask, 1);
                }
              }
              if(slack <= mgc || !(rc < 1e18f)) {
                // some pair lies inside the margin, or the squares may overflow
                // and t be a NaN, which the slack does not show: candidate by
                // candidate
                mask = 0u;
                for(int c = c0; c < c0 + 32 && c < ncand; ++c) {
                  const float dx = ax + cxs[c], dy = ay + cys[c], dz = az + czs[c];
                  const float rf = fmaxf(haf, sqrtf(chs[c]));
                  const float t = dx * dx + dy * dy + dz * dz - rf * rf;
                  if(decide(t, rf * (4.1e-5f * rf + kq), cidx[c]))
                    mask |= 0x80000000u >> (c - c0);
                }
              }
              while(mask) {
                const int k = __clz(mask);
                mask &= ~(0x80000000u >> k);
                const int b = cidx[c0 + k];
                if(refok(c0 + k, b, sqrtf(chs[c0 + k])))
                  append(b);
              }
            }
          }
        }
        __syncwarp();
        ncand = 0;
      }
    }
    if(!ORDERED && P.n <= LIST_STAT_MAX) {
      const unsigned kept = mem ? (unsigned)min(cnt, maxnb) : 0u;
      const unsigned longest = __reduce_max_sync(FULL, kept);
      const unsigned pairs = __reduce_add_sync(FULL, kept);
      if(lane == 0) {
        atomicMax(&Ls.stat[0], longest);
        atomicAdd(&Ls.stat[1], pairs);
      }
    }
    if(mem) {
      if(cnt > maxnb) {
        if(atomicCAS(&st->code, 0, (int)FSPH_ERR_LIST_OVERFLOW) == 0)
          st->index = a;
        cnt = maxnb;
      }
      Ls.cnt[a] = cnt;
      {
        // pad the last chunk of four with the particle itself
        int * o = Ls.idx + list_slot(a, 0, maxnb);
        for(int k = cnt; k < ((cnt + 3) & ~3); ++k)
          o[slot_off(k)] = a;
      }
      if(ORDERED && chunked) {
        // the candidates came in several sorted chunks: put the whole list
        // in (reference octree depth, index) order (Shell sort, Ciura gaps)
        int * out = Ls.idx + list_slot(a, 0, maxnb);
        auto key = [&](int b) {
          return ((unsigned long long)T.edepth[b] << 32) | (unsigned)b;
        };
        const int gaps[8] = {701, 301, 132, 57, 23, 10, 4, 1};
        for(int gi = 0; gi < 8; ++gi) {
          const int gap = gaps[gi];
          for(int i = gap; i < cnt; ++i) {
            const int v = out[slot_off(i)];
            const unsigned long long kv = key(v);
            int j = i;
            while(j >= gap && key(out[slot_off(j - gap)]) > kv) {
              out[slot_off(j)] = out[slot_off(j - gap)];
              j -= gap;
            }
            out[slot_off(j)] = v;
          }
        }
      }
    }
  }
}

cudaError_t launch_neighbors(const Launch & L, const Particles & P,
  const PhysParams & pp, const Tree & T, Lists & Ls, DevStatus * st, int nsm,
  const unsigned long long * rbits, const Packed & K, int ordered) {
  const size_t smem_o = (size_t)NB_WARPS * NB_CAND_ORDERED * 9 +
                        (size_t)NB_WARPS * NB_STACK * 4;
  const size_t smem_v = (size_t)NB_WARPS * NB_CAND * 21 +
                        (size_t)NB_WARPS * NB_STACK * 4;
  const size_t smem_u = (size_t)NB_WARPS * NB_UNI_CAND * 16 +
                        (size_t)NB_WARPS * NB_STACK * 4;
  static std::atomic<unsigned long long> attr_devices{0};
  cudaError_t ae = once_per_device(&attr_devices, [&]() {
    cudaError_t e = cudaFuncSetAttribute(k_neighbors<NB_MODE_ORDERED>,
      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_o);
    if(e == cudaSuccess)
      e = cudaFuncSetAttribute(k_neighbors<NB_MODE_VAR>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_v);
    if(e == cudaSuccess)
      e = cudaFuncSetAttribute(k_neighbors<NB_MODE_UNI>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_u);
    return e;
  });
  if(ae != cudaSuccess)
    return ae;
  const int maxb0 = (P.n + NB_WARPS * 32 - 1) / (NB_WARPS * 32) * 8;
  const int maxb = maxb0 > 0 ? maxb0 : 1;
  auto grid = [&](int per_sm) { return nsm * per_sm < maxb ? nsm * per_sm : maxb; };
  if(ordered) {
    chain(L, k_neighbors<NB_MODE_ORDERED>, grid(NB_ORDERED_BLOCKS_PER_SM), NB_WARPS * 32,
      smem_o, P, T, Ls, st, pp.dim, rbits, K);
    *L.counter += 1;
  }
  else {
    // both variants; the one the range words do not select returns at once
    chain(L, k_neighbors<NB_MODE_UNI>, grid(NB_UNI_BLOCKS_PER_SM), NB_WARPS * 32, smem_u,
      P, T, Ls, st, pp.dim, rbits, K);
    chain(L, k_neighbors<NB_MODE_VAR>, grid(NB_BLOCKS_PER_SM), NB_WARPS * 32, smem_v,
      P, T, Ls, st, pp.dim, rbits, K);
    *L.counter += 2;
  }
  return cudaGetLastError();
}

}  // namespace fsph

// ------------------------------------------- allocation-free key sort --
// Range, Morton keys and the radix sort of fsph_update_iteration for
// callers that must not allocate device memory themselves -- for example a
// host application whose device memory is owned by its own pool allocator,
// or a time-critical loop in which cudaMalloc/cudaFree (which may
// synchronise the device) are not acceptable.  Its scratch (range words,
// ping-pong keys and indices, digit histogram) is this file-scope array,
// sized for FSPH_NOALLOC_SORT_MAX particles: 12,846,336 bytes that every
// GPU loading the library holds until the process exits.
#define FSPH_NOALLOC_SORT_MAX (1 << 20)
#define NOALLOC_RANGE_BYTES 256
static_assert(RANGE_WORDS * 8 <= NOALLOC_RANGE_BYTES &&
                RANGE_PART <= FSPH_NOALLOC_SORT_MAX, "range scratch");
#define NOALLOC_KEYS_BYTES ((size_t)FSPH_NOALLOC_SORT_MAX * 8)
#define NOALLOC_VALS_BYTES ((size_t)FSPH_NOALLOC_SORT_MAX * 4)
#define NOALLOC_HIST_BYTES \
  ((size_t)(256 * ((FSPH_NOALLOC_SORT_MAX + RS_TILE - 1) / RS_TILE) + 256) * 4)
#define NOALLOC_TOTAL \
  (NOALLOC_RANGE_BYTES + NOALLOC_KEYS_BYTES + NOALLOC_VALS_BYTES + NOALLOC_HIST_BYTES)

namespace fsph {
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_TOTAL];
}  // namespace fsph

namespace {
// Device address of g_noalloc_scratch per device.  In host code the symbol
// names a host-side shadow, not device memory, so the address must come
// from cudaGetSymbolAddress, taken once per device with that device current.
std::mutex g_noalloc_mu;
void * g_noalloc_addr[64] = {};
}  // namespace

extern "C" fsph_status fsph_sort_keys_noalloc(const double * x,
  const double * y, const double * z, const double * h, int64_t n,
  int32_t dimension, uint64_t * keys_out, int32_t * perm_out, void * stream) {
  using namespace fsph;
  if(n < 2 || n > FSPH_NOALLOC_SORT_MAX || (dimension != 2 && dimension != 3) ||
     !x || !y || (dimension == 3 && !z) || !h || !keys_out || !perm_out)
    return FSPH_ERR_ARG;
  int dev = 0;
  if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return FSPH_ERR_NO_DEVICE;
  void * base = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if(!g_noalloc_addr[dev]) {
      void * ptr = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
      if(e != cudaSuccess || !ptr)
        return FSPH_ERR_CUDA;
      g_noalloc_addr[dev] = ptr;
    }
    base = g_noalloc_addr[dev];
  }
  unsigned char * b = (unsigned char *)base;
  unsigned long long * range = (unsigned long long *)b;
  unsigned long long * ktmp = (unsigned long long *)(b + NOALLOC_RANGE_BYTES);
  int * vtmp = (int *)(b + NOALLOC_RANGE_BYTES + NOALLOC_KEYS_BYTES);
  unsigned * hist =
    (unsigned *)(b + NOALLOC_RANGE_BYTES + NOALLOC_KEYS_BYTES + NOALLOC_VALS_BYTES);
  Particles P{};
  P.f[F_X] = const_cast<double *>(x);
  P.f[F_Y] = const_cast<double *>(y);
  P.f[F_Z] = const_cast<double *>(z ? z : y);
  P.f[F_H] = const_cast<double *>(h);
  P.n = (int)n;
  PhysParams pp{};
  pp.dim = dimension;
  long long launches = 0;
  Launch L{(cudaStream_t)stream, &launches};
  // every scratch word that is read is first written by this call: the range's
  // block counter here (calls that overlapped, which the caller must not make,
  // could have left it at any value), the rest by the launches (the range's
  // partial words share the keys' scratch), but SORT_CROWDED, which may hold
  // any value
  if(cudaMemsetAsync(range + RANGE_TICKET, 0, sizeof(*range), L.stream) != cudaSuccess)
    return FSPH_ERR_CUDA;
  if(launch_range(L, P, pp, range, ktmp) != cudaSuccess ||
     launch_keys(L, P, pp, range, (unsigned long long *)keys_out, perm_out) != cudaSuccess)
    return FSPH_ERR_CUDA;
  if(radix_sort_pairs(L, (unsigned long long *)keys_out, perm_out, ktmp, vtmp,
       (int)n, hist, 63 / dimension * dimension,
       (unsigned *)(range + RANGE_SORT)) != cudaSuccess)
    return FSPH_ERR_CUDA;
  return FSPH_OK;
}

