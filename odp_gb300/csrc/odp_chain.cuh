/*
 * odp_chain.cuh -- the random stream and the acceptance rule of the annealing
 * chains, shared by the kernels that step them.
 */
#ifndef ODP_CHAIN_CUH
#define ODP_CHAIN_CUH
#include <cuda_runtime.h>
#include "odp_engine.h"

namespace {

/* glibc's TYPE_3 stream (r[i] = r[i-31] + r[i-3], output r[i] >> 1) over a
 * ring of its last 31 words, ring[pos] = r[i-31]. */
struct dev_rng {
  unsigned int ring[31];
  int pos;
};

__device__ __forceinline__ int rng_next(dev_rng *g)
{
  const int p = g->pos;
  const unsigned int x = g->ring[p] + g->ring[p >= 3 ? p - 3 : p + 28];
  g->ring[p] = x;
  g->pos = (p == 30) ? 0 : p + 1;
  return (int)(x >> 1);
}

/* get_random (utils.c:361-364): the integer form is exact where the double
 * product is (max <= 2^22); above it the same double arithmetic. */
__device__ __forceinline__ int rng_below(dev_rng *g, int max)
{
  const int x = rng_next(g);
  if(max >= 0 && max <= (1 << 22))
    return (int)(((unsigned long long)(unsigned)x * (unsigned long long)max) >> 31);
  return (int)(x * ((double)max) / (1.0 + 2147483647.0));
}

/* accept_s (sample/SA/common.c:15-37); uniform_rand (common.c:10-13) is
 * (random() + 1) / (RAND_MAX + 2) from the same stream as the proposals. */
__device__ bool accept_move(gbx_chain &c, dev_rng *rng, int diameter, double aspl)
{
  if(c.hill_climbing) return aspl <= c.cur_aspl;
  if(diameter < c.cur_diameter && !c.aspl_priority) return true;
  if(diameter > c.cur_diameter && !c.aspl_priority) return false;
  if(aspl <= c.cur_aspl) return true;
  double diff = (c.cur_aspl - aspl) * c.n * (c.n - 1);
  if(c.s != 1) diff /= c.s;
  const int r = rng_next(rng);
  /* In 32 bits first: the estimate of exp(diff / temp) is good to 1e-4 (the
   * exponent, above -24, rounds by 4e-6, u by 1e-7), and below -24 the value is
   * less than any u.  Only a u within 1e-3 of it needs the 64-bit form, whose
   * divisions and exponential take 2k cycles. */
  const float x = (float)diff / (float)c.temp, uf = ((float)r + 1.0f) * (1.0f / 2147483648.0f);
  if(x < -24.0f) return false;
  if(x <= 0.0f){
    const float e = expf(x);
    if(uf < e * 0.999f) return true;
    if(uf > e * 1.001f) return false;
  }
  const double u = ((double)r + 1.0) / ((double)2147483647 + 2.0);
  return exp(diff / c.temp) > u;
}

}  // namespace
#endif
