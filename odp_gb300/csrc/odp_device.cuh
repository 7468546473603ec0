/*
 * odp_device.cuh -- device helpers shared by the kernels: bit counting, the
 * timer, the rules that turn the compact adjacency into row-space neighbour
 * entries, and the lanes of the lockstep kernels.
 */
#ifndef ODP_DEVICE_CUH
#define ODP_DEVICE_CUH
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include "odp_engine.h"

namespace {

__device__ __forceinline__ unsigned popc4(const uint4 &v)
{
  return __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
}

__device__ __forceinline__ void or_into(uint4 &a, const uint4 &b)
{
  a.x |= b.x; a.y |= b.y; a.z |= b.z; a.w |= b.w;
}

template <typename T>
__device__ __forceinline__ T vload(const T *p) { return *(const volatile T *)p; }

__device__ __forceinline__ unsigned long long globaltimer()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

/* ---------------------------------------------------------------------- */
/* Neighbour-table expansion.                                              */
/* ---------------------------------------------------------------------- */

/* ODP_ROTATE for the grid symmetries (reference utils_cuda.cu:3-14). */
__device__ __forceinline__ int grid_rotate(int v, int width, int height, int s, int deg)
{
  int x = v / height, y = v % height;
  if(s == 2) return (width - x - 1) * height + (height - y - 1);
  if(deg == 90)  return y * height + (height - x - 1);
  if(deg == 180) return (height - x - 1) * height + (height - y - 1);
  return (height - y - 1) * height + x;
}

/* Row of a base-quadrant vertex (utils_cuda.cu:16-23). */
__device__ __forceinline__ int grid_base_row(int x, int height, int s)
{
  if(s == 2) return x;
  return (x / height) * (height / 2) + x % height;
}

/* Neighbour j of global vertex v of a rotation-symmetric grid
 * (utils_cuda.cu:25-59), read from the compact adjacency `adj`; -1 when the
 * stored entry is out of range. */
__device__ __forceinline__ int grid_source_row(const gbx_expand_desc &e, int v, int &back)
{
  const int w = e.width, h = e.height, s = e.s;
  int x = v / h, y = v % h, bw = w / 2, bh = h / 2;
  if(s == 2){
    if(x < bw){ back = 0; return v; }
    back = 180;
    return grid_rotate(v, w, h, s, 180);
  }
  if(x < bw && y < bh){ back = 0; return grid_base_row(v, h, s); }
  if(x < bw)          { back = 90; return grid_base_row(grid_rotate(v, w, h, s, 270), h, s); }
  if(y >= bh)         { back = 180; return grid_base_row(grid_rotate(v, w, h, s, 180), h, s); }
  back = 270;
  return grid_base_row(grid_rotate(v, w, h, s, 90), h, s);
}

/* Compact-adjacency position of entry j of global vertex v, and the
 * rotation that maps the stored value back (grid symmetry) or the shift
 * that does (general symmetry). */
__device__ __forceinline__ size_t entry_source(const gbx_expand_desc &e, int v, int j, int &back)
{
  if(e.grid_s) return (size_t)grid_source_row(e, v, back) * e.d + j;
  const int base = e.n / e.s;
  back = (v / base) * base;
  return (size_t)(v % base) * e.d + j;
}

/* Row-table entry from the stored value `a` of entry (v, j) (entries at or
 * past the vertex's degree hold the row itself, and so does an out-of-range
 * value, which also sets `bad`): the rotated vertex's row for symmetric
 * grids, the shifted vertex (mod n) for general symmetry (its row, where the
 * plan orders the rows itself). */
__device__ __forceinline__ int expand_value(const gbx_expand_desc &e, int a, int back, int j, int deg, int row,
                                            bool &bad)
{
  if(j >= deg) return row;
  if(a < 0 || a >= e.n){ bad = true; return row; }
  if(e.grid_s) return e.itable[back ? grid_rotate(a, e.width, e.height, e.s, back) : a];
  int nb = a + back;
  if(nb >= e.n) nb -= e.n;
  return e.itable ? e.itable[nb] : nb;
}


/* A record into pinned host memory: its error word last, released to the host
 * when the launch has a number that the host looks for (the release costs a job
 * of the small kernel 1 to 2 us: 36 graphs of n = 200 to 1000 42.9 -> 40.9). */
__device__ __forceinline__ void store_record(gbx_small_rec *to, const gbx_small_rec &r)
{
  to->level = r.level;
  to->sum = r.sum;
  to->t_loaded = r.t_loaded;
  to->t_done = r.t_done;
  if(GBX_REC_SEQ(r.err)) asm volatile("st.release.sys.global.u32 [%0], %1;" :: "l"(&to->err), "r"(r.err) : "memory");
  else to->err = r.err;
}

/* ---------------------------------------------------------------------- */
/* Lanes: 32 bytes (256 source bits, one sector) of a row, the unit of the  */
/* lockstep kernels, moved by 256-bit accesses (L2 only: other SMs rewrite  */
/* the buffers between levels).                                             */
/* ---------------------------------------------------------------------- */

#define LANE_FULL 1u                  /* every source bit of the lane is set */
#define LANE_CHANGED 2u               /* the older buffer does not hold the lane's words yet */

#define ARRIVE_ONE (1ull << 48)       /* barrier words: CTAs done << 48 | bits counted */
#define ARRIVE_BITS (ARRIVE_ONE - 1)

__device__ __forceinline__ void ld_lane(unsigned (&r)[8], const void *p)
{
  asm volatile("ld.global.cg.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(p) : "memory");
}

__device__ __forceinline__ void st_lane(void *p, const unsigned (&r)[8])
{
  asm volatile("st.global.cg.v8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
               :: "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "l"(p)
               : "memory");
}

/* Set bits of eight words: full adders (one three-input operation for each
 * sum and carry) reduce them to four words of weights 1, 1, 2 and 4, as the
 * bit count runs at a quarter of the logic's rate. */
__device__ __forceinline__ unsigned popc_lane(const unsigned (&r)[8])
{
  const unsigned s1 = r[0] ^ r[1] ^ r[2], c1 = (r[0] & r[1]) | (r[2] & (r[0] | r[1]));
  const unsigned s2 = r[3] ^ r[4] ^ r[5], c2 = (r[3] & r[4]) | (r[5] & (r[3] | r[4]));
  const unsigned s3 = s1 ^ s2 ^ r[6], c3 = (s1 & s2) | (r[6] & (s1 | s2));
  const unsigned t1 = c1 ^ c2 ^ c3, f1 = (c1 & c2) | (c3 & (c1 | c2));
  return __popc(s3) + __popc(r[7]) + 2 * __popc(t1) + 4 * __popc(f1);
}

__device__ __forceinline__ unsigned and_lane(const unsigned (&r)[8])
{
  return r[0] & r[1] & r[2] & r[3] & r[4] & r[5] & r[6] & r[7];
}

/* Barrier words.  A CTA arrives with arrive_word (one thread, after a CTA
 * barrier: its release covers the CTA's stores) and one thread of it waits
 * with wait_for until `*word` reaches `target`; false past the limit. */
__device__ __forceinline__ void arrive_word(unsigned long long *word, unsigned long long v)
{
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" :: "l"(word), "l"(v) : "memory");
}

__device__ __forceinline__ void arrive_word(unsigned *word, unsigned v)
{
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" :: "l"(word), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned long long acquire_word(const unsigned long long *p)
{
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned acquire_word(const unsigned *p)
{
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <typename T>
__device__ __forceinline__ bool wait_for(const T *word, T target, T &seen, unsigned long long limit_ns)
{
  seen = acquire_word(word);
  if(seen < target){
    const unsigned long long t0 = globaltimer();
    do{
      if(globaltimer() - t0 > limit_ns) return false;
      seen = acquire_word(word);
    } while(seen < target);
  }
  return true;
}

__device__ __forceinline__ int lane_bits(int nsrc, int gl) { return min(max(nsrc - 256 * gl, 0), 256); }

__device__ __forceinline__ void mark(unsigned *s, int o, int n)
{
  if((unsigned)o < (unsigned)n) atomicOr(s + (o >> 5), 1u << (o & 31));
}

/* A lane's words OR its neighbours', NB of them in flight. */
template <int NB>
__device__ __forceinline__ void gather_lane(unsigned (&acc)[8], const char *X, const int *ids, int d, unsigned rb)
{
  int j = 0;
  for(; j + NB <= d; j += NB){
    unsigned t[NB][8];
#pragma unroll
    for(int i = 0; i < NB; i += 4){
      const int4 u = *reinterpret_cast<const int4 *>(ids + j + i);
      ld_lane(t[i], X + (size_t)(unsigned)u.x * rb);
      ld_lane(t[i + 1], X + (size_t)(unsigned)u.y * rb);
      ld_lane(t[i + 2], X + (size_t)(unsigned)u.z * rb);
      ld_lane(t[i + 3], X + (size_t)(unsigned)u.w * rb);
    }
#pragma unroll
    for(int i = 0; i < NB; i += 2)
#pragma unroll
      for(int k = 0; k < 8; k++) acc[k] |= t[i][k] | t[i + 1][k];
    if(and_lane(acc) == ~0u) return;
  }
  for(; j < d; j += 4){
    const int4 u = *reinterpret_cast<const int4 *>(ids + j);
    unsigned t0[8], t1[8] = {0, 0, 0, 0, 0, 0, 0, 0}, t2[8] = {0, 0, 0, 0, 0, 0, 0, 0},
             t3[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    ld_lane(t0, X + (size_t)(unsigned)u.x * rb);
    if(j + 1 < d) ld_lane(t1, X + (size_t)(unsigned)u.y * rb);
    if(j + 2 < d) ld_lane(t2, X + (size_t)(unsigned)u.z * rb);
    if(NB > 4 && j + 3 < d) ld_lane(t3, X + (size_t)(unsigned)u.w * rb);
#pragma unroll
    for(int k = 0; k < 8; k++) acc[k] |= (t0[k] | t1[k]) | (t2[k] | t3[k]);
  }
}

}  // namespace
#endif
