/*
 * odp_device.cuh -- device helpers shared by the kernels: bit counting, the
 * timer, and the rules that turn the compact adjacency into row-space
 * neighbour entries.
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

}  // namespace
#endif
