/*
 * anneal_resident.cu -- annealing chains that run many steps in one kernel.
 *
 * The stepwise form (anneal.cu) costs four launches per step: one thread per
 * chain proposes from global memory (17 us on GB300 for 16 chains of n = 1024,
 * d = 8), the engine evaluates every chain's graph (54 us) and a block per
 * chain decides (10 us).  Here a chain belongs to a team of CTAs for the whole
 * run.  Every CTA of the team keeps the chain's record, random stream and
 * compact adjacency (16-bit vertices) in shared memory and makes the same
 * proposal and the same decision from the same numbers, so nothing but the
 * bit counts of each level is exchanged: a step is one proposal, one pass over
 * the CTA's rows and one barrier per BFS level, and one decision.  Levels 1
 * and 2 come from the adjacency in shared memory (regular graphs without
 * symmetry; level 1 otherwise); later levels gather lanes as the lockstep
 * kernels do (sweep.cu).  Several teams run side by side.  A team of up to 16
 * CTAs is a thread-block cluster: the counts go to every CTA's shared memory
 * and a level's barrier is the cluster's.  Larger teams share one cooperative
 * launch and meet in global memory; every wait there has a time limit.
 *
 * The moves, results and records are those of the stepwise kernels.
 */
#include <cuda_runtime.h>
#include <climits>
#include <cstdint>
#include <cfloat>
#include <cooperative_groups.h>
#include "odp_engine.h"
#include "odp_device.cuh"
#include "odp_chain.cuh"

#define RESIDENT_THREADS GBX_RESIDENT_THREADS
#define RESIDENT_CLUSTER GBX_RESIDENT_CLUSTER

/* Rows marked at a time: 16 KB of them. */
__host__ __device__ static inline int resident_block(int rows, int lanes)
{
  const int fit = 16384 / (lanes * 32);
  return rows < fit ? rows : fit < 2 ? 2 : fit;
}

namespace {
namespace packed {                    /* the swap rules over 16-bit vertices */
typedef dev_rng mut_rng;
#define MUT_BELOW(rng, max) rng_below((rng), (max))
#define MUT_TRIES (1LL << 22)
#define MUT_FN static __device__ inline
#define MUT_VERTEX unsigned short
#include "odp_mutate.h"
}  // namespace packed

#define ANNEAL_MAX_ATTEMPTS (1 << 20) /* rejected 2-opt attempts per proposal */

struct ResidentSync {
  unsigned long long arrive[3][16];   /* step t's barrier word: [t % 3][0] */
  unsigned long long first[3][16];    /* bits at level 1 */
};

struct ResidentShared {
  gbx_chain c;
  dev_rng rng;
  packed::mut_general g;
  packed::mut_grid gg;
  int nw, wrow[4], wslot[4];          /* the last swap's (or undo's) writes */
  unsigned cnt[2], cnt1[2];           /* this CTA's bits of the pass, by the step's parity */
  uint2 peer[2][RESIDENT_CLUSTER];    /* cluster: every CTA's cnt and cnt1, the same */
  unsigned long long bits, bits1;     /* the team's */
  int ok, accept, copy;
};

struct Resident {                     /* uniform over the CTA */
  unsigned short *adj;                /* [base][d] */
  int *list;                          /* [rows][dp]: the CTA's rows of the neighbour table */
  unsigned *scratch;                  /* a block of rows being marked */
  unsigned char *flag;                /* [rows][lanes] */
  char *buf;
  ResidentSync *sync;
  unsigned step;
  int rank, size, rows, r0, nr, lanes, block;
};

template <class G>
__device__ __forceinline__ void swap_writes(ResidentShared &sh, const G &g)
{
  sh.nw = g.nw;
  for(int k = 0; k < 4; k++)
    if(k < g.nw){
      sh.wrow[k] = g.wrow[k];
      sh.wslot[k] = g.wslot[k];
    }
}

/* Thread 0: mut_two_opt's common way for regular general graphs without
 * symmetry, where nothing turns or has an antipode: five draws, four distinct
 * vertices, one exchange.  The draws, the two edges' slots and the rows that
 * point back are loaded side by side; one after another behind the general
 * form's branches they took 5k cycles a step, warm.  False, with nothing
 * drawn, when a vertex repeats (the general form draws again) or an edge has
 * no other end. */
__device__ bool propose_regular(ResidentShared &sh)
{
  unsigned short *adj = sh.g.adj;
  const int n = sh.g.n, d = sh.g.d, p = sh.rng.pos;
  unsigned x[5];
  int at[5];
#pragma unroll
  for(int k = 0; k < 5; k++){
    at[k] = p + k < 31 ? p + k : p + k - 31;
    const int q = at[k] >= 3 ? at[k] - 3 : at[k] + 28;
    x[k] = sh.rng.ring[at[k]];
    if(k < 3) x[k] += sh.rng.ring[q];
  }
  x[3] += x[0];
  x[4] += x[1];
  auto below = [&](int k, int max) { return (int)(((unsigned long long)(x[k] >> 1) * (unsigned long long)max) >> 31); };
  const int u0 = below(0, n), u1 = below(1, n), s0 = below(2, d), s1 = below(3, d);
  const int v0 = adj[u0 * d + s0], v1 = adj[u1 * d + s1];
  if(u0 == u1 || v0 == u1 || v1 == u0 || v0 == v1 || v0 == u0 || v1 == u1) return false;
  int b0 = -1, b1 = -1;
  for(int i0 = (d - 1) & ~7; i0 >= 0; i0 -= 8){            /* the first of equal entries */
    int e0[8], e1[8];
#pragma unroll
    for(int k = 0; k < 8; k++){
      const int i = min(i0 + k, d - 1);
      e0[k] = adj[v0 * d + i];
      e1[k] = adj[v1 * d + i];
    }
#pragma unroll
    for(int k = 7; k >= 0; k--){
      if(e0[k] == u0) b0 = min(i0 + k, d - 1);
      if(e1[k] == u1) b1 = min(i0 + k, d - 1);
    }
  }
  if(b0 < 0 || b1 < 0) return false;
  const bool cross = below(4, 2) != 0;                     /* u0--v1, v0--u1; else u0--u1, v0--v1 */
  adj[u0 * d + s0] = (unsigned short)(cross ? v1 : u1);
  adj[u1 * d + s1] = (unsigned short)(cross ? v0 : u0);
  adj[v0 * d + b0] = (unsigned short)(cross ? u1 : v1);
  adj[v1 * d + b1] = (unsigned short)(cross ? u0 : v0);
#pragma unroll
  for(int k = 0; k < 5; k++) sh.rng.ring[at[k]] = x[k];
  sh.rng.pos = p + 5 < 31 ? p + 5 : p + 5 - 31;
  sh.nw = 4;
  sh.wrow[0] = u0; sh.wslot[0] = s0;
  sh.wrow[1] = u1; sh.wslot[1] = s1;
  sh.wrow[2] = v0; sh.wslot[2] = b0;
  sh.wrow[3] = v1; sh.wslot[3] = b1;
  ODP_Restore &r = sh.c.last;
  r.u[0] = u0; r.u[1] = u1; r.v[0] = v0; r.v[1] = v1;
  r.u_d[0] = s0; r.u_d[1] = s1; r.v_d[0] = b0; r.v_d[1] = b1;
  return true;
}

/* Thread 0: the next swap into the shared adjacency; false when there is none.
 * The graph's record is a local copy: through shared memory every use of a
 * field would load it again, as the adjacency's stores might alias it. */
__device__ bool propose(ResidentShared &sh)
{
  int e = 0;
  ODP_Restore last;
  if(!sh.c.grid && sh.c.s == 1 && !sh.c.ndeg && propose_regular(sh)) return true;
  if(sh.c.grid){
    packed::mut_grid g = sh.gg;
    for(int attempt = 0; attempt < ANNEAL_MAX_ATTEMPTS && e == 0; attempt++) e = packed::mut_grid_two_opt(&sh.rng, &g, &last);
    if(e == 1) swap_writes(sh, g);
  }
  else{
    packed::mut_general g = sh.g;
    for(int attempt = 0; attempt < ANNEAL_MAX_ATTEMPTS && e == 0; attempt++) e = packed::mut_two_opt(&sh.rng, &g, &last);
    if(e == 1) swap_writes(sh, g);
  }
  if(e != 1) return false;
  sh.c.last = last;
  return true;
}

/* Thread 0: the last swap undone. */
__device__ void undo(ResidentShared &sh)
{
  const ODP_Restore last = sh.c.last;
  if(sh.c.grid){
    packed::mut_grid g = sh.gg;
    packed::mut_grid_restore(&g, &last);
    swap_writes(sh, g);
  }
  else{
    packed::mut_general g = sh.g;
    packed::mut_restore(&g, &last);
    swap_writes(sh, g);
  }
}

/* The slots a swap or its undo wrote, into the CTA's lists (s orbit rows per
 * slot) and, by the team's first CTA, into the chain's adjacency. */
template <int THREADS>
__device__ void spread_writes(const ResidentShared &sh, const Resident &t)
{
  const gbx_chain &c = sh.c;
  for(int i = threadIdx.x; i < sh.nw * c.s; i += THREADS){
    const int k = i / c.s, turn = i - k * c.s;
    const int m = sh.wrow[k], slot = sh.wslot[k], a = t.adj[m * c.d + slot];
    int row, nb;
    if(!c.grid || c.s == 1){
      row = m + turn * c.base;
      nb = a + turn * c.base;
      if(nb >= c.n) nb -= c.n;
    }
    else{
      const int bv = (c.s == 2) ? m : (m / sh.gg.bh) * c.height + (m % sh.gg.bh);
      int v = bv, u = a;
      if(turn > 0){
        const int deg = (c.s == 2) ? 180 : 90 * turn;
        v = packed::grid_rot(&sh.gg, bv, deg);
        u = packed::grid_rot(&sh.gg, a, deg);
      }
      row = c.itable[v];
      nb = c.itable[u];
    }
    if(row >= t.r0 && row < t.r0 + t.nr) t.list[(row - t.r0) * c.dp + slot] = nb;
    if(turn == 0 && t.rank == 0) c.adj[(long long)m * c.d + slot] = a;
  }
}

/* The whole team passes, with the level's bits of all CTAs (and level 1's, in
 * the first pass of a step).  False past the limit (never in a cluster, whose
 * barrier is the hardware's). */
template <bool CLUSTER>
__device__ bool team_pass(ResidentShared &sh, Resident &t, unsigned long long limit_ns, bool with_first,
                          unsigned long long &bits, unsigned long long &bits1)
{
  const unsigned par = t.step & 1;
  if(CLUSTER){
    /* at most n * n < 2^32 bits */
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    __syncthreads();
    if(threadIdx.x < t.size)
      cl.map_shared_rank(&sh, threadIdx.x)->peer[par][t.rank] = make_uint2(sh.cnt[par], sh.cnt1[par]);
    if(threadIdx.x == 0) sh.cnt[par ^ 1] = sh.cnt1[par ^ 1] = 0;     /* read before the last barrier */
    t.step++;
    cl.sync();
    const unsigned lane = threadIdx.x & 31;
    const uint2 c = lane < t.size ? sh.peer[par][lane] : make_uint2(0u, 0u);
    bits = __reduce_add_sync(0xffffffffu, c.x);
    bits1 = __reduce_add_sync(0xffffffffu, c.y);
    return true;
  }
  __syncthreads();
  if(threadIdx.x == 0){
    const unsigned cnt = sh.cnt[par], cnt1 = sh.cnt1[par];
    sh.cnt[par] = sh.cnt1[par] = 0;
    sh.ok = 1;
    if(t.size == 1){
      sh.bits = cnt;
      sh.bits1 = cnt1;
    }
    else{
      unsigned long long *word = &t.sync->arrive[t.step % 3][0], *first = &t.sync->first[t.step % 3][0], seen;
      if(t.rank == 0){
        /* the next step's words: their last readers have all passed the last step */
        t.sync->arrive[(t.step + 1) % 3][0] = 0;
        t.sync->first[(t.step + 1) % 3][0] = 0;
      }
      if(cnt1) atomicAdd(first, (unsigned long long)cnt1);
      arrive_word(word, ARRIVE_ONE | cnt);
      if(!wait_for(word, ARRIVE_ONE * (unsigned)t.size, seen, limit_ns)) sh.ok = 0;
      sh.bits = seen & ARRIVE_BITS;
      if(with_first) sh.bits1 = __ldcg(first);
    }
  }
  t.step++;
  __syncthreads();
  bits = sh.bits;
  bits1 = sh.bits1;
  return sh.ok != 0;
}

/* Levels 1 and 2 (two) or level 1 of the CTA's rows, marked in shared memory
 * a block of rows at a time by all threads (a warp per row took 14k cycles of
 * latency for 64 rows of n = 1024, d = 8). */
template <int THREADS>
__device__ void first_rows(ResidentShared &sh, const Resident &t, bool two)
{
  const gbx_chain &c = sh.c;
  const int tid = threadIdx.x, d = c.d, dp = c.dp, words = t.lanes * 8;
  const int magic = d > 0 ? (65536 + d - 1) / d : 1;       /* i / d for i < 1024 (two: d <= 12) */
  char *to = t.buf + (two ? 0 : (size_t)c.n * t.lanes * 32);
  unsigned n1 = 0, n2 = 0;
  for(int b0 = 0; b0 < t.nr; b0 += t.block){
    const int nb = min(t.block, t.nr - b0);
    uint4 *sv = reinterpret_cast<uint4 *>(t.scratch);
    for(int i = tid; i < nb * t.lanes * 2; i += THREADS) sv[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const int *ids = t.list + b0 * dp;
    for(int i = tid; i < nb * dp; i += THREADS) mark(t.scratch + (i / dp) * words, ids[i], c.base);
    for(int r = tid; r < nb; r += THREADS) mark(t.scratch + r * words, t.r0 + b0 + r, c.base);
    __syncthreads();
    if(two){
      for(int i = tid; i < nb * t.lanes * 2; i += THREADS) n1 += popc4(sv[i]);
      __syncthreads();
      /* eight threads a row: entries part, part + 8, ... of its d * d */
      const int part = tid & 7;
      for(int r = tid >> 3; r < nb; r += THREADS / 8){
        unsigned *s = t.scratch + r * words;
        const int *row = ids + r * dp;
        for(int i0 = part; i0 < d * d; i0 += 64){          /* eight loaded before any is marked */
          int id[8];
#pragma unroll
          for(int k = 0; k < 8; k++){
            const int i = i0 + 8 * k, j = (i * magic) >> 16;
            id[k] = i < d * d ? t.adj[row[j] * d + (i - j * d)] : -1;
          }
#pragma unroll
          for(int k = 0; k < 8; k++) mark(s, id[k], c.base);
        }
      }
      __syncthreads();
    }
    for(int i = tid; i < nb * t.lanes; i += THREADS){
      const int r = i / t.lanes, p = i - r * t.lanes;
      unsigned w[8];
      *reinterpret_cast<uint4 *>(w) = sv[2 * i];
      *reinterpret_cast<uint4 *>(w + 4) = sv[2 * i + 1];
      st_lane(to + ((size_t)(t.r0 + b0 + r) * t.lanes + p) * 32, w);
      const unsigned b = popc_lane(w);
      n2 += b;
      t.flag[(b0 + r) * t.lanes + p] = (unsigned char)(LANE_CHANGED | (b == (unsigned)lane_bits(c.base, p) ? LANE_FULL : 0u));
    }
    __syncthreads();
  }
  n1 = __reduce_add_sync(0xffffffffu, n1);
  n2 = __reduce_add_sync(0xffffffffu, n2);
  if((tid & 31) == 0){
    if(n1) atomicAdd(&sh.cnt1[t.step & 1], n1);
    if(n2) atomicAdd(&sh.cnt[t.step & 1], n2);
  }
}

/* A gathered level: a thread keeps its lane and walks the rows. */
template <int THREADS>
__device__ void next_rows(ResidentShared &sh, const Resident &t, int level)
{
  const gbx_chain &c = sh.c;
  const unsigned rb = (unsigned)t.lanes * 32u;
  const size_t half = (size_t)c.n * rb;
  unsigned cnt = 0;
  const int rr = threadIdx.x / t.lanes, rs = THREADS / t.lanes;
  if(rr < rs){
    const int gl = threadIdx.x - rr * t.lanes;
    const unsigned bits = (unsigned)lane_bits(c.base, gl);
    const char *X = t.buf + ((level & 1) ? 0 : half) + gl * 32;
    char *Y = t.buf + ((level & 1) ? half : 0) + gl * 32;
    for(int row = rr; row < t.nr; row += rs){
      const unsigned f = t.flag[row * t.lanes + gl];
      const size_t own = (size_t)(unsigned)(t.r0 + row) * rb;
      unsigned acc[8];
      if(f & LANE_FULL){
        cnt += bits;
        if(f & LANE_CHANGED){
          ld_lane(acc, X + own);
          st_lane(Y + own, acc);
          t.flag[row * t.lanes + gl] = LANE_FULL;
        }
        continue;
      }
      ld_lane(acc, X + own);
      gather_lane<8>(acc, X, t.list + row * c.dp, c.d, rb);
      st_lane(Y + own, acc);
      const unsigned b = popc_lane(acc);
      cnt += b;
      if(b == bits) t.flag[row * t.lanes + gl] = LANE_FULL | LANE_CHANGED;
    }
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if((threadIdx.x & 31) == 0 && cnt) atomicAdd(&sh.cnt[t.step & 1], cnt);
}

/* The graph's diameter (negative: some pair is unreachable) and ordered
 * distance sum, the same in every thread of the team; false past a wait's limit. */
template <bool CLUSTER>
__device__ bool evaluate(ResidentShared &sh, Resident &t, unsigned long long limit_ns, int &diameter, long long &sum)
{
  const gbx_chain &c = sh.c;
  /* marking d * d entries a row against one more gathered level: n = 4096, d =
   * 16 took 42k cycles against 30k, n = 1024, d = 8 5k against 6k */
  const bool two = c.s == 1 && !c.ndeg && c.d <= 12;
  const unsigned long long full = (unsigned long long)c.n * (unsigned long long)c.base;
  unsigned long long prev = (unsigned long long)c.base;
  sum = ((long long)c.n * c.base - c.base) * c.s;
  int level = 0;
  bool over = false;
  auto settle = [&](unsigned long long b) {
    level++;
    const bool complete = b == full, stalled = !complete && (b == prev || level >= c.n);
    if(!complete && !stalled){
      sum += (long long)(full - b) * c.s;
      prev = b;
      return;
    }
    over = true;
    diameter = stalled ? -level : level;
  };
  constexpr int THREADS = CLUSTER ? GBX_RESIDENT_CLUSTER_THREADS : RESIDENT_THREADS;
  first_rows<THREADS>(sh, t, two);
  unsigned long long bits = 0, bits1 = 0;
  if(!team_pass<CLUSTER>(sh, t, limit_ns, two, bits, bits1)) return false;
  if(two) settle(bits1);
  if(!over) settle(bits);
  while(!over){
    next_rows<THREADS>(sh, t, level + 1);
    if(!team_pass<CLUSTER>(sh, t, limit_ns, false, bits, bits1)) return false;
    settle(bits);
  }
  return true;
}

/* store(i, src[i]) for i = first, first + stride, ... below n, eight loads in
 * flight (a store into shared or host memory might alias the source, so loads
 * one by one would each wait for the one before). */
template <class Store>
__device__ __forceinline__ void each_int(const int *src, int n, int first, int stride, Store store)
{
  for(int i0 = first; i0 < n; i0 += 8 * stride){
    int x[8];
#pragma unroll
    for(int k = 0; k < 8; k++) x[k] = __ldcg(src + min(i0 + k * stride, n - 1));
#pragma unroll
    for(int k = 0; k < 8; k++)
      if(i0 + k * stride < n) store(i0 + k * stride, x[k]);
  }
}

/* Thread 0: the step's outcome, as anneal_decide_kernel. */
__device__ void decide(ResidentShared &sh, int level, long long total)
{
  gbx_chain &c = sh.c;
  int diameter;
  long long sum;
  double aspl;
  if(level < 0){ diameter = INT_MAX; sum = LLONG_MAX; aspl = DBL_MAX; }
  else{
    diameter = level;
    aspl = total / (((double)c.n - 1) * c.n);
    sum = (long long)(total / 2.0);
  }
  c.steps++;
  sh.copy = 0;
  if(diameter < c.best_diameter || (diameter == c.best_diameter && aspl < c.best_aspl)){
    c.best_diameter = diameter;
    c.best_sum = sum;
    c.best_aspl = aspl;
    sh.copy = 1;
  }
  sh.accept = accept_move(c, &sh.rng, diameter, aspl);
  if(sh.accept){
    c.cur_diameter = diameter;
    c.cur_sum = sum;
    c.cur_aspl = aspl;
    c.accepted++;
  }
  c.temp *= c.cooling;
}

template <bool CLUSTER>
__global__ void __launch_bounds__(CLUSTER ? GBX_RESIDENT_CLUSTER_THREADS : RESIDENT_THREADS, 2) anneal_resident_kernel(const gbx_resident p)
{
  extern __shared__ __align__(16) unsigned char resident_smem[];
  __shared__ ResidentShared sh;
  constexpr int THREADS = CLUSTER ? GBX_RESIDENT_CLUSTER_THREADS : RESIDENT_THREADS;
  const int tid = threadIdx.x, G = (int)gridDim.x;
  /* team i: CTAs [i * G / teams, (i + 1) * G / teams), a cluster of them */
  const int team = (int)((((long long)blockIdx.x + 1) * p.teams - 1) / G);
  const int lo = (int)((long long)team * G / p.teams), hi = (int)((long long)(team + 1) * G / p.teams);
  Resident t;
  t.rank = (int)blockIdx.x - lo;
  t.sync = reinterpret_cast<ResidentSync *>(p.sync) + team;
  t.step = 0;
  if(CLUSTER) cooperative_groups::this_cluster().sync();   /* every CTA's shared memory is there */
  for(int chain = team; chain < p.count; chain += p.teams){
    __syncthreads();
    {
      const unsigned *src = reinterpret_cast<const unsigned *>(p.chains + chain);
      unsigned *dst = reinterpret_cast<unsigned *>(&sh.c);
      for(int i = tid; i < (int)(sizeof(gbx_chain) / 4); i += THREADS) dst[i] = src[i];
    }
    __syncthreads();
    const gbx_chain &c = sh.c;
    t.lanes = (c.base + 255) >> 8;
    /* a lane per thread is enough: more CTAs only lengthen the barrier */
    const int want = (int)(((long long)c.n * t.lanes + THREADS - 1) / THREADS);
    t.size = CLUSTER ? hi - lo : min(hi - lo, want);
    /* This CTA has no part in the chain.  Its step counter stays behind the
     * team's, so it may have none in any other: a team of several CTAs has one
     * chain, and several chains share a team only where teams have one CTA. */
    if(t.rank >= t.size) continue;
    t.rows = (c.n + t.size - 1) / t.size;
    t.r0 = t.rank * t.rows;
    t.nr = max(0, min(t.rows, c.n - t.r0));
    t.buf = p.buf + p.buf_offset[chain];
    t.list = reinterpret_cast<int *>(resident_smem);
    t.scratch = reinterpret_cast<unsigned *>(t.list + t.rows * c.dp);
    t.block = resident_block(t.rows, t.lanes);
    t.adj = reinterpret_cast<unsigned short *>(t.scratch + t.block * t.lanes * 8);
    t.flag = reinterpret_cast<unsigned char *>(t.adj + ((c.base * c.d + 1) & ~1));
    each_int(c.adj, c.base * c.d, tid, THREADS, [&](int i, int x) { t.adj[i] = (unsigned short)x; });
    each_int(c.nbr + (size_t)t.r0 * c.dp, t.nr * c.dp, tid, THREADS, [&](int i, int x) { t.list[i] = x; });
    if(tid < 31) sh.rng.ring[tid] = c.ring[tid];
    if(tid == 0){
      sh.rng.pos = c.ring_pos;
      sh.cnt[0] = sh.cnt[1] = sh.cnt1[0] = sh.cnt1[1] = 0;
      sh.g.n = c.n; sh.g.d = c.d; sh.g.s = c.s; sh.g.base = c.base;
      sh.g.ndeg = c.ndeg; sh.g.adj = t.adj; sh.g.nw = 0;
      sh.gg.w = c.width; sh.gg.h = c.height; sh.gg.d = c.d; sh.gg.s = c.s; sh.gg.len = c.len; sh.gg.n = c.n;
      sh.gg.bw = c.width / 2; sh.gg.bh = (c.s == 2) ? c.height : c.height / 2;
      sh.gg.ndeg = c.ndeg; sh.gg.adj = t.adj; sh.gg.xy = nullptr; sh.gg.nw = 0;
    }
    /* every CTA has its copy of the adjacency before the first one writes to it */
    unsigned long long bits, bits1;
    bool met = team_pass<CLUSTER>(sh, t, p.limit_ns, false, bits, bits1);
    __syncthreads();                                     /* sh.ok is read before the proposal writes it */
    for(int step = 0; met && step < p.steps && !sh.c.status; step++){
      if(tid == 0) sh.ok = propose(sh);
      __syncthreads();
      if(!sh.ok){                                        /* in every CTA: out of draws */
        if(tid == 0) sh.c.status = GBX_CHAIN_ERR_SWAP;
        __syncthreads();
        break;
      }
      spread_writes<THREADS>(sh, t);
      __syncthreads();
      int level = 0;
      long long sum = 0;
      met = evaluate<CLUSTER>(sh, t, p.limit_ns, level, sum);
      if(!met) break;
      if(tid == 0) decide(sh, level, sum);
      __syncthreads();
      if(sh.copy && t.rank == 0)
        each_int(c.adj, c.base * c.d, tid, THREADS, [best = c.best_adj](int i, int x) { best[i] = x; });
      if(!sh.accept){
        __syncthreads();                                 /* the copy has read the adjacency before the undo */
        if(tid == 0) undo(sh);
        __syncthreads();
        spread_writes<THREADS>(sh, t);
        __syncthreads();
      }
    }
    /* A CTA whose wait ran out left with the rows it had, perhaps before a
     * decision that all others took: the first CTA then misses it here, if not
     * before, and the chain is stopped. */
    if(met && sh.c.status != GBX_CHAIN_ERR_EVAL) met = team_pass<CLUSTER>(sh, t, p.limit_ns, false, bits, bits1);
    if(!met && tid == 0){
      sh.c.status = GBX_CHAIN_ERR_EVAL;
      *p.late = 1u;
    }
    __syncthreads();
    /* the records and the neighbour table, for the host and the next launch;
     * after a run the chain also goes to host memory, a part from each CTA:
     * three copies and a synchronise per chain took 40 us.  A CTA that has not
     * met the others copies nothing: the first one may still be writing the
     * graph. */
    if(met && p.host_chains){
      const int ints = c.base * c.d;
      int *to = p.host_graphs + p.host_offset[chain];
      each_int(c.adj, ints, t.rank * THREADS + tid, t.size * THREADS, [to](int i, int x) { to[i] = x; });
      each_int(c.best_adj, ints, t.rank * THREADS + tid, t.size * THREADS, [to, ints](int i, int x) { to[ints + i] = x; });
    }
    for(int i = tid; i < t.nr * c.dp; i += THREADS) c.nbr[(size_t)t.r0 * c.dp + i] = t.list[i];
    if(t.rank == 0){
      if(tid < 31) sh.c.ring[tid] = sh.rng.ring[tid];
      if(tid == 0) sh.c.ring_pos = sh.rng.pos;
      __syncthreads();
      unsigned *dst = reinterpret_cast<unsigned *>(p.chains + chain);
      unsigned *host = reinterpret_cast<unsigned *>(p.host_chains + chain);
      const unsigned *src = reinterpret_cast<const unsigned *>(&sh.c);
      for(int i = tid; i < (int)(sizeof(gbx_chain) / 4); i += THREADS){
        dst[i] = src[i];
        if(p.host_chains) host[i] = src[i];
      }
    }
  }
}

}  // namespace

extern "C" {

size_t gbx_resident_sync_bytes(void) { return sizeof(ResidentSync); }

size_t gbx_resident_smem(int rows, int dp, int base, int d)
{
  const size_t lanes = ((size_t)base + 255) / 256;
  return (size_t)rows * dp * 4 + (size_t)resident_block(rows, (int)lanes) * lanes * 32 + (((size_t)base * d + 1) & ~(size_t)1) * 2 + rows * lanes;
}

int gbx_resident_blocks(size_t smem, int *per_sm)
{
  *per_sm = 0;
  if(smem > GBX_SWEEP_SMEM_MAX) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute((const void *)anneal_resident_kernel<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, GBX_SWEEP_SMEM_MAX);
  if(e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, (const void *)anneal_resident_kernel<false>,
                                                      RESIDENT_THREADS, smem);
  if(e != cudaSuccess) cudaGetLastError();
  return (int)e;
}

static void resident_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr, int blocks, size_t smem, int cluster)
{
  if(cluster){
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  }
  else{
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  cfg.gridDim = dim3((unsigned)blocks, 1, 1);
  cfg.blockDim = dim3(cluster ? GBX_RESIDENT_CLUSTER_THREADS : RESIDENT_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

int gbx_resident_clusters(int cluster, size_t smem, int *active)
{
  *active = 0;
  if(smem > GBX_SWEEP_SMEM_MAX || cluster > RESIDENT_CLUSTER) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute((const void *)anneal_resident_kernel<true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, GBX_SWEEP_SMEM_MAX);
  if(e == cudaSuccess)
    e = cudaFuncSetAttribute((const void *)anneal_resident_kernel<true>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if(e != cudaSuccess){
    cudaGetLastError();
    return (int)e;
  }
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  resident_config(cfg, attr, cluster, smem, cluster);
  e = cudaOccupancyMaxActiveClusters(active, (const void *)anneal_resident_kernel<true>, &cfg);
  if(e != cudaSuccess) cudaGetLastError();
  return (int)e;
}

int gbx_resident_launch(const gbx_resident *r, int blocks, size_t smem, int cluster, void *stream)
{
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  resident_config(cfg, attr, blocks, smem, cluster);
  cfg.stream = (cudaStream_t)stream;
  gbx_resident arg = *r;
  void *args[1] = { &arg };
  return (int)cudaLaunchKernelExC(&cfg, cluster ? (const void *)anneal_resident_kernel<true>
                                                : (const void *)anneal_resident_kernel<false>, args);
}

}  /* extern "C" */
