/*
 * sweep.cu -- graphs evaluated in lockstep: one graph by every SM, or many by
 * teams of CTAs.
 *
 * The persistent engine (aspl_engine.cu) hands every level of every job out
 * in tiles through a ticket.  That suits many uneven graphs, but a single
 * graph pays about 10 us per level for it on GB300 (read the ticket, fence,
 * read the slot, stage the neighbour lists, gather, count, fence, close),
 * where the level's traffic takes 1 to 5 us for a few thousand vertices.
 * Here the rows are split over the CTAs once: each CTA keeps its rows'
 * neighbour lists in shared memory for the whole call, and a level is one
 * pass over its own rows and one grid-wide barrier, whose word also carries
 * the level's bit count.  A call is one cooperative launch (all CTAs are
 * resident, so they may wait for one another; every wait has a time limit).
 *
 * The unit of work is a lane: 32 bytes of a row (256 sources, one sector),
 * moved by one 256-bit access.
 *
 * sweep_dense_kernel (general graphs): the first levels (one, two, or without
 * symmetry up to GBX_SWEEP_BASE) come from the neighbour lists, marked in shared
 * memory and stored once; after them every lane that is not full gathers, and
 * stops as soon as it is.
 *
 * sweep_track_kernel (grids): rows and sources follow a Hilbert curve, so the
 * 256 sources of a lane lie close together and a row's lane changes in a few
 * levels only.  Every row keeps one bit per lane, "changed at this level"
 * (65536 sources: one 32-byte sector per row); a lane with no changed
 * neighbour is not visited, and one that is gathers its changed neighbours
 * alone.
 */
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include "odp_engine.h"
#include "odp_device.cuh"

#define SWEEP_THREADS 256
#define SWEEP_WARPS (SWEEP_THREADS / 32)
#define SWEEP_SLOTS GBX_SWEEP_SLOTS   /* column chunks a phase runs at once, at most */

namespace {

/* Counters of one graph's evaluation by PH phases over at most CH chunks;
 * the evaluation before clears them. */
template <int PH, int CH>
struct SyncT {
  unsigned ready[3];                                 /* CTAs past the copy, the expansion, the start */
  unsigned err;                                      /* GBX_ERR_* */
  unsigned pad[28];
  unsigned long long arrive[PH][3][16];              /* step t's barrier word: [t % 3][0] */
  unsigned long long count[PH][3][SWEEP_SLOTS];      /* bits per chunk of step t */
  unsigned long long start[2 * CH];                  /* bits per chunk at levels 1 to `base`: [base][nchunks] */
};
typedef SyncT<GBX_SWEEP_PHASES, GBX_SWEEP_CHUNKS> SweepSync;

/* A phase's progress, the same in every CTA but for `prev`, `sum` and
 * `alive`, which CTA 0 keeps for the records. */
struct SweepPhase {
  unsigned long long total, full;                    /* bits set at the last level; bits of a complete group */
  unsigned long long t_loaded;
  int level, group;                                  /* level < 0: no group left */
  unsigned step, alive;
  unsigned long long prev[SWEEP_SLOTS];
  long long sum[SWEEP_SLOTS];
};

struct SweepShared {
  SweepPhase ph[GBX_SWEEP_PHASES];
  unsigned cnt[SWEEP_SLOTS];                         /* this CTA's bits per chunk of the current step */
  int todo;
  int rank, size;                                    /* of this CTA among those that evaluate the graph */
  unsigned long long begin;                          /* when it began the graph */
};

#define TODO_DONE 0
#define TODO_LEVEL 1
#define TODO_ABORT 2

/* The whole grid passes; false (in every thread) past the limit. */
__device__ __forceinline__ bool grid_pass(unsigned *word, SweepShared &sh, const gbx_sweep &a)
{
  __syncthreads();
  if(threadIdx.x == 0){
    unsigned seen;
    arrive_word(word, 1u);
    const bool ok = wait_for(word, (unsigned)sh.size, seen, a.limit_ns);
    sh.todo = ok ? TODO_LEVEL : TODO_ABORT;
    if(!ok) *a.abort_flag = GBX_ERR_TIMEOUT;           /* pinned host memory */
  }
  __syncthreads();
  const bool ok = sh.todo != TODO_ABORT;
  __syncthreads();                                     /* read before it is written again */
  return ok;
}

/* Sources of chunk c. */
__device__ __forceinline__ int chunk_sources(const gbx_sweep &a, int c)
{
  const int C = 64 << a.wc_log2;
  return c < a.nchunks ? min(C, a.B - c * C) : 0;
}

/* First chunk of the phase's group. */
__device__ __forceinline__ int group_chunk(const gbx_sweep &a, int group, int ph)
{
  return (group * a.phases + ph) * a.slots;
}

/* A chunk's bits after `level` (CTA 0, the thread of the chunk): records the
 * chunk when it is complete or stalled (then false), else adds the level's
 * share of the distance sum. */
template <class Sync>
__device__ __forceinline__ bool settle(const gbx_sweep &a, SweepPhase &p, const Sync &sy, int chunk, int q,
                                       int level, unsigned long long c)
{
  const unsigned long long full = (unsigned long long)a.e.n * (unsigned long long)chunk_sources(a, chunk);
  const bool complete = c == full;
  const bool stalled = !complete && (c == p.prev[q] || level >= a.e.n);
  if(!complete && !stalled){
    p.sum[q] += (long long)(full - c) * a.e.s;
    p.prev[q] = c;
    return true;
  }
  gbx_small_rec r;
  r.level = stalled ? -level : level;
  r.err = __ldcg(&sy.err) | a.seq << 8;
  r.sum = p.sum[q];
  r.t_loaded = p.t_loaded;
  r.t_done = globaltimer();
  store_record(a.rec + chunk, r);
  return false;
}

/* CTA 0, warp 0: the chunks' counts of step `step`, which ended `level`.
 * `added`: the counts are of bits added. */
template <class Sync>
__device__ __forceinline__ void settle_step(const gbx_sweep &a, SweepPhase &p, const Sync &sy, int ph,
                                            unsigned step, int level, bool added)
{
  const int q = threadIdx.x;
  bool go = (p.alive >> q) & 1u;
  if(go){
    unsigned long long c = __ldcg(&sy.count[ph][step % 3][q]);
    if(added) c += p.prev[q];
    go = settle(a, p, sy, group_chunk(a, p.group, ph) + q, q, level, c);
  }
  const unsigned alive = __ballot_sync(0xffffffffu, go);
  if(q == 0) p.alive = alive;
  __syncwarp();
}

/* Warp 0: a phase's state at the start of a group (no level counted yet). */
__device__ __forceinline__ void group_state(const gbx_sweep &a, SweepPhase &p, int ph, int group)
{
  const int q = threadIdx.x;
  const int nsrc = q < a.slots ? chunk_sources(a, group_chunk(a, group, ph) + q) : 0;
  if(q < a.slots){
    p.prev[q] = (unsigned long long)nsrc;
    p.sum[q] = ((long long)a.e.n * nsrc - nsrc) * a.e.s;
  }
  const unsigned alive = __ballot_sync(0xffffffffu, nsrc > 0);
  const unsigned all = __reduce_add_sync(0xffffffffu, (unsigned)nsrc);
  __syncwarp();                                        /* every lane has read the last group's state */
  if(q == 0){
    p.group = group;
    p.alive = alive;
    p.total = all;
    p.full = (unsigned long long)a.e.n * all;
    p.level = alive ? 0 : -1;
    p.t_loaded = globaltimer();
  }
  __syncwarp();
}

/* Warp 0 publishes the CTA's part of a step: the counts per chunk, then one
 * barrier word with their total.  CTA 0 first clears the next step's words:
 * their last readers (step - 2) have all arrived at step - 1, which this CTA
 * has waited for, and nobody adds to them before it arrives. */
template <class Sync>
__device__ __forceinline__ void arrive_step(const gbx_sweep &a, SweepShared &sh, Sync &sy, int ph)
{
  const int q = threadIdx.x;
  const unsigned step = sh.ph[ph].step;
  const unsigned c = q < a.slots ? sh.cnt[q] : 0u;
  if(q < a.slots){
    if(sh.rank == 0) sy.count[ph][(step + 1) % 3][q] = 0;
    if(c) atomicAdd(&sy.count[ph][step % 3][q], (unsigned long long)c);
    sh.cnt[q] = 0;
  }
  const unsigned total = __reduce_add_sync(0xffffffffu, c);   /* rows x lanes x 256 of one CTA: below 2^32 */
  __syncwarp();          /* lane 0's release covers the other lanes' counts (a reduction orders no memory) */
  if(q == 0){
    if(sh.rank == 0) sy.arrive[ph][(step + 1) % 3][0] = 0;
    arrive_word(&sy.arrive[ph][step % 3][0], ARRIVE_ONE | total);
    sh.ph[ph].step = step + 1;
  }
  __syncwarp();
}

/* Warp 0 waits for the phase's last step and takes its count (true), or past
 * the limit gives up.  CTA 0 settles the step before meanwhile.  Lane 0
 * acquires the barrier word; the warp barrier hands that on to the lanes that
 * read the chunks' counts, and has them past their reads of the phase's state
 * before lane 0 writes the next one. */
template <class Sync>
__device__ __forceinline__ bool wait_step(const gbx_sweep &a, SweepShared &sh, Sync &sy, int ph, bool added,
                                          int first_level, unsigned long long &bits)
{
  SweepPhase &p = sh.ph[ph];
  const unsigned step = p.step;
  if(sh.rank == 0 && p.level > first_level) settle_step(a, p, sy, ph, step - 2, p.level - 1, added);
  unsigned long long seen = 0;
  bool ok = true;
  if(threadIdx.x == 0) ok = wait_for(&sy.arrive[ph][(step - 1) % 3][0], ARRIVE_ONE * (unsigned)sh.size, seen, a.limit_ns);
  __syncwarp();
  ok = __all_sync(0xffffffffu, ok);
  bits = __shfl_sync(0xffffffffu, seen, 0) & ARRIVE_BITS;
  return ok;
}

/* This CTA's place among those that evaluate the graph, and clean counts. */
__device__ __forceinline__ void sweep_begin(SweepShared &sh, int rank, int size)
{
  if(threadIdx.x < SWEEP_SLOTS) sh.cnt[threadIdx.x] = 0;
  if(threadIdx.x < GBX_SWEEP_PHASES) sh.ph[threadIdx.x].step = 0;
  if(threadIdx.x == 0){
    sh.rank = rank;
    sh.size = size;
    sh.begin = globaltimer();
  }
  __syncthreads();
}

/* A launch of one graph alternates between two sets of counters; CTA 0
 * clears the other one for the next launch. */
__device__ __forceinline__ SweepSync &launch_sync(const gbx_sweep &a)
{
  SweepSync *sy = reinterpret_cast<SweepSync *>(a.sync);
  if(blockIdx.x == 0){
    unsigned *other = reinterpret_cast<unsigned *>(sy + (a.set ^ 1));
    for(int i = threadIdx.x; i < (int)(sizeof(SweepSync) / 4); i += SWEEP_THREADS) other[i] = 0;
  }
  return sy[a.set];
}

/* The CTA's slice of the compact adjacency out of host memory; then the
 * whole grid has the device copy.  False past the limit. */
template <class Sync>
__device__ __forceinline__ bool pull_adjacency(const gbx_sweep &a, SweepShared &sh, Sync &sy)
{
  if(!a.e.adj_dev || a.in_place) return true;
  const long long ints = (long long)a.B * a.e.d;
  const long long t0 = (long long)sh.rank * SWEEP_THREADS + threadIdx.x;
  const long long stride = (long long)sh.size * SWEEP_THREADS;
  if(((reinterpret_cast<uintptr_t>(a.e.adj) | reinterpret_cast<uintptr_t>(a.e.adj_dev)) & 15) == 0){
    /* several reads in flight per thread: a small team's copy is bound by the
     * host link's latency */
    const int4 *src = reinterpret_cast<const int4 *>(a.e.adj);
    int4 *dst = reinterpret_cast<int4 *>(a.e.adj_dev);
    const int q = (int)(ints >> 2), st = sh.size * SWEEP_THREADS;
    for(int i0 = (int)t0; i0 < q; i0 += st * 8){
      int4 x[8];
#pragma unroll
      for(int k = 0; k < 8; k++) x[k] = src[min(i0 + k * st, q - 1)];
#pragma unroll
      for(int k = 0; k < 8; k++) dst[min(i0 + k * st, q - 1)] = x[k];
    }
    if(sh.rank == 0)
      for(long long i = (ints & ~3LL) + threadIdx.x; i < ints; i += SWEEP_THREADS) a.e.adj_dev[i] = a.e.adj[i];
  }
  else
    for(long long i = t0; i < ints; i += stride) a.e.adj_dev[i] = a.e.adj[i];
  return grid_pass(&sy.ready[0], sh, a);
}

/* The neighbour lists of the CTA's rows row0 + i * drow, i < nr, in shared
 * memory (and the table, if given).  2^lr threads share a row, eight rows in
 * flight per thread. */
template <class Sync>
__device__ __forceinline__ void expand_rows(const gbx_sweep &a, Sync &sy, int *list, int row0, int drow, int nr,
                                            int *table)
{
  const int *adj = a.e.adj_dev && !a.in_place ? a.e.adj_dev : a.e.adj;
  const int d = a.e.d, dp = a.e.dp;
  int lr = 2;
  while((1 << lr) < dp && lr < 5) lr++;
  const int per = SWEEP_THREADS >> lr;
  const int base = a.B;
  const float inv = 1.0f / (float)base;
  bool bad = false;
  for(int j = threadIdx.x & ((1 << lr) - 1); j < dp; j += 1 << lr)
    for(int i0 = threadIdx.x >> lr; i0 < nr; i0 += per * 8){
      int val[8], back[8], deg[8];
#pragma unroll
      for(int k = 0; k < 8; k++){
        const int i = i0 + k * per;
        back[k] = val[k] = deg[k] = 0;
        if(i < nr){
          const int row = row0 + i * drow;
          const int v = a.row_vertex ? __ldg(a.row_vertex + row) : row;
          deg[k] = a.e.ndeg ? __ldg(a.e.ndeg + v) : d;
          if(deg[k] < 0 || deg[k] > d){ bad = true; deg[k] = deg[k] < 0 ? 0 : d; }
          if(a.e.grid_s){
            if(j < deg[k]) val[k] = __ldcg(adj + entry_source(a.e, v, j, back[k]));
          }
          else{
            /* entry_source's quotient v / base, estimated and put right */
            int q = (int)((float)v * inv), m = v - q * base;
            if(m < 0){ q--; m += base; }
            if(m >= base){ q++; m -= base; }
            back[k] = q * base;
            if(j < deg[k]) val[k] = __ldcg(adj + (size_t)m * d + j);
          }
        }
      }
#pragma unroll
      for(int k = 0; k < 8; k++){
        const int i = i0 + k * per;
        if(i < nr){
          const int row = row0 + i * drow;
          const int x = expand_value(a.e, val[k], back[k], j, deg[k], row, bad);
          list[i * dp + j] = x;
          if(table) __stcg(table + (size_t)row * dp + j, x);
        }
      }
    }
  if(bad) atomicOr(&sy.err, GBX_ERR_BAD_ADJ);
}

/* ---------------------------------------------------------------------- */
/* General graphs.                                                         */
/* ---------------------------------------------------------------------- */

/* Levels 1 and 2 of every chunk (level 1 alone for base 1), a warp per row.  The warp marks the
 * row, its neighbours and their neighbours in its scratch row (scratch_bits
 * sources at a time) and stores each lane once.  A level-2 gather would read
 * d whole rows per row, nearly all of them zeros; this reads d neighbour
 * lists once for all chunks, and level 1 is never stored. */
__device__ void start_rows(const gbx_sweep &a, const int *list, unsigned *scratch, unsigned *cnt1, unsigned *cnt2,
                           int r0, int nr)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lL = a.wc_log2 - 2, L = 1 << lL;             /* lanes per row of a chunk */
  const int dp = a.e.dp, d = a.e.d;
  const int q4 = dp >> 2, magic = (65536 + q4 - 1) / q4;  /* i / q4 for i < 1024, q4 <= 16 */
  unsigned *s = scratch + (size_t)warp * (a.scratch_bits >> 5);
  for(int r = warp; r < nr; r += SWEEP_WARPS){
    const int *ids = list + r * dp;
    for(int sb = 0; sb < a.B; sb += a.scratch_bits){
      const int sub = min(a.B - sb, a.scratch_bits);
      const int pieces = (sub + 255) >> 8;
      uint4 *sv = reinterpret_cast<uint4 *>(s);
      for(int i = lane; i < pieces * 2; i += 32) sv[i] = make_uint4(0u, 0u, 0u, 0u);
      __syncwarp();
      for(int i = lane; i <= dp; i += 32) mark(s, (i < dp ? ids[i] : r0 + r) - sb, sub);
      __syncwarp();
      if(a.base == 2){
        for(int p0 = 0; p0 < pieces; p0 += 32){          /* level 1's counts */
          const int p = p0 + lane;
          unsigned v = 0;
          if(p < pieces){
            const uint4 x = sv[2 * p], y = sv[2 * p + 1];
            v = popc4(x) + popc4(y);
          }
          for(int o = L >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if(v && (lane & (L - 1)) == 0) atomicAdd(cnt1 + (((sb >> 8) + p) >> lL), v);
        }
        __syncwarp();
        /* six pieces of lists in flight per lane */
        for(int i0 = lane; i0 < d * q4; i0 += 192){
          int4 x[6];
#pragma unroll
          for(int k = 0; k < 6; k++){
            const int i = i0 + 32 * k, j = (i * magic) >> 16;
            if(i < d * q4) x[k] = __ldcg(reinterpret_cast<const int4 *>(a.e.nbr + (size_t)ids[j] * dp) + (i - j * q4));
            else x[k] = make_int4(-1, -1, -1, -1);
          }
#pragma unroll
          for(int k = 0; k < 6; k++){
            mark(s, x[k].x - sb, sub);
            mark(s, x[k].y - sb, sub);
            mark(s, x[k].z - sb, sub);
            mark(s, x[k].w - sb, sub);
          }
        }
        __syncwarp();
      }
      for(int p0 = 0; p0 < pieces; p0 += 32){
        const int p = p0 + lane;
        unsigned w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        const int c = ((sb >> 8) + p) >> lL, gl = ((sb >> 8) + p) & (L - 1);
        if(p < pieces){
          *reinterpret_cast<uint4 *>(w) = sv[2 * p];
          *reinterpret_cast<uint4 *>(w + 4) = sv[2 * p + 1];
          char *to = reinterpret_cast<char *>(a.start + (size_t)c * a.start_stride);
          st_lane(to + ((size_t)(r0 + r) << (a.wc_log2 + 3)) + (size_t)gl * 32, w);
        }
        unsigned v = popc_lane(w);
        for(int o = L >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if(v && (lane & (L - 1)) == 0) atomicAdd(cnt2 + c, v);
      }
      __syncwarp();                                      /* the scratch row is read before it is cleared again */
    }
  }
}

/* Levels 1 to `base` > 2 of every chunk, a warp per row: a search from the row
 * over the neighbour table, the vertices reached as bits in the warp's scratch
 * row and in its queue.  A gathered level reads d whole rows a row however few
 * bits they hold: for n = 65536, d = 16 level 3 took 500 us gathered and takes
 * 190 from the lists.  The counts of the levels before the last are of
 * vertices added.  The queue holds a whole tree of the levels before the last,
 * whether or not the lists are symmetric. */
__device__ void ball_rows(const gbx_sweep &a, const int *list, unsigned *scratch, unsigned *cnt, int r0, int nr)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lL = a.wc_log2 - 2, L = 1 << lL;
  const int dp = a.e.dp, n = a.e.n, last = a.base;
  const int q4 = dp >> 2, magic = (65536 + q4 - 1) / q4;
  const int words = a.scratch_bits >> 5, pieces = a.scratch_bits >> 8;
  if(warp >= a.scratch_rows) return;
  unsigned *s = scratch + (size_t)warp * (words + a.queue);
  int *queue = reinterpret_cast<int *>(s + words);
  uint4 *sv = reinterpret_cast<uint4 *>(s);
  const unsigned below = (1u << lane) - 1u;
  for(int r = warp; r < nr; r += a.scratch_rows){
    const int own = r0 + r;
    const int *ids = list + r * dp;
    for(int i = lane; i < pieces * 2; i += 32) sv[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    if(lane == 0){
      s[own >> 5] = 1u << (own & 31);
      atomicAdd(cnt + (own >> (lL + 8)), 1u);
    }
    __syncwarp();
    int lo = 0, hi = 0;                                  /* the last level's vertices in the queue (level 1: the row itself) */
    for(int level = 1; level < last; level++){
      unsigned *c = cnt + (level - 1) * a.nchunks;
      const int total = level == 1 ? q4 : (hi - lo) * q4;
      int end = hi;
      for(int i0 = 0; i0 < total; i0 += 128){
        int4 x[4];
#pragma unroll
        for(int k = 0; k < 4; k++){
          const int i = i0 + 32 * k + lane;
          if(i >= total) x[k] = make_int4(-1, -1, -1, -1);
          else if(level == 1) x[k] = *reinterpret_cast<const int4 *>(ids + 4 * i);
          else{
            const int j = i < 1024 ? (i * magic) >> 16 : i / q4;
            x[k] = __ldcg(reinterpret_cast<const int4 *>(a.e.nbr + (size_t)queue[lo + j] * dp) + (i - j * q4));
          }
        }
#pragma unroll
        for(int k = 0; k < 4; k++){
          if(i0 + 32 * k >= total) break;
          const int v[4] = { x[k].x, x[k].y, x[k].z, x[k].w };
#pragma unroll
          for(int m = 0; m < 4; m++){
            bool add = false;
            if((unsigned)v[m] < (unsigned)n){
              const unsigned bit = 1u << (v[m] & 31);
              add = !(atomicOr(s + (v[m] >> 5), bit) & bit);
            }
            const unsigned who = __ballot_sync(0xffffffffu, add);
            if(add){
              queue[end + __popc(who & below)] = v[m];
              atomicAdd(c + (v[m] >> (lL + 8)), 1u);
            }
            end += __popc(who);
          }
        }
      }
      __syncwarp();
      lo = hi;
      hi = end;
    }
    {
      const int total = (hi - lo) * q4;
      for(int i0 = lane; i0 < total; i0 += 192){
        int4 x[6];
#pragma unroll
        for(int k = 0; k < 6; k++){
          const int i = i0 + 32 * k, j = i < 1024 ? (i * magic) >> 16 : i / q4;
          if(i < total) x[k] = __ldcg(reinterpret_cast<const int4 *>(a.e.nbr + (size_t)queue[lo + j] * dp) + (i - j * q4));
          else x[k] = make_int4(-1, -1, -1, -1);
        }
#pragma unroll
        for(int k = 0; k < 6; k++){
          mark(s, x[k].x, n);
          mark(s, x[k].y, n);
          mark(s, x[k].z, n);
          mark(s, x[k].w, n);
        }
      }
    }
    __syncwarp();
    unsigned *c = cnt + (last - 1) * a.nchunks;
    for(int p0 = 0; p0 < pieces; p0 += 32){
      const int p = p0 + lane, q = p >> lL;
      unsigned w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if(p < pieces){
        *reinterpret_cast<uint4 *>(w) = sv[2 * p];
        *reinterpret_cast<uint4 *>(w + 4) = sv[2 * p + 1];
        char *to = reinterpret_cast<char *>(a.start + (size_t)q * a.start_stride);
        st_lane(to + ((size_t)own << (a.wc_log2 + 3)) + (size_t)(p & (L - 1)) * 32, w);
      }
      unsigned v = popc_lane(w);
      for(int o = L >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if(v && (lane & (L - 1)) == 0) atomicAdd(c + q, v);
    }
    __syncwarp();
  }
}

/* One level of the phase's group over the CTA's rows: a thread keeps its lane
 * and walks the rows.  `first`: the group's first gathered level, whose lanes
 * have no state yet. */
template <int NB>
__device__ void level_rows(const gbx_sweep &a, SweepShared &sh, const int *list, unsigned char *flag, int ph,
                           bool first, int r0, int nr)
{
  const int lL = a.wc_log2 - 2, L = 1 << lL, Q = a.slots, dp = a.e.dp, d = a.e.d;
  const unsigned rb = 8u << a.wc_log2;
  const int level = sh.ph[ph].level, c0 = group_chunk(a, sh.ph[ph].group, ph);
  const int nsrc = min(Q << (lL + 8), a.B - (c0 << (lL + 8)));
  const int lanes = (nsrc + 255) >> 8;                   /* at most SWEEP_THREADS */
  const int rr = threadIdx.x / lanes, rs = SWEEP_THREADS / lanes;
  unsigned cnt = 0;
  int q = 0;
  if(rr < rs){
    const int at = threadIdx.x - rr * lanes, gl = at & (L - 1);
    q = at >> lL;
    const unsigned bits = (unsigned)lane_bits(nsrc, at);
    const size_t words = a.slot_words;
    const unsigned long long *x = first ? a.start + (size_t)(c0 + q) * a.start_stride
                                        : a.buf + ((size_t)(ph * Q + q) * 2 + ((level & 1) ^ 1)) * words;
    const char *X = reinterpret_cast<const char *>(x) + gl * 32;
    char *Y = reinterpret_cast<char *>(a.buf + ((size_t)(ph * Q + q) * 2 + (level & 1)) * words) + gl * 32;
    unsigned char *fl = flag + (((ph * Q + q) * a.rows) << lL) + gl;
    for(int row = rr; row < nr; row += rs){
      const unsigned f = first ? LANE_CHANGED : fl[row << lL];
      unsigned acc[8];
      if(f & LANE_FULL){
        cnt += bits;
        if(f & LANE_CHANGED){
          if(bits == 256u){
#pragma unroll
            for(int k = 0; k < 8; k++) acc[k] = ~0u;
          }
          else ld_lane(acc, X + (size_t)(unsigned)(r0 + row) * rb);
          st_lane(Y + (size_t)(unsigned)(r0 + row) * rb, acc);
          fl[row << lL] = LANE_FULL;
        }
        continue;
      }
      ld_lane(acc, X + (size_t)(unsigned)(r0 + row) * rb);
      gather_lane<NB>(acc, X, list + row * dp, d, rb);
      st_lane(Y + (size_t)(unsigned)(r0 + row) * rb, acc);
      const unsigned c = popc_lane(acc);
      cnt += c;
      if(first || c == bits) fl[row << lL] = LANE_CHANGED | (c == bits ? LANE_FULL : 0u);
    }
  }
  if(Q == 1){
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if((threadIdx.x & 31) == 0) atomicAdd(&sh.cnt[0], cnt);
  }
  else if(cnt) atomicAdd(&sh.cnt[q], cnt);
}

/* Warp 0: what the phase does next.  After the group's last level (complete,
 * or a level that added nothing) the next group begins. */
template <class Sync>
__device__ __forceinline__ void plan_dense(const gbx_sweep &a, SweepShared &sh, Sync &sy, int ph)
{
  SweepPhase &p = sh.ph[ph];
  const int base = a.base;                               /* the level that the start computed */
  int todo = -1;
  if(p.level > base){
    unsigned long long bits;
    if(!wait_step(a, sh, sy, ph, false, base + 1, bits)) todo = TODO_ABORT;
    else{
      const bool over = bits == p.full || bits == p.total || p.level >= a.e.n;
      __syncwarp();
      if(over){
        if(sh.rank == 0) settle_step(a, p, sy, ph, p.step - 1, p.level, false);
        group_state(a, p, ph, p.group + 1);
      }
      else{
        todo = TODO_LEVEL;
        if(threadIdx.x == 0){ p.total = bits; p.level++; }
      }
    }
  }
  while(todo < 0){
    /* the group's levels up to `base`, counted at the start */
    if(p.level < 0){ todo = TODO_DONE; break; }
    const int q = threadIdx.x, chunk = group_chunk(a, p.group, ph) + q;
    const bool mine = (p.alive >> q) & 1u;
    unsigned long long t1 = p.total;
    bool go = mine, over = false;
    for(int j = 1; j <= base; j++){
      const unsigned long long c = mine ? __ldcg(&sy.start[(j - 1) * a.nchunks + chunk]) : 0ull;
      unsigned long long t2 = c;
      for(int o = 16; o > 0; o >>= 1) t2 += __shfl_xor_sync(0xffffffffu, t2, o);
      if(sh.rank == 0 && go) go = settle(a, p, sy, chunk, q, j, c);
      over |= t2 == p.full || t2 == t1 || a.e.n <= j;
      t1 = t2;
    }
    if(sh.rank == 0){
      const unsigned alive = __ballot_sync(0xffffffffu, go);
      if(q == 0) p.alive = alive;
    }
    __syncwarp();                                      /* read before it is written */
    if(over) group_state(a, p, ph, p.group + 1);
    else{
      todo = TODO_LEVEL;
      if(q == 0){ p.total = t1; p.level = base + 1; }
    }
    __syncwarp();
  }
  if(threadIdx.x == 0) sh.todo = todo;
  __syncwarp();
}

/* The whole evaluation by the CTAs of sh (all threads; false past a wait's
 * limit).  after_pass() runs once, when every CTA has begun the graph. */
template <int NB, class Sync, class AfterPass>
__device__ bool dense_graph(const gbx_sweep &a, SweepShared &sh, Sync &sy, unsigned char *smem, AfterPass after_pass)
{
  const int tid = threadIdx.x, dp = a.e.dp;
  const int r0 = sh.rank * a.rows, nr = max(0, min(a.rows, a.e.n - r0));
  int *list = reinterpret_cast<int *>(smem);                                     /* [rows][dp] */
  unsigned *scratch = reinterpret_cast<unsigned *>(list + (size_t)a.rows * dp);  /* a row of marks per warp */
  unsigned *cnt = scratch + a.scratch_rows * ((a.scratch_bits >> 5) + a.queue);  /* [base][nchunks] */
  unsigned char *flag = reinterpret_cast<unsigned char *>(cnt + a.base * a.nchunks);  /* [phases * slots][rows][lanes] */
  for(int i = tid; i < a.base * a.nchunks; i += SWEEP_THREADS) cnt[i] = 0;
  if(!pull_adjacency(a, sh, sy)) return false;
  expand_rows(a, sy, list, r0, 1, nr, a.base > 1 ? a.e.nbr : nullptr);
  if(a.base > 1){
    if(!grid_pass(&sy.ready[1], sh, a)) return false;
  }
  else __syncthreads();
  if(a.base > 2) ball_rows(a, list, scratch, cnt, r0, nr);
  else start_rows(a, list, scratch, cnt, cnt + (a.base - 1) * a.nchunks, r0, nr);
  __syncthreads();
  for(int c = tid; c < a.nchunks; c += SWEEP_THREADS){
    unsigned sum = 0;
    for(int j = 0; j < a.base; j++){
      const unsigned x = cnt[j * a.nchunks + c];
      sum = a.base > 2 && j < a.base - 1 ? sum + x : x;  /* ball_rows counts what a level adds, but for the last */
      if(sum) atomicAdd(&sy.start[j * a.nchunks + c], (unsigned long long)sum);
    }
  }
  if(!grid_pass(&sy.ready[2], sh, a)) return false;
  after_pass();
  if(tid < 32)
    for(int ph = 0; ph < a.phases; ph++){
      group_state(a, sh.ph[ph], ph, 0);
      if(tid == 0) sh.ph[ph].t_loaded = sh.begin;
    }

  unsigned open = (1u << a.phases) - 1u;                 /* phases with groups left */
  while(open)
    for(int ph = 0; ph < a.phases; ph++){
      if(!((open >> ph) & 1u)) continue;
      __syncthreads();
      if(tid < 32) plan_dense(a, sh, sy, ph);
      __syncthreads();
      const int todo = sh.todo;
      if(todo == TODO_ABORT){
        if(tid == 0) *a.abort_flag = GBX_ERR_TIMEOUT;
        return false;
      }
      if(todo == TODO_DONE){ open &= ~(1u << ph); continue; }
      level_rows<NB>(a, sh, list, flag, ph, sh.ph[ph].level == a.base + 1, r0, nr);
      __syncthreads();
      if(tid < 32) arrive_step(a, sh, sy, ph);
    }
  __syncthreads();
  return true;
}

template <int NB, int MIN_BLOCKS>
__global__ void __launch_bounds__(SWEEP_THREADS, MIN_BLOCKS) sweep_dense_kernel(const gbx_sweep a)
{
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  __shared__ SweepShared sh;
  SweepSync &sy = launch_sync(a);
  sweep_begin(sh, (int)blockIdx.x, (int)gridDim.x);
  dense_graph<NB>(a, sh, sy, sweep_smem, [] {});
}

/* ---------------------------------------------------------------------- */
/* Grids.                                                                  */
/* ---------------------------------------------------------------------- */

#define TRACK_SOLO 1024               /* pairs of a CTA from which its warps work alone */

/* Working memory of a round over SWEEP_THREADS (row, word) pairs. */
struct TrackRound {
  unsigned newc[SWEEP_THREADS], newf[SWEEP_THREADS];   /* lanes that changed, lanes now full */
  unsigned count[SWEEP_SLOTS * 8];                     /* bits added per chunk, in eight parts */
  int warp_items[2][SWEEP_WARPS];
  int next;                                            /* the level's next block of 32 pairs */
  unsigned short queue[SWEEP_THREADS * 32];            /* pair << 5 | lane of the word */
};

struct TrackShared {
  int *list;                          /* [rows][dp] */
  unsigned *have, *full, *last;       /* per (row, word), a bit per lane: holds bits; is full; buffer of its words */
  unsigned *near;                     /* [dp][SWEEP_THREADS]: the neighbours' changed words of the round's pairs */
  TrackRound *round;
};

/* Level 0 of a group: every source's own bit.  Lanes that hold nothing are
 * never stored or read. */
__device__ void track_start(const gbx_sweep &a, const SweepShared &sh, const TrackShared &t, int src0, int nsrc, int nr)
{
  const int lw = a.word_log2, row_lanes = a.slots << (a.wc_log2 - 2);
  for(int c = threadIdx.x; c < (nr << lw); c += SWEEP_THREADS){
    const int row = sh.rank + (c >> lw) * sh.size, w = c & ((1 << lw) - 1);
    const int o = row - src0, l = o >> 8;
    unsigned bit = 0, full = 0;
    if(row < a.B && (unsigned)o < (unsigned)nsrc && (l >> 5) == w){
      unsigned x[8];
#pragma unroll
      for(int k = 0; k < 8; k++) x[k] = ((o >> 5) & 7) == k ? 1u << (o & 31) : 0u;
      st_lane(reinterpret_cast<char *>(a.buf) + ((size_t)row * row_lanes + l) * 32, x);
      bit = 1u << (l & 31);
      if(lane_bits(nsrc, l) == 1) full = bit;
    }
    t.have[c] = bit;
    t.full[c] = full;
    t.last[c] = 0;
    __stcg(a.changed + ((size_t)row << lw) + w, bit);
  }
}

/* One level over the CTA's (row, word) pairs (row rank + i * size, so that the
 * busy rows of a wavefront spread over the CTAs).  The pairs' lanes with a
 * changed neighbour are queued and shared out over the threads, whatever rows
 * they come from.  With few pairs the CTA goes round by round, a pair per
 * thread and the queue shared out evenly over all of them; with many (solo)
 * each warp takes blocks of 32 pairs by itself, with no barrier in between
 * (256 x 256: 5.26 ms against 5.6; 97 x 103: 0.34 against 0.32).  A neighbour
 * that did not change is not read: its words of the previous level may never
 * have been stored, or lie in the other buffer.  (Reading a row of zeros in
 * its place saves the predicates, but that row's sectors are then read by
 * everybody: a 97 x 103 grid took 0.49 to 0.55 ms that way.) */
template <int NB>
__device__ void track_level(const gbx_sweep &a, SweepShared &sh, const TrackShared &t, int level, int nsrc, int nr)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lw = a.word_log2, lL = a.wc_log2 - 2, dp = a.e.dp, d = a.e.d, n = a.e.n;
  const unsigned rb = (unsigned)(a.slots << lL) * 32u;   /* bytes of a row */
  const size_t half = a.slot_words * 8;                  /* bytes of a buffer */
  const unsigned *was = a.changed + (size_t)((level & 1) ^ 1) * ((size_t)n << lw);
  unsigned *now = a.changed + (size_t)(level & 1) * ((size_t)n << lw);
  const char *X = reinterpret_cast<const char *>(a.buf) + ((level & 1) ? 0 : half);
  char *Y = reinterpret_cast<char *>(a.buf) + ((level & 1) ? half : 0);
  TrackRound &tr = *t.round;
  const int pairs = nr << lw;
  const bool solo = pairs >= TRACK_SOLO;
  const unsigned short *queue = tr.queue + (solo ? warp * 1024 : 0);
  for(int x = tid; x < SWEEP_SLOTS * 8; x += SWEEP_THREADS) tr.count[x] = 0;
  __syncthreads();
  for(int round = 0;; round++){
    /* pair of this thread: first + tid */
    int first = round * SWEEP_THREADS;
    if(solo){
      int blk = 0;
      if(lane == 0) blk = atomicAdd(&tr.next, 1);
      blk = __shfl_sync(0xffffffffu, blk, 0);
      if(blk * 32 >= pairs) break;
      first = (blk - warp) * 32;
    }
    else if(first >= pairs) break;
    const int c = first + tid, w = c & ((1 << lw) - 1);
    const bool mine = c < pairs;
    unsigned act = 0;
    if(mine){
      const int *ids = t.list + (c >> lw) * dp;
      for(int j0 = 0; j0 < d; j0 += 8){
        unsigned x[8];
#pragma unroll
        for(int k = 0; k < 8; k++)
          x[k] = j0 + k < d ? __ldcg(was + ((size_t)(unsigned)ids[j0 + k] << lw) + w) : 0u;
#pragma unroll
        for(int k = 0; k < 8; k++)
          if(j0 + k < dp){
            t.near[(j0 + k) * SWEEP_THREADS + tid] = x[k];
            act |= x[k];
          }
      }
      act &= ~t.full[c];
    }
    tr.newc[tid] = tr.newf[tid] = 0;
    const int items = __popc(act);
    int at = items;
    for(int o = 1; o < 32; o <<= 1){
      const int x = __shfl_up_sync(0xffffffffu, at, o);
      if(lane >= o) at += x;
    }
    int total = __shfl_sync(0xffffffffu, at, 31);
    at += (solo ? warp * 1024 : 0) - items;
    if(!solo){
      if(lane == 31) tr.warp_items[round & 1][warp] = total;
      __syncthreads();
      total = 0;
      for(int k = 0; k < SWEEP_WARPS; k++){
        if(k == warp) at += total;
        total += tr.warp_items[round & 1][k];
      }
    }
    for(unsigned x = act; x; x &= x - 1) tr.queue[at++] = (unsigned short)(tid << 5 | (__ffs(x) - 1));
    if(solo) __syncwarp();
    else __syncthreads();
    for(int i = solo ? lane : tid; i < total; i += solo ? 32 : SWEEP_THREADS){
      const int code = queue[i], cl = code >> 5, b = code & 31, cc = first + cl;
      const int l = ((cc & ((1 << lw) - 1)) << 5) | b;   /* lane of the row */
      const int row = sh.rank + (cc >> lw) * sh.size;
      const int *ids = t.list + (cc >> lw) * dp;
      const unsigned *near = t.near + cl;
      const size_t own = (size_t)(unsigned)row * rb + (unsigned)l * 32u;
      const char *Xl = X + (unsigned)l * 32u;
      unsigned old[8], acc[8];
#pragma unroll
      for(int e = 0; e < 8; e++) old[e] = 0;
      if((t.have[cc] >> b) & 1u)
        ld_lane(old, reinterpret_cast<const char *>(a.buf) + (((t.last[cc] >> b) & 1u) ? half : 0) + own);
#pragma unroll
      for(int e = 0; e < 8; e++) acc[e] = 0;
      for(int j0 = 0; j0 < d; j0 += NB){
        unsigned v[NB][8];
#pragma unroll
        for(int k = 0; k < NB; k++){
#pragma unroll
          for(int e = 0; e < 8; e++) v[k][e] = 0;
          if(j0 + k < d && ((near[(j0 + k) * SWEEP_THREADS] >> b) & 1u))
            ld_lane(v[k], Xl + (size_t)(unsigned)ids[j0 + k] * rb);
        }
#pragma unroll
        for(int k = 0; k < NB; k += 2)
#pragma unroll
          for(int e = 0; e < 8; e++) acc[e] |= v[k][e] | v[k + 1][e];
      }
      unsigned diff[8];
#pragma unroll
      for(int e = 0; e < 8; e++){
        diff[e] = acc[e] & ~old[e];
        acc[e] |= old[e];
      }
      const unsigned added = popc_lane(diff);
      if(added){
        st_lane(Y + own, acc);
        atomicOr(&tr.newc[cl], 1u << b);
        const unsigned bits = (unsigned)lane_bits(nsrc, l);
        if(bits == 256u ? and_lane(acc) == ~0u : popc_lane(acc) == bits) atomicOr(&tr.newf[cl], 1u << b);
        atomicAdd(&tr.count[(l >> lL) * 8 + (tid & 7)], added);
      }
    }
    if(solo) __syncwarp();
    else __syncthreads();
    if(mine){
      const unsigned nc = tr.newc[tid];
      __stcg(now + ((size_t)(unsigned)(sh.rank + (c >> lw) * sh.size) << lw) + w, nc);
      t.have[c] |= nc;
      t.full[c] |= tr.newf[tid];
      t.last[c] = (t.last[c] & ~nc) | ((level & 1) ? nc : 0u);
    }
  }
  __syncthreads();
  if(warp == 0 && lane < a.slots){
    unsigned s = 0;
#pragma unroll
    for(int k = 0; k < 8; k++) s += tr.count[lane * 8 + k];
    sh.cnt[lane] = s;
  }
}

/* Warp 0: what comes next; level 0 (the sources themselves) starts a group. */
template <class Sync>
__device__ __forceinline__ void plan_track(const gbx_sweep &a, SweepShared &sh, Sync &sy)
{
  SweepPhase &p = sh.ph[0];
  int todo = TODO_LEVEL;
  unsigned long long bits;
  if(p.step > 0){
    if(!wait_step(a, sh, sy, 0, true, 1, bits)) todo = TODO_ABORT;
    else{
      const bool over = p.level > 0 && (p.total + bits == p.full || bits == 0 || p.level >= a.e.n);
      __syncwarp();
      if(over){
        if(sh.rank == 0) settle_step(a, p, sy, 0, p.step - 1, p.level, true);
        group_state(a, p, 0, p.group + 1);
        if(p.level < 0) todo = TODO_DONE;
      }
      else if(threadIdx.x == 0){
        p.total += bits;
        p.level++;
      }
    }
  }
  if(threadIdx.x == 0) sh.todo = todo;
  __syncwarp();
}

/* The whole evaluation by the CTAs of sh, as dense_graph. */
template <int NB, class Sync, class AfterPass>
__device__ bool track_graph(const gbx_sweep &a, SweepShared &sh, Sync &sy, unsigned char *smem, AfterPass after_pass)
{
  const int tid = threadIdx.x, dp = a.e.dp;
  const int nr = max(0, (a.e.n - sh.rank + sh.size - 1) / sh.size);
  TrackShared t;
  t.list = reinterpret_cast<int *>(smem);
  t.have = reinterpret_cast<unsigned *>(t.list + (size_t)a.rows * dp);
  t.full = t.have + ((size_t)a.rows << a.word_log2);
  t.last = t.full + ((size_t)a.rows << a.word_log2);
  t.near = t.last + ((size_t)a.rows << a.word_log2);
  t.round = reinterpret_cast<TrackRound *>(t.near + SWEEP_THREADS * dp);
  if(!pull_adjacency(a, sh, sy)) return false;
  expand_rows(a, sy, t.list, sh.rank, sh.size, nr, nullptr);
  if(tid < 32){
    group_state(a, sh.ph[0], 0, 0);
    if(tid == 0) sh.ph[0].t_loaded = sh.begin;
  }
  bool passed = false;
  for(;;){
    __syncthreads();
    if(tid < 32) plan_track(a, sh, sy);
    __syncthreads();
    const int todo = sh.todo, level = sh.ph[0].level, c0 = group_chunk(a, sh.ph[0].group, 0);
    if(todo == TODO_ABORT){
      if(tid == 0) *a.abort_flag = GBX_ERR_TIMEOUT;
      return false;
    }
    if(todo == TODO_DONE) break;
    if(level > 0 && !passed){
      passed = true;
      after_pass();
    }
    const int src0 = c0 * (64 << a.wc_log2), nsrc = min(a.slots * (64 << a.wc_log2), a.B - src0);
    if(level == 0) track_start(a, sh, t, src0, nsrc, nr);
    else track_level<NB>(a, sh, t, level, nsrc, nr);
    __syncthreads();
    if(tid == 0) t.round->next = 0;
    if(tid < 32) arrive_step(a, sh, sy, 0);
  }
  __syncthreads();
  return true;
}

/* The wide form has two CTAs per SM and six neighbours in flight, or eight where
 * that saves a turn: 190 x 190, d = 8 2069 -> 1884 us, 100 x 100 335 -> 318; at d
 * = 4 to 6 they cost 1 to 2 %.  The narrow one has three CTAs and four in
 * flight (79 registers; three with six in flight, and four CTAs, spilled: 256 x
 * 256, d = 6 6.0 and 5.9 ms against 5.3). */
template <int NB, int MIN_BLOCKS>
__global__ void __launch_bounds__(SWEEP_THREADS, MIN_BLOCKS) sweep_track_kernel(const gbx_sweep a)
{
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  __shared__ SweepShared sh;
  SweepSync &sy = launch_sync(a);
  sweep_begin(sh, (int)blockIdx.x, (int)gridDim.x);
  track_graph<NB>(a, sh, sy, sweep_smem, [] {});
}

/* ---------------------------------------------------------------------- */
/* Many graphs.                                                            */
/* ---------------------------------------------------------------------- */

/* Many graphs of uneven size by teams of CTAs.  A graph's team is a 2^k-th of
 * the grid: the large graphs are taken first by the large teams, and a team
 * that finds its size's queue empty splits in two, so that the small graphs
 * fill in behind.  Within a team a graph runs as in the kernels above, with
 * its barriers in the team's own words.  Against one grid-wide queue of tiles
 * there is no hand-off per tile, the neighbour lists stay in shared memory
 * over the levels, and one team's copy of its adjacency from host memory runs
 * while others compute. */
typedef SyncT<1, SWEEP_SLOTS> TeamSync;

struct TeamNode {
  TeamSync sync[2];                    /* by graph, alternating */
  unsigned long long box[2][16];       /* graph `seq` of the team: (seq + 1) << 32 | graph + 1, or 0: none left */
};

__global__ void __launch_bounds__(SWEEP_THREADS, 2) team_kernel(const gbx_team t)
{
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  __shared__ SweepShared sh;
  __shared__ gbx_sweep a;
  __shared__ int sh_graph;
  const int tid = threadIdx.x, G = (int)gridDim.x, b = (int)blockIdx.x;
  /* The first access of the GPU to a page of host memory takes it far longer
   * than to read the page, and a team that comes to a graph of new pages waits
   * for each in turn.  So all pages are asked for at the start, a word each, in
   * the graphs' order, by prefetches that nobody waits for.  256 graphs in
   * arrays just allocated, medians of two processes: 8.1 and 14.1 -> 6.0 and
   * 6.1 ms (pages in order, as of a large mapping, cost little either way: 3.0);
   * a word every 16 KB 6.3 and 7.1; known arrays 2.76 both ways. */
  if(t.adj)
    for(int q = b; q < t.queue[GBX_TEAM_SPLITS]; q += G){
      const int g = t.order ? t.order[q] : q;
      const int *src = reinterpret_cast<const int *>(__ldcg(t.adj + g));
      const long long ints = (long long)t.graphs[g].B * t.graphs[g].e.d;
      for(long long i = (long long)tid * t.page_ints; i < ints + t.page_ints && ints > 0; i += (long long)SWEEP_THREADS * t.page_ints)
        asm volatile("prefetch.global.L2 [%0];" :: "l"(src + min(i, ints - 1)));
    }
  for(int k = t.first_split; k <= t.last_split; k++){
    const int queued = t.queue[k + 1] - t.queue[k];
    if(queued <= 0) continue;
    /* team i of 2^k: CTAs [i * G >> k, (i + 1) * G >> k) */
    const int i = (int)((((long long)(b + 1) << k) - 1) / G);
    const int lo = (int)(((long long)i * G) >> k), hi = (int)(((long long)(i + 1) * G) >> k);
    TeamNode &node = reinterpret_cast<TeamNode *>(t.nodes)[(1 << k) - (1 << t.first_split) + i];
    /* CTA `lo` takes the next graph off the queue and posts it */
    auto post = [&](int seq) {
      const unsigned at = atomicAdd(t.next + k, 1u);
      const int from = t.queue[k] + (int)at;
      const unsigned g = at < (unsigned)queued ? (unsigned)(t.order ? t.order[from] : from) + 1u : 0u;
      __threadfence();
      atomicExch(&node.box[seq & 1][0], (unsigned long long)(seq + 1) << 32 | g);
    };
    if(b == lo && tid == 0) post(0);
    for(int seq = 0;; seq++){
      if(tid == 0){
        unsigned long long seen = 0;
        const bool ok = wait_for(&node.box[seq & 1][0], (unsigned long long)(seq + 1) << 32, seen, t.limit_ns);
        if(!ok) *t.abort_flag = GBX_ERR_TIMEOUT;
        sh_graph = ok ? (int)(unsigned)seen - 1 : -2;
      }
      __syncthreads();
      const int g = sh_graph;
      __syncthreads();                                   /* read before it is written again */
      if(g == -2) return;
      if(g < 0) break;
      {
        const unsigned *src = reinterpret_cast<const unsigned *>(t.graphs + g);
        unsigned *dst = reinterpret_cast<unsigned *>(&a);
        for(int x = tid; x < (int)(sizeof(gbx_sweep) / 4); x += SWEEP_THREADS) dst[x] = __ldg(src + x);
      }
      __syncthreads();
      if(tid == 0){
        a.limit_ns = t.limit_ns;
        if(t.adj) a.e.adj = reinterpret_cast<const int *>(__ldcg(t.adj + g));
        unsigned char *at = t.arena + (size_t)i * (t.arena_bytes >> k);   /* inside the parent's part: the size divides evenly */
        a.buf = reinterpret_cast<unsigned long long *>(at);
        a.start = a.buf + ((a.base & 1) ? a.slot_words : 0);
        a.start_stride = 2 * a.slot_words;
        a.changed = reinterpret_cast<unsigned *>(at + 16 * a.slot_words);
        a.rows = (a.e.n + (hi - lo) - 1) / (hi - lo);
      }
      /* every CTA applies all of the graph's changes itself, the same values
       * to the same places, and so needs no barrier of the team before it
       * reads them */
      for(int x = tid; x < a.nwrites; x += SWEEP_THREADS) *a.writes[x].at = a.writes[x].value;
      sweep_begin(sh, b - lo, hi - lo);
      TeamSync &sy = node.sync[seq & 1];
      auto clear = [&] {
        /* every CTA has begun this graph, so the last one's counters and box are free */
        if(b != lo) return;
        unsigned *other = reinterpret_cast<unsigned *>(&node.sync[(seq + 1) & 1]);
        for(int x = tid; x < (int)(sizeof(TeamSync) / 4); x += SWEEP_THREADS) other[x] = 0;
      };
      const bool ok = a.track ? track_graph<6>(a, sh, sy, sweep_smem, clear)
                              : dense_graph<8>(a, sh, sy, sweep_smem, clear);
      if(!ok) return;
      /* taken only now: a graph taken ahead would wait for this one, however long, while another team is free */
      if(b == lo && tid == 0) post(seq + 1);
    }
  }
}

}  // namespace

extern "C" {

/* Resident CTAs per SM of `entry` with that much shared memory: an answer, not
 * an error that the next launch would take for its own. */
static int resident(const void *entry, size_t smem, int *per_sm)
{
  cudaError_t e = cudaFuncSetAttribute(entry, cudaFuncAttributeMaxDynamicSharedMemorySize, GBX_SWEEP_SMEM_MAX);
  if(e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, entry, SWEEP_THREADS, smem);
  if(e != cudaSuccess) cudaGetLastError();
  return (int)e;
}

size_t gbx_sweep_sync_bytes(void) { return 2 * sizeof(SweepSync); }

size_t gbx_sweep_smem(const gbx_sweep *a)
{
  const size_t rows = (size_t)a->rows, lists = rows * (size_t)a->e.dp * 4;
  if(a->track)
    return lists + 3 * (rows << a->word_log2) * 4 + SWEEP_THREADS * (size_t)a->e.dp * 4 + sizeof(TrackRound);
  return lists + (size_t)a->scratch_rows * ((size_t)a->scratch_bits / 8 + 4 * (size_t)a->queue) + 4 * (size_t)a->base * (size_t)a->nchunks +
         (((size_t)a->phases * a->slots * rows) << (a->wc_log2 - 2));
}

/* The dense kernel's narrow form keeps four CTAs of 64 registers per SM, the
 * wide one two of 128 with eight neighbours in flight per lane. */
static const void *sweep_entry(const gbx_sweep *a)
{
  if(a->track && !a->wide) return (const void *)sweep_track_kernel<4, 3>;
  if(a->track)
    return (a->e.d + 7) / 8 < (a->e.d + 5) / 6 ? (const void *)sweep_track_kernel<8, 2>
                                               : (const void *)sweep_track_kernel<6, 2>;
  return a->wide ? (const void *)sweep_dense_kernel<8, 2> : (const void *)sweep_dense_kernel<4, 4>;
}

int gbx_sweep_blocks(const gbx_sweep *a, int *per_sm)
{
  *per_sm = 0;
  const size_t smem = gbx_sweep_smem(a);
  if(smem > GBX_SWEEP_SMEM_MAX) return (int)cudaErrorInvalidValue;
  return resident(sweep_entry(a), smem, per_sm);
}

static int launch_all(const void *entry, void *arg, int blocks, size_t smem, cudaStream_t stream)
{
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks, 1, 1);
  cfg.blockDim = dim3(SWEEP_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void *args[1] = { arg };
  return (int)cudaLaunchKernelExC(&cfg, entry, args);
}

int gbx_sweep_launch(const gbx_sweep *a, int blocks, void *stream)
{
  gbx_sweep arg = *a;
  return launch_all(sweep_entry(a), &arg, blocks, gbx_sweep_smem(a), (cudaStream_t)stream);
}

size_t gbx_team_node_bytes(void) { return sizeof(TeamNode); }

int gbx_team_blocks(size_t smem, int *per_sm)
{
  *per_sm = 0;
  if(smem > GBX_SWEEP_SMEM_MAX) return (int)cudaErrorInvalidValue;
  return resident((const void *)team_kernel, smem, per_sm);
}

int gbx_team_launch(const gbx_team *t, int blocks, size_t smem, void *stream)
{
  gbx_team arg = *t;
  return launch_all((const void *)team_kernel, &arg, blocks, smem, (cudaStream_t)stream);
}

}  /* extern "C" */
