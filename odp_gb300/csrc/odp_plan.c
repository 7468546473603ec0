/*
 * odp_plan.c -- builds and runs execution plans (odp_plan.h) on the CUDA
 * layer.  This is the host runtime of the library: it chooses the kernels of a
 * plan, sizes column chunks so the live bitsets stay in L2, orders jobs and lays
 * out device memory.  A call is one kernel that reads the callers' arrays from
 * host memory and leaves its records in pinned memory (small, lockstep and team
 * plans), or a replayed CUDA graph of pull, expand, engine and one copy back,
 * with no host round trip per BFS level (the reference does one per level,
 * aspl_cuda.cu:62-82).
 *
 * Result semantics follow the reference exactly (aspl_cuda.cu:84-85,
 * 121-125, 256-260): the ordered sum is accumulated in 64-bit integers,
 * ASPL = sum / ((double)n - 1) / n computed as sum / (((double)n-1)*n), the
 * returned sum is (long)(sum / 2.0), the diameter is the largest level at
 * which a chunk became complete, and a graph with unreachable pairs returns
 * INT_MAX / LONG_MAX / DBL_MAX.
 */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <limits.h>
#include <float.h>
#include <math.h>
#include <pthread.h>
#include <unistd.h>
#include <time.h>
#include "odp_plan.h"
#include "odp_gb300.h"

#define ALIGN_UP(x, a) ((((x) + (a) - 1) / (a)) * (a))

static int g_device_ready = 0, g_sm_count = 0;

int odp_device_ready(void)
{
  if(g_device_ready) return 0;
  int e = gbx_device_init(&g_sm_count);
  if(e) return e;
  g_device_ready = 1;
  return 0;
}

static int env_int(const char *name, int fallback)
{
  const char *v = getenv(name);
  return (v && *v) ? atoi(v) : fallback;
}

void odp_tuning_defaults(odp_tuning *t, int batch)
{
  t->wc_log2 = env_int("ODP_GB300_WC_LOG2", 0);
  t->slots = env_int("ODP_GB300_SLOTS", 0);
  t->tile_rows = env_int("ODP_GB300_TILE_ROWS", 0);
  t->l2_budget_mb = env_int("ODP_GB300_L2_MB", 80);
  t->local_kb = env_int("ODP_GB300_LOCAL_KB", batch ? 2048 : 96);
  t->use_graph = env_int("ODP_GB300_GRAPH", 1);
  t->blocks = env_int("ODP_GB300_BLOCKS", 0);
  t->activity = env_int("ODP_GB300_ACTIVITY", -2);
  t->local_kb_explicit = getenv("ODP_GB300_LOCAL_KB") != NULL;
  t->reorder = env_int("ODP_GB300_REORDER", 1);
  t->direct = env_int("ODP_GB300_DIRECT", 1);
  t->small_n = env_int("ODP_GB300_SMALL_N", 8192);
  t->small_cluster = env_int("ODP_GB300_SMALL_CLUSTER", 0);
  t->small_part = env_int("ODP_GB300_SMALL_PART", -1);
  t->sweep = env_int("ODP_GB300_SWEEP", 1);
}

/* Shared memory per CTA of the small kernel when `cluster` CTAs share a job:
 * both bitset buffers (whole, or with `part` the CTA's 1/cluster of the
 * rows) and the row table of 1/cluster of the rows. */
static size_t small_bytes(int n, int dp, int wl, int cluster, int part)
{
  const size_t rows = (size_t)(n + cluster - 1) / (size_t)cluster;
  return 2 * (part ? rows : (size_t)n) * ((size_t)8 << wl) + rows * (size_t)dp * 4;
}

/* Chunk width (log2 words) for a graph whose whole level runs in shared
 * memory on a cluster of `cluster` CTAs: the widest of at most 16 words, and
 * at most the graph's own width, that fits; 0 if none does. */
static int small_wc_log2(int n, int dp, int full_l2, int cluster, int part)
{
  for(int wl = full_l2 < 4 ? full_l2 : 4; wl >= 1; wl--)
    if(small_bytes(n, dp, wl, cluster, part) <= GBX_SMALL_SMEM_MAX) return wl;
  return 0;
}

/* Threads per CTA for a CTA's rows: one lane per 16 bytes of a row (at most
 * a warp per row), rounded up to whole warps, 64 to 512. */
static int small_threads_for(int n, int wl, int cluster)
{
  const int rows = (n + cluster - 1) / cluster;
  const int lanes = (1 << wl) / 2 < 32 ? (1 << wl) / 2 : 32;
  long long t = ((long long)rows * lanes + 31) / 32 * 32;
  if(t < 64) t = 64;
  if(t > 512) t = 512;
  return (int)t;
}

static int ilog2_ceil(long long x)
{
  int l = 0;
  while((1LL << l) < x) l++;
  return l;
}

/* Rows one CTA pass covers for a chunk of 2^wl words (see RowShape in the .cu). */
static int rows_per_pass(int wl)
{
  int vpr = (1 << wl) / 2;
  int g = vpr < 32 ? vpr : 32;
  return 8 * (32 / g);
}

static int validate_shape(const odp_shape *sh)
{
  int n = sh->grid ? sh->width * sh->height : sh->nodes;
  if(n <= 0 || sh->degree < 0 || sh->degree > GBX_MAX_DEGREE || sh->symmetries <= 0) return ODPX_ERR_INVALID;
  if(n % sh->symmetries != 0) return ODPX_ERR_INVALID;
  if(sh->grid && sh->symmetries != 1){
    int s = sh->symmetries, w = sh->width, h = sh->height;
    if(s != 2 && s != 4) return ODPX_ERR_INVALID;
    if(s == 2 && w % 2 != 0) return ODPX_ERR_INVALID;
    if(s == 4 && (w % 2 != 0 || h % 2 != 0 || w != h)) return ODPX_ERR_INVALID;
  }
  return 0;
}

/* ODP_ROTATE (reference utils.c:67-88) on the host, for row tables. */
static int rotate_host(int v, int width, int height, int s, int deg)
{
  int x = v / height, y = v % height;
  if(s == 2) return (width - x - 1) * height + (height - y - 1);
  if(deg == 90)  return y * height + (height - x - 1);
  if(deg == 180) return (height - x - 1) * height + (height - y - 1);
  return (height - y - 1) * height + x;
}

/* Vertex -> row table of a rotation-symmetric grid (ODP_Create_itable, utils.c:2103-2124). */
static void fill_itable(int width, int height, int s, int *itable)
{
  int base = (width * height) / s;
  if(s == 2){
    for(int i = 0; i < base; i++){
      itable[i] = i;
      itable[rotate_host(i, width, height, s, 180)] = i + base;
    }
  }
  else{
    int bh = height / 2;
    for(int i = 0; i < base; i++){
      int v = (i / bh) * height + (i % bh);
      itable[v] = i;
      itable[rotate_host(v, width, height, s, 90)]  = i + base;
      itable[rotate_host(v, width, height, s, 180)] = i + base * 2;
      itable[rotate_host(v, width, height, s, 270)] = i + base * 3;
    }
  }
}

/* Per-vertex degrees over all n vertices, as the reference's Init variants
 * expand them (aspl_cuda.cu:164-179 tiling, :200-217 rotation).  For s = 4
 * grids the base vertex of local index i is placed with the inverse of the
 * local index map, as the row table does. */
static void fill_degrees(const odp_shape *sh, int n, int *out)
{
  int s = sh->symmetries, base = n / s;
  const int *nd = sh->num_degrees;
  if(!sh->grid || s == 1){
    for(int t = 0; t < s; t++)
      for(int j = 0; j < base; j++) out[t * base + j] = nd[j];
    return;
  }
  int w = sh->width, h = sh->height;
  if(s == 2){
    for(int i = 0; i < base; i++){
      out[i] = nd[i];
      out[rotate_host(i, w, h, 2, 180)] = nd[i];
    }
  }
  else{
    for(int i = 0; i < base; i++){
      int v = (i / (h / 2)) * h + i % (h / 2);
      out[v] = nd[i];
      out[rotate_host(v, w, h, 4, 90)]  = nd[i];
      out[rotate_host(v, w, h, 4, 180)] = nd[i];
      out[rotate_host(v, w, h, 4, 270)] = nd[i];
    }
  }
}

/* Cells of a bw x bh rectangle along the Hilbert curve (D. Hilbert, 1891) of
 * the square of side 2^order around it: quadrant by quadrant, the first and
 * the last turned so that the curve stays connected; squares outside the
 * rectangle are passed over.  A square is its origin and the directions of
 * its two axes. */
typedef struct { int bw, bh, count, *x, *y; } curve_walk;

static void walk_curve(curve_walk *c, int order, int ox, int oy, int ux, int uy, int vx, int vy)
{
  const int far = (1 << order) - 1, ex = ox + far * (ux + vx), ey = oy + far * (uy + vy);
  if((ox < ex ? ox : ex) >= c->bw || (oy < ey ? oy : ey) >= c->bh) return;
  if(order == 0){
    c->x[c->count] = ox;
    c->y[c->count++] = oy;
    return;
  }
  const int side = 1 << (order - 1), last = side - 1;
  walk_curve(c, order - 1, ox, oy, vx, vy, ux, uy);
  walk_curve(c, order - 1, ox + side * vx, oy + side * vy, ux, uy, vx, vy);
  walk_curve(c, order - 1, ox + side * (ux + vx), oy + side * (uy + vy), ux, uy, vx, vy);
  walk_curve(c, order - 1, ox + side * ux + last * (ux + vx), oy + side * uy + last * (uy + vy), -vx, -vy, -ux, -uy);
}

/* Rows of a grid graph in the order of a Hilbert curve through its base
 * region (the whole grid, the left half for s = 2, the lower-left quadrant
 * for s = 4): vertex -> row, and row -> vertex.  The base rows come first, so
 * the sources are rows [0, B) in curve order; the rotations of base row r
 * are rows r + t*B, as in fill_itable. */
static int fill_curve_rows(const odp_plan_graph *g, int *itable, int *row_vertex)
{
  const int bw = g->s == 1 ? g->width : g->width / 2;
  const int bh = g->s == 4 ? g->height / 2 : g->height;
  int *xy = malloc(sizeof(int) * 2 * (size_t)g->B);
  if(!xy) return ODPX_ERR_MEMORY;
  curve_walk c = { bw, bh, 0, xy, xy + g->B };
  walk_curve(&c, ilog2_ceil(bw > bh ? bw : bh), 0, 0, 1, 0, 0, 1);
  for(int k = 0; k < g->B; k++){
    const int base = c.x[k] * g->height + c.y[k];
    for(int r = 0; r < g->s; r++){
      const int v = r == 0 ? base : rotate_host(base, g->width, g->height, g->s, g->s == 2 ? 180 : 90 * r);
      itable[v] = k + r * g->B;
      row_vertex[k + r * g->B] = v;
    }
  }
  free(xy);
  return 0;
}

/* Source ordinals of a grid graph, ordered by square tiles of the base
 * region (the whole grid, the left half for s = 2, the lower-left quadrant
 * for s = 4), so that each column chunk's sources are close together and its
 * BFS wavefront stays narrow.  Indexed by row; rows that are not sources get
 * -1.  Any assignment of sources to bits gives the same results: the sum and
 * the diameter do not depend on which sources share a chunk. */
static void fill_srcpos(const odp_plan_graph *g, int *srcpos)
{
  int bw = g->s == 1 ? g->width : g->width / 2;
  int bh = g->s == 4 ? g->height / 2 : g->height;
  int cap = 64 << g->wc_log2, ts = 1;
  while((ts + 1) * (ts + 1) <= cap) ts++;
  for(int r = 0; r < g->n; r++) srcpos[r] = -1;
  int ord = 0;
  for(int tx = 0; tx < bw; tx += ts)
    for(int ty = 0; ty < bh; ty += ts)
      for(int x = tx; x < tx + ts && x < bw; x++)
        for(int y = ty; y < ty + ts && y < bh; y++){
          /* rows of base vertices: v itself for s = 1, 2 (x < w/2); the local
           * index x * (h/2) + y for s = 4 */
          int row = (g->s == 4) ? x * bh + y : x * g->height + y;
          srcpos[row] = ord++;
        }
}

/* Per-bucket tuning table (ODPX_Set_tuning_table), filled by the autotuner:
 * a graph whose (ceil log2 n, degree class, grid) matches an entry takes its
 * chunk width, tile traffic and local-job threshold. */
#define TUNE_MAX 256
static ODPX_Tune_entry g_table[TUNE_MAX];
static int g_table_len = 0;

int ODPX_Set_tuning_table(const ODPX_Tune_entry *entries, int count)
{
  if(count < 0 || count > TUNE_MAX || (count > 0 && !entries)) return ODPX_ERR_INVALID;
  if(count) memcpy(g_table, entries, sizeof(ODPX_Tune_entry) * (size_t)count);
  g_table_len = count;
  return 0;
}

int ODPX_Degree_class(int degree) { return degree <= 8 ? 0 : degree <= 16 ? 1 : degree <= 32 ? 2 : 3; }

static const ODPX_Tune_entry *table_lookup(int n, int degree, int grid)
{
  int nl = ilog2_ceil(n);
  int dc = ODPX_Degree_class(degree);
  for(int i = 0; i < g_table_len; i++)
    if(g_table[i].n_log2 == nl && g_table[i].degree_class == dc && g_table[i].grid == grid) return &g_table[i];
  return NULL;
}

typedef struct { int job; double work; } job_order;

static int cmp_work_desc(const void *a, const void *b)
{
  double wa = ((const job_order *)a)->work, wb = ((const job_order *)b)->work;
  if(wa > wb) return -1;
  if(wa < wb) return 1;
  return ((const job_order *)a)->job - ((const job_order *)b)->job;
}

/* Initial engine state: the first nslots jobs loaded into the slots, the
 * job queue at nslots, everything else zero. */
static void fill_state_init(odp_plan *p)
{
  memset(p->h_state_init, 0, p->state_bytes);
  gbx_slot *sl = (gbx_slot *)p->h_state_init;
  for(int k = 0; k < p->nslots; k++){
    const gbx_job *j = &p->h_jobs[k];
    sl[k].ticket = (unsigned long long)j->ntiles << 32;
    sl[k].job = k;
    sl[k].desc = *j;
    sl[k].level = 1;
    sl[k].prev = (unsigned long long)j->nsrc;
    sl[k].sum = ((long long)j->n * j->nsrc - j->nsrc) * j->sym;
    sl[k].buf0 = p->d_slotbuf + (size_t)k * 2 * p->slot_words;
    sl[k].buf1 = sl[k].buf0 + p->slot_words;
    sl[k].mask0 = p->d_slotmask + (size_t)k * 2 * p->slot_rows;
    sl[k].mask1 = sl[k].mask0 + p->slot_rows;
  }
  gbx_ctrl *ctrl = (gbx_ctrl *)(p->h_state_init + p->out_off);
  ctrl->next_job = (unsigned)p->nslots;
}

/* Whether a graph's jobs track changes (gather only words that changed at
 * the previous level).  It is exact for every graph.  Without it, lanes whose
 * words are saturated already skip their gathers; with it, every row stages
 * its neighbours' change masks, which pays where levels are many and each
 * changes few words: single grids.  Plans whose every job tracks changes run
 * the engine built for those passes alone, with two vectors per lane.
 * Measured on GB300, on against off (ms): 100 x 100, d = 4: 1.27 / 1.10;
 * 128 x 128, d = 6: 1.63 / 1.42, but d = 4: 1.87 / 2.04; 160 x 160: 3.62 /
 * 3.96; 192 x 192: 6.26 / 9.15; 224 x 224: 12.9 / 17.4; 256 x 256, s = 4:
 * 6.86 / 7.04; 256 x 256, d = 8, s = 2: 9.76 / 13.3.  In batches the larger
 * staging area of every job cost more than it saved (the 512-graph batch:
 * 9.0 against 7.15 ms tuned).  So by default it is on for a single grid of
 * at least 20000 vertices. */
static int tracks_changes(const odp_tuning *t, int count, int grid, int n, int s)
{
  (void)s;
  if(t->activity == -2) return count == 1 && grid && n >= 20000;
  return t->activity == -1 ? grid : t->activity;
}

static int shape_n(const odp_shape *sh) { return sh->grid ? sh->width * sh->height : sh->nodes; }
static int shape_dp(const odp_shape *sh) { return ALIGN_UP(sh->degree > 0 ? sh->degree : 1, 4); }
static int shape_words(const odp_shape *sh) { return (shape_n(sh) / sh->symmetries + 63) / 64; }

/* Jobs of the small kernel with these chunk widths. */
static long long small_job_count(const odp_shape *shapes, int count, const int *wl)
{
  long long jobs = 0;
  for(int i = 0; i < count; i++) jobs += (shape_words(&shapes[i]) + (1 << wl[i]) - 1) >> wl[i];
  return jobs;
}

/* Shared memory and threads of a CTA for chunks of 2^wl[i] words. */
static void small_shape(const odp_shape *shapes, int count, const int *wl, int c, int part, size_t *smem, int *threads)
{
  *smem = 0;
  *threads = 64;
  for(int i = 0; i < count; i++){
    const size_t b = small_bytes(shape_n(&shapes[i]), shape_dp(&shapes[i]), wl[i], c, part);
    const int th = small_threads_for(shape_n(&shapes[i]), wl[i], c);
    if(b > *smem) *smem = b;
    if(th > *threads) *threads = th;
  }
}

/* Whether all jobs run at once: by the SMs and, for a single graph, by the
 * clusters that the GPU's parts really hold (with a CTA per SM, 36 of 4 and 15
 * of 8: 64 x 64 in 16 clusters of 8 took two turns, 184 us against 115). */
static int small_at_once(const odp_shape *shapes, int count, const int *wl, long long jobs, int c, int part, int sms)
{
  size_t smem;
  int threads, active = 0;
  if(jobs * c > sms) return 0;
  if(count > 1) return 1;
  small_shape(shapes, count, wl, c, part, &smem, &threads);
  return smem <= GBX_SMALL_SMEM_MAX && gbx_small_clusters(c, threads, smem, &active) == 0 && active >= jobs;
}

/* Whether a plan is of the small class, for the small-graph kernel, and its
 * shape there: the chunk width of each graph (wl), the CTAs per job (one
 * thread-block cluster), the threads and shared memory per CTA.  Every graph
 * must have at most small_n vertices and no schedule setting or change tracking
 * may ask for the engine.  The cluster is the largest power of two up to 8 at
 * which every graph fits and all jobs run at once; for each graph the widest
 * chunk that fits is halved, widest first, while they still do (the n = 1024, d
 * = 8 graph: 8 jobs of 2 words on clusters of 8 CTAs, 64 SMs).  Plans of more
 * than one wave are for the other kernels: every job reads its graph's adjacency
 * from host memory, and 32 jobs on clusters of 8 (n = 4096, d = 24 and 32) take
 * 147 and 216 us against 38 and 41 in lockstep.  The replicated layout (every CTA
 * holds the whole level) is tried first.  Plans of grid graphs whose whole level
 * does not fit in one CTA take the partitioned layout (each CTA holds its rows,
 * neighbour rows are read from the CTA that owns them through distributed shared
 * memory), which fits graphs up to `cluster` times larger.  Its gathers run at
 * about one 16-byte request per clock per SM, so it pays only where levels are
 * many and light: grids of 72 x 72 and 80 x 80, d = 4, 207 and 249 us against 276
 * and 298 in lockstep, but general graphs lose (n = 8192, d = 8: 260 against 63; n
 * = 4096, d = 24: 183 against 38).  A cluster size forced by
 * ODP_GB300_SMALL_CLUSTER is used if the graphs fit at it (else halved),
 * whatever the SM count; ODP_GB300_SMALL_PART=0 or 1 forces the layout. */
static int choose_small(const odp_shape *shapes, int count, const odp_tuning *t, int sms, int *wl,
                        int *cluster_out, int *threads_out, size_t *smem_out, int *part_out)
{
  if(count <= 0 || t->small_n <= 0 || t->wc_log2 > 0 || t->slots > 0 || t->tile_rows > 0 || t->local_kb_explicit)
    return 0;
  for(int i = 0; i < count; i++){
    const int n = shape_n(&shapes[i]);
    const ODPX_Tune_entry *te = table_lookup(n, shapes[i].degree, shapes[i].grid);
    if(n > t->small_n || (te && te->wc_log2 > 0) || tracks_changes(t, count, shapes[i].grid, n, shapes[i].symmetries))
      return 0;
  }
  if(gbx_small_prepare()) return 0;
  const int want = t->small_cluster > 0 && t->small_cluster <= GBX_SMALL_CLUSTER_MAX ? t->small_cluster : 0;
  int all_grids = 1;
  for(int i = 0; i < count; i++) all_grids &= shapes[i].grid != 0;
  /* A single grid of 1800 vertices or more first tries clusters of 4 with chunks
   * of two words (clusters of 8 have half the rows a CTA, but chunks twice as
   * wide, and send every changed word to twice the peers), partitioned up to
   * degree 4, and then clusters of 8, partitioned; but a grid more than twice as
   * high as wide, whose rows of a CTA (a few columns) border on every other
   * CTA's, replicated first.  Measured on GB300, us, clusters of 8 against 4
   * replicated and 4 and 8 partitioned: 50 x 50, d = 4 125 / 90 / 85 / 86, d = 10
   * 81 / 77 / 84 / 96; 64 x 64, d = 4 268 / 124 / 115 / 184, d = 8 233 / 131 / 133
   * / 202; 200 x 12, d = 4 264 / 177 / 179 / 212;
   * 20 x 195, d = 6 262 partitioned against 195; 110 x 45, d = 4 448 / 290 / 213
   * / 202 (2 CTAs, replicated: 245); but 40 x 40, d = 8 49 / 54 / 55 / 53. */
  const int one_grid = count == 1 && all_grids && !want && t->small_part < 0 && shape_n(shapes) >= 1800;
  const int tall = one_grid && shapes->height > 2 * shapes->width;
  for(int turn = one_grid ? 0 : 1; turn < 3; turn++){
    const int part = turn == 0 ? shapes->degree <= 4 && !tall : one_grid ? (turn == 1) != tall : turn - 1;
    if(turn == 0 && 2 * shape_words(shapes) > sms) continue;
    if(!one_grid && ((part && t->small_part == 0) || (!part && t->small_part > 0))) continue;
    for(int c = want ? want : turn == 0 ? 4 : GBX_SMALL_CLUSTER_MAX; c >= (turn == 0 ? 4 : 1); c >>= 1){
      if(part && c == 1) continue;                 /* one CTA: the replicated layout */
      if(part && t->small_part < 0 && !all_grids) continue;
      int ok = 1;
      for(int i = 0; i < count && ok; i++){
        const int W = shape_words(&shapes[i]);
        wl[i] = small_wc_log2(shape_n(&shapes[i]), shape_dp(&shapes[i]), ilog2_ceil(W < 2 ? 2 : W), c, part);
        if(!wl[i]) ok = 0;
      }
      if(!ok) continue;
      long long jobs = small_job_count(shapes, count, wl);
      if(!want && !small_at_once(shapes, count, wl, jobs, c, part, sms)) continue;
      for(;;){                                   /* narrower chunks while the jobs fit on the SMs */
        int k = -1;
        for(int i = 0; i < count; i++)
          if(wl[i] > 1 && (k < 0 || wl[i] > wl[k])) k = i;
        if(k < 0) break;
        wl[k]--;
        const long long more = small_job_count(shapes, count, wl);
        if(want ? more * c > sms : !small_at_once(shapes, count, wl, more, c, part, sms)){ wl[k]++; break; }
        jobs = more;
      }
      size_t smem;
      int threads, active = 0;
      small_shape(shapes, count, wl, c, part, &smem, &threads);
      if(smem <= GBX_SMALL_SMEM_MAX && gbx_small_clusters(c, threads, smem, &active) == 0 && active > 0){
        *cluster_out = c;
        *threads_out = threads;
        *smem_out = smem;
        *part_out = part;
        return 1;
      }
    }
  }
  return 0;
}

/* Whether a small plan of one graph, in chunks of 2^wl words, is faster on the
 * lockstep kernel (unless its cluster or layout is forced).  Every job of the
 * small kernel reads the whole adjacency from host memory, so for general
 * graphs the line lies at 450 KB read in all; measured on GB300 through
 * ODPX_Batch_run, small kernel against lockstep (us): n = 512, d = 8 (66 KB) 29 /
 * 33; n = 1182, d = 10, s = 2 (118 KB) 33 / 36; n = 1024, d = 8 (262 KB) 30 / 33; n =
 * 1024, d = 24 (786 KB) 37 / 29; n = 2048, d = 8 (1 MB) 43 / 36; n = 4096, d = 8 (4
 * MB) 65 / 41.  Grids are bound by their levels: replicated 40 x 40, d = 8 62 / 135,
 * 64 x 64, d = 8 157 / 216; partitioned 50 x 50, d = 4 90 / 186, 64 x 64 119 / 233.
 * Partitioned, a level's time grows with n and d in the small kernel and hardly
 * in lockstep, less so the longer the grid, where fewer rows change: 75 x 75, d =
 * 4 217 / 286, d = 8 268 / 270, d = 10 335 / 297; 80 x 80, d = 4 249 / 298; 90 x 90
 * 341 to 533 / 371; 171 x 33, d = 4 295 / 423, d = 8 334 / 374, d = 10 405 / 415; 190 x
 * 36, d = 4 366 / 477, d = 8 418 / 419.  Grids more than twice as high as wide,
 * whose CTAs border on all others: 33 x 171, d = 4 384 / 430, d = 8 506 / 374; 25 x
 * 200, d = 6 560 / 422.  (General graphs with the levels
 * of a grid lose a little: 64 x 64 as one 192 / 208.) */
static int small_yields(const odp_shape *sh, const odp_tuning *t, int part, int wl)
{
  if(t->small_cluster > 0 || t->small_part >= 0) return 0;
  if(sh->grid)
    return part && 2.0 * pow(shape_n(sh), 1.5) * (sh->degree + 2) >
                   (sh->height > 2 * sh->width ? 25e3 : 46e3) * (sh->width + sh->height);
  const double jobs = (shape_words(sh) + (1 << wl) - 1) >> wl;
  return jobs * 4.0 * (shape_n(sh) / sh->symmetries) * sh->degree > 450e3;
}

/* How many levels of a general graph come from its neighbour lists (at least
 * `base`, 1 or 2; `chunks` bounds the counters) and the scratch that takes.  A
 * gathered level reads d + 1 lanes per row and 256 sources.  A level from the
 * lists marks up to d^k vertices a row (symmetric lists reach fewer) and queued
 * all before them, at about 0.6 of a lane each, and saves a barrier; at least
 * three warps of a CTA need their scratch rows.  Measured on GB300, two levels
 * against more (us): n = 65536, d = 16 (3 levels) 1656 / 1350; d = 6 (4) 2019 /
 * 1547, 5 levels 1818; d = 20 (3) 1616 / 1548; d = 24 1796, 3 levels 2077; n =
 * 30000, d = 8 (3) 374 / 320, 4 levels 343; n = 16384, d = 12 115, 3 levels 117. */
static void choose_start(const odp_shape *sh, int base, int chunks, gbx_sweep *c)
{
  const int n = shape_n(sh), d = sh->degree;
  const double gathered = (d + 1.0) * ((c->B + 255) / 256);
  c->base = base;
  c->scratch_rows = 8;
  c->scratch_bits = c->B <= 32768 ? (c->B + 255) / 256 * 256 : 32768;
  if(base < 2 || sh->symmetries > 1) return;
  const double most = 1.57 * gathered + 64.0;
  double marks = (double)d * d;
  int queue = 1 + d, levels = 2;
  while(levels < GBX_SWEEP_BASE && marks * d + queue + marks <= most && (levels + 1) * c->nchunks <= 2 * chunks){
    queue += (int)marks;
    marks *= d;
    levels++;
  }
  const int bits = (n + 255) / 256 * 256, row = bits / 8 + (queue + 3) / 4 * 16;
  if(levels == 2 || 3 * row > 36 * 1024) return;
  c->base = levels;
  c->queue = (queue + 3) / 4 * 4;
  c->scratch_bits = bits;
  while(c->scratch_rows * row > 36 * 1024) c->scratch_rows--;      /* four CTAs per SM */
}

/* Whether no schedule setting asks for the persistent engine. */
static int lockstep_allowed(const odp_shape *sh, const odp_tuning *t)
{
  const ODPX_Tune_entry *te = table_lookup(shape_n(sh), sh->degree, sh->grid);
  return t->sweep && t->wc_log2 <= 0 && t->slots <= 0 && t->tile_rows <= 0 && !t->local_kb_explicit &&
         t->activity == -2 && !(te && (te->wc_log2 > 0 || te->tile_kb > 0 || te->local_kb > 0));
}

/* A grid of more neighbours than the tracking kernel takes: its levels gather
 * every lane that is not full, however many they are, where the engine tracks
 * changes. */
static int dense_grid(const odp_shape *sh) { return sh->grid && shape_dp(sh) > GBX_SWEEP_TRACK_DEGREE; }

/* Whether a single graph of very many rows and few sources is faster on the
 * engine, which moves rows of 16 bytes where lockstep moves 32 (up to 128
 * sources), and whole rows of up to 128 bytes where lockstep, whose two
 * buffers are to stay in L2, takes 32 bytes of each at a time (up to 1024).
 * Measured on GB300, lockstep against engine (us): 16 to 128 sources, n = 120000,
 * d = 4 132 / 158, d = 8 121 / 121, n = 140000, d = 4 148 / 161, d = 8 139 / 133, d =
 * 12 139 / 131, n = 200000, d = 4 186 / 168, n = 262144, d = 8 220 / 183, n = 10^6, d
 * = 4 751 / 404; but 140 sources, n = 200000 186 / 231; 1000 sources, n = 400000, d =
 * 8 461 / 445, d = 16 faster by 1.25; n = 450000, d = 8 520 / 476, d = 12 542 / 539; n
 * = 600000, d = 8 813 / 601, n = 10^6, d = 4 1385 / 1117; but 1500 sources, n =
 * 600000 1061 / 1381. */
static int few_sources(const odp_shape *sh)
{
  const int n = shape_n(sh), W = shape_words(sh);
  return (W <= 2 && n > (sh->degree > 4 ? 130000 : 170000)) || (W <= 16 && n > 420000 && sh->degree <= 10);
}

/* Whether a plan runs on the lockstep kernels (sweep.cu), and its shape.  One
 * graph, no schedule setting, and a CTA's rows must fit in its shared memory
 * beside their lane states.  Measured on GB300 against the persistent engine:
 * n = 4096, d = 24: 27 against 67 us; n = 9999, s = 3: 48 against 108; n =
 * 65536, d = 16: 1.34 against 2.63 ms; n = 262144, s = 64: 0.63 against 1.0;
 * 97 x 103 grid: 0.34 against 0.76; 256 x 256: 5.3 against 18.5.
 *  - Grids of degree up to 32 track changed lanes, 65536 sources at a time, in
 *    the wide form while two CTAs per SM have a thread for every word of their
 *    rows' changes; past that a level takes a second round, and three narrower
 *    CTAs are faster (us): 135 x 135, d = 4 536 / 554; 140 x 140, d = 4 1031 /
 *    872; 150 x 150, d = 6 910 / 823; 190 x 190, d = 10 1913 / 1756; 256 x 256, d
 *    = 6 5431 / 5281.
 *  - Graphs whose bitset buffers take at most 64 MB, and a row 64 lanes, run
 *    all chunks at once.  With at most one lane per thread of two CTAs per SM
 *    they take the wide form.
 *  - Larger ones keep the start's bits of all chunks (n * B / 8 bytes) apart
 *    and run groups of chunks: 256-byte rows while both buffers of a chunk
 *    stay within 70 MB, narrower above (n = 262144: 0.63 ms with 128-byte
 *    rows, 0.94 with 256, 0.82 with 64); as many chunks in a phase as fit in
 *    75 MB (n = 262144, two chunks of 67 MB: 1.07 ms); and two phases, one
 *    computing while the other's barrier is crossed, where two chunks fit in
 *    80 MB (n = 65536, with two levels from the lists: two phases of two
 *    chunks 1.65 ms, of one 1.71, one phase of two 1.69).
 *  - Dense grids of more than 25000 sources stay on the engine; lockstep against
 *    it (ms), edges up to 2 to 10 columns long: 150 x 150, d = 34 5.7 / 8.0, d = 40
 *    19.5 / 23.1; 170 x 170 13.9 / 12.0, 46.5 / 34.9, d = 64 6.5 / 7.9; 200 x 200 33.0 /
 *    26.8, 113 / 80; 256 x 256 159 / 84, 550 / 251, s = 2 30.9 / 20.6, s = 4 0.94 / 1.88.
 *  - Without symmetry, a compact adjacency of up to 1 MB is expanded straight
 *    from host memory (n = 4096: 27.2 against 29.8 us); larger ones are copied
 *    first, in wider pieces. */
static int choose_sweep(const odp_shape *sh, const odp_tuning *t, int sms, gbx_sweep *sw, int *grid_out)
{
  if(!lockstep_allowed(sh, t) || t->blocks > 0 || few_sources(sh)) return 0;
  if(dense_grid(sh) && shape_n(sh) / sh->symmetries > 25000) return 0;
  const int n = shape_n(sh), W = shape_words(sh), full_l2 = ilog2_ceil(W < 4 ? 4 : W);
  memset(sw, 0, sizeof(*sw));
  sw->e.d = sh->degree;
  sw->e.dp = shape_dp(sh);
  sw->B = n / sh->symmetries;
  sw->phases = 1;
  sw->track = sh->grid && sw->e.dp <= GBX_SWEEP_TRACK_DEGREE;
  sw->in_place = !sh->grid && sh->symmetries == 1 && (double)n * sh->degree * 4 <= 1e6;
  if(sw->track){
    sw->wc_log2 = full_l2 < 5 ? full_l2 : 5;
    sw->slots = (W + (1 << sw->wc_log2) - 1) >> sw->wc_log2;
    if(sw->slots > GBX_SWEEP_SLOTS) sw->slots = GBX_SWEEP_SLOTS;
    int words = 1;
    while(32 * words < (sw->slots << (sw->wc_log2 - 2))) words *= 2;
    sw->wide = (double)n * words <= 2.0 * 256 * sms;
  }
  else if(16.0 * n * W <= 64e6 && W <= 256){
    sw->wc_log2 = full_l2 < 6 ? full_l2 : 6;
    sw->slots = (W + (1 << sw->wc_log2) - 1) >> sw->wc_log2;
    sw->wide = (double)n * ((W + 3) / 4) <= 2.0 * 256 * sms;
  }
  else{
    int wl = full_l2 < 5 ? full_l2 : 5;
    while(wl > 2 && 16.0 * n * (1 << wl) > 70e6) wl--;
    const double pair = 16.0 * n * (1 << wl);            /* both buffers of a chunk */
    const int chunks = (W + (1 << wl) - 1) >> wl;
    sw->phases = 2.0 * pair <= 80e6 && chunks > 1 ? 2 : 1;
    int q = (int)(75e6 / pair);
    if(q > (chunks + sw->phases - 1) / sw->phases) q = (chunks + sw->phases - 1) / sw->phases;
    if(q > 8) q = 8;
    sw->slots = q < 1 ? 1 : q;
    sw->wc_log2 = wl;
  }
  sw->nchunks = (W + (1 << sw->wc_log2) - 1) >> sw->wc_log2;
  if(!sw->track) choose_start(sh, sw->e.dp <= GBX_SWEEP_TWO_LEVEL ? 2 : 1, GBX_SWEEP_CHUNKS, sw);
  if(sw->nchunks > GBX_SWEEP_CHUNKS) return 0;
  for(int per_sm = sw->wide ? 2 : sw->track ? 3 : 4; per_sm >= 1; per_sm--)
    for(int q = sw->slots; q >= 1; q = q > 1 ? (q + 1) / 2 : 0){
      gbx_sweep c = *sw;
      int fit = 0;
      c.slots = q;
      c.rows = (n + per_sm * sms - 1) / (per_sm * sms);
      while((32 << c.word_log2) < (q << (c.wc_log2 - 2))) c.word_log2++;
      if(gbx_sweep_blocks(&c, &fit) == 0 && fit >= per_sm){
        /* bitsets that would take more than half of the free memory are left
         * to the engine, whose slots hold a few chunks only */
        const double bitsets = 16.0 * n * c.phases * q * (1 << c.wc_log2) + (c.track ? 0.0 : 8.0 * n * W);
        size_t room = 0;
        if(gbx_mem_free(&room) || bitsets > 0.5 * (double)room) return 0;
        *sw = c;
        *grid_out = (n + c.rows - 1) / c.rows;
        return 1;
      }
      if(!sw->track) break;
    }
  return 0;
}

/* Whether the team kernel takes a graph of this shape: it must fit the lockstep
 * kernels in one group (bitsets of at most 64 MB, 64 lanes a row, 256 for
 * grids).  Its cost on the whole GPU is estimated from its traffic: a general
 * graph's gathered levels and lists at 10 TB/s; for tracked grids 6.5 visits per row and
 * lane, each reading d + 2 sectors, at 8 TB/s; its latency from its levels.
 * The constants are fitted to 785 graphs of seven batches on teams of 1/2 to
 * 1/256 of the GPU (error of a graph's time 25 %). */
int odp_team_shape(const odp_shape *sh, const odp_tuning *t, gbx_sweep *c, odp_team_graph *g)
{
  const int n = shape_n(sh), W = shape_words(sh), full_l2 = ilog2_ceil(W < 4 ? 4 : W);
  memset(c, 0, sizeof(*c));
  if(!lockstep_allowed(sh, t) || 16.0 * n * W > 64e6 || W > (sh->grid ? 1024 : 256)) return 0;
  /* ten dense grids, teams / engine, us: 40 x 60, d = 36 938 / 1085, 52 x 52 1279 /
   * 1297, 56 x 56 1891 / 1580, 60 x 60 2730 / 1940, 90 x 90, d = 40 20.2 / 15.3 ms */
  if(dense_grid(sh) && n > 3000) return 0;
  c->e.dp = shape_dp(sh);
  c->B = n / sh->symmetries;
  c->phases = 1;
  c->track = sh->grid && c->e.dp <= GBX_SWEEP_TRACK_DEGREE;
  if(!c->track && W > 256) return 0;
  c->wc_log2 = c->track ? (full_l2 < 5 ? full_l2 : 5) : (full_l2 < 6 ? full_l2 : 6);
  c->nchunks = c->slots = (W + (1 << c->wc_log2) - 1) >> c->wc_log2;
  /* Two levels from the lists where a gathered level 2 would read more than 5000
   * bytes a row (d rows of 8 W), nearly all zeros; below that the marks cost a team
   * more than the level.  256 graphs 2.86 ms, never two levels 2.92; by the single
   * graphs' rule drawn batches went from 277 us (geometric mean) to 320 or more. */
  if(!c->track) choose_start(sh, c->e.dp <= GBX_SWEEP_TWO_LEVEL && 8.0 * W * sh->degree > 5000 ? 2 : 1, GBX_SWEEP_SLOTS, c);
  while((32 << c->word_log2) < (c->slots << (c->wc_log2 - 2))) c->word_log2++;
  const double lanes = (c->B + 255) / 256;
  if(c->track){
    g->cost = n * lanes * 6.5 * (sh->degree + 2) * 32.0 / 8e6;
    g->latency = 1.1 * (sh->width + sh->height);
  }
  else{
    double levels = 2.0, ball = sh->degree + 1.0;      /* until a ball of branching d - 1 holds n, and one more */
    for(const double grow = sh->degree > 3 ? sh->degree - 1.0 : 2.0; ball < n; ball *= grow) levels += 1.0;
    g->cost = (n * 8.0 * W * (sh->degree + 1) * (levels > 3.0 ? levels - 2.5 : 0.5) + 4.0 * n * c->e.dp * sh->degree) / 10e6;
    g->latency = 10.0 * levels;
  }
  g->need = 16.0 * ((double)n * c->slots * (1 << c->wc_log2)) + (c->track ? 8.0 * n * (1 << c->word_log2) : 0) + 1024;
  return 1;
}

/* The smallest of `at`, a heap of n, is to move down to its place. */
static void sift_down(double *at, int n, int i)
{
  const double x = at[i];
  for(int c; (c = 2 * i + 1) < n; i = c){
    if(c + 1 < n && at[c + 1] < at[c]) c++;
    if(at[c] >= x) break;
    at[i] = at[c];
  }
  at[i] = x;
}

/* Makespan (us) of the graphs on their teams: every team takes the next graph
 * of its size when it is free, and splits when there is none.  *last: the graph
 * that ends it.  `ord` holds the graphs, largest first; `list` takes them by
 * size of team.  The times at which the teams of a size are free are a heap. */
static double team_makespan(const odp_team_graph *g, const job_order *ord, int count, int *list, int *last)
{
  double at[1 << (GBX_TEAM_SPLITS - 1)] = {0};
  int first_of[GBX_TEAM_SPLITS] = {0};
  double end = 0;
  for(int j = 0; j < count; j++) first_of[g[j].split]++;
  for(int k = 1; k < GBX_TEAM_SPLITS; k++) first_of[k] += first_of[k - 1];
  for(int j = count - 1; j >= 0; j--) list[--first_of[g[ord[j].job].split]] = ord[j].job;
  for(int k = 0; k < GBX_TEAM_SPLITS && first_of[k] < count; k++){
    const int teams = 1 << k, from = first_of[k], to = k + 1 < GBX_TEAM_SPLITS ? first_of[k + 1] : count;
    if(k) for(int i = teams - 1; i >= 0; i--) at[i] = at[i >> 1];
    if(from < to) for(int i = teams / 2 - 1; i >= 0; i--) sift_down(at, teams, i);
    for(int j = from; j < to; j++){
      const odp_team_graph *x = &g[list[j]];
      at[0] += x->cost * teams + x->latency;
      if(at[0] > end){
        end = at[0];
        *last = list[j];
      }
      sift_down(at, teams, 0);
    }
  }
  return end;
}

/* The smallest team (of a grid of `grid` CTAs) that each graph fits: its rows a
 * CTA, the teams' bitsets 160 MB.  0 if some graph does not even fit the whole
 * grid. */
static int fit_teams(const odp_shape *shapes, int count, int grid, const gbx_sweep *gs, odp_team_graph *g)
{
  for(int i = 0; i < count; i++){
    g[i].fits = -1;
    for(int k = 0; k < GBX_TEAM_SPLITS && (1 << k) <= grid; k++){
      gbx_sweep c = gs[i];
      const int size = grid >> k;
      c.rows = (shape_n(&shapes[i]) + size - 1) / size;
      if(gbx_sweep_smem(&c) > ODP_TEAM_SMEM || (k > 0 && g[i].need * (1 << k) > 160e6)) break;
      g[i].fits = k;
    }
    if(g[i].fits < 0) return 0;
  }
  return 1;
}

/* Each graph's team: the smallest that it fits and on which it takes at most
 * `most` us. */
static void assign_teams(int count, double most, odp_team_graph *g)
{
  for(int i = 0; i < count; i++){
    g[i].split = 0;
    while(g[i].split < g[i].fits && g[i].cost * (2 << g[i].split) <= most) g[i].split++;
  }
}

/* What a row of a graph with many rows a source costs more on a small team than
 * on the engine (us): the lists and the start are work a row, and the team
 * kernel has half of the engine's warps on an SM.  Of 20 graphs with 4 rows a
 * source or more, ns a row, teams / engine, d = 8: up to 128 sources, n = 20000
 * .83 / .46, 50000 .68 / .34; 500 sources .95 / .68, .70 / .61; 2000 sources, n =
 * 8000 1.84 / 1.46, but 20000 1.37 / 1.21.  Other graphs gain about a fifth of
 * their cost, and a call 20 us, 40 where few graphs have large teams (3 graphs
 * of n = 8000 to 20000 1.3 to 1.9 times faster).  A batch that would lose more
 * than it gains stays on the engine: 40 of n = 20000, s = 100 578 -> 431 us, 50 of
 * n = 8000, s = 4 551 -> 483, 20 of n = 2000 and 3 of n = 200000, s = 2000 432 -> 333. */
double odp_team_slower(const odp_shape *sh)
{
  const int W = shape_words(sh);
  if(sh->grid || sh->symmetries < 4 || W > 32) return 0;
  return W <= 2 ? 0.25e-3 : W <= 16 ? 0.2e-3 : 0.15e-3;
}

/* Whether a plan runs on the team kernel, and which team each graph gets.
 * A graph's team is the smallest on which it takes no more
 * than a share of all graphs' cost, its rows fit a CTA's shared memory and
 * the teams' bitsets together stay within 160 MB; of several shares the one
 * with the least makespan is taken.  Shares above 1 let a few graphs of many
 * levels run side by side on small teams: 18 graphs of n = 360 to 2880, 366 ->
 * 207 us on GB300 with the fitted estimates. */
static int choose_team(const odp_shape *shapes, int count, const odp_tuning *t, int sms, gbx_sweep *gs,
                       gbx_team *tm, int *order, int *grid_out, size_t *smem_out, double *estimate)
{
  if(count == 1) return 0;
  int fit = 0;
  if(gbx_team_blocks(0, &fit) || fit < 2) return 0;
  int grid = 2 * sms;
  if(t->blocks > 0 && t->blocks < grid) grid = t->blocks;
  odp_team_graph *g = calloc((size_t)count, sizeof(odp_team_graph));
  job_order *ord = calloc((size_t)count, sizeof(job_order));
  int *list = calloc((size_t)count, sizeof(int));
  int ok = g && ord && list;
  double all = 0, lost = 0, won = count <= 4 ? 40.0 : 20.0;
  for(int i = 0; i < count && ok; i++){
    ok = odp_team_shape(&shapes[i], t, &gs[i], &g[i]);
    all += g[i].cost;
    ord[i].job = i;
    ord[i].work = g[i].cost;
    const double slower = odp_team_slower(&shapes[i]);
    if(slower > 0) lost += slower * shape_n(&shapes[i]);
    else won += 0.2 * g[i].cost;
  }
  ok = ok && lost <= won;
  if(ok) ok = fit_teams(shapes, count, grid, gs, g);
  if(ok){
    qsort(ord, (size_t)count, sizeof(job_order), cmp_work_desc);
    static const double shares[] = { 0.1, 0.2, 0.35, 0.6, 1.0, 2.0, 4.0, 8.0 };
    double best = 0, best_share = 0;
    int last = 0;
    for(int s = 0; s < 8; s++){
      assign_teams(count, shares[s] * all, g);
      const double m = team_makespan(g, ord, count, list, &last);
      if(s == 0 || m < best){ best = m; best_share = shares[s]; }
    }
    assign_teams(count, best_share * all, g);
    /* then larger teams for the graphs that end the run, while that shortens it
     * (256 graphs 2.87 -> 2.74 ms, 17 of n = 688 to 4128 392 -> 327 us) */
    best = team_makespan(g, ord, count, list, &last);
    for(int tries = count < 64 ? 2 * count : 128; tries > 0; tries--){
      const int i = last;
      if(g[i].split == 0) break;
      g[i].split--;
      const double m = team_makespan(g, ord, count, list, &last);
      if(m >= best){
        g[i].split++;
        break;
      }
      best = m;
    }
    *estimate = best;
    for(int i = 0; i < count; i++){
      const int size = grid >> g[i].split;
      gs[i].rows = (shape_n(&shapes[i]) + size - 1) / size;
    }
  }
  size_t smem = 0;
  double arena = 0;
  if(ok){
    int at = 0;
    tm->first_split = GBX_TEAM_SPLITS;
    tm->last_split = 0;
    for(int k = 0; k < GBX_TEAM_SPLITS; k++){
      tm->queue[k] = at;
      for(int j = 0; j < count; j++){
        const int i = ord[j].job;
        if(g[i].split != k) continue;
        order[at++] = i;
        if(k < tm->first_split) tm->first_split = k;
        tm->last_split = k;
        const size_t b = gbx_sweep_smem(&gs[i]);
        if(b > smem) smem = b;
        const double need = (double)ALIGN_UP((size_t)g[i].need, 256) + 512;
        if(need * (1 << k) > arena) arena = need * (1 << k);
      }
    }
    tm->queue[GBX_TEAM_SPLITS] = at;
    /* parts of every split are whole multiples of 256 bytes, so that a team's
     * part lies inside its parent's, whose other half may still be in use */
    tm->arena_bytes = ALIGN_UP((size_t)arena, (size_t)256 << (GBX_TEAM_SPLITS - 1));
    size_t room = 0;
    ok = gbx_team_blocks(smem, &fit) == 0 && fit * sms >= grid && gbx_mem_free(&room) == 0 &&
         arena <= 0.5 * (double)room;
  }
  *grid_out = grid;
  *smem_out = smem;
  free(g);
  free(ord);
  free(list);
  return ok;
}

#define CK(call) do{ int _e = (call); if(_e){ rc = ODPX_ERR_CUDA; goto fail; } }while(0)

/* Copies the shapes of a lockstep plan, from which `beside` is made. */
static int keep_shapes(odp_plan *p, const odp_shape *shapes)
{
  if(!(p->shapes = calloc((size_t)p->ngraphs, sizeof(odp_shape)))) return ODPX_ERR_MEMORY;
  for(int i = 0; i < p->ngraphs; i++){
    const size_t bytes = sizeof(int) * (size_t)p->g[i].B;
    p->shapes[i] = shapes[i];
    if(!shapes[i].num_degrees) continue;
    int *nd = malloc(bytes);
    if(nd) memcpy(nd, shapes[i].num_degrees, bytes);
    p->shapes[i].num_degrees = nd;
    if(!nd) return ODPX_ERR_MEMORY;
  }
  return 0;
}

int odp_plan_create(const odp_shape *shapes, int count, const odp_tuning *tuning, odp_plan **out)
{
  int rc = 0;
  *out = NULL;
  if(count <= 0) return ODPX_ERR_INVALID;
  for(int i = 0; i < count; i++){          /* arguments first: refused the same with or without a device */
    rc = validate_shape(&shapes[i]);
    if(rc) return rc;
  }
  if(odp_device_ready()) return ODPX_ERR_CUDA;

  odp_plan *p = calloc(1, sizeof(odp_plan));
  p->tuning = *tuning;
  p->ngraphs = count;
  p->g = calloc((size_t)count, sizeof(odp_plan_graph));
  p->blocks = tuning->blocks;          /* 0: chosen per launch from the staging size */
  p->spin_limit_ns = 60ull * 1000000000ull;
  const double budget = (double)tuning->l2_budget_mb * 1024.0 * 1024.0;
  const double local_bytes = (double)tuning->local_kb * 1024.0;

  /* A small plan: every job runs in the small-graph kernel, its bitsets and
   * row table in the shared memory of one thread-block cluster, with no
   * device-wide hand-off per level.  Other plans, and single graphs past the
   * line, run in lockstep or on teams where they fit, else on the engine. */
  const int sms = g_sm_count > 0 ? g_sm_count : 1;
  int *small_wl = calloc((size_t)count, sizeof(int));
  int small = choose_small(shapes, count, tuning, sms, small_wl, &p->small_cluster, &p->small_threads,
                           &p->small_smem, &p->small_part);
  p->small_class = small;
  p->sweep = count == 1 && (!small || small_yields(shapes, tuning, p->small_part, small_wl[0])) &&
             choose_sweep(shapes, tuning, sms, &p->sw, &p->sweep_grid);
  if(p->sweep){
    gbx_sweep c;
    odp_team_graph g;
    p->estimate = odp_team_shape(shapes, tuning, &c, &g) ? g.cost + g.latency : HUGE_VAL;
    small = 0;
  }
  int *team_order = NULL;
  if(!small && !p->sweep){
    p->h_teams = calloc((size_t)count, sizeof(gbx_sweep));
    team_order = calloc((size_t)count, sizeof(int));
    p->team = p->h_teams && team_order &&
              choose_team(shapes, count, tuning, sms, p->h_teams, &p->tm, team_order, &p->sweep_grid, &p->team_smem, &p->estimate);
  }
  const int lockstep = p->sweep || p->team;

  /* Shapes, chunk widths, tiles. */
  int njobs = 0;
  for(int i = 0; i < count; i++){
    const odp_shape *sh = &shapes[i];
    odp_plan_graph *g = &p->g[i];
    g->grid = sh->grid;
    g->n = sh->grid ? sh->width * sh->height : sh->nodes;
    g->d = sh->degree;
    g->dp = ALIGN_UP(sh->degree > 0 ? sh->degree : 1, 4);
    if(g->dp > p->max_dp) p->max_dp = g->dp;
    g->s = sh->symmetries;
    g->grid_s = sh->grid && sh->symmetries != 1;
    g->width = sh->width;
    g->height = sh->height;
    g->B = g->n / g->s;
    g->W = (g->B + 63) / 64;
    int full_l2 = ilog2_ceil(g->W < 2 ? 2 : g->W);
    const ODPX_Tune_entry *te = table_lookup(g->n, g->d, g->grid);
    int wl;
    if(tuning->wc_log2 > 0) wl = tuning->wc_log2;
    else if(te && te->wc_log2 > 0) wl = te->wc_log2;
    else if(tracks_changes(tuning, count, sh->grid, g->n, g->s)){
      /* 512-byte rows for a grid with change tracking (the 256 x 256 grid:
       * 24.4 ms with 64 words and 16 slots against 28.8 ms with 32 and 8) */
      wl = full_l2 < 6 ? full_l2 : 6;
    }
    else{
      /* 256-byte rows (32 words): measured best on GB300 for the 512-graph
       * batch and for single graphs (n = 1024, 65536, the 262144-vertex s = 64
       * graph and grids without change tracking) */
      wl = full_l2 < 5 ? full_l2 : 5;
    }
    if(wl < 1) wl = 1;
    if(wl > 7) wl = 7;                 /* rows of at most 1 KB per chunk */
    if(wl > full_l2 && full_l2 >= 1) wl = full_l2;
    if(small) wl = small_wl[i];
    if(p->sweep) wl = p->sw.wc_log2;
    if(p->team) wl = p->h_teams[i].wc_log2;
    g->wc_log2 = wl;
    const int wc = 1 << wl;
    g->nchunks = (g->W + wc - 1) / wc;
    g->has_ndeg = sh->num_degrees != NULL;
    g->has_itable = g->grid_s || (lockstep && sh->grid);   /* the lockstep kernels' grid rows follow a curve */
    g->has_srcpos = sh->grid && !lockstep;   /* grids: spatially compact source chunks */
    g->adj_ints = (size_t)g->B * g->d;
    g->adj_off = p->adj_ints;       p->adj_ints += ALIGN_UP(g->adj_ints, 4);
    g->ndeg_off = p->ndeg_ints;     if(g->has_ndeg) p->ndeg_ints += ALIGN_UP((size_t)g->n, 4);
    g->itable_off = p->itable_ints; if(g->has_itable) p->itable_ints += ALIGN_UP((size_t)g->n, 4);
    g->nbr_off = p->nbr_ints;       p->nbr_ints += (size_t)g->n * g->dp;
    g->srcpos_off = p->srcpos_ints; if(g->has_srcpos) p->srcpos_ints += ALIGN_UP((size_t)g->n, 4);
    p->total_vertices += g->n;
    njobs += g->nchunks;
  }
  p->njobs = njobs;
  p->small = small;
  free(small_wl);

  /* Tiles: about 640 KB of traffic each, measured best on GB300 for large
   * single graphs and for most size buckets of the batch.  A plan with few
   * jobs for the grid (a single graph, a group of annealing chains) takes
   * smaller tiles, and splits jobs it would otherwise run in one CTA, so
   * that its concurrently active jobs give every CTA about two tiles per
   * level.  A graph with change tracking, whose tiles mostly have little to
   * do, takes tiles of about 1.6 MB (the 256 x 256 grid: 400-row tiles,
   * 21.9 ms, against 23.6 ms with 160 rows and 24.0 ms with 640 on GB300). */
  const int grid_blocks = tuning->blocks > 0 ? tuning->blocks : gbx_engine_blocks(0);
  double fill_tile = 0;
  if(njobs * 4 <= grid_blocks){
    double active = 0;
    for(int i = 0; i < count; i++){
      const odp_plan_graph *g = &p->g[i];
      double lb = (double)g->n * (1 << g->wc_log2) * 8.0 * (g->d + 2);
      int conc = g->nchunks;
      if(count == 1){
        int cap = !g->grid ? 4 : tracks_changes(tuning, 1, 1, g->n, g->s) ? 16 : 8;
        if(conc > cap) conc = cap;
      }
      active += lb * conc;
    }
    fill_tile = active / (2.0 * (grid_blocks > 0 ? grid_blocks : 1));
    if(fill_tile < 32.0 * 1024.0) fill_tile = 32.0 * 1024.0;
  }
  for(int i = 0; i < count; i++){
    odp_plan_graph *g = &p->g[i];
    const ODPX_Tune_entry *te = table_lookup(g->n, g->d, g->grid);
    const int wc = 1 << g->wc_log2;
    double level_bytes = (double)g->n * wc * 8.0 * (g->d + 2);
    int rpp = rows_per_pass(g->wc_log2);
    double local_here = (te && te->local_kb > 0 && tuning->local_kb_explicit == 0) ? te->local_kb * 1024.0
                                                                                   : local_bytes;
    double tile_bytes = tracks_changes(tuning, count, g->grid, g->n, g->s) ? 1600.0 * 1024.0 : 640.0 * 1024.0;
    if(te && te->tile_kb > 0) tile_bytes = te->tile_kb * 1024.0;
    else if(fill_tile > 0 && fill_tile < tile_bytes){
      tile_bytes = fill_tile;
      if(!tuning->local_kb_explicit && fill_tile < local_here) local_here = fill_tile;
    }
    if(tuning->tile_rows > 0) g->tile_rows = ALIGN_UP(tuning->tile_rows, 4);   /* blocks start on 16-byte mask boundaries */
    else if(level_bytes <= local_here) g->tile_rows = g->n;
    else{
      double per_row = (double)wc * 8.0 * (g->d + 2);
      int tr = (int)(tile_bytes / per_row);
      g->tile_rows = ALIGN_UP(tr < rpp ? rpp : tr, rpp);
    }
    if(p->sweep) g->tile_rows = p->sw.rows;
    if(p->team) g->tile_rows = p->h_teams[i].rows;
    if(g->tile_rows > g->n) g->tile_rows = g->n;
    if(g->tile_rows < 1) g->tile_rows = 1;
    g->ntiles = (g->n + g->tile_rows - 1) / g->tile_rows;
  }

  /* Jobs, largest first so the long ones start early. */
  gbx_job *jobs = calloc((size_t)njobs, sizeof(gbx_job));
  job_order *ord = calloc((size_t)njobs, sizeof(job_order));
  {
    int k = 0;
    for(int i = 0; i < count; i++){
      odp_plan_graph *g = &p->g[i];
      int wc = 1 << g->wc_log2;
      for(int c = 0; c < g->nchunks; c++, k++){
        gbx_job *j = &jobs[k];
        j->n = g->n; j->dp = g->dp; j->d = g->d; j->wc_log2 = g->wc_log2;
        j->src0 = c * wc * 64;
        j->nsrc = g->B - j->src0 < wc * 64 ? g->B - j->src0 : wc * 64;
        j->sym = g->s; j->graph = i;
        j->tile_rows = g->tile_rows; j->ntiles = g->ntiles;
        j->flags = tracks_changes(tuning, count, g->grid, g->n, g->s) ? GBX_JOB_ACTIVE : 0;
        ord[k].job = k;
        ord[k].work = (double)g->n * wc * (g->d + 2) * (count > 1 && !p->team ? 1.0 : 0.0);
      }
    }
  }
  qsort(ord, (size_t)njobs, sizeof(job_order), cmp_work_desc);
  p->h_jobs = calloc((size_t)njobs, sizeof(gbx_job));
  for(int k = 0; k < njobs; k++){
    p->h_jobs[k] = jobs[ord[k].job];
    if(p->h_jobs[k].flags & GBX_JOB_ACTIVE) p->any_active = 1;
    else p->some_plain = 1;
  }
  free(jobs);
  free(ord);

  /* Slots: for batches, as many concurrent jobs as the L2 budget holds, at
   * least 64; for a single graph a fixed count measured best on GB300 (4 for
   * general graphs; 8 for grids, whose many short levels leave hand-offs to
   * hide, 16 for grids with change tracking).  Capped by the job count. */
  size_t max_words = 0, max_rows = 0;
  double sum_fp = 0;
  int fit = 0;
  for(int k = 0; k < njobs; k++){
    size_t w = (size_t)p->h_jobs[k].n << p->h_jobs[k].wc_log2;
    if(w > max_words) max_words = w;
    if((size_t)p->h_jobs[k].n > max_rows) max_rows = (size_t)p->h_jobs[k].n;
    double fp = 2.0 * 8.0 * (double)w;
    if(sum_fp + fp <= budget){ sum_fp += fp; fit++; }
  }
  int nslots = tuning->slots > 0 ? tuning->slots : fit;
  if(tuning->slots <= 0){
    if(nslots < 2) nslots = 2;
    if(count == 1){
      const int n0 = shapes[0].grid ? shapes[0].width * shapes[0].height : shapes[0].nodes;
      nslots = !shapes[0].grid ? 4 : tracks_changes(tuning, 1, 1, n0, shapes[0].symmetries) ? 16 : 8;
    }
    if(count > 1 && nslots < 64) nslots = 64;
    if(nslots > 512) nslots = 512;
  }
  if(p->sweep) nslots = p->sw.phases * p->sw.slots;
  if(p->team) nslots = 1;
  const size_t buffers = (size_t)nslots;
  if(nslots > njobs) nslots = njobs;
  if(nslots < 1) nslots = 1;
  p->nslots = nslots;
  p->slot_words = ALIGN_UP(max_words, 32);
  p->slot_rows = ALIGN_UP(max_rows, 64);

  /* Device memory. */
  p->out_off = sizeof(gbx_slot) * (size_t)nslots;
  p->acc_off = p->out_off + sizeof(gbx_ctrl) + 64;
  p->levels_off = p->acc_off + ALIGN_UP(sizeof(gbx_graph_acc) * (size_t)count, 64);
  p->state_bytes = p->levels_off + ALIGN_UP(sizeof(gbx_job_out) * (size_t)njobs, 64);
  p->out_bytes = p->state_bytes - p->out_off;

  CK(gbx_stream_create(&p->stream));
  CK(gbx_malloc((void **)&p->d_adj, sizeof(int) * (p->adj_ints ? p->adj_ints : 4)));
  if(p->ndeg_ints) CK(gbx_malloc((void **)&p->d_ndeg, sizeof(int) * p->ndeg_ints));
  if(p->itable_ints) CK(gbx_malloc((void **)&p->d_itable, sizeof(int) * p->itable_ints));
  CK(gbx_malloc((void **)&p->d_nbr, sizeof(int) * (p->nbr_ints ? p->nbr_ints : 4)));
  if(p->team) CK(gbx_malloc((void **)&p->d_slotbuf, p->tm.arena_bytes));
  else CK(gbx_malloc((void **)&p->d_slotbuf, sizeof(unsigned long long) * p->slot_words * 2 * (p->sweep ? buffers : (size_t)nslots)));
  CK(gbx_malloc((void **)&p->d_slotmask, sizeof(unsigned int) * p->slot_rows * 2 * (size_t)nslots));
  if(p->srcpos_ints) CK(gbx_malloc((void **)&p->d_srcpos, sizeof(int) * p->srcpos_ints));
  CK(gbx_malloc((void **)&p->d_expand, sizeof(gbx_expand_desc) * (size_t)count));
  CK(gbx_malloc((void **)&p->d_jobs, sizeof(gbx_job) * (size_t)njobs));
  CK(gbx_malloc((void **)&p->d_state, p->state_bytes));
  p->direct = tuning->direct && gbx_pageable_access();
  /* Small plans read their descriptors (and through them the adjacency)
   * from pinned host memory and write per-job records there. */
  if(p->direct || small || lockstep) CK(gbx_host_alloc((void **)&p->h_expand, sizeof(gbx_expand_desc) * (size_t)count));
  if(!p->direct) CK(gbx_host_alloc((void **)&p->h_adj, sizeof(int) * (p->adj_ints ? p->adj_ints : 4)));
  if(lockstep){
    CK(gbx_host_alloc((void **)&p->h_small_rec, sizeof(gbx_small_rec) * (size_t)njobs));
    memset(p->h_small_rec, 0, sizeof(gbx_small_rec) * (size_t)njobs);
    CK(gbx_host_device_ptr(p->h_small_rec, (void **)&p->d_small_rec));
    CK(gbx_host_alloc((void **)&p->h_abort, sizeof(unsigned int)));
    *p->h_abort = 0;
    CK(gbx_host_device_ptr(p->h_abort, (void **)&p->sw.abort_flag));
    if(p->team){
      /* the queue counters (256 bytes), then the teams' nodes */
      const int nodes = (2 << p->tm.last_split) - (1 << p->tm.first_split);
      p->team_node_bytes = 256 + gbx_team_node_bytes() * (size_t)nodes;
      CK(gbx_malloc(&p->d_sync, p->team_node_bytes));
      CK(gbx_malloc(&p->d_teams, (sizeof(gbx_sweep) + sizeof(int) + 2 * sizeof(unsigned long long)) * (size_t)count));
      CK(gbx_host_alloc((void **)&p->h_ptrs, sizeof(unsigned long long) * (size_t)count));
      if(p->itable_ints) CK(gbx_malloc((void **)&p->d_row_vertex, sizeof(int) * p->itable_ints));
    }
    else{
      CK(gbx_malloc(&p->d_sync, gbx_sweep_sync_bytes()));
      CK(gbx_memset(p->d_sync, 0, gbx_sweep_sync_bytes(), p->stream));
    }
    if(p->team){}
    else if(p->sw.track)
      CK(gbx_malloc((void **)&p->d_changed, sizeof(unsigned int) * 2 * ((size_t)p->g[0].n << p->sw.word_log2)));
    else if(njobs > p->sw.phases * p->sw.slots)   /* more than one group: the start's bits of every chunk apart */
      CK(gbx_malloc((void **)&p->d_start, sizeof(unsigned long long) * p->slot_words * (size_t)njobs));
    if(p->sweep && p->itable_ints) CK(gbx_malloc((void **)&p->d_row_vertex, sizeof(int) * p->itable_ints));
  }
  else if(small){
    CK(gbx_host_alloc((void **)&p->h_small_rec, sizeof(gbx_small_rec) * (size_t)njobs));
    memset(p->h_small_rec, 0, sizeof(gbx_small_rec) * (size_t)njobs);
    CK(gbx_host_device_ptr(p->h_small_rec, (void **)&p->d_small_rec));
    CK(gbx_host_device_ptr(p->h_expand, (void **)&p->d_small_desc));
  }
  else if(p->direct){
    /* the pull kernel reads this call's descriptors from pinned memory and
     * resets the engine state from a device copy of its initial value */
    CK(gbx_host_device_ptr(p->h_expand, (void **)&p->d_hexpand));
    CK(gbx_malloc((void **)&p->d_state_init, p->state_bytes));
  }
  CK(gbx_host_alloc((void **)&p->h_state_init, p->state_bytes));
  CK(gbx_host_alloc((void **)&p->h_state_out, p->out_bytes));
  memset(p->h_state_out, 0, p->out_bytes);

  /* Static tables: degrees, row tables, expand descriptors, jobs. */
  {
    int *h_nd = p->ndeg_ints ? malloc(sizeof(int) * p->ndeg_ints) : NULL;
    int *h_it = p->itable_ints ? malloc(sizeof(int) * p->itable_ints) : NULL;
    int *h_sp = p->srcpos_ints ? malloc(sizeof(int) * p->srcpos_ints) : NULL;
    gbx_expand_desc *ed = calloc((size_t)count, sizeof(gbx_expand_desc));
    long long first = 0;
    for(int i = 0; i < count; i++){
      odp_plan_graph *g = &p->g[i];
      if(g->has_ndeg){
        fill_degrees(&shapes[i], g->n, h_nd + g->ndeg_off);
        g->row_reads = 0;
        for(int v = 0; v < g->n; v++) g->row_reads += (double)h_nd[g->ndeg_off + v] + 2.0;
      }
      else g->row_reads = (double)g->n * (g->d + 2);
      if(g->has_itable && !lockstep) fill_itable(g->width, g->height, g->s, h_it + g->itable_off);
      if(g->has_srcpos) fill_srcpos(g, h_sp + g->srcpos_off);
      gbx_expand_desc *e = &ed[i];
      e->adj = p->d_adj + g->adj_off;
      e->ndeg = g->has_ndeg ? p->d_ndeg + g->ndeg_off : NULL;
      e->itable = g->has_itable ? p->d_itable + g->itable_off : NULL;
      e->nbr = p->d_nbr + g->nbr_off;
      e->n = g->n; e->d = g->d; e->dp = g->dp; e->s = g->s;
      e->width = g->width; e->height = g->height; e->grid_s = g->grid_s;
      e->first_vertex = first;
      first += g->n;
    }
    for(int k = 0; k < njobs; k++){
      const odp_plan_graph *g = &p->g[p->h_jobs[k].graph];
      p->h_jobs[k].nbr = p->d_nbr + g->nbr_off;
      p->h_jobs[k].srcpos = g->has_srcpos ? p->d_srcpos + g->srcpos_off : NULL;
    }
    if(lockstep && p->itable_ints){
      int *h_rv = malloc(sizeof(int) * p->itable_ints);
      rc = h_rv ? 0 : ODPX_ERR_MEMORY;
      for(int i = 0; i < count && !rc; i++){
        const odp_plan_graph *g = &p->g[i];
        if(g->has_itable) rc = fill_curve_rows(g, h_it + g->itable_off, h_rv + g->itable_off);
      }
      if(!rc && (gbx_memcpy_h2d(p->d_row_vertex, h_rv, sizeof(int) * p->itable_ints, p->stream) ||
                 gbx_stream_sync(p->stream)))
        rc = ODPX_ERR_CUDA;
      free(h_rv);
      if(rc){
        free(h_nd); free(h_it); free(h_sp); free(ed);
        goto fail;
      }
    }
    if(h_sp) CK(gbx_memcpy_h2d(p->d_srcpos, h_sp, sizeof(int) * p->srcpos_ints, p->stream));
    if(h_nd) CK(gbx_memcpy_h2d(p->d_ndeg, h_nd, sizeof(int) * p->ndeg_ints, p->stream));
    if(h_it) CK(gbx_memcpy_h2d(p->d_itable, h_it, sizeof(int) * p->itable_ints, p->stream));
    CK(gbx_memcpy_h2d(p->d_expand, ed, sizeof(gbx_expand_desc) * (size_t)count, p->stream));
    if(p->team){
      char *dev = p->d_teams;
      const size_t args = sizeof(gbx_sweep) * (size_t)count, ptrs = sizeof(unsigned long long) * (size_t)count;
      int job = 0;
      for(int i = 0; i < count; i++){
        gbx_sweep *w = &p->h_teams[i];
        const odp_plan_graph *g = &p->g[i];
        const size_t words = (size_t)g->n << g->wc_log2;
        w->e = ed[i];
        w->e.adj_dev = p->direct ? (int *)ed[i].adj : NULL;
        w->row_vertex = g->has_itable ? p->d_row_vertex + g->itable_off : NULL;
        w->slot_words = ALIGN_UP(words, 4) * (w->track ? (size_t)w->slots : 1);
        w->rec = p->d_small_rec + job;
        w->abort_flag = p->sw.abort_flag;
        job += w->nchunks;
      }
      gbx_team *tm = &p->tm;
      tm->graphs = (const gbx_sweep *)dev;
      tm->adj = p->direct ? (const unsigned long long *)(dev + args) : NULL;
      tm->order = (const int *)(dev + args + ptrs);
      tm->next = (unsigned int *)p->d_sync;
      tm->nodes = (char *)p->d_sync + 256;
      tm->arena = (unsigned char *)p->d_slotbuf;
      tm->abort_flag = p->sw.abort_flag;
      const long page = sysconf(_SC_PAGESIZE);
      tm->page_ints = (int)((page > 0 ? page : 4096) / (long)sizeof(int));
      CK(gbx_memcpy_h2d(dev, p->h_teams, args, p->stream));
      CK(gbx_memcpy_h2d(dev + args + ptrs, team_order, sizeof(int) * (size_t)count, p->stream));
    }
    else if(p->sweep){
      /* the launch carries the descriptor: per call `adj` names the caller's
       * array, which the kernel copies to `adj_dev`; without direct reads the
       * call uploads it and `adj` names the device copy */
      p->h_expand[0] = ed[0];
      p->h_expand[0].adj_dev = p->direct ? (int *)ed[0].adj : NULL;
      gbx_sweep *w = &p->sw;
      w->row_vertex = p->d_row_vertex;
      w->buf = p->d_slotbuf;
      w->slot_words = p->slot_words * (w->track ? (size_t)w->slots : 1);
      if(p->d_start){
        w->start = p->d_start;
        w->start_stride = p->slot_words;
      }
      else{                            /* the buffer that the first gathered level reads */
        w->start = p->d_slotbuf + ((w->base & 1) ? p->slot_words : 0);
        w->start_stride = 2 * p->slot_words;
      }
      w->sync = p->d_sync;
      w->changed = p->d_changed;
      w->rec = p->d_small_rec;
    }
    else if(small){
      /* the small-graph kernel reads `adj` itself: the caller's array (set
       * per call) or this plan's pinned staging copy */
      memcpy(p->h_expand, ed, sizeof(gbx_expand_desc) * (size_t)count);
      for(int i = 0; i < count; i++){
        p->h_expand[i].adj_dev = NULL;
        p->h_expand[i].adj = p->direct ? NULL : p->h_adj + p->g[i].adj_off;
      }
    }
    else if(p->direct){
      /* per call: `adj` names the caller's host array, `adj_dev` the device
       * copy that gbx_pull fills and expand reads */
      memcpy(p->h_expand, ed, sizeof(gbx_expand_desc) * (size_t)count);
      for(int i = 0; i < count; i++) p->h_expand[i].adj_dev = (int *)ed[i].adj;
    }
    CK(gbx_memcpy_h2d(p->d_jobs, p->h_jobs, sizeof(gbx_job) * (size_t)njobs, p->stream));
    CK(gbx_stream_sync(p->stream));
    free(h_nd); free(h_it); free(h_sp); free(ed);
  }
  free(team_order);
  team_order = NULL;
  if(lockstep && (rc = keep_shapes(p, shapes))) goto fail;

  fill_state_init(p);
  if(p->d_state_init){
    CK(gbx_memcpy_h2d(p->d_state_init, p->h_state_init, p->state_bytes, p->stream));
    CK(gbx_stream_sync(p->stream));
  }
  *out = p;
  return 0;

fail:
  free(team_order);
  odp_plan_destroy(p);
  return rc;
}

void odp_plan_destroy(odp_plan *p)
{
  if(!p) return;
  odp_plan_destroy(p->beside);
  for(int i = 0; p->shapes && i < p->ngraphs; i++) free((void *)p->shapes[i].num_degrees);
  free(p->shapes);
  if(p->graph_exec) gbx_graph_destroy(p->graph_exec);
  gbx_free(p->d_adj); gbx_free(p->d_ndeg); gbx_free(p->d_itable); gbx_free(p->d_nbr);
  gbx_free(p->d_slotbuf); gbx_free(p->d_slotmask); gbx_free(p->d_srcpos); gbx_free(p->d_expand); gbx_free(p->d_jobs); gbx_free(p->d_state);
  gbx_free(p->d_state_init);
  gbx_host_free(p->h_adj); gbx_host_free(p->h_expand); gbx_host_free(p->h_state_init); gbx_host_free(p->h_state_out);
  gbx_host_free(p->h_small_rec);
  gbx_free(p->d_row_vertex); gbx_free(p->d_changed); gbx_free(p->d_sync); gbx_free(p->d_start);
  gbx_host_free(p->h_abort); gbx_host_free(p->h_ptrs);
  gbx_free(p->d_teams);
  free(p->h_teams);
  if(p->stream) gbx_stream_destroy(p->stream);
  free(p->h_jobs);
  free(p->g);
  free(p);
}

/* The per-call GPU work, in stream order.  A small plan is one kernel: it
 * reads the adjacency from host memory and writes its records there. */
static int enqueue(odp_plan *p)
{
  int e;
  if(p->small) return odp_plan_enqueue_engine(p);
  if(p->team){
    if(p->direct){
      if((e = gbx_memcpy_h2d((void *)p->tm.adj, p->h_ptrs, sizeof(unsigned long long) * (size_t)p->ngraphs, p->stream)))
        return e;
    }
    else if((e = gbx_memcpy_h2d(p->d_adj, p->h_adj, sizeof(int) * (p->adj_ints ? p->adj_ints : 4), p->stream))) return e;
    return odp_plan_enqueue_engine(p);
  }
  if(p->sweep){
    if(!p->direct &&
       (e = gbx_memcpy_h2d(p->d_adj, p->h_adj, sizeof(int) * (p->adj_ints ? p->adj_ints : 4), p->stream)))
      return e;
    p->sw.e = p->h_expand[0];
    p->sw.limit_ns = p->spin_limit_ns;
    p->sw.seq = p->seq = p->seq % 0xffffffu + 1;
    if((e = gbx_sweep_launch(&p->sw, p->sweep_grid, p->stream))) return e;
    p->sw.set ^= 1;                    /* this launch clears the other half of the counters for the next */
    return 0;
  }
  if(p->direct){
    /* one kernel: this call's descriptors (their host pointers) from pinned
     * memory, the callers' arrays into the device copy that expand reads,
     * and the engine state reset */
    if((e = gbx_pull(p->d_hexpand, p->d_expand, p->ngraphs, p->d_state, p->d_state_init, p->state_bytes, p->stream)))
      return e;
  }
  else{
    if((e = gbx_memcpy_h2d(p->d_adj, p->h_adj, sizeof(int) * (p->adj_ints ? p->adj_ints : 4), p->stream))) return e;
    if((e = gbx_memcpy_h2d(p->d_state, p->h_state_init, p->state_bytes, p->stream))) return e;
  }
  if((e = gbx_expand(p->d_expand, p->ngraphs, p->total_vertices, p->max_dp,
                     (unsigned int *)(p->d_state + p->out_off + sizeof(gbx_ctrl)), p->stream))) return e;
  if((e = odp_plan_enqueue_engine(p))) return e;
  return gbx_memcpy_d2h(p->h_state_out, p->d_state + p->out_off, p->out_bytes, p->stream);
}

int odp_plan_enqueue_engine(odp_plan *p)
{
  if(p->team){
    int e = gbx_memset(p->d_sync, 0, p->team_node_bytes, p->stream);
    if(e) return e;
    p->tm.limit_ns = p->spin_limit_ns;
    return gbx_team_launch(&p->tm, p->sweep_grid, p->team_smem, p->stream);
  }
  if(p->small){
    /* one graph: its descriptor (this call's adjacency pointer) travels in
     * the launch's parameters, so the plan is launched directly each call */
    const int one = p->ngraphs == 1;
    if(one) p->seq = p->seq % 0xffffffu + 1;
    return gbx_small_launch(p->d_jobs, p->njobs, one ? NULL : p->d_small_desc, one ? &p->h_expand[0] : NULL,
                            p->d_small_rec, one ? p->seq : 0, p->small_smem, p->small_cluster, p->small_threads, p->small_part,
                            p->stream);
  }
  return gbx_engine_launch(p->d_jobs, p->njobs, (gbx_slot *)p->d_state, p->nslots,
                           (gbx_ctrl *)(p->d_state + p->out_off), (gbx_graph_acc *)(p->d_state + p->acc_off),
                           (gbx_job_out *)(p->d_state + p->levels_off), p->spin_limit_ns, p->blocks,
                           !p->any_active ? 0 : p->some_plain ? 2 : 1, p->stream);
}

const gbx_job_out *odp_plan_job_out(const odp_plan *p)
{
  return (const gbx_job_out *)(p->h_state_out + (p->levels_off - p->out_off));
}

typedef struct {
  odp_plan *p;
  const int *const *adjacency;
  int first, last;
} stage_part;

static void *stage_worker(void *arg)
{
  stage_part *w = arg;
  for(int i = w->first; i < w->last; i++){
    const odp_plan_graph *g = &w->p->g[i];
    memcpy(w->p->h_adj + g->adj_off, w->adjacency[i], sizeof(int) * g->adj_ints);
  }
  return NULL;
}

/* Hands this call's adjacency arrays to the device.  When kernels can read
 * pageable host memory, a pull kernel reads the callers' arrays in place
 * (coalesced 16-byte loads over the CPU-GPU link) and only their pointers are
 * recorded here: no host-side copy.  Otherwise the arrays
 * are copied into the pinned staging buffer that the upload reads; large
 * batches are split over host threads by bytes, since one thread copies at a
 * fraction of the memory bandwidth. */
void odp_plan_stage(odp_plan *p, const int *const *adjacency)
{
  if(p->direct){
    /* The device reads pageable host memory: no staging copy, only the
     * pointers (the arrays must stay unchanged until the run is finished). */
    for(int i = 0; i < p->ngraphs; i++) p->h_expand[i].adj = adjacency[i];
    if(p->team)
      for(int i = 0; i < p->ngraphs; i++) p->h_ptrs[i] = (unsigned long long)(uintptr_t)adjacency[i];
    return;
  }
  size_t total = sizeof(int) * p->adj_ints;
  long cpus = sysconf(_SC_NPROCESSORS_ONLN);
  int nt = total < (4u << 20) ? 1 : (int)(cpus < 16 ? cpus : 16);
  if(nt > p->ngraphs) nt = p->ngraphs;
  if(nt <= 1){
    stage_part w = { p, adjacency, 0, p->ngraphs };
    stage_worker(&w);
    return;
  }
  stage_part parts[16];
  pthread_t th[16];
  size_t per = total / (size_t)nt, acc = 0;
  int start = 0, k = 0;
  for(int i = 0; i < p->ngraphs && k < nt - 1; i++){
    acc += sizeof(int) * p->g[i].adj_ints;
    if(acc >= per * (size_t)(k + 1)){
      parts[k] = (stage_part){ p, adjacency, start, i + 1 };
      start = i + 1;
      k++;
    }
  }
  parts[k++] = (stage_part){ p, adjacency, start, p->ngraphs };
  int launched[16] = {0};
  for(int t = 1; t < k; t++) launched[t] = pthread_create(&th[t], NULL, stage_worker, &parts[t]) == 0;
  stage_worker(&parts[0]);
  for(int t = 1; t < k; t++){
    if(launched[t]) pthread_join(th[t], NULL);
    else stage_worker(&parts[t]);
  }
}

int odp_plan_launch(odp_plan *p)
{
  /* single-graph plans of one kernel pass this call's descriptor by value: never captured */
  if(p->tuning.use_graph && !p->sweep && !(p->small && p->ngraphs == 1)){
    if(!p->graph_exec){
      if(gbx_capture_begin(p->stream)) return ODPX_ERR_CUDA;
      int e = enqueue(p);
      void *ge = NULL;
      int e2 = gbx_capture_end(p->stream, &ge);
      if(e || e2) return ODPX_ERR_CUDA;
      p->graph_exec = ge;
    }
    return gbx_graph_launch(p->graph_exec, p->stream) ? ODPX_ERR_CUDA : 0;
  }
  return enqueue(p) ? ODPX_ERR_CUDA : 0;
}

/* Longest-processing-time order learned from a finished run.  The first
 * order sorts jobs by their per-level traffic, which does not know how many
 * levels each job will run; a graph with a long diameter (a grid with a short
 * length limit) then starts late and ends the batch alone.  After the first
 * run the jobs are re-sorted by their measured device time (load to finish),
 * so the next runs start the longest ones first.  Results do not depend on
 * the order.  The per-job records of the finished run are permuted the same
 * way so that they stay matched with the job table.  Runs with the stream
 * idle (after the synchronisation in odp_plan_finish), so neither the job
 * table nor the initial state is being read by the device. */
static int reorder_by_duration(odp_plan *p)
{
  gbx_job_out *jo = (gbx_job_out *)(p->h_state_out + (p->levels_off - p->out_off));
  unsigned long long t0 = ((const gbx_ctrl *)p->h_state_out)->t_start;
  for(int k = 0; k < p->njobs; k++){
    if(jo[k].t_loaded && jo[k].t_loaded < t0) t0 = jo[k].t_loaded;
    if(jo[k].t_done && jo[k].t_done < t0) t0 = jo[k].t_done;
  }
  job_order *ord = malloc(sizeof(job_order) * (size_t)p->njobs);
  gbx_job *nj = malloc(sizeof(gbx_job) * (size_t)p->njobs);
  gbx_job_out *no = malloc(sizeof(gbx_job_out) * (size_t)p->njobs);
  if(!ord || !nj || !no){ free(ord); free(nj); free(no); return ODPX_ERR_MEMORY; }
  for(int k = 0; k < p->njobs; k++){
    unsigned long long a = jo[k].t_loaded ? jo[k].t_loaded : t0;
    ord[k].job = k;
    ord[k].work = jo[k].t_done > a ? (double)(jo[k].t_done - a) : 0.0;
  }
  qsort(ord, (size_t)p->njobs, sizeof(job_order), cmp_work_desc);
  for(int k = 0; k < p->njobs; k++){
    nj[k] = p->h_jobs[ord[k].job];
    no[k] = jo[ord[k].job];
  }
  memcpy(p->h_jobs, nj, sizeof(gbx_job) * (size_t)p->njobs);
  memcpy(jo, no, sizeof(gbx_job_out) * (size_t)p->njobs);
  free(ord); free(nj); free(no);
  fill_state_init(p);
  if(gbx_memcpy_h2d(p->d_jobs, p->h_jobs, sizeof(gbx_job) * (size_t)p->njobs, p->stream)) return ODPX_ERR_CUDA;
  if(p->d_state_init && gbx_memcpy_h2d(p->d_state_init, p->h_state_init, p->state_bytes, p->stream))
    return ODPX_ERR_CUDA;
  if(gbx_stream_sync(p->stream)) return ODPX_ERR_CUDA;
  return 0;
}

/* Plans of one kernel: the per-job records folded per graph, as the engine's
 * accumulators fold them (sum of the jobs' sums, the largest level, stalled
 * if any job stalled); the levels and stamps also go to the per-job outcome
 * table that the introspection calls read. */
static int finish_small(odp_plan *p, odp_result *results)
{
  gbx_job_out *jo = (gbx_job_out *)(p->h_state_out + (p->levels_off - p->out_off));
  unsigned int err = 0;
  for(int k = 0; k < p->njobs; k++){
    err |= GBX_REC_ERR(p->h_small_rec[k].err);
    jo[k].level = p->h_small_rec[k].level;
    jo[k].t_loaded = p->h_small_rec[k].t_loaded;
    jo[k].t_done = p->h_small_rec[k].t_done;
  }
  if(err & GBX_ERR_BAD_ADJ) return ODPX_ERR_ADJACENCY;
  for(int i = 0; i < p->ngraphs; i++){
    results[i].sum = 0;
    results[i].diameter = 0;
    results[i].aspl = 0.0;                       /* set when a job stalled */
  }
  for(int k = 0; k < p->njobs; k++){
    const gbx_small_rec *r = &p->h_small_rec[k];
    odp_result *res = &results[p->h_jobs[k].graph];
    const int l = r->level < 0 ? -r->level : r->level;
    res->sum += (long)r->sum;
    if(l > res->diameter) res->diameter = l;
    if(r->level < 0) res->aspl = 1.0;
  }
  for(int i = 0; i < p->ngraphs; i++){
    const odp_plan_graph *g = &p->g[i];
    odp_result *res = &results[i];
    if(res->aspl != 0.0){
      res->diameter = INT_MAX;
      res->sum = LONG_MAX;
      res->aspl = DBL_MAX;
      continue;
    }
    const long total = res->sum;
    res->aspl = total / (((double)g->n - 1) * g->n);
    res->sum = (long)(total / 2.0);
  }
  return 0;
}

/* Waits for the records of the last launch (plans of one graph and one
 * kernel).  Taking them as they arrive saves the kernel's teardown and the
 * driver's wake-up: n = 256, d = 5 through ODP_Set_aspl 25.1 -> 22.5 us, n =
 * 1024, d = 8 27.3 -> 24.5 us on GB300.  The kernel has long read the caller's
 * array by then, and the stream orders whatever is launched next after its
 * end.  Past two milliseconds, or when a wait ran out, the stream is
 * synchronised instead. */
static int take_records(odp_plan *p)
{
  struct timespec t0, t;
  clock_gettime(CLOCK_MONOTONIC, &t0);
  for(int k = 0, spins = 0; k < p->njobs;){
    if(GBX_REC_SEQ(__atomic_load_n(&p->h_small_rec[k].err, __ATOMIC_ACQUIRE)) == p->seq){
      k++;
      continue;
    }
    if(++spins & 255) continue;
    clock_gettime(CLOCK_MONOTONIC, &t);
    if((p->h_abort && __atomic_load_n(p->h_abort, __ATOMIC_ACQUIRE)) ||
       (t.tv_sec - t0.tv_sec) * 1000000000ll + (t.tv_nsec - t0.tv_nsec) > 2000000ll)
      return gbx_stream_sync(p->stream);
  }
  return 0;
}

/* Whether every record is the last launch's. */
static int records_current(const odp_plan *p)
{
  for(int k = 0; k < p->njobs; k++)
    if(GBX_REC_SEQ(__atomic_load_n(&p->h_small_rec[k].err, __ATOMIC_ACQUIRE)) != p->seq) return 0;
  return 1;
}

int odp_plan_finish(odp_plan *p, odp_result *results)
{
  if(p->seq ? take_records(p) : gbx_stream_sync(p->stream)) return ODPX_ERR_CUDA;
  if(p->h_abort && *p->h_abort){
    /* a wait that ran out behind the last record (a CTA with nothing left to
     * do; perhaps the launch's before this one) has spoiled nothing */
    *p->h_abort = 0;
    if(!p->seq || !records_current(p)) return ODPX_ERR_TIMEOUT;
  }
  if(p->small || p->sweep || p->team) return finish_small(p, results);
  const gbx_ctrl *ctrl = (const gbx_ctrl *)p->h_state_out;
  unsigned int err = *(const unsigned int *)(p->h_state_out + sizeof(gbx_ctrl)) | ctrl->error;
  if(err & GBX_ERR_TIMEOUT) return ODPX_ERR_TIMEOUT;
  if(err & GBX_ERR_BAD_ADJ) return ODPX_ERR_ADJACENCY;
  if(p->tuning.reorder && !p->small && !p->reordered && p->njobs > p->nslots){
    p->reordered = 1;
    int e = reorder_by_duration(p);
    if(e) return e;
  }
  const gbx_graph_acc *acc = (const gbx_graph_acc *)(p->h_state_out + (p->acc_off - p->out_off));
  p->bytes_alg_last = 0;
  for(int i = 0; i < p->ngraphs; i++){
    const odp_plan_graph *g = &p->g[i];
    odp_result *r = &results[i];
    if(acc[i].flags & 1){
      r->diameter = INT_MAX;
      r->sum = LONG_MAX;
      r->aspl = DBL_MAX;
      continue;
    }
    long sum = (long)acc[i].sum;
    r->diameter = acc[i].levels;
    r->aspl = sum / (((double)g->n - 1) * g->n);
    r->sum = (long)(sum / 2.0);
  }
  return 0;
}

/* The plan that a call of p runs.  A cooperative launch waits until all of its
 * CTAs fit on the GPU at once, and behind a busy server's long batches it waits
 * for all lanes to be free together, where the other kernels' CTAs start as
 * soon as one leaves.  So beside such batches a lockstep plan's call runs on
 * the kernels that its shapes take without lockstep (a plan of its own, made the
 * first time).  Measured on GB300, us, n = 4096, d = 24 through ODP_Set_aspl,
 * lockstep against this, beside chains of n = 8192: 966 / 395; 16384: 2618 / 155;
 * 32768: 7262 / 163; 90 x 90 grids: 6678 / 142; alone 33 / 76.  Behind team
 * batches, which leave less room to other kernels, a call of more than 200 us
 * waits: beside chains of n = 8192, n = 9999 (110 us by the estimate) 1035 / 547, 40
 * graphs of n = 300 to 2000 1556 / 735, but n = 20000 (230) 1278 / 1329, 97 x 103 grid
 * (300) 1077 / 2270. */
static odp_plan *plan_for_call(odp_plan *p)
{
  const int held = p->shapes ? odp_serving() : 0;
  if(!held || (held == 1 && p->estimate > 200.0)) return p;
  if(!p->beside){
    odp_tuning t = p->tuning;
    t.sweep = 0;
    if(odp_plan_create(p->shapes, p->ngraphs, &t, &p->beside)) return p;
    p->beside->spin_limit_ns = p->spin_limit_ns;
  }
  return p->beside;
}

int odp_plan_run(odp_plan *p, const int *const *adjacency, odp_result *results)
{
  odp_plan *q = plan_for_call(p);
  p->ran = q;
  odp_plan_stage(q, adjacency);
  if(q != p) odp_plan_stage(p, adjacency);       /* a timing call may ask for the last run's arrays */
  int rc = odp_plan_launch(q);
  if(rc) return rc;
  return odp_plan_finish(q, results);
}

unsigned long long odp_plan_tiles(const odp_plan *p)
{
  return ((const gbx_ctrl *)p->h_state_out)->tiles;
}

unsigned int odp_plan_error(const odp_plan *p)
{
  if(p->small || p->sweep || p->team){
    unsigned int err = p->h_abort ? *p->h_abort : 0;
    for(int k = 0; k < p->njobs; k++) err |= GBX_REC_ERR(p->h_small_rec[k].err);
    return err;
  }
  const gbx_ctrl *ctrl = (const gbx_ctrl *)p->h_state_out;
  return *(const unsigned int *)(p->h_state_out + sizeof(gbx_ctrl)) | ctrl->error;
}

double odp_plan_bytes_alg(const odp_plan *p)
{
  const gbx_job_out *jo = odp_plan_job_out(p);
  double total = 0;
  for(int k = 0; k < p->njobs; k++){
    const gbx_job *j = &p->h_jobs[k];
    int l = jo[k].level < 0 ? -jo[k].level : jo[k].level;
    /* only the chunk's words that hold sources count; padding words of a
     * narrow last chunk are moved but are not algorithmic */
    double words = (double)((j->nsrc + 63) / 64);
    total += (double)l * 8.0 * words * p->g[j->graph].row_reads;
  }
  return total;
}
