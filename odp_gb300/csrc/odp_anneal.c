/*
 * odp_anneal.c -- host side of the device-resident annealing chains
 * (ODPX_Anneal_*, kernels in anneal_resident.cu and anneal.cu).
 *
 * Chains whose compact adjacency fits a CTA's shared memory run many steps
 * per launch in the resident kernel.  The others step as follows.
 *
 * A set of chains is one batch plan (odp_plan.c): every chain's graph is a
 * graph of the plan, uploaded and expanded once.  A step is four stream-ordered
 * operations and no host round trip: the proposal kernel, a device-to-device
 * reset of the engine state, the engine, and the decision kernel.  The host
 * only reads state back when asked.
 *
 * Each chain follows the reference's annealing client (sample/SA/general.c:
 * 130-191, general_s.c:152-191): temp starts at max_temp and is multiplied by
 * cooling_rate = pow(min_temp / max_temp, 1.0 / ncalcs) after every step
 * (0 for hill climbing), the best graph is kept, and accept_s decides.
 */
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include "odp_plan.h"
#include "odp_rng.h"
#include "odp_gb300.h"

#define ANNEAL_GRAPH_STEPS 8   /* steps per replayed CUDA graph */
#define RESIDENT_STEPS 512     /* steps per launch of the resident kernel */
#define RESIDENT_LANES 32      /* lanes a thread walks per level, at most */
#define RESIDENT_HOST (64 << 20) /* pinned bytes of a group's records and graphs, at most */

struct odpx_anneal {
  odp_plan *p;
  int count;
  gbx_chain *h_chains, *d_chains;
  int *d_best, *d_rowdeg;
  char *d_state_init;
  void *steps_exec;            /* ANNEAL_GRAPH_STEPS steps captured as one CUDA graph */
  int resident;                /* the steps run in the resident kernel */
  gbx_resident res;
  int res_blocks, res_cluster;
  size_t res_smem;
  void *d_res;                 /* its barrier words, bitset and host offsets and bitsets */
  char *h_res;                 /* pinned: the chains' records and graphs after a run, or NULL */
  gbx_chain *dh_chains;
  int h_current;               /* they are the chains' state */
  unsigned int *h_late;        /* pinned: a wait of the last run ran out */
  unsigned long long *h_offset; /* in ints, chain k's graphs among them */
};

/* ODP_GB300_ANNEAL_RESIDENT=0 keeps the stepwise kernels. */
static int env_resident(void)
{
  const char *v = getenv("ODP_GB300_ANNEAL_RESIDENT");
  return v && *v ? atoi(v) : 1;
}

static int chain_nodes(const ODPX_Chain *c)
{
  return c->grid ? c->width * c->height : c->nodes;
}

static int check_chain(const ODPX_Chain *c)
{
  if(!c->adjacency || c->degree <= 0 || c->symmetries <= 0) return ODPX_ERR_INVALID;
  if(c->grid){
    /* the grid 2-opt takes s = 1, 2 or 4 (utils.c:125-133), 4 on square grids */
    if(c->width <= 0 || c->height <= 0 || c->length <= 0) return ODPX_ERR_INVALID;
    if(c->symmetries != 1 && c->symmetries != 2 && c->symmetries != 4) return ODPX_ERR_INVALID;
    if(c->symmetries > 1 && c->width % 2) return ODPX_ERR_INVALID;
    if(c->symmetries == 4 && (c->height % 2 || c->width != c->height)) return ODPX_ERR_INVALID;
  }
  else if(c->nodes <= 0) return ODPX_ERR_INVALID;
  if(chain_nodes(c) % c->symmetries) return ODPX_ERR_INVALID;
  if(!c->hill_climbing && (!(c->max_temp > 0) || !(c->min_temp > 0) || c->ncalcs <= 0)) return ODPX_ERR_INVALID;
  if(c->num_degrees){
    int base = chain_nodes(c) / c->symmetries;
    for(int i = 0; i < base; i++)
      if(c->num_degrees[i] < 0 || c->num_degrees[i] > c->degree) return ODPX_ERR_INVALID;
  }
  return 0;
}

void ODPX_Anneal_destroy(ODPX_Anneal *a)
{
  if(!a) return;
  if(a->steps_exec) gbx_graph_destroy(a->steps_exec);
  if(a->p) odp_plan_destroy(a->p);
  gbx_free(a->d_res);
  gbx_host_free(a->h_res);
  gbx_host_free(a->h_late);
  free(a->h_offset);
  gbx_free(a->d_chains); gbx_free(a->d_best); gbx_free(a->d_rowdeg); gbx_free(a->d_state_init);
  free(a->h_chains);
  free(a);
}

/* CTAs of a cluster for every chain, or 0 for teams in a cooperative launch.  A
 * cluster's barrier takes 0.6 us, the one in global memory 2.4; but a level
 * on fewer CTAs takes longer than that saves, so a cluster has at least 7/8 of
 * the grid's share of a chain (`range` CTAs) or a lane per thread (`lanes` in
 * all), and every chain's runs at once.  Measured on GB300, teams against
 * clusters, us a step: 32 chains of n = 300, d = 6: 14.7 / 11.8; 25 of n = 700,
 * d = 16: 17.8 / 16.3; 16 of n = 1024, d = 8: 16.0 / 15.1 (13 CTAs); 4 of them:
 * 16 / 12.  With too few CTAs, 16 of n = 2048, d = 8: 34 / 39 (13 of 19). */
static int resident_cluster(const ODPX_Anneal *a, int range, long long lanes, size_t *smem_out)
{
  const odp_plan *p = a->p;
  const long long enough = (lanes + GBX_RESIDENT_CLUSTER_THREADS - 1) / GBX_RESIDENT_CLUSTER_THREADS;
  const long long want = (lanes + GBX_RESIDENT_THREADS - 1) / GBX_RESIDENT_THREADS;
  const int share = (range * 7 + 7) / 8, least = enough < share ? (int)enough : share;
  for(int c = want < range ? (int)want : range; c >= least && c >= 2; c--){
    size_t smem = 0;
    int active = 0;
    if(c > GBX_RESIDENT_CLUSTER) continue;
    for(int i = 0; i < a->count; i++){
      const odp_plan_graph *g = &p->g[i];
      const size_t s = gbx_resident_smem((g->n + c - 1) / c, g->dp, g->B, g->d);
      if(s > smem) smem = s;
    }
    if(gbx_resident_clusters(c, smem, &active) == 0 && active >= a->count){
      *smem_out = smem;
      return c;
    }
  }
  return 0;
}

/* Whether every chain fits the resident kernel: 16-bit vertices, and the
 * compact adjacency beside a CTA's share of the rows in shared memory.  The
 * teams share two CTAs per SM, or one where two do not fit; a part of the GPU
 * (ODP_GB300_BLOCKS, in engine CTAs, four per SM) becomes the same part of
 * them.  Measured on GB300 against four launches per step (us): 16 chains of
 * n = 1024, d = 8: 14.5 / 70; one of them: 11.4 / 49; 8 of n = 4096, d = 16: 75 /
 * 141; 32 of n = 300, d = 6: 12 / 64.  With few CTAs for large graphs the
 * engine's four CTAs per SM are faster: 16 chains on a quarter of the GPU, n =
 * 2048, d = 16 (32 lanes a thread) 116 / 132, n = 3000, d = 12 (70) 360 / 270, n
 * = 4096, d = 8 (128) 466 / 348.  Allocates its memory; 0 if the chains do not
 * fit. */
static int plan_resident(ODPX_Anneal *a, int blocks)
{
  const odp_plan *p = a->p;
  const int sms = gbx_engine_blocks(0) / 4;
  if(env_resident() == 0 || sms < 1) return 0;
  for(int per_sm = 2; per_sm >= 1; per_sm--){
    int grid = blocks > 0 ? blocks * per_sm / 4 : sms * per_sm, fit = 0;
    if(grid < 1) grid = 1;
    if(grid > sms * per_sm) grid = sms * per_sm;
    const int teams = a->count < grid ? a->count : grid, range = grid / teams;
    size_t smem = 0;
    unsigned long long words = 0, ints = 0;
    long long most = 1;
    for(int i = 0; i < a->count; i++){
      const odp_plan_graph *g = &p->g[i];
      const long long lanes = (g->B + 255) / 256, want = ((long long)g->n * lanes + 255) / 256;
      const int size = range < want ? range : (int)want;
      const size_t s = gbx_resident_smem((g->n + size - 1) / size, g->dp, g->B, g->d);
      if(g->n > 65535 || lanes > 256 || (long long)g->n * lanes > RESIDENT_LANES * 256ll * size) return 0;
      if(s > smem) smem = s;
      if(g->n * lanes > most) most = g->n * lanes;
      words += 8ull * (unsigned long long)g->n * (unsigned long long)lanes;   /* two buffers, 4 words a lane */
      ints += 2ull * (unsigned long long)g->B * (unsigned long long)g->d;
    }
    if(gbx_resident_blocks(smem, &fit) || fit < per_sm) continue;
    a->res_cluster = resident_cluster(a, range, most, &smem);
    const size_t sync = gbx_resident_sync_bytes() * (size_t)teams, offs = (sizeof(unsigned long long) * (size_t)a->count + 255) & ~(size_t)255;
    unsigned long long *off = calloc(1, 2 * offs), at = 0, to = 0;
    if(!off || (!a->h_late && gbx_host_alloc((void **)&a->h_late, sizeof(unsigned int))) ||
       gbx_host_device_ptr(a->h_late, (void **)&a->res.late) || gbx_malloc(&a->d_res, sync + 2 * offs + 8 * words)){
      free(off);
      a->d_res = NULL;
      return 0;
    }
    for(int i = 0; i < a->count; i++){
      off[i] = to;
      off[offs / sizeof(off[0]) + (size_t)i] = at;
      at += 64ull * (unsigned long long)p->g[i].n * (unsigned long long)((p->g[i].B + 255) / 256);
      to += 2ull * (unsigned long long)p->g[i].B * (unsigned long long)p->g[i].d;
    }
    *a->h_late = 0;
    a->res.chains = a->d_chains;
    a->res.sync = a->d_res;
    a->res.host_offset = (const unsigned long long *)((char *)a->d_res + sync);
    a->res.buf_offset = (const unsigned long long *)((char *)a->d_res + sync + offs);
    a->res.buf = (char *)a->d_res + sync + 2 * offs;
    a->res.limit_ns = p->spin_limit_ns;
    a->res.count = a->count;
    a->res.teams = teams;
    a->res_blocks = a->res_cluster ? teams * a->res_cluster : grid;
    a->res_smem = smem;
    const size_t recs = sizeof(gbx_chain) * (size_t)a->count;
    if(recs + sizeof(int) * ints <= RESIDENT_HOST && gbx_host_alloc((void **)&a->h_res, recs + sizeof(int) * ints) == 0 &&
       gbx_host_device_ptr(a->h_res, (void **)&a->dh_chains) == 0)
      a->res.host_graphs = (int *)((char *)a->dh_chains + recs);
    const int e = gbx_memcpy_h2d((char *)a->d_res + sync, off, 2 * offs, p->stream) || gbx_stream_sync(p->stream);
    a->h_offset = off;
    return !e;
  }
  return 0;
}

#define CK(call) do{ if(call){ rc = ODPX_ERR_CUDA; goto fail; } }while(0)

int ODPX_Anneal_create(const ODPX_Chain *chains, int count, ODPX_Anneal **out)
{
  if(!out || !chains || count <= 0) return ODPX_ERR_INVALID;
  *out = NULL;
  for(int i = 0; i < count; i++){
    int e = check_chain(&chains[i]);
    if(e) return e;
  }
  if(odp_device_ready()) return ODPX_ERR_CUDA;
  int rc = 0;
  ODPX_Anneal *a = calloc(1, sizeof(ODPX_Anneal));
  odp_shape *shapes = calloc((size_t)count, sizeof(odp_shape));
  const int **adj = calloc((size_t)count, sizeof(int *));
  odp_result *res = calloc((size_t)count, sizeof(odp_result));
  if(!a || !shapes || !adj || !res){ rc = ODPX_ERR_MEMORY; goto fail; }
  a->count = count;
  for(int i = 0; i < count; i++){
    shapes[i].grid = chains[i].grid != 0;
    shapes[i].nodes = chain_nodes(&chains[i]);
    shapes[i].width = chains[i].width;
    shapes[i].height = chains[i].height;
    shapes[i].degree = chains[i].degree;
    shapes[i].symmetries = chains[i].symmetries;
    shapes[i].num_degrees = chains[i].num_degrees;
    adj[i] = chains[i].adjacency;
  }
  odp_tuning t;
  odp_tuning_defaults(&t, count > 1);
  t.reorder = 0;                      /* the job order is fixed once the steps run on the device */
  t.direct = 0;                       /* the chains update the plan's device copy of the adjacency */
  /* Chain groups run side by side on parts of the GPU.  The small-graph
   * kernel's CTAs (512 threads, up to 200 KB of shared memory) do not fit on
   * SMs that hold other groups' engine CTAs: with four groups on four
   * streams, 1024-vertex chains ran at 52k instead of 121k evals/s. */
  t.small_n = 0;
  t.sweep = 0;                        /* a step's evaluation is enqueued between its other kernels */
  if((rc = odp_plan_create(shapes, count, &t, &a->p))) goto fail;
  odp_plan *p = a->p;
  /* the starting graphs' evaluation; it also uploads and expands them */
  if((rc = odp_plan_run(p, adj, res))) goto fail;

  size_t best_ints = 0, deg_ints = 0;
  for(int i = 0; i < count; i++){
    best_ints += ((size_t)p->g[i].B * p->g[i].d + 3) & ~(size_t)3;   /* 16-byte aligned copies */
    if(chains[i].num_degrees) deg_ints += (size_t)p->g[i].B;
  }
  CK(gbx_malloc((void **)&a->d_best, sizeof(int) * (best_ints ? best_ints : 1)));
  if(deg_ints) CK(gbx_malloc((void **)&a->d_rowdeg, sizeof(int) * deg_ints));
  CK(gbx_malloc((void **)&a->d_state_init, p->state_bytes));
  CK(gbx_malloc((void **)&a->d_chains, sizeof(gbx_chain) * (size_t)count));
  a->h_chains = calloc((size_t)count, sizeof(gbx_chain));
  if(!a->h_chains){ rc = ODPX_ERR_MEMORY; goto fail; }

  size_t boff = 0, doff = 0;
  for(int i = 0; i < count; i++){
    const ODPX_Chain *in = &chains[i];
    const odp_plan_graph *g = &p->g[i];
    gbx_chain *c = &a->h_chains[i];
    size_t words = (size_t)g->B * g->d;
    c->n = g->n; c->d = g->d; c->dp = g->dp; c->s = g->s; c->base = g->B; c->graph = i;
    c->grid = in->grid != 0;
    c->width = in->width; c->height = in->height; c->len = in->length;
    c->itable = g->has_itable ? p->d_itable + g->itable_off : NULL;
    c->adj = p->d_adj + g->adj_off;
    c->nbr = p->d_nbr + g->nbr_off;
    c->best_adj = a->d_best + boff;
    CK(gbx_memcpy_h2d(c->best_adj, in->adjacency, sizeof(int) * words, p->stream));
    boff += (words + 3) & ~(size_t)3;
    if(in->num_degrees){
      CK(gbx_memcpy_h2d(a->d_rowdeg + doff, in->num_degrees, sizeof(int) * (size_t)g->B, p->stream));
      c->ndeg = a->d_rowdeg + doff;
      doff += (size_t)g->B;
    }
    odp_rng rng;
    odp_rng_seed(&rng, in->seed);     /* ODP_Srand(seed): no output drawn yet */
    for(int k = 0; k < 31; k++) c->ring[k] = rng.line[k];
    c->ring_pos = 0;
    c->cur_diameter = c->best_diameter = res[i].diameter;
    c->cur_sum = c->best_sum = res[i].sum;
    c->cur_aspl = c->best_aspl = res[i].aspl;
    c->temp = in->hill_climbing ? 0.0 : in->max_temp;
    c->cooling = in->hill_climbing ? 0.0 : pow(in->min_temp / in->max_temp, (double)1.0 / in->ncalcs);
    c->hill_climbing = in->hill_climbing != 0;
    c->aspl_priority = in->aspl_priority != 0;
  }
  CK(gbx_memcpy_h2d(a->d_state_init, p->h_state_init, p->state_bytes, p->stream));
  CK(gbx_memcpy_h2d(a->d_chains, a->h_chains, sizeof(gbx_chain) * (size_t)count, p->stream));
  CK(gbx_stream_sync(p->stream));
  a->resident = plan_resident(a, t.blocks);
  free(shapes); free(adj); free(res);
  *out = a;
  return 0;

fail:
  free(shapes); free(adj); free(res);
  ODPX_Anneal_destroy(a);
  return rc;
}

/* One step in stream order: propose, reset the engine state, evaluate, decide. */
static int enqueue_step(ODPX_Anneal *a)
{
  odp_plan *p = a->p;
  gbx_ctrl *ctrl = (gbx_ctrl *)(p->d_state + p->out_off);
  const unsigned int *err = (const unsigned int *)(p->d_state + p->out_off + sizeof(gbx_ctrl));
  const gbx_graph_acc *acc = (const gbx_graph_acc *)(p->d_state + p->acc_off);
  if(gbx_anneal_propose(a->d_chains, a->count, p->stream)) return ODPX_ERR_CUDA;
  if(gbx_memcpy_d2d(p->d_state, a->d_state_init, p->state_bytes, p->stream)) return ODPX_ERR_CUDA;
  if(odp_plan_enqueue_engine(p)) return ODPX_ERR_CUDA;
  if(gbx_anneal_decide(a->d_chains, a->count, acc, ctrl, err, p->stream)) return ODPX_ERR_CUDA;
  return 0;
}

int ODPX_Anneal_run(ODPX_Anneal *a, int steps)
{
  if(!a || steps < 0) return ODPX_ERR_INVALID;
  odp_plan *p = a->p;
  int s = 0;
  if(a->resident){
    const int host = a->res.host_graphs && steps > 0;
    if(steps > 0) a->h_current = 0;
    for(; s < steps; s += a->res.steps){
      a->res.steps = steps - s < RESIDENT_STEPS ? steps - s : RESIDENT_STEPS;
      a->res.host_chains = host && s + a->res.steps == steps ? a->dh_chains : NULL;
      if((!a->res_cluster &&
          gbx_memset(a->res.sync, 0, gbx_resident_sync_bytes() * (size_t)a->res.teams, p->stream)) ||
         gbx_resident_launch(&a->res, a->res_blocks, a->res_smem, a->res_cluster, p->stream))
        return ODPX_ERR_CUDA;
    }
    if(gbx_stream_sync(p->stream)) return ODPX_ERR_CUDA;
    /* after a wait that ran out the state is read from the device, as that of the stepwise kernels */
    a->h_current |= host && !*a->h_late;
    *a->h_late = 0;
    return 0;
  }
  if(steps >= ANNEAL_GRAPH_STEPS){
    /* full groups of steps replay one captured graph: a launch per group
     * instead of four operations per step */
    if(!a->steps_exec){
      if(gbx_capture_begin(p->stream)) return ODPX_ERR_CUDA;
      int e = 0;
      for(int k = 0; k < ANNEAL_GRAPH_STEPS && !e; k++) e = enqueue_step(a);
      void *ge = NULL;
      int e2 = gbx_capture_end(p->stream, &ge);
      if(e || e2) return ODPX_ERR_CUDA;
      a->steps_exec = ge;
    }
    for(; s + ANNEAL_GRAPH_STEPS <= steps; s += ANNEAL_GRAPH_STEPS)
      if(gbx_graph_launch(a->steps_exec, p->stream)) return ODPX_ERR_CUDA;
  }
  for(; s < steps; s++)
    if(enqueue_step(a)) return ODPX_ERR_CUDA;
  return gbx_stream_sync(p->stream) ? ODPX_ERR_CUDA : 0;
}

void ODPX_Anneal_set_wait_limit(ODPX_Anneal *a, unsigned long long ns)
{
  if(!a || a->p->spin_limit_ns == ns) return;
  a->p->spin_limit_ns = ns;
  a->res.limit_ns = ns;
  /* the limit is an argument of the captured engine launches: capture anew */
  if(a->steps_exec){
    gbx_stream_sync(a->p->stream);
    gbx_graph_destroy(a->steps_exec);
    a->steps_exec = NULL;
  }
}

static void fill_state(const gbx_chain *c, ODPX_Chain_state *st)
{
  if(!st) return;
  st->steps = c->steps;
  st->accepted = c->accepted;
  st->status = c->status;
  st->diameter = c->cur_diameter;
  st->sum = (long)c->cur_sum;
  st->aspl = c->cur_aspl;
  st->best_diameter = c->best_diameter;
  st->best_sum = (long)c->best_sum;
  st->best_aspl = c->best_aspl;
  st->temp = c->temp;
}

int ODPX_Anneal_state(ODPX_Anneal *a, int chain, ODPX_Chain_state *st, int *adjacency, int *best_adjacency)
{
  if(!a || chain < 0 || chain >= a->count) return ODPX_ERR_INVALID;
  odp_plan *p = a->p;
  gbx_chain *c = &a->h_chains[chain];
  if(a->h_current){
    const gbx_chain *now = (const gbx_chain *)a->h_res + chain;
    const int *graphs = (const int *)((const gbx_chain *)a->h_res + a->count) + a->h_offset[chain];
    const size_t ints = (size_t)now->base * now->d;
    *c = *now;
    if(adjacency) memcpy(adjacency, graphs, sizeof(int) * ints);
    if(best_adjacency) memcpy(best_adjacency, graphs + ints, sizeof(int) * ints);
    fill_state(c, st);
    return 0;
  }
  if(gbx_memcpy_d2h(c, a->d_chains + chain, sizeof(gbx_chain), p->stream)) return ODPX_ERR_CUDA;
  size_t words = (size_t)c->base * c->d;
  if(adjacency && gbx_memcpy_d2h(adjacency, c->adj, sizeof(int) * words, p->stream)) return ODPX_ERR_CUDA;
  if(best_adjacency && gbx_memcpy_d2h(best_adjacency, c->best_adj, sizeof(int) * words, p->stream))
    return ODPX_ERR_CUDA;
  if(gbx_stream_sync(p->stream)) return ODPX_ERR_CUDA;
  fill_state(c, st);
  return 0;
}
