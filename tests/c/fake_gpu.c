/*
 * fake_gpu.c -- the CUDA layer (csrc/odp_engine.h) without a GPU, for tests of
 * the host runtime: device memory is host memory, every operation completes at
 * once, and a launch only reports an outcome.  fake_fail says how the launch
 * with that number behaves.
 */
#include <stdlib.h>
#include <string.h>
#include "odp_engine.h"

enum { ENGINE, SMALL, SWEEP, TEAM, RESIDENT, STEP, PULL, KINDS };
int fake_launches[KINDS];
int fake_total;                /* launches of the evaluation kernels so far */
int fake_abort_at;             /* that launch (from 1): a wait runs out, no record is written */
int fake_late_at;              /* that launch: complete, and then a wait runs out all the same */
const int *fake_adjacency;     /* of the last lockstep launch */
int fake_pending;              /* events are not complete while set */
int fake_pending_from;         /* nor from that launch on */

static int next(int kind)
{
  fake_launches[kind]++;
  return ++fake_total;
}

int gbx_device_init(int *sms){ if(sms) *sms = 152; return 0; }
int gbx_malloc(void **p, size_t n){ *p = calloc(1, n ? n : 256); return *p ? 0 : 2; }
int gbx_mem_free(size_t *n){ *n = (size_t)64 << 30; return 0; }
int gbx_free(void *p){ free(p); return 0; }
int gbx_host_alloc(void **p, size_t n){ return gbx_malloc(p, n); }
int gbx_host_free(void *p){ free(p); return 0; }
int gbx_stream_create(void **s){ *s = malloc(1); return 0; }
int gbx_stream_destroy(void *s){ free(s); return 0; }
int gbx_memcpy_h2d(void *d, const void *s, size_t n, void *st){ (void)st; memmove(d, s, n); return 0; }
int gbx_memcpy_d2h(void *d, const void *s, size_t n, void *st){ (void)st; memmove(d, s, n); return 0; }
int gbx_memcpy_d2d(void *d, const void *s, size_t n, void *st){ (void)st; memmove(d, s, n); return 0; }
int gbx_memset(void *d, int v, size_t n, void *st){ (void)st; memset(d, v, n); return 0; }
int gbx_stream_sync(void *s){ (void)s; return 0; }
const char *gbx_error_string(int e){ (void)e; return ""; }
int gbx_expand(const gbx_expand_desc *d, int n, long long v, int dp, unsigned *e, void *s)
{ (void)d; (void)n; (void)v; (void)dp; (void)e; (void)s; return 0; }
int gbx_engine_blocks(int active){ (void)active; return 608; }
int gbx_pageable_access(void){ return 1; }
int gbx_l2_read_probe(size_t b, int r, double *g){ (void)b; (void)r; *g = 0; return 0; }
int gbx_host_device_ptr(void *h, void **d){ *d = h; return 0; }
int gbx_small_prepare(void){ return 0; }
int gbx_small_clusters(int c, int t, size_t m, int *a){ (void)t; (void)m; *a = 144 / c; return 0; }
int gbx_scatter(const gbx_write *w, int n, void *s)
{ (void)s; for(int i = 0; i < n; i++) *w[i].at = w[i].value; return 0; }
int gbx_event_create(void **e){ *e = malloc(1); return 0; }
int gbx_event_destroy(void *e){ free(e); return 0; }
int gbx_event_record(void *e, void *s){ (void)e; (void)s; return 0; }
int gbx_event_query(void *e)
{
  (void)e;
  const int from = __atomic_load_n(&fake_pending_from, __ATOMIC_ACQUIRE);
  return __atomic_load_n(&fake_pending, __ATOMIC_ACQUIRE) || (from && fake_total >= from);
}
int gbx_event_elapsed_ms(void *a, void *b, float *ms){ (void)a; (void)b; *ms = 1.0f; return 0; }
int gbx_capture_begin(void *s){ (void)s; return 1; }       /* plans are created with use_graph off */
int gbx_capture_end(void *s, void **g){ (void)s; *g = NULL; return 1; }
int gbx_graph_launch(void *g, void *s){ (void)g; (void)s; return 1; }
int gbx_graph_destroy(void *g){ (void)g; return 0; }

int gbx_pull(const gbx_expand_desc *h, gbx_expand_desc *d, int n, void *st, const void *init, size_t bytes, void *s)
{
  (void)s;
  fake_launches[PULL]++;
  memcpy(d, h, sizeof(*h) * (size_t)n);
  if(bytes) memcpy(st, init, bytes);
  return 0;
}

int gbx_engine_launch(const gbx_job *j, int nj, gbx_slot *sl, int ns, gbx_ctrl *c, gbx_graph_acc *acc, gbx_job_out *o,
                      unsigned long long limit, int blocks, int active, void *s)
{
  (void)sl; (void)ns; (void)limit; (void)blocks; (void)active; (void)s;
  for(int i = 0; i < nj; i++){
    o[i].level = 1;
    acc[j[i].graph].levels = 1;
  }
  if(next(ENGINE) == fake_abort_at) c->error = GBX_ERR_TIMEOUT;
  return 0;
}

static void record(gbx_small_rec *r, int n, unsigned seq)
{
  for(int i = 0; i < n; i++){
    memset(&r[i], 0, sizeof(r[i]));
    r[i].level = 1;
    r[i].err = seq << 8;
  }
}

int gbx_small_launch(const gbx_job *j, int nj, const gbx_expand_desc *d, const gbx_expand_desc *d0, gbx_small_rec *r,
                     unsigned seq, size_t m, int c, int t, int p, void *s)
{
  (void)j; (void)d; (void)d0; (void)m; (void)c; (void)t; (void)p; (void)s;
  next(SMALL);
  record(r, nj, seq);
  return 0;
}

size_t gbx_sweep_sync_bytes(void){ return 65536; }
int fake_asked;                /* gbx_sweep_smem calls */
size_t gbx_sweep_smem(const gbx_sweep *a){ fake_asked++; return (size_t)a->rows * (size_t)a->e.dp * 4 + 8192; }
int gbx_sweep_blocks(const gbx_sweep *a, int *per_sm){ *per_sm = gbx_sweep_smem(a) <= 56000 ? 4 : gbx_sweep_smem(a) <= 200000 ? 1 : 0; return 0; }
int gbx_sweep_launch(const gbx_sweep *a, int blocks, void *s)
{
  (void)blocks; (void)s;
  const int k = next(SWEEP);
  fake_adjacency = a->e.adj;
  if(k != fake_abort_at) record(a->rec, a->nchunks, a->seq);
  if(k == fake_abort_at || k == fake_late_at) *a->abort_flag = GBX_ERR_TIMEOUT;
  return 0;
}

size_t gbx_team_node_bytes(void){ return 4096; }
int gbx_team_blocks(size_t m, int *per_sm){ (void)m; *per_sm = 2; return 0; }
int gbx_team_launch(const gbx_team *t, int blocks, size_t m, void *s)
{
  (void)blocks; (void)m; (void)s;
  const int k = next(TEAM);
  if(k != fake_abort_at)
    for(int i = 0; i < t->queue[GBX_TEAM_SPLITS]; i++) record(t->graphs[i].rec, t->graphs[i].nchunks, t->graphs[i].seq);
  if(k == fake_abort_at) *t->abort_flag = GBX_ERR_TIMEOUT;
  return 0;
}

int gbx_anneal_propose(gbx_chain *c, int n, void *s){ (void)c; (void)n; (void)s; fake_launches[STEP]++; return 0; }
int gbx_anneal_decide(gbx_chain *c, int n, const gbx_graph_acc *a, const gbx_ctrl *t, const unsigned *e, void *s)
{ (void)c; (void)n; (void)a; (void)t; (void)e; (void)s; return 0; }
size_t gbx_resident_sync_bytes(void){ return 1024; }
size_t gbx_resident_smem(int rows, int dp, int base, int d){ return (size_t)rows * (size_t)dp * 4 + (size_t)base * (size_t)d * 2; }
int gbx_resident_blocks(size_t m, int *per_sm){ *per_sm = m <= 100000 ? 2 : m <= 200000 ? 1 : 0; return 0; }
int gbx_resident_clusters(int c, size_t m, int *a){ (void)c; (void)m; *a = 0; return 0; }
int gbx_resident_launch(const gbx_resident *r, int blocks, size_t m, int cluster, void *s)
{ (void)r; (void)blocks; (void)m; (void)cluster; (void)s; fake_launches[RESIDENT]++; return 0; }
