// cf_solve.cu -- the host side of one fused solve in one call: both pool tables and the screen
// table prepared into page-locked memory, one upload, the table join (tail tables, build, probe) or
// the class join queued behind it, the pair check, and the read-back of the counters and first
// results.  A campaign runs thousands of solves of 0.1 to 1 ms of device time each; table by table
// from Python a solve took 0.2 to 0.4 ms of host time, which was then the whole solve.
#include <string.h>
#include "cf_abi_internal.h"

extern "C" size_t cf_pool_bytes(int n, int r);
extern "C" int cf_pool_prepare_split(const u64* primes, int n, int r, u64 m, int a, u64 mult_odd, u64 mult2, void* out,
                                     size_t out_bytes);
extern "C" size_t cf_screen_bytes(void);
extern "C" int cf_screen_prepare(const u32* limbsB, int nlimbs, double lgP0, double lgB, double eps, void* out,
                                 size_t out_bytes);
extern "C" size_t cf_tail_bytes(int n, int r);
extern "C" int cf_build_tail(const void* pool_dev, int n, int r, void* tail, void* stream);
extern "C" size_t cf_dtab_bytes2(int bbits, int fbits);
extern "C" int cf_dtab_build3(const void* pool_dev, const void* tail, int n, int r, u64 lo, u64 count, void* tab,
                              int bbits, int fbits, int side_format, u32* err, void* stream);
extern "C" int cf_fused_probe3(const void* pool_dev, const void* tail, int n, int r, u64 lo, u64 count,
                               const void* tab, int bbits, int fbits, int side_format, u64 tab_rank0, int swap,
                               void* pairs, u32 max_pairs, u32* npairs, u32* err, u32 grid, void* stream);
extern "C" int cf_class_join(const void* plan, const void* poolD, const void* poolI, u32 multD_m, u32 multD_d,
                             void* ws, size_t ws_bytes, void* pairs, u32 max_pairs, u32* npairs, u32* err,
                             void* ev_built, void* stream);
bool cf_class_plan_fits(const void* plan, u64 m, int nD, int nI, int r, u64 i_lo, u64 i_n, int swap);
extern "C" size_t cf_pair_result_bytes(void);
extern "C" int cf_check_pairs(const void* poolD, const void* poolI, const void* screen, int r, const void* pairs,
                              const u32* npairs, u32 max_pairs, void* results, u32* err, void* stream);

// The same layout is declared in include/cfmitm.h; keep the two in step.
struct CfSolve {
  const u64 *primesD, *primesI;        // host, ascending
  u64 m;                               // odd part of M
  u64 multD_odd, multD_2;              // (prod B0)^-1 mod m and mod 2^a
  u64 n_D, i_lo, n_I;                  // records of the D side; window of the I side
  const u32* limbsB;                   // size bound, 32-bit limbs
  double lgP0, lgB, eps;
  const void* class_plan;              // host plan of cf_class_plan, or null: table join
  void* stage;                         // page-locked, cf_solve_table_bytes; unchanged until the solve has run
  void* tables;                        // device, as many bytes, 256-byte aligned
  void* tails;                         // device, 256-byte aligned: both tail tables (table join)
  void* ws;                            // device: class workspace, or the D table
  u64 tails_bytes, ws_bytes;
  void *pairs, *results, *misc;        // device: max_pairs pairs and results, 64 bytes of counters
  void* readback;                      // page-locked: 8 bytes of counters, then `rows` results; or null
  void* events[4];                     // CUDA events: before, after the build, the probe, the check; or null
  u32 multD_mp, multD_d;               // (prod B0)^-1 mod the class plan's mp and d
  u32 max_pairs, rows, fused_grid;
  int nlimbs, nD, nI, r, a, swap, bbits, fbits, side_format;
};

static size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

extern "C" size_t cf_solve_desc_bytes(void) { return sizeof(CfSolve); }

// Bytes of the tables of one solve (both pool tables and the screen table).
extern "C" size_t cf_solve_table_bytes(int nD, int nI, int r) {
  const size_t d = cf_pool_bytes(nD, r), i = cf_pool_bytes(nI, r);
  return d && i ? up256(d) + up256(i) + up256(cf_screen_bytes()) : 0;
}

// Bytes of both tail tables (table join).
extern "C" size_t cf_solve_tail_bytes(int nD, int nI, int r) {
  return up256(cf_tail_bytes(nD, r) + 16) + up256(cf_tail_bytes(nI, r) + 16);
}

static int mark(void* ev, cudaStream_t st) {
  return ev ? cf_cuda_status(cudaEventRecord((cudaEvent_t)ev, st), "cf_solve: event") : CF_OK;
}

// Queue one solve on the stream (see the top of the file); nothing is waited for.  The results are
// in s->results / s->readback when the stream has run: {npairs, err} and the checked rows.
extern "C" int cf_solve(const CfSolve* s, void* stream) {
  if (!s || !s->primesD || !s->primesI || !s->limbsB || !s->stage || !s->tables || !s->ws || !s->misc ||
      (s->max_pairs && (!s->pairs || !s->results)) || (!s->class_plan && !s->tails) ||
      cf_solve_table_bytes(s->nD, s->nI, s->r) == 0 ||
      (!s->class_plan && (s->tails_bytes < cf_solve_tail_bytes(s->nD, s->nI, s->r) ||
                          s->ws_bytes < cf_dtab_bytes2(s->bbits, s->fbits) || !cf_dtab_bytes2(s->bbits, s->fbits)))) {
    cf_set_error("cf_solve: bad arguments%s", "");
    return CF_EBADARG;
  }
  // a plan of other sides would index the pools past their ends
  if (s->class_plan && !cf_class_plan_fits(s->class_plan, s->m, s->nD, s->nI, s->r, s->i_lo, s->n_I, s->swap)) {
    cf_set_error("cf_solve: the class plan is of another instance or window%s", "");
    return CF_EBADARG;
  }
  if (s->class_plan && ((s->primesD[s->nD - 1] | s->primesI[s->nI - 1]) >> 31)) {   // 32-bit factors in its kernels
    cf_set_error("cf_solve: the class join takes primes below 2^31%s", "");
    return CF_EBADARG;
  }
  const cudaStream_t st = (cudaStream_t)stream;
  const int r = s->r;
  const size_t bD = up256(cf_pool_bytes(s->nD, r)), bI = up256(cf_pool_bytes(s->nI, r));
  const size_t total = cf_solve_table_bytes(s->nD, s->nI, r);
  unsigned char *h = (unsigned char*)s->stage, *d = (unsigned char*)s->tables;
  // a table prepared from the modulus's parts equals the one prepared from M where M is below 2^64
  int rc = cf_pool_prepare_split(s->primesD, s->nD, r, s->m, s->a, s->multD_odd, s->multD_2, h, bD);
  if (rc == CF_OK) rc = cf_pool_prepare_split(s->primesI, s->nI, r, s->m, s->a, 1, s->a ? 1 : 0, h + bD, bI);
  if (rc == CF_OK) rc = cf_screen_prepare(s->limbsB, s->nlimbs, s->lgP0, s->lgB, s->eps, h + bD + bI, cf_screen_bytes());
  if (rc != CF_OK) return rc;
  u32* misc = (u32*)s->misc;
  cudaError_t e = cudaMemcpyAsync(d, h, total, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(misc, 0, 64, st);
  if (e != cudaSuccess) return cf_cuda_status(e, "cf_solve: tables");
  void *poolD = d, *poolI = d + bD, *screen = d + bD + bI;
  if ((rc = mark(s->events[0], st)) != CF_OK) return rc;
  if (s->class_plan) {
    rc = cf_class_join(s->class_plan, poolD, poolI, s->multD_mp, s->multD_d, s->ws, s->ws_bytes, s->pairs, s->max_pairs,
                       misc, misc + 1, s->events[1], stream);
    if (rc != CF_OK) return rc;
  } else {
    unsigned char* t = (unsigned char*)s->tails;
    void *tailD = t, *tailI = t + up256(cf_tail_bytes(s->nD, r) + 16);
    unsigned char* tab = (unsigned char*)s->ws;
    const size_t nb = (size_t)1 << s->bbits, tb = cf_dtab_bytes2(s->bbits, s->fbits);
    e = cudaMemsetAsync(tab, 0, 32 * nb, st);                           // fingerprint sectors
    if (e == cudaSuccess) e = cudaMemsetAsync(tab + 160 * nb, 0, tb - 160 * nb, st);   // fill counters, Bloom filter
    if (e != cudaSuccess) return cf_cuda_status(e, "cf_solve: table");
    rc = cf_build_tail(poolD, s->nD, r, tailD, stream);
    if (rc == CF_OK) rc = cf_build_tail(poolI, s->nI, r, tailI, stream);
    // build on the smaller side (swap: the table holds the I window and the D side probes)
    if (rc == CF_OK)
      rc = s->swap ? cf_dtab_build3(poolI, tailI, s->nI, r, s->i_lo, s->n_I, tab, s->bbits, s->fbits, s->side_format,
                                    misc + 1, stream)
                   : cf_dtab_build3(poolD, tailD, s->nD, r, 0, s->n_D, tab, s->bbits, s->fbits, s->side_format, misc + 1,
                                    stream);
    if (rc != CF_OK) return rc;
    if ((rc = mark(s->events[1], st)) != CF_OK) return rc;
    rc = s->swap ? cf_fused_probe3(poolD, tailD, s->nD, r, 0, s->n_D, tab, s->bbits, s->fbits, s->side_format, s->i_lo, 1,
                                   s->pairs, s->max_pairs, misc, misc + 1, s->fused_grid, stream)
                 : cf_fused_probe3(poolI, tailI, s->nI, r, s->i_lo, s->n_I, tab, s->bbits, s->fbits, s->side_format, 0, 0,
                                   s->pairs, s->max_pairs, misc, misc + 1, s->fused_grid, stream);
    if (rc != CF_OK) return rc;
  }
  if ((rc = mark(s->events[2], st)) != CF_OK) return rc;
  rc = cf_check_pairs(poolD, poolI, screen, r, s->pairs, misc, s->max_pairs, s->results, misc + 1, stream);
  if (rc != CF_OK) return rc;
  if ((rc = mark(s->events[3], st)) != CF_OK) return rc;
  if (s->readback) {
    e = cudaMemcpyAsync(s->readback, misc, 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && s->rows)
      e = cudaMemcpyAsync((unsigned char*)s->readback + 8, s->results,
                          (size_t)(s->rows < s->max_pairs ? s->rows : s->max_pairs) * cf_pair_result_bytes(),
                          cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return cf_cuda_status(e, "cf_solve: read-back");
  }
  return CF_OK;
}
