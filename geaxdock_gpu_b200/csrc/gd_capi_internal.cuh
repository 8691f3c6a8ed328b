/*
 * gd_capi_internal.cuh -- what the host-side units of the C ABI share: the context (gd_ctx),
 * the per-complex bookkeeping, the error reporting, and the launch and buffer helpers.
 *
 *   gd_capi.cu          the context, its uploads and tile lists, the Monte Carlo calls,
 *                       records and state (the reference's Run and launcher, src/run.cu:33-288,
 *                       src/kernel_cuda_lancher_siglegpu.cu)
 *   gd_capi_layout.cu   the device layout of one complex
 *   gd_pocket.cu        the pocket grid's point lists of the short-range terms
 *   gd_farfield.cu      the far points of large proteins as fields over the pocket grid
 *   gd_capi_tile.cu     the tile, its autotuning, chains, RNG streams and the wait bound
 *   gd_capi_stream.cu   records downloaded while the run proceeds (gd_records_stream)
 *   gd_capi_eval.cu     pose energies, placed coordinates and the energy trace
 *   gd_capi_noalloc.cu  pose energies without allocation (gd_eval_energy_noalloc)
 *   gd_capi_da.cu       the surrogate, delayed acceptance and its fallback controller, the
 *                       standalone network and k-means entry points
 */
#ifndef GD_CAPI_INTERNAL_CUH
#define GD_CAPI_INTERNAL_CUH

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <condition_variable>
#include <deque>
#include <limits>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "gd_device.cuh"
#include "gd_kmeans.cuh"
#include "gd_mlp.cuh"
#include "gd_numerics.h"

namespace gd {
template <int UNROLL, int SPLITS, int KIND, int PACK>
__global__ void gd_mc_kernel(GdMcArgs a, GdForceConst f);
#define GD_EXT(U, S, K, P) \
  extern template __global__ void gd_mc_kernel<U, S, K, P>(GdMcArgs, GdForceConst);
GD_EXT(1, 0, 0, 1) GD_EXT(2, 0, 0, 1) GD_EXT(4, 0, 0, 1)
GD_EXT(1, 1, 0, 1) GD_EXT(2, 1, 0, 1) GD_EXT(4, 1, 0, 1)
GD_EXT(1, 0, 1, 1) GD_EXT(2, 0, 1, 1) GD_EXT(4, 0, 1, 1)
GD_EXT(1, 1, 1, 1) GD_EXT(2, 1, 1, 1) GD_EXT(4, 1, 1, 1)
GD_EXT(4, 2, 0, 1) GD_EXT(4, 2, 1, 1)
GD_EXT(1, 0, 0, 2) GD_EXT(2, 0, 0, 2)
GD_EXT(2, 0, 2, 1)
#undef GD_EXT
__global__ void gd_exchange_kernel(const GdDevComplex *cxs, const int *group_base, int n_complex,
                                   int g_begin, int g_end, GdExchange ex, GdForceConst f,
                                   const int *call_base, int call_off, int mode_t, int *open,
                                   int *open_list, unsigned *err);
__global__ void gd_reset_records_kernel(int *rec_next, int r0, int r1);
}  // namespace gd

namespace gdc {

/* the calling thread's last error message (gd_last_error_string) */
extern thread_local std::string g_err;
/* records a formatted message and returns code */
int fail(int code, const char *fmt, ...);

#define CK(call)                                                                     \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess)                                                           \
      return fail(GD_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), \
                  __FILE__, __LINE__);                                               \
  } while (0)

constexpr float kPi = 3.1415926535f; /* reference src/size.h:67 */

float contact_threshold(float pmf0);
/* Distance beyond which the pair loop's far form gives its full form's result. */
double pmf_far_radius(float pmf0);
float bits_as_float(int v);
float host_dist2(float ax, float ay, float az, float px, float py, float pz);

struct ComplexInfo {
  int n_lig, n_prt, n_tmp, lna, pnp, pnp_pad, pnk, pos;
  int rep_offset, n_rep, k;
  int stream;
  /* stored pieces of a split launch whose sums run in the points' order, by split count */
  int pieces[GD_MAX_SPLITS + 1], hpieces[GD_MAX_SPLITS + 1];
  int types_uniform; /* every ligand conformer has the same atom types (two replicas per
                        thread share their atom's pair parameters) */
};

/* The shape of one launch of the Monte Carlo kernel: lanes per CTA (pack lanes per thread), points
 * per ring buffer and per FP32 sum (fold), splits per atom, point pairs in flight, the largest
 * replica count of a tile, and the pieces of sums in the points' order (0: sums per split). */
struct LaunchShape {
  int lanes, chunk, fold, split, unroll, pack, kmax;
  int pieces = 0, hpieces = 0; /* GdMcArgs */
};

/* One chain of the fused loops: a contiguous range of (complex, protein conformer) blocks,
 * their replicas, exchange groups and tiles. Chains share nothing, so the graph runs them on
 * separate streams and one chain's kernels fill the other's tail. */
struct Chain {
  int g0, g1;    /* blocks [g0, g1) in (complex, protein conformer) order */
  int r0, r1;    /* replicas */
  int xg0, xg1;  /* exchange groups */
  int t_off, t_cnt; /* plain tiles in the chain tile list */
};

}  // namespace gdc

struct RecStream;
struct RecAsync;
struct DaState;

struct gd_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  gd_mc_params mc{};
  int n_complex = 0, n_rep = 0, n_groups = 0;
  int threads = 256, chunk = GD_CHUNK, fold = GD_CHUNK, unroll = 2, split = 1, num_sms = 148;
  int pieces = 0, hpieces = 0; /* LaunchShape */
  int pack = 1; /* replicas per thread of the plain launches: the tile's lanes (threads) run on
                   threads / pack threads */
  int fill_threads = 0, fill_cap = 0; /* the last gd_set_tile in fill mode (threads > 0) */
  bool tile_auto = true; /* the automatic tile: launches of few lanes are split over more warps */
  gdc::LaunchShape auto_shape{}; /* the automatic tile, and its replicas per CTA by complex */
  std::vector<int> auto_k;
  std::vector<gdc::ComplexInfo> info;
  std::vector<void *> allocs;      /* cudaMalloc'd buffers */
  std::vector<void *> pool_allocs; /* buffers from the device's context pool (ctx_pool) */
  std::vector<void *> field_allocs; /* those of them that hold the far fields' tables */
  size_t field_bytes = 0;
  GdForceConst fc{};
  GdDevComplex *d_cx = nullptr;
  GdPairParam *d_pp = nullptr;
  int *d_group_base = nullptr;
  /* replica state */
  gd_replica *d_replica = nullptr;
  float *d_mm = nullptr;
  gd_energy *d_eold = nullptr;
  float *d_etotal = nullptr;
  int *d_nacc = nullptr, *d_acs = nullptr;
  gd_record_step *d_rec = nullptr;
  int *d_rec_next = nullptr;
  int rec_cap = 0;
  /* work lists */
  GdTileDesc *d_tiles = nullptr;
  int tiles_cap = 0;
  int tiles_r0 = -1, tiles_r1 = -1, tiles_n = 0, tiles_gen = -1, tile_gen = 0;
  std::vector<GdTileDesc> full_tiles;
  int *d_counters = nullptr; /* [counters_cap] persistent-CTA queue heads */
  int counters_cap = 0;
  bool counters_pooled = false; /* d_counters came from ctx_pool */
  int *d_xopen = nullptr;    /* open exchange groups: [GD_MAX_CHAINS][2] counters, [n_groups] list */
  int *d_cursor = nullptr;   /* [2]: step base, exchange call base (graph replays) */
  int *h_cursor = nullptr;   /* pinned staging */
  unsigned *d_err = nullptr;
  bool initialized = false;
  int exchange_calls = 0;
  /* trace */
  float *d_trace_e = nullptr;
  int *d_trace_acc = nullptr;
  int trace_cap = 0, trace_step0 = 0, trace_steps = 0;
  /* graph cache */
  std::map<long long, cudaGraphExec_t> graphs;
  /* pose evaluation scratch */
  void *d_eval_in = nullptr; /* poses, or given coordinates and centres */
  size_t eval_in_cap = 0;    /* bytes */
  gd_energy *d_e_out = nullptr;
  int eval_cap = 0;
  char *h_eval = nullptr;    /* page-locked, GD_EVAL_STAGE bytes, made on first use */
  long long timeout_ns = 2000000000LL;
  /* surrogate and delayed acceptance (gd_sur_create) */
  struct DaState *da = nullptr;
  /* concurrent chains of the fused loops: plain (gd_mc_run_fused) and delayed acceptance */
  int chains = 1, chains_da = 3;
  std::vector<cudaStream_t> aux;             /* streams of chains 1.. */
  cudaEvent_t ev_fork = nullptr;
  std::vector<cudaEvent_t> ev_join;
  std::vector<gdc::Chain> chain;
  int chain_gen = -1;
  GdTileDesc *d_chain_tiles = nullptr;
  int chain_tiles_cap = 0;
  /* record streaming into host memory (gd_records_stream) */
  struct RecStream *rs = nullptr;
  /* a dump window downloaded in the background (gd_get_records_async) */
  struct RecAsync *ra = nullptr;
};

#define GD_MAX_DEVICES 64
#define GD_MAX_CHAINS 16
#define GD_EVAL_STAGE ((size_t)256 << 10) /* bytes of a context's staging buffer */

namespace gdc {

/* ---- the context's helpers (gd_capi.cu) ---- */
cudaError_t d2h_rows(void *dst, size_t hpitch, const void *src, size_t dpitch, size_t width,
                     int n);
/* makes d2h_rows' page-locked staging buffers (once per process) */
void stage_prepare();
/* The device's stream-ordered pool for the buffers gd_create sets up: it keeps freed memory
 * (no release threshold), so gd_destroy returns buffers without unmapping them and the next
 * context of the process reuses them; gd_release_memory trims it. Null if it cannot be made. */
cudaMemPool_t ctx_pool(int device);
/* n elements on the context's device, stream-ordered on its stream (gd_create synchronises
 * the stream before any other stream sees the buffer), freed by gd_destroy */
template <class T>
int dalloc(gd_ctx *c, T **p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  void *q = nullptr;
  cudaMemPool_t pool = ctx_pool(c->device);
  cudaError_t e = pool ? cudaMallocFromPoolAsync(&q, n * sizeof(T), pool, c->stream)
                       : cudaMalloc(&q, n * sizeof(T));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(GD_ERR_NOMEM, "allocation of %zu bytes failed: %s", n * sizeof(T),
                cudaGetErrorString(e));
  }
  (pool ? c->pool_allocs : c->allocs).push_back(q);
  *p = (T *)q;
  return GD_OK;
}

/* frees a buffer of dalloc before the context ends (stream-ordered) */
void dfree(gd_ctx *c, void *p);

/* Gives the far fields' tables back to the driver: every pair runs in the loop from then on. A
 * replica's energy keeps the fields' last digits until its next accepted move. False if there are
 * none. */
bool release_fields(gd_ctx *c);
/* cudaMalloc for a buffer the context needs: the optional tables make room for it */
template <class T>
cudaError_t cmalloc(gd_ctx *c, T **p, size_t bytes) {
  void *q = nullptr;
  cudaError_t e = cudaMalloc(&q, bytes);
  if (e == cudaErrorMemoryAllocation && release_fields(c)) {
    cudaGetLastError();
    e = cudaMalloc(&q, bytes);
  }
  *p = e == cudaSuccess ? static_cast<T *>(q) : nullptr;
  return e;
}

template <class T>
int upload(gd_ctx *c, T **p, const std::vector<T> &v) {
  int rc = dalloc(c, p, v.size());
  if (rc) return rc;
  if (!v.empty()) CK(cudaMemcpyAsync(*p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice,
                                     c->stream));
  return GD_OK;
}
int check_complex(const gd_complex_desc &d, int idx);
int pick_threads(const std::vector<ComplexInfo> &info);
void build_tiles(const gd_ctx *c, int r0, int r1, std::vector<GdTileDesc> &out);
size_t smem_bytes(const LaunchShape &s);
/* the shape of the context's tile */
LaunchShape ctx_shape(const gd_ctx *c);
/* chooses the automatic tile (gd_create) / makes it the context's tile */
void make_auto_tile(gd_ctx *c);
void use_auto_tile(gd_ctx *c);
/* One work list of a launch: n_blocks runs of `block` replicas (a protein conformer's) of an
 * lna-atom ligand, none sharing a tile with another. */
struct WorkList {
  long long n_blocks;
  int block, lna;
};
/* the splits of a launch of these lists (1: none), and the replicas a tile then takes of each */
int auto_split(const gd_ctx *c, const std::vector<WorkList> &w, std::vector<int> *k);
/* A split launch of complex ci (-1: of all): lanes for k replicas of lna atoms, the ring holding the
 * whole protein, sums in the points' order. False where shared memory does not hold their pieces;
 * the shape then has sums per split. */
bool split_shape(const gd_ctx *c, int ci, int split, int k_lna, int kmax, int pnp_pad,
                 LaunchShape *s);
int ensure_counters(gd_ctx *c, int n);
/* the pinned host cursor of the graph launches (made on first use) */
int ensure_cursor(gd_ctx *c);
typedef void (*McKernel)(GdMcArgs, GdForceConst);
/* kind: GD_KIND_* */
McKernel launch_kernel(const LaunchShape &s, int kind = GD_KIND_PLAIN);
int launch_threads(const LaunchShape &s);
int grid_for(gd_ctx *c, int n_tiles, const LaunchShape &s, int kind = GD_KIND_PLAIN);
GdMcArgs base_args(gd_ctx *c);
int set_kernel_attrs(const LaunchShape &s, int kind = GD_KIND_PLAIN);
/* The exchange of groups [ch.xg0, ch.xg1) of chain k after launches of shape s (unless `fused`:
 * those launches did it), and the launch that decides the groups it left open on the pair loop's
 * energies (contexts with far fields). mode_t -1: from the step, as the fused launches take it. */
int launch_exchange(gd_ctx *c, const Chain &ch, int k, const LaunchShape &s, bool fused, int step0,
                    const int *step_base, const int *call_base, int call_off, int mode_t,
                    cudaStream_t st);
/* sets up the second of them before a capture */
int prepare_exchange(const gd_ctx *c, const LaunchShape &s);
void set_open_lists(gd_ctx *c, const Chain &ch, int k, GdMcArgs *a);
/* the next launch on the device sets its kernel's attributes again */
void forget_kernel_attrs(int device);
int launch_mc(gd_ctx *c, GdMcArgs a, const GdTileDesc *d_tiles, int n_tiles, int *counter,
              const LaunchShape &s);
int upload_tiles(gd_ctx *c, int r0, int r1, int *n_out);
int check_range(const gd_ctx *c, int r0, int r1);
/* the status that the device error word stands for */
int device_status(unsigned err);
void build_chains(gd_ctx *c, int want, std::vector<Chain> &ch, std::vector<GdTileDesc> *tiles);
int ensure_chain_streams(gd_ctx *c, int n);
int ensure_chains(gd_ctx *c);
cudaStream_t chain_stream(gd_ctx *c, int k);
void chains_fork(gd_ctx *c, int n);
void chains_join(gd_ctx *c, int n);
void drop_graphs(gd_ctx *c);

/* ---- pose evaluation (gd_capi_eval.cu) ---- */
/* the launch shape and replicas per CTA of an evaluation of n poses of complex ci */
LaunchShape eval_shape(const gd_ctx *c, int ci, int n, int *k);

/* ---- the record stream (gd_capi_stream.cu) ---- */
int rs_enqueue(gd_ctx *c, int rows_per_rep);
int rs_flush(gd_ctx *c);
int rs_restart(gd_ctx *c, int r0, int r1);
void rs_stop(gd_ctx *c);
/* waits for, then frees, the background window download */
void ra_free(gd_ctx *c);

/* ---- delayed acceptance (gd_capi_da.cu) ---- */
void da_free(gd_ctx *c);
void da_drop_graphs(gd_ctx *c);

/* ---- the device layout of one complex (gd_capi_layout.cu) ---- */
/* builds complex ci's arrays on the host, uploads them (pool memory, synchronised) and fills g;
 * thr: the contact thresholds [ligand type][point type] */
int layout_complex(gd_ctx *c, const gd_enepara *ff, const float (*thr)[GD_MAXTP1],
                   const gd_complex_desc &d, int ci, GdDevComplex &g);

/* ---- the pocket grid's point lists (gd_pocket.cu): optional, left out without memory ---- */
int build_pocket_lists(gd_ctx *c, std::vector<GdDevComplex> &dcx);

/* ---- the far fields of large proteins (gd_farfield.cu): optional, in a quarter of the memory
 * that is free when the context has all it needs ---- */
int build_far_fields(gd_ctx *c, const gd_enepara *ff, const gd_complex_desc *cxs,
                     std::vector<GdDevComplex> &dcx);
/* Distance from the pocket centre beyond which a complex's points are mostly fields, given memory
 * for them (infinity: no tables for this force field and protein). */
double field_reach(const gd_enepara *ff, const gd_complex_desc &d);

/* ---- allocation-free pose evaluation (gd_capi_noalloc.cu) ---- */
int noalloc_prepare(int device);

}  // namespace gdc

#endif
