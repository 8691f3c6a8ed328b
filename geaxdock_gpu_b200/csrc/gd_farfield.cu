/*
 * gd_farfield.cu -- the far points of a large protein as fields over a grid at the pocket
 * (gd_create).
 *
 * For an atom in a 2 A cell of the grid, every point beyond the cell's far radius (the largest
 * distance of the cell's box from the pocket centre plus r_f) is at least r_f from the atom: its
 * pmf term is pmf1 to 2^-25, its hydrogen-bond term rounds to zero, and its vdw and ele terms are
 * smooth functions of the atom's place in the cell. Their sums over the far points are tabulated
 * per conformer and cell as Chebyshev series of total degree 4 in the cell's coordinates (35
 * coefficients): one field of sum (ele_p / el1) / r, one vdw field per ligand atom type in use, and
 * the pmf sums per radius bin. The Monte Carlo kernel adds the fields once per atom and step and
 * runs its pair loop over the near points of each (radially ordered) segment only.
 *
 * Why: the pair loop is bound by the FMA and XU pipes, and on 3,000 points two thirds of its pairs
 * are far ones; an evaluation of the two series is about as many operations as 6 pairs. The
 * points are at least 8 cell edges away, so that a Chebyshev degree gains a factor of about 30.
 * Largest error over 300 places of six cells, relative to an atom's sum of |vdw|: on 4 A cells
 * 2e-6 / 3e-7 / 5e-8 at degree 4 / 5 / 6, on 2 A cells at degree 4 5e-8 (ele 4e-9), under the FP32
 * sum's own rounding. Smaller cells also leave fewer points to the loop: a warp of the 40-atom
 * ligand runs 1,630 / 1,470 / 1,310 of 3,000 with cells of 4 / 3 / 2 A.
 *
 * Node values are sums (FP32x2 over at most 128 point pairs of a type, those sums in FP64, as
 * the pair loop's) on the 5 x 5 x 5 Chebyshev nodes of a cell, one thread per node, one
 * CTA per (conformer, cell). The vdw term (p1 - p2) / (1 + x), p1 = p1a r^-9, p2 = p2a r^-6, x =
 * p1l z, z = r^-9 + lj1 r^-7, is expanded in x, so that a segment (one point type) needs the sums of
 * r^-9 z^k and r^-6 z^k only, k = 0..3, for every ligand type at once; the tables are made only
 * when x <= 1/32 at r_f for every type pair: less than 2^-20, a tenth of GD_CERT, of such a pair's
 * term is left out (the reference's force field: x = 0.019).
 * Complexes of one batch on the same protein share one set of tables.
 */
#include <memory>

#include "gd_capi_internal.cuh"

namespace gd {
namespace {

constexpr int NN = GD_FF_DEG + 1, NODES = NN * NN * NN;
constexpr int THREADS = 128;
constexpr int BLOCK = 128;
static_assert(THREADS >= NODES, "one thread per node");

struct FfArgs {
  const GdDevComplex *cxs;
  const GdPairParam *pp;
  const int *cells;      /* [n_cells] the tabulated cells */
  int n_cells, rep;      /* rep: a complex of the group */
  int n_types;
  unsigned char types[GD_MAXTP2]; /* the tabulated ligand types */
  float lj1;
  float *tab;
};

__global__ void __launch_bounds__(THREADS) farfield_kernel(FfArgs g) {
  extern __shared__ double val[]; /* [1 + n_types][NODES] */
  __shared__ double tm[NN][NN];   /* tm[i][a] = T_i(node a) times the transform's weight */
  const GdDevComplex &cx = g.cxs[g.rep];
  const int ic = blockIdx.x % g.n_cells, pc = blockIdx.x / g.n_cells, cell = g.cells[ic];
  const int bin = gd_ff_bin(cx, cell);
  const int tid = threadIdx.x;
  const int nf = 1 + g.n_types;
  float *out = g.tab + ((size_t)pc * g.n_cells + ic) * nf * GD_FF_NC;
  if (tid < NN * NN) {
    const int i = tid / NN, a = tid % NN;
    tm[i][a] = cospi(i * (a + 0.5) / NN) * (i ? 2.0 : 1.0) / NN;
  }
  const int na = tid % NN, nb = (tid / NN) % NN, nc = tid / (NN * NN);
  const bool on = tid < NODES;
  const double half = 0.5 * GD_FF_EDGE;
  const int ix = cell % GD_FF_N, iy = (cell / GD_FF_N) % GD_FF_N, iz = cell / (GD_FF_N * GD_FF_N);
  const double x = (double)cx.pocket[0] + (2 * ix + 1 - GD_FF_N + cospi((na + 0.5) / NN)) * half;
  const double y = (double)cx.pocket[1] + (2 * iy + 1 - GD_FF_N + cospi((nb + 0.5) / NN)) * half;
  const double z = (double)cx.pocket[2] + (2 * iz + 1 - GD_FF_N + cospi((nc + 0.5) / NN)) * half;
  if (on)
    for (int f = 0; f < nf; ++f) val[f * NODES + tid] = 0.0;
  const int nseg = cx.seg_count[pc];
  const float4 *pa = cx.pt_a + (size_t)pc * (cx.pnp_pad >> 1),
               *pb = cx.pt_b + (size_t)pc * (cx.pnp_pad >> 1);
  const float2 x2 = make_float2((float)x, (float)x), y2 = make_float2((float)y, (float)y),
               z2n = make_float2((float)z, (float)z), one = make_float2(1.0f, 1.0f),
               lj1 = make_float2(g.lj1, g.lj1);
  double ele = 0.0;
  for (int sg = 0; on && sg < nseg; ++sg) {
    const int4 s = cx.seg[pc * GD_MAX_SEG + sg];
    const int n0 = gd_ff_near(cx, pc, sg, s, bin);
    if (n0 >= s.y) continue;
    double A[4] = {0.0, 0.0, 0.0, 0.0}, B[4] = {0.0, 0.0, 0.0, 0.0};
    /* n0 is even: pairs of slots in FP32x2 as in the pair loop, sums folded to FP64 every BLOCK
     * pairs; the segment's odd last slot is a single point (its partner weighs nothing) */
    const int m1 = (s.y + 1) >> 1;
    for (int m0 = n0 >> 1; m0 < m1; m0 += BLOCK) {
      const float2 z2 = make_float2(0.0f, 0.0f);
      float2 sa[4] = {z2, z2, z2, z2}, sb[4] = {z2, z2, z2, z2}, se = z2;
      const int me = min(m1, m0 + BLOCK);
#pragma unroll 2
      for (int m = m0; m < me; ++m) {
        const float4 P = __ldg(pa + m), Q = __ldg(pb + m);
        const float2 dx = __fadd2_rn(x2, make_float2(P.x, P.y)),
                     dy = __fadd2_rn(y2, make_float2(P.z, P.w)),
                     dz = __fadd2_rn(z2n, make_float2(Q.x, Q.y));
        const float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
        float2 r = make_float2(rsqrtf(d2.x), rsqrtf(d2.y));
        /* one Newton step: r + r / 2 (1 - d2 r r) */
        const float2 h = __fmul2_rn(r, make_float2(0.5f, 0.5f));
        const float2 t = __fmul2_rn(d2, r);
        r = __ffma2_rn(h, __ffma2_rn(make_float2(-t.x, -t.y), r, one), r);
        const bool pad = 2 * m + 1 >= s.y;
        float2 ep = make_float2(Q.z, Q.w);
        if (pad) {
          r.y = 0.0f;
          ep.y = 0.0f;
        }
        const float2 r3 = __fmul2_rn(__fmul2_rn(r, r), r), r6 = __fmul2_rn(r3, r3);
        const float2 r9 = __fmul2_rn(r6, r3);
        const float2 zz = __ffma2_rn(lj1, __fmul2_rn(r6, r), r9);
        se = __ffma2_rn(ep, r, se);
        sa[0] = __fadd2_rn(sa[0], r9);
        sb[0] = __fadd2_rn(sb[0], r6);
        float2 ta = __fmul2_rn(r9, zz), tb = __fmul2_rn(r6, zz);
        sa[1] = __fadd2_rn(sa[1], ta);
        sb[1] = __fadd2_rn(sb[1], tb);
        ta = __fmul2_rn(ta, zz);
        tb = __fmul2_rn(tb, zz);
        sa[2] = __fadd2_rn(sa[2], ta);
        sb[2] = __fadd2_rn(sb[2], tb);
        sa[3] = __ffma2_rn(ta, zz, sa[3]);
        sb[3] = __ffma2_rn(tb, zz, sb[3]);
      }
      ele += (double)se.x + (double)se.y;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        A[k] += (double)sa[k].x + (double)sa[k].y;
        B[k] += (double)sb[k].x + (double)sb[k].y;
      }
    }
    for (int k = 0; k < g.n_types; ++k) {
      const GdPairParam &q = g.pp[g.types[k] * GD_MAXTP1 + s.z];
      const double l = -(double)q.p1l;
      val[(1 + k) * NODES + tid] += (double)q.p1a * (A[0] + l * (A[1] + l * (A[2] + l * A[3]))) -
                                    (double)q.p2a * (B[0] + l * (B[1] + l * (B[2] + l * B[3])));
    }
  }
  if (on) val[tid] = ele;
  __syncthreads();
  /* node values to series coefficients, one axis after the other */
  for (int f = 0; f < nf; ++f) {
    double *v = val + f * NODES;
#pragma unroll 1
    for (int axis = 0; axis < 3; ++axis) {
      const int stride = axis == 0 ? 1 : axis == 1 ? NN : NN * NN;
      const int i = axis == 0 ? na : axis == 1 ? nb : nc;
      double c = 0.0;
      if (on)
        for (int a = 0; a < NN; ++a) c += tm[i][a] * v[tid + (a - i) * stride];
      __syncthreads();
      if (on) v[tid] = c;
      __syncthreads();
    }
    if (tid == 0)
      for (int o = NN * (NN + 1) * (NN + 2) / 6; o < GD_FF_NC; ++o) out[f * GD_FF_NC + o] = 0.0f;
    if (on && na + nb + nc <= GD_FF_DEG) {
      /* order: k of z outermost, then j of y, then i of x, i + j + k <= degree */
      int o = na;
      for (int k = 0; k < nc; ++k) o += (NN - k) * (NN - k + 1) / 2;
      for (int j = 0; j < nb; ++j) o += NN - nc - j;
      out[f * GD_FF_NC + o] = (float)v[tid];
    }
  }
}

/* pmf sums of the far points, one thread per (conformer, radius bin, ligand type) */
__global__ void farpmf_kernel(const GdDevComplex *cxs, int rep, const GdPairParam *pp, int n,
                              double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const GdDevComplex &cx = cxs[rep];
  const int tl = i % GD_MAXTP2, bin = (i / GD_MAXTP2) % GD_FAR_BINS,
            pc = i / (GD_MAXTP2 * GD_FAR_BINS);
  double s = 0.0;
  for (int sg = 0; sg < cx.seg_count[pc]; ++sg) {
    const int4 g = cx.seg[pc * GD_MAX_SEG + sg];
    s += (double)pp[tl * GD_MAXTP1 + g.z].pmf1 * (double)(g.y - gd_ff_near(cx, pc, sg, g, bin));
  }
  out[i] = s;
}

}  // namespace
}  // namespace gd

namespace gdc {

namespace {

/* the largest distance of the cell's box from the grid's centre, in cell edges squared */
int cell_reach2(int cell) {
  const int i[3] = {cell % GD_FF_N, (cell / GD_FF_N) % GD_FF_N, cell / (GD_FF_N * GD_FF_N)};
  int r2 = 0;
  for (int a = 0; a < 3; ++a) {
    const int m = std::max(GD_FF_N / 2 - i[a], i[a] + 1 - GD_FF_N / 2);
    r2 += m * m;
  }
  return r2;
}

uint64_t fnv(uint64_t h, const void *p, size_t n) {
  /* FNV-1a over 8-byte words (Fowler, Noll, Vo), the tail bytes last */
  const unsigned char *b = static_cast<const unsigned char *>(p);
  for (; n >= 8; n -= 8, b += 8) {
    uint64_t w;
    memcpy(&w, b, 8);
    h = (h ^ w) * 0x100000001b3ull;
  }
  for (; n; --n, ++b) h = (h ^ *b) * 0x100000001b3ull;
  return h;
}

/* the inputs that a protein's tables depend on */
uint64_t protein_hash(const gd_complex_desc &d) {
  const size_t n = (size_t)d.n_prt * d.pnp;
  uint64_t h = 0xcbf29ce484222325ull ^ (uint64_t)d.n_prt ^ ((uint64_t)d.pnp << 32);
  for (const void *p : {(const void *)d.prt_x, (const void *)d.prt_y, (const void *)d.prt_z,
                        (const void *)d.prt_t, (const void *)d.prt_ele})
    h = fnv(h, p, 4 * n);
  return fnv(h, d.pocket_center, 12);
}

bool same_protein(const gd_complex_desc &a, const gd_complex_desc &b) {
  if (a.n_prt != b.n_prt || a.pnp != b.pnp) return false;
  const size_t n = 4 * (size_t)a.n_prt * a.pnp;
  return !memcmp(a.prt_x, b.prt_x, n) && !memcmp(a.prt_y, b.prt_y, n) &&
         !memcmp(a.prt_z, b.prt_z, n) && !memcmp(a.prt_t, b.prt_t, n) &&
         !memcmp(a.prt_ele, b.prt_ele, n) && !memcmp(a.pocket_center, b.pocket_center, 12);
}

}  // namespace

/* r_f and the extra bins per point type: properties of the force field alone, so that a complex
 * has the same tables whatever ligand or batch it comes with. False: no tables. */
static bool ff_radii(const gd_enepara *ff, double *r_f, double *r_hdb) {
  *r_f = 0.0;
  for (int tl = 0; tl < GD_MAXTP2; ++tl)
    for (int tp = 0; tp < GD_MAXTP1; ++tp) *r_f = std::max(*r_f, pmf_far_radius(ff->pmf0[tl][tp]));
  *r_f += 0.01;
  for (int tp = 0; tp < GD_MAXTP1; ++tp) {
    r_hdb[tp] = 0.0;
    for (int tl = 0; tl < GD_MAXTP2; ++tl)
      if (ff->hdb0[tl][tp] > 0.1f) {
        /* exp2 of minus 0.5 log2(e) ((r - hdb0) hdb1)^2 is flushed to zero below -126 */
        const double r = ff->hdb0[tl][tp] + std::sqrt(127.0 / (0.5 * 1.4426950408889634)) /
                                                std::fabs((double)ff->hdb1[tl][tp]);
        if (!std::isfinite(r)) return false;
        r_hdb[tp] = std::max(r_hdb[tp], r);
      }
  }
  const double r3 = 1.0 / (*r_f * *r_f * *r_f), z = r3 * r3 * (r3 + std::fabs(ff->lj1) / *r_f);
  for (int tl = 0; tl < GD_MAXTP2; ++tl)
    for (int tp = 0; tp < GD_MAXTP1; ++tp)
      if (!(std::fabs((double)ff->p1a[tl][tp] * ff->lj0) * z <= 1.0 / 32.0)) return false;
  return true;
}

/* Complexes worth it: at least a quarter of the points lie beyond the far radius of a cell that
 * reaches 10 A (with 19 % beyond, 1,500 points, a step got slower by the evaluation's latency; with
 * 60 %, 3,000 points, faster). */
static bool field_worth(const gd_complex_desc &d, double r_f) {
  const size_t n = (size_t)d.n_prt * d.pnp;
  size_t beyond = 0;
  const double lim = (10.0 + r_f) * (10.0 + r_f);
  for (size_t i = 0; i < n; ++i) {
    const double x = (double)d.prt_x[i] - d.pocket_center[0],
                 y = (double)d.prt_y[i] - d.pocket_center[1],
                 z = (double)d.prt_z[i] - d.pocket_center[2];
    beyond += x * x + y * y + z * z > lim ? 1 : 0;
  }
  return beyond * 4 >= n;
}

double field_reach(const gd_enepara *ff, const gd_complex_desc &d) {
  double r_f, r_hdb[GD_MAXTP1];
  if (!ff_radii(ff, &r_f, r_hdb) || !field_worth(d, r_f))
    return std::numeric_limits<double>::infinity();
  return 10.0 + r_f;
}

/* Appends ff_cert of a complex (GD_CERT_ELE, GD_CERT_FAR), by protein and ligand conformer. */
static void certainty(const gd_ctx *c, const gd_enepara *ff, const gd_complex_desc &d, double r_f,
                      std::vector<float> &out) {
  double wa[3];
  for (int k = 0; k < 3; ++k) wa[k] = std::fabs((double)c->fc.w[k] * c->fc.a_para[k]);
  const double r3 = 1.0 / (r_f * r_f * r_f), r6 = r3 * r3, r9 = r6 * r3;
  for (int p = 0; p < d.n_prt; ++p) {
    double count[GD_MAXTP1] = {0.0}, by_type[GD_MAXTP2], ele = 0.0;
    for (int i = p * d.pnp; i < (p + 1) * d.pnp; ++i) {
      count[d.prt_t[i]] += 1.0;
      ele += std::fabs((double)d.prt_ele[i]);
    }
    for (int t = 0; t < GD_MAXTP2; ++t) {
      by_type[t] = 0.0;
      for (int tp = 0; tp < GD_MAXTP1; ++tp)
        by_type[t] += count[tp] * (wa[0] * (std::fabs((double)ff->p1a[t][tp]) * r9 +
                                            std::fabs((double)ff->p2a[t][tp]) * r6) +
                                   wa[2] * std::fabs((double)ff->pmf1[t][tp]));
    }
    ele *= wa[1] / ((double)ff->el1 * r_f);
    for (int l = 0; l < d.n_lig; ++l) {
      double s = 0.0;
      for (int i = l * d.lna; i < (l + 1) * d.lna; ++i)
        s += GD_CERT_ELE * ele * std::fabs((double)d.lig_c[i]) + GD_CERT_FAR * by_type[d.lig_t[i]];
      out.push_back((float)(s / d.lna));
    }
  }
}

/* Bytes the tables may take: a quarter of what the device has free once the context holds all it
 * must (the pool's idle memory is free too), so that records, samples and poses asked for later
 * and other users of the device find room; release_fields gives even that back. */
static size_t field_budget(gd_ctx *c) {
  size_t free_b = 0, total_b = 0;
  if (cudaStreamSynchronize(c->stream) != cudaSuccess ||
      cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  uint64_t held = 0, used = 0;
  cudaMemPool_t pool = ctx_pool(c->device);
  if (pool && cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) ==
                  cudaSuccess &&
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess &&
      held > used)
    free_b += held - used;
  return free_b / 4;
}

bool release_fields(gd_ctx *c) {
  if (c->field_allocs.empty()) return false;
  cudaStreamSynchronize(c->stream); /* no kernel reads the tables */
  for (int ci = 0; ci < c->n_complex; ++ci)
    cudaMemsetAsync(reinterpret_cast<char *>(c->d_cx + ci) + offsetof(GdDevComplex, ff_tab), 0,
                    sizeof(float *), c->stream);
  for (void *p : c->field_allocs) dfree(c, p);
  c->field_allocs.clear();
  c->field_bytes = 0;
  cudaStreamSynchronize(c->stream);
  if (cudaMemPool_t pool = ctx_pool(c->device)) cudaMemPoolTrimTo(pool, 0);
  return true;
}

int build_far_fields(gd_ctx *c, const gd_enepara *ff, const gd_complex_desc *cxs,
                     std::vector<GdDevComplex> &dcx) {
  double r_f, r_hdb[GD_MAXTP1];
  if (!ff_radii(ff, &r_f, r_hdb)) return GD_OK;
  /* the complexes worth it, grouped by protein */
  struct Group { std::vector<int> members; bool used[GD_MAXTP2] = {}; };
  std::vector<std::unique_ptr<Group>> groups;
  std::map<uint64_t, std::vector<Group *>> by_hash;
  for (int ci = 0; ci < c->n_complex; ++ci) {
    const gd_complex_desc &d = cxs[ci];
    Group *g = nullptr;
    const uint64_t h = c->n_complex > 1 ? protein_hash(d) : 0;
    for (Group *q : by_hash[h])
      if (same_protein(cxs[q->members[0]], d)) g = q;
    if (!g) {
      if (!field_worth(d, r_f)) continue;
      groups.push_back(std::make_unique<Group>());
      g = groups.back().get();
      by_hash[h].push_back(g);
    }
    g->members.push_back(ci);
    for (int i = 0; i < d.n_lig * d.lna; ++i) g->used[d.lig_t[i]] = true;
  }
  if (groups.empty()) return GD_OK;
  int rc;
  CK(cudaFuncSetAttribute(gd::farfield_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)((1 + GD_MAXTP2) * gd::NODES * sizeof(double))));
  std::vector<gd::FfArgs> jobs;
  std::vector<double *> pmf;
  const size_t budget = field_budget(c);
  for (auto &gp : groups) {
    gd::FfArgs a{};
    a.pp = c->d_pp;
    a.rep = gp->members[0];
    /* the tabulated cells: those whose far radius leaves a tenth of a ball of points beyond it,
     * at most the cube's inscribed ball (22 A; an atom outside runs all points in its loop) */
    const double rad_max = (GD_FAR_BINS - 1) / (double)dcx[a.rep].far_inv_w;
    const double reach =
        std::min(0.5 * GD_FF_N, std::max(4.0, (0.965 * rad_max - r_f) / GD_FF_EDGE));
    std::vector<int> cells;
    std::vector<short> id(GD_FF_CELLS, -1);
    for (int k = 0; k < GD_FF_CELLS; ++k)
      if (cell_reach2(k) <= reach * reach) {
        id[k] = (short)cells.size();
        cells.push_back(k);
      }
    a.n_cells = (int)cells.size();
    a.lj1 = ff->lj1;
    unsigned char slot[GD_MAXTP2] = {};
    for (int t = 0; t < GD_MAXTP2; ++t)
      if (gp->used[t]) {
        slot[t] = (unsigned char)a.n_types;
        a.types[a.n_types++] = (unsigned char)t;
      }
    const int n_prt = c->info[a.rep].n_prt;
    const size_t per = (size_t)cells.size() * (1 + a.n_types) * GD_FF_NC;
    std::vector<float> cert;
    for (int ci : gp->members) certainty(c, ff, cxs[ci], r_f, cert);
    const size_t n_pmf = (size_t)n_prt * GD_FAR_BINS * GD_MAXTP2;
    const size_t bytes = sizeof(float) * per * n_prt + sizeof(double) * n_pmf +
                         sizeof(int) * cells.size() + sizeof(short) * id.size() +
                         sizeof(float) * cert.size();
    /* a protein whose tables do not fit runs without them */
    if (c->field_bytes + bytes > budget) continue;
    int *d_cells = nullptr;
    short *d_id = nullptr;
    double *p = nullptr;
    float *d_cert = nullptr;
    const bool made = !upload(c, &d_cert, cert) && !upload(c, &d_cells, cells) && !upload(c, &d_id, id) &&
                      !dalloc(c, &a.tab, per * n_prt) && !dalloc(c, &p, n_pmf);
    CK(cudaStreamSynchronize(c->stream)); /* the host vectors end here */
    for (void *q : {(void *)d_cells, (void *)d_id, (void *)a.tab, (void *)p, (void *)d_cert}) {
      if (!q) continue;
      if (made)
        c->field_allocs.push_back(q);
      else
        dfree(c, q);
    }
    if (!made) continue;
    c->field_bytes += bytes;
    a.cells = d_cells;
    for (int ci : gp->members) {
      GdDevComplex &g = dcx[ci];
      g.ff_id = d_id;
      g.ff_tab = a.tab;
      g.ff_pmf = p;
      g.ff_cert = d_cert;
      d_cert += (size_t)cxs[ci].n_prt * cxs[ci].n_lig;
      g.ff_fields = 1 + a.n_types;
      g.ff_cells = (int)cells.size();
      g.ff_r = (float)(r_f + 0.05);
      for (int t = 0; t < GD_MAXTP2; ++t) g.ff_slot[t] = slot[t];
      for (int t = 0; t < GD_MAXTP1; ++t)
        g.ff_extra[t] = (unsigned char)std::min(
            255.0, std::max(0.0, std::ceil((r_hdb[t] - r_f) * (double)g.far_inv_w)));
    }
    jobs.push_back(a);
    pmf.push_back(p);
  }
  CK(cudaMemcpyAsync(c->d_cx, dcx.data(), sizeof(GdDevComplex) * dcx.size(),
                     cudaMemcpyHostToDevice, c->stream));
  for (size_t k = 0; k < jobs.size(); ++k) {
    gd::FfArgs &a = jobs[k];
    a.cxs = c->d_cx;
    const int n_prt = c->info[a.rep].n_prt;
    gd::farfield_kernel<<<(unsigned)(a.n_cells * n_prt), gd::THREADS,
                          (1 + a.n_types) * gd::NODES * sizeof(double), c->stream>>>(a);
    const int n = n_prt * GD_FAR_BINS * GD_MAXTP2;
    gd::farpmf_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(c->d_cx, a.rep, c->d_pp, n, pmf[k]);
    CK(cudaGetLastError());
  }
  CK(cudaStreamSynchronize(c->stream)); /* the host vectors end here */
  return GD_OK;
}

}  // namespace gdc
