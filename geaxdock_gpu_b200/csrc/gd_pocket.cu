/*
 * gd_pocket.cu -- the pocket grid's point lists (gd_create): for every 4 A cell of a cube around
 * the pocket centre, the points the short-range terms of an atom in that cell can involve.
 *
 * The Monte Carlo kernel's short-range pass used to walk the rows of the conformer's cell list
 * for every atom: per lane some 25 rows of 4-5 points each, whose lengths differ from lane to lane,
 * with a dependent load per point. A warp spent 87-135 k cycles of a step on it, whatever the
 * protein's size (31 % of the step of a 344-point pocket). The lists make it two streams per
 * lane, four points' loads in flight, and put the rarer terms on a shorter list:
 *   contact list   every point within the largest contact threshold (and the soft-core radius)
 *                  of the cell's box: contacts, the electrostatic soft core;
 *   kind list      the hydrophobic points within 9 A and the class-2 points within the contact
 *                  radius: hpc, psp.
 * Entries are 16-bit point indices of the conformer's cell list, in its order (rows of cells by
 * z, y, then x), so that the sums add the same terms in the same order as the row walk, which
 * atoms outside the cube still take; every list is padded to whole quads with the sentinel
 * point behind the conformer's points (infinitely far: no term). Memory: about 0.2 MB a conformer.
 * One warp builds one cell's two lists, in two passes (count, fill).
 */
#include "gd_capi_internal.cuh"

namespace gd {
namespace {

constexpr int WARPS = 8;

/* FILL: writes the indices; else the lists' padded lengths to start[2 cell], start[2 cell + 1] */
template <bool FILL>
__global__ void __launch_bounds__(32 * WARPS)
    pocket_kernel(const GdDevComplex *__restrict__ cxs, const int2 *__restrict__ conf,
                  long long n_cells, int *__restrict__ counts, unsigned short *__restrict__ out,
                  const long long *__restrict__ conf_base) {
  const long long w = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= n_cells) return;
  const int ic = (int)(w / GD_PG_CELLS), cell = (int)(w % GD_PG_CELLS);
  const int2 cf = conf[ic];
  const GdDevComplex &cx = cxs[cf.x];
  const int ix = cell % GD_PG_N, iy = (cell / GD_PG_N) % GD_PG_N, iz = cell / (GD_PG_N * GD_PG_N);
  const float lx = cx.pg_org[0] + ix * GD_PG_EDGE, ly = cx.pg_org[1] + iy * GD_PG_EDGE,
              lz = cx.pg_org[2] + iz * GD_PG_EDGE;
  const float R = fmaxf(cx.pg_rh, cx.pg_rc), rh2 = cx.pg_rh * cx.pg_rh, rc2 = cx.pg_rc * cx.pg_rc;
  const int nx = cx.sr_n[0], ny = cx.sr_n[1], nz = cx.sr_n[2];
  const float inv = cx.sr_inv_cell;
  auto lo = [&](float v, float o) { return (int)floorf(fmaxf((v - R - o) * inv, -1.0f)); };
  auto hi = [&](float v, float o, int n) {
    return (int)floorf(fminf((v + GD_PG_EDGE + R - o) * inv, (float)n));
  };
  const int x0 = max(0, lo(lx, cx.sr_org[0])), x1 = min(nx - 1, hi(lx, cx.sr_org[0], nx));
  const int y0 = max(0, lo(ly, cx.sr_org[1])), y1 = min(ny - 1, hi(ly, cx.sr_org[1], ny));
  const int z0 = max(0, lo(lz, cx.sr_org[2])), z1 = min(nz - 1, hi(lz, cx.sr_org[2], nz));
  const int *st = cx.sr_start + (size_t)cf.y * (cx.sr_n[3] + 1);
  const float4 *pa = cx.sr_a + (size_t)cf.y * (cx.pnp + 1);
  int *cnt = counts + 2 * w;
  unsigned short *oc = nullptr, *ok = nullptr;
  if (FILL) {
    /* counts holds the starts by now */
    oc = out + conf_base[ic] + cnt[0];
    ok = out + conf_base[ic] + cnt[1];
  }
  int nc = 0, nk = 0;
  if (x0 <= x1)
    for (int z = z0; z <= z1; ++z)
      for (int y = y0; y <= y1; ++y) {
        const int row = (z * ny + y) * nx;
        const int b0 = st[row + x0], b1 = st[row + x1 + 1];
        for (int i0 = b0; i0 < b1; i0 += 32) {
          const int i = i0 + lane;
          bool con = false, kind = false;
          if (i < b1) {
            const float4 p = pa[i];
            const float gx = fmaxf(0.0f, fmaxf(lx - p.x, p.x - (lx + GD_PG_EDGE)));
            const float gy = fmaxf(0.0f, fmaxf(ly - p.y, p.y - (ly + GD_PG_EDGE)));
            const float gz = fmaxf(0.0f, fmaxf(lz - p.z, p.z - (lz + GD_PG_EDGE)));
            const float d2 = gx * gx + gy * gy + gz * gz;
            const int meta = __float_as_int(p.w);
            con = d2 <= rc2;
            kind = ((meta & 256) && d2 <= rh2) || ((meta & 512) && con);
          }
          const unsigned mc = __ballot_sync(0xffffffffu, con);
          const unsigned mk = __ballot_sync(0xffffffffu, kind);
          if (FILL) {
            const unsigned below = (1u << lane) - 1u;
            if (con) oc[nc + __popc(mc & below)] = (unsigned short)i;
            if (kind) ok[nk + __popc(mk & below)] = (unsigned short)i;
          }
          nc += __popc(mc);
          nk += __popc(mk);
        }
      }
  if (FILL) {
    if (lane < ((4 - (nc & 3)) & 3)) oc[nc + lane] = (unsigned short)cx.pnp;
    if (lane < ((4 - (nk & 3)) & 3)) ok[nk + lane] = (unsigned short)cx.pnp;
  } else if (lane == 0) {
    cnt[0] = (nc + 3) & ~3;
    cnt[1] = (nk + 3) & ~3;
  }
}

}  // namespace
}  // namespace gd

namespace gdc {

namespace {

/* The lists of every conformer of the batch: counts on the device, starts on the host, the
 * lists in one buffer; fills in the complexes' pg_start / pg_idx. got: the buffers made */
int pocket_lists(gd_ctx *c, std::vector<GdDevComplex> &dcx, std::vector<void *> &got) {
  std::vector<int2> conf;
  for (int ci = 0; ci < c->n_complex; ++ci)
    for (int p = 0; p < c->info[ci].n_prt; ++p) conf.push_back(make_int2(ci, p));
  const size_t nconf = conf.size();
  const long long n_cells = (long long)nconf * GD_PG_CELLS;
  const size_t per = 2 * GD_PG_CELLS + 1;
  int2 *d_conf = nullptr;
  int *d_cnt = nullptr;
  int rc;
  if ((rc = upload(c, &d_conf, conf))) return rc;
  got.push_back(d_conf);
  if ((rc = dalloc(c, &d_cnt, (size_t)n_cells * 2))) return rc;
  got.push_back(d_cnt);
  const unsigned grid = (unsigned)((n_cells + gd::WARPS - 1) / gd::WARPS);
  gd::pocket_kernel<false><<<grid, 32 * gd::WARPS, 0, c->stream>>>(c->d_cx, d_conf, n_cells,
                                                                   d_cnt, nullptr, nullptr);
  CK(cudaGetLastError());
  std::vector<int> cnt((size_t)n_cells * 2);
  CK(cudaMemcpyAsync(cnt.data(), d_cnt, sizeof(int) * cnt.size(), cudaMemcpyDeviceToHost,
                     c->stream));
  CK(cudaStreamSynchronize(c->stream));
  /* starts within the conformer's lists, one past the last at the end */
  std::vector<int> start(nconf * per);
  std::vector<long long> base(nconf);
  long long total = 0;
  for (size_t k = 0; k < nconf; ++k) {
    base[k] = total;
    int off = 0;
    for (size_t j = 0; j < 2 * GD_PG_CELLS; ++j) {
      start[k * per + j] = off;
      int &n = cnt[k * 2 * GD_PG_CELLS + j];
      const int len = n;
      n = off;
      off += len;
    }
    start[k * per + 2 * GD_PG_CELLS] = off;
    total += off;
  }
  unsigned short *d_idx = nullptr;
  int *d_start = nullptr;
  long long *d_base = nullptr;
  if ((rc = upload(c, &d_start, start))) return rc;
  got.push_back(d_start);
  if ((rc = upload(c, &d_base, base))) return rc;
  got.push_back(d_base);
  if ((rc = dalloc(c, &d_idx, (size_t)total))) return rc;
  got.push_back(d_idx);
  CK(cudaMemcpyAsync(d_cnt, cnt.data(), sizeof(int) * cnt.size(), cudaMemcpyHostToDevice,
                     c->stream));
  gd::pocket_kernel<true><<<grid, 32 * gd::WARPS, 0, c->stream>>>(c->d_cx, d_conf, n_cells, d_cnt,
                                                                  d_idx, d_base);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c->stream)); /* the host vectors end here */
  size_t k = 0;
  for (int ci = 0; ci < c->n_complex; ++ci) {
    dcx[ci].pg_start = d_start + k * per;
    dcx[ci].pg_idx = d_idx;
    dcx[ci].pg_base = d_base + k;
    k += c->info[ci].n_prt;
  }
  dfree(c, d_conf);
  dfree(c, d_cnt);
  return GD_OK;
}

}  // namespace

/* (c->d_cx holds the complexes without the lists; the caller uploads dcx again.) Without the
 * memory for them no atom finds itself in the grid, and each walks the rows of the cell list. */
int build_pocket_lists(gd_ctx *c, std::vector<GdDevComplex> &dcx) {
  std::vector<void *> got;
  const int rc = pocket_lists(c, dcx, got);
  if (rc != GD_ERR_NOMEM) return rc;
  CK(cudaStreamSynchronize(c->stream)); /* the uploads' host arrays are gone */
  for (void *p : got) dfree(c, p);
  for (GdDevComplex &g : dcx)
    for (float &o : g.pg_org) o = std::numeric_limits<float>::quiet_NaN();
  return GD_OK;
}

}  // namespace gdc
