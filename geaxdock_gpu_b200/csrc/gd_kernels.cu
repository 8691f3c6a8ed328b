/*
 * gd_kernels.cu -- sm_100a kernels of the Monte Carlo docking path.
 *
 * gd_mc_kernel: one persistent kernel for MonteCarlo_Init_d, MonteCarlo_d and pose
 * evaluation (reference src/kernel_cuda_l1_montecarlo.cu:12-127). Each CTA pulls tiles from
 * a work queue; a tile is `count` replicas of one protein conformer. Lane (slot j, atom l)
 * owns one ligand atom of one replica for all steps of the launch (a thread holds one lane,
 * or with PACK = 2 the lanes of the same atom in two slots, which share every load; with SPLIT the
 * lanes of an atom in several warps run some of the protein's segments each):
 *   Move_d        (src/kernel_cuda_l2_move.cu:21-80)       placed in registers from a
 *                                                         Philox draw, no HBM traffic;
 *   CalcEnergy_d  (src/kernel_cuda_l2_calcenergy.cu:19-360) the terms every pair has (vdw,
 *                 ele in its far form, pmf, hdb) in a loop over all protein points staged by
 *                 cp.async.bulk into a shared-memory double buffer, points sorted by type so
 *                 each lane keeps its pair parameters in registers per segment, MUFU rsqrt /
 *                 rcp / ex2, FP32 range sums folded into FP64; the far points of a large
 *                 protein as tabulated fields (gd_farfield.cu), with the decisions that could
 *                 hang on their rounding taken on the pair loop's energies; the short-range
 *                 terms (contacts, psp, hpc, the ele soft core) from the point lists of the
 *                 atom's pocket-grid cell (gd_pocket.cu), outside the grid from a walk of the
 *                 conformer's cell list;
 *   CalcMcc_d     (src/kernel_cuda_l2_calcmcc.cu:148-206) contact count in the same pass,
 *                 true positives from the sparse reference-contact list;
 *   CalcRmsd_d, KDE, MCS, dst, CombineEnergy_d (src/kernel_cuda_l3_combineenergy.cu:23-37),
 *                 of moved poses (modes 0-3) or of given placed coordinates (mode 4),
 *   Accept_d (src/kernel_cuda_l2_accept.cu:13-46), RecordLigand_d
 *   (src/kernel_cuda_l3_util.cu:74-106) in the per-replica epilogue run by one warp per slot.
 * gd_exchange_kernel: ExchangeReplicas_d (src/kernel_cuda_l1_exchangereplicas.cu:27-77), one
 * thread per (protein conformer, ligand conformer) group instead of one thread for all; groups
 * that it, or the exchange fused into gd_mc_kernel, leaves open for the far fields' rounding are
 * exchanged by gd_mc_kernel's GD_KIND_EXCHANGE form.
 */
#include <cuda_runtime.h>

#include "gd_device.cuh"
#include "gd_numerics.h"

namespace gd {

/* ---------------- MUFU / PTX helpers ---------------- */
__device__ __forceinline__ float rsqrt_a(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_a(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_a(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ long long gtimer() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
/* Spins on the barrier phase for at most timeout_ns (globaltimer); false on timeout. */
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  long long timeout_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long deadline = gtimer() + timeout_ns;
  while (!mbar_try_wait(bar, parity))
    if (gtimer() > deadline) return false;
  return true;
}

/* Squared distance written the same way everywhere a contact decision is taken. */
__device__ __forceinline__ float dist2(float ax, float ay, float az, float px, float py,
                                       float pz) {
  const float dx = __fsub_rn(ax, px), dy = __fsub_rn(ay, py), dz = __fsub_rn(az, pz);
  return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

/* hpc switching polynomial 1 - (3.5 u/81 - 4.5 u^2/81^2 + 2.5 u^3/81^3 - 0.5 u^4/81^4), u = d^2 */
#define HPC_C1 (3.5f / 81.0f)
#define HPC_C2 (4.5f / 6561.0f)
#define HPC_C3 (2.5f / 531441.0f)
#define HPC_C4 (0.5f / 43046721.0f)
#define LOG2E_F 1.4426950408889634f

struct Acc {
  float2 vdw, ele, pmf, hdb;
};

/* Per-segment pair parameters, splatted over the two lanes of an FP32x2 register pair. */
struct Pair2 {
  float2 p1a, mp2a, p1l, p1ll, b2, c2, hc1, hc0, hs;
};

__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }

/* One pair of protein slots (2m, 2m+1) against the lane's atom: the terms every pair has
 * (vdw, the far form of ele, pmf; hdb on segments whose type has a live hydrogen-bond pair).
 * The short-range terms (contacts, psp, hpc, the electrostatic soft core) come from the cell
 * list pass, short_range(). PAIR = false: only the first slot is a point (the second is
 * segment padding) and nothing of the second is kept. FAR: both points lie beyond the atom's
 * far radius, where the pmf exponent is below -25.5 in base 2 (the host's radius has a margin
 * of 0.5 over the FP32 rounding of tt). There ee < 2^-25, so p4 + p4 ee rounds to p4 and
 * num + num ee to num: the full body's terms are num rcp(p4) and p4 rcp(p4), which the far
 * form computes without tt, ee, pd and vn, bit for bit; where a warp splits a segment into
 * its near and far parts therefore changes no result. */
template <bool HDB, bool PAIR, bool FAR>
__device__ __forceinline__ void pair_body(const float4 A, const float4 B, float2 ax, float2 ay,
                                          float2 az, const Pair2 &q, const GdForceConst &f,
                                          Acc &a) {
  const float2 one = f2(1.0f);
  /* squared distance, per lane exactly dist2(): a + (-p) == a - p */
  const float2 dx = __fadd2_rn(ax, make_float2(A.x, A.y));
  const float2 dy = __fadd2_rn(ay, make_float2(A.z, A.w));
  const float2 dz = __fadd2_rn(az, make_float2(B.x, B.y));
  const float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
  const float2 ri = make_float2(rsqrt_a(d2.x), rsqrt_a(d2.y));
  /* vdw: (p1 - p2) / (p1 lj0 (1 + lj1 d2) + 1), p1 = p1a r^-9, p2 = p2a r^-6; the
   * denominator is (p1l + p1ll d2) r^-9 + 1 with p1l = p1a lj0, p1ll = p1l lj1 */
  const float2 r2i = __fmul2_rn(ri, ri);
  const float2 r3i = __fmul2_rn(r2i, ri);
  const float2 r6i = __fmul2_rn(r3i, r3i);
  const float2 num = __fmul2_rn(r6i, __ffma2_rn(q.p1a, r3i, q.mp2a));
  const float2 p4 = __ffma2_rn(__ffma2_rn(q.p1ll, d2, q.p1l), __fmul2_rn(r6i, r3i), one);
  /* ele: q_l ele_p g(el1 r), q_l applied once per atom. The points hold ele_p / el1, so the
   * far form g = 1 / (el1 r) is one FMA with r^-1; pairs inside r < 1 / el1 get the soft-core
   * difference in short_range() */
  const float2 ep = make_float2(B.z, B.w);
  if constexpr (PAIR) {
    a.ele = __ffma2_rn(ep, ri, a.ele);
  } else {
    a.ele.x = __fmaf_rn(ep.x, ri.x, a.ele.x);
  }
  if constexpr (FAR) {
    const float2 inv = make_float2(rcp_a(p4.x), rcp_a(p4.y));
    if constexpr (PAIR) {
      a.vdw = __ffma2_rn(num, inv, a.vdw);
      a.pmf = __ffma2_rn(p4, inv, a.pmf);
    } else {
      a.vdw.x = __fmaf_rn(num.x, inv.x, a.vdw.x);
      a.pmf.x = __fmaf_rn(p4.x, inv.x, a.pmf.x);
    }
  } else {
  /* pmf: pmf1 / (1 + exp((6 - r/2)(r - pmf0))) as exp2 of the expanded quadratic
   * cA d2 + b2 r + c2 = d2 (b2 r^-1 + cA) + c2 (cA = -log2(e)/2, b2 = log2(e)(6 + pmf0/2),
   * c2 = -6 log2(e) pmf0). Its maximum over r is log2(e) (12 - pmf0)^2 / 8 < 100 for
   * pmf0 > -10 (checked when the force field is loaded), so den stays finite and p4 den does
   * wherever p4 does. */
  const float2 tt = __ffma2_rn(d2, __ffma2_rn(q.b2, ri, f2(-0.5f * LOG2E_F)), q.c2);
  const float2 ee = make_float2(ex2_a(tt.x), ex2_a(tt.y));
  /* one reciprocal for both quotients, den = 1 + ee: num / p4 = num den / (p4 den),
   * 1 / den = p4 / (p4 den), with p4 den = p4 + p4 ee and num den = num + num ee; the
   * segment's pmf1 multiplies the pmf sum when it is folded */
  const float2 pd = __ffma2_rn(p4, ee, p4);
  const float2 inv = make_float2(rcp_a(pd.x), rcp_a(pd.y));
  const float2 vn = __ffma2_rn(num, ee, num);
  if constexpr (PAIR) {
    a.vdw = __ffma2_rn(vn, inv, a.vdw);
    a.pmf = __ffma2_rn(p4, inv, a.pmf);
  } else {
    a.vdw.x = __fmaf_rn(vn.x, inv.x, a.vdw.x);
    a.pmf.x = __fmaf_rn(p4.x, inv.x, a.pmf.x);
  }
  }
  if (HDB) {
    const float2 h = __ffma2_rn(__fmul2_rn(d2, ri), q.hc1, q.hc0);
    const float2 hh = __fmul2_rn(h, h);
    if constexpr (PAIR)
      a.hdb = __ffma2_rn(q.hs, make_float2(ex2_a(-hh.x), ex2_a(-hh.y)), a.hdb);
    else
      a.hdb.x = __fmaf_rn(q.hs.x, ex2_a(-hh.x), a.hdb.x);
  }
}

/* Pair loop over slots [i0, i1) of one point-type segment held in shared memory; i0 is even,
 * an odd i1 leaves one point for a half iteration. HDB: the segment's point type has a live
 * hydrogen-bond pair with some atom type of the ligand (decided per complex on the host, so
 * every warp of the CTA runs the same code). UNROLL: point pairs in flight per lane. */
template <bool HDB, int UNROLL, bool FAR>
__device__ __forceinline__ void pair_range(const float4 *__restrict__ PA,
                                           const float4 *__restrict__ PB, int i0, int i1,
                                           float ax, float ay, float az, const Pair2 &q,
                                           const GdForceConst &f, Acc &a) {
  const float2 ax2 = f2(ax), ay2 = f2(ay), az2 = f2(az);
  const int m0 = i0 >> 1, m1 = i1 >> 1;
#pragma unroll UNROLL
  for (int m = m0; m < m1; ++m)
    pair_body<HDB, true, FAR>(PA[m], PB[m], ax2, ay2, az2, q, f, a);
  if (i1 & 1) pair_body<HDB, false, FAR>(PA[m1], PB[m1], ax2, ay2, az2, q, f, a);
}

/* One pair of slots of which the first n (0, 1, 2) are points of the range: the values of
 * pair_body, kept for those. */
template <bool HDB, bool FAR>
__device__ __forceinline__ void pair_body_n(const float4 A, const float4 B, float2 ax, float2 ay,
                                            float2 az, const Pair2 &q, const GdForceConst &f,
                                            Acc &a, int n) {
  Acc t = a;
  pair_body<HDB, true, FAR>(A, B, ax, ay, az, q, f, t);
  if (n > 0) {
    a.vdw.x = t.vdw.x;
    a.ele.x = t.ele.x;
    a.pmf.x = t.pmf.x;
    if (HDB) a.hdb.x = t.hdb.x;
  }
  if (n > 1) {
    a.vdw.y = t.vdw.y;
    a.ele.y = t.ele.y;
    a.pmf.y = t.pmf.y;
    if (HDB) a.hdb.y = t.hdb.y;
  }
}

/* pair_range for the split launches, where a warp has few others beside it and the latency of a
 * body counts: the points left after the whole groups of four pairs run as one more group, its
 * pairs in flight together, instead of one after the other (segments of a small pocket are some
 * seven pairs long). The slots read past the range lie in the CTA's shared memory. */
template <bool HDB, int UNROLL, bool FAR>
__device__ __forceinline__ void pair_range_lat(const float4 *__restrict__ PA,
                                               const float4 *__restrict__ PB, int i0, int i1,
                                               float ax, float ay, float az, const Pair2 &q,
                                               const GdForceConst &f, Acc &a) {
  const float2 ax2 = f2(ax), ay2 = f2(ay), az2 = f2(az);
  int m = i0 >> 1;
#pragma unroll 1
  for (; 2 * (m + UNROLL) <= i1; m += UNROLL)
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      pair_body<HDB, true, FAR>(PA[m + u], PB[m + u], ax2, ay2, az2, q, f, a);
  const int r = i1 - 2 * m;
  if (r > 0)
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      pair_body_n<HDB, FAR>(PA[m + u], PB[m + u], ax2, ay2, az2, q, f, a, r - 2 * u);
}

/* The same range for the same atom of two replicas (the lane's two slots): one load of each
 * point pair, one loop, the segment's parameters shared; each atom's sums are the operations
 * of pair_range in the same order, so its energies are bit-identical. */
template <bool HDB, int UNROLL, bool FAR>
__device__ __forceinline__ void pair_range2(const float4 *__restrict__ PA,
                                            const float4 *__restrict__ PB, int i0, int i1,
                                            const float *ax, const float *ay, const float *az,
                                            const Pair2 &q, const GdForceConst &f, Acc *a) {
  const float2 ax0 = f2(ax[0]), ay0 = f2(ay[0]), az0 = f2(az[0]);
  const float2 ax1 = f2(ax[1]), ay1 = f2(ay[1]), az1 = f2(az[1]);
  const int m0 = i0 >> 1, m1 = i1 >> 1;
#pragma unroll UNROLL
  for (int m = m0; m < m1; ++m) {
    const float4 A = PA[m], B = PB[m];
    pair_body<HDB, true, FAR>(A, B, ax0, ay0, az0, q, f, a[0]);
    pair_body<HDB, true, FAR>(A, B, ax1, ay1, az1, q, f, a[1]);
  }
  if (i1 & 1) {
    const float4 A = PA[m1], B = PB[m1];
    pair_body<HDB, false, FAR>(A, B, ax0, ay0, az0, q, f, a[0]);
    pair_body<HDB, false, FAR>(A, B, ax1, ay1, az1, q, f, a[1]);
  }
}

/* Sums of the short-range terms of one atom. */
struct ShortSums {
  double hsum;                /* sum of hpp * switch(d^2) over hydrophobic points, d^2 <= 81 */
  float psp;                  /* sum of the PSP entries of class-2 points in contact */
  float ele;                  /* soft-core minus far-form electrostatics, d^2 < (1 / el1)^2 */
  int ncon;                   /* contacts: d^2 <= the pair's contact threshold */
};

/* The terms of CalcEnergy_d that only pairs within a few angstrom have (contacts for mcc and
 * psp, hpc's switching polynomial, the soft core of ele), for one atom at (ax, ay, az), from
 * the conformer's cell list: the rows of cells (fixed y, z) that reach within sr_r of the
 * atom, each over the x range the remaining radius allows, so every point with
 * d^2 <= sr_r2 is visited once and the tests use the same d^2 as the pair loop. The next
 * row's bounds are read while the current row runs. thr: the contact thresholds of the atom's
 * type against every point type (shared memory). */
__device__ __forceinline__ void short_range(const GdDevComplex &cx, int pc,
                                            const float *__restrict__ thr,
                                            const float *__restrict__ psprow,
                                            const GdForceConst &f, float ax, float ay, float az,
                                            ShortSums &s) {
  const int nx = cx.sr_n[0], ny = cx.sr_n[1], nz = cx.sr_n[2];
  const float R = cx.sr_r, R2 = cx.sr_r * cx.sr_r, ic = cx.sr_inv_cell, e = cx.sr_cell;
  const float r2max = cx.sr_r2;
  const float ox = cx.sr_org[0], oy = cx.sr_org[1], oz = cx.sr_org[2];
  const int y0 = max(0, (int)floorf((ay - R - oy) * ic));
  const int y1 = min(ny - 1, (int)floorf((ay + R - oy) * ic));
  const int z0 = max(0, (int)floorf((az - R - oz) * ic));
  const int z1 = min(nz - 1, (int)floorf((az + R - oz) * ic));
  if (y0 > y1 || z0 > z1) return;
  const int *__restrict__ st = cx.sr_start + (size_t)pc * (cx.sr_n[3] + 1);
  const float4 *__restrict__ PA = cx.sr_a + (size_t)pc * (cx.pnp + 1);
  const float4 *__restrict__ PB = cx.sr_b + (size_t)pc * (cx.pnp + 1);
  /* point range of row (iy, iz) within the remaining radius; empty when out of reach */
  auto bounds = [&](int iy, int iz, int &b0, int &b1) {
    b0 = b1 = 0;
    const float zl = oz + (float)iz * e, yl = oy + (float)iy * e;
    const float gz = fmaxf(0.0f, fmaxf(zl - az, az - (zl + e)));
    const float gy = fmaxf(0.0f, fmaxf(yl - ay, ay - (yl + e)));
    const float rem = R2 - gy * gy - gz * gz;
    if (rem < 0.0f) return;
    const float hx = sqrtf(rem);
    const int x0 = max(0, (int)floorf((ax - hx - ox) * ic));
    const int x1 = min(nx - 1, (int)floorf((ax + hx - ox) * ic));
    if (x0 > x1) return;
    const int row = (iz * ny + iy) * nx;
    b0 = __ldg(st + row + x0);
    b1 = __ldg(st + row + x1 + 1);
  };
  int iy = y0, iz = z0, n0 = 0, n1 = 0;
  bool more = true;
  bounds(iy, iz, n0, n1);
  while (more) {
    const int c0 = n0, c1 = n1;
    if (++iy > y1) {
      iy = y0;
      ++iz;
    }
    more = iz <= z1;
    if (more) bounds(iy, iz, n0, n1);
    for (int i = c0; i < c1; ++i) {
      const float4 p = __ldg(PA + i);
      const float d2 = dist2(ax, ay, az, p.x, p.y, p.z);
      if (d2 > r2max) continue;
      const int meta = __float_as_int(p.w);
      const bool hpc = (meta & 256) && d2 <= 81.0f;
      const bool con = d2 <= thr[meta & 255];
      const bool cls2 = con && (meta & 512);
      const bool near = d2 < f.near2;
      s.ncon += con ? 1 : 0;
      if (hpc || cls2 || near) {
        const float4 b = __ldg(PB + i);
        if (hpc) {
          float t = __fmaf_rn(d2, HPC_C4, -HPC_C3);
          t = __fmaf_rn(d2, t, HPC_C2);
          t = __fmaf_rn(d2, t, -HPC_C1);
          s.hsum += (double)__fmul_rn(b.x, __fmaf_rn(d2, t, 1.0f));
        }
        if (cls2) s.psp += __ldg(psprow + __float_as_int(b.y));
        if (near) {
          const float ri = rsqrt_a(d2);
          const float s1 = __fmul_rn(f.el1, __fmul_rn(d2, ri));
          const float gn = __fmaf_rn(__fmul_rn(s1, s1), __fmaf_rn(f.b1, s1, f.a1), f.el0);
          /* ep (el1 gn) - ep ri = ele_p gn - ele_p g_far */
          s.ele += __fmaf_rn(b.z * f.el1, gn, -(b.z * ri));
        }
      }
    }
  }
}

/* The same terms for an atom inside the pocket grid, from its cell's two point lists
 * (gd_pocket.cu), the contact list (con), the kind list (kind) or both: the same points' terms
 * added in the same order as short_range. Bound by the latency of a load per point: four points
 * are in flight, and a point past the end of a list is the sentinel. A warp's pass went from
 * 87-135 k cycles (the row walk) to 20-34 k: 6,820 replicas of 40 atoms on 3,000 points, 11 steps,
 * 11.75 -> 9.64 ms with the epilogue's changes. */
__device__ __forceinline__ void short_range_lists(const GdDevComplex &cx, int pc, int cell,
                                                  const float *__restrict__ thr,
                                                  const float *__restrict__ psprow,
                                                  const GdForceConst &f, float ax, float ay,
                                                  float az, bool con, bool kind, ShortSums &s) {
  const int *__restrict__ st = cx.pg_start + (size_t)pc * (2 * GD_PG_CELLS + 1) + 2 * cell;
  const int s0 = __ldg(st), s1 = __ldg(st + 1), s2 = __ldg(st + 2);
  const ushort4 *__restrict__ ix =
      reinterpret_cast<const ushort4 *>(cx.pg_idx + __ldg(cx.pg_base + pc));
  const float4 *__restrict__ PA = cx.sr_a + (size_t)pc * (cx.pnp + 1);
  const float4 *__restrict__ PB = cx.sr_b + (size_t)pc * (cx.pnp + 1);
  for (int i = s0 >> 2; con && i < (s1 >> 2); ++i) {
    const ushort4 id = __ldg(ix + i);
    const int k[4] = {id.x, id.y, id.z, id.w};
    float4 p[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) p[u] = __ldg(PA + k[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float d2 = dist2(ax, ay, az, p[u].x, p[u].y, p[u].z);
      s.ncon += d2 <= thr[__float_as_int(p[u].w) & 255] ? 1 : 0;
      if (d2 < f.near2) {
        const float e = __ldg(&PB[k[u]].z);
        const float ri = rsqrt_a(d2);
        const float s1_ = __fmul_rn(f.el1, __fmul_rn(d2, ri));
        const float gn = __fmaf_rn(__fmul_rn(s1_, s1_), __fmaf_rn(f.b1, s1_, f.a1), f.el0);
        /* ep (el1 gn) - ep ri = ele_p gn - ele_p g_far */
        s.ele += __fmaf_rn(e * f.el1, gn, -(e * ri));
      }
    }
  }
  for (int i = s1 >> 2; kind && i < (s2 >> 2); ++i) {
    const ushort4 id = __ldg(ix + i);
    const int k[4] = {id.x, id.y, id.z, id.w};
    float4 p[4];
    float2 b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      p[u] = __ldg(PA + k[u]);
      b[u] = __ldg(reinterpret_cast<const float2 *>(PB + k[u]));
    }
    float ps[4];
    double h[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float d2 = dist2(ax, ay, az, p[u].x, p[u].y, p[u].z);
      const int meta = __float_as_int(p[u].w);
      float t = __fmaf_rn(d2, HPC_C4, -HPC_C3);
      t = __fmaf_rn(d2, t, HPC_C2);
      t = __fmaf_rn(d2, t, -HPC_C1);
      t = __fmul_rn(b[u].x, __fmaf_rn(d2, t, 1.0f));
      h[u] = (meta & 256) && d2 <= 81.0f ? (double)t : 0.0;
      ps[u] = (meta & 512) && d2 <= thr[meta & 255] ? __ldg(psprow + __float_as_int(b[u].y))
                                                    : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s.hsum += h[u];
      s.psp += ps[u];
    }
  }
}

/* The pocket-grid cell of a position, -1 outside the grid (a NaN position is outside). */
__device__ __forceinline__ int pocket_cell(const GdDevComplex &cx, float x, float y, float z) {
  const float inv = 1.0f / GD_PG_EDGE;
  const float fx = floorf((x - cx.pg_org[0]) * inv), fy = floorf((y - cx.pg_org[1]) * inv),
              fz = floorf((z - cx.pg_org[2]) * inv);
  const float n = (float)GD_PG_N;
  if (!(fx >= 0.0f && fx < n && fy >= 0.0f && fy < n && fz >= 0.0f && fz < n)) return -1;
  return ((int)fz * GD_PG_N + (int)fy) * GD_PG_N + (int)fx;
}

/* A float4 of the far-field tables: read once per atom and step, kept out of L1, which holds the
 * point lists. */
__device__ __forceinline__ float4 ldg_stream(const float4 *p) {
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p));
  return v;
}

/* The far points' ele and vdw sums at (x, y, z) of a tabulated cell (gd_farfield.cu): two
 * Chebyshev series of total degree 4 in the cell's coordinates, about 110 FMAs and 18 loads from
 * L2, for what the pair loop spent on more than half of 3,000 points. */
__device__ __forceinline__ void far_field(const GdDevComplex &cx, int pc, int cell, int id, int tl,
                                          float x, float y, float z, float &ele, float &vdw) {
  const float4 *te = reinterpret_cast<const float4 *>(
      cx.ff_tab + ((size_t)pc * cx.ff_cells + id) * cx.ff_fields * GD_FF_NC);
  const float4 *tv = te + (1 + cx.ff_slot[tl]) * (GD_FF_NC / 4);
  const int ix = cell % GD_FF_N, iy = (cell / GD_FF_N) % GD_FF_N, iz = cell / (GD_FF_N * GD_FF_N);
  const float s = 2.0f / GD_FF_EDGE;
  const float u = (x - cx.pocket[0]) * s - (float)(2 * ix + 1 - GD_FF_N),
              v = (y - cx.pocket[1]) * s - (float)(2 * iy + 1 - GD_FF_N),
              w = (z - cx.pocket[2]) * s - (float)(2 * iz + 1 - GD_FF_N);
  constexpr int N = GD_FF_DEG + 1;
  static_assert(GD_FF_NC % 4 == 0, "whole float4 per series");
  float tu[N], tw[N];
  tu[0] = tw[0] = 1.0f;
  tu[1] = u;
  tw[1] = w;
#pragma unroll
  for (int i = 2; i < N; ++i) {
    tu[i] = 2.0f * u * tu[i - 1] - tu[i - 2];
    tw[i] = 2.0f * w * tw[i - 1] - tw[i - 2];
  }
  ele = vdw = 0.0f;
  float4 ce, cv;
  int n = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    float ek = 0.0f, vk = 0.0f, t0 = 1.0f, t1 = v;
#pragma unroll
    for (int j = 0; j < N - k; ++j) {
      float ej = 0.0f, vj = 0.0f;
#pragma unroll
      for (int i = 0; i < N - k - j; ++i, ++n) {
        if ((n & 3) == 0) {
          ce = ldg_stream(te + (n >> 2));
          cv = ldg_stream(tv + (n >> 2));
        }
        const float a = (n & 3) == 0 ? ce.x : (n & 3) == 1 ? ce.y : (n & 3) == 2 ? ce.z : ce.w;
        const float b = (n & 3) == 0 ? cv.x : (n & 3) == 1 ? cv.y : (n & 3) == 2 ? cv.z : cv.w;
        ej = __fmaf_rn(a, tu[i], ej);
        vj = __fmaf_rn(b, tu[i], vj);
      }
      ek = __fmaf_rn(ej, t0, ek);
      vk = __fmaf_rn(vj, t0, vk);
      const float t2 = 2.0f * v * t1 - t0;
      t0 = t1;
      t1 = t2;
    }
    ele = __fmaf_rn(ek, tw[k], ele);
    vdw = __fmaf_rn(vk, tw[k], vdw);
  }
}

/* Per-replica state of the CTA's slots, in shared memory. */
struct Slot {
  int rep, lig_conf, accept, n_acc;
  int rec_next;
  float mag; /* e_old's terms (cert_mag) */
  float mb, u;
  float mm_old[6];
  float mm_new[6];
  float rot[9];
  float tx, ty, tz;
  gd_energy e_old;
  gd_replica replica;
  /* a decision too close to take from the fields' energies: the proposal's energies, and its total
   * by the pair loop over every point */
  gd_energy e_prop;
  float e_full;
  float cert; /* ff_cert of both poses */
  int open;
};
static_assert(sizeof(Slot) == GD_SLOT_BYTES, "slot layout");

/* Whether the slot's replica, or a proposal one root-mean-square move from it, lies GD_ROAM or more
 * from the pocket centre. */
__device__ __forceinline__ bool slot_roams(const GdMcArgs &a, const GdDevComplex &cx,
                                           const Slot &s, int id) {
  float v[3], step2 = 0.0f, d2 = 0.0f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    v[i] = a.mode == 4 ? a.center_in[(size_t)id * 3 + i]
                       : cx.lig_center[s.lig_conf * 3 + i] +
                             (a.mode >= 2 ? a.mm_in[(size_t)id * 6 + i] : s.mm_old[i]);
    d2 += (v[i] - cx.pocket[i]) * (v[i] - cx.pocket[i]);
    step2 += a.mode == 0 ? a.move_scale[i] * a.move_scale[i] : 0.0f;
  }
  return sqrtf(d2) + sqrtf(step2) > GD_ROAM;
}

#define NQ 10 /* vdw ele pmf psp hdb hsum->hpc kde rmsd ncon tp */
#define MCS_U 4 /* restraint positions in flight in the epilogue */

/* MCS position restraints of one replica's atoms, sum over positions of tcc rmsd (every lane of the
 * warp returns it): MCS_U positions at a time, so that their loads and shuffles overlap, and the
 * square roots of up to 32 positions at once, one per lane (one position after the other they took
 * 20-29 k cycles a step at 8-11 positions, with lane 0's square roots 8-10 k). */
__device__ __forceinline__ double restraints(const GdDevComplex &cx, int lig_conf, int L,
                                             const float4 *atoms, int lane) {
  double elhm = 0.0;
  const int *meta_y = &cx.lig_meta[lig_conf * L].y;
#pragma unroll 1
  for (int mb = 0; mb < cx.pos; mb += 32) {
    const int me = min(cx.pos, mb + 32);
    double mine = 0.0; /* lane's position mb + lane: squared distances, atoms */
    unsigned mine_n = 0;
#pragma unroll 1
    for (int m0 = mb; m0 < me; m0 += MCS_U) {
      double sm[MCS_U];
      unsigned cnt = 0; /* the positions' atom counts (<= GD_MAXLIG), 8 bits each */
#pragma unroll
      for (int u = 0; u < MCS_U; ++u) sm[u] = 0.0;
      for (int i = lane; i < L; i += 32) {
        const int idx = __ldg(meta_y + 2 * i);
        const float4 at = atoms[i];
#pragma unroll
        for (int u = 0; u < MCS_U; ++u) {
          const int m = min(m0 + u, cx.pos - 1);
          const float4 r = __ldg(cx.mcs + (size_t)m * cx.mcs_ld + idx);
          if (r.x != GD_MCS_INVALID_COORD) {
            const float dx = at.x - r.x, dy = at.y - r.y, dz = at.z - r.z;
            sm[u] += (double)(dx * dx + dy * dy + dz * dz);
            cnt += 1u << (8 * u);
          }
        }
      }
      cnt = __reduce_add_sync(0xffffffffu, cnt);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < MCS_U; ++u) sm[u] += __shfl_down_sync(0xffffffffu, sm[u], o);
#pragma unroll
      for (int u = 0; u < MCS_U; ++u) {
        const double v = __shfl_sync(0xffffffffu, sm[u], 0);
        if (mb + lane == m0 + u) {
          mine = v;
          mine_n = (cnt >> (8 * u)) & 255u;
        }
      }
    }
    double tcc = 0.0, root = 0.0;
    if (mb + lane < me && mine_n) {
      tcc = (double)cx.mcs_tcc[mb + lane];
      root = sqrt(mine / (double)mine_n);
    }
    /* added in position order */
    for (int m = mb; m < me; ++m)
      elhm += __shfl_sync(0xffffffffu, tcc, m - mb) * __shfl_sync(0xffffffffu, root, m - mb);
  }
  return elhm;
}

/* One segment range of the pair loop, dispatched on the segment's flags (bit 2: live
 * hydrogen-bond term). */
template <int UNROLL, int PACK, bool FAR, bool LAT = false>
__device__ __forceinline__ void pair_dispatch(int flags, const float4 *PA, const float4 *PB,
                                              int i0, int i1, const float *ax, const float *ay,
                                              const float *az, const Pair2 &pq,
                                              const GdForceConst &f, Acc *acc) {
#define GD_PR(H)                                                                             \
  if constexpr (PACK == 2)                                                                   \
    pair_range2<H, UNROLL, FAR>(PA, PB, i0, i1, ax, ay, az, pq, f, acc);                     \
  else if constexpr (LAT)                                                                    \
    pair_range_lat<H, UNROLL, FAR>(PA, PB, i0, i1, ax[0], ay[0], az[0], pq, f, acc[0]);      \
  else                                                                                       \
    pair_range<H, UNROLL, FAR>(PA, PB, i0, i1, ax[0], ay[0], az[0], pq, f, acc[0])
  if (flags & 4) {
    GD_PR(true);
  } else {
    GD_PR(false);
  }
#undef GD_PR
}

/* The magnitudes of an energy's weighted terms, which its far fields' rounding is a share of. */
__device__ __forceinline__ float cert_mag(const gd_energy &e, const GdForceConst &f) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < GD_MAXWEI - 1; ++i) m += fabsf(e.e[i] * f.w[i]);
  return m;
}

/* ExchangeReplicas_d (src/kernel_cuda_l1_exchangereplicas.cu:27-77) for one (protein
 * conformer, ligand conformer) group lg of complex cx: temperature pairs (2 j + mode_t, its
 * successor), accepted by the Metropolis test on their energies with one Philox draw per pair
 * of this exchange call. The group's replica states are read with L2 loads (.cg): inside the
 * Monte Carlo kernel other SMs wrote them in this launch.
 * Where energies come from far fields, a group with a pair whose decision could hang on their
 * rounding is left as it is: the result is nonzero, and list gets the temperature indexes of such
 * pairs' replicas, two a pair. With their energies by the pair loop in full[] (by temperature index)
 * those pairs decide on them. */
__device__ __forceinline__ unsigned gd_exchange_group(const GdDevComplex &cx, int lg,
                                                      const GdExchange &x, const GdForceConst &f,
                                                      int call, int mode_t,
                                                      const float *full = nullptr,
                                                      int *list = nullptr) {
  if (mode_t >= 2) return 0;
  const int nl = cx.n_lig, nt = cx.n_tmp;
  const int p = lg / nl, l = lg - p * nl, r0 = cx.rep_offset + nt * nl * p + l;
  const bool certify = cx.ff_tab != nullptr;
  const float cert = certify ? cx.ff_cert[lg] : 0.0f; /* lg = p n_lig + l */
  short temps[GD_MAXTMP], orders[GD_MAXTMP];
  float en[GD_MAXTMP], tol[GD_MAXTMP];
  for (int t = 0; t < nt; ++t) {
    const int r = r0 + nl * t;
    temps[t] = (short)__ldcg(&x.replica[r].idx_tmp);
    en[t] = __ldcg(x.etotal + r);
    orders[temps[t]] = (short)t;
    if (certify) {
      gd_energy e;
#pragma unroll
      for (int i = 0; i < GD_MAXWEI - 1; ++i) e.e[i] = __ldcg(&x.e_old[r].e[i]);
      tol[t] = GD_CERT * cert_mag(e, f) + cert;
    }
  }
  const int maxpair = nt / 2 - (nt % 2 == 0) * (mode_t == 1);
  unsigned taken = 0, open = 0;
  int n = 0;
  for (int pair = 0; pair < maxpair; ++pair) {
    const int i1 = (pair << 1) + mode_t, i2 = i1 + 1;
    const int o1 = orders[i1], o2 = orders[i2];
    const float mb1 = cx.minus_beta[temps[o1]], mb2 = cx.minus_beta[temps[o2]];
    const float u = gd_draw_exchange(x.seed, (uint32_t)cx.stream, (uint32_t)lg, (uint32_t)call,
                                     (uint32_t)pair);
    int acc = gd_exchange_accept(en[o1], en[o2], mb1, mb2, u);
    if (certify) {
      const float d = tol[o1] + tol[o2];
      if (gd_exchange_accept(en[o1], en[o2] + d, mb1, mb2, u) !=
          gd_exchange_accept(en[o1], en[o2] - d, mb1, mb2, u)) {
        if (full) {
          acc = gd_exchange_accept(full[o1], full[o2], mb1, mb2, u);
        } else {
          open |= 1u << pair;
          if (list) {
            list[n++] = o1;
            list[n++] = o2;
          }
        }
      }
    }
    if (acc) {
      const short tt = temps[o1];
      temps[o1] = temps[o2];
      temps[o2] = tt;
      taken |= 1u << pair;
    }
  }
  if (open) return open;
  /* (counts without a result: a load and a store each, one after the other, kept the thread up to
   * 3 us) */
  for (int pair = 0; pair < maxpair; ++pair)
    if ((taken >> pair) & 1u) {
      atomicAdd(x.acs + r0 + nl * orders[(pair << 1) + mode_t], 1);
      atomicAdd(x.acs + r0 + nl * orders[(pair << 1) + mode_t + 1], 1);
    }
  for (int t = 0; t < nt; ++t) x.replica[r0 + nl * t].idx_tmp = temps[t];
  return 0;
}

/* Lists a group for the launch that decides it. The list holds every group once; it is full only
 * when such a launch did not take place. */
__device__ __forceinline__ void open_group(int *open, int *list, int cap, int g, unsigned *err) {
  const int i = atomicAdd(open, 1);
  if (i < cap)
    list[i] = g;
  else
    atomicOr(err, GD_DEV_ERR_TIMEOUT);
}

/* Delayed acceptance, second stage, for the survivor in pose slot `pos` (mode 3): the
 * corrected Metropolis test u2 < exp(mb ((E_new - E_old) - (S_new - S_cur))) (gd_da_stage2)
 * on the energies ea and eb, surrogate-error sums, the collect step's training target, the trace,
 * and on acceptance the state update and the record, as the plain epilogue does them. tol > 0:
 * nothing is done, and the result is false, when the decision is not the same that much above and
 * below ea. */
__device__ __forceinline__ bool da_decide(const GdMcArgs &a, const GdDevComplex &cx, int ci, int pos,
                                          const gd_energy &en, float ea, float eb, float tol,
                                          const float *mm_new, int step) {
  const GdDaEpi &da = *a.da;
  const int r = da.pose_rep[pos];
  const gd_replica rp = a.replica[r];
  const float mb = cx.minus_beta[rp.idx_tmp];
  const float enew = en.e[GD_MAXWEI - 1];
  const float sn = da.s_new[r], so = da.s_cur[r], u2 = da.u2[r];
  const int acc = gd_da_stage2(ea, eb, sn, so, mb, u2);
  if (tol > 0.0f && gd_da_stage2(ea + tol, eb, sn, so, mb, u2) !=
                        gd_da_stage2(ea - tol, eb, sn, so, mb, u2))
    return false;
  const bool active = !a.da_collect && da.active[ci];
  if (active) {
    const double e = (double)sn - (double)enew;
    da.err2[r] += e * e;
    da.nerr[r] += 1;
  }
  if (a.da_collect && da.smp_cap > 0)
    da.smp_t[((long long)step * da.n_rep + r) % da.smp_cap] = enew;
  if (da.tr_flag) {
    const int ti = step - da.tr_step0;
    if (ti >= 0 && ti < da.tr_cap) {
      const size_t o = (size_t)r * da.tr_cap + ti;
      da.tr_s[o] = sn;
      da.tr_e[o] = enew;
      da.tr_flag[o] = 1 + acc;
    }
  }
  if (!acc) return true;
  a.e_old[r] = en;
  a.etotal[r] = enew;
#pragma unroll
  for (int i = 0; i < 6; ++i) a.mm_old[(size_t)r * 6 + i] = mm_new[i];
  a.n_accept[r] += 1;
  da.s_cur[r] = sn;
  if (active) da.acc[r] += 1; else da.plain_acc[r] += 1;
  if (a.rec) {
    const int kslot = a.rec_next[r];
    if (kslot < a.rec_cap) {
      gd_record_step *q = a.rec + (size_t)r * a.rec_cap + kslot;
      q->replica = rp;
      q->energy = en;
#pragma unroll
      for (int i = 0; i < 6; ++i) q->movematrix[i] = mm_new[i];
      q->step = step;
      a.rec_next[r] = kslot + 1;
    } else {
      atomicOr(a.err, GD_DEV_ERR_RECORD_FULL);
    }
  }
  return true;
}

/*
 * Shared memory: two mbarriers, two protein buffers of D points (float4 + float2), the
 * placed atoms, NQ FP64 partials per lane, the slots. The protein buffers form a two-stage
 * ring without CTA barriers: every warp waits on the buffer's "full" mbarrier by itself and,
 * when done, bumps the buffer's counter; the last warp to finish refills the buffer with the
 * chunk two ahead. Every wait is bounded (globaltimer); a wait that runs out sets the error
 * word, the CTA leaves at the next step barrier after letting its copies in flight land.
 */
template <int UNROLL, int SPLITS, int KIND, int PACK>
__global__ void __launch_bounds__(SPLITS ? GD_MAX_TPB_SPLIT : GD_MAX_TPB / PACK,
                                  SPLITS ? 1 : GD_MIN_BLOCKS_PACK(UNROLL, PACK, KIND != GD_KIND_PLAIN))
    gd_mc_kernel(GdMcArgs a, GdForceConst f) {
  constexpr bool SPLIT = SPLITS != GD_UNSPLIT, ordered = SPLITS == GD_SPLIT_ORDERED;
  constexpr bool DA = KIND == GD_KIND_DA, XCH = KIND == GD_KIND_EXCHANGE;
  static_assert(PACK == 1 || (PACK == 2 && !SPLIT && KIND == GD_KIND_PLAIN),
                "two replicas per lane: plain modes with one lane per atom");
  if (XCH && __ldcg(a.x_open) == 0) return; /* the usual case: no group is open */
  extern __shared__ __align__(16) unsigned char smem[];
  /* Sums in the points' order (ordered): the splits run contiguous ranges of segments; split 0 adds
   * its own up as the unsplit lanes do, the others store theirs piece by piece, and the pieces are
   * then added in order. The result is the unsplit launch's, bit for bit; otherwise each split has
   * partial sums, added in split order. */
  /* T: the stride of the placed atoms and partials: the tile's lanes (PACK per thread), of one split
   * when ordered */
  const int NT = blockDim.x, T = ordered ? NT / a.split : NT * PACK, tid = threadIdx.x, D = a.chunk;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
  /* contact thresholds [ligand type][point type], then the ring buffers: buffer b holds D
   * slots as D/2 pairs in two float4 streams */
  float *thr_s = reinterpret_cast<float *>(smem + 16);
  float4 *bpa = reinterpret_cast<float4 *>(smem + 16 + GD_THR_BYTES);
  float4 *bpb = bpa + D;
  float4 *atoms = bpb + D;
  double *part = reinterpret_cast<double *>(atoms + T);
  /* the stored pieces: three planes each (vdw, ele, pmf), then the hydrogen-bond pieces */
  double *pcs = part + NQ * T;
  const int n_planes = ordered ? 3 * a.pieces + a.hpieces : 0;
  Slot *slots = reinterpret_cast<Slot *>(pcs + n_planes * T);
  __shared__ int s_tile, s_abort, s_open;
  __shared__ int s_done[2];
  __shared__ unsigned s_issued[2];
  __shared__ double s_lhm[SPLIT ? GD_MAX_SLOTS : 1]; /* the slots' restraint sums */
  __shared__ double s_norm[3][GD_MAXWEI];            /* a_para, b_para, w */

  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = 0;
    s_open = 0;
    s_done[0] = s_done[1] = 0;
    s_issued[0] = s_issued[1] = 0;
  }
  for (int i = tid; i < GD_MAXTP2 * GD_MAXTP1; i += NT) thr_s[i] = a.pp[i].thr;
#pragma unroll
  for (int i = 0; i < GD_MAXWEI; ++i)
    if (tid == i) {
      s_norm[0][i] = (double)f.a_para[i];
      s_norm[1][i] = (double)f.b_para[i];
      s_norm[2][i] = (double)f.w[i];
    }
  __syncthreads();
  uint32_t consumed0 = 0, consumed1 = 0; /* completed phases waited for, per buffer */
  const int step_first = a.step0 + (a.step_base ? *a.step_base : 0);
  const int warp = tid >> 5, lane = tid & 31, nwarps = NT >> 5;
  if (DA && a.mode == 3 && blockIdx.x == 0)
    for (int g = a.da_g0 + tid; g < a.da_g1; g += NT) a.da_cnt_next[g] = 0;

  /* the open exchange groups (XCH): this CTA's xg-th, whose replicas x_list[xb .. xn) (temperature
   * indexes) are still to be evaluated, their energies going to x_e */
  __shared__ int x_list[XCH ? GD_MAXTMP : 1], x_n;
  __shared__ float x_e[XCH ? GD_MAXTMP : 1];
  int xg = (int)blockIdx.x - (int)gridDim.x, xb = 0, xn = 0, x_ci = 0, x_lg = 0;
  bool x_has = false;
  const int x_count = XCH ? min(__ldcg(a.x_open), a.x_open_cap) : 0;
  const int x_mode = !XCH ? 0
                     : a.x_mode_t >= 0 ? a.x_mode_t
                                       : !(((step_first % a.x_spd) / a.x_spe) % 2);

  for (;;) {
    int t = 0;
    GdTileDesc tile;
    if constexpr (XCH) {
      if (xb >= xn) {
        const GdExchange ex = {a.replica, a.etotal, a.e_old, a.x_acs, a.seed};
        const int call = (a.x_call_base ? *a.x_call_base : 0) + a.x_call_off;
        /* every replica of the group is evaluated: its pairs decide */
        if (tid == 0 && x_has) gd_exchange_group(a.cx[x_ci], x_lg, ex, f, call, x_mode, x_e);
        x_has = false;
        xg += (int)gridDim.x;
        if (xg >= x_count || s_abort) break;
        const int g = a.x_open_list[xg];
        int hi = a.n_complex - 1;
        x_ci = 0;
        while (x_ci < hi) {
          const int mid = (x_ci + hi + 1) >> 1;
          if (a.x_group_base[mid] <= g) x_ci = mid; else hi = mid - 1;
        }
        x_lg = g - a.x_group_base[x_ci];
        if (tid == 0)
          x_n = 2 * __popc(gd_exchange_group(a.cx[x_ci], x_lg, ex, f, call, x_mode, nullptr,
                                             x_list));
        __syncthreads();
        x_has = x_n > 0;
        xn = x_n;
        xb = 0;
        __syncthreads(); /* x_n is read before the next group's is written */
        if (!x_has) continue;
      }
      t = xg;
      tile = {x_ci, x_lg / a.cx[x_ci].n_lig, 0, min(min(a.u.count, T / a.cx[x_ci].lna), xn - xb)};
    } else {
      if (tid == 0) s_tile = atomicAdd(a.tile_counter, 1);
      __syncthreads();
      t = s_tile;
      if (t >= a.n_tiles || s_abort) break;
      if (a.tiles) {
        tile = a.tiles[t];
      } else {
        tile = a.u;
        tile.rep_begin = t * a.u.count;
        tile.count = min(a.u.count, a.u_n - tile.rep_begin);
      }
    }
    int k = tile.count;
    if (DA && a.mode == 3) {
      /* slot (group, capacity): the survivors of the group past this tile's first slot */
      const int g = tile.count >> 8, cap = tile.count & 255;
      k = max(0, min(cap, a.da_cnt[g] - (tile.rep_begin - a.da->group_b0[g])));
    }
    if (k <= 0) {
      /* an empty tile (a delayed-acceptance block with fewer survivors than tiles): no copy
       * issued, nothing to wait for; the barrier keeps s_tile until every thread read it */
      __syncthreads();
      continue;
    }
    const GdDevComplex &cx = a.cx[tile.complex_index];
    /* lane = (split sp, slot j, ligand atom l): the S copies of an atom, in different warps (A
     * lanes, whole warps, per split), each run some of the protein's segments and some of the
     * other per-atom terms; S = 1 is one lane per atom */
    const int L = cx.lna, S = SPLIT ? a.split : 1;
    const int A = SPLIT ? NT / S : T;
    const int kp = (k + PACK - 1) / PACK; /* lane groups */
    const int sp = SPLIT ? tid / A : 0;
    /* Unsplit lanes of a tile whose replicas are all at the pocket run over the atoms' ranks by
     * distance from the ligand's centre, the tile's slots within a rank: a warp's atoms lie about
     * as far out, so that its inner warps end their segments early (a warp runs to the largest near
     * radius among its atoms): 6,820 replicas of 40 atoms on 3,000 points, 11 steps from the
     * pocket, 7.24 -> 6.79 ms; of 60 atoms on 1,500 points, 20 steps, 15.8 -> 15.3 ms. One replica
     * further away (GD_ROAM) would make every warp of the CTA run about as far as its atoms need:
     * then each slot's atoms lie together, in the chain's order, whose neighbours share list
     * entries. The 6,820 replicas after 1,000 steps, by rank / by slot / as chosen, ms per 10
     * steps: moves of 0.1 A 6.60 / 6.76 / 6.56, of 2 A 9.33 / 8.36 / 8.38, of 6 A 10.66 / 9.97 /
     * 9.93 (six replicas a CTA and four pairs in flight 9.86 / 9.24 / 9.22); lines at 8 and 11 A
     * and at the ligand's radius are up to 3 % slower at 2 A. Delayed acceptance's tiles, of one
     * step each, keep to the ranks (by slot 28.9 -> 30.2 ms for 50 steps at 0.1 A). The warps'
     * place in the CTA goes round with the tile, so that the tiles an SM holds (about GD_NUM_SMS
     * apart) load its four schedulers alike. Split lanes keep the slots' order (2 % faster there). */
    const int wr = SPLIT ? warp - sp * (A >> 5) : (warp + t + t / GD_NUM_SMS) % nwarps;
    const int ai = wr * 32 + lane;
    const bool active = ai < kp * L;
    int jj = 0, rank = 0;
    auto take_lane = [&](bool by_slot) {
      const int n = by_slot ? L : kp, hi = active ? ai / n : 0, lo = active ? ai - hi * n : 0;
      jj = by_slot ? hi : lo;
      rank = by_slot ? lo : hi;
    };
    take_lane(SPLIT);
    /* the splits that run the short-range lists, the restraints and the per-atom tail (split 0: the
     * far field; with it, where sums run in order, the contact list, whose ele term comes first) */
    const int con_sp = ordered ? 0 : S - 1, tail_sp = ordered ? S - 1 : 0;
    const int kind_sp = ordered && S < 3 ? S - 1 : max(S - 2, 0);
    const int mcs_sp = S >= 4 ? S - 3 : ordered ? S - 1 : S == 2 ? 1 : 0;
    /* ---- slot set-up (one thread per replica) ---- */
    bool roams = false;
    if (tid < k) {
      Slot &s = slots[tid];
      const int id = XCH ? cx.rep_offset + cx.n_lig * (cx.n_tmp * tile.prt_conf + x_list[xb + tid]) +
                               x_lg % cx.n_lig
                         : tile.rep_begin + tid;
      s.rep = id;
      s.accept = 0;
      s.open = 0;
      s.cert = 0.0f;
      if (XCH) {
        s.lig_conf = a.replica[id].idx_lig;
      } else if (a.mode >= 2) {
        s.lig_conf = a.tiles ? a.lig_conf_in[id] : a.u.rep_begin;
        if (DA)
#pragma unroll
          for (int i = 0; i < 6; ++i) s.mm_old[i] = 0.0f; /* a slot left open: its replica's pose */
      } else {
        s.replica = a.replica[id];
        s.lig_conf = s.replica.idx_lig;
        s.mb = cx.minus_beta[s.replica.idx_tmp];
        if (a.mode == 0) {
          s.e_old = a.e_old[id];
          s.mag = cert_mag(s.e_old, f);
          s.n_acc = a.n_accept[id];
          s.rec_next = a.rec ? a.rec_next[id] : 0;
#pragma unroll
          for (int i = 0; i < 6; ++i) s.mm_old[i] = a.mm_old[(size_t)id * 6 + i];
        } else {
          s.n_acc = 0;
          s.rec_next = 0;
#pragma unroll
          for (int i = 0; i < 6; ++i) s.mm_old[i] = 0.0f;
        }
      }
      if (cx.ff_tab) s.cert = 2.0f * cx.ff_cert[tile.prt_conf * cx.n_lig + s.lig_conf];
      if constexpr (!SPLIT && KIND == GD_KIND_PLAIN) roams = slot_roams(a, cx, s, id);
    }

    /* ---- protein tile pipeline ---- */
    const int pc = tile.prt_conf;
    const size_t pbase = (size_t)pc * (cx.pnp_pad >> 1);
    const float4 *ga = cx.pt_a + pbase, *gb = cx.pt_b + pbase;
    const int P = cx.pnp, pnp_pad = cx.pnp_pad;
    const int nch = (pnp_pad + D - 1) / D;
    const bool resident = nch <= 2;
    const int nsteps = a.mode == 0 ? a.n_steps : 1;
    int total_q = resident ? nch : nsteps * nch;
    /* chunk q of the passes into its buffer (one thread) */
    auto issue = [&](int q) {
      const int b = q & 1, c0 = (q % nch) * D, n = min(D, pnp_pad - c0);
      s_issued[b] += 1;
      mbar_expect_tx(&bar[b], (uint32_t)(n * 16));
      bulk_g2s(bpa + b * (D >> 1), ga + (c0 >> 1), (uint32_t)(n * 8), &bar[b]);
      bulk_g2s(bpb + b * (D >> 1), gb + (c0 >> 1), (uint32_t)(n * 8), &bar[b]);
    };
    if (tid == 0) {
      s_done[0] = s_done[1] = 0;
      for (int q = 0; q < min(2, total_q); ++q) issue(q);
    }
    if constexpr (!SPLIT && KIND == GD_KIND_PLAIN)
      roams = __syncthreads_or(roams);
    else
      __syncthreads();

    /* ---- per-lane constants ---- */
    if (roams) take_lane(true);
    const bool by_slot = SPLIT || roams;
    /* the thread's lanes: slot jj (PACK 1), or slots 2 jj and 2 jj + 1, the same atom of two
     * replicas (PACK 2); a missing second slot (odd k) repeats the first one's atom and stores
     * nothing. sl_of: each lane's slot; vl: its index in the placed-atom and partial arrays */
    int sl_of[PACK], vl[PACK];
    bool ok[PACK];
#pragma unroll
    for (int h = 0; h < PACK; ++h) {
      const int jh = jj * PACK + h;
      ok[h] = active && jh < k;
      sl_of[h] = ok[h] ? jh : jj * PACK;
    }

    float4 orig[PACK];
    int l_of[PACK];
#pragma unroll
    for (int h = 0; h < PACK; ++h) {
      /* (a thread's two lanes hold the same atom of two slots, so PACK 2 keeps the atoms' order) */
      const int lc = slots[sl_of[h]].lig_conf;
      l_of[h] = PACK == 1 && !by_slot ? cx.lig_rank[lc * L + rank] : rank;
      orig[h] = cx.lig_pos[lc * L + l_of[h]];
      vl[h] = (ordered ? 0 : sp * A) + sl_of[h] * L + l_of[h];
    }
    /* atom types are the same in every conformer of a ligand when PACK is 2 (host-checked) */
    const int tl = cx.lig_meta[slots[sl_of[0]].lig_conf * L + l_of[0]].x;
    const float *psprow = cx.psp + (size_t)tl * cx.psp_ld;
    const GdPairParam *pprow = a.pp + tl * GD_MAXTP1;
    const int4 *segs = cx.seg + pc * GD_MAX_SEG;
    const int nseg = cx.seg_count[pc];
    unsigned own = 0, hseg = 0;
    int p0 = 0, h0 = 0; /* the first stored piece, of all and of the hydrogen-bond ones */
    if constexpr (SPLIT) {
      const unsigned *plan = cx.split_plan + (size_t)pc * GD_SPLIT_WORDS;
      own = __ldg(plan + (ordered ? GD_SPLIT_MASKS : 0) + GD_SPLIT_AT(S, sp));
      if (ordered) {
        const unsigned first = __ldg(plan + 2 * GD_SPLIT_MASKS + S - 1);
        p0 = first & 0xffffu;
        h0 = first >> 16;
        hseg = __ldg(plan + GD_SPLIT_WORDS - 1);
        /* pieces that no segment has (at a block's end) stay zero */
        for (int i = tid; i < n_planes * T; i += NT) pcs[i] = 0.0;
      }
    }
    bool aborted = false;
    /* the lane's piece (sg, block blk): vdw, ele, pmf, hydrogen bonds */
    auto store_piece = [&](int sg, int blk, int flags, double e0, double e1, double e2,
                           double e3) {
      if (!ok[0]) return;
      double *w = pcs + 3 * (sg + blk - p0) * T + vl[0];
      w[0] = e0;
      w[T] = e1;
      w[2 * T] = e2;
      if (flags & 4)
        pcs[(3 * a.pieces + __popc(hseg & ((1u << sg) - 1u)) + blk - h0) * T + vl[0]] = e3;
    };

    /* A step may take three passes. Energies from the far fields differ from those of the pair
     * loop over every point in the last FP32 digits; a Metropolis decision that could hang on
     * that (about one in 10^4, GD_CERT), of a plain step or of delayed acceptance's second stage, is
     * left open in the first pass (phase 0), the CTA then evaluates the proposal (phase 1) and the
     * current pose (phase 2) without the fields, and the slots left open decide on those: every
     * decision is the one the plain loop takes. Exchanges: gd_exchange_group. */
    const bool certify = (a.mode == 0 || (DA && a.mode == 3)) && cx.ff_tab != nullptr;
    /* a step's ring runs on into the next pass; delayed acceptance's single step issues the chunks
     * of another pass when there is one (a third more copies otherwise: 29 -> 31 ms for 50 steps of
     * 6,820 replicas on 3,000 points) */
    const bool run_on = !DA && certify;
    int phase = 0, q_run = 0;
    for (int s = 0; s < nsteps;) {
      /* ---- Move_d: four lanes per replica draw the move (a Box-Muller pair each) and build the
       * rotation (an angle each); one lane took 2.3-4 k cycles with every warp waiting ---- */
      for (int jb = 0; jb < k; jb += NT >> 2) {
        const int j = jb + (tid >> 2), q = tid & 3;
        const bool mine = j < k && q < 3;
        Slot &sl = slots[j < k ? j : 0];
        float m0 = 0.0f, m1 = 0.0f, u = 0.0f; /* movematrix[2 q], [2 q + 1] */
        const float *mm = phase == 2 ? sl.mm_old : sl.mm_new;
        if (mine && phase == 0) {
          if (a.mode == 0) {
            float d0, d1;
            gd_draw_pair(a.seed, (uint32_t)cx.stream, (uint32_t)(sl.rep - cx.rep_offset),
                         (uint32_t)(step_first + s), a.move_kind, q, &d0, &d1, &u);
            m0 = GD_ADD(sl.mm_old[2 * q], GD_MUL(a.move_scale[2 * q], d0));
            m1 = GD_ADD(sl.mm_old[2 * q + 1], GD_MUL(a.move_scale[2 * q + 1], d1));
          } else if (a.mode == 2 || a.mode == 3) {
            m0 = a.mm_in[(size_t)sl.rep * 6 + 2 * q];
            m1 = a.mm_in[(size_t)sl.rep * 6 + 2 * q + 1];
          }
          sl.mm_new[2 * q] = m0;
          sl.mm_new[2 * q + 1] = m1;
          if (q == 2) sl.u = u;
        }
        __syncwarp();
        float sn = 0.0f, cn = 0.0f;
        if (mine) gd_sincosf(mm[3 + q], &sn, &cn);
        const int l0 = lane & ~3;
        const float s1 = __shfl_sync(0xffffffffu, sn, l0), c1 = __shfl_sync(0xffffffffu, cn, l0),
                    s2 = __shfl_sync(0xffffffffu, sn, l0 + 1),
                    c2 = __shfl_sync(0xffffffffu, cn, l0 + 1),
                    s3 = __shfl_sync(0xffffffffu, sn, l0 + 2),
                    c3 = __shfl_sync(0xffffffffu, cn, l0 + 2);
        if (mine) {
          if (q == 0) gd_rotation_sc(s1, c1, s2, c2, s3, c3, sl.rot);
          if (q == 1) {
            const float *lc = cx.lig_center + sl.lig_conf * 3;
            sl.tx = GD_ADD(mm[0], lc[0]);
            sl.ty = GD_ADD(mm[1], lc[1]);
            sl.tz = GD_ADD(mm[2], lc[2]);
            if (a.mode == 4) {
              /* given coordinates: the ligand centre comes with them (Ligand.coord_new.center) */
              sl.tx = a.center_in[(size_t)sl.rep * 3];
              sl.ty = a.center_in[(size_t)sl.rep * 3 + 1];
              sl.tz = a.center_in[(size_t)sl.rep * 3 + 2];
            }
          }
        }
      }
      __syncthreads();
      float ax[PACK], ay[PACK], az[PACK];
#pragma unroll
      for (int h = 0; h < PACK; ++h) {
        ax[h] = ay[h] = az[h] = 0.0f;
        if (active) {
          const Slot &sl = slots[sl_of[h]];
          if (a.mode == 4) {
            const float *p = a.xyz_in + ((size_t)sl.rep * L + l_of[h]) * 3;
            ax[h] = p[0];
            ay[h] = p[1];
            az[h] = p[2];
          } else {
            gd_place_atom(sl.rot, sl.tx, sl.ty, sl.tz, orig[h].x, orig[h].y, orig[h].z, &ax[h],
                          &ay[h], &az[h]);
          }
          if (ok[h] && sp == 0) atoms[vl[h]] = make_float4(ax[h], ay[h], az[h], 0.0f);
        }
      }
      /* each lane clears its own partials (the only ones the epilogue reads) */
#pragma unroll
      for (int h = 0; h < PACK; ++h)
        if (ok[h] && (!ordered || sp == 0))
#pragma unroll
          for (int qi = 0; qi < NQ; ++qi) part[qi * T + vl[h]] = 0.0;

      if constexpr (SPLIT) {
        /* the restraints beside the pair loop, by the warps of one split */
        __syncthreads();
        const int wa = A >> 5, w0 = mcs_sp * wa;
        if (warp >= w0 && warp < w0 + wa)
          for (int js = warp - w0; js < k; js += wa) {
            const double v = restraints(cx, slots[js].lig_conf, L, atoms + js * L, lane);
            if (lane == 0) s_lhm[js] = v;
          }
      }

      /* ---- short-range terms from the pocket grid's lists (or the cell list), before the pair
       * loop: warps whose lists are short start the loop while the others still read ---- */
      /* lbin: the radius bin past which each lane's points come from the far fields
       * (GD_FAR_BINS - 1: every point runs in the loop) */
      int lbin[PACK];
#pragma unroll
      for (int h = 0; h < PACK; ++h) {
        lbin[h] = GD_FAR_BINS - 1;
        if (!ok[h]) continue;
        const int v = vl[h];
        const int cell = pocket_cell(cx, ax[h], ay[h], az[h]);
        /* outside the grid the contact split walks the rows for both lists */
        const bool con = sp == con_sp, kind = sp == (cell >= 0 ? kind_sp : con_sp);
        if (con || kind) {
          ShortSums sr = {0.0, 0.0f, 0.0f, 0};
          const float *thr = thr_s + tl * GD_MAXTP1;
          if (cell >= 0)
            short_range_lists(cx, pc, cell, thr, psprow, f, ax[h], ay[h], az[h], con, kind, sr);
          else
            short_range(cx, pc, thr, psprow, f, ax[h], ay[h], az[h], sr);
          if (con) {
            part[1 * T + v] = (double)sr.ele;
            part[8 * T + v] = (double)sr.ncon;
          }
          if (kind) {
            part[3 * T + v] = (double)sr.psp;
            const double hpc2 = (sr.hsum - (double)f.hpl0[tl]) / (double)f.hpl1[tl];
            part[5 * T + v] = 0.5 * hpc2 * hpc2 - (double)f.hpl2[tl];
          }
        }
        const int fcell =
            !XCH && cx.ff_tab != nullptr && phase == 0 ? gd_ff_cell(cx, ax[h], ay[h], az[h]) : -1;
        if (fcell >= 0) {
          const int id = __ldg(cx.ff_id + fcell);
          const int bin = gd_ff_bin(cx, fcell);
          if (id >= 0 && bin < GD_FAR_BINS - 1) {
            lbin[h] = bin;
            if (sp == 0) {
              float fe, fv;
              far_field(cx, pc, fcell, id, tl, ax[h], ay[h], az[h], fe, fv);
              part[0 * T + v] = (double)fv;
              part[1 * T + v] += (double)fe;
              part[2 * T + v] =
                  __ldg(cx.ff_pmf + ((size_t)pc * GD_FAR_BINS + bin) * GD_MAXTP2 + tl);
            }
          }
        }
      }

      /* ---- far-point bin of the warp: a point further from the pocket centre than far_r +
       * the largest distance of the warp's atoms from it is beyond far_r of each of them, and
       * takes the far form of the pair body (the same result, fewer operations) ---- */
      int fbin = 0;
#pragma unroll
      for (int h = 0; h < PACK; ++h) {
        if (!ok[h]) continue;
        const float dx = ax[h] - cx.pocket[0], dy = ay[h] - cx.pocket[1],
                    dz = az[h] - cx.pocket[2];
        const float rho = sqrtf(dx * dx + dy * dy + dz * dz) + cx.far_r;
        fbin = max(fbin, (int)fminf(rho * cx.far_inv_w, (float)(GD_FAR_BINS - 1)));
      }
      fbin = (int)__reduce_max_sync(0xffffffffu, (unsigned)fbin);
      const unsigned short *fcnt = cx.far_cnt + (size_t)pc * GD_MAX_SEG * GD_FAR_BINS + fbin;

      /* ---- CalcEnergy_d pair loop over the protein ring (sg0: the first segment that reaches
       * past the chunks done) ---- */
      int sg0 = 0;
      for (int ci = 0; ci < nch; ++ci) {
        const int q = resident ? ci : q_run + ci;
        const int b = q & 1;
        if (!resident || q_run == 0) {
          bool ok = !*(volatile int *)&s_abort;
          if (ok) ok = mbar_wait_bounded(&bar[b], b ? (consumed1 & 1u) : (consumed0 & 1u),
                                         a.timeout_ns);
          if (!ok) {
            aborted = true;
            if (lane == 0) { s_abort = 1; atomicOr(a.err, GD_DEV_ERR_TIMEOUT); }
            break;
          }
          if (b) ++consumed1; else ++consumed0;
        }
        if (active) {
          const float4 *PA = bpa + b * (D >> 1); /* local slot = slot - c0 */
          const float4 *PB = bpb + b * (D >> 1);
          const int c0 = ci * D, c1 = min(pnp_pad, c0 + D);
          /* blocks of `fold` slots, at whose ends a segment's sums go to FP64: the whole chunk, or
           * the default tile's chunks where the ring's are larger */
          int blk = SPLIT ? c0 / a.fold : 0;
          for (int b0 = c0; b0 < c1; b0 += a.fold, ++blk) {
            const int b1 = min(c1, b0 + a.fold);
            for (int sg = sg0; sg < nseg; ++sg) {
              const int4 g = segs[sg];
              if (g.x >= b1) break;
              if (g.y <= b1) sg0 = sg + 1;
              if (SPLIT && !((own >> sg) & 1u)) continue;
              const int i0 = max(g.x, b0) - c0;
              /* each lane's end of the segment: where its far field takes over */
              int il[PACK], i1 = 0;
#pragma unroll
              for (int h = 0; h < PACK; ++h) {
                const int e = PACK > 1 && !ok[h] ? g.x
                              : lbin[h] == GD_FAR_BINS - 1 ? g.y
                                                           : gd_ff_near(cx, pc, sg, g, lbin[h]);
                il[h] = min(e, b1) - c0;
                i1 = max(i1, il[h]);
              }
              if (i0 >= i1) {
                if (ordered && sp > 0) store_piece(sg, blk, g.w, 0.0, 0.0, 0.0, 0.0);
                continue;
              }
              const float4 *pr = reinterpret_cast<const float4 *>(pprow + g.z);
              const float4 q0 = __ldg(pr), q1 = __ldg(pr + 1), q2 = __ldg(pr + 2);
              Pair2 pq;
              pq.p1a = f2(q0.x); pq.mp2a = f2(-q0.y); pq.p1l = f2(q0.z);
              pq.p1ll = f2(q0.z * f.lj1); pq.hc1 = f2(q1.z); pq.hc0 = f2(q1.w);
              pq.hs = f2(q2.x); pq.b2 = f2(q2.z); pq.c2 = f2(q2.w);
              const float2 z2 = f2(0.0f);
              Acc acc[PACK];
#pragma unroll
              for (int h = 0; h < PACK; ++h) acc[h] = {z2, z2, z2, z2};
              /* the segment's near points [i0, im) and far points [im, i1); the split slot is
               * even (the segment starts on one), so the near part keeps whole slot pairs */
              const int fs = g.x + ((__ldg(fcnt + sg * GD_FAR_BINS) + 1) & ~1) - c0;
              const int im = min(i1, max(i0, fs));
              if constexpr (PACK == 1) {
                if (i0 < im)
                  pair_dispatch<UNROLL, 1, false, SPLIT>(g.w, PA, PB, i0, im, ax, ay, az, pq, f,
                                                         acc);
                if (im < i1)
                  pair_dispatch<UNROLL, 1, true, SPLIT>(g.w, PA, PB, im, i1, ax, ay, az, pq, f,
                                                        acc);
              } else {
                /* both lanes' points together, then the rest of the lane that has more */
                const int ib = max(i0, min(il[0], il[1])), imb = min(im, ib);
                if (i0 < imb)
                  pair_dispatch<UNROLL, 2, false>(g.w, PA, PB, i0, imb, ax, ay, az, pq, f, acc);
                if (imb < ib)
                  pair_dispatch<UNROLL, 2, true>(g.w, PA, PB, imb, ib, ax, ay, az, pq, f, acc);
#pragma unroll
                for (int h = 0; h < PACK; ++h) {
                  const int j0 = max(ib, im);
                  if (ib < min(im, il[h]))
                    pair_dispatch<UNROLL, 1, false>(g.w, PA, PB, ib, min(im, il[h]), ax + h, ay + h,
                                                    az + h, pq, f, acc + h);
                  if (j0 < il[h])
                    pair_dispatch<UNROLL, 1, true>(g.w, PA, PB, j0, il[h], ax + h, ay + h, az + h,
                                                   pq, f, acc + h);
                }
              }
#pragma unroll
              for (int h = 0; h < PACK; ++h) {
                if (!ok[h]) continue;
                const int v = vl[h];
                if (ordered && sp > 0) {
                  store_piece(sg, blk, g.w, (double)acc[h].vdw.x + (double)acc[h].vdw.y,
                              (double)acc[h].ele.x + (double)acc[h].ele.y,
                              (double)q1.y * ((double)acc[h].pmf.x + (double)acc[h].pmf.y),
                              (double)acc[h].hdb.x + (double)acc[h].hdb.y);
                  continue;
                }
                part[0 * T + v] += (double)acc[h].vdw.x + (double)acc[h].vdw.y;
                part[1 * T + v] += (double)acc[h].ele.x + (double)acc[h].ele.y;
                part[2 * T + v] += (double)q1.y * ((double)acc[h].pmf.x + (double)acc[h].pmf.y);
                part[4 * T + v] += (double)acc[h].hdb.x + (double)acc[h].hdb.y;
              }
            }
          }
        }
        if (!resident) {
          /* the last warp done with buffer b refills it with chunk q + 2 */
          __syncwarp();
          if (lane == 0) {
            __threadfence_block();
            const int prev = atomicAdd(&s_done[b], 1);
            if (prev == nwarps - 1) {
              s_done[b] = 0;
              if (run_on || q + 2 < total_q) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue(q + 2);
              }
            }
          }
        }
      }

      /* ---- per-atom tail (one split of each atom): kde, rmsd, reference contacts ---- */
#pragma unroll
      for (int h = 0; h < PACK; ++h) {
        if (!ok[h] || aborted) continue;
        const int v = vl[h];
        if (!ordered) part[1 * T + v] *= (double)orig[h].w;
        if (sp != tail_sp) continue;
        float ks = 0.0f;
        /* the KDE points lie sorted by type, in their given order within a type: the atom sums
         * its own type's points only. Latency-bound (a chain of additions per atom): four loads
         * in flight. One conformer of 454 points walked whole took 96 k cycles a step. */
        const int k0 = __ldg(cx.kde_start + tl), k1 = __ldg(cx.kde_start + tl + 1);
#pragma unroll 4
        for (int kk = k0; kk < k1; ++kk) {
          const float4 kd = __ldg(cx.kde + kk);
          const float dx = ax[h] - kd.x, dy = ay[h] - kd.y, dz = az[h] - kd.z;
          ks += expf(f.kde2 * (dx * dx + dy * dy + dz * dz));
        }
        const int kn = k1 - k0;
        part[6 * T + v] = kn ? (double)ks / (double)kn : 0.0;
        const Slot &sl = slots[sl_of[h]];
        const float *lc = cx.lig_center + sl.lig_conf * 3;
        const float rx = ax[h] - (orig[h].x + lc[0]), ry = ay[h] - (orig[h].y + lc[1]),
                    rz = az[h] - (orig[h].z + lc[2]);
        part[7 * T + v] = (double)(rx * rx + ry * ry + rz * rz);
        int tp = 0;
        const int *rs = cx.ref_start + pc * (L + 1);
        for (int i = rs[l_of[h]]; i < rs[l_of[h] + 1]; ++i) {
          const float4 rp = __ldg(cx.ref_pts + i);
          tp += dist2(ax[h], ay[h], az[h], rp.x, rp.y, rp.z) <= rp.w ? 1 : 0;
        }
        part[9 * T + v] = (double)tp;
      }
      if (__syncthreads_or(aborted)) {
        aborted = true;
        break;
      }

      if constexpr (SPLIT) {
        if constexpr (ordered) {
          /* each atom's pieces added to split 0's sums in the points' order, a sum per thread */
          for (int i = tid; i < 4 * k * L; i += NT) {
            const int q = i / (k * L), at = i - q * k * L, js = at / L;
            const bool hb = q == 3;
            double *p = part + (hb ? 4 : q) * T + at;
            const double *w = pcs + (hb ? 3 * a.pieces : q) * T + at;
            const int n = hb ? a.hpieces : a.pieces, st = hb ? T : 3 * T;
            const float charge =
                q == 1 ? __ldg(&cx.lig_pos[slots[js].lig_conf * L + at - js * L].w) : 1.0f;
            double t = p[0];
#pragma unroll 16
            for (int j = 0; j < n; ++j) t += w[j * st];
            p[0] = q == 1 ? t * (double)charge : t;
          }
        } else {
          /* each atom's partials of its splits, added in split order by all threads */
          for (int i = tid; i < NQ * k * L; i += NT) {
            const int q = i / (k * L);
            double *p = part + q * T + (i - q * k * L);
            double t = p[0];
            for (int z = 1; z < S; ++z) t += p[z * A];
            p[0] = t;
          }
        }
        __syncthreads();
      }

      /* ---- per-replica epilogue: one warp per slot ---- */
      for (int js = warp; js < k; js += nwarps) {
        Slot &sl = slots[js];
        /* slot totals are written back over the slot's first partial; five quantities at a time,
         * so that their shuffles overlap (one at a time the chain took 7-9 k cycles a step) */
        double *tot = part + js * L;
#pragma unroll 1
        for (int q0 = 0; q0 < NQ; q0 += 5) {
          double v[5];
#pragma unroll
          for (int u = 0; u < 5; ++u) v[u] = 0.0;
          for (int i = lane; i < L; i += 32)
#pragma unroll
            for (int u = 0; u < 5; ++u) v[u] += part[(q0 + u) * T + js * L + i];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < 5; ++u) v[u] += __shfl_down_sync(0xffffffffu, v[u], o);
          if (lane == 0)
#pragma unroll
            for (int u = 0; u < 5; ++u) tot[(q0 + u) * T] = v[u];
        }
        const double elhm =
            SPLIT ? s_lhm[js] : restraints(cx, sl.lig_conf, L, atoms + js * L, lane);
        /* the nine normalised terms, MCC and RMSD, a lane each; the total in term order (all by
         * lane 0 they took 3-5 k cycles) */
        __syncwarp();
        const double Ld = (double)L;
        /* every lane's division, square root and logarithm at the same time as the others' */
        const double tp = tot[9 * T];
        const double fp = tot[8 * T] - tp, fn = (double)cx.nref_total - tp;
        const double tn = Ld * (double)P - tp - fp - fn;
        double e =
            lane < 6 ? tot[lane * T] : lane == 6 ? tot[6 * T] : lane == 7 ? elhm : tot[7 * T];
        e /= lane == 6 ? (double)f.kde3 : lane == 7 ? (double)cx.pos : Ld;
        if (lane >= 8) {
          const double dx = (double)sl.tx - (double)cx.pocket[0];
          const double dy = (double)sl.ty - (double)cx.pocket[1];
          const double dz = (double)sl.tz - (double)cx.pocket[2];
          e = sqrt(lane == 8 ? dx * dx + dy * dy + dz * dz
                   : lane == 9 ? (tp + fp) * (tp + fn) * (tn + fp) * (tn + fn) : e);
        } else if (lane == 7) {
          e = log(e);
        }
        float side = 0.0f; /* lane 9: MCC, lane 10: RMSD */
        if (lane == 6 || lane == 9) {
          const double q = (lane == 6 ? e : tp * tn - fp * fn) / (lane == 6 ? Ld : e);
          side = e != 0.0 ? (float)q : 0.0f;
          if (lane == 6) e = q;
        } else if (lane == 10) {
          side = (float)e;
        }
        if (lane < GD_MAXWEI - 1) e = s_norm[0][lane] * e + s_norm[1][lane];
        gd_energy en;
        double etot = 0.0;
        float mag = 0.0f;
#pragma unroll
        for (int i = 0; i < GD_MAXWEI - 1; ++i) {
          const double v = __shfl_sync(0xffffffffu, e, i);
          en.e[i] = (float)v;
          etot += v * s_norm[2][i];
          mag += fabsf((float)(v * s_norm[2][i]));
        }
        en.e[GD_MAXWEI - 1] = (float)etot;
        en.cms = __shfl_sync(0xffffffffu, side, 9);
        en.rmsd = __shfl_sync(0xffffffffu, side, 10);
        if (lane == 0) {
          const int rid = sl.rep;
          const float etn = en.e[GD_MAXWEI - 1];
          if (XCH) {
            x_e[x_list[xb + js]] = etn;
          } else if (a.mode == 2 || a.mode == 4) {
            a.e_out[rid] = en;
          } else if (DA && a.mode == 3) {
            const int ci = tile.complex_index, step = step_first + s;
            if (phase == 0) {
              const int r = a.da->pose_rep[rid];
              const gd_energy &eo = a.e_old[r];
              const float tol = certify ? GD_CERT * (mag + cert_mag(eo, f)) + sl.cert : 0.0f;
              if (!da_decide(a, cx, ci, rid, en, etn, eo.e[GD_MAXWEI - 1], tol, sl.mm_new, step)) {
#pragma unroll
                for (int i = 0; i < 6; ++i) sl.mm_old[i] = a.mm_old[(size_t)r * 6 + i];
                sl.e_prop = en;
                sl.open = 1;
                s_open = 1;
              }
            } else if (sl.open) {
              if (phase == 1) {
                sl.e_full = etn;
              } else {
                sl.open = 0;
                da_decide(a, cx, ci, rid, sl.e_prop, sl.e_full, etn, 0.0f, sl.mm_new, step);
              }
            }
          } else {
            int acc = 1;
            bool decide = phase == 0;
            if (a.mode == 0) {
              const float eto = sl.e_old.e[GD_MAXWEI - 1];
              if (phase == 0) {
                acc = gd_metropolis(etn, eto, sl.mb, sl.u);
                if (certify) {
                  const float tol = GD_CERT * (mag + sl.mag) + sl.cert;
                  if (gd_metropolis(etn + tol, eto, sl.mb, sl.u) !=
                      gd_metropolis(etn - tol, eto, sl.mb, sl.u)) {
                    sl.e_prop = en;
                    sl.open = 1;
                    s_open = 1;
                    decide = false;
                  }
                }
              } else if (sl.open) {
                if (phase == 1) {
                  sl.e_full = etn;
                } else {
                  acc = gd_metropolis(sl.e_full, etn, sl.mb, sl.u);
                  en = sl.e_prop;
                  mag = cert_mag(en, f);
                  sl.open = 0;
                  decide = true;
                }
              }
            }
            if (decide) {
              sl.accept = acc;
              if (acc) {
                sl.e_old = en;
                sl.mag = mag;
#pragma unroll
                for (int i = 0; i < 6; ++i) sl.mm_old[i] = sl.mm_new[i];
                if (a.mode == 0) sl.n_acc += 1;
                if (a.rec) {
                  const int kslot = sl.rec_next;
                  if (kslot < a.rec_cap) {
                    gd_record_step *r = a.rec + (size_t)rid * a.rec_cap + kslot;
                    r->replica = sl.replica;
                    r->energy = en;
#pragma unroll
                    for (int i = 0; i < 6; ++i) r->movematrix[i] = sl.mm_new[i];
                    r->step = a.mode == 0 ? step_first + s : 0;
                    sl.rec_next = kslot + 1;
                  } else {
                    atomicOr(a.err, GD_DEV_ERR_RECORD_FULL);
                  }
                }
              }
              if (a.trace_e && a.mode == 0) {
                const int ti = step_first + s - a.trace_step0;
                if (ti >= 0 && ti < a.trace_cap) {
                  a.trace_e[(size_t)rid * a.trace_cap + ti] = en.e[GD_MAXWEI - 1];
                  a.trace_acc[(size_t)rid * a.trace_cap + ti] = acc;
                }
              }
            }
          }
        }
      }
      __syncthreads();
      q_run += nch;
      if (phase == 0 && !(certify && s_open)) {
        ++s;
      } else if (phase < 2) {
        ++phase;
        if (DA && !resident) {
          total_q = q_run + nch;
          if (tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(q_run);
            issue(q_run + 1);
          }
        }
      } else {
        phase = 0;
        ++s;
        if (tid == 0) s_open = 0; /* read again only after the next step's barriers */
      }
    }
    if (run_on && !resident && !aborted) {
      /* the ring was refilled for a pass that did not come: let its two chunks land */
      for (int i = 0; i < 2; ++i) {
        const int b = (q_run + i) & 1;
        if (!mbar_wait_bounded(&bar[b], b ? (consumed1 & 1u) : (consumed0 & 1u), a.timeout_ns)) {
          aborted = true;
          if (lane == 0) { s_abort = 1; atomicOr(a.err, GD_DEV_ERR_TIMEOUT); }
          break;
        }
        if (b) ++consumed1; else ++consumed0;
      }
      aborted = __syncthreads_or(aborted);
    }

    if (aborted) {
      /* a bounded wait gave up: let the copies still in flight land (bounded again, with
       * the fixed drain limit) before the CTA leaves, then stop */
      if (tid == 0) {
        const long long drain_ns = 2000000000LL;
        if (s_issued[0]) mbar_wait_bounded(&bar[0], (s_issued[0] - 1u) & 1u, drain_ns);
        if (s_issued[1]) mbar_wait_bounded(&bar[1], (s_issued[1] - 1u) & 1u, drain_ns);
      }
      __syncthreads();
      break;
    }

    /* ---- write back replica state ---- */
    if (a.mode < 2 && tid < k) {
      const Slot &sl = slots[tid];
      a.e_old[sl.rep] = sl.e_old;
      a.etotal[sl.rep] = sl.e_old.e[GD_MAXWEI - 1];
      a.n_accept[sl.rep] = sl.n_acc;
      if (a.rec) a.rec_next[sl.rep] = sl.rec_next;
#pragma unroll
      for (int i = 0; i < 6; ++i) a.mm_old[(size_t)sl.rep * 6 + i] = sl.mm_old[i];
      /* ExchangeReplicas_d fused: the replica that completes its group in this launch (the
       * group's last to be written back, counted with fences on both sides) exchanges the
       * group's temperatures; no CTA waits for another */
      if (a.mode == 0 && a.x_done) {
        const int local = sl.rep - cx.rep_offset, nl = cx.n_lig, nt = cx.n_tmp;
        const int lg = (local / (nt * nl)) * nl + local % nl;
        __threadfence();
        if (atomicAdd(a.x_done + a.x_group_base[tile.complex_index] + lg, 1) == nt - 1) {
          __threadfence();
          const int mode_t = !(((step_first % a.x_spd) / a.x_spe) % 2);
          const GdExchange ex = {a.replica, a.etotal, a.e_old, a.x_acs, a.seed};
          if (gd_exchange_group(cx, lg, ex, f, (a.x_call_base ? *a.x_call_base : 0) + a.x_call_off,
                                mode_t))
            open_group(a.x_open, a.x_open_list, a.x_open_cap,
                       a.x_group_base[tile.complex_index] + lg, a.err);
        }
      }
    }
    if (XCH) xb += k;
    __syncthreads();
  }
  if (XCH && tid == 0) {
    /* every CTA has read the count: the last one clears it for the next exchange */
    __threadfence();
    if (atomicAdd(a.x_open + 1, 1) == (int)gridDim.x - 1) a.x_open[0] = a.x_open[1] = 0;
  }
}

/* the kernel variants the host can launch: point pairs in flight per lane; no split, partial sums
 * per split, or split with sums in the points' order (the automatic shapes, four pairs); plain modes, the delayed-acceptance exact stage (mode 3) or the open exchange groups; replicas per
 * thread (two only for the plain modes without split) */
#define GD_INST(U, S, K, P) \
  template __global__ void gd_mc_kernel<U, S, K, P>(GdMcArgs, GdForceConst);
GD_INST(1, 0, 0, 1) GD_INST(2, 0, 0, 1) GD_INST(4, 0, 0, 1)
GD_INST(1, 1, 0, 1) GD_INST(2, 1, 0, 1) GD_INST(4, 1, 0, 1)
GD_INST(1, 0, 1, 1) GD_INST(2, 0, 1, 1) GD_INST(4, 0, 1, 1)
GD_INST(1, 1, 1, 1) GD_INST(2, 1, 1, 1) GD_INST(4, 1, 1, 1)
GD_INST(4, 2, 0, 1) GD_INST(4, 2, 1, 1)
GD_INST(1, 0, 0, 2) GD_INST(2, 0, 0, 2)
GD_INST(2, 0, 2, 1)
#undef GD_INST

/* ExchangeReplicas_d, one thread per (complex, protein conformer, ligand conformer) group of
 * the range [g_begin, g_end). */
__global__ void gd_exchange_kernel(const GdDevComplex *cxs, const int *group_base, int n_complex,
                                   int g_begin, int g_end, GdExchange ex, GdForceConst f,
                                   const int *call_base, int call_off, int mode_t, int *open,
                                   int *open_list, unsigned *err) {
  const int g = g_begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= g_end || mode_t >= 2) return;
  int lo = 0, hi = n_complex - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (group_base[mid] <= g) lo = mid; else hi = mid - 1;
  }
  if (gd_exchange_group(cxs[lo], g - group_base[lo], ex, f,
                        (call_base ? *call_base : 0) + call_off, mode_t))
    open_group(open, open_list, g_end - g_begin, g, err);
}

/* ResetCounter_d (src/kernel_cuda_l1_resetcounter.cu:12-22). */
__global__ void gd_reset_records_kernel(int *rec_next, int r0, int r1) {
  const int r = r0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (r <= r1) rec_next[r] = 0;
}

}  // namespace gd
