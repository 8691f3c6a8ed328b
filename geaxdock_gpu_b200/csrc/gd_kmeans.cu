/*
 * gd_kmeans.cu -- the k-means of the post-Monte-Carlo clustering on the GPU, many independent
 * problems (segments) per launch.
 *
 * Reference: clusterByKmeans (src/util.C:1801-1880) over seq_kmeans (src/seq_kmeans.c): the
 * records of a segment are shuffled, the first k become the initial centres, then Lloyd
 * iterations (nearest centre by squared Euclidean distance, ties to the lower index; centres
 * = member means) run while more than `threshold` of the objects changed cluster and at most
 * 501 passes; the representative of a cluster is its last member in shuffled order (the
 * reference's medoid loop never updates its running distance, so it keeps the last member).
 *
 * The shuffle here is a seeded pseudorandom permutation of each segment's positions: a
 * 4-round balanced Feistel network on the smallest even power of two covering the segment,
 * with cycle walking (every position is mapped independently, so the permutation needs no
 * sort); round keys come from the seed and the segment index through the lowbias32 integer
 * hash (C. Wellons). The reference shuffles with an unseeded random_shuffle, so only the
 * distribution of orders can be matched, not the order itself.
 *
 * Every float operation is the reference's, in its order: the distance sums the squared
 * coordinate differences dimension by dimension (no fused multiply-add); a centre sums its
 * members' coordinates in shuffled order and divides by the member count. One thread per
 * object assigns. For small segments one thread per cluster walks its segment in order to sum
 * its members; for large ones (the pooled second stage) a stable radix sort of the objects by
 * cluster (CUB, over the bits the cluster numbers have) lists each cluster's members in order and
 * one CTA per cluster sums them.
 * A segment stops iterating on its own criterion; the host reads one counter per pass, a pass
 * behind the launches, so that the device does not wait for it (the pass launched after the last
 * one finds no active segment).
 */
#include <cuda_runtime.h>

#include <cstdint>
#include <cub/device/device_radix_sort.cuh>
#include <mutex>
#include <vector>

#include "gd_kmeans.cuh"

namespace gd {
namespace {

__host__ __device__ inline uint32_t lowbias32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

struct PermKeys {
  uint32_t k[4];
  int half; /* bits per half */
};

__host__ __device__ inline PermKeys perm_keys(uint64_t seed, int seg, int n) {
  PermKeys p;
  int b = 0;
  while ((1u << b) < (uint32_t)n) ++b;
  if (b & 1) ++b;
  p.half = b / 2;
  for (int r = 0; r < 4; ++r)
    p.k[r] = lowbias32((uint32_t)seed ^
                       lowbias32((uint32_t)(seed >> 32) + 0x9E3779B9u * (uint32_t)(seg * 4 + r + 1)));
  return p;
}

/* position i (0 <= i < n) of the shuffled segment holds object perm_index(i) */
__host__ __device__ inline int perm_index(int i, int n, const PermKeys &p) {
  if (n <= 1) return 0;
  const uint32_t mask = (1u << p.half) - 1u;
  uint32_t x = (uint32_t)i;
  do {
    uint32_t l = x >> p.half, r = x & mask;
    for (int k = 0; k < 4; ++k) {
      const uint32_t f = lowbias32(r ^ p.k[k]) & mask;
      const uint32_t nl = r;
      r = l ^ f;
      l = nl;
    }
    x = (l << p.half) | r;
  } while (x >= (uint32_t)n);
  return (int)x;
}

struct Seg {
  int off, n, k, cbase; /* objects [off, off + n), clusters [cbase, cbase + k) */
};

__global__ void gather_kernel(const float *__restrict__ obj, int dim, const Seg *__restrict__ seg,
                              const int *__restrict__ seg_of, int n_obj, uint64_t seed,
                              float *__restrict__ sh, int *__restrict__ perm) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_obj) return;
  const int s = seg_of[p];
  const Seg g = seg[s];
  const PermKeys pk = perm_keys(seed, s, g.n);
  const int src = g.off + perm_index(p - g.off, g.n, pk);
  perm[p] = src;
  for (int j = 0; j < dim; ++j) sh[(size_t)p * dim + j] = obj[(size_t)src * dim + j];
}

__global__ void init_centres(const float *__restrict__ sh, int dim, const Seg *__restrict__ seg,
                             const int *__restrict__ cseg, int n_cl, float *__restrict__ cen) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cl) return;
  const Seg g = seg[cseg[c]];
  for (int j = 0; j < dim; ++j)
    cen[(size_t)c * dim + j] = sh[(size_t)(g.off + (c - g.cbase)) * dim + j];
}

/* Nearest centre of each object. The centres of the clusters of every segment the block's
 * objects belong to (a contiguous range) are staged in shared memory when they fit (SMEM_CL
 * clusters). A block whose objects are all of one segment (the pooled stage: 500 centres) reads
 * them as pairs: two centres per FP32x2 difference and sum, each separately rounded as the scalar
 * form's, and two objects per thread, which share every load. Bound by the
 * FMA pipe (27 operations per object and centre, 62 us for 170,484 objects and 500 centres, 69 us
 * on the SMs that hold five of the 666 blocks): 105 us; one centre and object at a time, with
 * nine loads each, took 139 us. */
constexpr int SMEM_CL = 1024;
constexpr int ASSIGN_T = 128; /* threads; 2 ASSIGN_T objects per block */

/* negated centres [c0, c0 + k) as pairs: sc[(c / 2) 2 D + 2 j + (c & 1)]; an odd last centre is
 * paired with itself (a tie, which the lower index wins) */
template <int D>
__device__ __forceinline__ void stage_pairs(const float *__restrict__ cen, int c0, int k,
                                            float *sc) {
  const int kp = (k + 1) >> 1;
  for (int i = threadIdx.x; i < kp * 2 * D; i += ASSIGN_T) {
    const int c = min(k - 1, i / (2 * D) * 2 + (i & 1)), j = (i % (2 * D)) >> 1;
    sc[i] = -cen[(size_t)(c0 + c) * D + j];
  }
}

/* squared distances of a thread's object: the nearest centre's index and distance as the scan
 * finds them, and (SECOND) the two smallest */
struct Nearest {
  int best = 0;
  float d = 0.0f, lo1 = INFINITY, lo2 = INFINITY;
  template <bool SECOND>
  __device__ __forceinline__ void see(float2 s, int c, bool first) {
    if (first || s.x < d) {
      d = s.x;
      best = c;
    }
    if (s.y < d) {
      d = s.y;
      best = c + 1;
    }
    if (SECOND) {
      lo2 = fminf(lo2, fmaxf(lo1, s.x));
      lo1 = fminf(lo1, s.x);
      lo2 = fminf(lo2, fmaxf(lo1, s.y));
      lo1 = fminf(lo1, s.y);
    }
  }
};

template <int D, bool SECOND>
__device__ __forceinline__ void scan_pairs(const float *sc, int c0, int c1,
                                           const float *__restrict__ sh, int pa, int pb, Nearest &a,
                                           Nearest &b) {
  float2 oa[D], ob[D];
#pragma unroll
  for (int j = 0; j < D; ++j) {
    const float va = pa >= 0 ? sh[(size_t)pa * D + j] : 0.0f;
    const float vb = pb >= 0 ? sh[(size_t)pb * D + j] : 0.0f;
    oa[j] = make_float2(va, va);
    ob[j] = make_float2(vb, vb);
  }
#pragma unroll 2
  for (int c = c0; c < c1; ++c) { /* centre pairs */
    const float2 *q = reinterpret_cast<const float2 *>(sc) + c * D;
    float2 sa = make_float2(0.0f, 0.0f), sb = sa;
#pragma unroll
    for (int j = 0; j < D; ++j) {
      const float2 n = q[j];
      const float2 ta = __fadd2_rn(oa[j], n), tb = __fadd2_rn(ob[j], n);
      /* scalar products: ptxas contracts a packed product and sum into FFMA2, even from
       * mul.rn.f32x2 and add.rn.f32x2, which rounds once */
      sa = __fadd2_rn(sa, make_float2(__fmul_rn(ta.x, ta.x), __fmul_rn(ta.y, ta.y)));
      sb = __fadd2_rn(sb, make_float2(__fmul_rn(tb.x, tb.x), __fmul_rn(tb.y, tb.y)));
    }
    a.see<SECOND>(sa, 2 * c, c == 0);
    b.see<SECOND>(sb, 2 * c, c == 0);
  }
}

template <int D>
__global__ void __launch_bounds__(ASSIGN_T) assign_kernel(
    const float *__restrict__ sh, const Seg *__restrict__ seg, const int *__restrict__ seg_of,
    const unsigned char *__restrict__ act, int n_obj, const float *__restrict__ cen,
    int *__restrict__ mem, int *__restrict__ changed) {
  __shared__ __align__(16) float sc[SMEM_CL * D];
  const int p0 = blockIdx.x * (2 * ASSIGN_T);
  const int pl = min(p0 + 2 * ASSIGN_T, n_obj) - 1;
  const int s0 = seg_of[p0], s1 = seg_of[pl];
  const int c0 = seg[s0].cbase;
  const Seg gl = seg[s1];
  const int nc = gl.cbase + gl.k - c0;
  const bool staged = nc <= SMEM_CL;
  if (s0 == s1 && staged && gl.k > 0) {
    if (!act[s0]) return;
    stage_pairs<D>(cen, c0, gl.k, sc);
    __syncthreads();
    const int ia = p0 + threadIdx.x, ib = ia + ASSIGN_T;
    const int pa = ia < n_obj ? ia : -1, pb = ib < n_obj ? ib : -1;
    Nearest a, b;
    scan_pairs<D, false>(sc, 0, (gl.k + 1) >> 1, sh, pa, pb, a, b);
    int n = 0;
    if (pa >= 0) {
      n += mem[pa] != a.best ? 1 : 0;
      mem[pa] = a.best;
    }
    if (pb >= 0) {
      n += mem[pb] != b.best ? 1 : 0;
      mem[pb] = b.best;
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(changed + s0, n);
    return;
  }
  if (staged)
    for (int i = threadIdx.x; i < nc * D; i += ASSIGN_T) sc[i] = cen[(size_t)c0 * D + i];
  __syncthreads();
  for (int p = p0 + threadIdx.x; p <= pl; p += ASSIGN_T) {
    const int s = seg_of[p];
    if (!act[s]) continue;
    const Seg g = seg[s];
    const float *cb = staged ? sc + (size_t)(g.cbase - c0) * D : cen + (size_t)g.cbase * D;
    float o[D];
#pragma unroll
    for (int j = 0; j < D; ++j) o[j] = sh[(size_t)p * D + j];
    int best = 0;
    float best_d = 0.0f;
    for (int c = 0; c < g.k; ++c) {
      const float *q = cb + (size_t)c * D;
      float d = 0.0f;
#pragma unroll
      for (int j = 0; j < D; ++j) {
        const float t = __fsub_rn(o[j], q[j]);
        d = __fadd_rn(d, __fmul_rn(t, t));
      }
      if (c == 0 || d < best_d) {
        best_d = d;
        best = c;
      }
    }
    if (mem[p] != best) atomicAdd(changed + s, 1);
    mem[p] = best;
  }
}

/* One large segment: most objects of a later pass cannot have changed their centre. Each keeps an
 * upper bound u of the distance to its centre and a lower bound l of that to any other (Hamerly,
 * "Making k-means even faster", SDM 2010); a pass adds its centre's move to u, takes the largest
 * move from l, and only objects with u not clearly below l are scanned again, with the distances
 * and the comparisons of assign_kernel. Rounding: a computed squared distance is within 8e-7 of
 * the exact one of the same FP32 operands (nine differences, products and sums) but for an
 * underflow of at most 9 x 2^-126, so u < l with KM_REL and KM_ABS to spare means that the scan
 * would find the same centre, strictly nearest; a NaN or an infinite move fails the comparison
 * and is scanned. 170,484 objects without structure (independent normal terms, the bounds' worst case:
 * 63 % scanned in the 6th pass, 50 % in the 30th, 25 % from the 46th on) and 500 clusters: a call
 * of 147 passes 26.4 -> 21.2 ms; of wandering energies, 22 passes, 5.0 -> 4.2 ms. */
constexpr float KM_REL = 4e-6f, KM_ABS = 4e-18f;

__global__ void __launch_bounds__(256)
    prune_kernel(const unsigned char *__restrict__ act, int n_obj, int first,
                 const int *__restrict__ mem, const float *__restrict__ move,
                 const unsigned *__restrict__ most, float2 *__restrict__ ul, int *__restrict__ list,
                 int *__restrict__ n_list) {
  const int p = blockIdx.x * 256 + threadIdx.x;
  if (!act[0]) return;
  bool scan = p < n_obj;
  if (scan && !first) {
    const float2 v = ul[p];
    const float u = (v.x + move[mem[p]]) * (1.0f + 2e-7f);
    const float l = (v.y - __uint_as_float(*most)) * (1.0f - 2e-7f);
    if (u * (1.0f + KM_REL) + KM_ABS < l) {
      ul[p] = make_float2(u, l);
      scan = false;
    }
  }
  const unsigned m = __ballot_sync(0xffffffffu, scan);
  if (!m) return;
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0) at = atomicAdd(n_list, __popc(m));
  at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
  if (scan) list[at] = p;
}

/* stage_pairs' layout in global memory (update_sorted_kernel keeps it up) */
template <int D>
__device__ __forceinline__ void put_pair(float *__restrict__ pairs, int c, int k, int j, float v) {
  float *p = pairs + (size_t)(c >> 1) * (2 * D) + 2 * j + (c & 1);
  p[0] = -v;
  if (c == k - 1 && !(c & 1)) p[1] = -v;
}

template <int D>
__global__ void pairs_kernel(const float *__restrict__ cen, int k, float *__restrict__ pairs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < k * D) put_pair<D>(pairs, i / D, k, i % D, cen[i]);
}

/* The listed objects, LIST_N a CTA: half of its threads scan the first half of the centres, half
 * the second, two objects a thread. Lists are shorter than the object array, and CTAs of 256
 * objects left two to three an SM: 22.3 -> 21.5 ms for the 147 passes; with the centres copied
 * from the paired layout that update_sorted_kernel keeps (float4 loads, no divisions) 21.2 ms.
 * The second half starts from no centre (infinity), so that a comparison between the halves is
 * the scan's own: only a strictly nearer centre replaces one of lower index, and a first centre
 * that is not a number is never replaced. */
constexpr int LIST_N = ASSIGN_T;

template <int D>
__global__ void __launch_bounds__(ASSIGN_T) assign_list_kernel(
    const float *__restrict__ sh, int k, const int *__restrict__ list,
    const int *__restrict__ n_list, const float4 *__restrict__ pairs, int *__restrict__ mem,
    float2 *__restrict__ ul, int *__restrict__ changed) {
  __shared__ __align__(16) float sc[SMEM_CL * D];
  __shared__ float4 other[LIST_N]; /* the second half's (best, d, lo1, lo2) */
  const int n = *n_list, i0 = blockIdx.x * LIST_N;
  if (i0 >= n) return;
  const int quads = (((k + 1) >> 1) * 2 * D + 3) >> 2;
#pragma unroll 8
  for (int i = threadIdx.x; i < quads; i += ASSIGN_T)
    reinterpret_cast<float4 *>(sc)[i] = pairs[i];
  __syncthreads();
  constexpr int G = ASSIGN_T / 2;
  const int half = threadIdx.x / G, t = threadIdx.x - half * G;
  const int ia = i0 + t, ib = ia + G;
  const int pa = ia < n ? list[ia] : -1, pb = ib < n ? list[ib] : -1;
  const int kp = (k + 1) >> 1, km = (kp + 1) >> 1;
  Nearest a, b;
  if (half) a.d = b.d = INFINITY;
  scan_pairs<D, true>(sc, half ? km : 0, half ? kp : km, sh, pa, pb, a, b);
  if (half) {
    other[t] = make_float4(__int_as_float(a.best), a.d, a.lo1, a.lo2);
    other[t + G] = make_float4(__int_as_float(b.best), b.d, b.lo1, b.lo2);
  }
  __syncthreads();
  if (half) return;
  int ch = 0;
  auto put = [&](int p, const Nearest &q, float4 o) {
    if (p < 0) return;
    const bool second = o.y < q.d;
    const int best = second ? __float_as_int(o.x) : q.best;
    const float d = second ? o.y : q.d;
    const float lo2 = fminf(fmaxf(q.lo1, o.z), fminf(q.lo2, o.w));
    ch += mem[p] != best ? 1 : 0;
    mem[p] = best;
    /* u from the scan's own distance, NaN if the first centre's is: then never skipped; l of a
     * square that overflowed is what is known of it */
    ul[p] = make_float2(sqrtf(d) * (1.0f + 1e-6f) + KM_ABS,
                        sqrtf(fminf(lo2, 3.4028235e38f)) * (1.0f - 1e-6f) - KM_ABS);
  };
  put(pa, a, other[t]);
  put(pb, b, other[t + G]);
  ch = __reduce_add_sync(0xffffffffu, ch);
  if ((threadIdx.x & 31) == 0 && ch) atomicAdd(changed, ch);
}

template <int D>
__global__ void update_kernel(const float *__restrict__ sh, const Seg *__restrict__ seg,
                              const int *__restrict__ cseg, const unsigned char *__restrict__ act,
                              int n_cl, const int *__restrict__ mem, float *__restrict__ cen) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cl) return;
  const int s = cseg[c];
  if (!act[s]) return;
  const Seg g = seg[s];
  const int kc = c - g.cbase;
  float sum[D];
#pragma unroll
  for (int j = 0; j < D; ++j) sum[j] = 0.0f;
  int cnt = 0;
  for (int p = g.off; p < g.off + g.n; ++p) {
    if (mem[p] != kc) continue;
    ++cnt;
#pragma unroll
    for (int j = 0; j < D; ++j) sum[j] = __fadd_rn(sum[j], sh[(size_t)p * D + j]);
  }
  if (cnt > 0) {
#pragma unroll
    for (int j = 0; j < D; ++j) cen[(size_t)c * D + j] = __fdiv_rn(sum[j], (float)cnt);
  }
}

__global__ void cluster_key_kernel(const Seg *__restrict__ seg, const int *__restrict__ seg_of,
                                   const int *__restrict__ mem, int n_obj, int n_cl,
                                   int *__restrict__ key, int *__restrict__ pos) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_obj) return;
  const int m = mem[p];
  key[p] = m >= 0 ? seg[seg_of[p]].cbase + m : n_cl; /* not clustered: past the last cluster */
  pos[p] = p;
}

/* first / one-past-last index of each cluster in the sorted key array */
__global__ void bounds_kernel(const int *__restrict__ key, int n_obj, int n_cl,
                              int *__restrict__ begin, int *__restrict__ end) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_obj) return;
  const int k = key[i];
  if (k >= n_cl) return;
  if (i == 0 || key[i - 1] != k) begin[k] = i;
  if (i == n_obj - 1 || key[i + 1] != k) end[k] = i + 1;
}

/* centre = in-order sum of its members / count, one CTA per cluster: its threads gather the
 * members' rows, a tile of UPD_T at a time and the next tile in flight, and one thread per
 * coordinate adds a tile's values in order. Bound by the chain of dependent additions of the
 * largest cluster; one thread per (cluster, coordinate) gathering for itself waited for its loads:
 * 72 us a pass for 170,484 objects in 500 clusters, now 11 us. */
constexpr int UPD_T = 128;

template <int D>
__global__ void __launch_bounds__(UPD_T)
    update_sorted_kernel(const float *__restrict__ sh, const int *__restrict__ cseg,
                         const unsigned char *__restrict__ act, const int *__restrict__ begin,
                         const int *__restrict__ end, const int *__restrict__ pos,
                         float *__restrict__ cen, float *__restrict__ move,
                         unsigned *__restrict__ most, float *__restrict__ pairs) {
  __shared__ float tile[2][UPD_T * D];
  const int c = blockIdx.x, t = threadIdx.x;
  if (!act[cseg[c]]) return;
  const int b = begin[c], e = end[c];
  if (e <= b) { /* the centre stays */
    if (move && t == 0) move[c] = 0.0f;
    return;
  }
  float v[D];
  int q = b + t < e ? pos[b + t] : 0, qn = b + UPD_T + t < e ? pos[b + UPD_T + t] : 0;
#pragma unroll
  for (int j = 0; j < D; ++j) v[j] = sh[(size_t)q * D + j];
  float s = 0.0f;
  for (int i0 = b, k = 0; i0 < e; i0 += UPD_T, k ^= 1) {
    float *w = tile[k];
#pragma unroll
    for (int j = 0; j < D; ++j) w[t * D + j] = v[j];
    __syncthreads();
    if (i0 + UPD_T < e) {
#pragma unroll
      for (int j = 0; j < D; ++j) v[j] = sh[(size_t)qn * D + j];
      const int i2 = i0 + 2 * UPD_T + t;
      qn = i2 < e ? pos[i2] : 0;
    }
    if (t < D) {
      const int n = min(UPD_T, e - i0);
      if (n == UPD_T) {
#pragma unroll 32
        for (int i = 0; i < UPD_T; ++i) s = __fadd_rn(s, w[i * D + t]);
      } else {
#pragma unroll 8
        for (int i = 0; i < n; ++i) s = __fadd_rn(s, w[i * D + t]);
      }
    }
  }
  float step = 0.0f;
  if (t < D) {
    const float v = __fdiv_rn(s, (float)(e - b));
    step = v - cen[(size_t)c * D + t];
    cen[(size_t)c * D + t] = v;
    if (move) put_pair<D>(pairs, c, (int)gridDim.x, t, v);
  }
  if (!move || t >= 32) return;
  /* how far the centre went, rounded up (prune_kernel); infinite when it is not a number */
  float d2 = step * step;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) d2 += __shfl_down_sync(0xffffffffu, d2, o);
  if (t == 0) {
    float m = sqrtf(d2) * (1.0f + 1e-6f) + KM_ABS;
    if (!(m >= 0.0f)) m = INFINITY;
    move[c] = m;
    atomicMax(most, __float_as_uint(m));
  }
}

/* per segment: delta = changed / n (float); keep iterating while delta > threshold and the
 * pass counter (post-incremented, as `loop++ < 500`) is below max_iter */
__global__ void step_kernel(const Seg *__restrict__ seg, int n_seg, int *__restrict__ changed,
                            int *__restrict__ loops, unsigned char *__restrict__ act,
                            float threshold, int max_iter, int *__restrict__ n_active) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_seg) return;
  if (act[s]) {
    const float delta = __fdiv_rn((float)changed[s], (float)seg[s].n);
    const bool more = delta > threshold && loops[s]++ < max_iter;
    act[s] = more ? 1 : 0;
    if (more) atomicAdd(n_active, 1);
  }
  changed[s] = 0;
}

/* the same from the sorted member lists (last member = the largest position in the list) */
__global__ void medoid_sorted_kernel(int n_cl, const int *__restrict__ begin,
                                     const int *__restrict__ end, const int *__restrict__ pos,
                                     const int *__restrict__ perm, int *__restrict__ medoid,
                                     int *__restrict__ size) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cl) return;
  const int b = begin[c], e = end[c];
  medoid[c] = e > b ? perm[pos[e - 1]] : -1;
  size[c] = e > b ? e - b : 0;
}

__global__ void medoid_kernel(const Seg *__restrict__ seg, const int *__restrict__ cseg, int n_cl,
                              const int *__restrict__ mem, const int *__restrict__ perm,
                              int *__restrict__ medoid, int *__restrict__ size) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cl) return;
  const Seg g = seg[cseg[c]];
  const int kc = c - g.cbase;
  int last = -1, cnt = 0;
  for (int p = g.off; p < g.off + g.n; ++p)
    if (mem[p] == kc) {
      last = p;
      ++cnt;
    }
  medoid[c] = last >= 0 ? perm[last] : -1;
  size[c] = cnt;
}

__global__ void unshuffle_kernel(const int *__restrict__ perm, const int *__restrict__ mem,
                                 int n_obj, int *__restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n_obj) out[perm[p]] = mem[p];
}

/* Page-locked pairs of counters for the pass loop (making one costs more than a pass): taken and
 * given back by each call, a few kept for the next ones of the process. */
std::mutex g_pin_mu;
std::vector<int *> g_pin;
constexpr size_t PIN_KEEP = 4;

cudaError_t pin_take(int **p) {
  {
    std::lock_guard<std::mutex> lock(g_pin_mu);
    if (!g_pin.empty()) {
      *p = g_pin.back();
      g_pin.pop_back();
      return cudaSuccess;
    }
  }
  return cudaHostAlloc(reinterpret_cast<void **>(p), 2 * sizeof(int), cudaHostAllocPortable);
}

void pin_give(int *p) {
  if (!p) return;
  {
    std::lock_guard<std::mutex> lock(g_pin_mu);
    if (g_pin.size() < PIN_KEEP) {
      g_pin.push_back(p);
      return;
    }
  }
  cudaFreeHost(p);
}

/* segment of every object and of every cluster, one CTA per segment */
__global__ void seg_of_kernel(const Seg *__restrict__ seg, int *__restrict__ seg_of,
                              int *__restrict__ cseg) {
  const int s = blockIdx.x;
  const Seg g = seg[s];
  for (int i = threadIdx.x; i < g.n; i += blockDim.x) seg_of[g.off + i] = s;
  for (int i = threadIdx.x; i < g.k; i += blockDim.x) cseg[g.cbase + i] = s;
}

/* One block of device memory for all of a call's arrays, each at a 256-byte boundary: sized in a
 * first round of take() calls, which return offsets, and made by alloc(). (Some twenty
 * cudaMalloc and cudaFree a call took 8-10 ms of host time, now and then 100 ms and more.) The pool
 * keeps what it is given back, so a block past POOL_MAX comes from the driver and goes back to it:
 * a call that large runs for tens of milliseconds, its cudaMalloc for about one. */
constexpr size_t POOL_MAX = (size_t)64 << 20;
struct Arena {
  char *base = nullptr;
  size_t used = 0;
  bool pooled = false;
  template <class T>
  size_t take(size_t n) {
    const size_t at = used;
    used += ((n ? n : 1) * sizeof(T) + 255) & ~(size_t)255;
    return at;
  }
  template <class T>
  T *at(size_t off) const {
    return reinterpret_cast<T *>(base + off);
  }
  cudaError_t alloc(void *pool, cudaStream_t st) {
    pooled = pool != nullptr && used <= POOL_MAX;
    return pooled ? cudaMallocFromPoolAsync(reinterpret_cast<void **>(&base), used,
                                            (cudaMemPool_t)pool, st)
                  : cudaMalloc(reinterpret_cast<void **>(&base), used);
  }
  void release(cudaStream_t st) {
    if (!base) return;
    if (pooled)
      cudaFreeAsync(base, st); /* after the stream's work; cudaFree waits for it by itself */
    else
      cudaFree(base);
    base = nullptr;
  }
};

}  // namespace

int kmeans_permutation(uint64_t seed, int seg, int n, int *out) {
  const PermKeys pk = perm_keys(seed, seg, n);
  for (int i = 0; i < n; ++i) out[i] = perm_index(i, n, pk);
  return 0;
}

int kmeans_device(const KmeansJob &job, KmeansResult &res, std::string &err) {
  const int D = job.dim;
  if (D != 9) {
    err = "k-means is built for 9 coordinates (the energy terms)";
    return -1;
  }
  const int n_seg = (int)job.seg_off.size() - 1;
  std::vector<Seg> seg(n_seg);
  int n_obj = job.seg_off.back(), n_cl = 0;
  for (int s = 0; s < n_seg; ++s) {
    Seg &g = seg[s];
    g.off = job.seg_off[s];
    g.n = job.seg_off[s + 1] - g.off;
    /* fewer objects than clusters: not clustered, every object is its own cluster in its
     * original order (clusterByKmeans returns the records as they are) */
    g.k = job.k[s] <= g.n ? job.k[s] : g.n;
    g.cbase = n_cl;
    n_cl += g.k;
  }
  res.membership.assign(n_obj, -1);
  res.medoid.assign(n_cl, -1);
  res.size.assign(n_cl, 0);
  res.cluster_base.resize(n_seg);
  for (int s = 0; s < n_seg; ++s) res.cluster_base[s] = seg[s].cbase;
  res.passes.assign(n_seg, 0);
  if (n_obj == 0 || n_cl == 0) return 0;

  int *h_act = nullptr; /* pinned: active segments after the even and the odd passes */
  cudaEvent_t ev[2] = {nullptr, nullptr};
  cudaStream_t st = (cudaStream_t)job.stream;
  cudaError_t e = cudaSuccess;
  auto ok = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
    return e == cudaSuccess;
  };
  ok(pin_take(&h_act));
  for (cudaEvent_t &v : ev) ok(cudaEventCreateWithFlags(&v, cudaEventDisableTiming));
  int max_n = 0;
  for (const Seg &g : seg) max_n = g.n > max_n ? g.n : max_n;
  const bool sorted = max_n > 8192;
  /* a single large segment whose centres fit in shared memory (the pooled stage): bounds decide
   * which objects a pass scans (26.4 -> 21.2 ms, above). Small segments are bound by their sums,
   * and several large ones at once do not occur in the clustering this serves */
  const bool pruned = sorted && n_seg == 1 && n_cl <= SMEM_CL;
  int key_bits = 1; /* keys 0 .. n_cl */
  while (key_bits < 31 && (n_cl >> key_bits)) ++key_bits;
  const size_t no = n_obj, nc = n_cl, ns = n_seg, srt = sorted ? no : 0;
  size_t tmp_bytes = 0;
  if (sorted)
    ok(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (int *)nullptr, (int *)nullptr,
                                       (int *)nullptr, (int *)nullptr, n_obj, 0, key_bits, st));
  Arena m;
  const size_t o_obj = m.take<float>(no * D), o_sh = m.take<float>(no * D),
               o_cen = m.take<float>(nc * D), o_seg = m.take<Seg>(ns), o_so = m.take<int>(no),
               o_cs = m.take<int>(nc), o_perm = m.take<int>(no), o_mem = m.take<int>(no),
               o_orig = m.take<int>(no), o_chg = m.take<int>(ns), o_loop = m.take<int>(ns),
               o_act = m.take<unsigned char>(ns), o_na = m.take<int>(2), o_med = m.take<int>(nc),
               o_size = m.take<int>(nc), o_key = m.take<int>(srt), o_key2 = m.take<int>(srt),
               o_pos = m.take<int>(srt), o_pos2 = m.take<int>(srt), o_cb = m.take<int>(2 * nc),
               o_tmp = m.take<char>(tmp_bytes), o_ul = m.take<float2>(pruned ? no : 0),
               o_list = m.take<int>(pruned ? no : 0), o_move = m.take<float>(nc),
               o_cnt = m.take<int>(2), o_pairs = m.take<float>(pruned ? (nc + 1) * D + 3 : 0);
  ok(m.alloc(job.pool, st));
  float *obj = m.at<float>(o_obj), *sh = m.at<float>(o_sh), *cen = m.at<float>(o_cen);
  Seg *dseg = m.at<Seg>(o_seg);
  int *dseg_of = m.at<int>(o_so), *dcseg = m.at<int>(o_cs), *perm = m.at<int>(o_perm),
      *mem = m.at<int>(o_mem), *orig = m.at<int>(o_orig), *changed = m.at<int>(o_chg),
      *loops = m.at<int>(o_loop), *n_act = m.at<int>(o_na), *medoid = m.at<int>(o_med),
      *size = m.at<int>(o_size), *key = m.at<int>(o_key), *key2 = m.at<int>(o_key2),
      *pos = m.at<int>(o_pos), *pos2 = m.at<int>(o_pos2), *cb = m.at<int>(o_cb),
      *ce = cb + n_cl, *list = m.at<int>(o_list), *n_list = m.at<int>(o_cnt);
  float2 *ul = m.at<float2>(o_ul);
  float *move = m.at<float>(o_move), *pairs = m.at<float>(o_pairs);
  unsigned *most = reinterpret_cast<unsigned *>(n_list + 1);
  unsigned char *act = m.at<unsigned char>(o_act);
  void *tmp = m.at<char>(o_tmp);
  if (e == cudaSuccess) {
    std::vector<unsigned char> a0(n_seg);
    for (int s = 0; s < n_seg; ++s) a0[s] = seg[s].k > 0 && job.k[s] <= seg[s].n;
    ok(cudaMemcpyAsync(obj, job.objects, sizeof(float) * (size_t)n_obj * D,
                       cudaMemcpyHostToDevice, st));
    ok(cudaMemcpyAsync(dseg, seg.data(), sizeof(Seg) * n_seg, cudaMemcpyHostToDevice, st));
    seg_of_kernel<<<n_seg, 128, 0, st>>>(dseg, dseg_of, dcseg);
    ok(cudaMemcpyAsync(act, a0.data(), n_seg, cudaMemcpyHostToDevice, st));
    ok(cudaMemsetAsync(mem, 0xff, sizeof(int) * n_obj, st));
    ok(cudaMemsetAsync(changed, 0, sizeof(int) * n_seg, st));
    ok(cudaMemsetAsync(loops, 0, sizeof(int) * n_seg, st));
    const int T = 256, bo = (n_obj + T - 1) / T, bc = (n_cl + T - 1) / T, bs = (n_seg + T - 1) / T;
    const int ba = (n_obj + 2 * ASSIGN_T - 1) / (2 * ASSIGN_T);
    gather_kernel<<<bo, T, 0, st>>>(obj, D, dseg, dseg_of, n_obj, job.seed, sh, perm);
    init_centres<<<bc, T, 0, st>>>(sh, D, dseg, dcseg, n_cl, cen);
    if (pruned) pairs_kernel<9><<<(n_cl * 9 + T - 1) / T, T, 0, st>>>(cen, n_cl, pairs);
    ok(cudaGetLastError());
    for (int pass = 0; e == cudaSuccess; ++pass) {
      if (pruned) {
        ok(cudaMemsetAsync(n_list, 0, sizeof(int), st));
        prune_kernel<<<bo, T, 0, st>>>(act, n_obj, pass == 0, mem, move, most, ul, list, n_list);
        assign_list_kernel<9><<<(n_obj + LIST_N - 1) / LIST_N, ASSIGN_T, 0, st>>>(
            sh, n_cl, list, n_list, reinterpret_cast<const float4 *>(pairs), mem, ul, changed);
        ok(cudaMemsetAsync(most, 0, sizeof(unsigned), st));
      } else {
        assign_kernel<9><<<ba, ASSIGN_T, 0, st>>>(sh, dseg, dseg_of, act, n_obj, cen, mem, changed);
      }
      if (sorted) {
        /* stable by key: each cluster's members in shuffled order */
        cluster_key_kernel<<<bo, T, 0, st>>>(dseg, dseg_of, mem, n_obj, n_cl, key, pos);
        ok(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, key, key2, pos, pos2, n_obj, 0, key_bits,
                                           st));
        ok(cudaMemsetAsync(cb, 0, sizeof(int) * 2 * n_cl, st));
        bounds_kernel<<<bo, T, 0, st>>>(key2, n_obj, n_cl, cb, ce);
        update_sorted_kernel<9><<<n_cl, UPD_T, 0, st>>>(sh, dcseg, act, cb, ce, pos2, cen,
                                                        pruned ? move : nullptr, most, pairs);
      } else {
        update_kernel<9><<<bc, T, 0, st>>>(sh, dseg, dcseg, act, n_cl, mem, cen);
      }
      const int slot = pass & 1;
      ok(cudaMemsetAsync(n_act + slot, 0, sizeof(int), st));
      step_kernel<<<bs, T, 0, st>>>(dseg, n_seg, changed, loops, act, job.threshold,
                                    job.max_iter, n_act + slot);
      ok(cudaMemcpyAsync(h_act + slot, n_act + slot, sizeof(int), cudaMemcpyDeviceToHost, st));
      ok(cudaEventRecord(ev[slot], st));
      /* the count of the pass before, while this one runs */
      if (pass > 0) {
        ok(cudaEventSynchronize(ev[slot ^ 1]));
        if (e != cudaSuccess || h_act[slot ^ 1] == 0 || pass > job.max_iter + 2) break;
      }
    }
    if (sorted) {
      /* member lists of the final memberships */
      cluster_key_kernel<<<bo, T, 0, st>>>(dseg, dseg_of, mem, n_obj, n_cl, key, pos);
      ok(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, key, key2, pos, pos2, n_obj, 0, key_bits,
                                         st));
      ok(cudaMemsetAsync(cb, 0, sizeof(int) * 2 * n_cl, st));
      bounds_kernel<<<bo, T, 0, st>>>(key2, n_obj, n_cl, cb, ce);
      medoid_sorted_kernel<<<bc, T, 0, st>>>(n_cl, cb, ce, pos2, perm, medoid, size);
    } else {
      medoid_kernel<<<bc, T, 0, st>>>(dseg, dcseg, n_cl, mem, perm, medoid, size);
    }
    unshuffle_kernel<<<bo, T, 0, st>>>(perm, mem, n_obj, orig);
    ok(cudaGetLastError());
    ok(cudaMemcpyAsync(res.membership.data(), orig, sizeof(int) * n_obj, cudaMemcpyDeviceToHost,
                       st));
    ok(cudaMemcpyAsync(res.medoid.data(), medoid, sizeof(int) * n_cl, cudaMemcpyDeviceToHost, st));
    ok(cudaMemcpyAsync(res.size.data(), size, sizeof(int) * n_cl, cudaMemcpyDeviceToHost, st));
    ok(cudaMemcpyAsync(res.passes.data(), loops, sizeof(int) * n_seg, cudaMemcpyDeviceToHost,
                       st));
    ok(cudaStreamSynchronize(st));
  }
  m.release(st);
  cudaStreamSynchronize(st); /* the pool can give the block back (gd_release_memory) */
  pin_give(h_act);
  for (cudaEvent_t v : ev)
    if (v) cudaEventDestroy(v);
  if (e != cudaSuccess) {
    err = cudaGetErrorString(e);
    return -2;
  }
  /* passes = loop + 1 of the reference (its loop_iterations) */
  for (int s = 0; s < n_seg; ++s) {
    const Seg &g = seg[s];
    if (job.k[s] > g.n) {
      for (int c = 0; c < g.n; ++c) {
        res.medoid[g.cbase + c] = g.off + c;
        res.size[g.cbase + c] = 1;
        res.membership[g.off + c] = c;
      }
      res.passes[s] = 0;
    } else {
      res.passes[s] = g.k > 0 ? res.passes[s] + 1 : 0;
    }
  }
  return 0;
}

}  // namespace gd
