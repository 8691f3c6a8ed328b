/*
 * gd_capi_eval.cu -- pose energies on demand (gd_eval_energy, gd_eval_energy_xyz): one launch of
 * the Monte Carlo kernel in its evaluation modes over given poses or placed coordinates; placed
 * ligand coordinates of given poses (gd_place_ligand, the reference's PlaceLigand as its trace
 * tool calls it); and the per-step energy trace of replica 0 (gd_trace_enable, gd_trace_get).
 */
#include "gd_capi_internal.cuh"

using namespace gdc;

namespace gdc {

LaunchShape eval_shape(const gd_ctx *c, int ci, int n, int *k) {
  const ComplexInfo &x = c->info[ci];
  if (!c->tile_auto) {
    *k = x.k;
    return ctx_shape(c);
  }
  std::vector<int> ks;
  LaunchShape s;
  for (int S = auto_split(c, {{1, n, x.lna}}, &ks); S > 1; --S) {
    *k = ks[0];
    if (split_shape(c, ci, S, *k * x.lna, *k, x.pnp_pad, &s)) return s;
  }
  /* one lane per atom: a CTA of 128..256 lanes with the least left over */
  int best = 256;
  for (int T = 128; T <= GD_MAX_TPB; T += 32)
    if (T >= x.lna && (T / x.lna) * x.lna * best > (best / x.lna) * x.lna * T) best = T;
  *k = std::min(GD_MAX_SLOTS, best / x.lna);
  return {best, GD_CHUNK, GD_CHUNK, 1, 2, 1, *k};
}

}  // namespace gdc

namespace {

/* Energies of n poses of one (complex, protein conformer, ligand conformer): moved by
 * movematrix rows (mm, kernel mode 2), or given as placed coordinates and centres (xyz and
 * center, mode 4). */
int eval_poses(gd_ctx *c, int ci, int prt_conf, int lig_conf, const float *mm, const float *xyz,
               const float *center, int n, gd_energy *out) {
  if (!c || !out || (!mm && !(xyz && center))) return fail(GD_ERR_INVALID, "null argument");
  if (ci < 0 || ci >= c->n_complex) return fail(GD_ERR_INVALID, "bad complex index");
  const ComplexInfo &x = c->info[ci];
  if (prt_conf < 0 || prt_conf >= x.n_prt || lig_conf < 0 || lig_conf >= x.n_lig)
    return fail(GD_ERR_INVALID, "conformer index out of range");
  if (n < 1) return GD_OK;
  CK(cudaSetDevice(c->device));
  const bool given = mm == nullptr;
  const size_t row = sizeof(float) * (given ? 3 * (size_t)x.lna + 3 : 6);
  if (row * n > c->eval_in_cap) {
    if (c->d_eval_in) cudaFree(c->d_eval_in);
    c->d_eval_in = nullptr;
    c->eval_in_cap = 0;
    CK(cmalloc(c, &c->d_eval_in, row * n));
    c->eval_in_cap = row * n;
  }
  if (n > c->eval_cap) {
    if (c->d_e_out) cudaFree(c->d_e_out);
    c->d_e_out = nullptr;
    c->eval_cap = 0;
    CK(cmalloc(c, &c->d_e_out, sizeof(gd_energy) * n));
    c->eval_cap = n;
  }
  /* small calls go through a page-locked buffer of the context, so that the copies and the kernel
   * queue up behind one another and the call waits once (24 poses: 51 us, 81 with a wait
   * and a pageable copy per array);
   * large ones, whose time is in the copies, straight from and to the caller's arrays */
  const size_t in = row * n, out_bytes = sizeof(gd_energy) * (size_t)n;
  const bool staged = std::max(in, out_bytes) + sizeof(unsigned) <= GD_EVAL_STAGE;
  if (staged && !c->h_eval) CK(cudaMallocHost(&c->h_eval, GD_EVAL_STAGE));
  float *d_xyz = static_cast<float *>(c->d_eval_in), *d_ctr = d_xyz + 3 * (size_t)x.lna * n;
  auto up = [&](float *dst, const float *src, size_t bytes, size_t at) -> cudaError_t {
    const void *from = src;
    if (staged) {
      memcpy(c->h_eval + at, src, bytes);
      from = c->h_eval + at;
    }
    return cudaMemcpyAsync(dst, from, bytes, cudaMemcpyHostToDevice, c->stream);
  };
  if (given) {
    const size_t xb = sizeof(float) * 3 * (size_t)x.lna * n;
    CK(up(d_xyz, xyz, xb, 0));
    CK(up(d_ctr, center, sizeof(float) * 3 * n, xb));
  } else {
    CK(up(d_xyz, mm, in, 0));
  }
  int k = 1;
  const LaunchShape shape = eval_shape(c, ci, n, &k);
  GdMcArgs a = base_args(c);
  a.mode = given ? 4 : 2;
  a.n_steps = 1;
  a.mm_in = given ? nullptr : d_xyz;
  a.xyz_in = given ? d_xyz : nullptr;
  a.center_in = given ? d_ctr : nullptr;
  a.u = GdTileDesc{ci, prt_conf, lig_conf, k};
  a.u_n = n;
  a.e_out = c->d_e_out;
  a.rec = nullptr;
  a.trace_e = nullptr;
  int rc = launch_mc(c, a, nullptr, (n + k - 1) / k, c->d_counters, shape);
  if (rc) {
    cudaStreamSynchronize(c->stream); /* the caller's arrays are no longer read */
    return rc;
  }
  unsigned err = 0;
  unsigned *h_err = staged ? reinterpret_cast<unsigned *>(c->h_eval + GD_EVAL_STAGE) - 1 : &err;
  /* the inputs have been read when the energies are written */
  CK(cudaMemcpyAsync(staged ? (void *)c->h_eval : (void *)out, c->d_e_out, out_bytes,
                     cudaMemcpyDeviceToHost, c->stream));
  CK(cudaMemcpyAsync(h_err, c->d_err, sizeof(err), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  if ((rc = device_status(*h_err))) return rc;
  if (staged) memcpy(out, c->h_eval, out_bytes);
  return GD_OK;
}

}  // namespace

extern "C" {

int gd_eval_energy(gd_ctx *c, int ci, int prt_conf, int lig_conf, const float *mm, int n,
                   gd_energy *out) {
  if (!mm) return fail(GD_ERR_INVALID, "null argument");
  return eval_poses(c, ci, prt_conf, lig_conf, mm, nullptr, nullptr, n, out);
}

int gd_eval_energy_xyz(gd_ctx *c, int ci, int prt_conf, int lig_conf, const float *xyz,
                       const float *center, int n, gd_energy *out) {
  if (!xyz || !center) return fail(GD_ERR_INVALID, "null argument");
  return eval_poses(c, ci, prt_conf, lig_conf, nullptr, xyz, center, n, out);
}

/* One thread per (pose, atom): the rotation of the pose and the placed atom, with the same
 * gd_rotation / gd_place_atom the Monte Carlo kernel places its ligands with. */
__global__ void gd_place_kernel(const GdDevComplex *cxs, int ci, int lig_conf, const float *mm,
                                int n, float *xyz) {
  const GdDevComplex &cx = cxs[ci];
  const int L = cx.lna;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)n * L) return;
  const int pose = (int)(i / L), l = (int)(i % L);
  float m[6], rot[9];
  for (int k = 0; k < 6; ++k) m[k] = mm[pose * 6 + k];
  gd_rotation(m, rot);
  const float *lc = cx.lig_center + lig_conf * 3;
  const float4 o = cx.lig_pos[lig_conf * L + l];
  gd_place_atom(rot, GD_ADD(m[0], lc[0]), GD_ADD(m[1], lc[1]), GD_ADD(m[2], lc[2]), o.x, o.y,
                o.z, &xyz[i * 3], &xyz[i * 3 + 1], &xyz[i * 3 + 2]);
}

int gd_place_ligand(gd_ctx *c, int ci, int lig_conf, const float *mm, int n, float *xyz) {
  if (!c || (n > 0 && (!mm || !xyz))) return fail(GD_ERR_INVALID, "null argument");
  if (ci < 0 || ci >= c->n_complex) return fail(GD_ERR_INVALID, "bad complex index");
  const ComplexInfo &x = c->info[ci];
  if (lig_conf < 0 || lig_conf >= x.n_lig)
    return fail(GD_ERR_INVALID, "ligand conformer %d out of range [0, %d)", lig_conf, x.n_lig);
  if (n < 0) return fail(GD_ERR_INVALID, "negative pose count");
  if (n == 0) return GD_OK;
  CK(cudaSetDevice(c->device));
  const size_t out_bytes = sizeof(float) * 3 * (size_t)x.lna * n;
  float *d_mm = nullptr, *d_xyz = nullptr;
  CK(cudaStreamSynchronize(c->stream));
  cudaError_t e = cmalloc(c, &d_mm, sizeof(float) * 6 * (size_t)n);
  if (e == cudaSuccess) e = cmalloc(c, &d_xyz, out_bytes);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_mm, mm, sizeof(float) * 6 * (size_t)n,
                                       cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) {
    const long long total = (long long)n * x.lna;
    gd_place_kernel<<<(unsigned)((total + 255) / 256), 256, 0, c->stream>>>(c->d_cx, ci, lig_conf,
                                                                           d_mm, n, d_xyz);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e == cudaSuccess) e = cudaMemcpy(xyz, d_xyz, out_bytes, cudaMemcpyDeviceToHost);
  cudaFree(d_mm);
  cudaFree(d_xyz);
  if (e != cudaSuccess) return fail(GD_ERR_CUDA, "gd_place_ligand: %s", cudaGetErrorString(e));
  return GD_OK;
}

int gd_trace_enable(gd_ctx *c, int max_steps) {
  if (!c || max_steps < 0) return fail(GD_ERR_INVALID, "bad argument");
  CK(cudaStreamSynchronize(c->stream));
  if (c->d_trace_e) cudaFree(c->d_trace_e);
  if (c->d_trace_acc) cudaFree(c->d_trace_acc);
  c->d_trace_e = nullptr;
  c->d_trace_acc = nullptr;
  c->trace_cap = 0;
  drop_graphs(c);
  if (max_steps == 0) return GD_OK;
  CK(cmalloc(c, &c->d_trace_e, sizeof(float) * (size_t)c->n_rep * max_steps));
  CK(cmalloc(c, &c->d_trace_acc, sizeof(int) * (size_t)c->n_rep * max_steps));
  CK(cudaMemsetAsync(c->d_trace_acc, 0xff, sizeof(int) * (size_t)c->n_rep * max_steps, c->stream));
  c->trace_cap = max_steps;
  c->trace_step0 = 0;
  return GD_OK;
}

int gd_trace_get(gd_ctx *c, float *e_new, int *acc, int *n_steps) {
  if (!c || !e_new || !acc || !n_steps) return fail(GD_ERR_INVALID, "null argument");
  if (!c->trace_cap) return fail(GD_ERR_STATE, "trace disabled");
  CK(cudaStreamSynchronize(c->stream));
  CK(cudaMemcpy(e_new, c->d_trace_e, sizeof(float) * (size_t)c->n_rep * c->trace_cap,
                cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(acc, c->d_trace_acc, sizeof(int) * (size_t)c->n_rep * c->trace_cap,
                cudaMemcpyDeviceToHost));
  *n_steps = c->trace_cap;
  return GD_OK;
}

}  // extern "C"
