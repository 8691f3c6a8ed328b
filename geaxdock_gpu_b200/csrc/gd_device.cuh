/*
 * gd_device.cuh -- device-resident data layout of the B200 Monte Carlo docking engine.
 *
 * HBM layout (one context, all complexes of a batch):
 *   ligand conformers   float4 (x, y, z, charge) + int2 (type, MCS field) per atom,
 *                       conformer-major; placed coordinates never touch HBM.
 *   protein conformers  two copies of every conformer's points:
 *                       (1) for the all-pairs loop (vdw, ele, pmf, hdb), sorted by point type,
 *                       every type segment starting on an even slot, stored as pairs of slots
 *                       in two float4 streams (negated coordinates and ele / el1) so one
 *                       16-byte shared load gives the two-lane register pairs of the FP32x2
 *                       loop; a segment table (start, end, type, flags) per conformer, flag
 *                       bit 2: the type has a live hydrogen-bond pair with the ligand;
 *                       (2) for the short-range terms (contacts, psp, hpc, the electrostatic
 *                       soft core), a cell list: points sorted by cell of a uniform grid (x
 *                       fastest) as float4 (x, y, z, type and kind bits) + float4 (hpp, PSP
 *                       column bits, ele / el1, 0), and the first point of every cell.
 *   pair parameters     per (ligand type, protein type) 12 floats, folded for the kernel.
 *   contact reference   per conformer and ligand atom, the list of reference contacts as
 *                       float4 (x, y, z, contact threshold): tp is counted over this sparse
 *                       list, so the pair loop only counts contacts.
 *   replica state       movematrix_old[6], Energy (48 B), Replica (16 B), counters; records
 *                       in the reference's LigRecordSingleStep layout.
 * Protein tiles are staged from HBM/L2 into shared memory with cp.async.bulk (TMA engine)
 * into a double buffer completed on mbarriers.
 */
#ifndef GD_DEVICE_CUH
#define GD_DEVICE_CUH

#include <cstdint>

#include "../../include/geauxdock_b200.h"

#define GD_MAX_SEG 32          /* point types (30), rounded up */
#define GD_FAR_BINS 64         /* radius bins of the far-point counts (GdDevComplex.far_cnt) */
#define GD_CELL 4.0f           /* edge of the short-range cell grid (A) */
/* shared-memory bytes of the contact-threshold table at the front of the kernel's buffer */
#define GD_THR_BYTES (GD_MAXTP2 * GD_MAXTP1 * 4)
/* the pocket grid: GD_PG_N^3 cells of GD_PG_EDGE A, a 40 A cube centred on the pocket centre */
#define GD_PG_N 10
#define GD_PG_CELLS (GD_PG_N * GD_PG_N * GD_PG_N)
#define GD_PG_EDGE 4.0f
/* the far fields: cells of GD_FF_EDGE A, a cube of GD_FF_N^3 centred on the pocket centre, of
 * which those of a ball are tabulated; Chebyshev series of total degree GD_FF_DEG, GD_FF_NC
 * coefficients (padded to whole float4) */
#define GD_FF_N 22
#define GD_FF_CELLS (GD_FF_N * GD_FF_N * GD_FF_N)
#define GD_FF_EDGE 2.0f
#define GD_FF_DEG 4
#define GD_FF_NC (((GD_FF_DEG + 1) * (GD_FF_DEG + 2) * (GD_FF_DEG + 3) / 6 + 3) / 4 * 4)
#define GD_MAX_CELLS (1 << 22) /* cells per conformer grid; a larger box widens the cells */
#define GD_MAX_CELLS_ALL (1 << 25) /* cells of all conformers of a complex together */
#define GD_MAX_TPB 256         /* threads per CTA: 3 CTAs of 256 fit the register file */
#define GD_NUM_SMS 148         /* B200 (only a placement hint: any value gives the same results) */
#define GD_CHUNK 512           /* slots per ring buffer and FP32 sum of the default tile */
#define GD_ROAM 5.0f           /* A from the pocket: where a tile's lanes go by slot, not by rank */
#define GD_MAX_TPB_SPLIT 512   /* threads per CTA of the split launches */
/* work of the per-atom terms that a split's segments are balanced against, in units of one point
 * pair: a segment's own set-up, the contact list, the kind list, the restraints, the tail */
#define GD_MAX_SPLITS 16
#define GD_SPLIT_AT(S, sp) ((S) * ((S) - 1) / 2 + (sp))
#define GD_SPLIT_MASKS GD_SPLIT_AT(GD_MAX_SPLITS + 1, 0)
#define GD_SPLIT_WORDS (2 * GD_SPLIT_MASKS + GD_MAX_SPLITS + 1)
#define GD_COST_SEG 8
#define GD_COST_CON 70
#define GD_COST_KIND 90
#define GD_COST_MCS 40
#define GD_COST_TAIL 40
#define GD_COST_FAR 40
#define GD_SLOT_BYTES 252      /* shared-memory bytes per replica slot (sizeof gd::Slot) */
/* A decision on field-based energies stands when it is the same above and below by what the fields
 * may change both poses' energies: GD_CERT of a pose's weighted terms' magnitudes (the rounding of
 * its FP32 results) and what the far points' sums can lose, GD_CERT_ELE of the electrostatic
 * magnitude of all points at the far radius and GD_CERT_FAR of their vdw and pmf magnitudes
 * (ff_cert). 600,000 poses of 5 to 100 atoms on 2,100 to 9,900 points, charges up to 90 times the
 * usual, alternating too, contact weights of both signs 40 times, dispersion 50 times the usual:
 * the largest change was 1.6e-7 of the magnitudes with usual charges (1.4e-5 with the largest),
 * 8.2e-9 of the electrostatic bound, and 1/7 of a pose's sum of the three. */
#define GD_CERT 1e-6f
#define GD_CERT_ELE 5e-8
#define GD_CERT_FAR 2.5e-7
/* resident 256-thread CTAs per SM the register budget is set for, per unroll depth: 80
 * registers at four point pairs in flight, 64 below (no spills); the delayed-acceptance
 * variants keep one CTA fewer (80 at two pairs, 128 at four), where 64 and 80 would spill */
#define GD_MIN_BLOCKS(u) ((u) >= 4 ? 3 : 4)
#define GD_MIN_BLOCKS_DA(u) ((u) >= 4 ? 2 : ((u) >= 2 ? 3 : 4))
/* two replicas per thread: CTAs of at most GD_MAX_TPB / 2 threads (the tile's lanes over two),
 * 4 resident per SM with one point pair in flight per replica, 3 with two */
#define GD_MIN_BLOCKS_PACK(u, p, da) \
  ((p) == 2 ? ((u) >= 2 ? 3 : 4) : ((da) ? GD_MIN_BLOCKS_DA(u) : GD_MIN_BLOCKS(u)))
#define GD_MAX_SLOTS 128       /* replicas per CTA */
#define GD_NQ 12               /* per-lane partial sums handed to the reducer */

/* device error word bits */
#define GD_DEV_ERR_TIMEOUT 1
#define GD_DEV_ERR_RECORD_FULL 2
#define GD_DEV_ERR_CONFIG 4

struct GdPairParam {
  float p1a, p2a, p1l, thr;    /* LJ numerators; p1a*lj0; contact threshold on d^2 */
  float pmf0, pmf1, hc1, hc0;  /* pmf; hdb argument h = r*hc1 + hc0 (scaled for exp2) */
  float hs, hneed, b2, c2;     /* hdb scale (0 when hdb0 <= 0.1); 1 if the hdb term is live;
                                  pmf exponent cA d2 + b2 r + c2 in base 2 */
};

struct GdDevComplex {
  int n_lig, n_prt, n_tmp, lna;
  int pnp, pnp_pad, pnk, pos;
  int rep_offset, n_rep, psp_ld, mcs_ld;
  int stream, nref_total, pad0, pad1;
  float pocket[4];
  /* short-range cell grid, one frame for every conformer of the complex: cell (ix, iy, iz)
   * covers [org + i * cell, org + (i + 1) * cell) per axis, index (iz * ny + iy) * nx + ix */
  float sr_org[3], sr_cell, sr_inv_cell;
  float sr_r;                 /* search radius: every pair with d^2 <= sr_r2 lies inside it */
  float sr_r2;                /* max(81 (hpc), largest contact threshold, (1 / el1)^2) */
  float sr_pad;
  int sr_n[4];                /* nx, ny, nz, cells */
  const float4 *lig_pos;      /* [n_lig*lna] */
  const int2 *lig_meta;       /* [n_lig*lna] type, MCS index (n + 1) */
  const unsigned char *lig_rank; /* [n_lig*lna] the conformer's atoms by distance from its centre */
  const float *lig_center;    /* [n_lig*3] */
  /* protein points in pairs (slots 2m, 2m+1), [n_prt*pnp_pad/2] each:
   *   pt_a = (-x0, -x1, -y0, -y1), pt_b = (-z0, -z1, ele0 / el1, ele1 / el1) */
  const float4 *pt_a;
  const float4 *pt_b;
  /* the cell list, [n_prt*(pnp + 1)] points (the last of a conformer a sentinel at infinity) and
   * [n_prt*(sr_n[3] + 1)] cell starts (conformer-local point indices): sr_a = (x, y, z, bits of type | 256 if hydrophobic | 512 if class 2),
   * sr_b = (hpp, PSP column bits, ele / el1, 0) */
  const float4 *sr_a;
  const float4 *sr_b;
  const int *sr_start;
  /* the pocket grid's point lists (gd_pocket.cu): cell c's contact list is pg_idx[pg_base[pc] +
   * pg_start[s] ..) with s = pc (2 GD_PG_CELLS + 1) + 2 c, up to entry s + 1, its kind list from
   * there to entry s + 2 (whole quads of indices into sr_a / sr_b) */
  const unsigned short *pg_idx;
  const int *pg_start;
  const long long *pg_base;   /* [n_prt] */
  float pg_org[3];
  float pg_rc, pg_rh;         /* the lists' radii around a cell's box: contacts, hydrophobic */
  /* who runs which segments of a split launch (layout_complex), GD_SPLIT_WORDS per conformer: the
   * segment masks of split sp of S at GD_SPLIT_AT(S, sp), for partial sums per split and (from
   * GD_SPLIT_MASKS on) for sums in the points' order; then for S = 1.. the first stored piece (low
   * half) and the first stored hydrogen-bond piece of the latter; last, the segments with a live
   * hydrogen-bond term */
  const unsigned *split_plan;
  const int4 *seg;            /* [n_prt*GD_MAX_SEG] */
  const int *seg_count;       /* [n_prt] */
  const float4 *kde;          /* [pnk] x, y, z, 0: sorted by type, in their given order within one */
  const int *kde_start;       /* [GD_MAXTP2 + 1] the first KDE point of each ligand type */
  const float4 *mcs;          /* [pos*mcs_ld] x, y, z, 0 (x invalid: GD_MCS_INVALID_COORD) */
  const float *mcs_tcc;       /* [pos] */
  const float *psp;           /* [GD_MAXTP2*psp_ld] */
  const float *minus_beta;    /* [n_tmp] */
  const int *ref_start;       /* [n_prt*(lna+1)] */
  const float4 *ref_pts;      /* [ref_start[n_prt*(lna+1)-1]] */
  /* Within each segment the points run by distance from the pocket centre. far_cnt[(pc *
   * GD_MAX_SEG + seg) * GD_FAR_BINS + b]: how many of the segment's points lie closer than
   * (b + 1) / far_inv_w to the centre (all of them at the last bin). A point further than
   * far_r + (an atom's distance from the centre) from the centre is further than far_r from
   * the atom, where every type pair's pmf exponent is below -25.5 in base 2. */
  const unsigned short *far_cnt;
  float far_r, far_inv_w;
  /* the far fields (gd_farfield.cu; ff_tab null: none). Cell c's table is number ff_id[c] (-1:
   * not tabulated) of its conformer's ff_cells, ff_fields series of GD_FF_NC coefficients: ele,
   * then vdw of ligand type t at 1 + ff_slot[t]. ff_pmf[(pc * GD_FAR_BINS + bin) * GD_MAXTP2 + t]:
   * the far points' pmf sum. A cell's far points: in each segment those past the count of bin
   * gd_ff_bin(cell) + ff_extra[point type]. */
  const float *ff_tab;
  const short *ff_id;
  const double *ff_pmf;
  const float *ff_cert;       /* [n_prt*n_lig] what the far points' sums may differ by, per pose */
  int ff_fields, ff_cells;
  float ff_r;                 /* r_f: a cell's far points are at least this far from its atoms */
  unsigned char ff_slot[GD_MAXTP2], ff_extra[GD_MAXTP1 + 2];
};

#ifdef __CUDACC__
/* The far-field cell of a position, -1 outside the cube (a NaN position is outside). */
__device__ __forceinline__ int gd_ff_cell(const GdDevComplex &cx, float x, float y, float z) {
  const float inv = 1.0f / GD_FF_EDGE, n = (float)GD_FF_N, o = 0.5f * GD_FF_N;
  const float fx = floorf((x - cx.pocket[0]) * inv + o), fy = floorf((y - cx.pocket[1]) * inv + o),
              fz = floorf((z - cx.pocket[2]) * inv + o);
  if (!(fx >= 0.0f && fx < n && fy >= 0.0f && fy < n && fz >= 0.0f && fz < n)) return -1;
  return ((int)fz * GD_FF_N + (int)fy) * GD_FF_N + (int)fx;
}
/* Radius bin of a far-field cell: every point past the bin's counts lies beyond the box's
 * largest distance from the pocket centre plus ff_r. GD_FAR_BINS - 1 counts every point. */
__device__ __forceinline__ int gd_ff_bin(const GdDevComplex &cx, int cell) {
  const int ix = cell % GD_FF_N, iy = (cell / GD_FF_N) % GD_FF_N, iz = cell / (GD_FF_N * GD_FF_N);
  const int mx = max(GD_FF_N / 2 - ix, ix + 1 - GD_FF_N / 2),
            my = max(GD_FF_N / 2 - iy, iy + 1 - GD_FF_N / 2),
            mz = max(GD_FF_N / 2 - iz, iz + 1 - GD_FF_N / 2);
  const float rho = GD_FF_EDGE * sqrtf((float)(mx * mx + my * my + mz * mz)) + cx.ff_r;
  return (int)fminf(rho * cx.far_inv_w, (float)(GD_FAR_BINS - 1));
}
/* First far slot of segment sg (range and type g) for a cell of that bin: an even slot, or the
 * segment's end. */
__device__ __forceinline__ int gd_ff_near(const GdDevComplex &cx, int pc, int sg, const int4 g,
                                          int bin) {
  const int b = min(bin + (int)cx.ff_extra[g.z], GD_FAR_BINS - 1);
  const int n = cx.far_cnt[((size_t)pc * GD_MAX_SEG + sg) * GD_FAR_BINS + b];
  return min(g.y, g.x + ((n + 1) & ~1));
}
#endif

/* One CTA's unit of work: `count` consecutive replicas of one protein conformer. */
struct GdTileDesc {
  int complex_index, prt_conf, rep_begin, count;  /* rep_begin: global replica index */
};

struct GdForceConst {
  float lj1, el0, el1, a1, b1, inv_el1;
  float near2;                /* (1 / el1)^2: soft-core electrostatics inside */
  float kde2, kde3;
  float a_para[GD_MAXWEI], b_para[GD_MAXWEI], w[GD_MAXWEI];
  float hpl0[GD_MAXTP2], hpl1[GD_MAXTP2], hpl2[GD_MAXTP2];
};

/* Delayed-acceptance state read by the exact kernel in mode 3 (device-resident). Survivors of
 * the surrogate stage are compacted per (complex, protein conformer) group into pose slots
 * [group_b0[g], group_b0[g] + count[g]); pose_rep maps a slot to its replica. */
struct GdDaEpi {
  const int *group_b0;        /* [n_groups] */
  int n_groups, n_rep;
  const int *pose_rep;        /* [n_rep] */
  const float *s_new;         /* [n_rep] surrogate energy of the proposal */
  float *s_cur;               /* [n_rep] surrogate energy of the current pose */
  const float *u2;            /* [n_rep] final accept uniform (the plain step's) */
  const int *active;          /* [n_complex] surrogate stage on */
  int *acc, *plain_acc;       /* [n_rep] accepted moves with the stage on / off */
  double *err2;               /* [n_rep] sum of (S_new - E_new)^2 with the stage on */
  int *nerr;                  /* [n_rep] its count */
  float *smp_t;               /* [smp_cap] training targets (collect steps) */
  long long smp_cap;
  float *tr_s, *tr_e;         /* decision trace, [n_rep*tr_cap] or null */
  int *tr_flag;
  int tr_cap, tr_step0;
};

/* What the Monte Carlo kernel is compiled for: plain steps and evaluations, delayed acceptance's
 * exact stage, the exchange groups left open (gd_exchange_group). */
enum { GD_KIND_PLAIN = 0, GD_KIND_DA = 1, GD_KIND_EXCHANGE = 2 };
/* How it treats an atom's work: one lane; several, each with partial sums; several, whose sums run
 * in the points' order. */
enum { GD_UNSPLIT = 0, GD_SPLIT_PARTIAL = 1, GD_SPLIT_ORDERED = 2 };

/* The replica state that exchanges read and write, and their draws' seed. */
struct GdExchange {
  gd_replica *replica;
  const float *etotal;
  const gd_energy *e_old;
  int *acs;                   /* exchanges taken, per replica */
  uint64_t seed;
};

/* Arguments of the fused Monte Carlo / energy kernel. */
struct GdMcArgs {
  const GdDevComplex *cx;     /* [n_complex] */
  const GdPairParam *pp;      /* [GD_MAXTP2*GD_MAXTP1] */
  const GdTileDesc *tiles;    /* [n_tiles], or null: tile i is poses [i u.count, ..) of u, up to u_n */
  GdTileDesc u;               /* (complex, protein conformer, ligand conformer in rep_begin, count) */
  int u_n;
  int n_tiles;
  int *tile_counter;          /* persistent-CTA work queue head */
  int mode;                   /* 0: MC steps, 1: init (energy at movematrix 0), 2: eval poses,
                                 3: delayed-acceptance exact stage (eval + decision), 4: eval
                                 given placed coordinates */
  int n_steps;                /* steps in this launch (mode 0) */
  int step0;                  /* step number of the first step (s1 + s2), added to *step_base */
  const int *step_base;       /* device cursor for graph replays (null: 0) */
  int chunk;                  /* protein points per shared-memory buffer (multiple of 4) */
  int fold;                   /* slots after which a segment's FP32 sums go to FP64 (divides chunk) */
  int split;                  /* lanes per ligand atom (protein split), >= 1 */
  int pieces, hpieces;        /* split launches whose sums run in the points' order: stored pieces
                                 per atom and sum, of them hydrogen-bond pieces (0: partial sums
                                 per split, added in split order) */
  int move_kind;
  uint64_t seed;
  float move_scale[6];
  /* replica state, global replica index */
  gd_replica *replica;
  float *mm_old;              /* [n_rep*6] */
  gd_energy *e_old;
  float *etotal;
  int *n_accept;
  /* records */
  gd_record_step *rec;        /* [n_rep*rec_cap] or null */
  int *rec_next;              /* [n_rep] */
  int rec_cap;
  /* trace (replay) */
  float *trace_e;             /* [n_rep*trace_cap] or null */
  int *trace_acc;
  int trace_cap, trace_step0;
  /* pose evaluation (mode 2): pose i of the tile uses mm_in[(rep_begin - 0 + j)*6] */
  const float *mm_in;
  const int *lig_conf_in;     /* per pose ligand conformer (mode 2) */
  gd_energy *e_out;
  /* mode 4: pose i's atoms at xyz_in[(i * lna + atom) * 3 + {0,1,2}], its centre at
   * center_in[i * 3 + {0,1,2}] (the lab frame, as Ligand.coord_new) */
  const float *xyz_in;
  const float *center_in;
  unsigned *err;              /* device error word */
  long long timeout_ns;       /* bounded waits */
  /* mode 3: tile.count holds (group << 8) | capacity; the survivors come from da_cnt */
  const GdDaEpi *da;
  const int *da_cnt;          /* [n_groups] survivors this step */
  int *da_cnt_next;           /* [n_groups] the next step's counters; block 0 zeroes the
                                 range [da_g0, da_g1) this launch serves */
  int da_g0, da_g1;
  int da_collect;             /* collect step: stage off everywhere, targets stored */
  /* ExchangeReplicas_d fused into mode 0 (launches that cover whole groups and one exchange
   * interval): per-group counts of replicas written back in this launch, the complexes' first
   * group, the exchange counters, and the exchange call (*x_call_base + x_call_off); mode_t
   * = !(((s mod x_spd) / x_spe) % 2) for the interval starting at step s, as the reference's
   * launcher derives it from the step within the dump window */
  int *x_done;                /* [n_groups] zeroed before the launch, or null */
  const int *x_group_base;    /* [n_complex] */
  int *x_acs;                 /* [n_rep] */
  const int *x_call_base;
  int x_call_off, x_spd, x_spe;
  /* exchange groups (global numbers) whose decisions wait for the pair loop's energies: x_open[0]
   * of them in x_open_list, taken by the GD_KIND_EXCHANGE launch that follows (its CTAs check out
   * in x_open[1]); it takes mode_t from x_mode_t, or (-1) from the step as above */
  int *x_open, *x_open_list;
  int x_mode_t, x_open_cap, n_complex;
};

#endif
