// ccfv_internal.h -- device-side data structures and launchers shared by the
// translation units of libccfv (not part of the public ABI).
#pragma once

#include <cstddef>
#include <cuda_runtime.h>
#include <cstdint>

namespace ccfv {

enum { BC_COMPAT = 0, BC_PERIODIC = 1 };
enum { VEL_REF_ROT4 = 0, VEL_CONST = 1, VEL_ROTATION = 2, VEL_SWIRL = 3 };

// Device status word bits (set by kernels, read by ccfv_check).
enum : unsigned { STATUS_HALO = 1u };

// Tile geometry of the fused sweep kernel.  A CTA owns LPG lines and a run
// of consecutive cells (positions) of those lines; a thread-block cluster of
// `cs` CTAs covers whole lines.  Lines sit in the fast (lane) index of the
// shared-memory tile, positions in the slow index, so every phase of the
// kernel reads shared memory without bank conflicts in both directions.
constexpr int LPG = 16;          // lines per tile (x-sweeps: 128 B rows)
constexpr int PITCH = LPG + 1;   // odd pitch: conflict-free column access
constexpr int NW = 8;            // warps per CTA
constexpr int NTH = NW * 32;     // threads per CTA
constexpr int CPW = 32 / LPG;    // chunks per warp
constexpr int NCH = NW * CPW;    // chunks per line per CTA
constexpr int LC_MAX = 256;      // max positions per CTA
constexpr int MAX_CLUSTER = 16;  // non-portable cluster size (lines <= 4096)
constexpr int MAX_DEVICES = 64;  // device ordinals with per-device library state

// One field (one instance at one time slice) in one sweep launch.
// x-sweep: lines are columns j (s_line = 1, s_pos = ny), positions i.
// y-sweep: lines are rows i (s_line = ny, s_pos = 1), positions j.
struct SweepField {
  void *data;            // T[ny*nx]: swept in place (pp = 0), or buffer A (pp = 1)
  void *data2;           // pp = 1: buffer B
  const void *in0;       // pp = 1: input of the first sweep of the sequence
  long long s_pos;       // element stride between positions of a line
  long long s_line;      // element stride between lines
  int L;                 // cells per line
  int M;                 // lines
  int dir;               // 0: x-sweep, 1: y-sweep
  int bc;                // BC_*
  int vel;               // VEL_*
  int group0;            // first tile index of this field in the launch
  int groups;            // tiles of this field = ceil(M / LPG)
  int dsrc;              // foot derivative of: 0 the sweep input, 1 the remapped field
  int hd;                // dsrc = 1: halo (cells) of the remapped field
  int uniform;           // 1: the velocity along the sweep depends only on the
                         // transverse coordinate (every foot of a line has the
                         // same displacement): stencil fast path
  int jf;                // filter kernel: recurrence warm-up length J
  int cta0;              // filter kernel: first CTA of this field in the launch
                         // (a multiple of the launch's cluster size)
  int halo_f;            // filter kernel: staged halo (cells) of this field
  // Batched launches (all zero for single-instance launches):
  int inst;              // instance index into the launch's `nlo` array
  int slice;             // >= 0: fixed slice of this field; -1: the launch's slice
  int jmax;              // the field takes part while jstep < jmax (0: always)
  int smax;              // slice-indexed fields: while slice < smax
  int gskip;             // slice-indexed fields: skip slice == nlo (zero increment)
  int jmin;              // ... and while jstep >= jmin
  int s0, sj;            // pass of the launch in an out-of-place sequence: s0 + sj jstep
  int pp;                // 1: out-of-place sequence: pass s writes A when s + par is
                         // odd, else B, and reads the other buffer (in0 for s = 0);
                         // 0: in place on `data`
  int par;               // pp = 1: parity offset (chosen so the last sweep writes A)
  int phase;             // slice-indexed fields: 0 every launch, 1 only while the
                         // instance's nlo < 0 (first coarse sweep), 2 only while
                         // nlo >= 0 (Parareal iterations)
  int src;               // source term: 0 none (the reference's f = 0), 1 Gaussian
  int src_tb;            // 1: the remapped source is f(t_b) too (third sub-step), else f(t_a)
  double sp[5];          // Gaussian source: sp0 exp(-((x-sp1)^2+(y-sp2)^2)/sp3) cos(sp4 t)
  double src_w;          // RHS weight of (remapped f(t_a or t_b) + f(t_b))
  double t_step;         // added per launch step: time = ... + jstep * t_step
  double t_slice;        // added per launch slice: time = ... + slice * t_slice
  double vp[4];          // velocity parameters
  double s_min, s_max, h;  // along-line edge coordinates: s_min + h*e
  double t_min, ht;        // transverse edges: t_min + ht*line
  double Dt;               // sub-step length
  double ta_rel, tb_rel;   // foot-tracing interval relative to the launch time
  double eps_remap;        // compat remap clamp (x: 1e-15, y: 1e-16)
  double kb;               // (1-theta)*K*(Dt/h): RHS diffusion coefficient
  double theta;            // implicit weight of the diffusion (0.5: Crank-Nicolson);
                           // host bookkeeping: the kernels read kb and the tables
  double inv12h;           // 1/(12 h)
  double sm_fac;           // periodic, scan kernels: a / gamma; filter kernel: mu
  double sm_inv_den;       // periodic, scan kernels: 1 / (1 + z0 + (a/gamma) z_{L-1});
                           // filter kernel: 1 / c
  const void *tab;         // T[3L]: alpha_k | g_k | z_k (solver factors)
  // Streaming kernels only (the tile kernels' copy of a descriptor ends here)
  int jd;                // cells over which a carry decays below rounding (jf, or more
                         // where the recurrences need no warm-up)
  int rk_tail;           // compat: the second term of the rank-one closure matters
  double rk_a;             // compat: mu^2 / (1 - mu^(2L+2)), rank-one closure
  // exact form, q = -mu: q^n of a whole segment and of the line's last one,
  // 1/(1 - q^2), 1/(1 - q^L), q^n of the last lane of the last one, and
  // q^-(positions that this lane walks behind it), 0 where that is above 2^24
  double ex[6];
  // per-line stencil of w's input, computed once per plan (the velocity fields
  // it serves do not depend on time).  wt: T[lines][stencil_taps(variant)];
  // nt: int[lines] shifts.
  const void *wt;
  const int *nt;
};

// Whether a field takes part in a batched launch (`nlo[inst]`: the first
// active slice of every instance, -1 before the first coarse sweep; null: a
// single-instance launch, always active).  The batched engine evaluates the
// same rule on the host to skip launches in which no field is active.
__host__ __device__ inline bool field_active(const SweepField &f, int jstep, int nslice,
                                             const int *nlo) {
  if ((f.jmax > 0 && jstep >= f.jmax) || jstep < f.jmin) return false;
  if (!nlo) return true;
  const int lo = nlo[f.inst];
  if (f.slice >= 0) return f.slice >= lo;
  if ((f.phase == 1 && lo >= 0) || (f.phase == 2 && lo < 0)) return false;
  return nslice < f.smax && nslice >= lo + f.gskip;
}

// Shared-memory slot of one descriptor at the head of every tile kernel's
// dynamic shared memory (the data behind it stays 64-byte aligned).
constexpr size_t FD_COPY = offsetof(SweepField, jd);
constexpr size_t FD_BYTES = (FD_COPY + 63) & ~size_t(63);
static_assert(FD_COPY % 8 == 0 && FD_BYTES == 384, "bounds the steps that are taken");

// Kernel variants: the per-cell kernel (any velocity / boundary / scheme) and
// the fused stencil kernel (uniform displacement, periodic, derivative of the
// sweep input).
// SWEEP_GENERAL_SRC is the per-cell kernel with the source tile staged.
// The streaming kernels (stream.cu) run SWEEP_FILTER (warm-up between a line's
// segments), SWEEP_FILTER_EXACT (the line closed exactly: any diffusion number),
// SWEEP_CELL / SWEEP_CELL_EXACT (the same with a per-cell right-hand side: feet
// that differ from edge to edge) and, with the reference's boundaries,
// SWEEP_COMPAT and (the reference scheme's third sweep, derivative of the
// remapped field) SWEEP_COMPAT_D.  SWEEP_FILTER_XX: the last x sweep of a step
// and the first of the next one in one pass over the field.
// SWEEP_CELL_COMPAT: the tile kernel with the reference's boundaries.
enum { SWEEP_GENERAL = 0, SWEEP_FAST = 1, SWEEP_FILTER = 2, SWEEP_GENERAL_SRC = 3,
       SWEEP_FILTER_EXACT = 4, SWEEP_CELL = 5, SWEEP_CELL_EXACT = 6, SWEEP_CELL_COMPAT = 7,
       SWEEP_COMPAT = 8, SWEEP_COMPAT_D = 9, SWEEP_FILTER_XX = 10 };
inline bool stream_variant(int v) {
  return v == SWEEP_FILTER || v == SWEEP_COMPAT || v == SWEEP_COMPAT_D ||
         v == SWEEP_FILTER_XX || v == SWEEP_CELL || v == SWEEP_FILTER_EXACT ||
         v == SWEEP_CELL_EXACT;
}
// Variants with the factored solve.
inline bool filter_variant(int v) {
  return stream_variant(v) || v == SWEEP_CELL_COMPAT;
}
// Warm-up (segmented) forms: lines longer than MAX_CLUSTER segments are
// allowed out of place.
inline bool warm_filter_variant(int v) {
  return (stream_variant(v) && v != SWEEP_FILTER_EXACT && v != SWEEP_CELL_EXACT) ||
         v == SWEEP_CELL_COMPAT;
}
// Variants whose right-hand side is the per-line stencil table (SweepField::wt),
// and its values per line.
inline bool stencil_filter_variant(int v) {
  return stream_variant(v) && v != SWEEP_CELL && v != SWEEP_CELL_EXACT;
}
constexpr int STREAM_TAPS_C = 10;   // 8 taps, the feet's offset in a cell last
constexpr int STREAM_TAPS_D = 24;   // 8 + 13 taps, likewise
constexpr int STREAM_TAPS_XX = 16;  // 15 taps, padded
inline int stencil_taps(int v) {
  return v == SWEEP_COMPAT_D ? STREAM_TAPS_D
         : v == SWEEP_COMPAT ? STREAM_TAPS_C
         : v == SWEEP_FILTER_XX ? STREAM_TAPS_XX : 8;
}
// Variants with the per-cell right-hand side.
inline bool cell_filter_variant(int v) {
  return v == SWEEP_CELL || v == SWEEP_CELL_EXACT || v == SWEEP_CELL_COMPAT;
}
// Lines closed exactly (several segments: one cluster).
inline bool exact_filter_variant(int v) { return v == SWEEP_FILTER_EXACT || v == SWEEP_CELL_EXACT; }
constexpr int FILTER_JMAX = 64;  // longest recurrence warm-up with 16 lanes per line

// Launch geometry shared by all fields of one sweep launch.
struct LaunchGeom {
  int cs = 1, lc_max = 0, halo = 0, groups = 0, variant = 0;
  int dir = 0;            // sweep direction
  int lanes = 0;          // streaming form: lanes per line
  int rows = 0;           // streaming form: staged positions per line (at most)
  int ends = 0;           // streaming form, reference's boundaries: scratch values per
                          // line end (edges and cells next to it)
  bool strong = false;    // streaming form: warm-up past FILTER_JMAX
  int lc_fit = 0, halo_fit = 0;  // tile of the scan kernels: a step whose scan tile
                                 // does not fit is refused whatever form runs it
};

// Buffers of a single-field launch that replace its descriptor's, and how the
// pass uses them (launch_sweep).
enum { IO_IN_PLACE = 1, IO_FLIP = 2 };
struct FieldIo {
  void *data = nullptr;
  const void *in = nullptr;
  int mode = 0;
};

// The fields of a plan's launch by value: they differ only in their buffers
// and time origins, and field i's buffers lie i * stride bytes behind field
// 0's.  tiles: tiles per field (0: not known to be so, read the descriptors).
struct PlanFields {
  SweepField f = {};
  long long stride = 0;
  int tiles = 0;
  int seg = 0;  // streaming form: cells per segment
};

// Streaming form (stream.cu): positions per lane; cells per segment of a line
// of L cells in cs segments (even: pairs of cells stay aligned); lines per CTA;
// shared memory of a launch.
constexpr int STREAM_CH = 17;
constexpr int FILTER_JLONG = 8 * STREAM_CH;  // longest warm-up with 32 lanes per line
__host__ __device__ inline int stream_seg(int L, int cs) { return ((L + cs - 1) / cs + 1) & ~1; }
// Exact form: whole walks, or one segment.
__host__ __device__ inline int exact_seg(int L, int cs, int lanes) {
  return cs > 1 ? lanes * STREAM_CH : (L + 1) & ~1;
}
int stream_tile_lines(int dir, int lanes);
size_t stream_smem_bytes(const LaunchGeom &G, bool fp64);
// Lines per CTA of a launch geometry.
inline int tile_lines(const LaunchGeom &G) {
  return stream_variant(G.variant) ? stream_tile_lines(G.dir, G.lanes) : LPG;
}

// Shared-memory bytes of the sweep kernels for a launch.
size_t sweep_smem_bytes(int lc_max, int halo, bool fp64, bool source = false);
size_t sweep_fast_smem_bytes(int lc_max, int halo, bool fp64);
size_t sweep_filter_smem_bytes(int lc_max, int halo, bool fp64, bool exact = false,
                               bool cell = false);
// Longest segment (cells per CTA along a line) of the filter kernel for a
// recurrence warm-up of J cells.
int filter_segment_max(int J);
// Fills the per-line stencil table of the filter kernel for field `*d_field`
// (device descriptor): wt = T[lines][stencil_taps(variant)], nt = int[lines], lines = groups*LPG
// (lines past M get zeros).
cudaError_t launch_filter_weights(bool fp64, const SweepField *d_field, void *wt, int *nt,
                                  int lines, cudaStream_t stream, int variant = SWEEP_FILTER);

// Launches one fused sweep over all fields of `d_fields` (device array,
// sorted by group0; tiles group_base .. group_base+groups_total-1).  All fields share G: the cluster size `cs`, their
// max positions per CTA `lc_max` and the halo `halo` (LaunchGeom).  `toff` is added to
// every field's ta_rel/tb_rel (the launch time); `data` (if non-null)
// replaces fields[0].data and `in` (if non-null, else `data`) its in0
// (single-field launches).  `jstep` is the step of an out-of-place sequence
// (SweepField::pp); `mode`: IO_IN_PLACE writes this pass over its input,
// IO_FLIP exchanges the two buffers of a pass; `inplace` says whether any field
// sweeps in place (the filter kernel's segments of a line then form a
// cluster).  `plan`: the same fields by value where they allow it (see
// PlanFields; the streaming form then reads no descriptor).
template <typename T>
cudaError_t launch_sweep(const LaunchGeom &G, const PlanFields &plan, const SweepField *d_fields,
                         int nfields, int group_base, int groups_total, double toff,
                         const FieldIo &io, unsigned *d_status, cudaStream_t stream,
                         int jstep = 0, bool inplace = true);

// Batched form: `jstep` / `nslice` select the step and slice of this launch,
// `nlo[inst]` the first active slice of every instance (see SweepField).
struct BatchStep {
  int jstep = 0, nslice = 0;
  const int *nlo = nullptr;
  bool inplace = true;
  bool pdl = false;            // programmatic dependent launch
  const int *g0idx = nullptr;  // the fields' group0 values (device), or null
};
template <typename T>
cudaError_t launch_sweep_batch(const LaunchGeom &G, const SweepField *d_fields, int nfields,
                               int group_base, int groups_total, const BatchStep &bs,
                               unsigned *d_status, cudaStream_t stream);
// The streaming form's launch (stream_variant), called by the two above.
template <typename T>
cudaError_t launch_stream(const LaunchGeom &G, const PlanFields &plan, const SweepField *d_fields,
                          int nfields, int group_base, int groups_total, double toff,
                          const FieldIo &io, unsigned *d_status,
                          int jstep, int nslice, const int *nlo, bool inplace,
                          cudaStream_t stream, const int *g0idx, bool pdl);

// Solver-table layout (T values): alpha[L] g[L] z[L] tP[L] tS[L]
// aggA[cs*NCH] PA[cs*(NCH+1)], where, for the chunk partition the sweep
// kernels use (cs = ceil(L/LC_MAX) CTAs per line, NCH chunks per CTA),
// tP[k] / tS[k] are the products of alpha from the chunk start to k / from k
// to the chunk end, aggA the chunk products and PA the CTA-local exclusive
// prefix products of the chunks (PA[NCH] = product over the CTA).
inline int table_cs(int L) { return (L + LC_MAX - 1) / LC_MAX; }
inline size_t table_len(int L) {
  const int cs = table_cs(L);
  return 5 * (size_t)L + (size_t)cs * NCH + (size_t)cs * (NCH + 1);
}
// Fills tP, tS, aggA, PA of a table whose alpha is already in place
// (heap-free; T = double or float, computed in double).
template <typename T>
void fill_chunk_products(int L, T *tab);

// Resident coarse propagator (coarse.cu): the whole G phase of one
// delta-form Parareal iteration of an instance whose coarse field fits in one
// SM's shared memory, one CTA per instance.  f: the instance's coarse sweep
// descriptors of the iterations (x, y, x; filter-kernel constants filled).
struct ResidentG {
  SweepField f[3];
  const double *F;  // F[0..S] fine results
  double *U;        // U[0..S] slice states (updated)
  double *norms;    // [2 (S + 1)]: sum dU^2, sum U^2 of every corrected slice
  int inst;         // index into the launch's nlo array
  int S, m, nx, ny, pitch;
};
// Dynamic shared memory of the resident kernel for an nx x ny field.
size_t resident_g_smem_bytes(int nx, int ny, bool fp64, bool cell);
// Whether an nx x ny coarse field can be resident (lines of at most 272
// cells, the field in shared memory).
bool resident_g_fits(int nx, int ny, bool fp64, bool cell);
// cell: the instances' right-hand side is per cell (else SweepField::wt / nt
// hold their stencil tables).
cudaError_t launch_resident_g(bool fp64, bool cell, const ResidentG *d_rg, int n, size_t smem,
                              const int *nlo, cudaStream_t st);

// Whether launches use programmatic dependent launch (CCFV_PDL).
bool pdl_enabled();

// Counts kernel launches made by the library.
void count_launch(uint64_t n = 1);
uint64_t launches();

}  // namespace ccfv
