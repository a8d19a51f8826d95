// stream.cu -- the streaming form of the factored sweep: velocity fields whose
// feet share one displacement per line, right-hand side from a per-line
// stencil table.
//
// The line system a x_{k-1} + b x_k + a x_{k+1} = r_k factors as
// c (1 + mu S^-1)(1 + mu S) with |mu| < 1 (sweep.cu, filter path), so a sweep
// is an eight-tap stencil of the staged cells and two first-order recurrences
//   w_k = r_k / c - mu w_{k-1},   x_k = w_k - mu x_{k+1},
// each warmed up over J cells with |mu|^J below the rounding of T.  LN lanes
// own one line's segment, SCH = 17 consecutive positions each (odd: the lanes'
// shared-memory columns are conflict free).
//
// Both directions move pairs of values with one asynchronous copy (16 bytes in
// FP64) where the pairs are aligned, single values where they are not (odd row
// length or an odd base address), and differ in how lines lie in memory:
//   y sweep (DIR 1): a line is contiguous, so a warp stages, solves and stores
//     its own one or two lines with no CTA barrier at all.  32 lanes per line
//     (544 positions) halve the warm-up of 16; short lines, where half of
//     those lanes would idle, take 16.
//   x sweep (DIR 0): 16 neighbouring lines are a 128-byte row; the CTA stages
//     rows, and lanes interleave a pair of lines (even lanes one, odd lanes the
//     other).  A row of 16 + 2 padding values keeps pairs aligned and makes the
//     half-warp's 8 chunks x 2 lines hit distinct banks: 17 * 18 / 2 is odd.
// A recurrence is walked twice per lane, first from zero for the chunk's end
// value, then from the true carry; that is two multiply-adds per position
// against the three operations of adding carry * (-mu)^i afterwards.  Carries
// decay by (-mu)^17 per lane, so the scan over lanes needs only as many
// doubling steps as the warm-up has chunks (0, 1 or 2 instead of 4).
//
// What bounds it: HBM, then issue.  A lone FP64 step of 4096^2, three passes of
// 268 MB (123 us at the copy rate), takes 183 us against 230 us for the tile
// kernel this replaced (8-byte copies, 16 lanes per line, carries added
// afterwards, two CTA barriers).  Instructions per cell: 50 an x sweep, 41 a y
// sweep, 68 two x sweeps in one pass; the tile kernel 69 a sweep.
#include <cooperative_groups.h>

#include <atomic>
#include <cstdlib>
#include <mutex>

#include "ccfv_internal.h"
#include "line_ends.cuh"
#include "sweep_device.cuh"
#include "sweep_math.cuh"

namespace cg = cooperative_groups;

namespace ccfv {

namespace {

constexpr int SCH = STREAM_CH;     // positions per lane
constexpr int X_LINES = 16;        // lines per CTA of an x sweep
constexpr int X_PITCH = X_LINES + 2;
constexpr int Y_WARPS = 4;

template <int DIR, int LN>
struct StreamCta {
  static constexpr int warps = DIR == 0 ? X_LINES * LN / 32 : Y_WARPS;
  static constexpr int lpw = 32 / LN;  // lines per warp
  static constexpr int lines = warps * lpw;
};

// One aligned pair or one value, copied asynchronously.
template <typename T>
__device__ __forceinline__ void copy_pair(T *d, const T *s) {
  if (sizeof(T) == 8) cp_async16(d, s); else cp_async8(d, s);
}
template <typename T>
__device__ __forceinline__ void copy_one(T *d, const T *s) {
  if (sizeof(T) == 8) cp_async8(d, s); else cp_async4(d, s);
}
template <typename T>
struct alignas(2 * sizeof(T)) Pair {
  T a, b;
};

__device__ __forceinline__ int wrap_pos(int pos, int L) {
  if ((unsigned)pos >= (unsigned)L) {
    pos %= L;
    if (pos < 0) pos += L;
  }
  return pos;
}

template <typename T>
__device__ __forceinline__ void load_taps(T (&o)[8], const T *__restrict__ wt) {
#pragma unroll
  for (int m = 0; m < 8; ++m) o[m] = __ldg(wt + m);
}

// v[i] (+)= sum_m o[m] C_{row + i + m}, NT taps of SCH positions (stride ES
// between positions) through a register window.
template <typename T, int ES, int NT, bool ADD>
__device__ __forceinline__ void stencil(const T *cp, const T (&o)[8], T (&v)[SCH]) {
  T q[NT];
#pragma unroll
  for (int m = 0; m < NT - 1; ++m) q[m] = cp[m * ES];
#pragma unroll
  for (int i = 0; i < SCH; ++i) {
    q[NT - 1] = cp[(NT - 1 + i) * ES];
    T t = ADD ? v[i] + o[0] * q[0] : o[0] * q[0];
#pragma unroll
    for (int m = 1; m < NT; ++m) t += o[m] * q[m];
    v[i] = t;
#pragma unroll
    for (int m = 0; m < NT - 1; ++m) q[m] = q[m + 1];
  }
}

// ---- the reference's boundaries (BND 1, 2) ----
//
// Cells whose stencil reaches a clamped or ghost cell, a few at either end of
// a line, take the reference's per-cell formulas; every other cell of the line
// takes the stencil.  The recurrence inputs r_k of those positions are
// prepared before the walk, the left end's by the first half of the line's
// lanes and the right end's by the second half at the same time: one foot,
// PPM integral and derivative per edge (not per cell and side), edges and
// cells spread over the half's lanes.
//
// Region of one end: positions [ka, kb) need r; that needs b of [ba, bb), the
// edges of those cells and, when the sweep differentiates the remapped field
// (BND 2), the remapped cells [ra, rb).
struct EndRegion {
  int ka, kb, ba, bb, ra, rb;
};

// Cells of one line in shared memory: position -> staged value (zero outside
// the line but for the four ghost cells).  near(k): whether the cells that a
// foot in cell k reads, k - 3 .. k + 3, are staged.
template <typename T, int ES>
struct StagedLine {
  T *c;  // cell 0
  int b0, b1;
  unsigned *status;
  __device__ __forceinline__ T operator()(int pos) const { return c[pos * ES]; }
  __device__ __forceinline__ bool near(int k) const {
    if (k - 3 >= b0 && k + 3 < b1) return true;
    atomicOr(status, STATUS_HALO);
    return false;
  }
};

// FootCell of a foot, clamped by eps to the line (T2S4:322-324, 414-415, 452-455).
__device__ __forceinline__ FootCell foot_cell(const SweepField &F, double f, double eps) {
  const double x = fmin(fmax(f, F.s_min + eps), F.s_max - eps);
  FootCell r;
  // the cell decides between ghosts: the reference's quotient, rounded alike
  r.k = (int)floor((x - F.s_min) / F.h);
  r.xi = (x - (F.s_min + F.h * r.k)) * (12.0 * F.inv12h);
  return r;
}
// edge_foot (sweep_math.cuh) of the velocity fields that do not depend on the
// position along the line, nor on time: Heun's two speeds are one.
__device__ __forceinline__ double line_foot(const SweepField &F, int line, int e) {
  const double s = F.s_min + F.h * e;
  auto corner = [&](double tau) {
    const double w = F.vel == VEL_REF_ROT4 ? (F.dir == 0 ? -4 * tau : 4 * tau)
                     : F.vel == VEL_CONST
                         ? (F.dir == 0 ? F.vp[0] : F.vp[1])
                         : (F.dir == 0 ? -F.vp[0] * (tau - F.vp[2]) : F.vp[0] * (tau - F.vp[1]));
    return s - 0.5 * F.Dt * (w + w);
  };
  const double tau0 = F.t_min + F.ht * (double)line;
  return 0.5 * (corner(tau0) + corner(tau0 + F.ht));
}
// The derivative's clamp of a foot on the end of the line (rare: kept out of
// the kernels, whose single pass over their code is bound by fetching it).
__device__ __noinline__ FootCell end_foot_cell(const SweepField &F, int line, int e) {
  return foot_cell(F, line_foot(F, line, e), 1e-15);
}

// Remap of one cell over [fl, fr] (T2S4:306-347, 396-438), its left foot clamped
// from below and its right one from above only: a left foot on the upper edge
// itself lies in no cell and the right one still counts the last cell.
template <typename T, typename V>
__device__ __noinline__ T remap_at_end(const SweepField &F, const V &cells, int line, int k) {
  const int L = F.L;
  const double fl = line_foot(F, line, k), fr = line_foot(F, line, k + 1);
  if (fl > F.s_max || fr < F.s_min || fl == fr) return T(0);
  const double xl = fmax(fl, F.s_min + F.eps_remap), xr = fmin(fr, F.s_max - F.eps_remap);
  const int kl = (int)floor((xl - F.s_min) / F.h), kr = (int)floor((xr - F.s_min) / F.h);
  if (!cells.near(kl) || !cells.near(kr)) return T(0);
  const T il = kl >= 0 && kl < L ? ppm_to(cells, kl, T((xl - (F.s_min + F.h * kl)) / F.h)) : T(0);
  const T ir = kr >= 0 && kr < L ? ppm_to(cells, kr, T((xr - (F.s_min + F.h * kr)) / F.h)) : T(0);
  if (kl == kr) return ir - il;
  T v = (kl >= 0 && kl < L ? cells(kl) : T(0)) - il;
  for (int j = kl + 1; j < min(kr, L); ++j) v += cells(j);
  return v + ir;
}

// Feet of the edges that the region's positions need, by HL lanes (this one:
// hc): kf, the cell with a mark for feet outside the line (zero inflow); d, the
// offset in the cell `at`, which is NO_CELL where the foot lies in no cell.
// They depend on the plan alone: done before the launch waits for its
// predecessor.
template <typename T, bool REMAPPED, int HL>
__device__ __forceinline__ void end_feet(const SweepField &F, int line, int n0, double x0,
                                         const EndRegion &R, int hc, T *at, T *d, int *kf) {
  const int L = F.L, e0 = REMAPPED ? R.ra : R.ba, e1 = REMAPPED ? R.rb : R.bb;
  if (R.ka >= R.kb) return;
  // Every foot of a line sits at the same offset n0 + x0 from its edge: one
  // clear of the ends needs no quotient of its own, one a cell beyond them lies
  // in no cell and neither do those of its cell.
  for (int e = e0 + hc; e <= e1; e += HL) {
    const int j = e + n0;
    int mark = j < 0 ? FOOT_BELOW : FOOT_ABOVE + L;
    FootCell p{j, x0};
    const bool cell = j > -2 && j < L + 1;
    if (cell) {
      mark = j;
      if (j < 2 || j > L - 4) {
        const double f = line_foot(F, line, e);
        p = foot_cell(F, f, F.eps_remap);
        mark = f < F.s_min               ? FOOT_BELOW
               : f > F.s_max             ? FOOT_ABOVE + p.k
               : f < F.s_min + F.eps_remap || f > F.s_max - F.eps_remap ? FOOT_ON_END
                                                                        : p.k;
      }
    }
    at[e - e0] = cell ? T(p.k) : T(NO_CELL);
    d[e - e0] = T(p.xi);
    kf[e - e0] = mark;
  }
}

// r_k = (1/12c)(b_{k-1} + 10 b_k + b_{k+1}) of the region's positions into
// `d`, from the feet that end_feet left (phi: their cells).  phi / d / tmp / kf:
// scratch of the half.  All lanes of the warp call it (empty region: nothing but
// the barriers).
template <typename T, int ES, bool REMAPPED, int HL>
__device__ __forceinline__ void end_inputs(const SweepField &F, const StagedLine<T, ES> &cells,
                                           int line, int n0, const EndRegion &R, int hc,
                                           T *phi, T *d, T *tmp, int *kf) {
  tmp += 2;  // room for two ghosts on either side
  const int L = F.L;
  const T kbc = T(F.kb), inv12h = T(F.inv12h);
  const bool any = R.ka < R.kb;
  // PPM integral of the feet's cells and derivative of the staged cells
  const int e0 = REMAPPED ? R.ra : R.ba, e1 = REMAPPED ? R.rb : R.bb;
  if (any)
    for (int e = e0 + hc; e <= e1; e += HL) {  // this lane's own edges
      const int i = e - e0;
      T ph = phi[i], dv = d[i];
      if (!foot_inputs<REMAPPED>(cells, L, inv12h, kf[i], F.eps_remap != 1e-15,
                                 [&] { return end_foot_cell(F, line, e); }, ph, dv))
        kf[i] = FOOT_ABOVE;
      phi[i] = ph;
      d[i] = dv;
    }
  __syncwarp();
  // remapped cells: whole cells between the feet plus the two integrals
  // (T2S4:306-347, 396-438); zero from outside the line
  T *const b = REMAPPED ? phi : tmp;
  const int c0 = REMAPPED ? R.ra : R.ba, c1 = REMAPPED ? R.rb : R.bb;
  if (any)
    for (int k = c0 + hc; k < c1; k += HL) {
      const int kl = kf[k - e0], kr = kf[k + 1 - e0];
      T v = T(0);
      if (kl == FOOT_ON_END || kr == FOOT_ON_END) {
        v = remap_at_end<T>(F, cells, line, k);
      } else if (kl < FOOT_ABOVE && kr != FOOT_BELOW) {
        const int l = max(kl, 0), r = min(kr & (FOOT_ABOVE - 1), L);
        for (int j = l; j < r; ++j) v += cells(j);
        v = (v + phi[k + 1 - e0]) - phi[k - e0];
      }
      if (!REMAPPED) v += kbc * (d[k + 1 - e0] - d[k - e0]);
      tmp[k - c0] = v;
    }
  __syncwarp();
  if (REMAPPED) {
    // derivative of the remapped field at the edges of [ba, bb)
    // (T2S4:929-932), its ghosts from the three remapped end cells
    if (any && hc == 0) {
      if (R.ra == 0) ghosts(tmp[0], tmp[1], tmp[2], tmp[-1], tmp[-2]);
      T *z = tmp + (L - 1 - R.ra);
      if (R.rb == L) ghosts(z[0], z[-1], z[-2], z[1], z[2]);
    }
    __syncwarp();
    auto remapped = [&](int k) -> T { return tmp[k - R.ra]; };
    if (any)
      for (int e = R.ba + hc; e <= R.bb; e += HL) {
        int k = kf[e - e0];
        T xi = d[e - e0], dv = T(0);
        if (k == FOOT_ON_END) {  // inside [s_min, s_max], within the clamp
          const FootCell q = end_foot_cell(F, line, e);
          k = q.k;
          xi = T(q.xi);
        }
        if (k >= 0 && k < FOOT_ABOVE)
          dv = derivative_at(remapped, k, xi, L, inv12h);
        d[e - e0] = dv;
      }
    __syncwarp();
    if (any)
      for (int k = R.ba + hc; k < R.bb; k += HL)
        b[k - R.ba] = tmp[k - R.ra] + kbc * (d[k + 1 - e0] - d[k - e0]);
    __syncwarp();
  }
  // compact mass matrix, b = 0 outside the line (T2S4:616-634)
  if (any) {
    const T icw = T(F.sm_inv_den / 12.0);
    for (int k = R.ka + hc; k < R.kb; k += HL) {
      const T bm = k > R.ba ? b[k - 1 - R.ba] : T(0), bp = k + 1 < R.bb ? b[k + 1 - R.ba] : T(0);
      d[k - R.ka] = icw * ((bm + bp) + T(10.0) * b[k - R.ba]);
    }
  }
  __syncwarp();
}

// What a CTA needs of its field.
struct StreamField {
  int L, M, J, JD, H, groups, cta0;
  long long s_line, s_pos;
  double mu;
  const void *wt;
  const int *nt;
};
__device__ __forceinline__ StreamField stream_field(const SweepField &f) {
  return StreamField{f.L, f.M, f.jf, f.jd, f.halo_f, f.groups, f.cta0, f.s_line, f.s_pos, f.sm_fac,
                     f.wt, f.nt};
}

// ---- feet that differ from edge to edge: the swirling field (BND 4) ----
//
// Speed along the line a(tau, t) sin^2(pi s): an edge's two corners share
// sin(pi s) and cos(pi s) (a table of the CTA's edges), and the speed at the
// predicted point s - Dt w is that of a small angle z away, so a corner foot is
// a short series instead of a sine of its own: orders 5 and 4 below 2^-8 (5e-18
// left out), 7 and 8 below 2^-5 (2e-18); longer steps call sinpi.  A loop over the
// edges two at a time: unrolled whole, the kernel waits for its instructions
// (23 us a sweep of 1024^2 against 18 us; the tile kernel, a sine per corner and
// divisions per edge, took 51 us).
template <int N>
struct Series {
  static constexpr int value = N;
};
struct CornerLine {
  double wb, wa, z;  // a(tau, tb), a(tau, ta), pi Dt a(tau, tb)
};
__device__ __noinline__ double far_sine(double x) { return sinpi(x); }
// w(s, tb) + w(s - Dt w, ta) of one corner; series: 2, 1 or 0 as above.
template <int series>
__device__ __forceinline__ double corner_speeds(const CornerLine &l, double S, double C, double s,
                                                double Dt) {
  const double s2 = S * S, w = l.wb * s2;
  double q;
  if (series) {
    const double z = l.z * s2, z2 = z * z;
    double a = 1.0 / 120, b = 1.0 / 24;
    if (series == 1) {
      a += z2 * (-1.0 / 5040);
      b += z2 * (-1.0 / 720 + z2 * (1.0 / 40320));
    }
    const double sn = z + z * z2 * (-1.0 / 6 + z2 * a);
    q = S + S * z2 * (-0.5 + z2 * b) - C * sn;
  } else {
    q = far_sine(s - Dt * w);
  }
  return w + l.wa * (q * q);
}

// One edge: its foot's cell, the PPM integral (T2S4:63-65, 260-304) and 12 h
// times the derivative at the foot (T2S4:440-547), both as polynomials of the
// offset in the cell, and the foot cell's value.  u: the foot in cells from its
// edge e (not from the line's start, where it would round to 1e-13 of a cell on
// a line of 1024).  A cell outside the staged rows (cannot happen) is replaced and
// marked in `bad`.
template <typename T>
struct SwirlEdge {
  int kf;
  T phi, d, z;
};
template <typename T, int ES>
__device__ __forceinline__ SwirlEdge<T> swirl_edge(int e, double u, const T *cells, int b0,
                                                   int rows, int &bad) {
  SwirlEdge<T> r;
  // floor by the rounding of u - 1/2 + 1.5 2^52 (an exact cell edge may count
  // as either cell's: the integrals meet there)
  const double t = (u - 0.5) + 6755399441055744.0;
  r.kf = e + __double2loint(t);
  const T x = T(u - (t - 6755399441055744.0));
  const int row = r.kf - b0, at = min(max(row, 2), rows - 3);
  bad |= row ^ at;
  const T *c = cells + at * ES;
  const T m2 = c[-2 * ES], m1 = c[-ES], z = c[0], p1 = c[ES], p2 = c[2 * ES];
  // left and right edge values, PPM integral x (cl + x (a + x b))
  const T dm = z - m1, e0 = m2 - p1, s1 = m1 + p1;
  const T cl = T(7.0 / 12.0) * (z + m1) - T(1.0 / 12.0) * (p1 + m2);
  const T cr = T(7.0 / 12.0) * (p1 + z) - T(1.0 / 12.0) * (p2 + m1);
  const T cs = cl + cr;
  r.phi = x * (cl + x * ((T(3.0) * z - cs) - cl + x * (cs - T(2.0) * z)));
  // derivative: c0 + x (3 c1 + x (-6 c2 + 2 x c3))
  const T c0 = e0 + T(15.0) * dm, c2 = e0 + T(3.0) * dm;
  const T c1 = (m2 - p2) + T(2.0) * m1 + T(6.0) * p1 - T(8.0) * z;
  const T c3 = (m2 + p2) - T(4.0) * s1 + T(6.0) * z;
  r.d = c0 + x * (T(3.0) * c1 + x * (T(2.0) * x * c3 - T(6.0) * c2));
  r.z = z;
  return r;
}
// Whole cells between two feet that are not one apart (compensated, signed).
template <typename T, int ES>
__device__ __noinline__ T cells_between(int kl, int kr, const T *cells, int b0, int rows,
                                        unsigned *status) {
  const int lo = min(kl, kr), hi = max(kl, kr);
  if (lo < b0 || hi > b0 + rows) {
    atomicOr(status, STATUS_HALO);
    return T(0);
  }
  T s = T(0), comp = T(0);
  for (int k = lo; k < hi; ++k) {
    const T x = cells[(k - b0) * ES], t = s + x;
    comp += (fabs(s) >= fabs(x)) ? ((s - t) + x) : ((x - t) + s);
    s = t;
  }
  s += comp;
  return kr > kl ? s : -s;
}

// BND 0: periodic lines; 1: the reference's boundaries, derivative of the sweep
// input; 2: the reference's third sweep, which differentiates the remapped
// field.  Its interior right-hand side R_k + sum_t wq_t R_{k+n0-2+t} with R_j =
// sum_s wr_s C_{j+n0-2+s} is two tap groups of the cells, 8 taps from k+n0-3
// and 13 from k+2n0-5 with the mass matrix, in three windowed passes (8, 8, 5)
// that keep the register window at eight values for any displacement.  BND 3
// (x sweeps, periodic): the last x sweep of a step and the first of the next
// one in one pass.  Both solve the same circulant systems, so their operators
// commute: the two stencils compose into 15 taps from k+2n0-6 and the forward
// recurrence runs twice, then the backward one; the warm-up of such a double
// recurrence is a few cells longer.  2048^2: one pass of 21.3 us for two of
// 18.2 us (eight steps 317 -> 255 us).
//
// EXACT (BND 0 and 4; any diffusion number): no warm-up.  Every segment of a
// line runs both recurrences over its own cells from zero, which leaves it an
// affine map of its carries, w_end = q^np w_in + E and x_start = q^np x_in + X
// (q = -mu); the segments, one cluster, write E and X to each other and close
// the periodic line exactly.  Segments are whole walks and a shorter last one;
// a y line of 544 cells is one warp's and needs no exchange.  Bound by the
// clusters' latency: 64 registers for the y kernel too, so that the next
// launch's clusters find room beside this one's (1024^2, eight steps with every
// sweep closed: 264 us with 80 registers, 213 us with 64).  Eight steps at
// K dt / h^2 = 90 against the tile kernel: 256^2 175 -> 122 us, 1024^2 222 -> 212
// us, 2048^2 602 -> 556 us, 4096^2 2491 -> 2455 us; swirling field at 20, 1024^2
// 792 -> 405 us, 2048^2 2988 -> 1510 us.
template <typename T, int DIR, int LN, int BND, bool EXACT>
__global__ void __launch_bounds__(StreamCta<DIR, LN>::warps * 32,
                                  BND == 4 ? (DIR == 0 ? 2 : 4) : DIR == 0 ? 64 / LN : EXACT ? 8 : 6)
    stream_kernel(const __grid_constant__ PlanFields plan, const SweepField *__restrict__ fields,
                  int nfields, int first, const FieldIo io, int rows, unsigned *status,
                  int jstep, int nslice, const int *nlo, int cs, int clustered,
                  const int *g0idx, int ends, double toff) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NT = StreamCta<DIR, LN>::warps * 32;
  constexpr int LPW = StreamCta<DIR, LN>::lpw;
  constexpr int ES = DIR == 0 ? X_PITCH : 1;    // element stride of a position
  constexpr int LS = DIR == 0 ? LPW : 1;        // lane stride of a chunk
  constexpr unsigned FULL = 0xffffffffu;
  constexpr bool ENDS = BND == 1 || BND == 2;  // the reference's boundaries
  constexpr bool XX = BND == 3;
  constexpr bool SWIRL = BND == 4;
  T *tile_s = reinterpret_cast<T *>(smem_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  // field, tile and segment of this CTA.  A plan's fields differ only in their
  // buffers, a constant stride apart: their descriptor is a kernel argument and
  // the grid is (tile, segment, field), so nothing has to be fetched or divided
  // before the copies start.  Batched launches (one-dimensional) search for
  // their field.  The tiles of one segment come before the next segment, so
  // that the CTAs in flight cover whole rows of the field (x sweep of 4096^2:
  // 46.6 us against 48.3 us with a line's segments side by side).
  StreamField F;
  const SweepField *D;  // whole descriptor (line ends only)
  int tile, rank;
  const void *vs;
  void *vd;
  if (plan.tiles > 0) {
    F = stream_field(plan.f);
    // (the swirling field's times differ from slice to slice)
    D = SWIRL ? fields + (first + (int)blockIdx.z) : &plan.f;
    tile = blockIdx.x;
    rank = blockIdx.y;
    field_io(plan.f, jstep, io, &vs, &vd);
    const long long off = (first + (int)blockIdx.z) * plan.stride;
    vs = static_cast<const char *>(vs) + off;
    vd = static_cast<char *>(vd) + off;
  } else {
    const int cta = (int)blockIdx.x + first;
    const SweepField &f = fields[find_field(fields, g0idx, nfields, cta / cs)];
    F = stream_field(f);
    D = &f;
    if (SWIRL) toff = field_time(f, toff, jstep, nslice);
    const int q = cta - F.cta0;
    rank = clustered ? q % cs : q / F.groups;
    tile = clustered ? q / cs : q - rank * F.groups;
    field_io(f, jstep, io, &vs, &vd);
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (!field_active(f, jstep, nslice, nlo)) return;  // uniform over a cluster
  }
  // exact form: its constants, then the values that the cluster exchanges
  T *exs = tile_s + (size_t)(DIR == 0 ? X_PITCH : StreamCta<DIR, LN>::lines) * rows +
           (SWIRL ? 2 * (LN * SCH + 3) * (sizeof(double) / sizeof(T)) : 0);
  if (EXACT) {
    if (threadIdx.x < 6) exs[threadIdx.x] = T(D->ex[threadIdx.x]);
    __syncwarp();  // an aligned cluster barrier takes converged warps only
    // the peers may write to this CTA once it runs
    if (cs > 1) asm volatile("barrier.cluster.arrive.aligned;\n" ::: "memory");
  }
  const T *src = reinterpret_cast<const T *>(vs);
  T *dst = reinterpret_cast<T *>(vd);
  const int L = F.L, M = F.M, J = F.J, H = F.H;
  const long long s_line = F.s_line, s_pos = F.s_pos;
  const int Lc = plan.tiles > 0 ? plan.seg : EXACT ? exact_seg(L, cs, LN) : stream_seg(L, cs);
  const int p0 = min(L, rank * Lc), p1 = min(L, p0 + Lc), np = p1 - p0;
  const int line0 = tile * StreamCta<DIR, LN>::lines;        // first line of the CTA
  if (np <= 0 && !clustered) return;

  // ---- stage the cells (periodic wrap) ----
  // Positions p0-J .. p1+J-1 are walked by the first `act` lanes of a line, and
  // the cells of all positions of those lanes are staged: past p1+J they only
  // lengthen the backward warm-up, so nothing is masked inside a lane.
  // (The reference's lines end: nothing is walked past position L - 1.)
  const int walked = ENDS ? min(np + 2 * J, L - p0 + J) : np + 2 * J;
  const int act = min(LN, (walked + SCH - 1) / SCH);
  // first position of the first lane: p0 - J, or (the reference's lines) as much
  // earlier as makes the last lane end with the line, so that nothing is masked
  // there either (also where the line ends within the warm-up of a segment
  // before the last one)
  const int org = ENDS ? min(p0 - J, L - act * SCH) : p0 - J;
  const int nr = (act * SCH + 2 * (H - J) + (ENDS ? 2 : 1)) & ~1;
  // position of staged row 0, row of position p0 (both even with p0 and H)
  const int b0 = ENDS ? (org - (H - J)) & ~1 : p0 - H, h0 = ENDS ? p0 - b0 : H;
  const bool inside = b0 >= 0 && b0 + nr <= L;
  const bool pairs = ((DIR == 0 ? s_pos : s_line) & 1) == 0 && (DIR == 0 || (L & 1) == 0) &&
                     (((size_t)src | (size_t)dst) & (2 * sizeof(T) - 1)) == 0;
  // What depends on the plan alone comes before the wait, beside the launch
  // before this one: the line's shift, the feet of its ends, the swirl's tables.
  // Small grids are chains of dependent launches, bound by each one's latency:
  // one step of the reference's setting at 128^2 28.5 -> 20.6 us, ten at 600^2
  // 259 -> 226 us, its Parareal at 256^2 20.4 -> 19.1 ms, six swirl steps of
  // 1024^2 323 -> 311 us.  (Batched launches have waited: their tables may be
  // this launch's predecessor's work.)
  // this lane's line
  const int c = DIR == 0 ? lane / LPW : lane % LN;           // chunk
  const int lw = DIR == 0 ? lane % LPW : lane / LN;          // line within the warp
  const int line = line0 + warp * LPW + lw;
  const T mmu = T(-F.mu);
  const T *wt = reinterpret_cast<const T *>(F.wt) +  // padded past M
                (size_t)line *
                    (BND == 2 ? STREAM_TAPS_D : BND == 1 ? STREAM_TAPS_C : XX ? STREAM_TAPS_XX : 8);
  // whether positions next to the line's ends are walked here (both regions are
  // shorter than their scratch): other segments copy first and skip them (2048^2,
  // eight steps: 513 us with the feet before every segment's copies, 492 us so)
  const bool near = ENDS && (org < ends || org + act * SCH > L - ends);
  int n0 = 0;
  if (!SWIRL && (!ENDS || near)) n0 = __ldg(F.nt + line);
  // swirling field: sin and cos of the edges org-1 .. of the walked positions,
  // and the speeds of the line's two corner lines
  double2 *const sc_edge = reinterpret_cast<double2 *>(
      tile_s + (size_t)(DIR == 0 ? X_PITCH : StreamCta<DIR, LN>::lines) * rows);
  CornerLine c0{0, 0, 0}, c1{0, 0, 0};
  int series = 0;
  if (SWIRL) {
    for (int i = threadIdx.x; i < act * SCH + 3; i += NT) {
      const double s = D->s_min + D->h * (org - 1 + i);
      sc_edge[i] = double2{sinpi(s), cospi(s)};
    }
    const double ca = cospi((toff + D->ta_rel) / D->vp[0]);
    const double cb = cospi((toff + D->tb_rel) / D->vp[0]);
    const double sg = DIR == 0 ? 1.0 : -1.0, Dt = D->Dt;
    const double g0 = sg * sinpi(2.0 * (D->t_min + D->ht * (double)line));
    const double g1 = sg * sinpi(2.0 * (D->t_min + D->ht * (double)(line + 1)));
    const double pd = 3.14159265358979323846 * Dt;
    c0 = CornerLine{g0 * cb, g0 * ca, pd * (g0 * cb)};
    c1 = CornerLine{g1 * cb, g1 * ca, pd * (g1 * cb)};
    series = fabs(pd) <= 0.00390625 ? 2 : fabs(pd) <= 0.03125 ? 1 : 0;  // |speed| <= 1
  }
  // inputs of the positions next to the line's ends (BND): the left region is
  // r[k - lo.ka], k in [lo.ka, lo.kb), the right one likewise
  EndRegion lo{}, hi{};
  hi.ka = L;
  T *rl = nullptr, *rr = nullptr, *half = nullptr;
  int *kf = nullptr;
  if (near) {
    const int kend = org + act * SCH;  // first position not walked
    // positions whose stencil, with the mass matrix's neighbours, stays clear
    // of clamps and ghosts: [sl, sr)
    int bl = max(2 - n0, 0), bh = min(L - 4 - n0, L - 1);
    if (BND == 2) {
      bl = max(bl, 4 - 2 * n0);
      bh = min(bh, L - 7 - 2 * n0);
    }
    const int sl = min(bl + 1, L), sr = min(max(bh, sl), L);
    auto region = [&](int ka, int kb) {
      EndRegion e;
      e.ka = ka;
      e.kb = kb;
      e.ba = max(0, ka - 1);
      e.bb = min(L, kb + 1);
      e.ra = max(0, min(e.ba, e.ba + n0 - 4));
      e.rb = min(L, max(e.bb, e.bb + n0 + 5));
      if (e.ra < 3) e.ra = 0;  // with the cells its ghosts come from
      if (e.rb > L - 3) e.rb = L;
      return e;
    };
    lo = region(max(0, org), min(sl, kend));
    hi = region(max(sr, org), min(L, kend));
    if (line >= M) lo.kb = lo.ka, hi.kb = hi.ka;
    // scratch: per line and end 3 arrays of `ends` values and one of cells
    T *sc = tile_s + (size_t)(DIR == 0 ? X_PITCH : StreamCta<DIR, LN>::lines) * rows;
    kf = reinterpret_cast<int *>(sc + (size_t)StreamCta<DIR, LN>::lines * 6 * ends);
    const int li = warp * LPW + lw, side = c >= LN / 2;
    sc += (size_t)li * 6 * ends;
    kf += (size_t)(2 * li + side) * ends;
    rl = sc + ends;
    rr = sc + 4 * ends;
    half = sc + side * 3 * ends;
    const double x0 = __ldg(wt + (BND == 2 ? STREAM_TAPS_D : STREAM_TAPS_C) - 1);
    end_feet<T, BND == 2, LN / 2>(*D, line, n0, x0, side ? hi : lo, c % (LN / 2), half,
                                  half + ends, kf);
  }
  if (plan.tiles > 0) {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  }

  if (DIR == 0) {
    constexpr int G = X_LINES / 2;
    const int g = pairs ? 2 * ((int)threadIdx.x % G) : (int)threadIdx.x % X_LINES;
    const int r0 = pairs ? (int)threadIdx.x / G : (int)threadIdx.x / X_LINES;
    const int rs = pairs ? NT / G : NT / X_LINES;
    if (line0 + g < M) {
      const T *s = src + line0 + g;
      T *d = tile_s + r0 * X_PITCH + g;
      if (pairs && inside) {
        s += (long long)(b0 + r0) * s_pos;
        const long long step = (NT / G) * s_pos;
#pragma unroll 5
        for (int r = r0; r < nr; r += NT / G, s += step, d += NT / G * X_PITCH) copy_pair(d, s);
      } else {
        for (int r = r0; r < nr; r += rs, d += rs * X_PITCH) {
          if (ENDS && (unsigned)(b0 + r) >= (unsigned)L) {
            d[0] = T(0);
            if (pairs) d[1] = T(0);
            continue;
          }
          const T *p = s + (long long)(ENDS ? b0 + r : wrap_pos(b0 + r, L)) * s_pos;
          if (pairs) copy_pair(d, p); else copy_one(d, p);
        }
      }
    }
  } else {
#pragma unroll
    for (int l = 0; l < LPW; ++l) {
      const int gl = line0 + warp * LPW + l;
      if (gl < M) {
        const T *s = src + (long long)gl * s_line;
        T *d = tile_s + (size_t)(warp * LPW + l) * rows;
        if (pairs && inside) {
          s += b0;
#pragma unroll 5
          for (int e = 2 * lane; e < nr; e += 64) copy_pair(d + e, s + e);
        } else if (pairs) {
          for (int e = 2 * lane; e < nr; e += 64) {
            if (ENDS && (unsigned)(b0 + e) >= (unsigned)L)
              d[e] = d[e + 1] = T(0);
            else
              copy_pair(d + e, s + (ENDS ? b0 + e : wrap_pos(b0 + e, L)));
          }
        } else {
          for (int e = lane; e < nr; e += 32) {
            if (ENDS && (unsigned)(b0 + e) >= (unsigned)L)
              d[e] = T(0);
            else
              copy_one(d + e, s + (ENDS ? b0 + e : wrap_pos(b0 + e, L)));
          }
        }
      }
    }
  }
  cp_async_commit();
  if (ENDS && !near) n0 = __ldg(F.nt + line);
  // the stencil, while the cells arrive
  T o[8];
  if (!ENDS && !SWIRL) load_taps(o, wt);
  static_assert(SCH == 17, "pw");
  T pw = mmu * mmu;  // (-mu)^17
  pw *= pw;
  pw *= pw;
  pw *= pw * mmu;
  cp_async_wait_all_committed();
  if (DIR == 0 || SWIRL || EXACT) __syncthreads(); else __syncwarp();
  // In place, the segments of a line are read (halo) by the neighbouring CTAs
  // of its cluster: no CTA stores before every CTA has staged.
  if (clustered && !EXACT) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.aligned;\n" ::: "memory");
  }

  // ---- stencil and recurrences ----
  T *const col = DIR == 0 ? tile_s + warp * LPW + lw : tile_s + (size_t)(warp * LPW + lw) * rows;
  const int k0 = (ENDS ? org - b0 : H - J) + c * SCH;  // staged row of this lane's first position
  const int r0 = XX ? k0 + 2 * n0 - 6 : k0 + n0 - 3;  // row of the first tap
  bool ok = SWIRL || (r0 >= 0 && r0 + SCH + (XX ? 14 : 7) <= rows);
  if (BND == 2) ok = ok && k0 + 2 * n0 - 5 >= 0 && k0 + 2 * n0 + SCH + 8 <= rows;
  if (!ok && line < M) atomicOr(status, STATUS_HALO);
  if (near) {
    const StagedLine<T, ES> cells{col - b0 * ES, b0, b0 + nr, status};
    if (c == 0 && line < M) {  // ghost cells of the staged line
      T g1, g2;
      if (b0 <= -2) {
        ghosts(cells(0), cells(1), cells(2), g1, g2);
        col[(-1 - b0) * ES] = g1;
        col[(-2 - b0) * ES] = g2;
      }
      if (L + 2 - b0 <= nr && L - 3 >= b0) {
        ghosts(cells(L - 1), cells(L - 2), cells(L - 3), g1, g2);
        col[(L - b0) * ES] = g1;
        col[(L + 1 - b0) * ES] = g2;
      }
    }
    __syncwarp();
    end_inputs<T, ES, BND == 2, LN / 2>(*D, cells, line, n0, c < LN / 2 ? lo : hi, c % (LN / 2),
                                        half, half + ends, half + 2 * ends, kf);
  }
  // doubling steps that bring a carry in from every chunk of the warm-up (FP32:
  // one more, so that what is left out, |mu|^J of it at every chunk start, is
  // far below a rounding and not a share of one with the same sign everywhere)
  // (the reference's lines of one segment: no warm-up, any decay length).
  int ns = (F.JD <= SCH ? 0 : F.JD <= 2 * SCH ? 1 : F.JD <= 4 * SCH ? 2 : F.JD <= 8 * SCH ? 3 : 4) + (sizeof(T) == 4 ? 1 : 0);
  if (EXACT || (ENDS && F.JD > 4 * SCH)) ns = LN == 32 ? 5 : 4;
  T v[SCH];
  if (ENDS) load_taps(o, wt);
  if (SWIRL) {
    // b of the positions k0-1 .. k0+17 from the feet of their edges, then the
    // mass matrix: v_i = (1/12c)(b_{i-1} + 10 b_i + b_{i+1})
    if (c < act) {
      const int kp = org + c * SCH;
      const double s_min = D->s_min, h = D->h, Dt = D->Dt;
      const double hd = 3.0 * Dt * D->inv12h;  // Dt / (4 h)
      const T kbc = T(D->kb * D->inv12h), icw = T(D->sm_inv_den / 12.0);
      int bad = 0;
      T bl[SCH + 2];  // b, in a loop small enough for the instruction cache
      auto cells_b = [&](auto order) {
        constexpr int SERIES = decltype(order)::value;
        auto edge = [&](int i) {  // edge kp - 1 + i
          const double2 t = sc_edge[c * SCH + i];
          const double s = SERIES ? 0.0 : s_min + h * (kp - 1 + i);
          const double u = -hd * (corner_speeds<SERIES>(c0, t.x, t.y, s, Dt) +
                                  corner_speeds<SERIES>(c1, t.x, t.y, s, Dt));
          return swirl_edge<T, ES>(kp - 1 + i, u, col, b0, nr, bad);
        };
        SwirlEdge<T> l = edge(0);
#pragma unroll 2
        for (int i = 0; i < SCH + 2; ++i) {
          const SwirlEdge<T> r = edge(i + 1);
          T m = r.phi - l.phi;
          if (r.kf == l.kf + 1) m += l.z;
          else if (r.kf != l.kf) m += cells_between<T, ES>(l.kf, r.kf, col, b0, nr, status);
          bl[i] = m + kbc * (r.d - l.d);
          l = r;
        }
      };
      if (series == 2) cells_b(Series<2>());
      else if (series == 1) cells_b(Series<1>());
      else cells_b(Series<0>());
#pragma unroll
      for (int i = 0; i < SCH; ++i) v[i] = icw * ((bl[i] + bl[i + 2]) + T(10.0) * bl[i + 1]);
      if (bad && line < M) atomicOr(status, STATUS_HALO);
    } else {
#pragma unroll
      for (int i = 0; i < SCH; ++i) v[i] = T(0);
    }
  } else {
    stencil<T, ES, 8, false>(col + (ok ? r0 : 0) * ES, o, v);
  }
  if (XX) {
    load_taps(o, wt + 8);
    stencil<T, ES, 7, true>(col + (ok ? r0 + 8 : 0) * ES, o, v);
  }
  if (BND == 2) {
    load_taps(o, wt + 8);
    stencil<T, ES, 8, true>(col + (ok ? k0 + 2 * n0 - 5 : 0) * ES, o, v);
    load_taps(o, wt + 16);
    stencil<T, ES, 5, true>(col + (ok ? k0 + 2 * n0 + 3 : 0) * ES, o, v);
  }
  const int kp = org + c * SCH;  // this lane's first position
  if (ENDS) {
    // lanes next to the line's ends take the prepared inputs (zero before the
    // line) through their own rows: a loop over a few positions instead of 17
    // predicated selects
    __syncwarp();  // the cells of these rows have been read
    if (kp < lo.kb || kp < 0 || kp + SCH > hi.ka) {
      T *row = col + k0 * ES;
#pragma unroll
      for (int i = 0; i < SCH; ++i) row[i * ES] = v[i];
      for (int k = kp; k < min(kp + SCH, lo.kb); ++k)
        row[(k - kp) * ES] = k < 0 ? T(0) : rl[k - lo.ka];
      for (int k = max(kp, hi.ka); k < min(kp + SCH, hi.kb); ++k)
        row[(k - kp) * ES] = rr[k - hi.ka];
#pragma unroll
      for (int i = 0; i < SCH; ++i) v[i] = row[i * ES];
    }
  }
  // one recurrence over the line: the chunk from zero for its end value, the
  // carry into it by doubling steps over the lanes, the chunk again
  auto forward = [&] {
    T w = T(0);
#pragma unroll
    for (int i = 0; i < SCH; ++i) w = v[i] + mmu * w;
    T pd = pw;
    for (int s = 0; s < ns; ++s) {
      const T t = __shfl_up_sync(FULL, w, LS << s, DIR == 0 ? 32 : LN);
      if (c >= (1 << s)) w += pd * t;
      pd *= pd;
    }
    w = __shfl_up_sync(FULL, w, LS, DIR == 0 ? 32 : LN);
    if (c == 0) w = T(0);
#pragma unroll
    for (int i = 0; i < SCH; ++i) {
      w = v[i] + mmu * w;
      v[i] = w;
    }
  };
  // carry of the backward recurrence from the right of this chunk
  auto backward_carry = [&] {
    T x = T(0);
#pragma unroll
    for (int i = SCH - 1; i >= 0; --i) x = v[i] + mmu * x;
    if (c >= act) x = T(0);  // lanes whose cells are not staged
    T pd = pw;
    for (int s = 0; s < ns; ++s) {
      const T t = __shfl_down_sync(FULL, x, LS << s, DIR == 0 ? 32 : LN);
      if (c + (1 << s) < LN) x += pd * t;
      pd *= pd;
    }
    x = __shfl_down_sync(FULL, x, LS, DIR == 0 ? 32 : LN);
    return c == LN - 1 ? T(0) : x;
  };
  forward();
  if (XX) {
    forward();
    T x = backward_carry();
#pragma unroll
    for (int i = SCH - 1; i >= 0; --i) {
      x = v[i] + mmu * x;
      v[i] = x;
    }
  }
  T x, rise = T(0);  // rise (EXACT): the forward carry's share, before this lane's first position
  if (!EXACT) {
    x = backward_carry();
  } else {
    constexpr int W = DIR == 0 ? 32 : LN;      // shuffle width of a line
    const int l0 = DIR == 0 ? lane % LPW : 0;  // its first lane
    auto from = [&](T a, int ch) { return __shfl_sync(FULL, a, l0 + LS * ch, W); };
    const int mine = np - c * SCH;  // positions from this lane's first one on
    // E; nothing behind the segment for the backward recurrence
    T E = v[SCH - 1];
    if (np < LN * SCH) {
#pragma unroll
      for (int i = 0; i < SCH; ++i) {
        if (i == mine - 1) E = v[i];
        if (i >= mine) v[i] = T(0);
      }
    }
    x = T(0);
#pragma unroll
    for (int i = SCH - 1; i >= 0; --i) x = v[i] + mmu * x;
    // with the scan: q^(17 c), q^(17 (act-1-c))
    T pd = pw, up = T(1), down = T(1);
#pragma unroll
    for (int b = 0; b < (LN == 32 ? 5 : 4); ++b) {
      const T t = __shfl_down_sync(FULL, x, LS << b, W);
      if (c + (1 << b) < LN) x += pd * t;
      if (c >> b & 1) up *= pd;
      if ((act - 1 - c) >> b & 1) down *= pd;
      pd *= pd;
    }
    // The forward carry cr into a segment adds cr q^(j+1) to w_j (q = -mu),
    // which the backward recurrence turns into A q^(j+1) - A q^(np+1) q^(np-j),
    // A = cr / (1 - mu^2); the backward carry d from the right adds d q^(np-j).
    const T whole = exs[0], last = exs[1], inv1m = exs[2], inv_line = exs[3];
    T cr, d;  // this segment's carries
    if (cs == 1) {
      cr = from(E, act - 1) * inv_line;
      d = (from(x, 0) + cr * (mmu * (T(1) - last * last) * inv1m)) * inv_line;
    } else {
      // every CTA writes its E and X to all of its cluster
      T *ex = exs + 8 + 2 * MAX_CLUSTER * (warp * LPW + lw);
      E = from(E, act - 1);
      const T X = from(x, 0);
      __syncwarp();
      asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
      if (c < cs) {
        T *p = cg::this_cluster().map_shared_rank(ex, c) + 2 * rank;
        p[0] = E;
        p[1] = X;
      }
      __syncwarp();
      asm volatile("barrier.cluster.arrive.aligned;\n" ::: "memory");
      asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
      // lane r: segment r.  All but the last are Lc long, q^Lc = whole
      const T e = c < cs ? ex[2 * c] : T(0), xr = c < cs ? ex[2 * c + 1] : T(0);
      T S = e, pc = T(1), ps = whole;  // S: w at the end of segment r from a zero line start
      for (int b = 0; (1 << b) < cs; ++b) {
        const T t = __shfl_up_sync(FULL, S, LS << b, W);
        if (c >= (1 << b)) S += ps * t;
        if (c >> b & 1) pc *= ps;
        ps *= ps;
      }
      const T w0 = (last * from(S, cs - 2) + from(e, cs - 1)) * inv_line;
      S = __shfl_up_sync(FULL, S, LS, W);
      const T cr_c = pc * w0 + (c > 0 ? S : T(0));
      const T pr = c == cs - 1 ? last : whole;
      T R = c < cs ? xr + cr_c * (mmu * (T(1) - pr * pr) * inv1m) : T(0);
      ps = whole;
      for (int b = 0; (1 << b) < cs; ++b) {
        const T t = __shfl_down_sync(FULL, R, LS << b, W);
        if (c + (1 << b) < LN) R += ps * t;
        ps *= ps;
      }
      const T x0 = from(R, 0) * inv_line;  // x at the line's start
      cr = from(cr_c, rank);
      const T dn = from(R, min(rank + 1, cs - 1)) + from(pc, max(cs - 2 - rank, 0)) * last * x0;
      d = rank + 1 < cs ? dn : x0;
    }
    const bool end = rank + 1 == cs;
    rise = cr * inv1m * up;
    const T far = d - cr * inv1m * mmu * (end ? last : whole);
    x = __shfl_down_sync(FULL, x, LS, W);
    if (c == LN - 1) x = T(0);
    // Carry into this lane.  The last one, where it ends behind the segment,
    // starts with q^-(positions behind) as much.  Where that factor is large
    // (lines of a few cells and |q| far below one: q^-13 at 4 cells leaves FP32's
    // range) the carry enters right behind the segment's last position.
    const T back = end ? exs[5] : T(1);
    if (back != T(0)) {
      if (c < act) x += far * down * back;
    } else if (c < act - 1) {
      x += far * exs[4] * T(powi(-F.mu, SCH * (act - 2 - c)));
    } else {
#pragma unroll
      for (int i = 1; i < SCH; ++i)
        if (i == mine) v[i] = far;
    }
  }
  __syncwarp();  // every lane of the line has read its cells
  T *xp = col + k0 * ES;
#pragma unroll
  for (int i = SCH - 1; i >= 0; --i) {
    x = v[i] + mmu * x;
    if (ENDS || EXACT) v[i] = x;
    if (!EXACT) xp[i * ES] = x;
  }
  if (EXACT) {
#pragma unroll
    for (int i = 0; i < SCH; ++i) {
      rise *= mmu;
      xp[i * ES] = v[i] + rise;
    }
  }
  if (ENDS && p0 == 0) {
    // non-cyclic system: A = c (1 + mu S^-1)(1 + mu S) + c mu^2 e_0 e_0^T, so
    // x = y - y_0 g with g_k = mu^2 ((-mu)^k - (-mu)^(2L-k)) / (1 - mu^(2L+2))
    // (Sherman-Morrison); y_0 is this segment's value at position 0, and g has
    // decayed below rounding within the segment
    __syncwarp();
    const double q = -F.mu, a = (double)col[-b0 * ES] * D->rk_a;
    __syncwarp();
    if (kp < F.JD) {
      double g = -a * powi(q, max(kp, 0));
#pragma unroll
      for (int i = 0; i < SCH; ++i)
        if (kp + i >= 0) {
          v[i] += T(g);
          g *= q;
        }
      if (D->rk_tail) {
        g = a * powi(q, 2 * L - min(kp + SCH, L) + 1);
#pragma unroll
        for (int i = SCH - 1; i >= 0; --i)
          if (kp + i < L) {
            v[i] += T(g);
            g *= q;
          }
      }
#pragma unroll
      for (int i = 0; i < SCH; ++i) xp[i * ES] = v[i];
    }
  }
  if (DIR == 0) __syncthreads(); else __syncwarp();
  if (clustered && !EXACT) asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");

  // ---- store positions p0 .. p1-1 ----
  if (DIR == 0) {
    if (pairs) {
      constexpr int G = X_LINES / 2;
      const int g = 2 * ((int)threadIdx.x % G);
      if (line0 + g < M) {
        T *d = dst + (long long)p0 * s_pos + line0 + g;
        const T *s = tile_s + h0 * X_PITCH + g;
#pragma unroll 4
        for (int r = (int)threadIdx.x / G; r < np; r += NT / G)
          *reinterpret_cast<Pair<T> *>(d + (long long)r * s_pos) =
              *reinterpret_cast<const Pair<T> *>(s + r * X_PITCH);
      }
    } else {
      const int g = (int)threadIdx.x % X_LINES;
      if (line0 + g < M)
        for (int r = (int)threadIdx.x / X_LINES; r < np; r += NT / X_LINES)
          dst[(long long)(p0 + r) * s_pos + line0 + g] = tile_s[(r + h0) * X_PITCH + g];
    }
  } else {
#pragma unroll
    for (int l = 0; l < LPW; ++l) {
      const int gl = line0 + warp * LPW + l;
      if (gl < M) {
        T *d = dst + (long long)gl * s_line + p0;
        const T *s = tile_s + (size_t)(warp * LPW + l) * rows + h0;
        if (pairs)
          for (int e = 2 * lane; e < np; e += 64)
            *reinterpret_cast<Pair<T> *>(d + e) = *reinterpret_cast<const Pair<T> *>(s + e);
        else
          for (int e = lane; e < np; e += 32) d[e] = s[e];
      }
    }
  }
}

template <typename T>
using StreamKernelT = void (*)(const PlanFields, const SweepField *, int, int, const FieldIo, int,
                               unsigned *, int, int, const int *, int, int, const int *, int,
                               double);

template <typename T, int BND, bool EXACT = false>
StreamKernelT<T> stream_kernel_of(int dir, int lanes) {
  if constexpr (BND == 0 && !EXACT)
    if (dir == 0 && lanes == 32) return stream_kernel<T, 0, 32, 0, false>;
  if (dir == 0) return stream_kernel<T, 0, 16, BND, EXACT>;
  return lanes == 32 ? stream_kernel<T, 1, 32, BND, EXACT> : stream_kernel<T, 1, 16, BND, EXACT>;
}
template <typename T>
StreamKernelT<T> stream_kernel_for(int variant, int dir, int lanes) {
  if (variant == SWEEP_CELL) return stream_kernel_of<T, 4>(dir, lanes);
  if constexpr (sizeof(T) == 8)  // (fused_x_geom: FP64 only)
    if (variant == SWEEP_FILTER_XX)
      return lanes == 32 ? stream_kernel<T, 0, 32, 3, false> : stream_kernel<T, 0, 16, 3, false>;
  if (variant == SWEEP_FILTER_EXACT) return stream_kernel_of<T, 0, true>(dir, lanes);
  if (variant == SWEEP_CELL_EXACT) return stream_kernel_of<T, 4, true>(dir, lanes);
  return variant == SWEEP_COMPAT     ? stream_kernel_of<T, 1>(dir, lanes)
         : variant == SWEEP_COMPAT_D ? stream_kernel_of<T, 2>(dir, lanes)
                                     : stream_kernel_of<T, 0>(dir, lanes);
}

}  // namespace

int stream_tile_lines(int dir, int lanes) {
  return dir == 0 ? X_LINES : Y_WARPS * (32 / lanes);
}

size_t stream_smem_bytes(const LaunchGeom &G, bool fp64) {
  const size_t el = fp64 ? 8 : 4, lines = stream_tile_lines(G.dir, G.lanes);
  return (G.dir == 0 ? (size_t)X_PITCH : lines) * G.rows * el +
         lines * 2 * (size_t)G.ends * (3 * el + sizeof(int)) +
         (exact_filter_variant(G.variant) ? (8 + (G.cs > 1 ? lines * 2 * MAX_CLUSTER : 0)) * el : 0) +
         (G.variant == SWEEP_CELL || G.variant == SWEEP_CELL_EXACT ? sizeof(double2) * ((size_t)G.lanes * STREAM_CH + 3) : 0);
}

template <typename T>
cudaError_t launch_stream(const LaunchGeom &G, const PlanFields &plan, const SweepField *d_fields,
                          int nfields, int group_base, int groups_total, double toff, const FieldIo &io,
                          unsigned *d_status, int jstep, int nslice, const int *nlo,
                          bool inplace, cudaStream_t stream, const int *g0idx, bool pdl) {
  // Function attributes apply to the device that is current when they are
  // set: configure each device once (several host threads may launch).
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
  static std::atomic<bool> configured[MAX_DEVICES];
  static std::mutex config_mu;
  if (!configured[dev].load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> lk(config_mu);
    if (!configured[dev].load(std::memory_order_relaxed)) {
      for (int v : {SWEEP_FILTER, SWEEP_COMPAT, SWEEP_COMPAT_D, SWEEP_FILTER_XX, SWEEP_CELL,
                    SWEEP_FILTER_EXACT, SWEEP_CELL_EXACT})
        for (int i = 0; i < 4; ++i) {
          const void *fn = (const void *)stream_kernel_for<T>(v, i / 2, i % 2 ? 32 : 16);
          err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
          if (err != cudaSuccess) return err;
          err = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
          if (err != cudaSuccess) return err;
        }
      configured[dev].store(true, std::memory_order_release);
    }
  }
  if (groups_total <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  const bool by_value = plan.tiles > 0;
  cfg.gridDim = by_value ? dim3((unsigned)plan.tiles, (unsigned)G.cs,
                                (unsigned)(groups_total / plan.tiles))
                         : dim3((unsigned)(groups_total * G.cs), 1, 1);
  cfg.blockDim = dim3((unsigned)(G.dir == 0 ? X_LINES * G.lanes : Y_WARPS * 32), 1, 1);
  cfg.dynamicSmemBytes = stream_smem_bytes(G, sizeof(T) == 8);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned na = 0;
  // in place, or closed exactly, with several segments per line: they form one
  // cluster
  const int clustered = (inplace || exact_filter_variant(G.variant)) && G.cs > 1 ? 1 : 0;
  if (clustered) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = by_value ? 1 : (unsigned)G.cs;
    attr[na].val.clusterDim.y = by_value ? (unsigned)G.cs : 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  count_launch();
  return cudaLaunchKernelEx(&cfg, stream_kernel_for<T>(G.variant, G.dir, G.lanes), plan, d_fields, nfields,
                            by_value ? group_base / plan.tiles : group_base * G.cs, io, G.rows,
                            d_status, jstep, nslice, nlo, G.cs, clustered, g0idx, G.ends, toff);
}

template cudaError_t launch_stream<double>(const LaunchGeom &, const PlanFields &,
                                           const SweepField *, int, int, int, double, const FieldIo &, unsigned *,
                                           int, int, const int *, bool, cudaStream_t, const int *,
                                           bool);
template cudaError_t launch_stream<float>(const LaunchGeom &, const PlanFields &,
                                          const SweepField *, int, int, int, double, const FieldIo &, unsigned *,
                                          int, int, const int *, bool, cudaStream_t, const int *,
                                          bool);

}  // namespace ccfv
