// sweep.cu -- the fused T2S4 CC-CFV sweep for sm_100a.
//
// One launch performs one directional sub-step (an x(dt/2) or y(dt) sweep of
// GpuOneStep, T2S4_Parareal.cu:824-963) for any number of fields.  Per line
// of cells it fuses what the reference spreads over ~11 kernels and ~40
// N^2-sized global arrays:
//   characteristic feet of the cell edges     (T2S4:203-258)
//   PPM reconstruction + conservative remap   (T2S4:260-438)
//   4th-order derivative at the edge feet     (T2S4:440-547)
//   Crank-Nicolson RHS + compact mass matrix  (T2S4:550-654)
//   tridiagonal solve                         (T2S4:657-719)
// Each cell is read once from HBM and written once.
//
// Work decomposition.  A tile is LPG = 16 neighbouring lines.  A cluster of
// cs CTAs covers the whole length of the tile's lines, each CTA a run of up
// to LC_MAX consecutive positions plus a halo on both sides (loaded from
// global memory; in place is safe because every store happens after a
// cluster-wide barrier that follows all loads).  The shared tile is
// [position][line] with an odd pitch: for x-sweeps global rows of 16
// doubles (128 B) land in shared rows; for y-sweeps each line is a
// contiguous global run written down a shared column.
//
// Thread mapping: lane % 16 = line, each thread owns a chunk of consecutive
// positions of its line.  The constant-coefficient tridiagonal system is
// solved as two first-order linear recurrences (LU forward / backward) with
// line-invariant factors alpha_k, g_k precomputed per (L, dt, K): every
// chunk runs its recurrence locally from a zero carry, the chunk maps
// (prod alpha, local value) are composed across the CTA (shared memory) and
// across the cluster (distributed shared memory), and a fix-up pass adds the
// carried-in value times the running product.  The periodic (cyclic) system
// adds a Sherman-Morrison rank-one correction with a line-invariant vector.
#include <cooperative_groups.h>

#include <atomic>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "ccfv_internal.h"
#include "sweep_device.cuh"
#include "sweep_math.cuh"

namespace cg = cooperative_groups;

namespace ccfv {

namespace {

// Bounds-checked view of one line in the shared tile, indexed by position.
template <typename T>
struct LineView {
  const T *cs;
  int base;   // row of position 0 = H - p0
  int nrows;
  unsigned *status;
  __device__ __forceinline__ T operator()(int pos) const {
    int row = pos + base;
    if (row < 0 || row >= nrows) {
      atomicOr(status, STATUS_HALO);
      return T(0);
    }
    return cs[row * PITCH];
  }
};

template <typename T>
struct Ppm {
  T CL, D, C6;
};

// PPM coefficients of cell i (x_step_ppm_coef_on_gpu, T2S4:260-304); ghost
// cells are already in the tile (compat) or it holds wrapped cells (periodic).
template <typename T>
__device__ __forceinline__ Ppm<T> ppm(const LineView<T> &v, int i) {
  const T one_twelfth = T(1.0 / 12.0), seven_twelfths = T(7.0 / 12.0);
  T cm2 = v(i - 2), cm1 = v(i - 1), c0 = v(i), cp1 = v(i + 1), cp2 = v(i + 2);
  T cl = seven_twelfths * (c0 + cm1) - one_twelfth * (cp1 + cm2);
  T cr = seven_twelfths * (cp1 + c0) - one_twelfth * (cp2 + cm1);
  Ppm<T> p;
  p.CL = cl;
  p.D = cr - cl;
  p.C6 = T(6.0) * (c0 - T(0.5) * (cl + cr));
  return p;
}

// PPM antiderivative in cell units (d_intC_ppm4th, T2S4:63-65).
template <typename T>
__device__ __forceinline__ T ppm_int(const Ppm<T> &p, T xi) {
  T xi2 = xi * xi;
  return T(-1.0 / 3) * p.C6 * (xi2 * xi) + T(0.5) * (p.D + p.C6) * xi2 + p.CL * xi;
}

// Neumaier-compensated sum of cells lo..hi.
template <typename T>
__device__ __forceinline__ T sum_cells(const LineView<T> &v, int lo, int hi) {
  T s = T(0), comp = T(0);
  for (int k = lo; k <= hi; ++k) {
    T x = v(k);
    T t = s + x;
    comp += (fabs(s) >= fabs(x)) ? ((s - t) + x) : ((x - t) + s);
    s = t;
  }
  return s + comp;
}

// Conservative remap of one cell over its departure interval [fL, fR].
// compat: x_step_intC_ppm_on_gpu / y_step_intC_ppm_on_gpu (T2S4:306-438):
// zero inflow from outside the domain, feet clamped by eps_remap.  The
// reference's y-remap reads the next row's first cell when its right foot
// is clamped onto the top edge (jR == Ny, an O(2^-53 * Ny) contribution);
// here that term is zero.
template <typename T>
__device__ __forceinline__ T remap_cell(const SweepField &f, const LineView<T> &v, double fL,
                                        double fR) {
  const int L = f.L;
  if (f.bc == BC_COMPAT) {
    if (fL > f.s_max || fR < f.s_min || fL == fR) return T(0);
    double xL = fmax(fL, f.s_min + f.eps_remap);
    double xR = fmin(fR, f.s_max - f.eps_remap);
    int iL = (int)floor((xL - f.s_min) / f.h);
    int iR = (int)floor((xR - f.s_min) / f.h);
    T xiL = (T)((xL - (f.s_min + f.h * iL)) / f.h);
    T xiR = (T)((xR - (f.s_min + f.h * iR)) / f.h);
    Ppm<T> z{T(0), T(0), T(0)};
    Ppm<T> pL = (iL >= 0 && iL < L) ? ppm(v, iL) : z;
    if (iR == iL) return ppm_int(pL, xiR) - ppm_int(pL, xiL);
    Ppm<T> pR = (iR >= 0 && iR < L) ? ppm(v, iR) : z;
    T IntCL = ppm_int(pL, T(1)) - ppm_int(pL, xiL);
    T IntCR = ppm_int(pR, xiR);
    T IntCM = T(0);
    int hi = iR - 1 < L - 1 ? iR - 1 : L - 1;
    for (int k = iL + 1; k <= hi; ++k) IntCM += v(k);
    return IntCL + IntCM + IntCR;
  } else {
    double uL = (fL - f.s_min) / f.h, uR = (fR - f.s_min) / f.h;
    double fkL = floor(uL), fkR = floor(uR);
    int kL = (int)fkL, kR = (int)fkR;
    T xiL = (T)(uL - fkL), xiR = (T)(uR - fkR);
    Ppm<T> pL = ppm(v, kL);
    if (kR == kL) return ppm_int(pL, xiR) - ppm_int(pL, xiL);
    if (abs(kR - kL) > v.nrows) {  // cannot happen within the staged halo
      atomicOr(v.status, STATUS_HALO);
      return T(0);
    }
    Ppm<T> pR = ppm(v, kR);
    if (kR > kL) return sum_cells(v, kL, kR - 1) + ppm_int(pR, xiR) - ppm_int(pL, xiL);
    return -(sum_cells(v, kR, kL - 1) + ppm_int(pL, xiL) - ppm_int(pR, xiR));
  }
}

// Fourth-order derivative at a foot (dcdx_bar_on_gpu / dcdy_bar_on_gpu,
// T2S4:440-547).  compat keeps the reference's ghost selection at iL = L-2
// (+2 tap reads C_{N+1}) and iL = 1 (-2 tap reads C_{-2}).
template <typename T>
__device__ __forceinline__ T foot_derivative(const SweepField &f, const LineView<T> &v, double fb) {
  const int L = f.L;
  int iL, pm2, pp2;
  T xi;
  if (f.bc == BC_COMPAT) {
    if (!(fb >= f.s_min && fb <= f.s_max)) return T(0);
    double ixb = fmin(fmax(fb, f.s_min + 1e-15), f.s_max - 1e-15);
    iL = (int)floor((ixb - f.s_min) / f.h);
    xi = (T)((ixb - (f.s_min + f.h * iL)) / f.h);
    pm2 = (iL == 1) ? -2 : iL - 2;
    pp2 = (iL == L - 2) ? L + 1 : iL + 2;
  } else {
    double u = (fb - f.s_min) / f.h, fk = floor(u);
    iL = (int)fk;
    xi = (T)(u - fk);
    pm2 = iL - 2;
    pp2 = iL + 2;
  }
  T Cim2 = v(pm2), Cim1 = v(iL - 1), Ci = v(iL), Cip1 = v(iL + 1), Cip2 = v(pp2);
  T xi2 = xi * xi, xi3 = xi2 * xi;
  return T(f.inv12h) * ((T(2.0) * xi3 - T(6.0) * xi2 + T(3.0) * xi + T(1.0)) * Cim2 +
                        (T(-8.0) * xi3 + T(18.0) * xi2 + T(6.0) * xi - T(15.0)) * Cim1 +
                        (T(12.0) * xi3 - T(18.0) * xi2 - T(24.0) * xi + T(15.0)) * Ci +
                        (T(-8.0) * xi3 + T(6.0) * xi2 + T(18.0) * xi - T(1.0)) * Cip1 +
                        (T(2.0) * xi3 - T(3.0) * xi) * Cip2);
}

// Compat ghost cells C_{-2}, C_{-1}, C_N, C_{N+1} of one line of a tile
// (3-point extrapolation, T2S4:275-286), written where the tile's rows
// [lo, hi) cover them.  base = row of position 0.
template <typename T>
__device__ __forceinline__ void compat_ghosts(T *c, int base, int lo, int hi, int L) {
  const T one_eleventh = T(1.0 / 11.0);
  if (lo <= -2 && hi > 2) {
    T c0 = c[(base + 0) * PITCH], c1 = c[(base + 1) * PITCH], c2 = c[(base + 2) * PITCH];
    c[(base - 1) * PITCH] = one_eleventh * (-c2 + T(3) * c1 + T(9) * c0);
    c[(base - 2) * PITCH] = one_eleventh * (T(-15) * c2 + T(56) * c1 - T(30) * c0);
  }
  if (hi >= L + 2 && lo <= L - 3) {
    T a = c[(base + L - 3) * PITCH], b = c[(base + L - 2) * PITCH], d = c[(base + L - 1) * PITCH];
    c[(base + L) * PITCH] = one_eleventh * (-a + T(3) * b + T(9) * d);
    c[(base + L + 1) * PITCH] = one_eleventh * (T(-15) * a + T(56) * b - T(30) * d);
  }
}

// Source f(x, y, t) (the reference's f is identically zero, T2S4:58-61;
// Gaussian: sp0 exp(-((x-sp1)^2 + (y-sp2)^2) / sp3) cos(sp4 t)).
__device__ __forceinline__ double src_f(const SweepField &f, double x, double y, double t) {
  const double dx = x - f.sp[1], dy = y - f.sp[2];
  return f.sp[0] * exp(-(dx * dx + dy * dy) / f.sp[3]) * cos(f.sp[4] * t);
}

// 3x3 Simpson cell average of f over cell `pos` of line `gl` at time t
// (get_source_term_on_gpu, T2S4:142-165).
__device__ double src_cell(const SweepField &f, int pos, long long gl, double t) {
  const double s = f.s_min + (pos + 0.5) * f.h, tau = f.t_min + (gl + 0.5) * f.ht;
  const double x_i = f.dir == 0 ? s : tau, y_j = f.dir == 0 ? tau : s;
  const double dx = f.dir == 0 ? f.h : f.ht, dy = f.dir == 0 ? f.ht : f.h;
  const double xm = x_i - 0.5 * dx, xp = x_i + 0.5 * dx, ym = y_j - 0.5 * dy, yp = y_j + 0.5 * dy;
  return 1.0 / 36.0 *
         (src_f(f, xm, ym, t) + src_f(f, xp, ym, t) + src_f(f, xm, yp, t) + src_f(f, xp, yp, t) +
          4.0 * (src_f(f, xm, y_j, t) + src_f(f, xp, y_j, t) + src_f(f, x_i, ym, t) +
                 src_f(f, x_i, yp, t)) +
          16.0 * src_f(f, x_i, y_j, t));
}

// Uniform displacement: every edge foot of a line sits at e - sigma
// (position units), -sigma = n0 + xi0 from the foot f0 of edge 0.  Remap,
// foot derivative and RHS then reduce to fixed 6-tap stencils whose weights
// depend on xi0 only:
//   remap_k = sum_t w_t C_{k+n0+t},  kb (D_{k+1}-D_k) = sum_t q_t C_{k+n0+t}
// (t = -2..3; q includes (1-theta) K Dt/h and 1/(12h)), the same PPM integral
// and cubic derivative weights as the per-cell formulas (T2S4:63-65,
// 440-547), so the stencil and per-cell paths agree to rounding.
template <typename T>
__device__ __forceinline__ void uniform_weights(const SweepField &F, double f0, T w[6], T qd[6],
                                                int *n0) {
  const double u = (f0 - F.s_min) / F.h;
  const double fl = floor(u);
  *n0 = (int)fl;
  const double x = u - fl, x2 = x * x, x3 = x2 * x;
  const double A = x - 2.0 * x2 + x3, B = x3 - x2, Cc = 3.0 * x2 - 2.0 * x3;
  w[0] = T(A / 12.0);
  w[1] = T((B - 8.0 * A) / 12.0);
  w[2] = T(1.0 - Cc - 2.0 * B / 3.0);
  w[3] = T(Cc + 2.0 * A / 3.0);
  w[4] = T((8.0 * B - A) / 12.0);
  w[5] = T(-B / 12.0);
  const double pm2 = 2.0 * x3 - 6.0 * x2 + 3.0 * x + 1.0;
  const double pm1 = -8.0 * x3 + 18.0 * x2 + 6.0 * x - 15.0;
  const double pz = 12.0 * x3 - 18.0 * x2 - 24.0 * x + 15.0;
  const double pp1 = -8.0 * x3 + 6.0 * x2 + 18.0 * x - 1.0;
  const double pp2 = 2.0 * x3 - 3.0 * x;
  const double kq = F.kb * F.inv12h;
  qd[0] = T(kq * -pm2);
  qd[1] = T(kq * (pm2 - pm1));
  qd[2] = T(kq * (pm1 - pz));
  qd[3] = T(kq * (pz - pp1));
  qd[4] = T(kq * (pp1 - pp2));
  qd[5] = T(kq * pp2);
}

// Shared-memory carve-up of the sweep kernel.
template <typename T>
struct Smem {
  T *C;      // [(lc_max + 2H) * PITCH]  tile 0: the input cells
  T *B;      // [(lc_max + 2H) * PITCH]  tile 1
  // Both tiles are indexed by row = position - p0 + H.  Derivative of the
  // input: b -> tile 1, q/x -> tile 0.  Derivative of the remapped field:
  // remap -> tile 1, b -> tile 0, q/x -> tile 1.
  T *tA;     // [lc_max]  alpha_k
  T *tG;     // [lc_max]  g_k
  T *tZ;     // [lc_max]  z_k (periodic)
  T *aggA;   // [NCH * LPG] chunk products
  T *aggF;   // [NCH * LPG] chunk forward values
  T *aggR;   // [NCH * LPG] chunk backward values
  T *xch;    // [8 * LPG] cluster exchange: fwdA fwdB bwdA bwdB y0 yL
  T *Fs;     // [(lc_max + 2H) * PITCH] source cell averages at t_a (source variant only)
  SweepField *fd;
};

template <typename T>
__device__ __forceinline__ Smem<T> carve(unsigned char *raw, int lc_max, int H) {
  Smem<T> s;
  s.fd = reinterpret_cast<SweepField *>(raw);
  T *p = reinterpret_cast<T *>(raw + FD_BYTES);
  s.C = p;
  p += (lc_max + 2 * H) * PITCH;
  s.B = p;
  p += (lc_max + 2 * H) * PITCH;
  s.tA = p;
  p += lc_max;
  s.tG = p;
  p += lc_max;
  s.tZ = p;
  p += lc_max;
  s.aggA = p;
  p += NCH * LPG;
  s.aggF = p;
  p += NCH * LPG;
  s.aggR = p;
  p += NCH * LPG;
  s.xch = p;
  p += 8 * LPG;
  s.Fs = p;
  return s;
}

template <typename T>
__global__ void __launch_bounds__(NTH, 2) sweep_kernel(const SweepField *__restrict__ fields,
                                                    int nfields, int group_base, double toff,
                                                    const FieldIo io, int lc_max, int H,
                                                    unsigned *status, int jstep, int nslice,
                                                    const int *nlo, const int *g0idx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int tile = blockIdx.x / cs + group_base;
  Smem<T> S = carve<T>(smem_raw, lc_max, H);

  // ---- descriptor of this tile's field (binary search on group0) ----
  if (threadIdx.x == 0) {
    *S.fd = fields[find_field(fields, g0idx, nfields, tile)];
  }
  __syncthreads();
  const SweepField &F = *S.fd;
  if (!field_active(F, jstep, nslice, nlo)) return;  // uniform over the cluster
  toff = field_time(F, toff, jstep, nslice);
  const int L = F.L;
  const int g = tile - F.group0;
  const long long line0 = (long long)g * LPG;
  const int Lc = (L + cs - 1) / cs;
  const int p0 = min(L, rank * Lc);
  const int p1 = min(L, p0 + Lc);
  const int np = p1 - p0;
  const int nrows = np + 2 * H;
  const bool periodic = F.bc == BC_PERIODIC;
  const T *gsrc;
  T *gdst;
  {
    const void *vs;
    void *vd;
    field_io(F, jstep, io, &vs, &vd);
    gsrc = reinterpret_cast<const T *>(vs);
    gdst = reinterpret_cast<T *>(vd);
  }

  // ---- phase 0: stage the tile (+halo) and the solver factors ----
  {
    const int total = nrows * LPG;
    const bool xs = (F.s_line == 1);
    for (int e = threadIdx.x; e < total; e += NTH) {
      int row, ln;
      if (xs) { row = e / LPG; ln = e - row * LPG; }
      else { ln = e / nrows; row = e - ln * nrows; }
      int pos = p0 - H + row;
      long long gl = line0 + ln;
      T val = T(0);
      if (gl < F.M) {
        bool ok = true;
        if (pos < 0 || pos >= L) {
          if (periodic) { pos %= L; if (pos < 0) pos += L; }
          else ok = false;
        }
        if (ok) val = gsrc[(long long)pos * F.s_pos + gl * F.s_line];
      }
      S.C[row * PITCH + ln] = val;
    }
    const T *tab = reinterpret_cast<const T *>(F.tab);
    for (int k = threadIdx.x; k < np; k += NTH) {
      S.tA[k] = tab[p0 + k];
      S.tG[k] = tab[L + p0 + k];
      S.tZ[k] = periodic ? tab[2 * L + p0 + k] : T(0);
    }
  }
  __syncthreads();
  if (!periodic && threadIdx.x < LPG) compat_ghosts(S.C + threadIdx.x, H - p0, p0 - H, p1 + H, L);
  // source: f(t_a) (f(t_b) in the third sub-step) on the staged rows, remapped
  // like C (T2S4:846-853, 893-900, 944-951); f(t_b) enters unremapped
  const double t_src0 = toff + (F.src_tb ? F.tb_rel : F.ta_rel);
  const double t_src1 = toff + F.tb_rel;
  if (F.src) {
    for (int e = threadIdx.x; e < nrows * LPG; e += NTH) {
      const int row = e / LPG, l = e - row * LPG;
      int pos = p0 - H + row;
      T val = T(0);
      if (periodic) {
        pos %= L;
        if (pos < 0) pos += L;
        val = T(src_cell(F, pos, line0 + l, t_src0));
      } else if (pos >= 0 && pos < L) {
        val = T(src_cell(F, pos, line0 + l, t_src0));
      }
      S.Fs[row * PITCH + l] = val;
    }
    __syncthreads();
    if (!periodic && threadIdx.x < LPG) compat_ghosts(S.Fs + threadIdx.x, H - p0, p0 - H, p1 + H, L);
  }
  __syncthreads();

  // ---- thread -> (line, chunk) ----
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ln = lane % LPG;
  const int c = warp * CPW + lane / LPG;
  const long long gl = line0 + ln;
  const int m = (np + NCH - 1) / NCH;
  const int s = min(p1, p0 + c * m);
  const int e = min(p1, s + m);
  const int clast = (np - 1) / m;  // last non-empty chunk
  LineView<T> v{S.C + ln, H - p0, nrows, status};

  // ---- phase 1: feet, remap, foot derivative, RHS b ----
  // b_k = remap_k + w (remap(f)_k + f_k) + 0.5 K Dt/h (D_{k+1} - D_k)
  // (x_b_RHS_on_gpu / y_b_RHS_on_gpu, T2S4:564-613); w = src_w, 0 without a
  // source (the reference's f is identically zero, T2S4:58-61).
  T *bArr, *qArr;
  {
    const LineView<T> vf{S.Fs + ln, H - p0, nrows, status};  // read only when F.src
    const T srcw = T(F.src_w);
    auto src_term = [&](int k, double fa, double fb) -> T {
      int kk = k;
      if (periodic) { kk %= L; if (kk < 0) kk += L; }
      return srcw * (remap_cell(F, vf, fa, fb) + T(src_cell(F, kk, line0 + ln, t_src1)));
    };
    // the shared-foot stencils cover C only; with a source every cell takes
    // the per-cell path
    const bool stencil = F.uniform && !F.src;
    int kb = s, ke = e;
    if (c == 0 && (periodic || p0 > 0)) kb = p0 - 1;
    if (c == clast && (periodic || p1 < L)) ke = p1 + 1;
    const double tau0 = F.t_min + F.ht * (double)gl;
    const double tau1 = F.t_min + F.ht * (double)(gl + 1);
    const double ta = toff + F.ta_rel, tb = toff + F.tb_rel;
    const LineFeet lf(F, tau0, tau1, ta, tb);
    const T kbc = T(F.kb);
    // uniform displacement: shared-foot stencils (uniform_weights)
    int n0 = 0, klo = 1, khi = 0;
    T w[6], qd[6];
    if (stencil) {
      uniform_weights<T>(F, lf.foot(F, 0), w, qd, &n0);
      if (periodic) { klo = INT_MIN; khi = INT_MAX; }
      else { klo = 2 - n0; khi = L - 4 - n0; }  // clear of clamps and ghost quirks
    }
    if (F.dsrc == 0) {
      bArr = S.B;
      qArr = S.C;
      if (stencil) {
        for (int k = kb; k < ke; ++k) {
          T bk;
          if (k >= klo && k <= khi) {
            const int r = k + n0 + H - p0 - 2;
            const T *cp = S.C + r * PITCH + ln;
            if (r < 0 || r + 5 >= nrows) { atomicOr(status, STATUS_HALO); bk = T(0); }
            else {
              bk = T(0);
#pragma unroll
              for (int t = 0; t < 6; ++t) bk += (w[t] + qd[t]) * cp[t * PITCH];
            }
          } else {
            double fa = lf.foot(F, k);
            double fb = lf.foot(F, k + 1);
            bk = remap_cell(F, v, fa, fb) + kbc * (foot_derivative(F, v, fb) - foot_derivative(F, v, fa));
          }
          bArr[(k - p0 + H) * PITCH + ln] = bk;
        }
      } else if (kb < ke) {
        double fprev = lf.foot(F, kb);
        T dprev = foot_derivative(F, v, fprev);
        for (int k = kb; k < ke; ++k) {
          double fnext = lf.foot(F, k + 1);
          T dnext = foot_derivative(F, v, fnext);
          T ic = remap_cell(F, v, fprev, fnext);
          T bk = ic + kbc * (dnext - dprev);
          if (F.src) bk += src_term(k, fprev, fnext);
          bArr[(k - p0 + H) * PITCH + ln] = bk;
          fprev = fnext;
          dprev = dnext;
        }
      }
    } else {
      // The reference's third sweep differentiates the remapped field
      // (dcdx_bar_on_gpu(v_d_Cnphf_bar_x, ...), T2S4:929-932): remap the
      // cells p0-hd .. p1+hd-1 into tile 1 first, then differentiate it.
      T *R = S.B;
      int q0 = p0 - F.hd, q1 = p1 + F.hd;
      if (!periodic) { q0 = max(q0, 0); q1 = min(q1, L); }
      const int m1 = (q1 - q0 + NCH - 1) / NCH;
      const int r0 = q0 + c * m1, r1 = min(q1, r0 + m1);
      for (int k = r0; k < r1; ++k) {
        T ik;
        if (stencil && k >= klo && k <= khi) {
          const int r = k + n0 + H - p0 - 2;
          const T *cp = S.C + r * PITCH + ln;
          if (r < 0 || r + 5 >= nrows) { atomicOr(status, STATUS_HALO); ik = T(0); }
          else {
            ik = T(0);
#pragma unroll
            for (int t = 0; t < 6; ++t) ik += w[t] * cp[t * PITCH];
          }
        } else {
          double fa = lf.foot(F, k);
          double fb = lf.foot(F, k + 1);
          ik = remap_cell(F, v, fa, fb);
        }
        R[(k - p0 + H) * PITCH + ln] = ik;
      }
      __syncthreads();
      if (!periodic && threadIdx.x < LPG) compat_ghosts(R + threadIdx.x, H - p0, q0 - 2, q1 + 2, L);
      __syncthreads();
      LineView<T> vr{R + ln, H - p0, nrows, status};
      bArr = S.C;
      qArr = S.B;
      for (int k = kb; k < ke; ++k) {
        T bk;
        if (stencil && k >= klo && k <= khi) {
          const int r = k + n0 + H - p0 - 2;
          const T *rp = R + r * PITCH + ln;
          if (r < 0 || r + 5 >= nrows) { atomicOr(status, STATUS_HALO); bk = T(0); }
          else {
            T acc = T(0);
#pragma unroll
            for (int t = 0; t < 6; ++t) acc += qd[t] * rp[t * PITCH];
            bk = vr(k) + acc;
          }
        } else {
          double fa = lf.foot(F, k);
          double fb = lf.foot(F, k + 1);
          bk = vr(k) + kbc * (foot_derivative(F, vr, fb) - foot_derivative(F, vr, fa));
          if (F.src) bk += src_term(k, fa, fb);
        }
        bArr[(k - p0 + H) * PITCH + ln] = bk;
      }
    }
  }
  __syncthreads();

  // ---- phase 2: compact mass matrix + local forward recurrence ----
  T *Cl = qArr + ln;
  const int rb = H - p0;  // row of position 0 in both tiles
  {
    T A = T(1), q = T(0);
    if (s < e) {
      const T *Bl = bArr + ln;
      T bm = Bl[(s - 1 + rb) * PITCH], bc = Bl[(s + rb) * PITCH];
      for (int k = s; k < e; ++k) {
        T bp = Bl[(k + 1 + rb) * PITCH];
        T mb;
        if (!periodic && k == 0) mb = (T(10.0) * bc + bp) / T(12.0);
        else if (!periodic && k == L - 1) mb = (T(10.0) * bc + bm) / T(12.0);
        else mb = (bp + T(10.0) * bc + bm) / T(12.0);
        const T a = S.tA[k - p0];
        q = S.tG[k - p0] * mb + a * q;
        A *= a;
        Cl[(k + rb) * PITCH] = q;
        bm = bc;
        bc = bp;
      }
    }
    S.aggA[c * LPG + ln] = A;
    S.aggF[c * LPG + ln] = q;
  }
  __syncthreads();

  // ---- phase 3: forward carries (CTA prefix, then cluster prefix) ----
  {
    T PA = T(1), PB = T(0);  // composite of chunks 0..c-1
    for (int j = 0; j < c; ++j) {
      T a = S.aggA[j * LPG + ln], b = S.aggF[j * LPG + ln];
      PB = a * PB + b;
      PA = a * PA;
    }
    T cin = T(0);
    if (cs > 1) {
      T *xA = S.xch, *xB = S.xch + LPG;
      if (c == NCH - 1) {
        T a = S.aggA[c * LPG + ln], b = S.aggF[c * LPG + ln];
        xA[ln] = a * PA;
        xB[ln] = a * PB + b;
      }
      cluster.sync();
      for (int r = 0; r < rank; ++r) {
        const T *ra = cluster.map_shared_rank(xA, r);
        const T *rbv = cluster.map_shared_rank(xB, r);
        cin = ra[ln] * cin + rbv[ln];
      }
    }
    const T carry = PA * cin + PB;
    T P = T(1);
    for (int k = s; k < e; ++k) {
      P *= S.tA[k - p0];
      Cl[(k + rb) * PITCH] += P * carry;
    }
    // ---- phase 4: local backward recurrence ----
    T x = T(0);
    for (int k = e - 1; k >= s; --k) {
      x = Cl[(k + rb) * PITCH] + S.tA[k - p0] * x;
      Cl[(k + rb) * PITCH] = x;
    }
    S.aggR[c * LPG + ln] = x;
  }
  __syncthreads();

  // ---- phase 5: backward carries (CTA suffix, then cluster suffix) ----
  {
    T SA = T(1), SB = T(0);  // composite of chunks NCH-1 .. c+1
    for (int j = NCH - 1; j > c; --j) {
      T a = S.aggA[j * LPG + ln], b = S.aggR[j * LPG + ln];
      SB = b + a * SB;
      SA = a * SA;
    }
    T cin = T(0);
    if (cs > 1) {
      T *xA = S.xch + 2 * LPG, *xB = S.xch + 3 * LPG;
      if (c == 0) {
        T a = S.aggA[ln], b = S.aggR[ln];
        xA[ln] = a * SA;
        xB[ln] = b + a * SB;
      }
      cluster.sync();
      for (int r = cs - 1; r > rank; --r) {
        const T *ra = cluster.map_shared_rank(xA, r);
        const T *rbv = cluster.map_shared_rank(xB, r);
        cin = rbv[ln] + ra[ln] * cin;
      }
    }
    const T carry = SB + SA * cin;
    T P = T(1);
    for (int k = e - 1; k >= s; --k) {
      P *= S.tA[k - p0];
      Cl[(k + rb) * PITCH] += P * carry;
    }
  }

  // ---- phase 6: periodic rank-one (Sherman-Morrison) correction ----
  if (periodic) {
    T *y0 = S.xch + 4 * LPG, *yL = S.xch + 5 * LPG;
    __syncthreads();
    if (rank == 0 && threadIdx.x < LPG) y0[threadIdx.x] = qArr[(H)*PITCH + threadIdx.x];
    if (rank == cs - 1 && threadIdx.x < LPG) yL[threadIdx.x] = qArr[(H + np - 1) * PITCH + threadIdx.x];
    T a0, aL;
    if (cs > 1) {
      cluster.sync();
      a0 = cluster.map_shared_rank(y0, 0)[ln];
      aL = cluster.map_shared_rank(yL, cs - 1)[ln];
    } else {
      __syncthreads();
      a0 = y0[ln];
      aL = yL[ln];
    }
    const T fct = (a0 + T(F.sm_fac) * aL) * T(F.sm_inv_den);
    for (int k = s; k < e; ++k) Cl[(k + rb) * PITCH] -= fct * S.tZ[k - p0];
  }
  __syncthreads();

  // ---- phase 7: store ----
  {
    const int total = np * LPG;
    const bool xs = (F.s_line == 1);
    for (int q = threadIdx.x; q < total; q += NTH) {
      int row, l2;
      if (xs) { row = q / LPG; l2 = q - row * LPG; }
      else { l2 = q / np; row = q - l2 * np; }
      long long gl2 = line0 + l2;
      if (gl2 < F.M)
        gdst[(long long)(p0 + row) * F.s_pos + gl2 * F.s_line] = qArr[(row + H) * PITCH + l2];
    }
  }
  if (cs > 1) cluster.sync();  // keep shared memory alive for remote readers
}


// ---------------------------------------------------------------------------
// Fast path: uniform displacement + periodic cells, derivative of the input.
// Every cell of a line uses the same 6-tap RHS stencil, so phase 1 and the
// forward recurrence fuse into one walk with a sliding register window (one
// shared-memory read per cell).  The chunk prefix / suffix products of
// alpha_k are line-invariant and kept once per chunk, which lets the forward
// fix-up and the backward recurrence fuse into a single reverse walk, and the
// backward fix-up, the Sherman-Morrison correction and the store into a final
// walk.

template <typename T>
struct FastSmem {
  T *C;      // [(lc_max + 2H) * PITCH]
  T *Q;      // [lc_max * PITCH]   q, then x (row = position - p0)
  T *tA, *tG, *tZ, *tP, *tS;  // [lc_max] factors and chunk prefix/suffix products
  T *aggA;   // [NCH]        chunk products (line-invariant)
  T *PA;     // [NCH + 1]    CTA-local exclusive prefix products of the chunks
  T *aggF;   // [NCH * LPG]  chunk forward values
  T *aggR;   // [NCH * LPG]  chunk backward values
  T *om;     // [6 * LPG]    per-line stencil weights
  T *cin;    // [2 * LPG]    per-line carries from the other CTAs of the cluster
  T *xch;    // [8 * LPG]    cluster exchange
  int *n0;   // [LPG]        per-line foot offset
  SweepField *fd;
};

template <typename T>
__device__ __forceinline__ FastSmem<T> carve_fast(unsigned char *raw, int lc_max, int H) {
  FastSmem<T> s;
  s.fd = reinterpret_cast<SweepField *>(raw);
  s.n0 = reinterpret_cast<int *>(raw + FD_BYTES);
  T *p = reinterpret_cast<T *>(raw + FD_BYTES + 64 * sizeof(int));
  s.C = p; p += (lc_max + 2 * H) * PITCH;
  s.Q = p; p += lc_max * PITCH;
  s.tA = p; p += lc_max;
  s.tG = p; p += lc_max;
  s.tZ = p; p += lc_max;
  s.tP = p; p += lc_max;
  s.tS = p; p += lc_max;
  s.aggA = p; p += NCH;
  s.PA = p; p += NCH + 1;
  s.aggF = p; p += NCH * LPG;
  s.aggR = p; p += NCH * LPG;
  s.om = p; p += 6 * LPG;
  s.cin = p; p += 2 * LPG;
  s.xch = p;
  return s;
}

template <typename T>
__global__ void __launch_bounds__(NTH, 2)
    sweep_fast_kernel(const SweepField *__restrict__ fields, int nfields, int group_base,
                      double toff, const FieldIo io, int lc_max, int H, unsigned *status,
                      int jstep, int nslice, const int *nlo, const int *g0idx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int tile = blockIdx.x / cs + group_base;
  FastSmem<T> S = carve_fast<T>(smem_raw, lc_max, H);
  {
    // every thread finds the field; the descriptor is copied cooperatively
    const int lo = find_field(fields, g0idx, nfields, tile);
    constexpr int NW8 = (int)(FD_COPY / 8);
    if (threadIdx.x < NW8)
      reinterpret_cast<long long *>(S.fd)[threadIdx.x] =
          __ldg(reinterpret_cast<const long long *>(&fields[lo]) + threadIdx.x);
  }
  __syncthreads();
  const SweepField &F = *S.fd;
  if (!field_active(F, jstep, nslice, nlo)) return;  // uniform over the cluster
  toff = field_time(F, toff, jstep, nslice);
  const int L = F.L;
  const long long line0 = (long long)(tile - F.group0) * LPG;
  const int Lc = (L + cs - 1) / cs;
  const int p0 = min(L, rank * Lc);
  const int p1 = min(L, p0 + Lc);
  const int np = p1 - p0;
  const int nrows = np + 2 * H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  const T *gsrc;
  T *gdst;
  {
    const void *vs;
    void *vd;
    field_io(F, jstep, io, &vs, &vd);
    gsrc = reinterpret_cast<const T *>(vs);
    gdst = reinterpret_cast<T *>(vd);
  }
  // ---- stage the tile (cp.async, no integer division) ----
  {
    const T *gdata = gsrc;
    if (F.s_line == 1) {
      // x-sweep: a warp copies two rows of 16 consecutive doubles per step
      const int ln = lane & (LPG - 1);
      const long long gl = line0 + ln;
      const bool okl = gl < F.M;
      for (int row = warp * 2 + (lane >> 4); row < nrows; row += 2 * NW) {
        int pos = p0 - H + row;
        if (pos < 0 || pos >= L) { pos %= L; if (pos < 0) pos += L; }
        T *dst = S.C + row * PITCH + ln;
        if (okl) {
          const T *src = gdata + (long long)pos * F.s_pos + gl;
          if (sizeof(T) == 8) cp_async8(dst, src); else cp_async4(dst, src);
        } else {
          *dst = T(0);
        }
      }
    } else {
      // y-sweep: a warp copies 32 consecutive cells of one line per step
      for (int ln = warp; ln < LPG; ln += NW) {
        const long long gl = line0 + ln;
        const bool okl = gl < F.M;
        const T *lbase = gdata + gl * F.s_line;
        for (int row = lane; row < nrows; row += 32) {
          int pos = p0 - H + row;
          if (pos < 0 || pos >= L) { pos %= L; if (pos < 0) pos += L; }
          T *dst = S.C + row * PITCH + ln;
          if (okl) {
            if (sizeof(T) == 8) cp_async8(dst, lbase + pos); else cp_async4(dst, lbase + pos);
          } else {
            *dst = T(0);
          }
        }
      }
    }
    cp_async_commit();
    // solver factors and chunk products of this CTA's positions
    const T *tab = reinterpret_cast<const T *>(F.tab);
    for (int k = threadIdx.x; k < np; k += NTH) {
      S.tA[k] = tab[p0 + k];
      S.tG[k] = tab[L + p0 + k];
      S.tZ[k] = tab[2 * L + p0 + k];
      S.tP[k] = tab[3 * L + p0 + k];
      S.tS[k] = tab[4 * L + p0 + k];
    }
    if (threadIdx.x < NCH) S.aggA[threadIdx.x] = tab[5 * L + rank * NCH + threadIdx.x];
    if (threadIdx.x <= NCH)
      S.PA[threadIdx.x] = tab[5 * L + cs * NCH + rank * (NCH + 1) + threadIdx.x];
    // per-line stencil: b_k = sum_t om_t C_{k+n0+t}, t = -2..3 (see sweep_kernel)
    if (threadIdx.x < LPG) {
      const int l = threadIdx.x;
      const long long gl = line0 + l;
      const double tau0 = F.t_min + F.ht * (double)gl;
      const double tau1 = F.t_min + F.ht * (double)(gl + 1);
      const double f0 = edge_foot(F, 0, tau0, tau1, toff + F.ta_rel, toff + F.tb_rel);
      const double u = (f0 - F.s_min) / F.h;
      const double fl = floor(u);
      S.n0[l] = (int)fl;
      const double x = u - fl, x2 = x * x, x3 = x2 * x;
      const double A = x - 2.0 * x2 + x3, B = x3 - x2, Cc = 3.0 * x2 - 2.0 * x3;
      const double kq = F.kb * F.inv12h;
      const double pm2 = 2.0 * x3 - 6.0 * x2 + 3.0 * x + 1.0;
      const double pm1 = -8.0 * x3 + 18.0 * x2 + 6.0 * x - 15.0;
      const double pz = 12.0 * x3 - 18.0 * x2 - 24.0 * x + 15.0;
      const double pp1 = -8.0 * x3 + 6.0 * x2 + 18.0 * x - 1.0;
      const double pp2 = 2.0 * x3 - 3.0 * x;
      T *om = S.om + 6 * l;
      om[0] = T(A / 12.0 - kq * pm2);
      om[1] = T((B - 8.0 * A) / 12.0 + kq * (pm2 - pm1));
      om[2] = T(1.0 - Cc - 2.0 * B / 3.0 + kq * (pm1 - pz));
      om[3] = T(Cc + 2.0 * A / 3.0 + kq * (pz - pp1));
      om[4] = T((8.0 * B - A) / 12.0 + kq * (pp1 - pp2));
      om[5] = T(-B / 12.0 + kq * pp2);
    }
    cp_async_wait_all_committed();
  }
  __syncthreads();

  const int ln = lane % LPG;
  const int c = warp * CPW + lane / LPG;
  const long long gl = line0 + ln;
  const int m = (np + NCH - 1) / NCH;
  const int s = min(p1, p0 + c * m);
  const int e = min(p1, s + m);

  // ---- fused RHS + compact mass matrix + local forward recurrence ----
  {
    T q = T(0);
    if (s < e) {
      const int n0 = S.n0[ln];
      const int r0 = (s - 1) + n0 - 2 - p0 + H;   // row of tap -2 of cell s-1
      const int rlast = e + n0 + 3 - p0 + H;       // row of tap +3 of cell e
      if (r0 < 0 || rlast >= nrows) {
        atomicOr(status, STATUS_HALO);
      } else {
        const T *omp = S.om + 6 * ln;
        const T o0 = omp[0], o1 = omp[1], o2 = omp[2], o3 = omp[3], o4 = omp[4], o5 = omp[5];
        const T *cp = S.C + r0 * PITCH + ln;
        T w0 = cp[0], w1 = cp[PITCH], w2 = cp[2 * PITCH], w3 = cp[3 * PITCH],
          w4 = cp[4 * PITCH], w5 = cp[5 * PITCH];
        T bm = o0 * w0 + o1 * w1 + o2 * w2 + o3 * w3 + o4 * w4 + o5 * w5;
        w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5; w5 = cp[6 * PITCH];
        T bc = o0 * w0 + o1 * w1 + o2 * w2 + o3 * w3 + o4 * w4 + o5 * w5;
        const T *nxt = cp + 7 * PITCH;
        T *qp = S.Q + (s - p0) * PITCH + ln;
        const T *ta = S.tA + (s - p0), *tg = S.tG + (s - p0);
        const int n = e - s;
#pragma unroll 4
        for (int i = 0; i < n; ++i) {
          w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5; w5 = nxt[i * PITCH];
          const T bp = o0 * w0 + o1 * w1 + o2 * w2 + o3 * w3 + o4 * w4 + o5 * w5;
          const T mb = (bp + T(10.0) * bc + bm) * T(1.0 / 12.0);
          q = tg[i] * mb + ta[i] * q;
          qp[i * PITCH] = q;
          bm = bc;
          bc = bp;
        }
      }
    }
    S.aggF[c * LPG + ln] = q;
  }
  __syncthreads();

  // ---- forward carries: CTA prefix (this line) + cluster prefix ----
  T carry;
  {
    T PB = T(0);
    for (int j = 0; j < c; ++j) PB = S.aggA[j] * PB + S.aggF[j * LPG + ln];
    if (cs > 1) {
      T *xB = S.xch + LPG;
      if (c == NCH - 1) xB[ln] = S.aggA[c] * PB + S.aggF[c * LPG + ln];
      cluster.sync();
      if (threadIdx.x < LPG) {  // compose the preceding CTAs once per line
        const T *tab = reinterpret_cast<const T *>(F.tab);
        const T *PAg = tab + 5 * L + cs * NCH;
        T cin = T(0);
        for (int r = 0; r < rank; ++r) {
          const T *rb = cluster.map_shared_rank(xB, r);
          cin = PAg[r * (NCH + 1) + NCH] * cin + rb[threadIdx.x];
        }
        S.cin[threadIdx.x] = cin;
      }
      __syncthreads();
      carry = S.PA[c] * S.cin[ln] + PB;
    } else {
      carry = PB;
    }
  }
  // ---- fused forward fix-up + local backward recurrence (reverse walk) ----
  {
    T x = T(0);
    const int n = e - s;
    T *qp = S.Q + (s - p0) * PITCH + ln;
    const T *ta = S.tA + (s - p0), *tp = S.tP + (s - p0);
#pragma unroll 4
    for (int i = n - 1; i >= 0; --i) {
      x = (qp[i * PITCH] + tp[i] * carry) + ta[i] * x;
      qp[i * PITCH] = x;
    }
    S.aggR[c * LPG + ln] = x;
  }
  __syncthreads();
  // ---- backward carries: CTA suffix + cluster suffix ----
  T carry2;
  {
    T SB = T(0), SA = T(1);
    for (int j = NCH - 1; j > c; --j) {
      const T a = S.aggA[j];
      SB = S.aggR[j * LPG + ln] + a * SB;
      SA = a * SA;
    }
    if (cs > 1) {
      T *xB = S.xch + 3 * LPG;
      if (c == 0) xB[ln] = S.aggR[ln] + S.aggA[0] * SB;
      cluster.sync();
      if (threadIdx.x < LPG) {
        const T *tab = reinterpret_cast<const T *>(F.tab);
        const T *PAg = tab + 5 * L + cs * NCH;
        T cin = T(0);
        for (int r = cs - 1; r > rank; --r) {
          const T *rb = cluster.map_shared_rank(xB, r);
          cin = rb[threadIdx.x] + PAg[r * (NCH + 1) + NCH] * cin;
        }
        S.cin[LPG + threadIdx.x] = cin;
      }
      __syncthreads();
      carry2 = SB + SA * S.cin[LPG + ln];
    } else {
      carry2 = SB;
    }
  }
  // ---- cyclic correction (Sherman-Morrison): needs y_0 and y_{L-1} ----
  T fct;
  {
    T *y0 = S.xch + 4 * LPG, *yL = S.xch + 5 * LPG;
    if (p0 == 0 && s == p0 && s < e) y0[ln] = S.Q[ln] + S.tS[0] * carry2;
    if (p1 == L && e == p1 && s < e) yL[ln] = S.Q[(np - 1) * PITCH + ln] + S.tS[np - 1] * carry2;
    if (cs > 1) {
      cluster.sync();
      if (threadIdx.x < LPG) {
        S.cin[threadIdx.x] = cluster.map_shared_rank(y0, 0)[threadIdx.x];
        S.cin[LPG + threadIdx.x] = cluster.map_shared_rank(yL, cs - 1)[threadIdx.x];
      }
      __syncthreads();
      fct = (S.cin[ln] + T(F.sm_fac) * S.cin[LPG + ln]) * T(F.sm_inv_den);
    } else {
      __syncthreads();
      fct = (y0[ln] + T(F.sm_fac) * yL[ln]) * T(F.sm_inv_den);
    }
  }
  // ---- backward fix-up + correction + store ----
  T *gdata = gdst;
  {
    const int n = e - s;
    T *qp = S.Q + (s - p0) * PITCH + ln;
    const T *ts = S.tS + (s - p0), *tz = S.tZ + (s - p0);
    if (F.s_line == 1) {
      // x-sweep: a half-warp writes 16 consecutive doubles of one row
      if (gl < F.M) {
        T *gp = gdata + (long long)s * F.s_pos + gl;
#pragma unroll 4
        for (int i = 0; i < n; ++i) gp[i * F.s_pos] = qp[i * PITCH] + ts[i] * carry2 - fct * tz[i];
      }
    } else {
#pragma unroll 4
      for (int i = 0; i < n; ++i) qp[i * PITCH] = qp[i * PITCH] + ts[i] * carry2 - fct * tz[i];
      __syncthreads();
      for (int l2 = warp; l2 < LPG; l2 += NW) {
        const long long gl2 = line0 + l2;
        if (gl2 >= F.M) continue;
        T *lbase = gdata + gl2 * F.s_line + p0;
        for (int row = lane; row < np; row += 32) lbase[row] = S.Q[row * PITCH + l2];
      }
    }
  }
  if (cs > 1) cluster.sync();  // keep shared memory alive for remote readers
}

// ---------------------------------------------------------------------------
// Filter path, tile form: the reference's boundaries where the streaming
// kernels (stream.cu) do not apply, i.e. feet that differ from edge to edge
// (swirling deformation) and lines whose ends need more scratch than fits.
//
// The constant system a x_{k-1} + b x_k + a x_{k+1} = r_k factors as
// c (1 + mu S^-1)(1 + mu S) x = r with |mu| < 1, mu / (1 + mu^2) = a / b,
// c = a / mu (plus a rank-one term at the line's start), so it is solved by two
// first-order recurrences,
//   w_k = r_k / c - mu w_{k-1},   x_k = w_k - mu x_{k+1}.
// A recurrence started from zero J positions early agrees with the exact one
// to |mu|^J, and J is chosen on the host so that |mu|^J is below the rounding
// of T.
//
// A CTA owns a segment [p0, p1) of 16 lines.  The 16 lanes of a half-warp
// own one line: lane c holds FCH consecutive positions in registers.  The
// forward recurrence runs over [p0 - J, p1 + J) (zero start J cells early),
// the backward one over [p0, p1 + J) (zero start at its end); inside a line
// the chunks are joined exactly by a 4-step shuffle scan of the chunk maps
// x -> (-mu)^FCH x + e, so only the segment ends are warmed up.  Every phase
// of a line stays inside its half-warp: the only CTA barriers are after the
// staging and before the cooperative store.

constexpr int FCH = 17;  // positions per lane (odd: conflict-free shared-memory columns)
constexpr int FLANES = 16;
// Longest segment for a recurrence warm-up J: 16 * FCH >= np + 2J.
__host__ __device__ constexpr int filter_seg_max(int J) { return FLANES * FCH - 2 * J; }

// Rows of the staged tile: enough for the longest chunk walk, so the solve
// loops need no bounds predicates (rows past the staged ones are only read
// by lanes whose positions lie past the range; their values are masked).
__host__ __device__ inline int filter_tile_rows(int lc_max, int H) {
  return (lc_max > FLANES * FCH ? lc_max : FLANES * FCH) + 2 * H + 8;
}

// The tile of a step is bounded with the room of a power table and of its edges.
constexpr int FPW = FLANES * FCH + 8;
template <typename T>
struct FiltSmem {
  T *C;      // [filter_tile_rows * PITCH]  input cells, then w, then x
  T *B;      // [filter_tile_rows * PITCH]  b of every position
  T *pwt;    // [32]       (-mu)^(i+1), i = 0 .. FCH-1
  SweepField *fd;
  int rows;
};

template <typename T>
__device__ __forceinline__ FiltSmem<T> carve_filt(unsigned char *raw, int lc_max, int H) {
  FiltSmem<T> s;
  s.fd = reinterpret_cast<SweepField *>(raw);
  s.pwt = reinterpret_cast<T *>(raw + FD_BYTES);
  s.C = s.pwt + 32;
  s.rows = filter_tile_rows(lc_max, H);
  s.B = s.C + (size_t)s.rows * PITCH;
  return s;
}

// Compat boundaries (the reference's): an edge whose foot lies inside
// [s_min + eps, s_max - eps] is "normal" (its remap clamps are no-ops); cells
// next to an edge that is not, or whose feet cross, take the reference's
// per-cell remap with its clamps and zero inflow (remap_cell, T2S4:306-438).
// The foot derivative keeps the reference's ghost selection (foot_derivative).
template <typename T>
struct CompatEdge {
  double f;
  int kf;
  bool normal;
  T phi, d;
};

template <typename T>
__device__ __forceinline__ CompatEdge<T> compat_edge(const SweepField &F, const LineFeet &lf,
                                                     const LineView<T> &vc,
                                                     const LineView<T> &vd, int e) {
  CompatEdge<T> r;
  r.f = lf.foot(F, e);
  r.normal = r.f >= F.s_min + F.eps_remap && r.f <= F.s_max - F.eps_remap;
  r.kf = 0;
  r.phi = T(0);
  if (r.normal) {
    const double u = (r.f - F.s_min) / F.h;
    const double fk = floor(u);
    r.kf = (int)fk;
    r.phi = ppm_int(ppm(vc, r.kf), T(u - fk));
  }
  r.d = foot_derivative(F, vd, r.f);
  return r;
}

template <typename T>
__device__ __forceinline__ T compat_remap(const SweepField &F, const CompatEdge<T> &l,
                                          const CompatEdge<T> &r, const LineView<T> &vc) {
  if (l.normal && r.normal && r.kf >= l.kf && l.f != r.f) {
    T s = T(0);
    for (int k = l.kf; k < r.kf; ++k) s += vc(k);
    return (s + r.phi) - l.phi;
  }
  return remap_cell(F, vc, l.f, r.f);
}

// The per-line stencil table of one field (one thread per line): eight taps
// from C_{k+n0-3}.  SWEEP_COMPAT_D (the reference scheme's third sweep, uniform
// displacement): b_k = R_k + sum_t wq_t R_{k+n0-2+t} with R_j = sum_s wr_s
// C_{j+n0-2+s} (the interior formulas of the line) is two groups of taps, with
// the mass matrix 8 from C_{k+n0-3} and 13 from C_{k+2n0-5}.  SWEEP_FILTER_XX:
// the eight taps twice, 15 from C_{k+2n0-6}.
template <typename T>
__global__ void filter_weights_kernel(const SweepField *__restrict__ f, T *__restrict__ wt,
                                      int *__restrict__ nt, int lines, int variant) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= lines) return;
  const SweepField F = *f;
  if (variant == SWEEP_COMPAT_D) {
    double om[STREAM_TAPS_D];
    for (int m = 0; m < STREAM_TAPS_D; ++m) om[m] = 0.0;
    int n0 = 0;
    if (l < F.M) {
      const double tau0 = F.t_min + F.ht * (double)l;
      const double f0 = edge_foot(F, 0, tau0, tau0 + F.ht, F.ta_rel, F.tb_rel);
      double wr[6], wq[6], wd[11];
      uniform_weights<double>(F, f0, wr, wq, &n0);
      for (int j = 0; j < 11; ++j) wd[j] = 0.0;
      for (int t = 0; t < 6; ++t)
        for (int s = 0; s < 6; ++s) wd[t + s] += wq[t] * wr[s];
      // mass matrix (1/12c)(b_{k-1} + 10 b_k + b_{k+1}) of n taps at w
      const double icw = F.sm_inv_den / 12.0;
      auto mass = [&](const double *w, int n, double *out) {
        for (int m = 0; m < n + 2; ++m)
          out[m] = icw * ((m < n ? w[m] : 0.0) + 10.0 * (m >= 1 && m <= n ? w[m - 1] : 0.0) +
                          (m >= 2 ? w[m - 2] : 0.0));
      };
      mass(wr, 6, om);
      mass(wd, 11, om + 8);
      om[STREAM_TAPS_D - 1] = (f0 - F.s_min) / F.h - n0;
    }
    for (int m = 0; m < STREAM_TAPS_D; ++m) wt[(size_t)l * STREAM_TAPS_D + m] = T(om[m]);
    nt[l] = n0;
    return;
  }
  if (variant == SWEEP_FILTER_XX) {
    double o[8], om[STREAM_TAPS_XX];
    int n0 = 0;
    for (int m = 0; m < 8; ++m) o[m] = 0.0;
    if (l < F.M) filter_line_stencil<double>(F, l, 0.0, o, &n0);
    for (int m = 0; m < STREAM_TAPS_XX; ++m) om[m] = 0.0;
    for (int m = 0; m < 8; ++m)
      for (int t = 0; t < 8; ++t) om[m + t] += o[m] * o[t];
    if (l < F.M) {
      // gain of a constant field: the taps sum to (1 + mu)^4, each product
      // rounded off by its own; the difference goes to an outer tap, in
      // two-term arithmetic (eight steps of 1024^2 at K dt / h^2 = 20: mean of
      // the field off by 2.5e-14 as rounded, 1.1e-14 so)
      double hi = 0.0, lo = 0.0;  // sum
      for (int m = 0; m < STREAM_TAPS_XX; ++m) {
        const double t = hi + om[m], z = t - hi;
        lo += (hi - (t - z)) + (om[m] - z);
        hi = t;
      }
      const double g = 1.0 + F.sm_fac, ge = F.sm_fac - (g - 1.0);
      const double g2 = g * g, e2 = __fma_rn(g, g, -g2) + 2.0 * g * ge;
      const double g4 = g2 * g2, e4 = __fma_rn(g2, g2, -g4) + 2.0 * g2 * e2;
      om[0] += (g4 - hi) + (e4 - lo);
    }
    for (int m = 0; m < STREAM_TAPS_XX; ++m) wt[(size_t)l * STREAM_TAPS_XX + m] = T(om[m]);
    nt[l] = n0;
    return;
  }
  const int nw = variant == SWEEP_COMPAT ? STREAM_TAPS_C : 8;
  T *row = wt + (size_t)l * nw;
  if (l < F.M) {
    T om[8];
    int n0 = 0;
    filter_line_stencil<T>(F, l, 0.0, om, &n0);
    for (int m = 0; m < 8; ++m) row[m] = om[m];
    nt[l] = n0;
    if (nw > 8) {
      const double tau0 = F.t_min + F.ht * (double)l;
      row[nw - 1] = T((edge_foot(F, 0, tau0, tau0 + F.ht, 0.0, 0.0) - F.s_min) / F.h - n0);
    }
  } else {
    for (int m = 0; m < nw; ++m) row[m] = T(0);
    nt[l] = 0;
  }
}

// The staged cells first give every position's b (the reference's per-cell
// remap with its clamps, foot derivatives with its ghost selection) in a second
// tile, each line's half-warp filling its own column; the forward filter then
// takes w's input as the mass-matrix stencil (1/12c)(b_{k-1} + 10 b_k +
// b_{k+1}).  Bound by the per-edge arithmetic; two tiles: two CTAs per SM.
template <typename T>
__global__ void __launch_bounds__(NTH, 2)
    sweep_filter_kernel(const SweepField *__restrict__ fields, int nfields, int group_base,
                        double toff, const FieldIo io, int lc_max, int H, unsigned *status,
                        int jstep, int nslice, const int *nlo, int cs, int clustered,
                        const int *g0idx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // Programmatic dependent launch: nothing is read before the previous grid
  // of the stream has completed (a no-op when launched without the
  // attribute), and the next grid may be scheduled onto the SMs this grid's
  // CTAs free.
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  // CTA -> (field, tile of LPG lines, segment).  The launch's clusters are the
  // cs segments of one tile; fields carry their first CTA and halo, so fields
  // of different segment lengths share one launch (lc_max and H size the
  // shared memory only)
  const int cta = (int)blockIdx.x + group_base;
  FiltSmem<T> S = carve_filt<T>(smem_raw, lc_max, H);
  {
    // a field's CTAs start at cta0 = group0 * cs (cs is uniform over a launch);
    // only the threads that copy the descriptor search for it
    constexpr int NW8 = (int)(FD_COPY / 8);
    if (threadIdx.x < NW8) {
      const int lo = find_field(fields, g0idx, nfields, cta / cs);
      reinterpret_cast<long long *>(S.fd)[threadIdx.x] =
          __ldg(reinterpret_cast<const long long *>(&fields[lo]) + threadIdx.x);
    }
  }
  __syncthreads();
  const SweepField &F = *S.fd;
  if (!field_active(F, jstep, nslice, nlo)) return;
  toff = field_time(F, toff, jstep, nslice);
  const int L = F.L;
  H = F.halo_f;
  const int q = cta - F.cta0;
  const int rank = q % cs;
  const long long line0 = (long long)(q / cs) * LPG;
  const int Lc = (L + cs - 1) / cs;
  const int p0 = min(L, rank * Lc);
  const int p1 = min(L, p0 + Lc);
  const int np = p1 - p0;
  const int nrows = np + 2 * H;
  const int J = F.jf;
  const T mu = T(F.sm_fac);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T *gsrc;
  T *gdst;
  {
    const void *vs;
    void *vd;
    field_io(F, jstep, io, &vs, &vd);
    gsrc = reinterpret_cast<const T *>(vs);
    gdst = reinterpret_cast<T *>(vd);
  }

  // Descriptor fields used in the loops live in registers: the descriptor is
  // in shared memory, and the copies' memory clobbers and the generic-pointer
  // stores would otherwise make the compiler reload it every iteration.
  const long long s_pos = F.s_pos, s_line = F.s_line, M = F.M;
  const bool xsweep = s_line == 1;
  // ---- stage rows p0-H .. p1+H-1 (zero outside the line) ----
  {
    const int rlo = max(0, H - p0), rhi = min(nrows, H - p0 + L);
    if (xsweep) {
      // a warp copies two rows of 16 consecutive values (128 B for FP64) per step
      const int ln = lane & (LPG - 1);
      const long long gl = line0 + ln;
      T *dcol = S.C + ln;
      int row = warp * 2 + (lane >> 4);
      if (gl < M) {
        const T *gcol = gsrc + gl;
        for (; row < rlo; row += 2 * NW) dcol[row * PITCH] = T(0);
        const T *src = gcol + (long long)(p0 - H + row) * s_pos;
        T *dst = dcol + row * PITCH;
        const long long gstep = 2LL * NW * s_pos;
#pragma unroll 4
        for (; row < rhi; row += 2 * NW, src += gstep, dst += 2 * NW * PITCH) {
          if (sizeof(T) == 8) cp_async8(dst, src); else cp_async4(dst, src);
        }
        for (; row < nrows; row += 2 * NW) dcol[row * PITCH] = T(0);
      } else {
        for (; row < nrows; row += 2 * NW) dcol[row * PITCH] = T(0);
      }
    } else {
      // a warp copies 32 consecutive values of one line per step
      for (int ln = warp; ln < LPG; ln += NW) {
        const long long gl = line0 + ln;
        T *dcol = S.C + ln;
        int row = lane;
        if (gl < M) {
          const T *lbase = gsrc + gl * s_line;
          for (; row < rlo; row += 32) dcol[row * PITCH] = T(0);
          const T *src = lbase + (p0 - H + row);
          T *dst = dcol + row * PITCH;
#pragma unroll 4
          for (; row < rhi; row += 32, src += 32, dst += 32 * PITCH) {
            if (sizeof(T) == 8) cp_async8(dst, src); else cp_async4(dst, src);
          }
          for (; row < nrows; row += 32) dcol[row * PITCH] = T(0);
        } else {
          for (; row < nrows; row += 32) dcol[row * PITCH] = T(0);
        }
      }
    }
  }
  cp_async_commit();
  if (threadIdx.x == 9 * LPG) {
    const T mmu = T(-F.sm_fac);
    T pk = mmu;
    for (int i = 0; i < FCH; ++i) {
      S.pwt[i] = pk;
      pk *= mmu;
    }
  }
  cp_async_wait_all_committed();
  __syncthreads();
  // extrapolated ghost cells C_{-2}, C_{-1}, C_L, C_{L+1} (T2S4:275-286)
  if (threadIdx.x < LPG) compat_ghosts(S.C + threadIdx.x, H - p0, p0 - H, p1 + H, L);
  __syncthreads();
  // In place, the segments of a line are read (halo) by the neighbouring CTAs
  // of its cluster: this CTA's reads are complete here, and no CTA of the
  // cluster stores before every CTA has arrived.  Out of place (ping-pong),
  // the launch has no clusters and needs no barrier.
  if (clustered) asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");

  // ---- one line per half-warp, FCH positions per lane ----
  if (np + 2 * J > FLANES * FCH) {
    // the host keeps segments within filter_seg_max(J)
    if (threadIdx.x == 0) atomicOr(status, STATUS_HALO);
    return;
  }
  {
    const int c = lane & (FLANES - 1);
    const int ln = warp * 2 + (lane >> 4);
    const unsigned fm = 0xffffffffu;  // the warp is converged at every shuffle
    const int rb = H - p0;            // row of position 0
    const T mmu = -mu;
    const T pw = S.pwt[FCH - 1];      // (-mu)^FCH

    {
      // b of positions [p0 - J - 1, p0 - J + FLANES * FCH + 1) into this
      // line's column of the second tile: every row the forward walk reads
      // (zero past p1 + J + 1, where the walk's values are masked); lane c
      // takes a contiguous run and carries the previous edge
      const long long gl = line0 + ln;
      const int kb = p0 - J - 1;
      const int kw = p0 - J + FLANES * FCH + 1;
      const int kv = min(kw, p1 + J + 1);
      const int mm = (kw - kb + FLANES - 1) / FLANES;
      const int s0 = kb + c * mm, s1 = min(kw, s0 + mm);
      const double tau0 = F.t_min + F.ht * (double)gl;
      const T kbc = T(F.kb);
      const LineFeet lf(F, tau0, tau0 + F.ht, toff + F.ta_rel, toff + F.tb_rel);
      // b = 0 outside the line (the compact mass matrix's zero ghosts).
      // Uniform displacement (the reference's rotation, constant, rotation):
      // cells clear of the clamps and ghost selections take the
      // shared-foot stencils, the rest the per-cell formulas of the
      // reference (remap_cell, foot_derivative); other velocity fields the
      // per-edge path (compat_edge)
      const int ka = max(s0, 0), kz = min(min(s1, kv), L);
      const LineView<T> vc{S.C + ln, rb, nrows, status};
      const bool uni = F.uniform != 0;
      T wr[6], wq[6];
      int n0 = 0, klo = 1, khi = 0;
      if (uni) {
        uniform_weights<T>(F, lf.foot(F, 0), wr, wq, &n0);
        klo = 2 - n0;
        khi = L - 4 - n0;
      }
      if (!F.dsrc) {
        T *bcol = S.B + ln;
        if (uni) {
          // the lane's run in three ranges: the cells clear of the clamps
          // and ghost selections [i0, i1) take the stencil with no
          // per-cell branches, the others the reference's formulas (or 0
          // outside the line)
          auto edge_cell = [&](int k) {
            T b = T(0);
            if (k >= ka && k < kz) {
              const double fa = lf.foot(F, k), fb = lf.foot(F, k + 1);
              b = remap_cell(F, vc, fa, fb) +
                  kbc * (foot_derivative(F, vc, fb) - foot_derivative(F, vc, fa));
            }
            bcol[(k + rb) * PITCH] = b;
          };
          const int i0 = max(s0, max(ka, klo)), i1 = max(i0, min(s1, min(kz, khi + 1)));
          const int ia = min(i0, s1);
          for (int k = i0; k < i1; ++k) {
            const T *cp = S.C + (k + n0 - 2 + rb) * PITCH + ln;
            T b = T(0);
#pragma unroll
            for (int t = 0; t < 6; ++t) b += (wr[t] + wq[t]) * cp[t * PITCH];
            bcol[(k + rb) * PITCH] = b;
          }
          for (int k = s0; k < s1; ++k) {  // the rest, skipping [i0, i1)
            if (k == ia) k = max(ia, i1);
            if (k >= s1) break;
            edge_cell(k);
          }
        } else {
          if (ka < kz) {
            CompatEdge<T> el = compat_edge<T>(F, lf, vc, vc, ka);
            for (int k = ka; k < kz; ++k) {
              const CompatEdge<T> er = compat_edge<T>(F, lf, vc, vc, k + 1);
              bcol[(k + rb) * PITCH] = compat_remap<T>(F, el, er, vc) + kbc * (er.d - el.d);
              el = er;
            }
          }
          for (int k = s0; k < s1; ++k)
            if (k < ka || k >= kz) bcol[(k + rb) * PITCH] = T(0);
        }
      } else {
        // the reference's third sweep differentiates the remapped field
        // (dcdx_bar_on_gpu(v_d_Cnphf_bar_x, ...), T2S4:929-932): remap the
        // cells [ra0, ra1) into the second tile, its ghosts, then
        // b = R + kbc (D_R(f_{k+1}) - D_R(f_k)) into the first tile (this
        // line's cells are no longer read)
        const int ra0 = max(0, kb - F.hd), ra1 = min(L, kv + F.hd);
        const int m1 = (ra1 - ra0 + FLANES - 1) / FLANES;
        const int q0 = ra0 + c * m1, q1 = min(ra1, q0 + m1);
        T *rcol = S.B + ln;
        if (uni) {
          auto edge_remap = [&](int k) {
            rcol[(k + rb) * PITCH] = remap_cell(F, vc, lf.foot(F, k), lf.foot(F, k + 1));
          };
          const int j0 = max(q0, klo), j1 = max(j0, min(q1, khi + 1));
          const int ja = min(j0, q1);
          for (int k = j0; k < j1; ++k) {
            const T *cp = S.C + (k + n0 - 2 + rb) * PITCH + ln;
            T r = T(0);
#pragma unroll
            for (int t = 0; t < 6; ++t) r += wr[t] * cp[t * PITCH];
            rcol[(k + rb) * PITCH] = r;
          }
          for (int k = q0; k < q1; ++k) {  // the rest, skipping [j0, j1)
            if (k == ja) k = max(ja, j1);
            if (k >= q1) break;
            edge_remap(k);
          }
        } else if (q0 < q1) {
          CompatEdge<T> el = compat_edge<T>(F, lf, vc, vc, q0);
          for (int k = q0; k < q1; ++k) {
            const CompatEdge<T> er = compat_edge<T>(F, lf, vc, vc, k + 1);
            rcol[(k + rb) * PITCH] = compat_remap<T>(F, el, er, vc);
            el = er;
          }
        }
        __syncwarp(fm);
        if (c == 0) compat_ghosts(rcol, rb, ra0 - 2, ra1 + 2, L);
        __syncwarp(fm);
        const LineView<T> vr{rcol, rb, nrows, status};
        T *bcol = S.C + ln;
        auto edge_cell = [&](int k) {
          T b = T(0);
          if (k >= ka && k < kz) {
            const double fa = lf.foot(F, k), fb = lf.foot(F, k + 1);
            b = vr(k) + kbc * (foot_derivative(F, vr, fb) - foot_derivative(F, vr, fa));
          }
          bcol[(k + rb) * PITCH] = b;
        };
        // interior cells of a uniform displacement [i0, i1): the stencil
        // (empty range for other fields: klo > khi)
        const int i0 = max(s0, max(ka, klo)), i1 = max(i0, min(s1, min(kz, khi + 1)));
        const int ia = min(i0, s1);
        for (int k = i0; k < i1; ++k) {
          const T *rp = rcol + (k + n0 - 2 + rb) * PITCH;
          T acc = T(0);
#pragma unroll
          for (int t = 0; t < 6; ++t) acc += wq[t] * rp[t * PITCH];
          bcol[(k + rb) * PITCH] = rcol[(k + rb) * PITCH] + acc;
        }
        for (int k = s0; k < s1; ++k) {  // the rest, skipping [i0, i1)
          if (k == ia) k = max(ia, i1);
          if (k >= s1) break;
          edge_cell(k);
        }
      }
      __syncwarp(fm);
    }

    // forward: w_k = (1/c) M b_k - mu w_{k-1} over [p0 - J, qb), qb = p1 + J.
    // Lanes past qb walk stage rows that are allocated but not staged: their
    // values only flow further right and are masked by the backward load.
    const int qb = p1 + J;
    const int k0 = p0 - J + c * FCH;
    const int r0 = k0 - 1 + rb;  // row of the first tap
    const bool ok = r0 >= 0 && r0 + FCH + 2 <= S.rows;
    if (!ok) atomicOr(status, STATUS_HALO);
    T v[FCH];
    {
      // w_k = (1/12c)(b_{k-1} + 10 b_k + b_{k+1}) - mu w_{k-1}; zero input
      // outside the line (non-cyclic system, exact zero start at 0)
      const T icw = T(F.sm_inv_den / 12.0);
      const T *bp = (F.dsrc ? S.C : S.B) + (ok ? r0 : 0) * PITCH + ln;
      T b0 = bp[0], b1 = bp[PITCH];
      T w = T(0);
#pragma unroll
      for (int i = 0; i < FCH; ++i) {
        const T b2 = bp[(2 + i) * PITCH];
        T in = icw * ((b0 + b2) + T(10.0) * b1);
        if ((unsigned)(k0 + i) >= (unsigned)L) in = T(0);
        w = in + mmu * w;
        v[i] = w;
        b0 = b1;
        b1 = b2;
      }
    }
    {
      // carries: chunk map x -> pw x + e_c, inclusive scan over the line's lanes
      T sa = pw, sb = v[FCH - 1];
#pragma unroll
      for (int d = 1; d < FLANES; d <<= 1) {
        const T pa = __shfl_up_sync(fm, sa, d, FLANES);
        const T pb = __shfl_up_sync(fm, sb, d, FLANES);
        if (c >= d) {
          sb = sa * pb + sb;
          sa = sa * pa;
        }
      }
      T cin = __shfl_up_sync(fm, sb, 1, FLANES);
      if (c == 0) cin = T(0);
      // + cin (-mu)^(i+1), the powers by a running product (no table loads)
#pragma unroll
      for (int i = 0; i < FCH; ++i) {
        cin *= mmu;
        v[i] += cin;
      }
    }
    // The backward filter runs on the same positions k0 .. k0+FCH-1 of each
    // lane (w stays in registers); positions left of p0 are warm-up values
    // whose x is discarded, positions from qb on start it from zero.
    const int k1 = k0;
    // positions of this lane inside the backward range (the zero start is at
    // the line's end, x_L = 0)
    const int qe = min(qb, L), nb = qe - k1;
    // zero from qe on; a backward range that covers every lane's positions
    // needs none (uniform over the CTA)
    if (qe - (p0 - J) < FLANES * FCH) {
#pragma unroll
      for (int i = 0; i < FCH; ++i) v[i] = (i < nb) ? v[i] : T(0);
    }

    // backward: x over [k0, qb), zero start at qb
    {
      T x = T(0);
#pragma unroll
      for (int i = FCH - 1; i >= 0; --i) {
        x = v[i] + mmu * x;
        v[i] = x;
      }
      T sa = pw, sb = v[0];
#pragma unroll
      for (int d = 1; d < FLANES; d <<= 1) {
        const T pa = __shfl_down_sync(fm, sa, d, FLANES);
        const T pb = __shfl_down_sync(fm, sb, d, FLANES);
        if (c + d < FLANES) {
          sb = sa * pb + sb;
          sa = sa * pa;
        }
      }
      T cin = __shfl_down_sync(fm, sb, 1, FLANES);
      if (c == FLANES - 1) cin = T(0);
#pragma unroll
      for (int i = FCH - 1; i >= 0; --i) {
        cin *= mmu;  // cin (-mu)^(FCH - i)
        v[i] += cin;
      }
    }
    if (p0 == 0) {
      // non-cyclic system: A = c (1 + mu S^-1)(1 + mu S) + c mu^2 e_0 e_0^T,
      // so x = y - y_0 g with g_k = mu^2 ((-mu)^k - (-mu)^(2L-k)) /
      // (1 - mu^(2L+2)) (Sherman-Morrison); y_0 is this segment's x at 0
      const int c0 = J / FCH, i0 = J - c0 * FCH;
      T y0 = T(0);
#pragma unroll
      for (int i = 0; i < FCH; ++i) y0 = (i == i0) ? v[i] : y0;
      y0 = __shfl_sync(fm, y0, c0, FLANES);
      const double q = -F.sm_fac;
      const double A = q * q / (1.0 - powi(q * q, L + 1));
      const bool tail = powi(fabs(q), L) >= 0x1p-60;  // (-mu)^(2L-k) still matters
      double qk = powi(q, max(k0, 0));
#pragma unroll
      for (int i = 0; i < FCH; ++i) {
        const int k = k0 + i;
        if (k >= 0 && k < L) {
          const double gk = A * (tail ? qk - powi(q, 2 * L - k) : qk);
          v[i] -= y0 * T(gk);
          qk *= q;
        }
      }
    }
    __syncwarp(fm);
    {
      T *xp = S.C + (k1 + rb) * PITCH + ln;
#pragma unroll
      for (int i = 0; i < FCH; ++i) xp[i * PITCH] = v[i];
    }
  }
  __syncthreads();
  if (clustered) asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");

  // ---- cooperative store of rows H .. H+np-1 ----
  if (xsweep) {
    const int l = lane & (LPG - 1);
    const long long gl = line0 + l;
    if (gl < M) {
      const int row0 = warp * 2 + (lane >> 4);
      T *gp = gdst + (long long)(p0 + row0) * s_pos + gl;
      const T *sp = S.C + (row0 + H) * PITCH + l;
      const long long gstep = 2LL * NW * s_pos;
      for (int row = row0; row < np; row += 2 * NW) {
        *gp = *sp;
        gp += gstep;
        sp += 2 * NW * PITCH;
      }
    }
  } else {
    for (int l2 = warp; l2 < LPG; l2 += NW) {
      const long long gl2 = line0 + l2;
      if (gl2 >= M) continue;
      T *lbase = gdst + gl2 * s_line + p0;
      const T *scol = S.C + H * PITCH + l2;
      for (int row = lane; row < np; row += 32) lbase[row] = scol[row * PITCH];
    }
  }
}

}  // namespace

size_t sweep_smem_bytes(int lc_max, int halo, bool fp64, bool source) {
  size_t el = fp64 ? 8 : 4;
  size_t n = (source ? 3 : 2) * (size_t)(lc_max + 2 * halo) * PITCH +
             3 * (size_t)lc_max + 3 * (size_t)NCH * LPG + 8 * (size_t)LPG;
  return FD_BYTES + n * el;
}

// The filter kernel's tile; exact, cell: the larger and smaller tiles that bound
// which steps are taken.
size_t sweep_filter_smem_bytes(int lc_max, int halo, bool fp64, bool exact, bool cell) {
  size_t el = fp64 ? 8 : 4;
  return FD_BYTES + 64 * sizeof(int) +
         (8 * (size_t)LPG + 32 + (exact ? (size_t)FPW + 2 * LPG : 0) +
          (cell ? 2 : 1) * (size_t)filter_tile_rows(lc_max, halo) * PITCH) * el +
         (cell ? 8 * (size_t)FPW + 8 : 0);
}

int filter_segment_max(int J) { return filter_seg_max(J); }

cudaError_t launch_filter_weights(bool fp64, const SweepField *d_field, void *wt, int *nt,
                                  int lines, cudaStream_t stream, int variant) {
  const int bt = 128, grid = (lines + bt - 1) / bt;
  count_launch();
  if (fp64)
    filter_weights_kernel<double><<<grid, bt, 0, stream>>>(d_field, static_cast<double *>(wt), nt,
                                                           lines, variant);
  else
    filter_weights_kernel<float><<<grid, bt, 0, stream>>>(d_field, static_cast<float *>(wt), nt,
                                                          lines, variant);
  return cudaGetLastError();
}

size_t sweep_fast_smem_bytes(int lc_max, int halo, bool fp64) {
  size_t el = fp64 ? 8 : 4;
  size_t n = (size_t)(lc_max + 2 * halo) * PITCH + (size_t)lc_max * PITCH + 5 * (size_t)lc_max +
             2 * (size_t)NCH + 1 + 2 * (size_t)NCH * LPG + 16 * (size_t)LPG;
  return FD_BYTES + 64 * sizeof(int) + n * el;
}

// Programmatic dependent launch: the filter kernels wait for their predecessor
// before reading cells, after fetching what is constant.  Batch of 64 mixed
// instances: 1323 ms without, 1276 ms with; 12 instances up to 583^2: 120 ms
// without, 101 ms with.  CCFV_PDL=0 turns it off.
bool pdl_enabled() {
  static const bool on = [] {
    const char *e = std::getenv("CCFV_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

template <typename T>
static cudaError_t launch_impl(const LaunchGeom &G, const PlanFields &plan,
                               const SweepField *d_fields, int nfields, int group_base, int groups_total, double toff,
                               const FieldIo &io,
                               unsigned *d_status, int jstep, int nslice, const int *nlo,
                               bool inplace, cudaStream_t stream, const int *g0idx, bool pdl_ok) {
  const int variant = G.variant, cs = G.cs, lc_max = G.lc_max, halo = G.halo;
  if (stream_variant(variant))
    return launch_stream<T>(G, plan, d_fields, nfields, group_base, groups_total, toff, io, d_status,
                            jstep, nslice, nlo, inplace, stream, g0idx, pdl_ok && pdl_enabled());
  const bool fast = (variant == SWEEP_FAST);
  const bool filt = filter_variant(variant);
  const bool src = (variant == SWEEP_GENERAL_SRC);
  const size_t smem = filt ? sweep_filter_smem_bytes(lc_max, halo, sizeof(T) == 8, false, true)
                      : fast ? sweep_fast_smem_bytes(lc_max, halo, sizeof(T) == 8)
                             : sweep_smem_bytes(lc_max, halo, sizeof(T) == 8, src);
  {
    // Function attributes apply to the device that is current when they are
    // set: configure each device once (contexts, batches, servers and the
    // allocation-free step may run on different devices of one process, from
    // several host threads).
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    static std::atomic<bool> configured[MAX_DEVICES];
    static std::mutex config_mu;
    if (!configured[dev].load(std::memory_order_acquire)) {
      std::lock_guard<std::mutex> lk(config_mu);
      if (!configured[dev].load(std::memory_order_relaxed)) {
        for (const void *fn :
             {(const void *)sweep_kernel<T>, (const void *)sweep_fast_kernel<T>,
              (const void *)sweep_filter_kernel<T>}) {
          err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     227 * 1024);
          if (err != cudaSuccess) return err;
          err = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
          if (err != cudaSuccess) return err;
        }
        configured[dev].store(true, std::memory_order_release);
      }
    }
  }
  if (groups_total <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(groups_total * cs), 1, 1);
  cfg.blockDim = dim3(NTH, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  if (filt) {
    // whole lines per CTA, or out of place: no cluster
    int clustered = 0;
    cudaLaunchAttribute fattr[2];
    unsigned na = 0;
    if (cs > 1 && inplace) {
      fattr[na++] = attr[0];
      clustered = 1;
    }
    if (pdl_ok && pdl_enabled()) {
      fattr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      fattr[na].val.programmaticStreamSerializationAllowed = 1;
      ++na;
    }
    cfg.attrs = fattr;
    cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, sweep_filter_kernel<T>, d_fields, nfields, group_base * cs, toff, io, lc_max,
                              halo, d_status, jstep, nslice, nlo, cs, clustered, g0idx);
  }
  if (fast)
    return cudaLaunchKernelEx(&cfg, sweep_fast_kernel<T>, d_fields, nfields, group_base, toff,
                              io, lc_max, halo, d_status, jstep, nslice, nlo, g0idx);
  return cudaLaunchKernelEx(&cfg, sweep_kernel<T>, d_fields, nfields, group_base, toff, io,
                            lc_max, halo, d_status, jstep, nslice, nlo, g0idx);
}

template <typename T>
cudaError_t launch_sweep(const LaunchGeom &G, const PlanFields &plan, const SweepField *d_fields,
                         int nfields, int group_base, int groups_total, double toff,
                               const FieldIo &io,
                         unsigned *d_status, cudaStream_t stream, int jstep, bool inplace) {
  return launch_impl<T>(G, plan, d_fields, nfields, group_base, groups_total, toff, io,
                        d_status, jstep, 0, nullptr, inplace, stream, nullptr, true);
}

template <typename T>
cudaError_t launch_sweep_batch(const LaunchGeom &G, const SweepField *d_fields, int nfields,
                               int group_base, int groups_total, const BatchStep &bs,
                               unsigned *d_status, cudaStream_t stream) {
  return launch_impl<T>(G, PlanFields(), d_fields, nfields, group_base, groups_total, 0.0,
                        FieldIo(), d_status,
                        bs.jstep, bs.nslice, bs.nlo, bs.inplace, stream, bs.g0idx, bs.pdl);
}

template cudaError_t launch_sweep<double>(const LaunchGeom &, const PlanFields &,
                                          const SweepField *, int, int, int, double, const FieldIo &,
                                          unsigned *, cudaStream_t, int, bool);
template cudaError_t launch_sweep<float>(const LaunchGeom &, const PlanFields &,
                                         const SweepField *, int, int, int, double, const FieldIo &,
                                         unsigned *, cudaStream_t, int, bool);
template cudaError_t launch_sweep_batch<double>(const LaunchGeom &, const SweepField *, int, int,
                                                int, const BatchStep &, unsigned *, cudaStream_t);
template cudaError_t launch_sweep_batch<float>(const LaunchGeom &, const SweepField *, int, int,
                                               int, const BatchStep &, unsigned *, cudaStream_t);

}  // namespace ccfv
