// line_ends.cuh -- the reference's per-edge formulas next to the ends of a line
// (stream.cu).  No CUDA header is needed: a host compiler takes the file with
// the function qualifiers defined away.
#pragma once

namespace ccfv {

// A foot in cell units: cell and offset in it.
struct FootCell {
  int k;
  double xi;
};

// Marks of the feet that are in no cell of the line: below it (clamped to cell
// 0), above it (added to the cell it is clamped to: L - 1, or L by rounding),
// and within the clamp of one of its ends (remap_at_end).
constexpr int FOOT_BELOW = -1, FOOT_ON_END = -2, FOOT_ABOVE = 1 << 30;

// `at` of a foot that lies in no cell.
constexpr double NO_CELL = -4096.0;

// Ghost cells C_{-2}, C_{-1} (left) or C_L, C_{L+1} (3-point extrapolation,
// T2S4:275-286) of the line ends: near to far cells a, b, d; ghosts at `g`.
template <typename T>
__device__ __forceinline__ void ghosts(T a, T b, T d, T &g1, T &g2) {
  const T e = T(1.0 / 11.0);
  g1 = e * (-d + T(3) * b + T(9) * a);
  g2 = e * (T(-15) * d + T(56) * b - T(30) * a);
}

// PPM integral of a cell from its left edge to xi (d_intC_ppm4th, T2S4:63-65,
// with the coefficients of T2S4:260-304).
template <typename T, typename V>
__device__ __forceinline__ T ppm_to(const V &c, int k, T xi) {
  const T m2 = c(k - 2), m1 = c(k - 1), z = c(k), p1 = c(k + 1), p2 = c(k + 2);
  const T cl = T(7.0 / 12.0) * (z + m1) - T(1.0 / 12.0) * (p1 + m2);
  const T cr = T(7.0 / 12.0) * (p1 + z) - T(1.0 / 12.0) * (p2 + m1);
  const T D = cr - cl, C6 = T(6.0) * (z - T(0.5) * (cl + cr));
  const T xi2 = xi * xi;
  return T(-1.0 / 3) * C6 * (xi2 * xi) + T(0.5) * (D + C6) * xi2 + cl * xi;
}

// Fourth-order derivative at a foot in cell k (T2S4:440-547) with the
// reference's choice of ghosts at k = 1 (-2 tap reads C_{-2}) and k = L - 2
// (+2 tap reads C_{L+1}).
template <typename T, typename V>
__device__ __forceinline__ T derivative_at(const V &c, int k, T xi, int L, T inv12h) {
  const T m2 = c(k == 1 ? -2 : k - 2), m1 = c(k - 1), z = c(k), p1 = c(k + 1),
          p2 = c(k == L - 2 ? L + 1 : k + 2);
  const T xi2 = xi * xi, xi3 = xi2 * xi;
  return inv12h * ((T(2.0) * xi3 - T(6.0) * xi2 + T(3.0) * xi + T(1.0)) * m2 +
                   (T(-8.0) * xi3 + T(18.0) * xi2 + T(6.0) * xi - T(15.0)) * m1 +
                   (T(12.0) * xi3 - T(18.0) * xi2 - T(24.0) * xi + T(15.0)) * z +
                   (T(-8.0) * xi3 + T(6.0) * xi2 + T(18.0) * xi - T(1.0)) * p1 +
                   (T(2.0) * xi3 - T(3.0) * xi) * p2);
}

// PPM integral up to one edge's foot and derivative there.  In: phi, the foot's
// cell (NO_CELL: none, both are zero), and d, its offset in it; out: the integral
// and the derivative of the line's cells (REMAPPED: d stays the offset, for the
// derivative of the remapped field).  A foot on the end of the line has its
// derivative in end_cell() where the derivative's clamp is not the remap's
// (own_clamp).  False: the cells around the foot are not staged; nothing has
// been read, both are zero, and the caller marks the foot FOOT_ABOVE, so that
// no cell is summed up to it either.
template <bool REMAPPED, typename T, typename V, typename E>
__device__ __forceinline__ bool foot_inputs(const V &cells, int L, T inv12h, const int &mark,
                                            bool own_clamp, const E &end_cell, T &phi, T &d) {
  const T at = phi;
  T xi = d;
  phi = d = T(0);
  if (at == T(NO_CELL)) return true;
  int k = (int)at;
  if (!cells.near(k)) return false;
  if (k >= 0 && k < L) phi = ppm_to(cells, k, xi);
  if (REMAPPED) {
    d = xi;
  } else if (mark != FOOT_BELOW && mark < FOOT_ABOVE) {
    if (mark == FOOT_ON_END && own_clamp) {
      const FootCell q = end_cell();
      k = q.k;
      xi = T(q.xi);
    }
    d = derivative_at(cells, k, xi, L, inv12h);
  }
  return true;
}

}  // namespace ccfv
