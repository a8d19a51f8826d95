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
// What bounds it: HBM.  One FP64 sweep of 4096^2 (268 MB): y 41.2 us, x 47 us,
// against 41.0 us for the copy rate and 62 us for the tile kernel this
// replaced (8-byte copies, 16 lanes per line, carries added afterwards, two
// CTA barriers; it issued 69 instructions per cell, this one about 26).
#include <atomic>
#include <cstdlib>
#include <mutex>

#include "ccfv_internal.h"
#include "sweep_device.cuh"

namespace ccfv {

namespace {

constexpr int SCH = STREAM_CH;     // positions per lane
constexpr int X_LINES = 16;        // lines per CTA of an x sweep
constexpr int X_PITCH = X_LINES + 2;
constexpr int X_WARPS = X_LINES / 2;
constexpr int Y_WARPS = 4;

template <int DIR, int LN>
struct StreamCta {
  static constexpr int warps = DIR == 0 ? X_WARPS : Y_WARPS;
  static constexpr int lpw = DIR == 0 ? 2 : 32 / LN;  // lines per warp
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

// v[i] = sum_m o[m] C_{row + i + m}, the stencil input of SCH positions
// (stride ES between positions).
template <typename T, int ES>
__device__ __forceinline__ void stencil8(const T *cp, const T (&o)[8], T (&v)[SCH]) {
  T q[7];
#pragma unroll
  for (int m = 0; m < 7; ++m) q[m] = cp[m * ES];
#pragma unroll
  for (int i = 0; i < SCH; ++i) {
    const T q7 = cp[(7 + i) * ES];
    T t = o[0] * q[0];
#pragma unroll
    for (int m = 1; m < 7; ++m) t += o[m] * q[m];
    v[i] = t + o[7] * q7;
#pragma unroll
    for (int m = 0; m < 6; ++m) q[m] = q[m + 1];
    q[6] = q7;
  }
}

// What a CTA needs of its field.
struct StreamField {
  int L, M, J, H, groups, cta0;
  long long s_line, s_pos;
  double mu;
  const void *wt;
  const int *nt;
};
__device__ __forceinline__ StreamField stream_field(const SweepField &f) {
  return StreamField{f.L, f.M, f.jf, f.halo_f, f.groups, f.cta0, f.s_line, f.s_pos, f.sm_fac,
                     f.wt, f.nt};
}

template <typename T, int DIR, int LN>
__global__ void __launch_bounds__(StreamCta<DIR, LN>::warps * 32, DIR == 0 ? 4 : 8)
    stream_kernel(const __grid_constant__ PlanFields plan, const SweepField *__restrict__ fields,
                  int nfields, int first, void *data_override, int rows, unsigned *status,
                  int jstep, int nslice, const int *nlo, int cs, int clustered,
                  const int *g0idx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NT = StreamCta<DIR, LN>::warps * 32;
  constexpr int LPW = StreamCta<DIR, LN>::lpw;
  constexpr int ES = DIR == 0 ? X_PITCH : 1;    // element stride of a position
  constexpr int LS = DIR == 0 ? 2 : 1;          // lane stride of a chunk
  constexpr unsigned FULL = 0xffffffffu;
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
  int tile, rank;
  const void *vs;
  void *vd;
  if (plan.tiles > 0) {
    F = stream_field(plan.f);
    tile = blockIdx.x;
    rank = blockIdx.y;
    field_io(plan.f, jstep, &vs, &vd, data_override);
    const long long off = (first + (int)blockIdx.z) * plan.stride;
    vs = static_cast<const char *>(vs) + off;
    vd = static_cast<char *>(vd) + off;
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  } else {
    const int cta = (int)blockIdx.x + first;
    const SweepField &f = fields[find_field(fields, g0idx, nfields, cta / cs)];
    F = stream_field(f);
    const int q = cta - F.cta0;
    rank = clustered ? q % cs : q / F.groups;
    tile = clustered ? q / cs : q - rank * F.groups;
    field_io(f, jstep, &vs, &vd, data_override);
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (!field_active(f, jstep, nslice, nlo)) return;  // uniform over a cluster
  }
  const T *src = reinterpret_cast<const T *>(vs);
  T *dst = reinterpret_cast<T *>(vd);
  const int L = F.L, M = F.M, J = F.J, H = F.H;
  const long long s_line = F.s_line, s_pos = F.s_pos;
  const int Lc = plan.tiles > 0 ? plan.seg : stream_seg(L, cs);
  const int p0 = min(L, rank * Lc), p1 = min(L, p0 + Lc), np = p1 - p0;
  const int line0 = tile * StreamCta<DIR, LN>::lines;        // first line of the CTA
  if (np <= 0 && !clustered) return;

  // ---- stage the cells (periodic wrap) ----
  // Positions p0-J .. p1+J-1 are walked by the first `act` lanes of a line, and
  // the cells of all positions of those lanes are staged: past p1+J they only
  // lengthen the backward warm-up, so nothing is masked inside a lane.
  const int act = min(LN, (np + 2 * J + SCH - 1) / SCH);
  const int nr = (act * SCH + 2 * (H - J) + 1) & ~1;
  const int b0 = p0 - H;  // position of staged row 0
  const bool inside = b0 >= 0 && b0 + nr <= L;
  const bool pairs = ((DIR == 0 ? s_pos : s_line) & 1) == 0 && (DIR == 0 || (L & 1) == 0) &&
                     (((size_t)src | (size_t)dst) & (2 * sizeof(T) - 1)) == 0;
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
          const T *p = s + (long long)wrap_pos(b0 + r, L) * s_pos;
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
          for (int e = 2 * lane; e < nr; e += 64) copy_pair(d + e, s + wrap_pos(b0 + e, L));
        } else {
          for (int e = lane; e < nr; e += 32) copy_one(d + e, s + wrap_pos(b0 + e, L));
        }
      }
    }
  }
  cp_async_commit();
  // this lane's line and its stencil, while the cells arrive
  const int c = DIR == 0 ? lane >> 1 : lane % LN;            // chunk
  const int lw = DIR == 0 ? (lane & 1) : lane / LN;          // line within the warp
  const int line = line0 + warp * LPW + lw;
  const T mmu = T(-F.mu);
  T o[8];
  {
    const T *w = reinterpret_cast<const T *>(F.wt) + (size_t)line * 8;  // padded past M
#pragma unroll
    for (int m = 0; m < 8; ++m) o[m] = __ldg(w + m);
  }
  const int n0 = __ldg(F.nt + line);
  static_assert(SCH == 17, "pw");
  T pw = mmu * mmu;  // (-mu)^17
  pw *= pw;
  pw *= pw;
  pw *= pw * mmu;
  cp_async_wait_all_committed();
  if (DIR == 0) __syncthreads(); else __syncwarp();
  // In place, the segments of a line are read (halo) by the neighbouring CTAs
  // of its cluster: no CTA stores before every CTA has staged.
  if (clustered) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.aligned;\n" ::: "memory");
  }

  // ---- stencil and recurrences ----
  T *const col = DIR == 0 ? tile_s + warp * LPW + lw : tile_s + (size_t)(warp * LPW + lw) * rows;
  const int k0 = H - J + c * SCH;  // staged row of this lane's first position
  const int r0 = k0 + n0 - 3;
  const bool ok = r0 >= 0 && r0 + SCH + 7 <= rows;
  if (!ok && line < M) atomicOr(status, STATUS_HALO);
  // doubling steps that bring a carry in from every chunk of the warm-up (FP32:
  // one more, so that what is left out, |mu|^J of it at every chunk start, is
  // far below a rounding and not a share of one with the same sign everywhere)
  const int ns = (J <= SCH ? 0 : J <= 2 * SCH ? 1 : 2) + (sizeof(T) == 4 ? 1 : 0);
  T v[SCH];
  stencil8<T, ES>(col + (ok ? r0 : 0) * ES, o, v);
  T w = T(0);
#pragma unroll
  for (int i = 0; i < SCH; ++i) w = v[i] + mmu * w;
  {
    T pd = pw;
    for (int s = 0; s < ns; ++s) {
      const T t = __shfl_up_sync(FULL, w, LS << s, DIR == 0 ? 32 : LN);
      if (c >= (1 << s)) w += pd * t;
      pd *= pd;
    }
    w = __shfl_up_sync(FULL, w, LS, DIR == 0 ? 32 : LN);
    if (c == 0) w = T(0);
  }
#pragma unroll
  for (int i = 0; i < SCH; ++i) {
    w = v[i] + mmu * w;
    v[i] = w;
  }
  T x = T(0);
#pragma unroll
  for (int i = SCH - 1; i >= 0; --i) x = v[i] + mmu * x;
  if (c >= act) x = T(0);  // lanes whose cells are not staged
  {
    T pd = pw;
    for (int s = 0; s < ns; ++s) {
      const T t = __shfl_down_sync(FULL, x, LS << s, DIR == 0 ? 32 : LN);
      if (c + (1 << s) < LN) x += pd * t;
      pd *= pd;
    }
    x = __shfl_down_sync(FULL, x, LS, DIR == 0 ? 32 : LN);
    if (c == LN - 1) x = T(0);
  }
  __syncwarp();  // every lane of the line has read its cells
  {
    T *xp = col + k0 * ES;
#pragma unroll
    for (int i = SCH - 1; i >= 0; --i) {
      x = v[i] + mmu * x;
      xp[i * ES] = x;
    }
  }
  if (DIR == 0) __syncthreads(); else __syncwarp();
  if (clustered) asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");

  // ---- store positions p0 .. p1-1 ----
  if (DIR == 0) {
    if (pairs) {
      constexpr int G = X_LINES / 2;
      const int g = 2 * ((int)threadIdx.x % G);
      if (line0 + g < M) {
        T *d = dst + (long long)p0 * s_pos + line0 + g;
        const T *s = tile_s + H * X_PITCH + g;
#pragma unroll 4
        for (int r = (int)threadIdx.x / G; r < np; r += NT / G)
          *reinterpret_cast<Pair<T> *>(d + (long long)r * s_pos) =
              *reinterpret_cast<const Pair<T> *>(s + r * X_PITCH);
      }
    } else {
      const int g = (int)threadIdx.x % X_LINES;
      if (line0 + g < M)
        for (int r = (int)threadIdx.x / X_LINES; r < np; r += NT / X_LINES)
          dst[(long long)(p0 + r) * s_pos + line0 + g] = tile_s[(r + H) * X_PITCH + g];
    }
  } else {
#pragma unroll
    for (int l = 0; l < LPW; ++l) {
      const int gl = line0 + warp * LPW + l;
      if (gl < M) {
        T *d = dst + (long long)gl * s_line + p0;
        const T *s = tile_s + (size_t)(warp * LPW + l) * rows + H;
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
using StreamKernelT = void (*)(const PlanFields, const SweepField *, int, int, void *, int,
                               unsigned *, int, int, const int *, int, int, const int *);

template <typename T>
StreamKernelT<T> stream_kernel_for(int dir, int lanes) {
  if (dir == 0) return stream_kernel<T, 0, 16>;
  return lanes == 32 ? stream_kernel<T, 1, 32> : stream_kernel<T, 1, 16>;
}

}  // namespace

int stream_tile_lines(int dir, int lanes) {
  return dir == 0 ? X_LINES : Y_WARPS * (32 / lanes);
}

size_t stream_smem_bytes(int dir, int lanes, int rows, bool fp64) {
  const size_t n = dir == 0 ? (size_t)X_PITCH * rows
                            : (size_t)stream_tile_lines(dir, lanes) * rows;
  return n * (fp64 ? 8 : 4);
}

template <typename T>
cudaError_t launch_stream(const LaunchGeom &G, const PlanFields &plan, const SweepField *d_fields,
                          int nfields, int group_base, int groups_total, void *data,
                          unsigned *d_status,
                          int jstep, int nslice, const int *nlo, bool inplace,
                          cudaStream_t stream, const int *g0idx, bool pdl) {
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
      for (auto fn : {stream_kernel_for<T>(0, 16), stream_kernel_for<T>(1, 16),
                      stream_kernel_for<T>(1, 32)}) {
        err = cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   227 * 1024);
        if (err != cudaSuccess) return err;
        err = cudaFuncSetAttribute((const void *)fn,
                                   cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
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
  cfg.blockDim = dim3((unsigned)((G.dir == 0 ? X_WARPS : Y_WARPS) * 32), 1, 1);
  cfg.dynamicSmemBytes = stream_smem_bytes(G.dir, G.lanes, G.rows, sizeof(T) == 8);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned na = 0;
  // in place with several segments per line: they form one cluster
  const int clustered = inplace && G.cs > 1 ? 1 : 0;
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
  return cudaLaunchKernelEx(&cfg, stream_kernel_for<T>(G.dir, G.lanes), plan, d_fields, nfields,
                            by_value ? group_base / plan.tiles : group_base * G.cs, data, G.rows, d_status, jstep, nslice, nlo, G.cs,
                            clustered, g0idx);
}

template cudaError_t launch_stream<double>(const LaunchGeom &, const PlanFields &,
                                           const SweepField *, int, int, int, void *, unsigned *,
                                           int, int, const int *, bool, cudaStream_t, const int *,
                                           bool);
template cudaError_t launch_stream<float>(const LaunchGeom &, const PlanFields &,
                                          const SweepField *, int, int, int, void *, unsigned *,
                                          int, int, const int *, bool, cudaStream_t, const int *,
                                          bool);

}  // namespace ccfv
