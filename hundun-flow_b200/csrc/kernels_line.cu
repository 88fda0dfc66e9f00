// Zebra line relaxation (y-line relaxation for stretched grids) on sm_100a.
//
// The reference relaxes strong-axis lines by lexicographic line Gauss-Seidel
// with one Thomas solve per line (line_smooth_axis, src/solver_mg.cpp:
// 3352-3539).  Here lines are coloured by the parity of their transverse
// index (zebra): a colour's lines couple only to the other colour, so all of
// them are solved at once.  The line matrices depend only on the level
// coefficients, so every factorisation is computed once per coefficient
// update and each sweep does only right-hand-side work:
//   * many lines per colour: a chunked scan over precomputed Thomas
//     factors.  Lanes run across lines (loads coalesce along x), each
//     thread owns a chunk of up to 16 rows of its line, and the chunks of a
//     line combine the affine maps of the forward and backward recurrences
//     through shared memory;
//   * few lines per colour (coarse levels): one CTA row per line runs
//     parallel cyclic reduction with precomputed elimination factors held
//     in registers;
//   * the coarsest level keeps x and rhs in shared memory for all of its
//     coarse sweeps in one launch.
#include "kernels.hpp"
#include "phase_device.cuh"

#include <algorithm>
#include <type_traits>

namespace hfps {
namespace {


// Right-hand side of the rows of one line with everything that is constant
// along the line hoisted: the transverse neighbours' offsets (0 where the
// neighbour is outside the level, read as 0 for Dirichlet and as the cell
// itself for Neumann), the face arrays with their index at row 0 and stride
// per row, and the line-end boundary faces.  Every load of a row is
// unconditional, so a thread can keep many rows' loads in flight.  The
// arithmetic and its order are line_rhs's.  Transverse neighbours belong to
// the other colour, which a colour pass never writes, so they are read
// through the read-only path.  With hx > 0 the vectors are in split rows
// (SplitPos): an x neighbour sits in the other half of the row, a y or z
// neighbour in the same half of the previous or next row.  A neighbour
// outside the level reads the cell itself (Neumann), so it counts as this
// colour's value for the zero flags of the first sweep.
// Variants of a scan colour pass by what is known of x (LineRhs::row).
enum ScanMode : int { kScanNormal = 0, kScanOwnZero = 1, kScanFresh = 2 };

template <class T, int AXIS, bool SPLIT>
struct LineRhs {
  static constexpr int kA0 = AXIS == 0 ? 1 : 0;  // first transverse axis
  static constexpr int kA1 = AXIS == 2 ? 1 : 2;  // second transverse axis
  const T* face[2];
  int fbase[2], fstride[2], fhigh[2];
  int off[4];
  bool keep[4];
  T end_low, end_high;   // line-end boundary faces (rows 0 and extent-1)
  bool lkeep_low, lkeep_high;

  __device__ static void axis_faces(const Level<T>& L, int axis, int i, int j,
                                    int k, int line_axis, const T*& f,
                                    int& b, int& st, int& hi) {
    // Face index of cell (i, j, k) on `axis`, its step per row along
    // line_axis, and the offset of the cell's high face.
    const int nx = L.nx, ny = L.ny, nz = L.nz;
    if (axis == 0) {
      f = L.fx;
      b = i + (nx + 1) * (j + ny * k);
      st = line_axis == 0 ? 1 : (line_axis == 1 ? nx + 1 : (nx + 1) * ny);
      hi = 1;
    } else if (axis == 1) {
      f = L.fy;
      b = i + nx * (j + (ny + 1) * k);
      st = line_axis == 0 ? 1 : (line_axis == 1 ? nx : nx * (ny + 1));
      hi = nx;
    } else {
      f = L.fz;
      b = i + nx * (j + ny * k);
      st = line_axis == 0 ? 1 : (line_axis == 1 ? nx : nx * ny);
      hi = nx * ny;
    }
    (void)nz;
  }

  // own_zero: this colour's x counts as zero, so a neighbour that is the cell
  // itself is left out.
  __device__ LineRhs(const Level<T>& L, int fa, int fb, int hx, bool own_zero = false) {
    int i0, j0, k0;
    line_cell(AXIS, fa, fb, 0, i0, j0, k0);
    const int idx[3] = {i0, j0, k0};
    const int ext[3] = {L.nx, L.ny, L.nz};
    const int step[3] = {1, L.nx, L.nx * L.ny};
    const int axes[2] = {kA0, kA1};
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int a = axes[n];
      axis_faces(L, a, i0, j0, k0, AXIS, face[n], fbase[n], fstride[n], fhigh[n]);
      const bool low_in = idx[a] > 0, high_in = idx[a] + 1 < ext[a];
      int lo = -step[a], hi = step[a];
      if (SPLIT) {
        const int odd = i0 & 1;
        lo = a == 0 ? (odd ? -hx : hx - 1) : (a == 1 ? -2 * hx : -2 * hx * L.ny);
        hi = a == 0 ? (odd ? 1 - hx : hx) : (a == 1 ? 2 * hx : 2 * hx * L.ny);
      }
      off[2 * n] = low_in ? lo : 0;
      off[2 * n + 1] = high_in ? hi : 0;
      keep[2 * n] = low_in || (!own_zero && ((L.neumann >> (2 * a)) & 1u));
      keep[2 * n + 1] = high_in || (!own_zero && ((L.neumann >> (2 * a + 1)) & 1u));
    }
    const T* lface;
    int lbase, lstride, lhigh;
    axis_faces(L, AXIS, i0, j0, k0, AXIS, lface, lbase, lstride, lhigh);
    end_low = __ldg(lface + lbase);
    end_high = __ldg(lface + lbase + (ext[AXIS] - 1) * lstride + lhigh);
    lkeep_low = (L.neumann >> (2 * AXIS)) & 1u;
    lkeep_high = (L.neumann >> (2 * AXIS + 1)) & 1u;
  }

  // Row s, c its vector index.  MODE kScanFresh: x is zero everywhere, so the
  // row is the rhs alone (every term is a finite face times zero).  ENDS: a
  // Neumann face at a line end may be nonzero; otherwise the end terms are exact
  // zeros and the cell's own x is not read.
  template <int MODE, bool ENDS>
  __device__ __forceinline__ T row(const T* x, const T* __restrict__ rhs, int c,
                                   int s, int extent) const {
    T d = __ldg(rhs + c);
    if (MODE == kScanFresh) return d;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int f = fbase[n] + s * fstride[n];
      const T lo = __ldg(x + c + off[2 * n]);
      const T hi = __ldg(x + c + off[2 * n + 1]);
      d += __ldg(face[n] + f) * (keep[2 * n] ? lo : T(0));
      d += __ldg(face[n] + f + fhigh[n]) * (keep[2 * n + 1] ? hi : T(0));
    }
    if (!ENDS) return d;
    const T self_value = MODE == kScanNormal ? x[c] : T(0);
    const T dl = d + end_low * (lkeep_low ? self_value : T(0));
    d = s == 0 ? dl : d;
    const T dh = d + end_high * (lkeep_high ? self_value : T(0));
    return s + 1 == extent ? dh : d;
  }
};

// ---------------------------------------------------------------------------
// Chunked-scan line solve.
//
// Each line's matrix is factorised once (full-line Thomas, in FP64): for row
// s, den_s = b_s - a_s c'_{s-1}, and the sweep needs
//   inv_s = 1 / den_s,   l_s = a_s / den_s,   u_s = c'_s = c_s / den_s.
// A sweep is then two first-order linear recurrences,
//   forward   y_s = d_s inv_s - l_s y_{s-1},
//   backward  x_s = y_s - u_s x_{s+1}.
// The line matrix is symmetric (a_s and c_{s-1} are the same face), so
// a_s / den_{s-1} = u_{s-1}, and the LDL^T form of the forward recurrence
//   z_s = d_s - u_{s-1} z_{s-1},   y_s = z_s inv_s
// needs no l array.  FP64 sweeps use it (one stream of 8 B per row less);
// FP32 sweeps keep the l array, because the extra load in the forward
// replay costs the FP32 kernel registers and occupancy.
// Each recurrence is an affine map per row.  A thread owns a chunk of up to
// ScanConfig<T>::rows consecutive rows of one line: it composes its chunk's
// maps, the chunks of a line combine their compositions through shared
// memory, and every thread replays its chunk from the incoming value.  No spike vectors or interface
// systems are stored, no division happens in a sweep, and the right-hand
// side of a chunk (the costly part: rhs, transverse faces and neighbours)
// stays in registers between the passes.
//
// Factor layout is colour-packed so that threads with consecutive line
// indices of one colour read consecutive addresses: array e (0 inv, then
// 1 u in the symmetric form, or 1 l and 2 u) of row s of colour line t sits at
//   ((e * 2 + colour) * extent + s) * colour_lines + t.

// Rows per chunk (held in registers) and the block-size bound, per
// precision: FP64 rows take twice the registers of FP32 rows.
// Measured on B200 at 256^3 (level-0 y-line colour pass): FP64 16 rows in
// blocks of <= 128 threads (8 lines x 16 chunks), FP32 8 rows in blocks of
// <= 512 threads (16 lines x 32 chunks).
#ifndef HFPS_SCAN_ROWS_F64
#define HFPS_SCAN_ROWS_F64 16
#endif
#ifndef HFPS_SCAN_THREADS_F64
#define HFPS_SCAN_THREADS_F64 128
#endif
#ifndef HFPS_SCAN_ROWS_F32
#define HFPS_SCAN_ROWS_F32 8
#endif
#ifndef HFPS_SCAN_THREADS_F32
#define HFPS_SCAN_THREADS_F32 512
#endif
template <class T>
struct ScanConfig;
template <>
struct ScanConfig<double> {
  static constexpr int rows = HFPS_SCAN_ROWS_F64;
  static constexpr int threads = HFPS_SCAN_THREADS_F64;
  static constexpr bool symmetric = true;
  static constexpr int arrays = 2;
};
// FP32 factors in the symmetric two-array form when HFPS_SCAN_SYM_F32 is 1.
#ifndef HFPS_SCAN_SYM_F32
#define HFPS_SCAN_SYM_F32 0
#endif
template <>
struct ScanConfig<float> {
  static constexpr int rows = HFPS_SCAN_ROWS_F32;
  static constexpr int threads = HFPS_SCAN_THREADS_F32;
  static constexpr bool symmetric = HFPS_SCAN_SYM_F32 != 0;
  static constexpr int arrays = symmetric ? 2 : 3;
};
// Longest line both precisions can solve: every chunk of a line lives in
// one block.
constexpr int kScanMaxExtent =
    HFPS_SCAN_ROWS_F64 * HFPS_SCAN_THREADS_F64 < HFPS_SCAN_ROWS_F32 * HFPS_SCAN_THREADS_F32
        ? HFPS_SCAN_ROWS_F64 * HFPS_SCAN_THREADS_F64
        : HFPS_SCAN_ROWS_F32 * HFPS_SCAN_THREADS_F32;

//
// x-lines (k_line_scan_x) keep a line's rows together instead, as their
// vectors do: ((e * 2 + colour) * colour_lines + t) * extent + s.
struct ScanLayout {
  int extent;
  int colour_lines;
  bool rows_together;
  __host__ __device__ size_t cell(int e, int colour, int s, int t) const {
    const size_t block = (static_cast<size_t>(e) * 2 + colour);
    return rows_together ? (block * colour_lines + t) * extent + s
                         : (block * extent + s) * colour_lines + t;
  }
  __host__ __device__ size_t values(int arrays) const {
    return static_cast<size_t>(arrays) * 2 * extent * colour_lines;
  }
};

// Thomas factors of every line, one thread per line, in FP64 whatever T is.
template <class T>
__global__ void k_scan_factors(Level<T> L, int axis, T* __restrict__ fac) {
  grid_dependency_sync();
  const int a_extent = axis == 0 ? L.ny : L.nx;
  const int b_extent = axis == 2 ? L.ny : L.nz;
  const int lines = a_extent * b_extent;
  const int extent = line_extent(axis, L.nx, L.ny, L.nz);
  const int ha = (a_extent + 1) >> 1;
  const ScanLayout lay{extent, ha * b_extent, axis == 0};
  for (int line = blockIdx.x * blockDim.x + threadIdx.x; line < lines;
       line += gridDim.x * blockDim.x) {
    const int fb = line / a_extent;
    const int fa = line - fb * a_extent;
    const int colour = (fa + fb) & 1;
    const int t = fb * ha + (fa >> 1);
    int base, stride;
    line_geometry(L, axis, fa, fb, base, stride);
    double prev_u = 0.0;
    for (int s = 0; s < extent; ++s) {
      const int c = base + s * stride;
      int i, j, k;
      line_cell(axis, fa, fb, s, i, j, k);
      T lowf, highf;
      line_faces(L, axis, c, j, k, lowf, highf);
      const double a = s == 0 ? 0.0 : -static_cast<double>(lowf);
      const double cc = s + 1 == extent ? 0.0 : -static_cast<double>(highf);
      const double den = static_cast<double>(L.diag[c]) - a * prev_u;
      const double u = cc / den;
      fac[lay.cell(0, colour, s, t)] = static_cast<T>(1.0 / den);
      if constexpr (ScanConfig<T>::symmetric) {
        fac[lay.cell(1, colour, s, t)] = static_cast<T>(u);
      } else {
        fac[lay.cell(1, colour, s, t)] = static_cast<T>(a / den);
        fac[lay.cell(2, colour, s, t)] = static_cast<T>(u);
      }
      prev_u = u;
    }
  }
}

// One zebra colour: blockDim = (LPB lines, S chunks), chunk q holds rows
// [q*m, min(extent, (q+1)*m) - 1] with m <= ScanConfig<T>::rows.  Shared memory holds
// the chunk compositions: forward (A, B) and backward (A, B), S x LPB each.
template <class T, int AXIS, int LPB, int MODE, bool SPLIT, bool ENDS>
__global__ void __launch_bounds__(ScanConfig<T>::threads)
    k_line_scan_color(Level<T> L, T* x, const T* __restrict__ rhs,
                      const T* __restrict__ fac, int color, int m, int hx, bool own_zero) {
  grid_dependency_sync();
  extern __shared__ unsigned char scan_smem[];
  const int S = blockDim.y;
  constexpr bool kSym = ScanConfig<T>::symmetric;
  constexpr int kScanRows = ScanConfig<T>::rows;
  T* fA = reinterpret_cast<T*>(scan_smem);
  T* fB = fA + S * LPB;
  T* bA = fB + S * LPB;
  T* bB = bA + S * LPB;
  const int extent = line_extent(AXIS, L.nx, L.ny, L.nz);
  const int a_extent = L.nx;
  const int b_extent = AXIS == 2 ? L.ny : L.nz;
  const int ha = (a_extent + 1) >> 1;
  const ScanLayout lay{extent, ha * b_extent, false};
  const int lane = threadIdx.x;
  const int q = threadIdx.y;
  const int t = blockIdx.x * LPB + lane;
  const int fb = t / ha;
  const int fa = 2 * (t - fb * ha) + ((fb + color) & 1);
  const bool valid = t < ha * b_extent && fa < a_extent;
  // Vector index of row 0 and its step per row (natural or split rows).
  int base = 0, stride = 0;
  if (valid) {
    line_geometry(L, AXIS, fa, fb, base, stride);
    if (SPLIT) {
      int i0, j0, k0;
      line_cell(AXIS, fa, fb, 0, i0, j0, k0);
      base = 2 * hx * (j0 + L.ny * k0) + (i0 & 1) * hx + (i0 >> 1);
      stride = AXIS == 1 ? 2 * hx : 2 * hx * L.ny;
    }
  }
  const int r0 = q * m;
  const int rows = valid ? max(0, min(m, extent - r0)) : 0;
  const int row = lay.colour_lines;
  const int tt = valid ? t : 0;
  const T* inv = fac + lay.cell(0, color, 0, tt);
  const T* lf = fac + lay.cell(1, color, 0, tt);
  const T* uf = fac + lay.cell(kSym ? 1 : 2, color, 0, tt);
  // Rows past the chunk's end (padding, and every row of an idle thread)
  // re-read the line's last row so that all loads are unconditional; their
  // values are never used.
  const auto srow = [&](int u) { return min(r0 + u, extent - 1); };
  // Forward multiplier of row s: u_{s-1} (zero on row 0), or l_s.
  const auto lower = [&](int u) -> T {
    const int s = srow(u);
    if constexpr (kSym) {
      const T g = __ldg(uf + max(s - 1, 0) * row);
      return s > 0 ? g : T(0);
    } else {
      return __ldg(lf + s * row);
    }
  };

  // Pass 1: right-hand sides (scaled by 1/den unless symmetric), and the
  // forward composition.
  const LineRhs<T, AXIS, SPLIT> lr(L, valid ? fa : 0, valid ? fb : 0, hx,
                                    MODE == kScanOwnZero || (!ENDS && own_zero));
  T v[kScanRows];
#pragma unroll
  for (int u = 0; u < kScanRows; ++u) {
    v[u] = lr.template row<MODE, ENDS>(x, rhs, base + srow(u) * stride, srow(u), extent);
    if constexpr (!kSym) v[u] = v[u] * __ldg(inv + srow(u) * row);
  }
  T A = T(1), B = T(0);
#pragma unroll
  for (int u = 0; u < kScanRows; ++u) {
    const T l = lower(u);
    const bool on = u < rows;
    B = on ? v[u] - l * B : B;
    A = on ? -l * A : A;
  }
  fA[q * LPB + lane] = A;
  fB[q * LPB + lane] = B;
  __syncthreads();
  // Forward replay from z_{r0-1} (y_{r0-1}); v becomes y.
  T z = T(0);
  for (int p = 0; p < q; ++p) z = fA[p * LPB + lane] * z + fB[p * LPB + lane];
#pragma unroll
  for (int u = 0; u < kScanRows; ++u) {
    z = v[u] - lower(u) * z;
    if constexpr (kSym) {
      v[u] = z * __ldg(inv + srow(u) * row);
    } else {
      v[u] = z;
    }
  }
  // Backward composition x_{r0} = A x_{r1+1} + B.
  A = T(1);
  B = T(0);
#pragma unroll
  for (int u = kScanRows - 1; u >= 0; --u) {
    const T uu = __ldg(uf + srow(u) * row);
    const bool on = u < rows;
    B = on ? v[u] - uu * B : B;
    A = on ? -uu * A : A;
  }
  bA[q * LPB + lane] = A;
  bB[q * LPB + lane] = B;
  __syncthreads();
  T xn = T(0);
  for (int p = S - 1; p > q; --p) xn = bA[p * LPB + lane] * xn + bB[p * LPB + lane];
#pragma unroll
  for (int u = kScanRows - 1; u >= 0; --u) {
    const T xv = v[u] - __ldg(uf + srow(u) * row) * xn;
    xn = u < rows ? xv : xn;
    if (u < rows) x[base + srow(u) * stride] = xn;
  }
}

// The same colour pass for x-lines, whose rows are contiguous.  Lanes across
// lines would touch a 32-byte sector per value (the pass took 155 us on
// 456x256x52 in FP64, 1.4 TB/s), so here a warp walks each line along its
// rows: the right-hand sides are formed coalesced and left in shared memory,
// the factors follow by asynchronous copies that hold no registers, each
// thread then scans its chunk of up to ScanConfig<T>::rows rows out of shared
// memory (chunks padded to an odd length, so that the lanes of a line fall in
// different banks), and the solution goes back coalesced: 75 us, 2.9 TB/s of
// the 36 bytes per cell that a pass needs (the transverse faces are 16 of them,
// the factors 8).  A FP64 block of some 1280 rows takes 35 KB of shared memory,
// so that six blocks per SM overlap their load and scan phases; what bounds
// it now is the rest of that overlap.  Chunks, compositions and their
// order are k_line_scan_color's, so the results are bit for bit its results.
constexpr int kScanXThreads = 128;

template <class T>
__device__ __forceinline__ void copy_async(T* shared, const T* global) {
  const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(shared));
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(global),
               "n"(sizeof(T)));
}

struct ScanXShape {
  int lines;        // per block
  int chunks, rows; // per line, per chunk
  int pitch;        // shared-memory stride of a chunk
};

// PARTS: a block has at most half as many lines as warps (long lines), and
// several warps take a part each of a line in the load and store phases.  With a
// warp per line whatever the block held, one warp of eight loaded 1030 FP32 rows
// while the others waited (with the threads trimmed to the chunks, level-0 passes in
// FP32: 700x140x140 206 -> 110 us, 1030x120x120 357 -> 128, 2048x90x90 372 -> 149;
// FP64: 1030x120x120 370 -> 168, 2048x90x90 469 -> 189).  Shorter lines keep the
// plain form, which the parts' bounds slow down (300x200x200 FP32 87 -> 105).
template <class T, bool PARTS>
__global__ void __launch_bounds__(kScanXThreads * (sizeof(T) == 4 ? 2 : 1))
    k_line_scan_x(Level<T> L, T* x, const T* __restrict__ rhs, const T* __restrict__ fac,
                  int color, ScanXShape sh) {
  grid_dependency_sync();
  extern __shared__ unsigned char scan_x_smem[];
  constexpr bool kSym = ScanConfig<T>::symmetric;
  constexpr int kScanRows = ScanConfig<T>::rows;
  const int extent = L.nx;
  const int ha = (L.ny + 1) >> 1;
  const ScanLayout lay{extent, ha * L.nz, true};
  const int m = sh.rows, S = sh.chunks;
  const int line_pitch = S * sh.pitch;
  const int span = sh.lines * line_pitch;
  T* d = reinterpret_cast<T*>(scan_x_smem);
  T* inv = d + span;
  T* up = inv + span;
  T* low = kSym ? up : up + span;
  T* fA = low + span;
  T* fB = fA + sh.lines * S;
  T* bA = fB + sh.lines * S;
  T* bB = bA + sh.lines * S;
  // s / m for s < 2048 and m <= 16.
  const unsigned reciprocal = (65536u + m - 1) / m;
  const auto place = [&](int s) {
    const int q = static_cast<int>((static_cast<unsigned>(s) * reciprocal) >> 16);
    return q * sh.pitch + (s - q * m);
  };
  const int t0 = blockIdx.x * sh.lines;
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5, lane = threadIdx.x & 31;
  // A line's index in its colour, or false past the colour's lines.
  const auto locate = [&](int t, int& fa, int& fb) {
    fb = t / ha;
    fa = 2 * (t - fb * ha) + ((fb + color) & 1);
    return t < ha * L.nz && fa < L.ny;
  };
  // A warp's lines, and its rows of them.
  const int share = PARTS ? max(1, warps / sh.lines) : 1;
  const int first = PARTS ? warp / share : warp, next = PARTS ? warps / share : warps;
  const int part = PARTS ? (extent + 32 * share - 1) / (32 * share) * 32 : 0;
  const int row0 = PARTS ? (warp - first * share) * part + lane : lane;
  const int row1 = PARTS ? min(extent, row0 - lane + part) : extent;
  for (int l = first; l < sh.lines; l += next) {
    int fa, fb;
    if (!locate(t0 + l, fa, fb)) continue;
    const T* finv = fac + lay.cell(0, color, 0, t0 + l);
    const T* flow = fac + lay.cell(1, color, 0, t0 + l);
    const T* fup = fac + lay.cell(kSym ? 1 : 2, color, 0, t0 + l);
    for (int s = row0; s < row1; s += 32) {
      const int at = l * line_pitch + place(s);
      copy_async(inv + at, finv + s);
      copy_async(up + at, fup + s);
      if constexpr (!kSym) copy_async(low + at, flow + s);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int l = first; l < sh.lines; l += next) {
    int fa, fb;
    if (!locate(t0 + l, fa, fb)) continue;
    const LineRhs<T, 0, false> lr(L, fa, fb, 0);
    const int base = L.nx * (fa + L.ny * fb);
    // Eight rows in flight in FP32 (97x201x55 MG application 800 -> 686 us); in
    // FP64 their registers cost more than they give (13.0 -> 14.4 us a pass).
    constexpr int kInFlight = sizeof(T) == 4 ? 8 : 4;
#pragma unroll kInFlight
    for (int s = row0; s < row1; s += 32) {
      const int c = base + s;
      T v = __ldg(rhs + c);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int f = lr.fbase[n] + s * lr.fstride[n];
        const T lo = __ldg(x + c + lr.off[2 * n]);
        const T hi = __ldg(x + c + lr.off[2 * n + 1]);
        v += __ldg(lr.face[n] + f) * (lr.keep[2 * n] ? lo : T(0));
        v += __ldg(lr.face[n] + f + lr.fhigh[n]) * (lr.keep[2 * n + 1] ? hi : T(0));
      }
      if (s == 0) v += lr.end_low * (lr.lkeep_low ? x[c] : T(0));
      if (s + 1 == extent) v += lr.end_high * (lr.lkeep_high ? x[c] : T(0));
      d[l * line_pitch + place(s)] = v;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int l = threadIdx.x / S, q = threadIdx.x - l * S;
  int fa, fb;
  const bool valid = l < sh.lines && locate(t0 + l, fa, fb);
  const int rows = valid ? max(0, min(m, extent - q * m)) : 0;
  const int at = valid ? l * line_pitch + q * sh.pitch : 0;
  const int slot = valid ? l * S + q : 0;
  // Forward multiplier of row u of the chunk: u_{s-1} (zero on row 0), or l_s.
  const auto lower = [&](int u) -> T {
    if constexpr (kSym) {
      if (u > 0) return up[at + u - 1];
      return q > 0 ? up[at - sh.pitch + m - 1] : T(0);
    } else {
      return low[at + u];
    }
  };
  T v[kScanRows];
  T A = T(1), B = T(0);
#pragma unroll
  for (int u = 0; u < kScanRows; ++u) {
    if (u < rows) {
      v[u] = d[at + u];
      if constexpr (!kSym) v[u] = v[u] * inv[at + u];
      const T f = lower(u);
      B = v[u] - f * B;
      A = -f * A;
    }
  }
  if (valid) {
    fA[slot] = A;
    fB[slot] = B;
  }
  __syncthreads();
  T z = T(0);
  if (valid)
    for (int p = 0; p < q; ++p) z = fA[slot - q + p] * z + fB[slot - q + p];
#pragma unroll
  for (int u = 0; u < kScanRows; ++u) {
    if (u < rows) {
      z = v[u] - lower(u) * z;
      if constexpr (kSym) v[u] = z * inv[at + u];
      else v[u] = z;
    }
  }
  A = T(1);
  B = T(0);
#pragma unroll
  for (int u = kScanRows - 1; u >= 0; --u) {
    if (u < rows) {
      const T f = up[at + u];
      B = v[u] - f * B;
      A = -f * A;
    }
  }
  if (valid) {
    bA[slot] = A;
    bB[slot] = B;
  }
  __syncthreads();
  T xn = T(0);
  if (valid)
    for (int p = S - 1; p > q; --p) xn = bA[slot - q + p] * xn + bB[slot - q + p];
#pragma unroll
  for (int u = kScanRows - 1; u >= 0; --u) {
    if (u < rows) {
      xn = v[u] - up[at + u] * xn;
      d[at + u] = xn;
    }
  }
  __syncthreads();
  for (int k = first; k < sh.lines; k += next) {
    if (!locate(t0 + k, fa, fb)) continue;
    T* out = x + L.nx * (fa + L.ny * fb);
    for (int s = row0; s < row1; s += 32) out[s] = d[k * line_pitch + place(s)];
  }
}

// ---------------------------------------------------------------------------
// PCR elimination factors of every line: per halving step the multipliers
// k1 = a_s / b_{s-h}, k2 = c_s / b_{s+h}, then the final diagonal.  Layout
// [2*steps+1][lines][P] so a line's threads read consecutive addresses.
template <class T>
__global__ void __launch_bounds__(1024) k_pcr_factors(Level<T> L, int axis, int P, T* __restrict__ fac) {
  grid_dependency_sync();
  extern __shared__ unsigned char pcr_factor_smem[];
  T* sa = reinterpret_cast<T*>(pcr_factor_smem) + threadIdx.y * 3 * P;
  T* sb = sa + P;
  T* sc = sb + P;
  const int a_extent = axis == 0 ? L.ny : L.nx;
  const int b_extent = axis == 2 ? L.ny : L.nz;
  const int lines = a_extent * b_extent;
  const int extent = line_extent(axis, L.nx, L.ny, L.nz);
  const int line = blockIdx.x * blockDim.y + threadIdx.y;
  const bool valid = line < lines;
  const int fb = valid ? line / a_extent : 0;
  const int fa = valid ? line - fb * a_extent : 0;
  const int s = threadIdx.x;
  T a = T(0), bb = T(1), cc = T(0);
  if (valid && s < extent) {
    int i, j, k;
    line_cell(axis, fa, fb, s, i, j, k);
    const int c = i + L.nx * (j + L.ny * k);
    T lowf, highf;
    line_faces(L, axis, c, j, k, lowf, highf);
    a = s == 0 ? T(0) : -lowf;
    bb = L.diag[c];
    cc = s + 1 == extent ? T(0) : -highf;
  }
  sa[s] = a;
  sb[s] = bb;
  sc[s] = cc;
  __syncthreads();
  const size_t slab = static_cast<size_t>(lines) * P;
  const size_t at = static_cast<size_t>(valid ? line : 0) * P + s;
  int step = 0;
  for (int h = 1; h < P; h <<= 1, ++step) {
    const int lo = s - h, hi = s + h;
    const T as = sa[s], bs = sb[s], cs = sc[s];
    T k1 = T(0), k2 = T(0), alo = T(0), clo = T(0), ahi = T(0), chi = T(0);
    if (lo >= 0) {
      k1 = as / sb[lo];
      alo = sa[lo];
      clo = sc[lo];
    }
    if (hi < P) {
      k2 = cs / sb[hi];
      ahi = sa[hi];
      chi = sc[hi];
    }
    const T na = -alo * k1;
    const T nc = -chi * k2;
    const T nb = bs - clo * k1 - ahi * k2;
    if (valid) {
      fac[(2 * step) * slab + at] = k1;
      fac[(2 * step + 1) * slab + at] = k2;
    }
    __syncthreads();
    sa[s] = na;
    sb[s] = nb;
    sc[s] = nc;
    __syncthreads();
  }
  if (valid) fac[(2 * step) * slab + at] = sb[s];
}

// One zebra colour with PCR: blockDim = (P, lines per block), P = 2^STEPS.
template <class T, int STEPS>
__global__ void __launch_bounds__(1024) k_line_pcr_factored_color(Level<T> L, T* __restrict__ x,
                                          const T* __restrict__ rhs,
                                          const T* __restrict__ fac, int axis,
                                          int color) {
  grid_dependency_sync();
  extern __shared__ unsigned char pcr_rhs_smem[];
  T* sd = reinterpret_cast<T*>(pcr_rhs_smem) + threadIdx.y * (2 << STEPS);
  pcr_line_slot<T, STEPS>(L, x, rhs, fac, axis, color, blockIdx.x * blockDim.y + threadIdx.y,
                          threadIdx.x, sd, [] {});
}

// All colour passes of one axis of a small level in one launch: a cluster of up
// to 8 CTAs holds a colour's lines at once, and a cluster barrier stands where
// separate passes have a launch.  The next pass's factors are loaded ahead of the
// barrier.  Bound by latency, a pass being one round of L2 loads, the exchanges
// and the barrier: visits of 60 lines of 16 rows 9.5 -> 7.4 us, of 32 lines of
// 32 rows 9.5 -> 8.0, of 8 lines of 256 rows 9.5 -> 8.8 (2 and 4 passes,
// averaged), each with two fewer gaps of 0.7 us; 456x256x52 step 105.2 -> 103.5
// ms, wrinkled 256^3 MG application 2769 -> 2726 us (both under the profiler).
template <class T, int STEPS>
__global__ void __launch_bounds__(256)
    k_line_pcr_sweeps(Level<T> L, T* x, const T* rhs, const T* __restrict__ fac, int axis,
                      int first, int passes) {
  extern __shared__ unsigned char pcr_rhs_smem[];
  T* sd = reinterpret_cast<T*>(pcr_rhs_smem) + threadIdx.y * (2 << STEPS);
  for (int pass = 0; pass < passes; ++pass) {
    pcr_line_slot<T, STEPS>(L, x, rhs, fac, axis, (first + pass) & 1,
                            blockIdx.x * blockDim.y + threadIdx.y, threadIdx.x, sd, [&] {
                              if (pass == 0) grid_dependency_sync();
                              else asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
                            });
    if (pass + 1 < passes) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  }
}

// One zebra colour pass of the coarsest-level kernel for the lines handled
// by this thread row (factors already in registers).  One CTA that solves a level
// spends a pass on the latency of its factors and faces from L2, and which exchange
// is faster depends on the rows: pcr_apply's where they fill the threads of a line
// (ONE_BARRIER; MG application with two barriers a step, then with one: 32x72x72 2551
// and 2367 us, 256x48x48 1544 and 1498), two barriers a step where some threads hold
// no row (31x72x72 2591 and 2837, 60x60x40 1335 and 1420, 240x40x40 1557 and 1570,
// 257x48x48 2858 and 2959).  The CTAs that build the dense map's columns hide the
// latency and take pcr_apply's (update of 200x40x40 7.02 -> 6.74 ms).
template <class TC, int STEPS, bool ONE_BARRIER>
__device__ __forceinline__ void coarse_line_pass(const Level<TC>& L, TC* xs,
                                                 const TC* bs, TC* sd, int axis,
                                                 int fa, int fb, bool valid,
                                                 int c, int s, int extent,
                                                 const PcrRow<TC, STEPS>& r) {
  TC d = TC(0);
  if (valid && s < extent) d = line_rhs_any(L, xs, bs, axis, fa, fb, s, extent, c);
  TC value;
  if constexpr (ONE_BARRIER) {
    value = pcr_apply(r, sd, s, d);
  } else {
    constexpr int P = 1 << STEPS;
    sd[s] = d;
    __syncthreads();
#pragma unroll
    for (int step = 0; step < STEPS; ++step) {
      const int lo = s - (1 << step), hi = s + (1 << step);
      const TC dlo = lo >= 0 ? sd[lo] : TC(0);
      const TC dhi = hi < P ? sd[hi] : TC(0);
      const TC next = sd[s] - dlo * r.k[2 * step] - dhi * r.k[2 * step + 1];
      __syncthreads();
      sd[s] = next;
      __syncthreads();
    }
    value = sd[s] / r.k[2 * STEPS];
  }
  if (valid && s < extent) xs[c] = value;
  __syncthreads();
}

// Coarsest level, line mode: all sweeps in one CTA with x and rhs resident
// in shared memory (widened to TC).  When each colour's lines fit the CTA's
// thread rows, both colours' PCR factors stay in registers for all sweeps.
//
// COLUMNS: with kCoarseColumns, block j instead starts from unit data, x = e_j and
// b = 0 for j < n, x = 0 and b = e_{j-n} for j >= n, and writes its result
// to x + j*n: the columns of the affine map x_out = P x_in + M b that the
// sweeps apply (coarse_dense_operator).  kCoarseColumnsOn starts from the
// column that is there, with the same b.
template <class T, class TC, int STEPS, bool COLUMNS, bool ONE_BARRIER>
__global__ void __launch_bounds__(512)
    k_coarse_line_smem(Level<TC> L, T* __restrict__ x, const T* __restrict__ b,
                       const TC* __restrict__ fac, int sweeps, int axis,
                       int columns) {
  grid_dependency_sync();
  constexpr int P = 1 << STEPS;
  extern __shared__ unsigned char coarse_smem[];
  const int n = L.nx * L.ny * L.nz;
  TC* xs = reinterpret_cast<TC*>(coarse_smem);
  TC* bs = xs + n;
  TC* sd = bs + n + threadIdx.y * 2 * P;
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int nthreads = blockDim.x * blockDim.y;
  if (COLUMNS) {
    const int j = blockIdx.x;
    x += static_cast<size_t>(j) * n;
    for (int c = tid; c < n; c += nthreads) {
      xs[c] = columns == kCoarseColumnsOn ? static_cast<TC>(x[c])
                                          : ((j < n && c == j) ? TC(1) : TC(0));
      bs[c] = (j >= n && c == j - n) ? TC(1) : TC(0);
    }
  } else {
    for (int c = tid; c < n; c += nthreads) {
      xs[c] = static_cast<TC>(x[c]);
      bs[c] = static_cast<TC>(b[c]);
    }
  }
  __syncthreads();
  const int extent = line_extent(axis, L.nx, L.ny, L.nz);
  const int a_extent = axis == 0 ? L.ny : L.nx;
  const int b_extent = axis == 2 ? L.ny : L.nz;
  const int ha = (a_extent + 1) >> 1;
  const int lines = ha * b_extent;
  const size_t slab = static_cast<size_t>(a_extent) * b_extent * P;
  const int s = threadIdx.x;
  const auto locate = [&](int t, int color, int& fa, int& fb, bool& valid, int& c,
                          size_t& at) {
    fb = t / ha;
    fa = 2 * (t - fb * ha) + ((fb + color) & 1);
    valid = t < lines && fa < a_extent;
    at = static_cast<size_t>(valid ? fa + a_extent * fb : 0) * P + s;
    c = 0;
    if (valid && s < extent) {
      int i, j, k;
      line_cell(axis, fa, fb, s, i, j, k);
      c = i + L.nx * (j + L.ny * k);
    }
  };
  if (lines <= static_cast<int>(blockDim.y)) {
    int fa0, fb0, c0, fa1, fb1, c1;
    bool v0, v1;
    size_t at0, at1;
    locate(threadIdx.y, 0, fa0, fb0, v0, c0, at0);
    locate(threadIdx.y, 1, fa1, fb1, v1, c1, at1);
    PcrRow<TC, STEPS> r0, r1;
    pcr_load(fac, slab, at0, r0);
    pcr_load(fac, slab, at1, r1);
    for (int sweep = 0; sweep < sweeps; ++sweep) {
      coarse_line_pass<TC, STEPS, ONE_BARRIER>(L, xs, bs, sd, axis, fa0, fb0, v0, c0, s, extent,
                                               r0);
      coarse_line_pass<TC, STEPS, ONE_BARRIER>(L, xs, bs, sd, axis, fa1, fb1, v1, c1, s, extent,
                                               r1);
    }
  } else {
    for (int sweep = 0; sweep < sweeps; ++sweep) {
      for (int color = 0; color < 2; ++color) {
        for (int base = 0; base < lines; base += blockDim.y) {
          int fa, fb, c;
          bool valid;
          size_t at;
          locate(base + threadIdx.y, color, fa, fb, valid, c, at);
          PcrRow<TC, STEPS> r;
          pcr_load(fac, slab, at, r);
          coarse_line_pass<TC, STEPS, ONE_BARRIER>(L, xs, bs, sd, axis, fa, fb, valid, c, s,
                                                   extent, r);
        }
      }
    }
  }
  for (int c = tid; c < n; c += nthreads) x[c] = static_cast<T>(xs[c]);
}

// Lines per PCR block.  One line per block (P threads) spreads a colour's
// few lines over as many SMs and keeps each step's barrier to P threads:
// measured on B200 at 256^3, one MG application 3.42 ms with 4 lines per
// block, 3.18 with 2, 3.08 with 1.
#ifndef HFPS_PCR_LINES
#define HFPS_PCR_LINES 1
#endif
void pcr_shape(int extent, int& P, int& lines_per_block, int& steps) {
  P = 1;
  steps = 0;
  while (P < extent) {
    P <<= 1;
    ++steps;
  }
  lines_per_block = std::max(1, std::min(1024 / P, HFPS_PCR_LINES));
}

// Lines per block and chunks per line of the scan kernel: at least 296
// blocks (two per SM) where the level allows, at most ScanConfig<T>::threads
// threads, at least 8 lines per block while that still allows chunks of at
// most ScanConfig<T>::rows rows.
struct ScanShape {
  int lpb, chunks, rows;
};

// Lines per block are halved (down to HFPS_SCAN_MIN_LPB) while a colour has
// fewer than two blocks per SM.
#ifndef HFPS_SCAN_MIN_LPB
#define HFPS_SCAN_MIN_LPB 8
#endif
template <class T>
ScanShape scan_shape(long long per_color, int extent) {
  constexpr int rows = ScanConfig<T>::rows;
  ScanShape sh{32, (extent + rows - 1) / rows, 0};
  while (sh.lpb > HFPS_SCAN_MIN_LPB && per_color < 296LL * sh.lpb) sh.lpb >>= 1;
  while (sh.lpb > 1 && sh.lpb * sh.chunks > ScanConfig<T>::threads) sh.lpb >>= 1;
  sh.rows = (extent + sh.chunks - 1) / sh.chunks;
  return sh;
}

// Without end terms the FP64 kernel needs 128 registers instead of 165: 16 resident
// warps per SM, not 12.  Along y that pays where the colour's blocks then take fewer
// waves (level-0 pass of 256^3 142 -> 123 us, 128x256x128 42 -> 36, 128^3 15.5 ->
// 10.8, 250x140x200 78 -> 70) and costs a little where they do not (128x192x128 29.1
// -> 30.2 us, 131x160x133 27.0 -> 27.9, 64x256x64 7.7 -> 8.0).  Along z it gained in
// one of seventeen shapes (256^3 162 either way, 128x256x256 76 -> 81, 256x256x160 96
// -> 100), and in natural order the half-used sectors of the fourth block cost more
// than it gives (456x256x52 y-lines 65.6 -> 71 us).  Those keep the kernel with the
// end terms, which are exact zeros then.  FP32 has 64 registers and two blocks per SM
// either way, and its level-0 pass is slower without them (94.5 -> 100.3 us).  A fresh
// pass reads nothing but rhs in either form.
struct ScanFlags {
  int hx;
  bool zero_other, zero_self, ends;
};

template <class T, int AXIS, int LPB>
void launch_scan(cudaStream_t s, const Level<T>& L, T* x, const T* b, const T* fac,
                 int color, long long per_color, const ScanShape& sh, ScanFlags f) {
  const int blocks = static_cast<int>((per_color + LPB - 1) / LPB);
  const size_t smem = static_cast<size_t>(4) * sh.chunks * LPB * sizeof(T);
  const dim3 block(LPB, sh.chunks);
  const bool split = f.hx != 0;
  const auto run = [&](auto kernel) {
    launch(kernel, blocks, block, smem, s, L, x, b, fac, color, sh.rows, f.hx, f.zero_self);
  };
  // The kernel without end terms takes the zero flag as an argument (a kernel of
  // its own takes more registers); with them it is a mode.
  if constexpr (sizeof(T) == 8 && AXIS == 1) {
    const int warps = (LPB * sh.chunks + 31) / 32;
    const int resident = 148 * (12 / warps), resident_none = 148 * (16 / warps);
    const bool fewer_waves =
        (blocks + resident_none - 1) / resident_none < (blocks + resident - 1) / resident;
    if (!f.ends && split && fewer_waves && !(f.zero_other && f.zero_self)) {
      run(k_line_scan_color<T, AXIS, LPB, kScanNormal, true, false>);
      return;
    }
  }
  if (f.zero_other && f.zero_self) {
    if (split) run(k_line_scan_color<T, AXIS, LPB, kScanFresh, true, true>);
    else run(k_line_scan_color<T, AXIS, LPB, kScanFresh, false, true>);
  } else if (f.zero_self) {
    if (split) run(k_line_scan_color<T, AXIS, LPB, kScanOwnZero, true, true>);
    else run(k_line_scan_color<T, AXIS, LPB, kScanOwnZero, false, true>);
  } else {
    if (split) run(k_line_scan_color<T, AXIS, LPB, kScanNormal, true, true>);
    else run(k_line_scan_color<T, AXIS, LPB, kScanNormal, false, true>);
  }
}

// As many lines per block as its threads have chunks for, halved (down to one
// per warp of the load phase) while that leaves fewer than four blocks per SM:
// with 42 lines of 40 cells per block a level of 1024 lines ran on 25 SMs.
template <class T>
void launch_scan_x(cudaStream_t s, const Level<T>& L, T* x, const T* b, const T* fac, int color,
                   long long per_color) {
  constexpr int rows = ScanConfig<T>::rows;
  constexpr int threads = kScanXThreads * (sizeof(T) == 4 ? 2 : 1);
  ScanXShape sh{};
  sh.chunks = (L.nx + rows - 1) / rows;
  sh.rows = (L.nx + sh.chunks - 1) / sh.chunks;
  sh.pitch = sh.rows | 1;
  // FP64 blocks of more than about 80 chunks take so much shared memory that the few
  // of them on an SM leave loads waiting for scans (110x243x107 69 us a pass, 51 before
  // the x scan; 47 so).  Lines of up to 3 chunks want the threads for their loads
  // (24x300x300 34 and 42 us), those of more than 32 the lines (520x160x160 159 and 185).
  const int most = sizeof(T) == 8 && sh.chunks > 3 && sh.chunks <= 32 ? 80 : threads;
  sh.lines = std::max(1, most / sh.chunks);
  while (sh.lines > threads / 32 && per_color < 592LL * sh.lines)
    sh.lines = std::max(threads / 32, sh.lines / 2);
  // A multiple of the warps, or some load a line more than the others (213x168x138 with
  // 9 and 8 lines a block 88 and 71 us, FP32 52 and 37; 300x200x200 with 6 and 4 175 and
  // 123); two a warp rather than one where they fit (40x80x80 with 5, 4 and 8 lines 7.9,
  // 9.3 and 7.2).  FP32 blocks lose from fewer lines unless the last round was mostly
  // empty (138x175x163 with 14 and 8 lines 26.4 and 30.2, 100x150x150 with 19 and 16
  // 17.8 and 19.1).
  constexpr int warps = threads / 32;
  if (sizeof(T) == 8 && sh.lines > warps) {
    if (sh.lines >= 2 * warps) sh.lines = sh.lines / warps * warps;
    else sh.lines = 2 * warps * sh.chunks <= most + 8 ? 2 * warps : warps;
  } else if (sh.lines > warps) {
    const int nearest = (sh.lines + warps / 2) / warps * warps;
    const int lines = nearest * sh.chunks <= most ? nearest : sh.lines / warps * warps;
    const int rounds = (sh.lines + warps - 1) / warps;
    const bool uneven = 5 * rounds * warps >= 7 * sh.lines;
    if (uneven ? 3 * lines >= 2 * sh.lines : 10 * lines >= 9 * sh.lines) sh.lines = lines;
  }
  constexpr size_t arrays = 1 + ScanConfig<T>::arrays;
  const size_t smem =
      static_cast<size_t>(sh.lines) * sh.chunks * (arrays * sh.pitch + 4) * sizeof(T);
  const size_t largest = threads * (arrays * (rows | 1) + 4) * sizeof(T);
  // Threads for the chunks, and a warp per line to load with: 1030 FP32 rows are
  // 129 chunks, and of a block of 256 threads half would only hold registers.
  const int used =
      std::min(threads, std::max((sh.lines * sh.chunks + 31) / 32 * 32, 32 * sh.lines));
  const auto run = [&](auto kernel) {
    allow_shared(kernel, smem, largest);
    launch(kernel, static_cast<int>((per_color + sh.lines - 1) / sh.lines), used, smem, s, L, x, b,
           fac, color, sh);
  };
  if (2 * 32 * sh.lines <= used) run(k_line_scan_x<T, true>);
  else run(k_line_scan_x<T, false>);
}

template <class T, int AXIS>
void launch_scan_axis(cudaStream_t s, const Level<T>& L, T* x, const T* b, const T* fac,
                      int color, long long per_color, const ScanShape& sh, ScanFlags f) {
  switch (sh.lpb) {
    case 32: launch_scan<T, AXIS, 32>(s, L, x, b, fac, color, per_color, sh, f); break;
    case 16: launch_scan<T, AXIS, 16>(s, L, x, b, fac, color, per_color, sh, f); break;
    case 8: launch_scan<T, AXIS, 8>(s, L, x, b, fac, color, per_color, sh, f); break;
    case 4: launch_scan<T, AXIS, 4>(s, L, x, b, fac, color, per_color, sh, f); break;
    case 2: launch_scan<T, AXIS, 2>(s, L, x, b, fac, color, per_color, sh, f); break;
    default: launch_scan<T, AXIS, 1>(s, L, x, b, fac, color, per_color, sh, f); break;
  }
}

}  // namespace

int line_kind(int nx, int ny, int nz, int axis) {
  const int extent = line_extent(axis, nx, ny, nz);
  const int a_extent = axis == 0 ? ny : nx;
  const int b_extent = axis == 2 ? ny : nz;
  const long long per_color = static_cast<long long>((a_extent + 1) / 2) * b_extent;
  const long long threshold =
      extent >= kLinePcrLongExtent ? kLinePcrThresholdLong : kLinePcrThreshold;
  if (per_color < threshold && extent <= 1024) return kLinePcr;
  return extent <= kScanMaxExtent ? kLineScan : kLineNone;
}

template <class T>
size_t line_factor_values(int nx, int ny, int nz, int axis) {
  const int extent = line_extent(axis, nx, ny, nz);
  const int a_extent = axis == 0 ? ny : nx;
  const int b_extent = axis == 2 ? ny : nz;
  const size_t lines = static_cast<size_t>(a_extent) * b_extent;
  const int kind = line_kind(nx, ny, nz, axis);
  if (kind == kLineNone) return 0;
  if (kind == kLineScan)
    return ScanLayout{extent, ((a_extent + 1) / 2) * b_extent, axis == 0}.values(ScanConfig<T>::arrays);
  int P, lpb, steps;
  pcr_shape(extent, P, lpb, steps);
  return static_cast<size_t>(2 * steps + 1) * lines * P;
}

template <class T>
void launch_line_factors(cudaStream_t s, const Level<T>& L, int axis, T* fac) {
  const int extent = line_extent(axis, L.nx, L.ny, L.nz);
  const int a_extent = axis == 0 ? L.ny : L.nx;
  const int b_extent = axis == 2 ? L.ny : L.nz;
  const int lines = a_extent * b_extent;
  const int kind = line_kind(L.nx, L.ny, L.nz, axis);
  if (kind == kLineNone) return;
  if (kind == kLineScan) {
    launch(k_scan_factors<T>, (lines + 127) / 128, 128, 0, s, L, axis, fac);
    return;
  }
  int P, lpb, steps;
  pcr_shape(extent, P, lpb, steps);
  const size_t smem = static_cast<size_t>(3) * P * lpb * sizeof(T);
  launch(k_pcr_factors<T>, (lines + lpb - 1) / lpb, dim3(P, lpb), smem, s, L, axis, P, fac);
}

template <class T>
void launch_line_pass(cudaStream_t s, const Level<T>& L, T* x, const T* b,
                      const T* fac, T* scratch, int axis, int color, int hx,
                      bool zero_other, bool zero_self, bool ends) {
  (void)scratch;
  const int extent = line_extent(axis, L.nx, L.ny, L.nz);
  const int a_extent = axis == 0 ? L.ny : L.nx;
  const int b_extent = axis == 2 ? L.ny : L.nz;
  const long long per_color = static_cast<long long>((a_extent + 1) / 2) * b_extent;
  const int kind = line_kind(L.nx, L.ny, L.nz, axis);
  if (kind == kLineNone) return;
  if (kind == kLineScan) {
    if (axis == 0) {
      launch_scan_x<T>(s, L, x, b, fac, color, per_color);
      return;
    }
    const ScanShape sh = scan_shape<T>(per_color, extent);
    const ScanFlags f{hx, zero_other, zero_self, ends};
    if (axis == 1) launch_scan_axis<T, 1>(s, L, x, b, fac, color, per_color, sh, f);
    else launch_scan_axis<T, 2>(s, L, x, b, fac, color, per_color, sh, f);
    return;
  }
  int P, lpb, steps;
  pcr_shape(extent, P, lpb, steps);
  const size_t smem = static_cast<size_t>(2) * P * lpb * sizeof(T);
  const int blocks = static_cast<int>((per_color + lpb - 1) / lpb);
  const dim3 block(P, lpb);
  switch (steps) {
#define HFPS_PCR_CASE(N)                                                        \
  case N:                                                                       \
    launch(k_line_pcr_factored_color<T, N>, blocks, block, smem, s, L, x, b, fac, axis, \
                                                                 color);        \
    break;
    HFPS_PCR_CASE(0) HFPS_PCR_CASE(1) HFPS_PCR_CASE(2) HFPS_PCR_CASE(3) HFPS_PCR_CASE(4)
    HFPS_PCR_CASE(5) HFPS_PCR_CASE(6) HFPS_PCR_CASE(7) HFPS_PCR_CASE(8) HFPS_PCR_CASE(9)
    HFPS_PCR_CASE(10)
#undef HFPS_PCR_CASE
    default: break;
  }
}

// Where a colour's rows fit 8 CTAs of at most 256 threads, few threads per CTA
// first: 512 rows per CTA lose what the launches cost (112 lines of 64 rows 3 x
// 3.5 -> 9.6 us on 16 CTAs, 12.3 on 8 of 1024 threads), and so do several rounds.
constexpr int kSweepCtas = 8, kSweepMinThreads = 64, kSweepMaxThreads = 256;

template <class T>
bool launch_line_sweeps(cudaStream_t s, const Level<T>& L, T* x, const T* b, const T* fac,
                        int axis, int first, int passes) {
  if (line_kind(L.nx, L.ny, L.nz, axis) != kLinePcr) return false;
  const int extent = line_extent(axis, L.nx, L.ny, L.nz);
  const int a_extent = axis == 0 ? L.ny : L.nx;
  const int b_extent = axis == 2 ? L.ny : L.nz;
  const long long per_color = static_cast<long long>((a_extent + 1) / 2) * b_extent;
  int P, lpb, steps;
  pcr_shape(extent, P, lpb, steps);
  int threads = kSweepMinThreads;
  while (threads < kSweepMaxThreads && kSweepCtas * static_cast<long long>(threads / P) < per_color)
    threads *= 2;
  lpb = threads / P;
  if (kSweepCtas * static_cast<long long>(lpb) < per_color) return false;
  int ctas = 1;
  while (ctas * lpb < per_color) ctas *= 2;
  const size_t smem = static_cast<size_t>(2) * P * lpb * sizeof(T);
  switch (steps) {
#define HFPS_SWEEPS_CASE(N)                                                                   \
  case N:                                                                                     \
    launch_cluster(k_line_pcr_sweeps<T, N>, ctas, dim3(P, lpb), smem, s, L, x, b, fac, axis, \
                   first, passes);                                                           \
    return true;
    HFPS_SWEEPS_CASE(0) HFPS_SWEEPS_CASE(1) HFPS_SWEEPS_CASE(2) HFPS_SWEEPS_CASE(3)
    HFPS_SWEEPS_CASE(4) HFPS_SWEEPS_CASE(5) HFPS_SWEEPS_CASE(6) HFPS_SWEEPS_CASE(7)
    HFPS_SWEEPS_CASE(8)
#undef HFPS_SWEEPS_CASE
    default: return false;
  }
}

template <class T, class TC>
bool launch_coarse_line(cudaStream_t s, const Level<TC>& L, T* x, const T* b,
                        const TC* fac, int sweeps, int axis, int columns) {
  const int extent = line_extent(axis, L.nx, L.ny, L.nz);
  if (line_kind(L.nx, L.ny, L.nz, axis) != kLinePcr) return false;
  int P, lpb, steps;
  pcr_shape(extent, P, lpb, steps);
  const int a_extent = axis == 0 ? L.ny : L.nx;
  const int b_extent = axis == 2 ? L.ny : L.nz;
  if (P > 512) return false;
  lpb = std::max(1, std::min({512 / P, 4, ((a_extent + 1) / 2) * b_extent}));
  const size_t cells = static_cast<size_t>(L.nx) * L.ny * L.nz;
  constexpr size_t kCoarseLineShared = 200 * 1024;
  if ((2 * cells + static_cast<size_t>(P) * lpb) * sizeof(TC) > kCoarseLineShared) return false;
  const size_t smem = (2 * cells + static_cast<size_t>(2) * P * lpb) * sizeof(TC);
  const auto run = [&](auto kernel, int blocks) {
    allow_shared(kernel, smem, kCoarseLineShared + 512 * sizeof(TC));
    launch(kernel, blocks, dim3(P, lpb), smem, s, L, x, b, fac, sweeps, axis, columns);
  };
  switch (steps) {
#define HFPS_COARSE_CASE(N)                                                      \
  case N:                                                                        \
    if (columns == kCoarseVector && extent == 1 << N)                             \
      run(k_coarse_line_smem<T, TC, N, false, true>, 1);                          \
    else if (columns == kCoarseVector)                                            \
      run(k_coarse_line_smem<T, TC, N, false, false>, 1);                         \
    else if constexpr (std::is_same<T, TC>::value)                                \
      run(k_coarse_line_smem<T, TC, N, true, true>, 2 * static_cast<int>(cells)); \
    else return false;                                                            \
    break;
    HFPS_COARSE_CASE(0) HFPS_COARSE_CASE(1) HFPS_COARSE_CASE(2) HFPS_COARSE_CASE(3)
    HFPS_COARSE_CASE(4) HFPS_COARSE_CASE(5) HFPS_COARSE_CASE(6) HFPS_COARSE_CASE(7)
    HFPS_COARSE_CASE(8) HFPS_COARSE_CASE(9)
#undef HFPS_COARSE_CASE
    default: return false;
  }
  return true;
}

template size_t line_factor_values<double>(int, int, int, int);
template size_t line_factor_values<float>(int, int, int, int);
template void launch_line_factors<double>(cudaStream_t, const Level<double>&, int, double*);
template void launch_line_factors<float>(cudaStream_t, const Level<float>&, int, float*);
template void launch_line_pass<double>(cudaStream_t, const Level<double>&, double*,
                                       const double*, const double*, double*, int, int, int,
                                       bool, bool, bool);
template void launch_line_pass<float>(cudaStream_t, const Level<float>&, float*, const float*,
                                      const float*, float*, int, int, int, bool, bool, bool);
template bool launch_line_sweeps<double>(cudaStream_t, const Level<double>&, double*,
                                         const double*, const double*, int, int, int);
template bool launch_line_sweeps<float>(cudaStream_t, const Level<float>&, float*, const float*,
                                        const float*, int, int, int);
template bool launch_coarse_line<double, double>(cudaStream_t, const Level<double>&, double*,
                                                 const double*, const double*, int, int, int);
template bool launch_coarse_line<float, double>(cudaStream_t, const Level<double>&, float*,
                                                const float*, const double*, int, int, int);

// ---------------------------------------------------------------------------
// Coarsest level as a dense affine map: out = P x + M b, with P and M
// (n x n each, FP64) stored column-major one after the other, as the
// columns mode of k_coarse_line_smem writes them.  A block owns 32 rows (one
// per lane); its 32 warps take every 32nd column with 8 column loads in
// flight per thread, and the 32 partial sums of a row are added in warp
// order, so the result is reproducible (dense_rows).
template <class T>
__global__ void __launch_bounds__(32 * kDenseWarps)
    k_coarse_dense(int n, const double* __restrict__ op, const T* __restrict__ x,
                   const T* __restrict__ b, T* __restrict__ out, bool x_zero) {
  grid_dependency_sync();
  extern __shared__ double dense_smem[];
  double* v = dense_smem;                    // [2n]: x then b, widened
  double* part = dense_smem + 2 * n;         // [kDenseWarps][32]
  const int tid = threadIdx.y * 32 + threadIdx.x;
  for (int j = tid; j < n; j += 32 * kDenseWarps) {
    v[j] = x_zero ? 0.0 : static_cast<double>(x[j]);
    v[n + j] = static_cast<double>(b[j]);
  }
  __syncthreads();
  dense_rows<T>(n, op, v, part, blockIdx.x, threadIdx.x, threadIdx.y, x_zero, out);
}

template <class T>
void launch_coarse_dense(cudaStream_t s, int n, const double* op, const T* x,
                         const T* b, T* out, bool x_zero) {
  static_assert((2 * kCoarseDenseMaxCells + 32 * kDenseWarps) * sizeof(double) <= 48 * 1024,
                "default shared memory limit");
  const size_t smem = (2 * static_cast<size_t>(n) + 32 * kDenseWarps) * sizeof(double);
  launch(k_coarse_dense<T>, (n + 31) / 32, dim3(32, kDenseWarps), smem, s, n, op, x, b, out,
         x_zero);
}

template void launch_coarse_dense<double>(cudaStream_t, int, const double*, const double*,
                                          const double*, double*, bool);
template void launch_coarse_dense<float>(cudaStream_t, int, const double*, const float*,
                                         const float*, float*, bool);

}  // namespace hfps
