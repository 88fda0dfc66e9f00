// The cold path's diagonal IC(0) (ColdPressureIccg, src/solver_iccg.hpp:
// 224-293; ColdPressureDilu, src/solver_cold.hpp:484-560, identical on the
// symmetric pressure rows): factorisation and both triangular sweeps in the
// reference's lexicographic order, one launch each.
//
// A cell depends on its lower (backward sweep: upper) neighbours only, so
// cells with equal i + j + k are independent.  One launch per such plane took
// 1.85 us per plane whatever its size, 640 us per application at 64^3.  Here a
// CTA owns a tile of kDicY x kDicZ columns in (j, k), one per compute thread, and
// marches them along x one step apart: thread (ty, tz) takes cell
// i = t - ty - tz at step t, so its x neighbour is its own last value and its
// y and z neighbours are what threads (ty - 1, tz) and (ty, tz - 1) formed in
// the step before, exchanged through shared memory with one barrier per step.
//
// Tiles follow one another value by value: the edge threads of a tile also
// write their results to a border array whose entries start as a pattern no
// result has (all bits set, a NaN that arithmetic does not make), and the next
// tile waits for the entries themselves.  No flag, fence or barrier lies between
// two tiles (a flag per 8 steps cost 3.4 us each in its wait, loads and fence).
//
// What bounds it: the chain of nx + ny + nz - 2 dependent steps, and 2.2 us per
// tile border on the longest path beyond the steps of its skew: the copy warps wait
// for all border entries of a chunk before the barrier that starts it, up to seven
// steps more than the skew needs, and the entries take a trip through L2.  A step is
// some twenty instructions of one warp per scheduler, so nothing else may run in
// the compute warps: four more warps copy the next chunk's inputs to shared memory
// (cp.async, the skewed windows of all rows, kDicChunk steps), wait for its border
// entries and write the last chunk's results back.  With all of it in the four
// compute warps a step took 0.36 us, now 0.18 forward and 0.25 backward.  Steps outside the grid compute on whatever
// is there and are set to zero, which is also the neighbour outside it, so a step
// has no branches.  The sweeps of an application take 72 + 83 us at 64^3, where the
// longest path has 190 steps (34 + 47 us) and ten borders (22 us a sweep; some 15 us
// a sweep are neither), and 236 + 257 at 128^3.
//
// Waits cannot deadlock: tiles are taken in the order of a ticket, diagonal by
// diagonal, so a tile waits only for tiles whose CTAs are already running.
// They are bounded too: a wait that runs out sets flag bit 4 and ends the
// sweep on every CTA, and the solver reports it at its next check.
//
// Each cell's arithmetic is the reference's, operation for operation.
#include "kernels.hpp"

namespace hfps {
namespace {

constexpr int kDicY = 16;
constexpr int kDicZ = 8;
constexpr int kDicColumns = kDicY * kDicZ;       // compute threads
constexpr int kDicThreads = 2 * kDicColumns;     // and as many that copy
constexpr int kDicChunk = 8;
constexpr int kDicPitch = kDicChunk + 1;  // rows of a window fall in different banks
// Values a step reads: the columns' last ones, then the y and the z border.
constexpr int kDicValues = kDicColumns + kDicZ + kDicY;
constexpr size_t kDicHeader = 16;  // the ticket, on a 128-byte line of its own
constexpr long long kDicSpinLimit = 1LL << 20;  // polls of an L2 round trip: under a second
constexpr unsigned long long kDicAbsent = ~0ull;
constexpr int kDicTimeout = 16;

enum DicMode : int { kDicForward = 0, kDicBackward = 1, kDicPivots = 2 };

__device__ __forceinline__ void copy_async8(double* shared, const double* global) {
  const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(shared));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(global));
}

__device__ __forceinline__ unsigned long long dic_peek(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// A border entry for the next tile; a result with the absent pattern's bits (a
// NaN that came in) goes as the canonical NaN.
__device__ __forceinline__ void dic_post(double* p, double value) {
  unsigned long long v = static_cast<unsigned long long>(__double_as_longlong(value));
  if (v == kDicAbsent) v = 0x7ff8000000000000ull;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Waits for a border entry; zero when the limit ran out here or in another CTA.
__device__ double dic_wait(const double* p, Scalars* sc) {
  for (long long polls = 0;; ++polls) {
    const unsigned long long seen = dic_peek(p);
    if (seen != kDicAbsent) return __longlong_as_double(static_cast<long long>(seen));
    if (polls >= kDicSpinLimit) {
      atomicOr(&sc->flags, kDicTimeout);
      return 0.0;
    }
    if ((polls & 63) == 63 && (*reinterpret_cast<volatile int*>(&sc->flags) & kDicTimeout) != 0)
      return 0.0;
  }
}

// The tile of ticket t, diagonal (y + z) by diagonal.
__device__ void dic_tile(int t, int tiles_y, int tiles_z, int& y, int& z) {
  int d = 0;
  for (;; ++d) {
    const int low = max(0, d - tiles_z + 1), high = min(d, tiles_y - 1);
    if (t <= high - low) {
      y = low + t;
      z = d - y;
      return;
    }
    t -= high - low + 1;
  }
}

// in, out: forward r and z, backward z and z, pivots the decorated row
// diagonals and the inverse pivots.  border: the ticket, then per tile the last
// y column of each z ([kDicZ][nx]) and the last z column of each y
// ([kDicY][nx]); the ticket is zero less one and every entry absent at the
// start.  The backward sweep runs in mirrored indices, so that all modes march
// upwards.
template <int MODE>
__global__ void __launch_bounds__(kDicThreads)
    k_dic_sweep(Level<double> L, const double* in, double* out, const double* __restrict__ inv,
                double* border, Scalars* scalars, int tiles_y, int tiles_z) {
  grid_dependency_sync();
  constexpr bool kMirror = MODE == kDicBackward;
  constexpr int kArrays = MODE == kDicPivots ? 4 : 5;  // in, x-, y-, z-faces, inverse pivots
  extern __shared__ double dic_smem[];
  // [2][kArrays][kDicColumns][kDicPitch] windows, then [2][kDicChunk][kDicValues]:
  // what step u of a chunk reads.
  constexpr int kWindow = kDicColumns * kDicPitch;
  double* const values = dic_smem + 2 * kArrays * kWindow;
  __shared__ int tile_y, tile_z;
  const int tid = threadIdx.x;
  if (tid == 0) {
    int y, z;
    // The header starts as all bits set, so the first ticket comes as ~0u.
    const unsigned ticket = atomicAdd(reinterpret_cast<unsigned*>(border), 1u) + 1u;
    dic_tile(static_cast<int>(ticket), tiles_y, tiles_z, y, z);
    tile_y = y;
    tile_z = z;
  }
  for (int v = tid; v < 2 * kDicChunk * kDicValues; v += kDicThreads) values[v] = 0.0;
  __syncthreads();
  const int nx = L.nx, ny = L.ny, nz = L.nz, plane = nx * ny;
  const int j0 = tile_y * kDicY, k0 = tile_z * kDicZ;
  const size_t per_tile = static_cast<size_t>(kDicY + kDicZ) * nx;
  double* const mine = border + kDicHeader + per_tile * (tile_y + tiles_y * tile_z);
  const int steps = nx + kDicY + kDicZ - 2;
  const int chunks = (steps + kDicChunk - 1) / kDicChunk;

  if (tid >= kDicColumns) {
    // Copies: thread (row of the y edge, step of the chunk), one z per turn.
    const int t = tid - kDicColumns;
    const int row_y = t / kDicChunk, u = t % kDicChunk;
    const int j = j0 + row_y;
    const int jj = kMirror ? ny - 1 - j : j;
    const auto each = [&](int chunk, auto f) {
#pragma unroll
      for (int z = 0; z < kDicZ; ++z) {
        const int k = k0 + z;
        const int i = chunk * kDicChunk + u - row_y - z;
        if (i < 0 || i >= nx || j >= ny || k >= nz) continue;
        const int ii = kMirror ? nx - 1 - i : i, kk = kMirror ? nz - 1 - k : k;
        f(ii + nx * (jj + ny * kk), kk, (z * kDicY + row_y) * kDicPitch + u);
      }
    };
    const auto load = [&](int chunk) {
      double* const w = dic_smem + (chunk & 1) * kArrays * kWindow;
      each(chunk, [&](int c, int kk, int at) {
        // The face towards the neighbour the sweep comes from.
        copy_async8(w + at, in + c);
        copy_async8(w + at + kWindow, L.fx + face_x_index(L, c, jj, kk) + (kMirror ? 1 : 0));
        copy_async8(w + at + 2 * kWindow, L.fy + face_y_index(L, c, kk) + (kMirror ? nx : 0));
        copy_async8(w + at + 3 * kWindow, L.fz + c + (kMirror ? plane : 0));
        if (MODE != kDicPivots) copy_async8(w + at + 4 * kWindow, inv + c);
      });
    };
    const auto flush = [&](int chunk) {
      const double* const w = dic_smem + (chunk & 1) * kArrays * kWindow;
      each(chunk, [&](int c, int, int at) { out[c] = w[at]; });
    };
    // Border entries: (edge row, step) pairs, the y border's rows first.
    const double* const before_y = mine - per_tile;
    const double* const before_z = mine - per_tile * tiles_y + static_cast<size_t>(kDicZ) * nx;
    const auto wait = [&](int chunk) {
      double* const v = values + (chunk & 1) * kDicChunk * kDicValues;
      for (int e = t; e < (kDicZ + kDicY) * kDicChunk; e += kDicColumns) {
        const int row = e / kDicChunk, step = e % kDicChunk;
        const bool y_edge = row < kDicZ;
        const int across = y_edge ? row : row - kDicZ;
        const int i = chunk * kDicChunk + step - across;
        if (i < 0 || i >= nx) continue;
        if (y_edge ? (tile_y == 0 || k0 + across >= nz) : (tile_z == 0 || j0 + across >= ny))
          continue;
        v[step * kDicValues + kDicColumns + row] =
            dic_wait((y_edge ? before_y : before_z) + static_cast<size_t>(across) * nx + i, scalars);
      }
    };
    load(0);
    wait(0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (int chunk = 0; chunk < chunks; ++chunk) {
      __syncthreads();
      if (chunk > 0) flush(chunk - 1);
      if (chunk + 1 < chunks) {
        load(chunk + 1);
        wait(chunk + 1);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    flush(chunks - 1);
    return;
  }

  const int ty = tid % kDicY, tz = tid / kDicY;
  const int j = j0 + ty, k = k0 + tz;
  const bool column = j < ny && k < nz;
  const bool post_y = column && ty == kDicY - 1 && tile_y + 1 < tiles_y;
  const bool post_z = column && tz == kDicZ - 1 && tile_z + 1 < tiles_z;
  double* const to_y = mine + static_cast<size_t>(tz) * nx;
  double* const to_z = mine + static_cast<size_t>(kDicZ + ty) * nx;
  const int from_y = ty > 0 ? tid - 1 : kDicColumns + tz;
  const int from_z = tz > 0 ? tid - kDicY : kDicColumns + kDicZ + ty;
  double x_last = 0.0;
  int i = -ty - tz, bad = 0;
  for (int chunk = 0; chunk < chunks; ++chunk) {
    __syncthreads();
    double* const row = dic_smem + (chunk & 1) * kArrays * kWindow + tid * kDicPitch;
    double* const v = values + (chunk & 1) * kDicChunk * kDicValues;
    double* const v_next = values + ((chunk + 1) & 1) * kDicChunk * kDicValues;
#pragma unroll
    for (int u = 0; u < kDicChunk; ++u, ++i) {
      const double ax = row[kWindow + u], ay = row[2 * kWindow + u], az = row[3 * kWindow + u];
      const double own = row[u];
      const double y_last = v[u * kDicValues + from_y], z_last = v[u * kDicValues + from_z];
      const bool on = column && i >= 0 && i < nx;
      double value;
      if (MODE == kDicPivots) {
        value = own;
        value -= ax * ax * x_last;
        value -= ay * ay * y_last;
        value -= az * az * z_last;
        if (on && (!(value > 0) || !isfinite(value))) bad = 1;
        value = 1 / value;
      } else {
        value = MODE == kDicForward ? own : 0.0;
        value += ax * x_last;
        value += ay * y_last;
        value += az * z_last;
        value = value * row[4 * kWindow + u];
        if (MODE == kDicBackward) value = own + value;
      }
      value = on ? value : 0.0;
      if (post_y && on) dic_post(to_y + i, value);
      if (post_z && on) dic_post(to_z + i, value);
      row[u] = value;
      x_last = value;
      (u + 1 < kDicChunk ? v + (u + 1) * kDicValues : v_next)[tid] = value;
      if (u + 1 < kDicChunk) asm volatile("bar.sync 1, %0;" ::"n"(kDicColumns) : "memory");
    }
  }
  __syncthreads();
  if (MODE == kDicPivots && bad) atomicOr(&scalars->flags, 1);
}

int dic_tiles(int ny, int nz) {
  return ((ny + kDicY - 1) / kDicY) * ((nz + kDicZ - 1) / kDicZ);
}

template <int MODE>
void launch_sweep(cudaStream_t s, const Level<double>& L, const double* in, double* out,
                  const double* inv, double* border, Scalars* scalars) {
  constexpr int arrays = MODE == kDicPivots ? 4 : 5;
  constexpr size_t smem =
      (2 * arrays * kDicColumns * kDicPitch + 2 * kDicChunk * kDicValues) * sizeof(double);
  allow_shared(k_dic_sweep<MODE>, smem, smem);
  launch(k_dic_sweep<MODE>, dic_tiles(L.ny, L.nz), kDicThreads, smem, s, L, in, out, inv, border,
         scalars, (L.ny + kDicY - 1) / kDicY, (L.nz + kDicZ - 1) / kDicZ);
}

// Doubles of one sweep's header and borders.
size_t sweep_border(int nx, int ny, int nz) {
  return kDicHeader + static_cast<size_t>(dic_tiles(ny, nz)) * (kDicY + kDicZ) * nx;
}

}  // namespace

size_t dic_border_values(int nx, int ny, int nz) { return 2 * sweep_border(nx, ny, nz); }

void launch_dic_pivots(cudaStream_t s, const Level<double>& L, const double* rows, double* inv,
                       double* border, Scalars* scalars) {
  cudaMemsetAsync(border, 0xff, sweep_border(L.nx, L.ny, L.nz) * sizeof(double), s);
  launch_sweep<kDicPivots>(s, L, rows, inv, nullptr, border, scalars);
}

void launch_dic_apply(cudaStream_t s, const Level<double>& L, const double* in, double* out,
                      const double* inv, double* border, Scalars* scalars) {
  const size_t values = sweep_border(L.nx, L.ny, L.nz);
  cudaMemsetAsync(border, 0xff, 2 * values * sizeof(double), s);
  launch_sweep<kDicForward>(s, L, in, out, inv, border, scalars);
  launch_sweep<kDicBackward>(s, L, out, out, inv, border + values, scalars);
}

}  // namespace hfps
