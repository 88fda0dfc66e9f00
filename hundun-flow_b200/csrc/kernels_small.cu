// The smallest levels of a cycle as one launch.
//
// Below about a thousand cells a phase of the cycle (a Chebyshev stage, a
// colour pass, a transfer) is under a microsecond of work, but as a kernel
// of its own it takes 1.6-5 us on the device, and an F-cycle visits level l
// l + 1 times: at 64^3 these levels were 60 of 87 launches and 225 of the
// 370 us of an FP64 MG application, 117 us of them in the one-CTA coarsest
// solve, whose 48 colour passes each waited on global memory.  Here one CTA
// keeps the coefficients and vectors of all of these levels in shared memory
// and runs the whole sub-cycle (both visits of an F-cycle, which follow one
// another) from a list of phases built on the host, with a CTA barrier
// between phases.  The coarsest sweeps run in one warp, a cell per lane, the
// neighbours exchanged by shuffles and nothing but registers touched.  Line
// levels with lines of at most 32 cells run their colour passes as PCR within
// a warp, and their coarsest sweeps as the dense affine map.
//
// What bounds it: latency.  A phase is one round of shared-memory loads, the
// row's chain of seven dependent operations and a division, and a barrier;
// the coarsest solve is 48 such chains in a row.  One CTA is the right size
// because a phase of a thousand cells is shorter than any wait between CTAs.
//
// Every cell update is the one of the per-kernel path, operation for
// operation (row_value, prolongate_at, the same stage formulas, PCR), so results
// are bit-identical to it; only the dense map groups its sums differently.
#include "kernels.hpp"
#include "phase_device.cuh"

#include <algorithm>

namespace hfps {
namespace {

constexpr int kSmallThreads = 512;

// A cell's indices packed in one word (extents of at most kSmallMaxCells).
__device__ __forceinline__ unsigned small_pack(int i, int j, int k) {
  return static_cast<unsigned>(i) | (static_cast<unsigned>(j) << 10) |
         (static_cast<unsigned>(k) << 20);
}
__device__ __forceinline__ void small_unpack(unsigned v, int& i, int& j, int& k) {
  i = v & 1023u;
  j = (v >> 10) & 1023u;
  k = v >> 20;
}

// All red-black sweeps of a coarsest level of at most 32 cells in one warp:
// lane l holds cell l, its coefficients and its x.  A neighbour outside the
// level is the lane itself with its coefficient kept (Neumann) or zeroed
// (Dirichlet: the term is then an exact zero, as coefficient * 0 is).
template <class T>
__device__ __forceinline__ void small_coarse_warp(const Level<double>& L, T* x, const T* b,
                                                  int sweeps) {
  const int lane = threadIdx.x;
  const int n = L.nx * L.ny * L.nz;
  const bool on = lane < n;
  const int c = on ? lane : 0;
  int i, j, k;
  cell_coords(c, L.nx, L.ny, i, j, k);
  const int plane = L.nx * L.ny;
  const int fxi = face_x_index(L, c, j, k);
  const int fyi = face_y_index(L, c, k);
  double f[6] = {L.fx[fxi], L.fx[fxi + 1], L.fy[fyi], L.fy[fyi + L.nx], L.fz[c], L.fz[c + plane]};
  int from[6] = {c - 1, c + 1, c - L.nx, c + L.nx, c - plane, c + plane};
  const bool in[6] = {i > 0, i + 1 < L.nx, j > 0, j + 1 < L.ny, k > 0, k + 1 < L.nz};
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    if (in[e]) continue;
    from[e] = c;
    if (!((L.neumann >> e) & 1u)) f[e] = 0.0;
  }
  const double d = L.diag[c];
  const double rhs = static_cast<double>(b[c]);
  double xc = static_cast<double>(x[c]);
  const double omega = 0.72;
  const int parity = (i + j + k) & 1;
  for (int s = 0; s < sweeps; ++s) {
#pragma unroll
    for (int color = 0; color < 2; ++color) {
      double xn[6];
#pragma unroll
      for (int e = 0; e < 6; ++e) xn[e] = __shfl_sync(0xffffffffu, xc, from[e]);
      double v = d * xc;
#pragma unroll
      for (int e = 0; e < 6; ++e) v -= f[e] * xn[e];
      const double next = xc + omega * (rhs - v) / d;
      xc = parity == color ? next : xc;
    }
  }
  if (on) x[c] = static_cast<T>(xc);
}

// One zebra colour of line relaxation along `axis` (lines of at most 32 cells):
// P = 2^steps lanes hold a line, its PCR steps exchange by shuffles
// (pcr_line_slot's arithmetic, without its barriers).
template <class T>
__device__ __forceinline__ void small_line_pass(const Level<T>& L, T* x, const T* b,
                                                const T* __restrict__ fac, int axis, int steps,
                                                int color) {
  const int P = 1 << steps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int a_extent = axis == 0 ? L.ny : L.nx;
  const int b_extent = axis == 2 ? L.ny : L.nz;
  const int ha = (a_extent + 1) >> 1;
  const int lines = ha * b_extent;
  const int extent = line_extent(axis, L.nx, L.ny, L.nz);
  const size_t slab = static_cast<size_t>(a_extent) * b_extent * P;
  const int per_warp = 32 >> steps;
  const int s = lane & (P - 1);
  for (int t0 = warp * per_warp; t0 < lines; t0 += (kSmallThreads / 32) * per_warp) {
    const int t = t0 + (lane >> steps);
    const int fb = t / ha;
    const int fa = 2 * (t - fb * ha) + ((fb + color) & 1);
    const bool valid = t < lines && fa < a_extent;
    const size_t at = static_cast<size_t>(valid ? fa + a_extent * fb : 0) * P + s;
    T k[2 * kSmallMaxSteps + 1];
#pragma unroll
    for (int e = 0; e <= 2 * kSmallMaxSteps; ++e)
      k[e] = e <= 2 * steps ? __ldg(fac + e * slab + at) : T(0);
    int c = 0;
    T d = T(0);
    if (valid && s < extent) {
      int i, j, m;
      line_cell(axis, fa, fb, s, i, j, m);
      c = i + L.nx * (j + L.ny * m);
      d = line_rhs_any<T, PlainLoad>(L, x, b, axis, fa, fb, s, extent, c);
    }
    T pivot = k[0];
#pragma unroll
    for (int step = 0; step < kSmallMaxSteps; ++step) {
      if (step < steps) {
        const int h = 1 << step;
        const T up = __shfl_up_sync(0xffffffffu, d, h);
        const T down = __shfl_down_sync(0xffffffffu, d, h);
        const T dlo = s - h >= 0 ? up : T(0);
        const T dhi = s + h < P ? down : T(0);
        d = d - dlo * k[2 * step] - dhi * k[2 * step + 1];
        pivot = k[2 * step + 2];
      }
    }
    if (valid && s < extent) x[c] = d / pivot;
  }
}

// The coarsest sweeps as the dense affine map P x + M b (FP64, column-major,
// P then M): groups of threads take interleaved columns of all rows, and a
// row's partial sums are added in group order.  With x_zero the P half is not
// read.  v holds 2n doubles, part one per thread.
template <class T>
__device__ __forceinline__ void small_dense(int n, const double* __restrict__ op, T* x, const T* b,
                                            double* v, double* part, bool x_zero) {
  const int tid = threadIdx.x;
  for (int c = tid; c < n; c += kSmallThreads) {
    v[c] = static_cast<double>(x[c]);
    v[n + c] = static_cast<double>(b[c]);
  }
  __syncthreads();
  const int width = (n + 31) & ~31;
  const int groups = kSmallThreads / width;
  const int group = tid / width, row = tid - group * width;
  double acc = 0.0;
  if (group < groups && row < n) {
#pragma unroll 8
    for (int j = (x_zero ? n : 0) + group; j < 2 * n; j += groups)
      acc += __ldg(op + static_cast<size_t>(j) * n + row) * v[j];
  }
  part[tid] = acc;
  __syncthreads();
  if (tid < n) {
    double sum = part[tid];
    for (int g = 1; g < groups; ++g) sum += part[g * width + tid];
    x[tid] = static_cast<T>(sum);
  }
}

template <class T>
__global__ void __launch_bounds__(kSmallThreads) k_small_cycle(const SmallProgram<T> prog) {
  extern __shared__ double small_smem[];
  char* const smem = reinterpret_cast<char*>(small_smem);
  const int tid = threadIdx.x;
  // Coefficients and cell indices of every level.  They were written before
  // the kernel that this launch waits for began, so they are loaded ahead of
  // the wait.
  for (int l = 0; l < prog.count; ++l) {
    const SmallLevel<T>& S = prog.level[l];
    const Level<T>& L = S.view;
    const int n = L.nx * L.ny * L.nz;
    const int nfx = (L.nx + 1) * L.ny * L.nz, nfy = L.nx * (L.ny + 1) * L.nz,
              nfz = L.nx * L.ny * (L.nz + 1);
    T* d = reinterpret_cast<T*>(smem + S.coefficients);
    T* fx = d + n;
    T* fy = fx + nfx;
    T* fz = fy + nfy;
    unsigned* ijk = reinterpret_cast<unsigned*>(smem + S.cells);
    for (int c = tid; c < n; c += kSmallThreads) {
      d[c] = L.diag[c];
      int i, j, k;
      cell_coords(c, L.nx, L.ny, i, j, k);
      ijk[c] = small_pack(i, j, k) | (L.fluid[c] != 0 ? 1u << 30 : 0u);
    }
    for (int f = tid; f < nfx; f += kSmallThreads) fx[f] = L.fx[f];
    for (int f = tid; f < nfy; f += kSmallThreads) fy[f] = L.fy[f];
    for (int f = tid; f < nfz; f += kSmallThreads) fz[f] = L.fz[f];
  }
  grid_dependency_sync();
  {
    const SmallLevel<T>& S = prog.level[0];
    const int n = S.view.nx * S.view.ny * S.view.nz;
    T* v = reinterpret_cast<T*>(smem + S.vectors);
    for (int c = tid; c < n; c += kSmallThreads) {
      v[kSmallX * n + c] = T(0);
      v[kSmallB * n + c] = prog.b[c];
    }
  }
  __syncthreads();

  for (int op = 0; op < prog.ops; ++op) {
    const unsigned word = prog.op[op];
    const int kind = word & 15u;
    const int lv = (word >> 4) & 15u;
    const int arg = (word >> 8) & 255u;
    const int slot = (word >> 16) & 1u;  // which of the two x vectors is current
    const SmallLevel<T>& S = prog.level[lv];
    const int n = S.view.nx * S.view.ny * S.view.nz;
    const T* diag = reinterpret_cast<const T*>(smem + S.coefficients);
    Level<T> L = S.view;
    L.diag = diag;
    L.fx = diag + n;
    L.fy = L.fx + (L.nx + 1) * L.ny * L.nz;
    L.fz = L.fy + L.nx * (L.ny + 1) * L.nz;
    const unsigned* ijk = reinterpret_cast<const unsigned*>(smem + S.cells);
    T* vec = reinterpret_cast<T*>(smem + S.vectors);
    T* x = vec + slot * n;
    T* other = vec + (slot ^ 1) * n;
    T* b = vec + kSmallB * n;
    T* r = vec + kSmallR * n;
    switch (kind) {
      case kSmallStage: {
        // chebyshev_cell, from x into the other x vector.
        const T previous = prog.previous_factor[arg], residual = prog.residual_factor[arg];
        for (int c = tid; c < n; c += kSmallThreads) {
          int i, j, k;
          small_unpack(ijk[c] & 0x3fffffffu, i, j, k);
          const T value = row_value<T>(L, x, i, j, k, c);
          const T defect = b[c] - value;
          const T scaled = residual * defect / L.diag[c];
          const T d = arg == 0 ? scaled : previous * r[c] + scaled;
          r[c] = d;
          other[c] = x[c] + d;
        }
        break;
      }
      case kSmallColour:
        // rb_slot, in place: a cell reads only the other colour and itself.
        for (int c = tid; c < n; c += kSmallThreads) {
          int i, j, k;
          small_unpack(ijk[c] & 0x3fffffffu, i, j, k);
          if (((i + j + k) & 1) != arg) continue;
          const T value = row_value<T>(L, x, i, j, k, c);
          x[c] = x[c] + T(0.72) * (b[c] - value) / L.diag[c];
        }
        break;
      case kSmallDefect:
        for (int c = tid; c < n; c += kSmallThreads) {
          int i, j, k;
          small_unpack(ijk[c] & 0x3fffffffu, i, j, k);
          r[c] = b[c] - row_value<T>(L, x, i, j, k, c);
        }
        break;
      case kSmallGather: {
        // restrict_residual: level lv's rhs from the finer level's defects
        // (vector R), children in dz, dy, dx order; then x = 0 or the first
        // smoothing step from it (zero_start).
        const SmallLevel<T>& FS = prog.level[lv - 1];
        const int fnx = FS.view.nx, fny = FS.view.ny, fnz = FS.view.nz;
        const int m = FS.mask;
        const int mx = m & 1, my = (m >> 1) & 1, mz = (m >> 2) & 1;
        const T* fr = reinterpret_cast<const T*>(smem + FS.vectors) + kSmallR * (fnx * fny * fnz);
        for (int c = tid; c < n; c += kSmallThreads) {
          int i, j, k;
          small_unpack(ijk[c] & 0x3fffffffu, i, j, k);
          T sum = T(0);
          for (int dz = 0; dz <= mz; ++dz)
            for (int dy = 0; dy <= my; ++dy)
              for (int dx = 0; dx <= mx; ++dx) {
                const int fi = (i << mx) + dx, fj = (j << my) + dy, fk = (k << mz) + dz;
                if (fi >= fnx || fj >= fny || fk >= fnz) continue;
                sum += fr[fi + fnx * (fj + fny * fk)];
              }
          b[c] = sum;
          T d;
          x[c] = zero_start_value<T>(arg, prog.residual_factor[0], sum, L.diag[c],
                                     (i + j + k) & 1, d);
          r[c] = d;
        }
        break;
      }
      case kSmallStart:
        // The same start from x = 0 on the first level (its rhs came in).
        for (int c = tid; c < n; c += kSmallThreads) {
          int i, j, k;
          small_unpack(ijk[c] & 0x3fffffffu, i, j, k);
          T d;
          x[c] = zero_start_value<T>(arg, prog.residual_factor[0], b[c], L.diag[c],
                                     (i + j + k) & 1, d);
          r[c] = d;
        }
        break;
      case kSmallProlong: {
        // x of level lv plus the correction of level lv + 1 (its vector `arg`).
        const SmallLevel<T>& CS = prog.level[lv + 1];
        const int cn = CS.view.nx * CS.view.ny * CS.view.nz;
        const T* cx = reinterpret_cast<const T*>(smem + CS.vectors) + arg * cn;
        for (int c = tid; c < n; c += kSmallThreads) {
          int i, j, k;
          const unsigned word_c = ijk[c];
          small_unpack(word_c & 0x3fffffffu, i, j, k);
          const T value = prolongate_at<T, PlainLoad>(CS.view, cx, S.mask, i, j, k, NaturalPos());
          x[c] = (word_c >> 30) != 0u ? x[c] + value : T(0);
        }
        break;
      }
      case kSmallLine:
        small_line_pass<T>(L, x, b, S.factors[arg & 3], arg & 3, arg >> 3, (arg >> 2) & 1);
        break;
      case kSmallDense: {
        double* v = reinterpret_cast<double*>(smem + prog.wide);
        small_dense<T>(n, prog.dense, x, b, v, v + 2 * n, arg != 0);
        break;
      }
      default: {  // kSmallCoarse
        if (n <= 32) {
          if (tid < 32) small_coarse_warp<T>(prog.coarse, x, b, prog.coarse_sweeps);
          break;
        }
        // Wider coarsest levels: the sweeps in FP64 over shared memory.
        double* xw = reinterpret_cast<double*>(smem + prog.wide);
        double* bw = xw + n;
        for (int c = tid; c < n; c += kSmallThreads) {
          xw[c] = static_cast<double>(x[c]);
          bw[c] = static_cast<double>(b[c]);
        }
        __syncthreads();
        for (int s = 0; s < prog.coarse_sweeps; ++s)
          for (int color = 0; color < 2; ++color) {
            for (int c = tid; c < n; c += kSmallThreads) {
              int i, j, k;
              small_unpack(ijk[c] & 0x3fffffffu, i, j, k);
              if (((i + j + k) & 1) != color) continue;
              const double value = row_value(prog.coarse, xw, i, j, k, c);
              xw[c] += 0.72 * (bw[c] - value) / prog.coarse.diag[c];
            }
            __syncthreads();
          }
        for (int c = tid; c < n; c += kSmallThreads) x[c] = static_cast<T>(xw[c]);
        break;
      }
    }
    __syncthreads();
  }
  {
    const SmallLevel<T>& S = prog.level[0];
    const int n = S.view.nx * S.view.ny * S.view.nz;
    const T* x = reinterpret_cast<const T*>(smem + S.vectors) + prog.result * n;
    for (int c = tid; c < n; c += kSmallThreads) prog.x[c] = x[c];
  }
}

}  // namespace

// Shared-memory layout of a program: per level the coefficients, the packed
// cell indices and four vectors, and FP64 scratch for the coarsest level.
template <class T>
size_t small_layout(SmallProgram<T>& prog) {
  size_t bytes = 0;
  const auto add = [&](size_t b) {
    const size_t at = bytes;
    bytes += (b + 15) & ~static_cast<size_t>(15);
    return static_cast<int>(at);
  };
  for (int l = 0; l < prog.count; ++l) {
    SmallLevel<T>& S = prog.level[l];
    const size_t nx = S.view.nx, ny = S.view.ny, nz = S.view.nz, n = nx * ny * nz;
    S.coefficients =
        add((n + (nx + 1) * ny * nz + nx * (ny + 1) * nz + nx * ny * (nz + 1)) * sizeof(T));
    S.cells = add(n * sizeof(unsigned));
    S.vectors = add(kSmallVectors * n * sizeof(T));
  }
  const SmallLevel<T>& last = prog.level[prog.count - 1];
  prog.wide = add((2 * static_cast<size_t>(last.view.nx) * last.view.ny * last.view.nz +
                   kSmallThreads) *
                  sizeof(double));
  return bytes;
}

template <class T>
bool launch_small_cycle(cudaStream_t s, SmallProgram<T>& prog) {
  const size_t smem = small_layout(prog);
  if (smem > kSmallMaxShared) return false;
  allow_shared(k_small_cycle<T>, smem, kSmallMaxShared);
  launch(k_small_cycle<T>, 1, kSmallThreads, smem, s, prog);
  return true;
}

template size_t small_layout<double>(SmallProgram<double>&);
template size_t small_layout<float>(SmallProgram<float>&);
template bool launch_small_cycle<double>(cudaStream_t, SmallProgram<double>&);
template bool launch_small_cycle<float>(cudaStream_t, SmallProgram<float>&);

}  // namespace hfps
