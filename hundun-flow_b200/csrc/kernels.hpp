// Host-callable launchers for the sm_100a kernels (kernels.cu).
//
// Every launcher enqueues on the given stream and never synchronises.  Level
// operands are passed as hfps::Level<T> (hfps_device.cuh); vectors are dense
// x-fastest arrays of the level's shape.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "hfps_device.cuh"

namespace hfps {

// Device-resident Krylov scalars.  Kernels read alpha/beta from here, so a
// whole iteration runs without a host round trip; the host reads back only
// what steers control flow.
struct Scalars {
  double rho;        // r.z of the current search direction
  double pap;        // p.Ap
  double alpha;      // rho / pap
  double rr;         // last r.r (recursive or true residual)
  double rho_next;   // r.z after the preconditioner
  double beta;       // rho_next / rho (0 after a restart)
  double proj[3];    // MG projection sums r.r, r.Az, Az.Az
  double mg_alpha;   // MG correction scale
  double misc[4];
  double hcol[72];   // FGMRES: projections of the current column and |w|^2
  int flags;         // bit 0 non-finite, bit 1 breakdown, bit 2 invalid assembly input,
                     // bit 3 a grid barrier of the small-level kernel timed out
  unsigned marks;    // bit 0: a difference had a nonzero entry (recycle capture)
  unsigned counters[12];  // last-block arrival counters, one per reduction
  double constant_mean;   // volume-weighted mean of the last project_constant
  // The small-level kernel's grid barrier: arrivals (on a 128-byte line of
  // its own).
  unsigned tail_pad0[32];
  unsigned tail_count;
  unsigned tail_pad1[31];
};

enum ScalarOp : int {
  kOpPap = 0,        // pap = sum; alpha = rho / pap
  kOpRecursive = 1,  // rr = sum
  kOpRhoNext = 2,    // rho_next = sum; beta = rho_next / rho; rho = rho_next
  kOpRhoRestart = 3, // rho = sum; beta = 0
  kOpMisc = 4,       // misc[0] = sum
  kOpScaledNorm = 7, // misc[3] = misc[2] * sqrt(sum): the max-scaled norm (counter 7)
};
// Arrival counters of reductions that apply no scalar op: 5 MG projection,
// 6 FGMRES multidot, 8 project_constant.  Counter 7 serves both passes of
// the max-scaled norm.
constexpr int kCounterProjection = 5;
constexpr int kCounterMultidot = 6;
constexpr int kCounterProjectConstant = 8;
constexpr int kMaxFgmresRestart = 64;

struct Reduce {
  Scalars* scalars;
  double* partials;   // >= gridDim.x * kBasisChunk doubles
  int op;
};

int reduction_blocks(long long items);

// Layout of a level's vectors (x, b): hx == 0 the natural x-fastest order,
// otherwise split rows (SplitPos) whose even- and odd-i halves are hx cells
// long, 2 * hx * ny * nz values in all.  Coefficients and every other vector
// stay in the natural order.
struct VecLayout {
  int nx, ny, hx;
};

// ---- level operators (T = double or float) -------------------------------
template <class T>
void launch_level_apply(cudaStream_t s, const Level<T>& L, const T* x, T* y);
// r (natural order) = b - A x with x, b in layout hx.
template <class T>
void launch_level_defect(cudaStream_t s, const Level<T>& L, const T* x,
                         const T* b, T* r, int hx = 0);
template <class T>
void launch_rb_color(cudaStream_t s, const Level<T>& L, T* x, const T* b,
                     int color);
template <class T>
void launch_chebyshev_stage(cudaStream_t s, const Level<T>& L, const T* x,
                            const T* b, T* direction, T* next,
                            T previous_factor, T residual_factor, bool first, bool last);
// What the producer of a level's rhs b writes to its x: zero, or the first
// pre-smoothing step from x = 0, which needs no neighbour (the row of a zero
// x is zero): the first Chebyshev stage x = factor * b / D (also the stage's
// direction, written when another stage follows), or the first red-black
// colour.  kZeroNone leaves x unwritten.
enum ZeroKind : int { kZeroClear = 0, kZeroChebyshev = 1, kZeroRedBlack = 2, kZeroNone = 3 };
template <class T>
struct ZeroStart {
  int kind;
  T factor;
  const T* diag;   // the level's, natural order
  T* direction;    // null when no further Chebyshev stage follows
};
// Fine x, b in layout hx, coarse b, x in layout hxc (zero: point levels, natural order).
template <class T>
void launch_defect_restrict(cudaStream_t s, const Level<T>& F, const T* x,
                            const T* b, const Level<T>& C, T* cb, T* cx,
                            int coarsen_mask, int hx, int hxc, const ZeroStart<T>& zero);
// Fine x in layout hx, coarse x in layout hxc.  even_only: the cells of odd
// i + k may be left alone, because a y-line colour pass overwrites them before
// anything reads them (honoured where it saves traffic, in split rows).
template <class T>
void launch_prolongate(cudaStream_t s, const Level<T>& F, T* x,
                       const Level<T>& C, const T* cx, int coarsen_mask, int hx = 0,
                       int hxc = 0, bool even_only = false);
// out = x after prolongation of cx and the first post-smoothing step: Chebyshev
// stage 0 (factor; its direction unless `last`) or red-black colour 1.  All three
// axes coarsened, natural order, at most kStepCells cells; out must not alias x.
constexpr long long kStepCells = 1LL << 17;
template <class T>
void launch_prolong_step(cudaStream_t s, const Level<T>& F, const T* x, const T* b,
                         const Level<T>& C, const T* cx, T* direction, T* out, bool chebyshev,
                         T factor, bool last);
// ---- zebra line relaxation (kernels_line.cu) --------------------------------
// Line-colour passes with at least kLinePcrThreshold lines (kLinePcrThresholdLong
// for lines of kLinePcrLongExtent cells or more) run the chunked-scan solve
// (lanes across lines, warps along chunks of one line); fewer lines run PCR
// with one CTA row per line.  Lines longer than 2048 cells are not supported
// (kLineNone).  The long-line boundary is lower because PCR's factor block
// grows with the line (2 log2(extent) + 1 arrays against the scan's two):
// measured MG applications, 512 lines per colour on the scan against PCR,
// 256-cell lines (32x256x32 in the 256^3 hierarchy) 2.74 against 2.80 ms,
// 128-cell lines (32x128x32 in the 128^3 one) 0.78 against 0.75 ms; fewer
// than 512 lines leave most SMs idle on the scan (2.82 ms with 8x256x8 on
// it as well).
#ifndef HFPS_LINE_PCR_THRESHOLD
#define HFPS_LINE_PCR_THRESHOLD 1024
#endif
#ifndef HFPS_LINE_PCR_THRESHOLD_LONG
#define HFPS_LINE_PCR_THRESHOLD_LONG 512
#endif
constexpr long long kLinePcrThreshold = HFPS_LINE_PCR_THRESHOLD;
constexpr long long kLinePcrThresholdLong = HFPS_LINE_PCR_THRESHOLD_LONG;
constexpr int kLinePcrLongExtent = 256;
enum LineKind : int { kLineNone = 0, kLineScan = 1, kLinePcr = 2 };
int line_kind(int nx, int ny, int nz, int axis);
// Values of the factor block of one level and line axis in precision T: the
// Thomas reciprocal and upper multiplier (2 per cell, FP64), plus the lower
// multiplier (3 per cell, FP32), or PCR multipliers and final diagonals.
template <class T>
size_t line_factor_values(int nx, int ny, int nz, int axis);
template <class T>
void launch_line_factors(cudaStream_t s, const Level<T>& L, int axis, T* fac);
// One zebra colour of line relaxation along `axis`, x and b in layout hx
// (split rows only with the scan solve, axis 1 or 2).  zero_other: the other
// colour's x is known to be zero (not read); zero_self: this colour's x is
// (the first pass and the first sweep of a cycle started from x = 0).  ends: a
// Neumann boundary face of the level may be nonzero (launch_neumann_faces).
template <class T>
void launch_line_pass(cudaStream_t s, const Level<T>& L, T* x, const T* b,
                      const T* fac, T* scratch, int axis, int color, int hx = 0,
                      bool zero_other = false, bool zero_self = false, bool ends = true);
// Coarsest level in line mode with x/rhs resident in shared memory; returns
// false when the level is too large for that form.  With kCoarseColumns,
// launches 2n blocks that write the columns of the sweeps' affine map x_out =
// P x_in + M b (P then M, column-major) to x, n = cells of the level;
// kCoarseColumnsOn applies the sweeps to columns already there (a further
// axis after the first).
enum CoarseColumns : int { kCoarseVector = 0, kCoarseColumns = 1, kCoarseColumnsOn = 2 };
// All `passes` colour passes of one axis, starting with colour `first`, in one
// launch.  False: not launched, the level is not a small PCR level.
template <class T>
bool launch_line_sweeps(cudaStream_t s, const Level<T>& L, T* x, const T* b, const T* fac,
                        int axis, int first, int passes);
template <class T, class TC>
bool launch_coarse_line(cudaStream_t s, const Level<TC>& L, T* x, const T* b,
                        const TC* fac, int sweeps, int axis, int columns = kCoarseVector);
// out = P x + M b with the dense coarsest-level map built by the columns
// mode above (n <= kCoarseDenseMaxCells; out must not alias x or b).  With
// x_zero (x is known to be zero) the P half is not read.
constexpr int kCoarseDenseMaxCells = 2048;
template <class T>
void launch_coarse_dense(cudaStream_t s, int n, const double* op, const T* x,
                         const T* b, T* out, bool x_zero);

// Coarsest level: `sweeps` smoother sweeps in one CTA, arithmetic in TC.
// Line mode when line_axis >= 0 (zebra line Gauss-Seidel).
template <class T, class TC>
void launch_coarse_solve(cudaStream_t s, const Level<TC>& L, T* x, const T* b,
                         TC* xs, TC* bs, TC* work, TC* dprime, int sweeps,
                         int line_axis);

// ---- small levels as one persistent launch (kernels_tail.cu) ---------------
// A program of cycle phases for the levels below the scan levels, executed
// by one cooperative launch with a bounded grid barrier between phases.
enum TailKind : int { kTailPcr = 0, kTailRestrict = 1, kTailProlong = 2, kTailDense = 3 };
struct TailOp {
  int kind;
  int level;   // index into TailProgram::levels (the fine level of a transfer)
  int arg;     // PCR: colour; transfers: coarsening mask; dense: x is zero
  int pad;
  // PCR: x, rhs, factors.  Restrict: fine x, fine b, coarse b, coarse x.
  // Prolong: fine x, coarse x.  Dense: x, b, out.
  void* p0;
  void* p1;
  void* p2;
  void* p3;
};
constexpr int kTailMaxOps = 480;
constexpr int kTailMaxLevels = 8;
// Passed by value as the kernel parameter (kept under the 32 KB limit).
template <class T>
struct TailProgram {
  int count;
  int dense_n;
  // Added to every barrier's target count: 0, or 1 to make the first
  // barrier run out its wait limit (the failure path's test).
  int barrier_offset;
  int pad;
  int axis[kTailMaxLevels];
  Level<T> levels[kTailMaxLevels];
  const double* dense_op;
  Scalars* scalars;
  TailOp ops[kTailMaxOps];
};
static_assert(sizeof(TailProgram<double>) < 32000, "kernel parameter limit");
// log2 of the PCR width for lines of `extent` cells, or -1 if unsupported.
int tail_steps(int extent);
// Lines of one PCR pass a CTA of the persistent launch relaxes at once.
int tail_lines_per_cta(int steps);
// CTAs that can be co-resident on `sms` SMs (0: cannot run).
template <class T>
int tail_grid(int steps, int dense_n, int sms);
template <class T>
bool launch_tail(cudaStream_t s, const TailProgram<T>& prog, int steps, int blocks);

// ---- the smallest levels as one launch (kernels_small.cu) -------------------
// Levels with at most kSmallMaxCells cells (and, where lines are relaxed, lines
// of at most 2^kSmallMaxSteps cells), from the first such level to the coarsest.  One CTA runs them: measured at 64^3
// (FP64 MG application, levels 8^3 and below; with the first smoothing step
// folded into the producers of the rhs) 357 -> 223 us.  At 16^3 a stage reads
// its coefficients at one SM's rate, no faster than a launch of 16 CTAs.
// The dense map of a line hierarchy's coarsest level reads 16 n^2 bytes in
// batches of L2 latency: with 180 rows in one CTA it took 15 us, against 4 us
// spread over several (k_coarse_dense), so such hierarchies keep that kernel
// and all their launches; with two strong axes (456x256x52, 8 rows, 24 sweeps
// along both axes before) one MG application went from 4.2 to 2.9 ms.
constexpr int kSmallMaxCells = 1023;
constexpr int kSmallMaxLevels = 12;
constexpr int kSmallMaxOps = 1024;
constexpr int kSmallMaxStages = 16;
constexpr int kSmallMaxSteps = 5;      // PCR steps of a line within a warp
constexpr int kSmallDenseCells = 64;  // rows of the coarsest dense map (below)
constexpr size_t kSmallMaxShared = 200 * 1024;
enum SmallKind : int {
  kSmallStage = 0,    // Chebyshev stage `arg`
  kSmallColour = 1,   // red-black colour `arg`
  kSmallDefect = 2,   // defect into vector R
  kSmallGather = 3,   // rhs from the finer level's defects, x by ZeroKind `arg`
  kSmallStart = 4,    // x by ZeroKind `arg` from the level's own rhs
  kSmallProlong = 5,  // add the next level's vector `arg`
  kSmallCoarse = 6,   // all red-black sweeps of the coarsest level
  kSmallLine = 7,     // line colour pass: axis | colour << 2 | PCR steps << 3
  kSmallDense = 8     // all line sweeps of the coarsest level; 1: x is zero
};
// Vectors of a level: two x (a Chebyshev stage writes the other one), b, and
// the direction or defect.
enum SmallVector : int { kSmallX = 0, kSmallX2 = 1, kSmallB = 2, kSmallR = 3, kSmallVectors = 4 };
template <class T>
struct SmallLevel {
  Level<T> view;
  const T* factors[3];  // PCR factors per strong axis
  int mask;           // axes that coarsen to the next level
  int coefficients, cells, vectors;  // byte offsets in shared memory
};
template <class T>
struct SmallProgram {
  int count;          // levels
  int ops;
  int coarse_sweeps;
  int result;         // x vector of the first level that holds the result
  int wide;           // byte offset of the coarsest level's FP64 copies
  const T* b;         // first level's rhs
  T* x;               // and result
  Level<double> coarse;
  const double* dense;  // coarsest affine map of line levels
  T previous_factor[kSmallMaxStages];
  T residual_factor[kSmallMaxStages];
  SmallLevel<T> level[kSmallMaxLevels];
  // kind | level << 4 | arg << 8 | current x vector << 16
  unsigned op[kSmallMaxOps];
};
static_assert(sizeof(SmallProgram<double>) < 32000, "kernel parameter limit");
// Lays the program out in shared memory and returns the bytes it takes.
template <class T>
size_t small_layout(SmallProgram<T>& prog);
// False (nothing launched) when it takes more than kSmallMaxShared.
template <class T>
bool launch_small_cycle(cudaStream_t s, SmallProgram<T>& prog);

// ---- MG entry/exit ------------------------------------------------------
// b = active ? r : 0 (converted to T), and x by `zero` (its Chebyshev and
// red-black starts only in natural order); b and x in layout v, r natural.
template <class T>
void launch_mg_enter(cudaStream_t s, int n, const double* r,
                     const uint8_t* active, T* b, T* x, VecLayout v, const ZeroStart<T>& zero);
// z = active ? x * scale : 0 (scale read from device when scale_ptr).
template <class T>
void launch_mg_exit(cudaStream_t s, int n, const T* x, const uint8_t* active,
                    const double* scale_ptr, double* z, VecLayout v);
// launch_mg_exit (unit scaling) fused with the PCG's r.z through red.
template <class T>
void launch_mg_exit_dot(cudaStream_t s, int n, const T* x, const uint8_t* active, double* z,
                        VecLayout v, const double* r, Reduce red);
template <class T>
void launch_diagonal_solve(cudaStream_t s, int n, const T* b, const T* diag,
                           T* x, VecLayout v);
// Projection sums for the residual-minimising MG scale (level-0, FP64 r).
template <class T>
void launch_mg_projection(cudaStream_t s, int n, const double* r,
                          const uint8_t* active, const T* recursive,
                          Reduce red);

// project_constant (src/solver_mg.cpp:1411-1453) on a level vector v in
// layout hx: v - mean on cells of positive volume and 0 on the others, mean
// = sum(volume v) / sum(volume) (kept in scalars->constant_mean).  A total
// volume that is not positive or a non-finite sum sets flag bit 0.
template <class T>
void launch_project_constant(cudaStream_t s, int nx, int ny, int nz, int hx, T* v,
                             const double* volume, Scalars* scalars, double* partials);

// ---- Krylov (FP64) --------------------------------------------------------
// y = A x and x.y: over 3-D shared-memory tiles when `tiled` and the tiles'
// partial sums fit the partials block, else a warp per x-row (the same rows).
void launch_spmv_dot(cudaStream_t s, const Level<double>& L, const double* x,
                     double* y, Reduce red, bool tiled = true);
void launch_residual_norm(cudaStream_t s, const Level<double>& L,
                          const double* x, const double* b, double* r,
                          Reduce red);
void launch_pcg_update(cudaStream_t s, int n, double* x, const double* p,
                       double* r, const double* ap, Reduce red);
void launch_dot(cudaStream_t s, int n, const double* a, const double* b,
                Reduce red);
void launch_p_update(cudaStream_t s, int n, double* p, const double* z,
                     const Scalars* sc);
void launch_norm2(cudaStream_t s, int n, const double* v, Reduce red);
// The max-scaled 2-norm of global_norm (src/solver_krylov.cpp:650-711) into
// scalars->misc[3]: pass 1 forms max |v| (misc[2]; a non-finite entry sets
// flag bit 0), pass 2 max * sqrt(sum of (v / max)^2), zero when max is zero.
void launch_scaled_norm(cudaStream_t s, int n, const double* v, Scalars* scalars,
                        double* partials);
void launch_copy(cudaStream_t s, int n, const double* src, double* dst);
// ---- the steps either side of the solve ----------------------------------------
// Pressure-correction system assembly (diag, rhs) from densities, the
// density derivative, the predicted face fluxes and the face coefficients.
void launch_assemble(cudaStream_t s, int nx, int ny, int nz, const double* xf,
                     const double* yf, const double* zf, double a0, double a1, double a2,
                     bool bdf2, const double* rho, const double* rho_n, const double* rho_nm1,
                     const double* psi, const double* source, const double* phix,
                     const double* phiy, const double* phiz, const double* fx,
                     const double* fy, const double* fz, double* diag, double* rhs,
                     Scalars* scalars);
// flux += mass-flux response of the correction p (in place).
void launch_correct_flux(cudaStream_t s, int nx, int ny, int nz, unsigned neumann,
                         const double* p, const double* cx, const double* cy,
                         const double* cz, double scale, double* qx, double* qy, double* qz,
                         Scalars* scalars);
// ---- cold path: diagonal IC(0) and BiCGSTAB ----------------------------------
// Decorated-row diagonal of the cold-path factorisation.
void launch_dic_rows(cudaStream_t s, int nx, int ny, int nz, unsigned neumann,
                     const double* diag, const double* fx, const double* fy, const double* fz,
                     const uint8_t* active, double* out);
// Doubles of the sweeps' tickets and tile borders (kernels_dic.cu).
size_t dic_border_values(int nx, int ny, int nz);
// Inverse pivots (flags bit 0 on a non-positive pivot; bit 4 when a wait
// between blocks ran out).
void launch_dic_pivots(cudaStream_t s, const Level<double>& L, const double* rows, double* inv,
                       double* border, Scalars* scalars);
// out = M^{-1} in: forward then backward sweep (flags bit 4 as above); out must
// not alias in.
void launch_dic_apply(cudaStream_t s, const Level<double>& L, const double* in, double* out,
                      const double* inv, double* border, Scalars* scalars);
void launch_bicg_direction(cudaStream_t s, int n, double* p, const double* r, const double* v,
                           double beta, double omega);
// s = r - alpha v, with |s|^2 through red.
void launch_bicg_intermediate(cudaStream_t s, int n, double* sv, const double* r,
                              const double* v, double alpha, Reduce red);
// x = (x + alpha ph) + omega sh, r = s - omega t, with |r|^2 through red.
void launch_bicg_update(cudaStream_t s, int n, double* x, const double* ph, const double* sh,
                        double* r, const double* sv, const double* t, double alpha,
                        double omega, Reduce red);
// ---- FGMRES (solve_fgmres) ---------------------------------------------------
// Basis vectors handled by one multidot / basis-update launch.
constexpr int kBasisChunk = 16;
struct BasisRefs {
  const double* v[kBasisChunk];
  double s[kBasisChunk];
  int count;
};
// w = A z - shift v.
void launch_operator_shift(cudaStream_t s, const Level<double>& L, const double* z,
                           const double* v, double shift, double* w);
// out[r] = v_r . w for r < count, and out[count] = w . w when `self`
// (count + self <= kBasisChunk); non-finite sums set flags bit 0.
void launch_multidot(cudaStream_t s, int n, const BasisRefs& basis, const double* w,
                     bool self, double* out, Reduce red);
// snap = x - snap; marks bit 0 when any entry is nonzero
// (difference_recycle_field, src/solver_linear_state.cpp:162-181).
void launch_difference_nonzero(cudaStream_t s, int n, const double* x, double* snap,
                               Scalars* scalars);
// out = (scaled ? scale : 1) * (dst + sum_r s_r v_r), per cell in basis order.
void launch_basis_update(cudaStream_t s, int n, const double* dst, const BasisRefs& basis,
                         double scale, bool scaled, double* out);

// ---- setup (FP64) ---------------------------------------------------------
void launch_mask_finest(cudaStream_t s, int nx, int ny, int nz,
                        const double* x_faces, const double* y_faces,
                        const double* z_faces, const double* diag_in,
                        const double* fx_in, const double* fy_in,
                        const double* fz_in, const uint8_t* active,
                        double* diag, double* fx, double* fy, double* fz,
                        double* volume, uint8_t* fluid);
void launch_reaction(cudaStream_t s, const Level<double>& L,
                     const double* volume, double* reaction);
// One axis of the tensor aggregation (aggregate_tensor_channel).
void launch_aggregate_axis(cudaStream_t s, const double* src, int ex, int ey,
                           int ez, double* dst, int dx, int dy, int dz,
                           int axis, int face_axis, int global_extent);
void launch_coarse_diagonal(cudaStream_t s, int nx, int ny, int nz,
                            double* diag, const double* fx, const double* fy,
                            const double* fz, const double* volume,
                            uint8_t* fluid);
void launch_beta_coefficients(cudaStream_t s, int nx, int ny, int nz,
                              const double* x_faces, const double* y_faces,
                              const double* z_faces, unsigned neumann,
                              const double* beta, const double* storage,
                              double* diag, double* fx, double* fy,
                              double* fz);
void launch_shortcut_ratio(cudaStream_t s, const Level<double>& L,
                           Reduce red);
// Sets bit 1 of scalars->marks when any Neumann boundary face is not zero.
void launch_neumann_faces(cudaStream_t s, const Level<double>& L, Scalars* scalars);
template <class TO, class TI>
void launch_convert(cudaStream_t s, size_t n, const TI* src, TO* dst);

// ---- adjoint ---------------------------------------------------------------
void launch_face_gradients(cudaStream_t s, const Level<double>& L,
                           const double* lambda, const double* p,
                           const double* fx_in, const double* fy_in,
                           const double* fz_in, double* gx, double* gy,
                           double* gz);
void launch_adjoint_source(cudaStream_t s, int n, const double* dl_dp,
                           const uint8_t* active, double* out);

}  // namespace hfps
