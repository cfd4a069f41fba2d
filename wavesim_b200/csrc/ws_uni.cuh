// Loop kernels for line lengths without a compile-time schedule of their own
// (any length that factors into two to four radices of at most 16): the same
// passes as the split step (column pass, x pencils, outer pencils), with the
// schedule chosen at run time and every radix's butterfly compiled once.
//
// A line of N = R0 R1 .. RS-1 points is transformed in place by decimation in
// frequency: stage s splits each block of n_s = N / (R0 .. Rs-1) elements
// into butterflies {j + r sub}, sub = n_s / R_s, and multiplies output r by
// W_{n_s}^{j r}.  Forward transforms go from natural order to digit-reversed
// order, inverse transforms run the stages backwards (conjugate twiddles
// first, then the butterfly) from digit-reversed to natural order.  A thread
// takes one butterfly at a time: it reads and writes the same R elements, so
// a stage needs one barrier, no second buffer, and R complex registers
// whatever N is.  Two consequences shape the passes:
//
// * The spectrum never needs its natural order: only the Green's function
//   looks at k, through tables of p that are permuted once when the solver is
//   made (uni_permutation).  In global memory, element i of the last stage's
//   butterfly u sits at u + i N / RS-1, so that consecutive threads touch
//   consecutive elements; a pass therefore starts with the last stage
//   straight from global memory, or ends with it straight into it.
// * Where an inverse transform is followed by a forward one (the column pass:
//   inverse y, f_mix, forward y; the outer pencils: forward, Green's function,
//   inverse), the last stage of the first and the first stage of the second
//   are the same butterfly on the same elements and stay in registers.  A
//   two-stage line crosses shared memory twice in the whole pass.
//
// The constants of the butterflies and the twiddles are rounded, so that a
// forward and an inverse transform in a row multiply by N (1 + g) with |g| up
// to a few 1e-8 per axis: the same in every iteration, which a solve of 200
// iterations adds up to a few 1e-6.  g is known from the schedule, as a part by
// position and one by frequency (uni_gains in ws_mbs.cu).  The first goes into
// the rounding of the ramps (k_balance_ramps), the second into the Green's
// function.  Converged fields (energies) against 64 bits on the same tables,
// without and with it: 252 x 432 4.6e-6 (2.3e-6) and 7e-7 (8e-8), 81 x 360
// 2.1e-6 (1.2e-6) and 8e-7 (1.3e-7), the latter half by the order of f_mix in
// 2-D (col_body).  The times stay within 3% (batches between compile-time columns and
// these pencils 2-6% longer).
//
// T has its y pitch rounded up to 4 elements (one 32-byte sector), so that
// the pencils' rows start on sectors for odd Ny too.
//
// Measured against the generic three-pass kernels (ws_kernels.cuh), which
// hold every radix inlined with all of a thread's elements in local memory
// (1.3-3.7 KB a thread), device time of one iteration of the launched passes:
// 125 x 144 x 99 62 us against 361, 210 x 189 x 216 305 against 2311, 1100 x
// 768 36 against 102, 63 x 77 x 70 x 3 49 against 138, 105 x 120 x 63 x 3 85
// against 490.  Single solves of 2-D grids run them in k_loop instead, where
// their columns fit the SMs' shared memory (1100 x 768: 30).  Grids whose
// passes fit the L2 are bound by the latency of a pass (load, two butterflies,
// store) and the launches; larger ones by memory, at 2-3 times the bytes' time.  The compile-time schedules stay where they exist: 192^3
// takes 153 us with them and 232 with these.
#pragma once
#include "ws_kernels.cuh"

namespace ws {
namespace uni {

constexpr int kStages = 4;
constexpr int kMaxThreads = 256;

struct Stage {
  int R;           // radix
  int sub;         // distance between the elements of a butterfly
  int units;       // butterflies of a line: n / R
  int two;         // its twiddles in the plan's table: W^{j r} at two + r sub + j
  int subp, blkp;  // sub and the block R sub in a padded column (Plan::pad)
  unsigned msub, munits;  // multipliers of the division by sub and units (magic)
};

struct Plan {
  int n, nst;
  int cls;       // kernels (kClassRadix) that its radices need
  int pad;       // columns: one slot of padding after every last-stage butterfly (its radix even), else 0
  int np;        // elements of a padded column
  unsigned mrl;  // multiplier of the division by the last stage's radix
  int ntw;       // elements of the twiddle table
  const float2* tw;
  Stage st[kStages];
};

// a / d for 0 <= a < 65536 from m = magic(d)
__host__ __device__ constexpr unsigned magic(int d) {
  return d == 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / (unsigned)d);
}
__device__ __forceinline__ int quot(int a, unsigned m) { return m ? (int)__umulhi((unsigned)a, m) : a; }

// what changes from one iteration to the next
struct ColIter {
  const float2 *gx, *gy, *gz;     // ramps of this iteration's wiggle (its conjugate ramps)
  const float2 *gx1, *gy1, *gz1;  // ramps applied before the forward transform
  const float2* src;              // added with weight A before the forward transform, or null
  double* partials;               // ROI energy of each block's columns
  int acc;                        // kAccEach ..
};

struct ColArgs {
  Geom g;
  Plan py;
  ColIter it;
  const float2* dE_in;  // forward pass: the field to transform
  float2 A;
  float2 *T, *dE, *E;
  const float2* gamma;
  const DevState* st;
  long long pitch;    // T: elements between columns
  long long fstride;  // fields: elements between right-hand sides
  long long tstride;  // T: elements between right-hand sides
  long long gstride;
  int total;          // columns of a right-hand side
  int lines;          // columns per block
  int bpr;            // blocks per right-hand side
};

struct PencilArgs {
  Geom g;
  Plan po;
  Wig w;  // p tables in the order of T
  float2 k02e, ik02e;  // k0^2 e + i e and its inverse
  float norm, norm_e;  // 1/N, and what the float lacks of it (relative)
  const float *ex, *ey, *ez;  // the gains' inverses by frequency, in the order of T
  float2* T;
  const DevState* st;
  long long pitch, tstride, cstride;  // cstride: elements between the components of T
  int lty, nyt, bpr, mode3d;  // lty: log2 of the y per block
  int pstd;  // the PSTD Laplacian instead of the Green's function; 1: output conjugated
};

struct XArgs {
  Plan px;
  float2* T;
  const DevState* st;
  long long pitch, tstride;
  int ny, nx, lty, nyt, bpr;
};

// The whole loop of a 2-D grid in one cooperative launch (k_loop): each block owns one
// column tile, whose gamma and dE' (and E') stay in its shared memory from the
// first iteration to the last, walks the pencils' tiles, and meets the others
// at a barrier in global memory after each pass.
constexpr int kLoopRhs = 16;  // right-hand sides that it takes
constexpr int kLoopThreads = 512;
constexpr long long kBarrierClocks = 2000000000LL;  // ~1 s: a bound, not a delay that ever occurs
struct LoopArgs {
  ColArgs col;
  PencilArgs pen;
  const Wig* wig;  // nw of them, the p tables in the order of T
  const float2* src;
  double* partials;  // slot i: bpr nrhs energies of iteration i of a cycle
  DevState* st;
  StopRule rule;
  Hist hist;
  unsigned* arrived;  // zero at launch
  int* err;
  long long limit;    // clocks that a block waits for the others
  long long max_cycles;  // of this launch
  int tile_elems;        // shared memory: the passes' tile, in float2
  int groups;            // energies of 32 butterflies of a column tile
  int e_resident;        // E' fits too
  int nw, nrhs;
};

// PSTD's stepping of a 2-D grid (PSTD.m:103-127) in one cooperative launch
// (k_pstd_loop): the outer pencils with the Laplacian, then the column pass
// with the leapfrog between its two transforms.  Each block keeps the two
// fields, the coefficients and the source of its columns in shared memory.
struct PstdStepAmp {
  float2 A;   // the source's amplitude in the step
  float2 ps;  // e^{i (arg A - arg A before)}
  double A2;  // |A|^2
  int may_end;  // real(A) > 0.9
};
struct PstdLoopArgs {
  ColArgs col;  // gamma: (c1, c2) per point
  PencilArgs pen;
  const float* c3;
  const float2* src;
  float2* fields;  // two of npts: step it reads (it - 1) % 2 and writes it % 2
  const PstdStepAmp* amp;  // of the launch's steps
  double* partials;
  DevState* st;
  double* hist;
  long long hist_cap, max_iter;
  double threshold;
  unsigned* arrived;
  int* err;
  long long limit;
  int steps, interval;
  int tile_elems, groups;
};

enum { kFwd = 0, kInv = 1, kStep = 2, kPstd = 3 };

// the kernels compiled for radices up to kClassRadix[c]
constexpr int kClasses = 3;
constexpr int kClassRadix[kClasses] = {8, 12, 16};
struct Kernels {
  const void* col[2][3];  // 2-D, 3-D; by kFwd, kInv, kStep
  const void* x[2];       // forward, inverse
  const void* pencil[2];  // one component, three
  const void* loop;
  const void* pstd_loop;
};
template <int RM>
Kernels kernels_up_to();

}  // namespace uni
}  // namespace ws
