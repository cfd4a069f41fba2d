// C ABI of the B200 MBS loop (declared in include/wavesim_b200.h).
//
// Host runtime: FFT planning (radix schedules, twiddle tables, tile and
// cluster shapes), device buffers, the per-solver CUDA stream, and the loop
// driver.  The loop runs as one cooperative launch (small 2-D grids), as one
// CUDA graph (first wiggle cycle with the source, then a device-side while node
// over the steady cycle whose condition the cycle's stop-rule launch sets) or,
// when a host callback needs the history, as launches from a host loop.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <memory>
#include <mutex>
#include <numeric>
#include <vector>

#include "wavesim_b200.h"
#include "ws_fast.cuh"
#include "ws_hostout.h"
#include "ws_kernels.cuh"
#include "ws_mixed.cuh"
#include "ws_tma.cuh"
#include "ws_uni.cuh"

namespace ws {

constexpr int kEmax = 16;           // max elements per thread per FFT stage
constexpr int kMaxThreadsPow2 = 512;
constexpr int kMaxThreadsMixed = 512;
constexpr size_t kSmemBudget = 150 * 1024;  // per-block tile budget (bytes)
constexpr size_t kSmemMax = 227 * 1024;     // what a block can have
constexpr int kNumSms = 148;
constexpr long long kLoopCycles = 512;  // wiggle cycles of one cooperative launch (uni::k_loop)

thread_local std::string g_last_error;

static int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

#define WS_CUDA(call)                                                                          \
  do {                                                                                         \
    cudaError_t err__ = (call);                                                                \
    if (err__ != cudaSuccess) {                                                                \
      return fail(err__ == cudaErrorMemoryAllocation ? WS_ERR_OUT_OF_MEMORY : WS_ERR_CUDA,     \
                  std::string(#call) + ": " + cudaGetErrorString(err__));                      \
    }                                                                                          \
  } while (0)

// ---------------------------------------------------------------------------
// planning
// ---------------------------------------------------------------------------
// Radix schedules of the generic kernels: 0 the largest radices first (the
// default), 1 radices of at most 8 first (more, lighter stages), 2 the
// default radices in reverse order.  Any order is a valid Stockham schedule;
// the autotuner picks one by time.
constexpr int kNumSchedules = 3;
static bool plan_radices(int n, std::vector<int>& out, int sched = 0) {
  out.clear();
  static const int pref0[] = {16, 12, 13, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  static const int pref1[] = {8, 7, 6, 5, 4, 3, 9, 10, 11, 12, 13, 16, 2};
  const int* pref = sched == 1 ? pref1 : pref0;
  while (n > 1) {
    bool found = false;
    for (int i = 0; i < 13; ++i) {
      const int r = pref[i];
      if (n % r == 0) {
        out.push_back(r);
        n /= r;
        found = true;
        break;
      }
    }
    if (!found) return false;
  }
  if (sched == 2) std::reverse(out.begin(), out.end());
  return (int)out.size() <= kMaxStages;
}

static bool length_supported(int n) {
  std::vector<int> r;
  return n >= 1 && n <= 65536 && plan_radices(n, r);
}

// Fast power-of-two kernels (ws_fast.cuh), instantiated for these shapes.
struct FastInner {
  int n, c, do_x;
  const void* fwd;
  const void* inv;
  size_t smem;      // bytes (3-D, enough for both kernels); 2-D: bytes per held column, one extra column of scratch
  size_t smem_fwd, smem_inv;  // 3-D: what each kernel needs
  const void* fused = nullptr;  // K3 of one iteration + K1 of the next (3-D planes on a cluster), or null
  size_t smem_fused = 0;
  const void* fused_tma = nullptr;  // the same with K3's rows loaded by a tensor copy (first argument: the map)
  const void* col_step = nullptr;   // the column pass of the split fused step (kc_col_step), or null
  size_t smem_col = 0;              // its dynamic shared memory (kc_col_step2d, kmc_col_step)
  int lines = 0;                    // 2-D: columns per block (0: 4096 / N, 16 elements per thread)
};
struct FastPencil {
  int no, ty;
  const void* fn;
  int nc;        // components it transforms together (1, or 3 with the dyadic Green's function)
  int threads;
  size_t smem;
  int dims;      // 3: z pencils of 3-D grids only; 2: x pencils of 2-D grids only; 0: both
};

template <int N, int C, bool DX>
static FastInner fast_inner() {
  using G = fast::PlaneGeom<N, C, DX>;
  FastInner f{N, C, DX ? 1 : 0, (const void*)fast::kf_plane_fwd<N, C, DX>,
              (const void*)fast::kf_plane_inv<N, C, DX>, DX ? G::smem : (size_t)G::CS * sizeof(float2),
              DX ? (G::PUSH ? G::smem_push : G::smem_a) : 0, DX ? G::smem_max_ab : 0};
  if constexpr (DX) {
    f.col_step = (const void*)fast::kc_col_step<N, C>;
  } else {
    f.col_step = (const void*)fast::kc_col_step2d<N>;
    f.smem_col = fast::smem_col_step2d<N>();
  }
  if constexpr (DX && C > 1) {
    if constexpr (C >= 16) {  // small tiles: the column tile and the row tile fit side by side
      f.fused = (const void*)fast::kf_plane_fused_push<N, C>;
      f.smem_fused = fast::FusedPushGeom<N, C>::smem;
    } else {
      f.fused = (const void*)fast::kf_plane_fused<N, C>;
      f.fused_tma = (const void*)fast::kf_plane_fused_tma<N, C>;
      f.smem_fused = G::smem_max_ab;
    }
  }
  return f;
}
template <int NO, int TY>
static FastPencil fast_pencil() {
  return FastPencil{NO, TY, (const void*)fast::kf_pencil<NO, TY>, 1, TY * (NO / 16),
                    (size_t)(TY + 1) * NO * sizeof(float2), 0};
}
// mixed-radix / vector kernels (ws_mixed.cuh)
using Plan192 = mixed::Plan<192, 12, 12, 4, 4>;
using Plan96 = mixed::Plan<96, 12, 12, 4, 2>;
using Plan160 = mixed::Plan<160, 20, 10, 4, 4>;
using Plan224 = mixed::Plan<224, 28, 14, 4, 4>;
// (radix orders by register use: 5 x 4 x 4 x 4 spilled 416 bytes a thread in
// the 2-D column pass, 4 x 4 x 4 x 5 16; 7 x 4 x 4 x 4 84, 14 x 4 x 4 x 2 40)
using Plan320 = mixed::Plan<320, 20, 4, 4, 4, 5>;
using Plan448 = mixed::Plan<448, 28, 14, 4, 4, 2>;
using Plan576 = mixed::Plan<576, 36, 12, 12, 4>;
template <class PL, int C>
static FastInner mixed_inner() {
  using G = mixed::MGeom<PL, C>;
  FastInner f{PL::N, C, 1, (const void*)mixed::km_plane_fwd<PL, C>, (const void*)mixed::km_plane_inv<PL, C>,
              G::smem, G::smem, G::smem};
  f.fused = (const void*)mixed::km_plane_fused<PL, C>;
  f.fused_tma = (const void*)mixed::km_plane_fused_tma<PL, C>;
  f.col_step = (const void*)mixed::kmc_col_step<PL, C>;
  f.smem_col = mixed::smem_col_step<PL, C>();
  f.smem_fused = G::smem;
  static_assert((size_t)PL::N * G::LR * sizeof(float2) + 128 <= G::smem, "the dense row tile fits");
  return f;
}
// 2-D columns on the mixed-radix lines (kmc_col_*2d), one round of lines per block
template <class PL>
static FastInner mixed_inner2d() {
  using G = mixed::MGeom2d<PL>;
  FastInner f{PL::N, 1, 0, (const void*)mixed::kmc_col_fwd2d<PL>, (const void*)mixed::kmc_col_inv2d<PL>,
              (size_t)G::CS * sizeof(float2), 0, 0};
  f.col_step = (const void*)mixed::kmc_col_step2d<PL>;
  f.smem_col = mixed::smem_col_step2d<PL>();
  f.lines = G::LPR;
  return f;
}
// z pencils of 3-D grids (one or three components), and x pencils of 2-D grids (one)
template <class PL, int TY, int NC>
static FastPencil mixed_pencil() {
  return FastPencil{PL::N, TY, (const void*)mixed::km_pencil<PL, TY, NC, true>, NC, TY * PL::P,
                    (size_t)(TY + 1) * PL::N * sizeof(float2), 3};
}
template <class PL, int TY>
static FastPencil mixed_pencil2d() {
  return FastPencil{PL::N, TY, (const void*)mixed::km_pencil<PL, TY, 1, false>, 1, TY * PL::P,
                    (size_t)(TY + 1) * PL::N * sizeof(float2), 2};
}

static const std::vector<FastInner>& fast_inner_table() {
  // 96^2 planes on 3 blocks (288 column-pass blocks at 96^3): 24.9 us an
  // iteration against 29.6 with one block per plane (96 of the 148 SMs);
  // 128^2 on 2: 41.5 against 43.8 on 4
  static const std::vector<FastInner> t = {
      fast_inner<64, 1, true>(),     fast_inner<128, 2, true>(),    fast_inner<256, 8, true>(),
      fast_inner<256, 16, true>(),
      fast_inner<64, 1, false>(),    fast_inner<128, 1, false>(),   fast_inner<256, 1, false>(),
      fast_inner<512, 1, false>(),   fast_inner<1024, 1, false>(),  fast_inner<2048, 1, false>(),
      mixed_inner<Plan192, 6>(),     mixed_inner<Plan96, 3>(),      mixed_inner<Plan160, 5>(),
      mixed_inner<Plan224, 7>(),
      mixed_inner2d<Plan192>(),      mixed_inner2d<Plan320>(),      mixed_inner2d<Plan448>(),
      mixed_inner2d<Plan576>()};
  return t;
}
// Persistent TMA-pipelined K2 (ws_tma.cuh) for z pencils of a 3-D grid.
struct TmaPencil {
  int no, ty, stages;
  const void* fn;
  size_t smem;
  int threads;
  int nc = 1;  // components (3: the vector form, kt_pencil_vec)
};
template <int NO, int TY, int S>
static TmaPencil tma_pencil() {
  using PT = tma::PencilTile<NO, TY, S>;
  return TmaPencil{NO, TY, S, (const void*)tma::kt_pencil<NO, TY, S>, PT::smem, PT::kThreads};
}
template <class PL, int TY, int S>
static TmaPencil tma_pencil_vec() {
  using PT = tma::VecPencilTile<PL, TY, S>;
  return TmaPencil{PL::N, TY, S, (const void*)tma::kt_pencil_vec<PL, TY, S>, PT::smem, PT::kThreads, 3};
}
// The x passes of the split fused step (kt_xpencil, ws_tma.cuh).
struct XPencil {
  int no, ty, stages;
  const void* fwd;
  const void* inv;
  size_t smem;
  int threads;
};
template <int NO, int TY, int S>
static XPencil x_pencil() {
  using PT = tma::PencilTile<NO, TY, S>;
  return XPencil{NO, TY, S, (const void*)tma::kt_xpencil<NO, TY, S, false>,
                 (const void*)tma::kt_xpencil<NO, TY, S, true>, PT::smem, PT::kThreads};
}
template <class PL, int TY, int S>
static XPencil x_pencil_m() {
  using PT = tma::MixedXTile<PL, TY, S>;
  return XPencil{PL::N, TY, S, (const void*)tma::kt_xpencil_m<PL, TY, S, false>,
                 (const void*)tma::kt_xpencil_m<PL, TY, S, true>, PT::smem, PT::kThreads};
}
static const std::vector<XPencil>& x_pencil_table() {
  // the first match of (no, ty) is the default
  static const std::vector<XPencil> t = {x_pencil<64, 16, 3>(), x_pencil<128, 16, 3>(), x_pencil<256, 8, 3>(),
                                         x_pencil<256, 8, 4>(), x_pencil<256, 16, 3>(), x_pencil<256, 8, 2>(),
                                         x_pencil_m<Plan192, 8, 4>(),
                                         x_pencil_m<Plan192, 16, 3>(), x_pencil_m<Plan96, 16, 3>(),
                                         x_pencil_m<Plan160, 16, 3>(), x_pencil_m<Plan224, 16, 3>()};
  return t;
}
using Plan192t = mixed::Plan<192, 12, 12, 4, 4>;
static const std::vector<TmaPencil>& tma_pencil_table() {
  // the first match of (no, ty) is the default; the autotuner tries the rest
  // (at 256: 8 y x 3 stages, 4 blocks of 128 threads per SM at 128 registers,
  // measured 0.0667 ms against 0.0732 for 8 x 4 stages at 3 blocks per SM,
  // 0.070 for 16 x 3, 0.081 for 4 x 4 and 0.096 for 8 x 6)
  static const std::vector<TmaPencil> t = {tma_pencil<64, 16, 3>(), tma_pencil<128, 16, 3>(),
                                           tma_pencil<256, 8, 3>(),  tma_pencil<256, 8, 4>(),
                                           tma_pencil<256, 8, 2>(),  tma_pencil<256, 16, 3>(),
                                           tma_pencil<256, 16, 2>(), tma_pencil<256, 8, 6>(),
                                           tma_pencil<256, 4, 4>(),
                                           // 192 x 3 components, one at a time in registers: 8 y x 2 stages
                                           // (3 blocks per SM) measured 0.120 ms at 192^3 against 0.143
                                           // (8 x 3), 0.154 (4 x 3) and 0.145 (16 x 2); all three lines in
                                           // registers took 0.131 at best
                                           tma_pencil_vec<Plan192t, 8, 2>(), tma_pencil_vec<Plan192t, 8, 3>(),
                                           tma_pencil_vec<Plan192t, 4, 3>(), tma_pencil_vec<Plan192t, 16, 2>()};
  return t;
}

// ... for the x pencils of 2-D grids, in batches
template <int NO, int TY, int S>
static TmaPencil tma_pencil2d() {
  using PT = tma::PencilTile<NO, TY, S>;
  return TmaPencil{NO, TY, S, (const void*)tma::kt_pencil<NO, TY, S, false>, PT::smem, PT::kThreads};
}
static const std::vector<TmaPencil>& tma_pencil2d_table() {
  // 16 x 1024^2: 4 y x 3 stages 267 us an iteration, 8 x 3 271, 4 x 2 (80
  // registers) 371; kf_pencil (32-byte rows, nothing in flight while it
  // computes) 336.  64 x 512^2: 8 x 3 220, 4 x 3 231, 8 x 2 270, kf_pencil 254
  static const std::vector<TmaPencil> t = {tma_pencil2d<1024, 4, 3>(), tma_pencil2d<512, 8, 3>()};
  return t;
}

static const std::vector<FastPencil>& fast_pencil_table() {
  static const std::vector<FastPencil> t = {
      fast_pencil<32, 16>(),  fast_pencil<64, 16>(),  fast_pencil<128, 16>(),
      fast_pencil<256, 16>(), fast_pencil<512, 8>(),  fast_pencil<1024, 4>(),
      mixed_pencil<Plan192, 8, 3>(),   // (a TY = 8 variant first: the later TY = 16 is the default)
      mixed_pencil<Plan192, 16, 1>(),
      mixed_pencil<Plan192, 16, 3>(),
      mixed_pencil<Plan96, 16, 1>(),
      mixed_pencil<Plan96, 16, 3>(),
      mixed_pencil<Plan160, 16, 1>(),
      mixed_pencil<Plan224, 16, 1>(),
      mixed_pencil2d<Plan192, 16>(),
      mixed_pencil2d<Plan320, 8>(),
      mixed_pencil2d<Plan448, 8>(),
      mixed_pencil2d<Plan576, 8>(),
      mixed_pencil<mixed::Plan<64, 16, 16, 4>, 16, 3>(),
      mixed_pencil<mixed::Plan<128, 16, 16, 8>, 16, 3>(),
      mixed_pencil<mixed::Plan<256, 16, 16, 16>, 16, 3>()};
  return t;
}

// A pass of the run-time scheduled kernels (ws_uni.cuh).
struct UniPass {
  uni::Plan plan{};
  int lines = 0;  // column pass: columns per block; pencils: consecutive y per block
  int threads = 0;
  size_t smem = 0;
  long long grid = 0;  // blocks of a right-hand side
};

// The line's schedule: the fewest stages of radices 2 .. 16, of those the
// smallest largest radix (registers), then the smallest sum; in ascending
// order, so that the column pass's epilogue (stage 0) has the fewest elements
// in registers.  False where the length has none (1, primes, factors above 16).
static bool uni_plan(int n, uni::Plan& P) {
  int best[uni::kStages] = {}, best_n = 0, best_max = 1 << 30, best_sum = 1 << 30;
  int cur[uni::kStages];
  auto search = [&](auto&& self, int left, int from, int k) -> void {
    if (left == 1) {
      if (k < 2) return;
      int sum = 0;
      for (int i = 0; i < k; ++i) sum += cur[i];
      if (best_n && (k > best_n || (k == best_n && (cur[k - 1] > best_max || (cur[k - 1] == best_max && sum >= best_sum)))))
        return;
      best_n = k;
      best_max = cur[k - 1];
      best_sum = sum;
      std::copy(cur, cur + k, best);
      return;
    }
    if (k == uni::kStages) return;
    for (int r = from; r <= 16 && r <= left; ++r)
      if (left % r == 0) {
        cur[k] = r;
        self(self, left / r, r, k + 1);
      }
  };
  search(search, n, 2, 0);
  if (!best_n) return false;
  P = uni::Plan{};
  P.n = n;
  P.nst = best_n;
  P.cls = 0;
  while (uni::kClassRadix[P.cls] < best_max) ++P.cls;
  const int rl = best[best_n - 1];
  P.pad = rl % 2 == 0 ? 1 : 0;
  auto padded = [&](int i) { return i + (P.pad ? i / rl : 0); };
  P.np = padded(n);
  P.mrl = uni::magic(rl);
  int block = n;
  for (int s = 0; s < best_n; ++s) {
    uni::Stage& S = P.st[s];
    S.R = best[s];
    S.sub = block / S.R;
    S.units = n / S.R;
    S.subp = padded(S.sub);
    S.blkp = padded(block);
    S.msub = uni::magic(S.sub);
    S.munits = uni::magic(S.units);
    S.two = P.ntw;
    P.ntw += block;
    block = S.sub;
  }
  return true;
}

// W_n^{j r} of a stage on blocks of n
static float2 uni_twiddle(int j, int r, int n) {
  const double a = -2.0 * M_PI * (double)((long long)j * r % n) / (double)n;
  return make_float2((float)std::cos(a), (float)std::sin(a));
}

// The frequency of each element of a forward transform in the order of T.
static std::vector<int> uni_permutation(const uni::Plan& P) {
  std::vector<int> k(P.n);
  const uni::Stage& L = P.st[P.nst - 1];
  for (int u = 0; u < L.units; ++u) {
    int rev = 0, w = 1, rest = u, span = L.units;
    for (int s = 0; s < P.nst - 1; ++s) {  // digit of stage s, the most significant first
      span /= P.st[s].R;
      rev += w * (rest / span);
      rest %= span;
      w *= P.st[s].R;
    }
    for (int i = 0; i < L.R; ++i) k[u + i * L.units] = rev + i * L.units;
  }
  return k;
}

// |w| - 1 of a rounded twiddle
static double excess(float2 w) { return 0.5 * ((double)w.x * w.x + (double)w.y * w.y - 1.0); }

// The rounded constants of the butterflies and the twiddles make a forward and
// an inverse transform in a row multiply by N (1 + a few 1e-8) instead of N, the same
// in every iteration of a solve.  To first order the factor is 1 + p + f: p a
// function of the position (each stage's butterfly on that input, and the mean
// |W|^2 - 1 of its twiddles over the butterfly's outputs), f one of the frequency with
// a mean of zero (the butterflies' outputs, and the mean over the positions).
// pos: p of j + r n / R0 is pos[j] + round_trip(1, R0, r); freq, in the order of
// T: f of u + i n / RL is freq[u] + round_trip(0, RL, i) (both are 0 for r = i = 0).
// tw: the plan's twiddles.
static void uni_gains(const uni::Plan& P, const float2* tw, std::vector<double>& pos, std::vector<double>& freq) {
  pos.assign(P.n, 0.0);
  freq.assign(P.n, 0.0);
  double mean = 0.0;
  for (int s = 0, span = P.n; s < P.nst; ++s) {
    const uni::Stage& S = P.st[s];
    std::vector<double> tin(S.sub, 0.0), out(S.R, 0.0);
    for (int r = 0; r < S.R; ++r) {
      for (int j = 0; j < S.sub; ++j) {
        const double g = 2.0 * excess(tw[S.two + r * S.sub + j]);
        tin[j] += g / S.R;
        out[r] += g / S.sub;
      }
      out[r] += round_trip(0, S.R, r);
      mean += out[r] / S.R;
    }
    for (int i = 0; i < P.n; ++i) pos[i] += tin[i % S.sub] + round_trip(1, S.R, i / S.sub % S.R);
    // the digit of stage s of element u + i n / RL: of u, or i
    const int units = P.st[P.nst - 1].units;
    span = s < P.nst - 1 ? span / S.R : 1;
    for (int k = 0; k < P.n; ++k)
      freq[k] += s < P.nst - 1 ? out[k % units / (span / P.st[P.nst - 1].R) % S.R] : out[k / units];
  }
  for (double& f : freq) f -= mean;
}

// The same for the compile-time schedules of columns (Stockham: stage s takes
// the digit of weight N / (R0 .. Rs) of its input, multiplies it by W_{Ns Rs}^{jm r},
// jm the digits of the output so far, and gives the output's digit of weight
// Ns = R0 .. Rs-1; the inverse is the same with conjugate constants).
static void line_gains(const std::vector<int>& radix, std::vector<double>& pos, std::vector<double>& freq) {
  const int n = std::accumulate(radix.begin(), radix.end(), 1, std::multiplies<int>());
  pos.assign(n, 0.0);
  freq.assign(n, 0.0);
  int Ns = 1, rest = n;
  for (int R : radix) {
    rest /= R;
    std::vector<double> by_input(R, 0.0), by_output(Ns, 0.0);  // of the twiddles
    for (int r = 0; r < R; ++r)
      for (int j = 0; j < Ns; ++j) {
        const double g = excess(uni_twiddle(j, r, Ns * R));
        by_input[r] += g / Ns;
        by_output[j] += g / R;
      }
    for (int i = 0; i < n; ++i) {
      const int in = i / rest % R, out = i / Ns % R;
      pos[i] += butterfly_gain(0, R, in) + by_input[in] + butterfly_gain(3, R, out) + by_output[i % Ns];
      freq[i] += butterfly_gain(1, R, out) + by_output[i % Ns] + butterfly_gain(2, R, in) + by_input[in];
    }
    Ns *= R;
  }
  const double mean = std::accumulate(freq.begin(), freq.end(), 0.0) / n;
  for (double& f : freq) f -= mean;
}

static int uni_units(const uni::Plan& P) {
  int m = 1;
  for (int s = 0; s < P.nst; ++s) m = std::max(m, P.st[s].units);
  return m;
}

// energies that a block of the column pass sums: one per 32 butterflies of its first stage
static int uni_groups(const UniPass& p) { return (p.lines * p.plan.st[0].units + 31) / 32; }

// The column pass: one butterfly per thread, as many columns as fill 256 threads,
// fewer where the grid would not give every SM two blocks, at least a warp.
static void uni_columns(UniPass& p, long long total, int lines = 0) {
  const int um = uni_units(p.plan);
  const long long most = std::max(1, uni::kMaxThreads / um), least = (32 + um - 1) / um;
  long long l = std::min(most, std::max(least, total / (2 * kNumSms)));
  while (l > 1 && l * p.plan.np * sizeof(float2) > 64 * 1024) l /= 2;
  p.lines = lines ? lines : (int)std::min(l, total);
  p.threads = (int)std::min<long long>(uni::kMaxThreads, (p.lines * (long long)um + 31) / 32 * 32);
  p.smem = p.lines * (p.plan.np * sizeof(float2) + 32) + 2 * p.plan.n * sizeof(float2) + uni_groups(p) * sizeof(float);
  p.grid = (total + p.lines - 1) / p.lines;
}

// Pencils: 16 consecutive y (one 128-byte row segment) per block, 8 where a
// butterfly per thread would not fit 256 threads or the tile 72 KB (three
// blocks per SM), down to 4 (one sector) where the grid would not give every
// SM two blocks.  Measured at 150 x 80 x 198 (66 butterflies a line): 8 y with
// two butterflies per thread 93 us an iteration, 4 y 105 us; at 512^2 4 y 21.8
// us, 8 y (64 blocks) 24.8 us.
static void uni_pencils(UniPass& p, int ny, int nc, long long mids) {
  const int um = uni_units(p.plan);
  const size_t row = (size_t)nc * p.plan.n * sizeof(float2);
  int ty = 16;
  while (ty > 8 && (ty * um > uni::kMaxThreads || ty * row > 72 * 1024)) ty /= 2;
  while (ty > 4 && (ny + ty - 1) / ty * mids < 2 * kNumSms) ty /= 2;
  while (ty > 1 && ty * row > 150 * 1024) ty /= 2;
  p.lines = ty;
  int w = std::max(1, std::min(um, uni::kMaxThreads / ty));
  while ((w * ty) % 32 && w * ty + ty <= uni::kMaxThreads) ++w;
  p.threads = w * ty;
  p.smem = ty * row + (p.plan.n + p.plan.st[p.plan.nst - 1].units) * sizeof(float);
  p.grid = (long long)((ny + ty - 1) / ty) * mids;
}

static const uni::Kernels& uni_kernels(int cls) {
  static const uni::Kernels t[uni::kClasses] = {uni::kernels_up_to<uni::kClassRadix[0]>(),
                                                uni::kernels_up_to<uni::kClassRadix[1]>(),
                                                uni::kernels_up_to<uni::kClassRadix[2]>()};
  return t[cls];
}

struct Layout {
  const FastInner* fi = nullptr;   // fast K1/K3, or null (generic)
  const FastPencil* fp = nullptr;  // fast K2, or null (generic)
  const TmaPencil* tp = nullptr;   // persistent TMA K2 (takes precedence over fp), or null
  const TmaPencil* tp2 = nullptr;  // persistent TMA x pencils of 2-D grids, for batches, or null
  const XPencil* xp = nullptr;     // x passes of the split fused step, or null (one-kernel fused step)
  int rset = kPow2;  // radix set of every plan of the solver
  int mode3d = 0;
  int csize = 1;     // 3-D: blocks (cluster) per plane
  int ncols = 1;     // 2-D: columns per block
  int ty = 16;       // outer pass: consecutive y per block
  int th_inner = 256, th_outer = 256;
  size_t smem_inner = 0, smem_outer = 0;
  long long grid_inner = 0, grid_outer = 0;
  bool uni_in = false, uni_out = false;  // the run-time scheduled kernels for the inner / the outer pass
  UniPass ucol, ux, uout;
  long long pitch = 0;  // elements between the columns of T
};

static int log2_of(int n) { return n > 1 ? 1 + log2_of(n / 2) : 0; }
static bool is_pow2(long long n) { return n >= 1 && (n & (n - 1)) == 0; }

// Overrides of the layout heuristics, for the autotuner (0 = heuristic).
struct LayoutChoice {
  int inner = 0;  // 1: fast inner kernels when a shape matches, 2: generic
  int outer = 0;  // 1: fast pencil when a shape matches, 2: generic, 3 + k: TMA pencil of k stages
  int csize = 0;  // 3-D generic: smallest blocks per plane to try
  int ncols = 0;  // 2-D generic: columns per block
  int ty = 0;     // generic outer: consecutive y per block
  int sched = 0;  // radix schedule of the generic kernels' plans (plan_radices)
  int xp = 0;     // split step: 1 + index of the x pencil in x_pencil_table (0: the default)
  bool operator==(const LayoutChoice& o) const {
    return inner == o.inner && outer == o.outer && csize == o.csize && ncols == o.ncols && ty == o.ty &&
           sched == o.sched && xp == o.xp;
  }
};

// The loop of a 2-D grid in one launch: a column tile per SM, the tables of
// all nw wiggles, gamma and dE' of the tile (E' where it fits) in shared memory.
static size_t loop_smem(const Layout& L, const Geom& g, int nw, bool e_resident, int* tile_elems = nullptr) {
  const size_t l = L.ucol.lines;
  const size_t tile = std::max(l * L.ucol.plan.np, (size_t)L.uout.lines * L.uout.plan.n);
  if (tile_elems) *tile_elems = (int)tile;
  const size_t tables = L.ucol.plan.ntw + L.uout.plan.ntw + nw * (g.ny + l);
  return (tile + tables + l * g.ny * (e_resident ? 3 : 2)) * sizeof(float2) + l * 16 +
         (uni_groups(L.ucol) + (size_t)nw * L.uout.plan.n + L.uout.plan.st[L.uout.plan.nst - 1].units) * sizeof(float);
}
constexpr size_t kLoopSmem = 225 * 1024;
// ... of PSTD's stepping: two fields, the source and three coefficients a point
static size_t pstd_loop_smem(const Layout& L, const Geom& g, int* tile_elems = nullptr) {
  const size_t l = L.ucol.lines;
  const size_t tile = std::max(l * L.ucol.plan.np, (size_t)L.uout.lines * L.uout.plan.n);
  if (tile_elems) *tile_elems = (int)tile;
  return (tile + L.ucol.plan.ntw + L.uout.plan.ntw + 4 * l * g.ny) * sizeof(float2) + l * 16 +
         (uni_groups(L.ucol) + (size_t)L.uout.plan.n + l * g.ny + L.uout.plan.st[L.uout.plan.nst - 1].units) * sizeof(float);
}
// The layout of single solves of small 2-D grids, `L` being the one of the
// grid's launched passes; false if there is none.  Measured against the
// launched passes, us an iteration: 64 x 56 7.6 (12.8), 160 x 264 12.4 (21.4),
// 396 x 315 11.0 (19.7), 512^2 12.6 (18.8, compile-time kernels), 632^2 20.3
// (23.9), 1100 x 768 30 (38); 1024^2 38.7 (34.2, compile-time kernels).  So
// it takes every grid whose columns fit the SMs' shared memory, but those with
// compile-time kernels in both passes only up to 400 000 points.  A choice of
// the launched passes' kernels (the autotuner's, which times only those) leaves
// it as it is: `heuristic` is their layout without one.
static bool loop_layout(const Geom& g, const Layout& heuristic, bool pstd, Layout& out) {
  const Layout& L = heuristic;
  if (L.mode3d || g.nc != 1) return false;
  const char* path = std::getenv("WAVESIM_B200_PATH");
  if (path && std::strcmp(path, "generic") == 0) return false;
  if (L.fi && L.fp && g.npts > 400000 && !pstd) return false;
  Layout t{};
  if (!uni_plan(g.nx, t.uout.plan) || !uni_plan(g.ny, t.ucol.plan)) return false;
  t.uni_in = t.uni_out = true;
  uni_pencils(t.uout, g.ny, 1, 1);
  // a tile per SM; up to 8192 points the tiles of 16 SMs, which then form one
  // cluster and meet at its hardware barrier (64 x 56: 7.6 us against 8.6)
  const int sms = t.uout.grid <= 16 && g.npts <= 8192 ? 16 : kNumSms;
  uni_columns(t.ucol, g.nx, (g.nx + sms - 1) / sms);
  if ((pstd ? pstd_loop_smem(t, g) : loop_smem(t, g, 4, false)) > kLoopSmem) return false;
  t.grid_inner = t.ucol.grid;
  t.grid_outer = t.uout.grid;
  t.rset = L.rset;
  t.pitch = (g.ny + 3) / 4 * 4;
  out = t;
  return true;
}

static int make_layout(const Geom& g, Layout& L, std::string& why, const LayoutChoice& ch = LayoutChoice{},
                       bool pstd = false) {
  L = Layout{};
  L.pitch = g.ny;
  L.mode3d = g.nz > 1;
  L.rset = kPow2;
  for (long long n : {(long long)g.ny, (long long)g.nx, (long long)g.nz})
    if (!is_pow2(n)) L.rset = kMixed;
  const int kMaxThreads = L.rset == kPow2 ? kMaxThreadsPow2 : kMaxThreadsMixed;
  auto threads_for = [&](long long elems) {
    long long t = (elems + kEmax - 1) / kEmax;
    t = ((t + 31) / 32) * 32;
    return (int)std::max(32LL, std::min((long long)kMaxThreads, t));
  };
  const int ny = g.ny;
  const size_t col_bytes = (size_t)padded(ny) * sizeof(float2);
  if (L.mode3d) {
    // smallest divisor C of Nx (<= 16) whose tile fits
    int best = 0;
    for (int c = ch.csize ? ch.csize : 1; c <= 16; ++c) {
      if (g.nx % c) continue;
      const long long cols = g.nx / c;
      const long long elems = cols * ny;
      if (elems > (long long)kMaxThreads * kEmax) continue;
      if (cols * col_bytes > kSmemBudget) continue;
      if (c > 1 && !length_supported((int)cols)) continue;
      best = c;
      break;
    }
    if (!best) {
      why = "an Ny x Nx plane of this size does not fit a cluster of 16 blocks";
      return WS_ERR_UNSUPPORTED;
    }
    L.csize = best;
    const long long cols = g.nx / best;
    L.th_inner = threads_for(cols * ny);
    L.smem_inner = cols * col_bytes;
    L.grid_inner = (long long)g.nz * g.nc * best;
  } else {
    const long long total_cols = (long long)g.nx * g.nc;
    const long long max_cols_fit = std::max(1LL, std::min((long long)(kSmemBudget / col_bytes),
                                                          (long long)kMaxThreads * kEmax / (long long)ny));
    if ((long long)ny > (long long)kMaxThreads * kEmax || col_bytes > kSmemBudget) {
      why = "Ny too large for one block";
      return WS_ERR_UNSUPPORTED;
    }
    // aim for >= 2 blocks per SM, at most ~8K elements per block
    long long want = std::max(1LL, std::min(max_cols_fit, (8192LL + ny - 1) / ny));
    while (want > 1 && (total_cols + want - 1) / want < 2 * kNumSms) want /= 2;
    if (ch.ncols) want = std::max(1LL, std::min<long long>(ch.ncols, max_cols_fit));
    L.ncols = (int)want;
    L.th_inner = threads_for((long long)want * ny);
    L.smem_inner = want * col_bytes;
    L.grid_inner = (total_cols + want - 1) / want;
  }
  // outer pass
  const int no = L.mode3d ? g.nz : g.nx;
  const long long mids = L.mode3d ? g.nx : 1;
  int ty = 16;
  while (ty > 1 && ((long long)padded(g.nc * ty) * no * sizeof(float2) > kSmemBudget ||
                    (long long)g.nc * ty * no > (long long)kMaxThreads * kEmax))
    ty /= 2;
  if (ty > g.ny) ty = std::max(1, g.ny);
  while (ty > 4 && ((g.ny + ty - 1) / ty) * mids < 2 * kNumSms) ty /= 2;
  if (ch.ty) ty = std::max(1, std::min(ch.ty, g.ny));
  if ((long long)padded(g.nc * ty) * no * sizeof(float2) > kSmemBudget ||
      (long long)g.nc * ty * no > (long long)kMaxThreads * kEmax) {
    why = "outer dimension too long for one block";
    return WS_ERR_UNSUPPORTED;
  }
  L.ty = ty;
  L.th_outer = threads_for((long long)g.nc * ty * no);
  L.smem_outer = (size_t)padded(g.nc * ty) * no * sizeof(float2);
  L.grid_outer = (long long)((g.ny + ty - 1) / ty) * mids;
  // fast power-of-two kernels where a shape matches
  const char* path = std::getenv("WAVESIM_B200_PATH");
  if (path && std::strcmp(path, "generic") == 0) return WS_OK;
  // 3-D: the first plane kernel of the grid's size, or the one with the
  // cluster size asked for (autotuner: ch.csize; WAVESIM_B200_CLUSTER)
  int want_c = ch.csize;
  if (!want_c)
    if (const char* e = std::getenv("WAVESIM_B200_CLUSTER")) want_c = std::atoi(e);
  const FastInner* first3 = nullptr;
  const FastInner* pick3 = nullptr;
  for (const FastInner& f : fast_inner_table()) {
    if (ch.inner == 2) break;
    if (L.mode3d && f.do_x && g.ny == f.n && g.nx == f.n) {
      if (!first3) first3 = &f;
      if (want_c && f.c == want_c) pick3 = &f;
    }
    if (!L.mode3d && !f.do_x && g.ny == f.n) L.fi = &f;
  }
  if (L.mode3d) L.fi = pick3 ? pick3 : first3;
  if (L.fi && !L.mode3d) {
    // one round of lines per block: 256 threads, 16 elements each (mixed-radix lines: E each)
    const long long total_cols = (long long)g.nx * g.nc;
    const long long want = L.fi->lines ? L.fi->lines : std::max(1, 4096 / g.ny);
    L.ncols = (int)want;
    L.grid_inner = (total_cols + want - 1) / want;
  }
  if (L.fi && L.mode3d) L.grid_inner = (long long)g.nz * g.nc * L.fi->c;
  if (ch.outer != 2) {
    // the last pencil of the shape, or the one with the y tile asked for
    // (autotuner: outer = 1 with ty; WAVESIM_B200_PENCIL_TY)
    int want_ty = ch.outer == 1 ? ch.ty : 0;
    if (!want_ty)
      if (const char* e = std::getenv("WAVESIM_B200_PENCIL_TY")) want_ty = std::atoi(e);
    for (const FastPencil& f : fast_pencil_table())
      if (f.no == no && g.ny % f.ty == 0 && f.nc == g.nc && (f.dims == 0 || f.dims == (L.mode3d ? 3 : 2)) && (!want_ty || f.ty == want_ty))
        L.fp = &f;
  }
  if (L.fp) L.grid_outer = (long long)(g.ny / L.fp->ty) * mids;  // blocks of the fast pencil kernel
  // the TMA pencil where a shape matches: by default (WAVESIM_B200_K2=plain keeps kf_pencil), or the
  // autotuner's choice of stages
  const char* k2 = std::getenv("WAVESIM_B200_K2");
  const bool tma_ok = L.mode3d && (ch.outer == 0 || ch.outer >= 3) &&
                      !(ch.outer == 0 && k2 && std::strcmp(k2, "plain") == 0);
  int want_tty = 0, want_ts = 0;  // WAVESIM_B200_TMA_TY / _TMA_STAGES: the y tile and stages of the TMA pencil
  if (const char* e = std::getenv("WAVESIM_B200_TMA_TY")) want_tty = std::atoi(e);
  if (const char* e = std::getenv("WAVESIM_B200_TMA_STAGES")) want_ts = std::atoi(e);
  if (tma_ok)
    for (const TmaPencil& f : tma_pencil_table())
      if (f.no == no && f.nc == g.nc && g.ny % f.ty == 0 && (ch.outer < 3 || f.stages == ch.outer - 3) &&
          (!want_tty || f.ty == want_tty) && (!want_ts || f.stages == want_ts)) {
        L.tp = &f;
        break;
      }
  if (!L.mode3d && g.nc == 1 && L.fp && ch.outer == 0 && !(k2 && std::strcmp(k2, "plain") == 0))
    for (const TmaPencil& f : tma_pencil2d_table())
      if (f.no == no && g.ny % f.ty == 0 && (!want_tty || f.ty == want_tty) && (!want_ts || f.stages == want_ts)) {
        L.tp2 = &f;
        break;
      }
  // the split fused step (x pencils + column pass) on power-of-two planes;
  // WAVESIM_B200_STEP=cluster keeps the one-kernel step with the cluster
  // exchange, WAVESIM_B200_XTY picks the x pencils' y tile
  const char* step = std::getenv("WAVESIM_B200_STEP");
  int want_xty = 0, want_xs = 0;  // WAVESIM_B200_XTY / _XSTAGES: the y tile and stages of the x pencils
  if (const char* e = std::getenv("WAVESIM_B200_XTY")) want_xty = std::atoi(e);
  if (const char* e = std::getenv("WAVESIM_B200_XSTAGES")) want_xs = std::atoi(e);
  if (L.mode3d && L.fi && L.fi->col_step && !(step && std::strcmp(step, "cluster") == 0)) {
    const auto& xt = x_pencil_table();
    if (ch.xp > 0 && ch.xp <= (int)xt.size()) {
      const XPencil& f = xt[ch.xp - 1];
      if (f.no != g.nx || g.ny % f.ty) {
        why = "the x pencil asked for does not fit the grid";
        return WS_ERR_UNSUPPORTED;
      }
      L.xp = &f;
    } else {
      for (const XPencil& f : xt)
        if (f.no == g.nx && g.ny % f.ty == 0 && (!want_xty || f.ty == want_xty) && (!want_xs || f.stages == want_xs)) {
          L.xp = &f;
          break;
        }
    }
  }
  // lengths without a compile-time schedule: the run-time scheduled kernels
  // (3-6 times the generic ones' speed at 2-D and 3-D grids of 45 to 1100
  // points a side, see ws_uni.cuh), unless the generic ones are asked for.  T is then in digit-reversed order
  // along the lines that those kernels transform: along the outer dimension
  // for every pairing, along y and x only if they run both passes.  (PSTD
  // feeds T through K1 a second time, which needs natural order there.)
  if (!L.tp && !L.fp && ch.outer != 2 && uni_plan(no, L.uout.plan)) {
    uni_pencils(L.uout, g.ny, g.nc, mids);
    L.uni_out = L.uout.smem <= kSmemMax;
    if (L.uni_out) L.grid_outer = L.uout.grid;
  }
  if (L.uni_out && !L.fi && !pstd && ch.inner != 2 && !ch.csize && !ch.ncols && !ch.sched &&
      uni_plan(g.ny, L.ucol.plan) && (!L.mode3d || uni_plan(g.nx, L.ux.plan))) {
    uni_columns(L.ucol, (long long)g.nx * g.nz * g.nc);
    if (L.mode3d) uni_pencils(L.ux, g.ny, 1, (long long)g.nz * g.nc);
    L.uni_in = std::max(L.ucol.smem, L.ux.smem) <= kSmemMax;  // a column of 8192 points does not fit
    if (L.uni_in) {
      L.grid_inner = L.ucol.grid;
      L.pitch = (g.ny + 3) / 4 * 4;
    }
  }
  return WS_OK;
}

// ---------------------------------------------------------------------------
// solver object
// ---------------------------------------------------------------------------
struct GraphKey {
  double threshold = -1;
  long long max_iter = -1;
  int interval = -1, stop_rule = -1, nan_stop = -1, nrhs = -1, warm = -1, layout = -1;
  double warm_ratio = -1;
  bool operator==(const GraphKey& o) const {
    return threshold == o.threshold && max_iter == o.max_iter && interval == o.interval &&
           stop_rule == o.stop_rule && nan_stop == o.nan_stop && nrhs == o.nrhs && warm == o.warm && layout == o.layout &&
           warm_ratio == o.warm_ratio;
  }
};

// Device tables of a layout's run-time scheduled plans, in one buffer: the
// wiggles (p tables in the order of T, ramps of k_balance_ramps), the twiddles,
// the ramps, the permutation of the p tables, what takes the transforms' gains
// out again by frequency and by position (minus uni_gains; 0 along the axes that
// other kernels transform), the permuted p tables.
struct UniTables {
  void* buf = nullptr;
  Wig* wigs = nullptr;
  float2* ramp = nullptr;
  int* perm = nullptr;
  int axes = 0;  // bit d: axis d (x, y, z) takes its ramps from k_balance_ramps
  float* efreq = nullptr;
  float* epos = nullptr;
  float* p = nullptr;
  std::vector<Wig> uwig;
};

struct Solver {
  int device = 0;
  cudaStream_t stream = nullptr;
  Geom g{};
  Layout lay;
  int nw = 0;
  float eps = 0.f;
  float2 k02e{};
  std::vector<Wig> wig;
  float* d_wigf = nullptr;   // all pxe/pye/pze
  float2* d_wigc = nullptr;  // all gx/gy/gz
  float2* d_gamma = nullptr;      // n_media gammas of npts elements each
  int n_media = 1;                // > 1: a batch of media, right-hand side r on gamma r
  // per right-hand side (batch of nrhs, capacity batch_cap): fields at r * field elements
  float2 *d_E = nullptr, *d_dE = nullptr, *d_T = nullptr, *d_src = nullptr;
  int batch_cap = 0;
  int nrhs = 1;
  float2* d_stage = nullptr;
  size_t stage_cap = 0;
  float2* d_out = nullptr;
  size_t out_cap = 0;
  DevState* d_state = nullptr;
  double* d_hist = nullptr;  // diff | fresh
  long long hist_cap = 0;
  double* d_energy = nullptr;
  double* d_partials = nullptr;  // per-block ROI energy of K3
  long long partials_cap = 0;    // elements of d_partials
  float2* d_init = nullptr;      // warm starts: v = gamma psi0 / Nw per right-hand side (batch_cap of them)
  int* d_err = nullptr;          // set by a fast kernel whose cluster exchange or TMA wait gave up
  CUtensorMap tmap_T{};          // T as {2 Ny floats, Nx, Nz * tmap_nrhs}, for the TMA pencil
  const void* tmap_base = nullptr;
  int tmap_nrhs = 0;
  const void* tmap_kernel = nullptr;  // the TMA pencil the map and tma_blocks were made for
  int tma_blocks = 0;            // resident blocks of the TMA pencil (its persistent grid)
  CUtensorMap tmap_X{};          // T as {2 Ny floats, Nx, Nz Nc nrhs}, box {2 TY, Nx, 1}, for the x pencils
  const void* xmap_base = nullptr;
  int xmap_nrhs = 0;
  const void* xmap_kernel = nullptr;
  int x_blocks = 0;              // resident blocks of the x pencil (its persistent grid)
  CUtensorMap tmap_slab{};       // T as 2-D {2 Ny floats, Nx Nz Nc nrhs}, box {2 LR, N}, for kf_plane_fused_tma
  const void* slab_base = nullptr;
  int slab_nrhs = 0;
  const void* slab_kernel = nullptr;
  int fused_tma = 1;             // the fused step loads K3's rows by a tensor copy (WAVESIM_B200_FUSED_TMA=0: not)
  int pf_inner = 0, pf_outer = 0;  // L2 prefetch distance of the fast kernels, in blocks (0: off)
  bool warm = false;             // the current solve starts from d_init
  int pstd = 0;                  // a PSTD stepper's solver: K2 applies the Laplacian (see ws_pstd_*)
  int fuse = 0;                  // the loop runs K3 of each iteration fused with K1 of the next
  LayoutChoice tuned{};          // the autotuner's choice (all zero: the heuristics)
  double warm_ratio = 0.0;       // discard threshold of the current solve
  long long wait_clocks = 0;     // bound of the TMA pencils' tile waits and the loop's barrier (0: the defaults)
  int pdl = 0;                   // WAVESIM_B200_PDL=1: launch the loop's kernels with programmatic
                                 // dependent launch (measured: 256^3 solve 46.3 against 44.3 ms,
                                 // 96^3 3.38 against 2.80 ms, 1024^2 8.50 against 8.71 ms; off)
  float2* d_tw = nullptr;
  Layout lays[2];                // the layouts of the launched passes [0] and of the loop in one launch [1];
  bool has_loop = false;         //   `lay` is the one in use, lays[active]
  int loop_blocks = 0;           // the loop's blocks that run at a time
  bool loop_clusters = false;    // up to 16 of them as one cluster
  int active = 0;
  int fuses[2] = {};             // `fuse` of each
  UniTables ut[2];               // their tables
  FftPlan py{}, pxl{}, po{};
  const float2* twx = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t gexec = nullptr;
  GraphKey gkey;
  cudaEvent_t ev[8] = {};
};

static void free_graph(Solver* s) {
  if (s->gexec) cudaGraphExecDestroy(s->gexec);
  if (s->graph) cudaGraphDestroy(s->graph);
  s->gexec = nullptr;
  s->graph = nullptr;
}

// The fused K3 + K1 step is used where the layout has one (3-D fast planes on
// a cluster); WAVESIM_B200_FUSE=0 keeps the three kernels separate.
static int fuse_of(const Solver* s, const Layout& L) {
  const char* e = std::getenv("WAVESIM_B200_FUSE");
  const bool on3 = L.fi && (L.fi->fused || L.xp) && L.mode3d;
  const bool on2 = L.fi && !L.mode3d && L.fi->col_step;  // 2-D: K2 + the column pass
  return ((on3 || on2 || L.uni_in) && !s->pstd && !(e && std::strcmp(e, "0") == 0)) ? 1 : 0;
}

static void destroy_solver(Solver* s) {
  if (!s) return;
  cudaSetDevice(s->device);
  free_graph(s);
  void* ptrs[] = {s->d_wigf, s->d_wigc,  s->d_gamma,  s->d_E,        s->d_dE, s->d_T,   s->d_src,
                  s->d_stage, s->d_out, s->d_state, s->d_hist, s->d_energy, s->d_tw, s->d_partials, s->d_init,
                  s->d_err, s->ut[0].buf, s->ut[1].buf};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  for (auto& e : s->ev)
    if (e) cudaEventDestroy(e);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
}

static int build_plan(int n, const std::vector<float2>& tw_all_offset_dummy, FftPlan& p, int sched = 0) {
  (void)tw_all_offset_dummy;
  std::vector<int> r;
  if (!plan_radices(n, r, sched)) return WS_ERR_UNSUPPORTED;
  p.n = n;
  p.nst = (int)r.size();
  for (int i = 0; i < kMaxStages; ++i) p.radix[i] = i < (int)r.size() ? r[i] : 1;
  return WS_OK;
}

// The radices of the compile-time schedules (empty: none).
static std::vector<int> line_radices(int n) {
  switch (n) {
    case 96: return {12, 4, 2};
    case 160: return {10, 4, 4};
    case 192: return {12, 4, 4};
    case 224: return {14, 4, 4};
    case 320: return {4, 4, 4, 5};
    case 448: return {14, 4, 4, 2};
    case 576: return {12, 12, 4};
  }
  if (n < 32 || n > 2048 || (n & (n - 1))) return {};
  if (n <= 256) return {16, n / 16};
  return {16, 16, n / 256};
}

// The table exp(-2 pi i k / n); behind it, for the lengths with a compile-time
// schedule, the tables of its second stage and on: W_{Ns R}^{jm r} at r Ns + jm
// (fast::line_stage with ST, mixed::Plan::table).
static void push_twiddles(std::vector<float2>& all, int n, size_t& off) {
  off = all.size();
  auto push = [&](double k, int of) {
    const double a = -2.0 * M_PI * k / (double)of;
    all.push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
  };
  for (int k = 0; k < n; ++k) push(k, n);
  const std::vector<int> radix = line_radices(n);
  if (radix.empty()) return;
  for (int s = 1, Ns = radix[0]; s < (int)radix.size(); Ns *= radix[s++])
    for (int r = 0; r < radix[s]; ++r)
      for (int j = 0; j < Ns; ++j) push((double)j * r * (n / (Ns * radix[s])), n);
}

template <typename K>
static cudaError_t allow_dynamic_smem(K kernel, int optin) {
  cudaFuncAttributes fa{};
  cudaError_t e = cudaFuncGetAttributes(&fa, (const void*)kernel);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              optin - (int)fa.sharedSizeBytes);
}

template <int RS>
static cudaError_t set_attributes_for(int optin) {
  cudaError_t e;
  if ((e = allow_dynamic_smem(k_fwd_inner<kEmax, RS>, optin))) return e;
  if ((e = allow_dynamic_smem(k_inv_inner<kEmax, RS>, optin))) return e;
  if ((e = allow_dynamic_smem(k_outer<kEmax, RS>, optin))) return e;
  if ((e = cudaFuncSetAttribute(k_fwd_inner<kEmax, RS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))) return e;
  return cudaFuncSetAttribute(k_inv_inner<kEmax, RS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

static int set_kernel_attributes() {
  // per device: attributes are per-context
  static int done_mask = 0;
  int dev = 0;
  WS_CUDA(cudaGetDevice(&dev));
  if (dev < 31 && (done_mask >> dev) & 1) return WS_OK;
  int optin = 0;
  WS_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  WS_CUDA(set_attributes_for<kPow2>(optin));
  WS_CUDA(set_attributes_for<kMixed>(optin));
  for (const FastInner& f : fast_inner_table()) {
    WS_CUDA(allow_dynamic_smem(f.fwd, optin));
    WS_CUDA(allow_dynamic_smem(f.inv, optin));
    WS_CUDA(cudaFuncSetAttribute(f.fwd, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    WS_CUDA(cudaFuncSetAttribute(f.inv, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (f.fused) {
      WS_CUDA(allow_dynamic_smem(f.fused, optin));
      WS_CUDA(cudaFuncSetAttribute(f.fused, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    if (f.col_step) WS_CUDA(allow_dynamic_smem(f.col_step, optin));
    if (f.fused_tma) {
      WS_CUDA(allow_dynamic_smem(f.fused_tma, optin));
      WS_CUDA(cudaFuncSetAttribute(f.fused_tma, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
  }
  for (const FastPencil& f : fast_pencil_table()) WS_CUDA(allow_dynamic_smem(f.fn, optin));
  for (const TmaPencil& f : tma_pencil_table()) WS_CUDA(allow_dynamic_smem(f.fn, optin));
  for (const TmaPencil& f : tma_pencil2d_table()) WS_CUDA(allow_dynamic_smem(f.fn, optin));
  for (int c = 0; c < uni::kClasses; ++c) {
    const uni::Kernels& k = uni_kernels(c);
    for (const auto& dims : k.col)
      for (const void* f : dims) WS_CUDA(allow_dynamic_smem(f, optin));
    for (const void* f : k.x) WS_CUDA(allow_dynamic_smem(f, optin));
    for (const void* f : k.pencil) WS_CUDA(allow_dynamic_smem(f, optin));
    for (const void* f : {k.loop, k.pstd_loop}) {
      WS_CUDA(allow_dynamic_smem(f, optin));
      WS_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
  }
  for (const XPencil& f : x_pencil_table()) {
    WS_CUDA(allow_dynamic_smem(f.fwd, optin));
    WS_CUDA(allow_dynamic_smem(f.inv, optin));
  }
  if (dev < 31) done_mask |= 1 << dev;
  return WS_OK;
}

static int check_args(const int64_t N[4], int64_t n_wiggles, const ws_wiggle* wiggles, const ws_complex* gamma,
                      const int64_t roi[8], Geom& g) {
  if (!N || !gamma || !wiggles || !roi) return fail(WS_ERR_INVALID_ARGUMENT, "null argument");
  for (int i = 0; i < 4; ++i)
    if (N[i] < 1) return fail(WS_ERR_INVALID_ARGUMENT, "N must be positive");
  if (N[3] != 1 && N[3] != 3) return fail(WS_ERR_INVALID_ARGUMENT, "N(4) must be 1 (scalar) or 3 (vector)");
  if (N[0] > 65536 || N[1] > 65536 || N[2] > 65536)
    return fail(WS_ERR_UNSUPPORTED, "grid dimension larger than 65536");
  if (n_wiggles < 1 || n_wiggles > 64) return fail(WS_ERR_INVALID_ARGUMENT, "Nwiggles must be in [1, 64]");
  g.ny = (int)N[0];
  g.nx = (int)N[1];
  g.nz = (int)N[2];
  g.nc = (int)N[3];
  g.npts = (long long)g.ny * g.nx * g.nz;
  if (g.npts * g.nc > (1LL << 31)) return fail(WS_ERR_UNSUPPORTED, "grid larger than 2^31 elements");
  for (int d = 0; d < 4; ++d) {
    const int64_t a = roi[2 * d], b = roi[2 * d + 1];
    if (a < 1 || b < a || b > N[d]) return fail(WS_ERR_INVALID_ARGUMENT, "roi outside the grid");
    g.r0[d] = (int)(a - 1);
    g.r1[d] = (int)b;
  }
  for (int d = 0; d < 3; ++d)
    if (!length_supported((int)N[d]))
      return fail(WS_ERR_UNSUPPORTED, "grid dimension " + std::to_string(N[d]) +
                                          " has a prime factor above 13 (use an efficient size)");
  return WS_OK;
}

static cudaMemcpyKind kind_from(int memory) { return memory == WS_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice; }

static size_t field_elems(const Solver* s) { return (size_t)s->g.npts * s->g.nc; }
// T of one right-hand side: allocated for a y pitch of whole sectors, used with the layout's
static size_t t_alloc_elems(const Solver* s) { return (size_t)((s->g.ny + 3) / 4 * 4) * s->g.nx * s->g.nz * s->g.nc; }
static long long t_stride(const Solver* s) { return s->lay.pitch * s->g.nx * s->g.nz * s->g.nc; }

// The wiggles' p tables in the order in which a layout's run-time scheduled
// plans leave T (natural along the axes that other kernels transform):
// per[w][i] = nat[w][perm[i]].
static __global__ void k_permute_tables(float* __restrict__ per, const float* __restrict__ nat,
                                        const int* __restrict__ perm, int nf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nf) per[(long long)blockIdx.y * nf + i] = nat[(long long)blockIdx.y * nf + perm[i]];
}
// The ramps with moduli that take the transforms' gains by position out:
// |g|^2 = 1 - pos, 1e-8 from 1, is no pair of floats, so each element takes the
// neighbour (of up to one ulp each way) that brings the sum over its 32
// elements nearest to it.  That also takes out the mean of the plain rounding.
// (Ramps of another modulus than 1 keep it.)  Rounding the ramps alone moves
// the converged field of 81 x 360 points by 6.0e-7, these by 2.6e-7 (165 x 400:
// 3.9e-7, 2.6e-7).
static __global__ void k_balance_ramps(float2* __restrict__ out, const float2* __restrict__ ramp,
                                       const float* __restrict__ epos, int nx, int ny, int nf, int axes) {
  const int i0 = 32 * (blockIdx.x * blockDim.x + threadIdx.x);
  out += (long long)blockIdx.y * nf;
  ramp += (long long)blockIdx.y * nf;
  double carry = 0.0;
  for (int i = i0; i < min(nf, i0 + 32); ++i) {
    const float2 g = ramp[i];
    float2 best = g;
    if (i == nx || i == nx + ny) carry = 0.0;
    if (axes >> (i < nx ? 0 : (i < nx + ny ? 1 : 2)) & 1) {
      double m = (double)g.x * g.x + (double)g.y * g.y;
      if (fabs(m - 1.0) < 1e-6) m = 1.0;
      const double want = m * (1.0 + epos[i]) + carry;
      double least = 1e300, rest = 0.0;
      for (int k = 0; k < 9; ++k) {
        const int a = k / 3, b = k % 3;
        if (b && g.y == 0.f) continue;
        const float2 c = make_float2(a ? nextafterf(g.x, a == 1 ? 2.f : -2.f) : g.x,
                                     b ? nextafterf(g.y, b == 1 ? 2.f : -2.f) : g.y);
        const double left = want - ((double)c.x * c.x + (double)c.y * c.y);
        const double cost = fabs(left) + 0.05 * (fabs((double)c.x - g.x) + fabs((double)c.y - g.y));
        if (cost < least) {
          least = cost;
          rest = left;
          best = c;
        }
      }
      carry = fabs(rest) < 1e-6 ? rest : 0.0;
    }
    out[i] = best;
  }
}
static cudaError_t permute_wiggles(Solver* s) {
  cudaError_t e = cudaStreamSynchronize(cudaStreamLegacy);  // the tables' uploads
  if (e != cudaSuccess) return e;
  const int nf = s->g.nx + s->g.ny + s->g.nz;
  for (const UniTables& t : s->ut)
    if (t.wigs) {
      k_permute_tables<<<dim3((nf + 255) / 256, s->nw), 256, 0, s->stream>>>(t.p, s->d_wigf, t.perm, nf);
      k_balance_ramps<<<dim3((nf + 1023) / 1024, s->nw), 32, 0, s->stream>>>(t.ramp, s->d_wigc, t.epos, s->g.nx, s->g.ny,
                                                                           nf, t.axes);
    }
  return cudaGetLastError();
}

// The tables of layout k.
static cudaError_t make_tables(Solver* s, int k) {
  Layout& L = s->lays[k];
  UniTables& t = s->ut[k];
  const Geom& g = s->g;
  const int len[3] = {g.nx, g.ny, g.nz};  // the order of d_wigf
  const uni::Plan* axis[3] = {L.mode3d ? (L.uni_in ? &L.ux.plan : nullptr) : &L.uout.plan,
                              L.uni_in ? &L.ucol.plan : nullptr, L.mode3d ? &L.uout.plan : nullptr};
  std::vector<float2> tw;
  uni::Plan* plans[3] = {&L.ucol.plan, &L.ux.plan, &L.uout.plan};
  size_t at[3];
  for (int q = 0; q < 3; ++q) {
    at[q] = tw.size();
    for (int i = 0; i < plans[q]->nst; ++i) {
      const uni::Stage& S = plans[q]->st[i];
      const int n = S.R * S.sub;
      for (int r = 0; r < S.R; ++r)
        for (int j = 0; j < S.sub; ++j) tw.push_back(uni_twiddle(j, r, n));
    }
  }
  const size_t nf = (size_t)g.nx + g.ny + g.nz;
  std::vector<int> perm;
  std::vector<float> efreq, epos;
  for (int d = 0; d < 3; ++d) {
    const int off = (int)perm.size();
    const std::vector<int> f = axis[d] ? uni_permutation(*axis[d]) : std::vector<int>();
    std::vector<double> pos(len[d], 0.0), freq(len[d], 0.0);
    const bool columns = d == 1 && L.fi && !L.mode3d;  // compile-time columns, inside these kernels' pencils
    for (int q = 0; q < 3; ++q)
      if (axis[d] && axis[d] == plans[q]) uni_gains(*axis[d], tw.data() + at[q], pos, freq);
    if (columns) line_gains(line_radices(g.ny), pos, freq);
    // without ramps of its own (PSTD, other column passes), the mean of the part by position
    const bool ramps = (L.uni_in || (L.fi && !L.mode3d)) && !s->pstd;
    const double mean = ramps ? 0.0 : std::accumulate(pos.begin(), pos.end(), 0.0) / len[d];
    if (ramps && (axis[d] || columns)) t.axes |= 1 << d;
    for (int i = 0; i < len[d]; ++i) {
      perm.push_back(off + (axis[d] ? f[i] : i));
      efreq.push_back((float)-(freq[i] + mean));
      epos.push_back((float)-pos[i]);
    }
  }
  // one buffer: the ramps, what the host has (in one copy), the p tables
  const size_t rb = nf * s->nw * sizeof(float2), wb = s->nw * sizeof(Wig), twb = tw.size() * sizeof(float2),
               tb = nf * sizeof(float);
  std::vector<char> host(wb + twb + 3 * tb);
  char* buf = nullptr;
  cudaError_t e = cudaMalloc(&buf, rb + host.size() + tb * s->nw);
  if (e != cudaSuccess) return e;
  t.ramp = reinterpret_cast<float2*>(buf);
  t.wigs = reinterpret_cast<Wig*>(buf + rb);
  float2* const d_tw = reinterpret_cast<float2*>(buf + rb + wb);
  t.perm = reinterpret_cast<int*>(buf + rb + wb + twb);
  t.efreq = reinterpret_cast<float*>(buf + rb + wb + twb + tb);
  t.epos = t.efreq + nf;
  t.p = t.epos + nf;
  for (int q = 0; q < 3; ++q) plans[q]->tw = d_tw + at[q];
  t.uwig = s->wig;
  for (int w = 0; w < s->nw; ++w) {
    const float* f = t.p + nf * w;
    t.uwig[w].pxe = f;
    t.uwig[w].pye = f + g.nx;
    t.uwig[w].pze = f + g.nx + g.ny;
    const float2* c = t.ramp + nf * w;
    t.uwig[w].gx = c;
    t.uwig[w].gy = c + g.nx;
    t.uwig[w].gz = c + g.nx + g.ny;
  }
  std::memcpy(host.data(), t.uwig.data(), wb);
  std::memcpy(host.data() + wb, tw.data(), twb);
  std::memcpy(host.data() + wb + twb, perm.data(), tb);
  std::memcpy(host.data() + wb + twb + tb, efreq.data(), tb);
  std::memcpy(host.data() + wb + twb + 2 * tb, epos.data(), tb);
  e = cudaMemcpyAsync(t.wigs, host.data(), host.size(), cudaMemcpyHostToDevice, s->stream);  // pageable: taken at once
  if (e != cudaSuccess) {  // nothing half made is kept
    cudaFree(buf);
    t = UniTables{};
    return e;
  }
  t.buf = buf;
  return cudaSuccess;
}

// Makes lays[k] the layout in use, with its tables (made on its first use:
// few solvers run both).
static cudaError_t use_layout(Solver* s, int k) {
  if (s->lays[k].uni_out && !s->ut[k].buf) {
    cudaError_t e = make_tables(s, k);
    if (e != cudaSuccess) return e;
    if ((e = permute_wiggles(s)) != cudaSuccess) {
      cudaFree(s->ut[k].buf);
      s->ut[k] = UniTables{};
      return e;
    }
  }
  s->active = k;
  s->lay = s->lays[k];
  s->fuse = s->fuses[k];
  return cudaSuccess;
}

// Threads of the loop's blocks: a butterfly each, or 512.
static int loop_threads(const Layout& L) {
  const int work = std::max(L.ucol.lines * uni_units(L.ucol.plan), L.uout.lines * uni_units(L.uout.plan));
  return work <= 256 ? 256 : uni::kLoopThreads;
}
// Tiles of the loop, and whether its blocks form one cluster.
static long long loop_tiles(const Solver* s, int nrhs) {
  return std::max(s->lays[1].ucol.grid, s->lays[1].uout.grid) * nrhs;
}
static bool loop_cluster(const Solver* s, int nrhs) { return s->loop_clusters && loop_tiles(s, nrhs) <= 16; }

// How many of the loop's blocks run at a time: one an SM, as many as the device
// has free for this process (a share of it has fewer than kNumSms, and would
// refuse the launch).  WAVESIM_B200_LOOP=n: at most n (0: no loop in one launch).
static cudaError_t loop_room(Solver* s) {
  const Layout& L = s->lays[1];
  const uni::Kernels& k = uni_kernels(std::max(L.ucol.plan.cls, L.uout.plan.cls));
  const void* fn = s->pstd ? k.pstd_loop : k.loop;
  size_t smem = s->pstd ? pstd_loop_smem(L, s->g) : loop_smem(L, s->g, s->nw, true);
  if (smem > kLoopSmem) smem = loop_smem(L, s->g, s->nw, false);
  const int threads = loop_threads(L);
  int sms = 0, per_sm = 0, clusters = 0;
  s->loop_blocks = 0;
  s->loop_clusters = false;
  if (smem > kLoopSmem) return cudaSuccess;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  if (e != cudaSuccess) return e;
  s->loop_blocks = per_sm > 0 ? std::min(sms, kNumSms) : 0;
  if (const char* most = std::getenv("WAVESIM_B200_LOOP")) s->loop_blocks = std::min(s->loop_blocks, std::max(0, std::atoi(most)));
  const long long tiles = loop_tiles(s, 1);
  if (tiles > std::min(16, s->loop_blocks)) return cudaSuccess;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)tiles;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)tiles);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  s->loop_clusters = cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters > 0;
  cudaGetLastError();
  return cudaSuccess;
}

// The layouts beside that of the launched passes (lays[0], made by the
// caller); the one of single solves is then in use.
static cudaError_t set_layouts(Solver* s) {
  Layout heuristic;
  std::string why;
  s->has_loop = make_layout(s->g, heuristic, why, LayoutChoice{}, s->pstd != 0) == WS_OK &&
                loop_layout(s->g, heuristic, s->pstd != 0, s->lays[1]);
  if (s->has_loop) {
    const cudaError_t e = loop_room(s);
    if (e != cudaSuccess) return e;
    s->has_loop = s->lays[1].ucol.grid <= s->loop_blocks;
  }
  for (int k = 0; k < 2; ++k) {
    if (s->ut[k].buf) cudaFree(s->ut[k].buf);
    s->ut[k] = UniTables{};
    s->fuses[k] = fuse_of(s, s->lays[k]);
  }
  return use_layout(s, s->has_loop ? 1 : 0);
}

// Buffers for nrhs right-hand sides (kept when large enough).
// d_partials holds at least n per-block energies (graphs hold the old pointer)
static int ensure_partials(Solver* s, long long n) {
  if (n <= s->partials_cap) return WS_OK;
  double* p = nullptr;
  WS_CUDA(cudaMalloc(&p, (size_t)n * sizeof(double)));
  if (s->d_partials) cudaFree(s->d_partials);
  s->d_partials = p;
  s->partials_cap = n;
  free_graph(s);
  return WS_OK;
}

static int ensure_batch(Solver* s, int nrhs) {
  if (nrhs <= s->batch_cap) return WS_OK;
  void* old[] = {s->d_E, s->d_dE, s->d_T, s->d_src, s->d_state, s->d_energy, s->d_partials, s->d_init};
  for (void* p : old)
    if (p) cudaFree(p);
  s->d_E = s->d_dE = s->d_T = s->d_src = s->d_init = nullptr;
  s->d_state = nullptr;
  s->d_energy = s->d_partials = nullptr;
  s->batch_cap = 0;
  if (s->d_hist) cudaFree(s->d_hist);
  s->d_hist = nullptr;
  s->hist_cap = 0;
  free_graph(s);
  const size_t nb = field_elems(s) * nrhs * sizeof(float2);
  WS_CUDA(cudaMalloc(&s->d_E, nb));
  WS_CUDA(cudaMalloc(&s->d_dE, nb));
  WS_CUDA(cudaMalloc(&s->d_T, t_alloc_elems(s) * nrhs * sizeof(float2)));
  WS_CUDA(cudaMalloc(&s->d_src, nb));
  WS_CUDA(cudaMalloc(&s->d_state, nrhs * sizeof(DevState)));
  WS_CUDA(cudaMalloc(&s->d_energy, nrhs * sizeof(double)));
  s->partials_cap = std::max<long long>(1, std::max(s->lays[0].grid_inner, s->lays[1].grid_inner)) * nrhs * s->nw;
  WS_CUDA(cudaMalloc(&s->d_partials, (size_t)s->partials_cap * sizeof(double)));
  WS_CUDA(cudaMemset(s->d_E, 0, nb));
  WS_CUDA(cudaMemset(s->d_dE, 0, nb));
  WS_CUDA(cudaMemset(s->d_state, 0, nrhs * sizeof(DevState)));
  s->batch_cap = nrhs;
  return WS_OK;
}

static int create_solver(const int64_t N[4], const ws_complex* gamma, int64_t n_wiggles, const ws_wiggle* wiggles,
                         float epsilon, ws_complex k02e, const int64_t roi[8], int memory, int device, Solver** out,
                         bool pstd = false) {
  Geom g{};
  int rc = check_args(N, n_wiggles, wiggles, gamma, roi, g);
  if (rc) return rc;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(WS_ERR_NO_DEVICE, "no CUDA device");
  if (device < 0 || device >= ndev) return fail(WS_ERR_INVALID_ARGUMENT, "bad device ordinal");
  WS_CUDA(cudaSetDevice(device));
  rc = set_kernel_attributes();
  if (rc) return rc;
  Solver* s = new Solver();
  s->device = device;
  s->g = g;
  s->nw = (int)n_wiggles;
  s->eps = epsilon;
  s->k02e = make_float2(k02e.re, k02e.im);
  std::string why;
  s->pstd = pstd ? 1 : 0;
  rc = make_layout(g, s->lay, why, LayoutChoice{}, pstd);
  if (rc) {
    destroy_solver(s);
    return fail(rc, why);
  }
  {
    // L2 prefetch distance of the fast kernels: about one wave of resident
    // blocks (2 per SM), a whole number of clusters.  WAVESIM_B200_PREFETCH
    // sets the waves' size in blocks per SM (0 switches the prefetch off).
    int per_sm = 2;
    if (const char* e = std::getenv("WAVESIM_B200_PREFETCH")) per_sm = std::max(0, std::atoi(e));
    const int c = s->lay.fi ? std::max(1, s->lay.fi->c) : 1;
    s->pf_inner = (per_sm * kNumSms / c) * c;
    s->pf_outer = per_sm * kNumSms;
    if (const char* e = std::getenv("WAVESIM_B200_FUSED_TMA")) s->fused_tma = std::atoi(e) ? 1 : 0;
    if (const char* e = std::getenv("WAVESIM_B200_PDL")) s->pdl = std::atoi(e) ? 1 : 0;
  }
#define WS_TRY(call)                 \
  do {                               \
    cudaError_t e__ = (call);        \
    if (e__ != cudaSuccess) {        \
      destroy_solver(s);             \
      return fail(e__ == cudaErrorMemoryAllocation ? WS_ERR_OUT_OF_MEMORY : WS_ERR_CUDA, \
                  std::string(#call) + ": " + cudaGetErrorString(e__)); \
    }                                \
  } while (0)
  WS_TRY(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
  WS_TRY(cudaMalloc(&s->d_err, 2 * sizeof(int)));  // and the loop's barrier counter
  WS_TRY(cudaMemset(s->d_err, 0, 2 * sizeof(int)));
  for (auto& e : s->ev) WS_TRY(cudaEventCreate(&e));
  // plans and twiddle tables
  std::vector<float2> tw;
  size_t off_y, off_x, off_xl, off_o;
  const int no = s->lay.mode3d ? g.nz : g.nx;
  const int nxl = s->lay.mode3d ? g.nx / s->lay.csize : 1;
  push_twiddles(tw, g.ny, off_y);
  push_twiddles(tw, g.nx, off_x);
  push_twiddles(tw, nxl, off_xl);
  push_twiddles(tw, no, off_o);
  WS_TRY(cudaMalloc(&s->d_tw, tw.size() * sizeof(float2)));
  WS_TRY(cudaMemcpy(s->d_tw, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice));
  build_plan(g.ny, tw, s->py);
  s->py.tw = s->d_tw + off_y;
  build_plan(nxl, tw, s->pxl);
  s->pxl.tw = s->d_tw + off_xl;
  build_plan(no, tw, s->po);
  s->po.tw = s->d_tw + off_o;
  s->twx = s->d_tw + off_x;
  // wiggles
  const size_t nf = (size_t)g.nx + g.ny + g.nz;
  WS_TRY(cudaMalloc(&s->d_wigf, nf * n_wiggles * sizeof(float)));
  WS_TRY(cudaMalloc(&s->d_wigc, nf * n_wiggles * sizeof(float2)));
  const cudaMemcpyKind kind = kind_from(memory);
  for (int w = 0; w < n_wiggles; ++w) {
    const ws_wiggle& W = wiggles[w];
    if (!W.pxe || !W.pye || !W.pze || !W.gx || !W.gy || !W.gz) {
      destroy_solver(s);
      return fail(WS_ERR_INVALID_ARGUMENT, "null wiggle array");
    }
    float* f = s->d_wigf + nf * w;
    float2* c = s->d_wigc + nf * w;
    WS_TRY(cudaMemcpy(f, W.pxe, g.nx * sizeof(float), kind));
    WS_TRY(cudaMemcpy(f + g.nx, W.pye, g.ny * sizeof(float), kind));
    WS_TRY(cudaMemcpy(f + g.nx + g.ny, W.pze, g.nz * sizeof(float), kind));
    WS_TRY(cudaMemcpy(c, W.gx, g.nx * sizeof(float2), kind));
    WS_TRY(cudaMemcpy(c + g.nx, W.gy, g.ny * sizeof(float2), kind));
    WS_TRY(cudaMemcpy(c + g.nx + g.ny, W.gz, g.nz * sizeof(float2), kind));
    s->wig.push_back(Wig{f, f + g.nx, f + g.nx + g.ny, c, c + g.nx, c + g.nx + g.ny});
  }
  s->lays[0] = s->lay;
  WS_TRY(set_layouts(s));
  WS_TRY(cudaMalloc(&s->d_gamma, (size_t)g.npts * sizeof(float2)));
  WS_TRY(cudaMemcpy(s->d_gamma, gamma, (size_t)g.npts * sizeof(float2), kind));
#undef WS_TRY
  const int rc2 = ensure_batch(s, 1);
  if (rc2) {
    destroy_solver(s);
    return rc2;
  }
  *out = s;
  return WS_OK;
}

// A new medium (gamma, wiggles, epsilon, k02e, roi) of the same grid and
// wiggle count into an existing solver: uploads only, no allocation.  The
// solver's stream must be idle (it is after a solve returns).
static int reload_medium(Solver* s, const int64_t N[4], const ws_complex* gamma, int64_t n_wiggles,
                         const ws_wiggle* wiggles, float epsilon, ws_complex k02e, const int64_t roi[8], int memory) {
  Geom g{};
  int rc = check_args(N, n_wiggles, wiggles, gamma, roi, g);
  if (rc) return rc;
  WS_CUDA(cudaSetDevice(s->device));
  const cudaMemcpyKind kind = kind_from(memory);
  const size_t nf = (size_t)g.nx + g.ny + g.nz;
  for (int w = 0; w < n_wiggles; ++w) {
    const ws_wiggle& W = wiggles[w];
    if (!W.pxe || !W.pye || !W.pze || !W.gx || !W.gy || !W.gz) return fail(WS_ERR_INVALID_ARGUMENT, "null wiggle array");
    float* f = s->d_wigf + nf * w;
    float2* c = s->d_wigc + nf * w;
    WS_CUDA(cudaMemcpy(f, W.pxe, g.nx * sizeof(float), kind));
    WS_CUDA(cudaMemcpy(f + g.nx, W.pye, g.ny * sizeof(float), kind));
    WS_CUDA(cudaMemcpy(f + g.nx + g.ny, W.pze, g.nz * sizeof(float), kind));
    WS_CUDA(cudaMemcpy(c, W.gx, g.nx * sizeof(float2), kind));
    WS_CUDA(cudaMemcpy(c + g.nx, W.gy, g.ny * sizeof(float2), kind));
    WS_CUDA(cudaMemcpy(c + g.nx + g.ny, W.gz, g.nz * sizeof(float2), kind));
  }
  WS_CUDA(permute_wiggles(s));
  WS_CUDA(cudaMemcpy(s->d_gamma, gamma, (size_t)g.npts * sizeof(float2), kind));
  const float2 k = make_float2(k02e.re, k02e.im);
  bool same = s->eps == epsilon && s->k02e.x == k.x && s->k02e.y == k.y;
  for (int d = 0; d < 4; ++d) same = same && s->g.r0[d] == g.r0[d] && s->g.r1[d] == g.r1[d];
  if (!same) {
    // scalars and the roi are kernel arguments inside the graph
    s->eps = epsilon;
    s->k02e = k;
    s->g = g;
    free_graph(s);
  }
  return WS_OK;
}

// what E' takes in iteration i of a cycle (counted from 0)
static int acc_of(const Solver* s, int i) { return s->nw % 2 ? kAccEach : (i % 2 ? kAccPair : kAccSkip); }
// the energy partials of iteration i of a cycle
static double* partials_of(const Solver* s, int i) {
  return s->d_partials + (long long)(i % s->nw) * s->lay.grid_inner * s->nrhs;
}

// the ramps of the inner passes: those that take the gains out, if pencils of ws_uni.cuh follow
static const Wig& ramps_of(const Solver* s, int w) {
  return s->lay.uni_out ? s->ut[s->active].uwig[w] : s->wig[w];
}

// iteration i of a cycle (wiggle i mod Nw)
static InnerArgs inner_args(const Solver* s, int i) {
  const int w = i % s->nw;
  InnerArgs a{};
  a.g = s->g;
  a.w = ramps_of(s, w);
  a.py = s->py;
  a.pxl = s->pxl;
  a.twx = s->twx;
  a.csize = s->lay.csize;
  a.mode3d = s->lay.mode3d;
  a.ncols = s->lay.ncols;
  a.bpr = (int)s->lay.grid_inner;
  a.fstride = (long long)field_elems(s);
  a.err = s->d_err;
  a.gstride = s->n_media > 1 ? (long long)s->g.npts : 0;
  a.pf = 0;  // K3 (and the generic kernels) measured slower with it
  a.acc2 = acc_of(s, i);
  return a;
}

static OuterArgs outer_args(const Solver* s, int w) {
  OuterArgs a{};
  a.g = s->g;
  a.w = s->wig[w];
  a.po = s->po;
  a.k02e = s->k02e;
  a.norm = (float)(1.0 / ((double)s->g.npts));
  a.ty = s->lay.ty;
  a.mode3d = s->lay.mode3d;
  a.bpr = (int)s->lay.grid_outer;
  a.fstride = (long long)field_elems(s);
  a.pf = 0;  // K2 measured slower with it
  a.pstd = s->pstd;
  a.wait_clocks = s->wait_clocks;
  return a;
}

template <int RS>
static cudaError_t launch_k1_t(const Solver* s, int w, const float2* in, const float2* src, float2* out,
                              float a_mult) {
  const float2 A = make_float2(0.f, a_mult * (float)(1.0f / s->eps / (float)s->nw));  // 1i/epsilon/Nwiggles
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(s->lay.grid_inner * s->nrhs));
  cfg.blockDim = dim3(s->lay.th_inner);
  cfg.dynamicSmemBytes = s->lay.smem_inner;
  cfg.stream = s->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = s->lay.mode3d ? s->lay.csize : 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_fwd_inner<kEmax, RS>, inner_args(s, w), in, src, A, out,
                            (const DevState*)s->d_state);
}

template <int RS>
static cudaError_t launch_k2_t(const Solver* s, int w) {
  k_outer<kEmax, RS><<<(unsigned)(s->lay.grid_outer * s->nrhs), s->lay.th_outer, s->lay.smem_outer, s->stream>>>(
      outer_args(s, w), s->d_T, s->d_state);
  return cudaGetLastError();
}

template <int RS>
static cudaError_t launch_k3_t(const Solver* s, int w) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(s->lay.grid_inner * s->nrhs));
  cfg.blockDim = dim3(s->lay.th_inner);
  cfg.dynamicSmemBytes = s->lay.smem_inner;
  cfg.stream = s->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = s->lay.mode3d ? s->lay.csize : 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_inv_inner<kEmax, RS>, inner_args(s, w), (const float2*)s->d_T, s->d_dE,
                            s->d_E, (const float2*)s->d_gamma, (const DevState*)s->d_state, partials_of(s, w));
}

static size_t fast_inner_smem(const Solver* s, bool fwd) {
  const FastInner* f = s->lay.fi;
  return f->do_x ? (fwd ? f->smem_fwd : f->smem_inv) : f->smem * (size_t)(s->lay.ncols + 1);
}

static cudaError_t launch_fast_inner(const Solver* s, const void* fn, void** args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(s->lay.grid_inner * s->nrhs));
  cfg.blockDim = dim3(fast::kThreads);
  cfg.dynamicSmemBytes = fast_inner_smem(s, fn == s->lay.fi->fwd);
  cfg.stream = s->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = s->lay.fi->do_x ? s->lay.fi->c : 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// A loop kernel that begins with pdl_begin(): launched with programmatic
// stream serialisation, so that it may be scheduled while the kernel before
// it finishes (it waits for that kernel's completion before touching global
// memory); captured into the loop's graph as a programmatic edge.
static cudaError_t launch_pdl(const Solver* s, const void* fn, dim3 grid, dim3 block, void** args, size_t smem) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = s->pdl ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// The passes of the run-time scheduled kernels (ws_uni.cuh).
static cudaError_t launch_uni(const Solver* s, const void* fn, const UniPass& p, void* args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(p.grid * s->nrhs));
  cfg.blockDim = dim3(p.threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s->stream;
  void* argv[] = {args};
  return cudaLaunchKernelExC(&cfg, fn, argv);
}

// mode kFwd: K1's column transforms of `in`; kInv: K3's; kStep: K3 with
// wiggle w and K1 of the next iteration with wiggle w1
static uni::ColArgs uni_col_args(const Solver* s, int w, int w1, const float2* in, const float2* src, float2* T,
                                 float a_mult) {
  const UniPass& p = s->lay.ucol;
  uni::ColArgs a{};
  a.g = s->g;
  a.py = p.plan;
  const std::vector<Wig>& wig = s->ut[s->active].uwig;
  a.it.gx = wig[w].gx;
  a.it.gy = wig[w].gy;
  a.it.gz = wig[w].gz;
  a.it.gx1 = wig[w1].gx;
  a.it.gy1 = wig[w1].gy;
  a.it.gz1 = wig[w1].gz;
  a.dE_in = in;
  a.it.src = src;
  a.A = make_float2(0.f, a_mult * (float)(1.0f / s->eps / (float)s->nw));  // 1i/epsilon/Nwiggles
  a.T = T;
  a.dE = s->d_dE;
  a.E = s->d_E;
  a.gamma = s->d_gamma;
  a.st = s->d_state;
  a.it.partials = partials_of(s, w);
  a.pitch = s->lay.pitch;
  a.fstride = (long long)field_elems(s);
  a.tstride = t_stride(s);
  a.gstride = s->n_media > 1 ? (long long)s->g.npts : 0;
  a.total = s->g.nx * s->g.nz * s->g.nc;
  a.lines = p.lines;
  a.bpr = (int)p.grid;
  a.it.acc = acc_of(s, w);
  return a;
}
static cudaError_t launch_uni_col(const Solver* s, int mode, int w, int w1, const float2* in, const float2* src,
                                  float2* T, float a_mult) {
  uni::ColArgs a = uni_col_args(s, w, w1, in, src, T, a_mult);
  return launch_uni(s, uni_kernels(a.py.cls).col[s->lay.mode3d][mode], s->lay.ucol, &a);
}

static uni::XArgs uni_x_args(const Solver* s, float2* T) {
  const UniPass& p = s->lay.ux;
  uni::XArgs a{};
  a.px = p.plan;
  a.T = T;
  a.st = s->d_state;
  a.pitch = s->lay.pitch;
  a.tstride = t_stride(s);
  a.ny = s->g.ny;
  a.nx = s->g.nx;
  a.lty = log2_of(p.lines);
  a.nyt = p.lines ? (s->g.ny + p.lines - 1) / p.lines : 0;
  a.bpr = (int)p.grid;
  return a;
}
static cudaError_t launch_uni_x(const Solver* s, bool inv, float2* T) {
  uni::XArgs a = uni_x_args(s, T);
  return launch_uni(s, uni_kernels(a.px.cls).x[inv ? 1 : 0], s->lay.ux, &a);
}

static uni::PencilArgs uni_pencil_args(const Solver* s, int w) {
  const UniPass& p = s->lay.uout;
  uni::PencilArgs a{};
  a.g = s->g;
  a.po = p.plan;
  a.w = s->ut[s->active].uwig[w];
  a.k02e = s->k02e;
  const double kk = (double)s->k02e.x * s->k02e.x + (double)s->k02e.y * s->k02e.y;
  if (kk > 0) a.ik02e = make_float2((float)(s->k02e.x / kk), (float)(-s->k02e.y / kk));
  a.norm = (float)(1.0 / ((double)s->g.npts));
  a.norm_e = (float)(1.0 / ((double)s->g.npts * a.norm) - 1.0);
  a.ex = s->ut[s->active].efreq;
  a.ey = a.ex + s->g.nx;
  a.ez = a.ey + s->g.ny;
  a.T = s->d_T;
  a.st = s->d_state;
  a.pitch = s->lay.pitch;
  a.tstride = t_stride(s);
  a.cstride = s->lay.pitch * s->g.nx * s->g.nz;
  a.lty = log2_of(p.lines);
  a.nyt = (s->g.ny + p.lines - 1) / p.lines;
  a.bpr = (int)p.grid;
  a.mode3d = s->lay.mode3d;
  a.pstd = s->pstd;
  return a;
}
static cudaError_t launch_uni_k2(const Solver* s, int w) {
  uni::PencilArgs a = uni_pencil_args(s, w);
  return launch_uni(s, uni_kernels(a.po.cls).pencil[s->g.nc == 3 ? 1 : 0], s->lay.uout, &a);
}

// K1 on explicit buffers: out = inner FFT of (in + a_mult A src) times the
// ramps of wiggle w (A = i/epsilon/Nw, the reference's per-iteration share of
// the source; a_mult = Nw gives the whole source, for the warm start's
// residual probe)
static cudaError_t launch_k1_io(const Solver* s, int w, const float2* in, const float2* src, float2* out,
                                float a_mult = 1.f) {
  if (s->lay.uni_in) {
    cudaError_t e = launch_uni_col(s, uni::kFwd, w, w, in, src, out, a_mult);
    return e != cudaSuccess || !s->lay.mode3d ? e : launch_uni_x(s, false, out);
  }
  if (s->lay.fi) {
    InnerArgs a = inner_args(s, w);
    a.ncols = s->lay.ncols;
    a.pf = s->pf_inner;  // K1 only: its loads come first, so the next wave's columns are worth pulling early
    float2 A = make_float2(0.f, a_mult * (float)(1.0f / s->eps / (float)s->nw));
    const DevState* st = s->d_state;
    void* args[] = {&a, &in, &src, &A, &out, &st};
    return launch_fast_inner(s, s->lay.fi->fwd, args);
  }
  return s->lay.rset == kPow2 ? launch_k1_t<kPow2>(s, w, in, src, out, a_mult)
                              : launch_k1_t<kMixed>(s, w, in, src, out, a_mult);
}
static cudaError_t launch_k1(const Solver* s, int w, bool with_source) {
  return launch_k1_io(s, w, s->d_dE, with_source ? s->d_src : nullptr, s->d_T);
}
// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against libcuda)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}

// T of the current batch as a 3-D float tensor {2 Ny, Nx, Nz Nc nrhs}, box
// {2 TY, 1, Nz}: every x coordinate the kernel issues is 2 TY yt floats, a
// multiple of 16 floats (TY >= 8), so each copy starts on a 64-byte boundary.
static cudaError_t ensure_tmap(Solver* s, const TmaPencil* f) {
  if (s->tmap_base == s->d_T && s->tmap_nrhs == s->nrhs && s->tmap_kernel == f->fn) return cudaSuccess;
  s->tmap_kernel = nullptr;
  s->tma_blocks = 0;
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return cudaErrorNotSupported;
  const Geom& g = s->g;
  const cuuint64_t dims[3] = {(cuuint64_t)2 * g.ny, (cuuint64_t)g.nx, (cuuint64_t)g.nz * g.nc * s->nrhs};
  const cuuint64_t strides[2] = {(cuuint64_t)g.ny * sizeof(float2), (cuuint64_t)g.ny * g.nx * sizeof(float2)};
  const cuuint32_t line = (cuuint32_t)std::min(f->no, 256);  // along z, or along x of a 2-D grid
  const cuuint32_t box[3] = {(cuuint32_t)(2 * f->ty), s->lay.mode3d ? 1u : line, s->lay.mode3d ? line : 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  if (enc(&s->tmap_T, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, s->d_T, dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  s->tmap_base = s->d_T;
  s->tmap_nrhs = s->nrhs;
  s->tmap_kernel = f->fn;
  return cudaSuccess;
}

static cudaError_t launch_k2_tma(const Solver* cs, int w, const TmaPencil* f) {
  Solver* s = const_cast<Solver*>(cs);  // the tensor-map cache only
  cudaError_t e = ensure_tmap(s, f);
  if (e != cudaSuccess) return e;
  if (s->tma_blocks <= 0) {
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f->fn, f->threads, f->smem);
    if (e != cudaSuccess) return e;
    s->tma_blocks = std::max(1, per_sm) * kNumSms;
  }
  OuterArgs a = outer_args(s, w);
  int ntiles = s->nrhs * (s->lay.mode3d ? s->g.nx : 1) * (s->g.ny / f->ty);
  const unsigned grid = (unsigned)std::min(ntiles, s->tma_blocks);
  const DevState* st = s->d_state;
  int* err = s->d_err;
  void* args[] = {&s->tmap_T, &a, &st, &ntiles, &err};
  return launch_pdl(s, f->fn, dim3(grid), dim3(f->threads), args, f->smem);
}

static cudaError_t launch_k2(const Solver* s, int w) {
  if (s->lay.tp) return launch_k2_tma(s, w, s->lay.tp);
  // the pipeline pays from about two tiles per resident block on
  if (s->lay.tp2 && (long long)s->nrhs * (s->g.ny / s->lay.tp2->ty) >= 4 * kNumSms) return launch_k2_tma(s, w, s->lay.tp2);
  if (s->lay.fp) {
    OuterArgs a = outer_args(s, w);
    const FastPencil* f = s->lay.fp;
    const unsigned grid = (unsigned)(s->lay.grid_outer * s->nrhs);
    float2* T = s->d_T;
    const DevState* st = s->d_state;
    void* args[] = {&a, &T, &st};
    return launch_pdl(s, f->fn, dim3(grid), dim3(f->threads), args, f->smem);
  }
  if (s->lay.uni_out) return launch_uni_k2(s, w);
  return s->lay.rset == kPow2 ? launch_k2_t<kPow2>(s, w) : launch_k2_t<kMixed>(s, w);
}
static cudaError_t launch_k3_only(const Solver* s, int w) {
  cudaError_t e;
  if (s->lay.uni_in) {
    if (s->lay.mode3d && (e = launch_uni_x(s, true, s->d_T)) != cudaSuccess) return e;
    return launch_uni_col(s, uni::kInv, w, w, nullptr, nullptr, s->d_T, 1.f);
  }
  if (s->lay.fi) {
    InnerArgs a = inner_args(s, w);
    a.ncols = s->lay.ncols;
    const float2* T = s->d_T;
    float2* dE = s->d_dE;
    float2* E = s->d_E;
    const float2* gamma = s->d_gamma;
    const DevState* st = s->d_state;
    double* partials = partials_of(s, w);
    void* args[] = {&a, &T, &dE, &E, &gamma, &st, &partials};
    e = launch_fast_inner(s, s->lay.fi->inv, args);
  } else {
    e = s->lay.rset == kPow2 ? launch_k3_t<kPow2>(s, w) : launch_k3_t<kMixed>(s, w);
  }
  return e;
}

// The stop rule for the iterations first .. first + slots - 1 of a cycle.
static cudaError_t launch_finish(const Solver* s, const StopRule& rule, const Hist& h, int first, int slots,
                                 CycleGuard guard = CycleGuard{}) {
  DevState* st = s->d_state;
  StopRule r = rule;
  Hist hh = h;
  const double* partials = partials_of(s, first);
  int nparts = (int)s->lay.grid_inner;
  long long stride = s->lay.grid_inner * s->nrhs;
  void* args[] = {&st, &r, &hh, &partials, &nparts, &stride, &slots, &guard};
  return launch_pdl(s, (const void*)k_finish_iterations, dim3(s->nrhs), dim3(256), args, 0);
}
// ... of a whole cycle, with the guard of the graph's while loop
static cudaError_t launch_cycle_end(const Solver* s, const StopRule& rule, const Hist& h, CycleGuard guard) {
  const CycleGuard one = s->nrhs == 1 ? guard : CycleGuard{};
  cudaError_t e = launch_finish(s, rule, h, 0, s->nw, one);
  if (e != cudaSuccess || !guard.on || one.on) return e;
  k_cycle_guard<<<1, 32, 0, s->stream>>>(s->d_state, s->nrhs, guard);
  return cudaGetLastError();
}

static cudaError_t launch_iteration(const Solver* s, int it0, bool with_source);

// K3 of the iteration with wiggle w fused with K1 of the next (wiggle w1,
// with the source when that iteration is one of the first Nw)
// T as a 2-D float tensor {2 Ny, Nx Nz Nc nrhs} (one row per y column), box
// {2 LR, N}: the x coordinate of every copy is 2 LR rank floats (a multiple
// of 128 bytes), the row coordinate rhs Nx Nz Nc + plane Nx >= 0.
static cudaError_t ensure_slab_map(Solver* s) {
  const FastInner* f = s->lay.fi;
  if (s->slab_base == s->d_T && s->slab_nrhs == s->nrhs && s->slab_kernel == f->fused_tma) return cudaSuccess;
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return cudaErrorNotSupported;
  const Geom& g = s->g;
  const int LR = g.ny / f->c;
  const cuuint64_t dims[2] = {(cuuint64_t)2 * g.ny, (cuuint64_t)g.nx * g.nz * g.nc * s->nrhs};
  const cuuint64_t strides[1] = {(cuuint64_t)g.ny * sizeof(float2)};
  const cuuint32_t box[2] = {(cuuint32_t)(2 * LR), (cuuint32_t)g.nx};
  const cuuint32_t estr[2] = {1u, 1u};
  if (enc(&s->tmap_slab, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, s->d_T, dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  s->slab_base = s->d_T;
  s->slab_nrhs = s->nrhs;
  s->slab_kernel = f->fused_tma;
  return cudaSuccess;
}

static cudaError_t launch_k3k1(const Solver* s, int w, int w1, bool src_next) {
  const bool tma = s->fused_tma && s->lay.fi->fused_tma;
  if (tma) {
    cudaError_t e = ensure_slab_map(const_cast<Solver*>(s));  // the map cache only
    if (e != cudaSuccess) return e;
  }
  InnerArgs a = inner_args(s, w);
  a.ncols = s->lay.ncols;
  Wig W1 = ramps_of(s, w1);
  const float2* src1 = src_next ? s->d_src : nullptr;
  float2 A = make_float2(0.f, (float)(1.0f / s->eps / (float)s->nw));
  float2* T = s->d_T;
  float2* dE = s->d_dE;
  float2* E = s->d_E;
  const float2* gamma = s->d_gamma;
  const DevState* st = s->d_state;
  double* partials = partials_of(s, w);
  void* args[] = {&a, &W1, &src1, &A, &T, &dE, &E, &gamma, &st, &partials};
  void* args_tma[] = {const_cast<CUtensorMap*>(&s->tmap_slab), &a, &W1, &src1, &A, &T, &dE, &E, &gamma, &st,
                      &partials};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(s->lay.grid_inner * s->nrhs));
  cfg.blockDim = dim3(fast::kThreads);
  cfg.dynamicSmemBytes = s->lay.fi->smem_fused;
  cfg.stream = s->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = s->lay.fi->c;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return tma ? cudaLaunchKernelExC(&cfg, s->lay.fi->fused_tma, args_tma)
             : cudaLaunchKernelExC(&cfg, s->lay.fi->fused, args);
}

// T of the current batch as a 3-D float tensor {2 Ny, Nx, Nz Nc nrhs}, box
// {2 TY, Nx, 1}, for the x pencils: every x coordinate the kernel issues is
// 2 TY yt floats (a multiple of 16 floats, TY >= 8), the others 0 and the
// plane index, both >= 0.
static cudaError_t ensure_xmap(Solver* s) {
  const XPencil* f = s->lay.xp;
  if (s->xmap_base == s->d_T && s->xmap_nrhs == s->nrhs && s->xmap_kernel == f->fwd) return cudaSuccess;
  s->xmap_kernel = nullptr;
  s->x_blocks = 0;
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return cudaErrorNotSupported;
  const Geom& g = s->g;
  const cuuint64_t dims[3] = {(cuuint64_t)2 * g.ny, (cuuint64_t)g.nx, (cuuint64_t)g.nz * g.nc * s->nrhs};
  const cuuint64_t strides[2] = {(cuuint64_t)g.ny * sizeof(float2), (cuuint64_t)g.ny * g.nx * sizeof(float2)};
  const cuuint32_t box[3] = {(cuuint32_t)(2 * f->ty), (cuuint32_t)f->no, 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  if (enc(&s->tmap_X, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, s->d_T, dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  s->xmap_base = s->d_T;
  s->xmap_nrhs = s->nrhs;
  s->xmap_kernel = f->fwd;
  return cudaSuccess;
}

// The x transforms of every (y, z) line of T in place: forward or inverse.
static cudaError_t launch_xpencil(const Solver* cs, bool inv) {
  Solver* s = const_cast<Solver*>(cs);  // the tensor-map cache only
  const XPencil* f = s->lay.xp;
  cudaError_t e = ensure_xmap(s);
  if (e != cudaSuccess) return e;
  if (s->x_blocks <= 0) {
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f->fwd, f->threads, f->smem);
    if (e != cudaSuccess) return e;
    s->x_blocks = std::max(1, per_sm) * kNumSms;
  }
  int ntiles = s->nrhs * s->g.nz * s->g.nc * (s->g.ny / f->ty);
  const unsigned grid = (unsigned)std::min(ntiles, s->x_blocks);
  Geom g = s->g;
  const float2* tw = s->twx;
  const DevState* st = s->d_state;
  long long wc = s->wait_clocks;
  int* err = s->d_err;
  void* args[] = {&s->tmap_X, &g, &tw, &st, &ntiles, &wc, &err};
  return launch_pdl(s, inv ? f->inv : f->fwd, dim3(grid), dim3(f->threads), args, f->smem);
}

// The column pass of the split fused step (kc_col_step): the columns of every
// plane kernel block, no cluster.
static cudaError_t launch_colstep(const Solver* s, int w, int w1, bool src_next) {
  InnerArgs a = inner_args(s, w);
  a.ncols = s->lay.ncols;
  Wig W1 = ramps_of(s, w1);
  const float2* src1 = src_next ? s->d_src : nullptr;
  float2 A = make_float2(0.f, (float)(1.0f / s->eps / (float)s->nw));
  float2* T = s->d_T;
  float2* dE = s->d_dE;
  float2* E = s->d_E;
  const float2* gamma = s->d_gamma;
  const DevState* st = s->d_state;
  double* partials = partials_of(s, w);
  void* args[] = {&a, &W1, &src1, &A, &T, &dE, &E, &gamma, &st, &partials};
  return launch_pdl(s, s->lay.fi->col_step, dim3((unsigned)(s->lay.grid_inner * s->nrhs)), dim3(fast::kThreads), args,
                    s->lay.fi->smem_col);
}

// K3 of an iteration and K1 of the next: one kernel on a cluster, or the
// split step (inverse x pencils, column pass, forward x pencils).
static cudaError_t launch_step(const Solver* s, int w, int w1, bool src_next) {
  if (s->lay.uni_in) {
    cudaError_t e = s->lay.mode3d ? launch_uni_x(s, true, s->d_T) : cudaSuccess;
    if (e != cudaSuccess) return e;
    e = launch_uni_col(s, uni::kStep, w, w1, nullptr, src_next ? s->d_src : nullptr, s->d_T, 1.f);
    return e != cudaSuccess || !s->lay.mode3d ? e : launch_uni_x(s, false, s->d_T);
  }
  if (!s->lay.mode3d) return launch_colstep(s, w, w1, src_next);  // 2-D: K2 already transformed along x
  if (!s->lay.xp) return launch_k3k1(s, w, w1, src_next);
  cudaError_t e = launch_xpencil(s, true);
  if (e != cudaSuccess) return e;
  if ((e = launch_colstep(s, w, w1, src_next)) != cudaSuccess) return e;
  return launch_xpencil(s, false);
}

// One iteration of the fused loop: T already holds K1's output for it.
static cudaError_t launch_iteration_fused(const Solver* s, int i, bool src_next) {
  const int w = i % s->nw, w1 = (i + 1) % s->nw;
  cudaError_t e = launch_k2(s, w);
  return e != cudaSuccess ? e : launch_step(s, w, w1, src_next);
}

// A steady iteration (no source) of the loop, fused or not.
static cudaError_t launch_steady(const Solver* s, int i) {
  return s->fuse ? launch_iteration_fused(s, i, false) : launch_iteration(s, i, false);
}

static cudaError_t launch_iteration(const Solver* s, int it0, bool with_source) {
  const int w = it0 % s->nw;
  cudaError_t e = launch_k1(s, w, with_source);
  if (e != cudaSuccess) return e;
  e = launch_k2(s, w);
  if (e != cudaSuccess) return e;
  return launch_k3_only(s, w);
}

// Whether nrhs right-hand sides can run as one launch of the loop
// (uni::k_loop): a column tile of each on an SM of its own.
static bool loop_fits(const Solver* s, int nrhs) {
  return s->has_loop && nrhs <= uni::kLoopRhs && nrhs * s->lays[1].ucol.grid <= s->loop_blocks &&
         loop_smem(s->lays[1], s->g, s->nw, false) <= kLoopSmem;
}

// A launch of a loop kernel with arguments `args`, whose barrier counter is at
// *arrived: cooperative, or one cluster where 16 blocks have all the tiles (then
// without a counter).
static cudaError_t launch_coop(const Solver* s, const void* fn, size_t smem, int nrhs, void* args, unsigned** arrived) {
  const Layout& L = s->lay;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)std::min<long long>(loop_tiles(s, nrhs), s->loop_blocks));
  const bool cluster = loop_cluster(s, nrhs);
  *arrived = cluster ? nullptr : (unsigned*)(s->d_err + 1);
  if (!cluster) {
    const cudaError_t e = cudaMemsetAsync(*arrived, 0, sizeof(unsigned), s->stream);
    if (e != cudaSuccess) return e;
  }
  cfg.blockDim = dim3(loop_threads(L));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s->stream;
  cudaLaunchAttribute attr[1];
  if (cluster) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cfg.gridDim.x;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* argv[] = {args};
  return cudaLaunchKernelExC(&cfg, fn, argv);
}

static long long barrier_limit(const Solver* s) { return s->wait_clocks > 0 ? s->wait_clocks : uni::kBarrierClocks; }

// Cycles of the loop in one cooperative launch, from T as K1 left it, until
// every right-hand side is done or max_cycles have run.
static cudaError_t launch_loop(const Solver* s, const StopRule& rule, const Hist& h, long long max_cycles) {
  const Layout& L = s->lay;
  uni::LoopArgs a{};
  a.col = uni_col_args(s, 0, 0, nullptr, nullptr, s->d_T, 1.f);
  a.pen = uni_pencil_args(s, 0);
  a.wig = s->ut[1].wigs;
  a.src = s->d_src;
  a.partials = s->d_partials;
  a.st = s->d_state;
  a.rule = rule;
  a.hist = h;
  a.err = s->d_err;
  a.limit = barrier_limit(s);
  a.max_cycles = max_cycles;
  a.nw = s->nw;
  a.nrhs = s->nrhs;
  const void* fn = uni_kernels(std::max(L.ucol.plan.cls, L.uout.plan.cls)).loop;
  a.groups = uni_groups(L.ucol);
  a.e_resident = loop_smem(L, s->g, s->nw, true) <= kLoopSmem;
  const size_t smem = loop_smem(L, s->g, s->nw, a.e_resident != 0, &a.tile_elems);
  return launch_coop(s, fn, smem, s->nrhs, &a, &a.arrived);
}

// Energy histories: per right-hand side r, diff at r * 2cap and fresh at r * 2cap + cap.
static int ensure_hist(Solver* s, long long cap) {
  if (s->hist_cap >= cap) return WS_OK;
  if (s->d_hist) cudaFree(s->d_hist);
  s->d_hist = nullptr;
  s->hist_cap = 0;
  free_graph(s);  // graphs hold the old pointer
  WS_CUDA(cudaMalloc(&s->d_hist, 2 * cap * std::max(1, s->batch_cap) * sizeof(double)));
  s->hist_cap = cap;
  return WS_OK;
}

// The prologue and first wiggle cycle of a solve (with the source).  Cold:
// the reference's iterations 1..Nw from E' = dE' = 0.  Warm (d_init holds
// v = u/Nw, see k_warm_scale): a cold probe iteration for diff_energy(1),
// the residual probe of the start and the discard check (k_warm_resid_*,
// k_warm_check), the restart from dE' = v, E' = 0, iterations 1..Nw with the
// source and the shift dE' -= v.
static cudaError_t launch_prologue(const Solver* s, const StopRule& rule, const Hist& h, CycleGuard guard) {
  const size_t nbytes = field_elems(s) * s->nrhs * sizeof(float2);
  cudaError_t e;
  if ((e = cudaMemsetAsync(s->d_E, 0, nbytes, s->stream)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(s->d_dE, 0, nbytes, s->stream)) != cudaSuccess) return e;
  k_reset_state<<<1, 256, 0, s->stream>>>(s->d_state, s->nrhs);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (s->warm) {
    if ((e = launch_iteration(s, 0, true)) != cudaSuccess) return e;  // the probe
    if ((e = launch_finish(s, rule, h, 0, 1)) != cudaSuccess) return e;
    const long long n = (long long)field_elems(s) * s->nrhs;
    const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 8 * kNumSms);
    const float nw = (float)s->nw;
    if (s->warm_ratio > 0.0) {
      // residual of the start: one iteration from dE' = u with the whole source
      k_warm_resid_begin<<<blocks, 256, 0, s->stream>>>(s->d_dE, s->d_init, n, nw);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      if ((e = launch_k1_io(s, 0, s->d_dE, s->d_src, s->d_T, nw)) != cudaSuccess) return e;
      if ((e = launch_k2(s, 0)) != cudaSuccess) return e;
      if ((e = launch_k3_only(s, 0)) != cudaSuccess) return e;
      const long long fe = (long long)field_elems(s);
      const unsigned bpr = (unsigned)std::max<long long>(1, std::min<long long>((fe + 255) / 256, 4 * kNumSms));
      k_warm_resid_energy<<<dim3(bpr, s->nrhs), 256, 0, s->stream>>>(s->d_dE, s->d_init, s->g, fe, nw,
                                                                     s->d_state);
    }
    k_warm_begin<<<blocks, 256, 0, s->stream>>>(s->d_dE, s->d_E, s->d_init, n);
    k_warm_restart<<<1, 256, 0, s->stream>>>(s->d_state, s->nrhs);
    if (s->warm_ratio > 0.0)
      k_warm_check<<<1, 256, 0, s->stream>>>(s->d_state, s->nrhs, s->warm_ratio, (double)s->nw * s->nw);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (s->fuse) {
    // K1 of the first iteration, then each fused step also computes K1 of the
    // next iteration (with the source while that one is among the first Nw)
    if ((e = launch_k1(s, 0, true)) != cudaSuccess) return e;
    for (int i = 0; i < s->nw; ++i)
      if ((e = launch_iteration_fused(s, i, i + 1 < s->nw)) != cudaSuccess) return e;
  } else {
    for (int i = 0; i < s->nw; ++i)
      if ((e = launch_iteration(s, i, true)) != cudaSuccess) return e;
  }
  if (!s->warm) return launch_cycle_end(s, rule, h, guard);
  if ((e = launch_finish(s, rule, h, 0, s->nw)) != cudaSuccess) return e;
  {
    const long long fe = (long long)field_elems(s);
    const unsigned bpr = (unsigned)std::max<long long>(1, std::min<long long>((fe + 255) / 256, 4 * kNumSms));
    k_warm_shift<<<dim3(bpr, s->nrhs), 256, 0, s->stream>>>(s->d_dE, s->d_init, s->g, fe, s->d_state);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // the shift changed dE': the fused loop's T is recomputed from it
    if (s->fuse && (e = launch_k1(s, 0, false)) != cudaSuccess) return e;
  }
  if (guard.on) k_cycle_guard<<<1, 32, 0, s->stream>>>(s->d_state, s->nrhs, guard);
  return cudaGetLastError();
}

static int build_graph(Solver* s, const StopRule& rule, const Hist& h) {
  free_graph(s);
  // the stop rule can only end the loop at a multiple of Nw, at the latest at
  // the first multiple >= max_iter: this many cycles always suffice
  const long long max_cycles = (rule.max_iter + s->nw - 1) / s->nw + 1;
  cudaGraph_t graph;
  WS_CUDA(cudaGraphCreate(&graph, 0));
  cudaGraphConditionalHandle cond;
  cudaError_t e = cudaGraphConditionalHandleCreate(&cond, graph, 1, cudaGraphCondAssignDefault);
  if (e != cudaSuccess) {
    cudaGraphDestroy(graph);
    return fail(WS_ERR_CUDA, std::string("cudaGraphConditionalHandleCreate: ") + cudaGetErrorString(e));
  }
  // prologue + first cycle (with the source)
  e = cudaStreamBeginCaptureToGraph(s->stream, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    e = launch_prologue(s, rule, h, CycleGuard{1, cond, max_cycles});
    cudaGraph_t g2 = graph;
    cudaError_t e2 = cudaStreamEndCapture(s->stream, &g2);
    if (e == cudaSuccess) e = e2;
  }
  if (e != cudaSuccess) {
    cudaGraphDestroy(graph);
    return fail(WS_ERR_CUDA, std::string("graph capture (first cycle): ") + cudaGetErrorString(e));
  }
  // sink node of the captured chain
  size_t nn = 0;
  cudaGraphGetNodes(graph, nullptr, &nn);
  std::vector<cudaGraphNode_t> nodes(nn);
  cudaGraphGetNodes(graph, nodes.data(), &nn);
  std::vector<cudaGraphNode_t> sinks;
  for (auto n : nodes) {
    size_t nd = 0;
    cudaGraphNodeGetDependentNodes(n, nullptr, &nd);
    if (nd == 0) sinks.push_back(n);
  }
  cudaGraphNodeParams cp{};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = cond;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t cnode;
  e = cudaGraphAddNode(&cnode, graph, sinks.data(), sinks.size(), &cp);
  if (e != cudaSuccess) {
    cudaGraphDestroy(graph);
    return fail(WS_ERR_CUDA, std::string("cudaGraphAddNode(while): ") + cudaGetErrorString(e));
  }
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  e = cudaStreamBeginCaptureToGraph(s->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    for (int i = 0; i < s->nw && e == cudaSuccess; ++i) e = launch_steady(s, i);
    if (e == cudaSuccess) e = launch_cycle_end(s, rule, h, CycleGuard{1, cond, max_cycles});
    cudaGraph_t b2 = body;
    cudaError_t e2 = cudaStreamEndCapture(s->stream, &b2);
    if (e == cudaSuccess) e = e2;
  }
  if (e != cudaSuccess) {
    cudaGraphDestroy(graph);
    return fail(WS_ERR_CUDA, std::string("graph capture (while body): ") + cudaGetErrorString(e));
  }
  e = cudaGraphInstantiate(&s->gexec, graph, 0);
  if (e != cudaSuccess) {
    cudaGraphDestroy(graph);
    s->gexec = nullptr;
    return fail(WS_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
  }
  s->graph = graph;
  return WS_OK;
}

// Source.add_to for every block of every right-hand side into the dense
// source fields (r at r * field elements); source energies into energy[r].
static int upload_sources(Solver* s, int nrhs, const int64_t* counts, const ws_source_block* src, int memory,
                          std::vector<double>& energy) {
  const Geom& g = s->g;
  const size_t F = field_elems(s);
  WS_CUDA(cudaMemsetAsync(s->d_src, 0, F * nrhs * sizeof(float2), s->stream));
  WS_CUDA(cudaMemsetAsync(s->d_energy, 0, nrhs * sizeof(double), s->stream));
  size_t need = 0, sum = 0;
  long long total = 0;
  for (int r = 0; r < nrhs; ++r) total += counts[r];
  for (long long b = 0; b < total; ++b) {
    const ws_source_block& B = src[b];
    size_t n = 1;
    for (int d = 0; d < 4; ++d) {
      const int64_t lim = d == 0 ? g.ny : d == 1 ? g.nx : d == 2 ? g.nz : g.nc;
      if (B.size[d] < 1 || B.position[d] < 1 || B.position[d] + B.size[d] - 1 > lim)
        return fail(WS_ERR_INVALID_ARGUMENT, "source block outside the grid (crop it first, Source.m:81-103)");
      n *= (size_t)B.size[d];
    }
    if (!B.values) return fail(WS_ERR_INVALID_ARGUMENT, "null source values");
    need = std::max(need, n);
    sum += n;
  }
  if (need > s->stage_cap && memory != WS_DEVICE) {
    if (s->d_stage) cudaFree(s->d_stage);
    s->d_stage = nullptr;
    s->stage_cap = 0;
    WS_CUDA(cudaMalloc(&s->d_stage, need * sizeof(float2)));
    s->stage_cap = need;
  }
  // the energies (only whether there is a source) of small host blocks come
  // from the host, so that nothing waits for the device here; the copies and
  // kernels share the staging buffer in stream order, and a pageable copy has
  // taken its values when it returns
  energy.assign(nrhs, 0.0);
  const bool on_host = memory != WS_DEVICE && sum <= (1u << 16);
  long long b = 0;
  for (int r = 0; r < nrhs; ++r) {
    for (int64_t k = 0; k < counts[r]; ++k, ++b) {
      const ws_source_block& B = src[b];
      const size_t n = (size_t)(B.size[0] * B.size[1] * B.size[2] * B.size[3]);
      const float2* vals = (const float2*)B.values;
      if (on_host)
        for (size_t i = 0; i < n; ++i) energy[r] += (double)std::fmaf(vals[i].x, vals[i].x, vals[i].y * vals[i].y);
      if (memory != WS_DEVICE) {
        WS_CUDA(cudaMemcpyAsync(s->d_stage, B.values, n * sizeof(float2), cudaMemcpyHostToDevice, s->stream));
        vals = s->d_stage;
      }
      const int th = 256;
      const long long blocks = std::min<long long>((n + th - 1) / th, 4096);
      k_scatter_source<<<(unsigned)std::max(1LL, blocks), th, 0, s->stream>>>(
          s->d_src + F * r, vals, g, (int)B.position[0] - 1, (int)B.position[1] - 1, (int)B.position[2] - 1,
          (int)B.position[3] - 1, (int)B.size[0], (int)B.size[1], (int)B.size[2], (int)B.size[3], s->d_energy + r);
      WS_CUDA(cudaGetLastError());
    }
  }
  if (on_host) return WS_OK;
  WS_CUDA(cudaMemcpyAsync(energy.data(), s->d_energy, nrhs * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
  WS_CUDA(cudaStreamSynchronize(s->stream));
  return WS_OK;
}

// One plane-wave block per right-hand side into the dense source fields.
static int generate_plane_waves(Solver* s, int nrhs, const ws_plane_wave* waves, std::vector<double>& energy) {
  const Geom& g = s->g;
  const size_t F = field_elems(s);
  WS_CUDA(cudaMemsetAsync(s->d_src, 0, F * nrhs * sizeof(float2), s->stream));
  WS_CUDA(cudaMemsetAsync(s->d_energy, 0, nrhs * sizeof(double), s->stream));
  for (int r = 0; r < nrhs; ++r) {
    const ws_plane_wave& W = waves[r];
    PlaneWaveArgs a{};
    long long n = 1;
    for (int d = 0; d < 4; ++d) {
      const int64_t lim = d == 0 ? g.ny : d == 1 ? g.nx : d == 2 ? g.nz : g.nc;
      if (W.size[d] < 1 || W.position[d] < 1 || W.position[d] + W.size[d] - 1 > lim)
        return fail(WS_ERR_INVALID_ARGUMENT, "plane-wave block outside the grid (crop it first, Source.m:81-103)");
      a.p[d] = (int)W.position[d] - 1;
      a.sz[d] = (int)W.size[d];
      n *= W.size[d];
    }
    a.amp_re = W.amplitude.re;
    a.amp_im = W.amplitude.im;
    a.phase0 = W.phase0;
    for (int d = 0; d < 3; ++d) a.phase[d] = W.phase[d];
    const long long blocks = std::min<long long>((n + 255) / 256, 4096);
    k_plane_wave_source<<<(unsigned)std::max(1LL, blocks), 256, 0, s->stream>>>(s->d_src + F * r, g, a,
                                                                                s->d_energy + r);
    WS_CUDA(cudaGetLastError());
  }
  energy.assign(nrhs, 0.0);
  WS_CUDA(cudaMemcpyAsync(energy.data(), s->d_energy, nrhs * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
  WS_CUDA(cudaStreamSynchronize(s->stream));
  return WS_OK;
}

static size_t roi_elems(const Geom& g) {
  return (size_t)(g.r1[0] - g.r0[0]) * (g.r1[1] - g.r0[1]) * (g.r1[2] - g.r0[2]) * (g.r1[3] - g.r0[3]);
}

// One batch of nrhs right-hand sides on the solver's medium.  Each one follows
// the reference loop and stop rule on its own; a converged one stops working
// while the others continue.
static int solve_batch(Solver* s, int nrhs, const int64_t* counts, const ws_source_block* src, int source_memory,
                       const ws_solve_options* o, ws_complex* E_out, int out_memory, double* diff_out,
                       int64_t diff_cap, int64_t* n_it, int* converged, const ws_plane_wave* waves = nullptr) {
  WS_CUDA(cudaSetDevice(s->device));
  ws_solve_options opt;
  ws_default_options(&opt);
  if (o) opt = *o;
  if (nrhs < 1 || nrhs > 65536) return fail(WS_ERR_INVALID_ARGUMENT, "number of right-hand sides must be in [1, 65536]");
  if (s->n_media > 1 && nrhs != s->n_media)
    return fail(WS_ERR_INVALID_ARGUMENT, "a solver of several media takes one right-hand side per medium");
  if (opt.max_iterations < 1 || opt.max_iterations > 100000000LL)
    return fail(WS_ERR_INVALID_ARGUMENT, "max_iterations must be in [1, 1e8]");
  if (opt.energy_interval < 1) return fail(WS_ERR_INVALID_ARGUMENT, "energy_interval must be >= 1");
  if (!waves) {
    if (!counts || !src) return fail(WS_ERR_NO_SOURCE, "no source blocks");
    for (int r = 0; r < nrhs; ++r)
      if (counts[r] < 1) return fail(WS_ERR_NO_SOURCE, "a right-hand side has no source blocks");
  }
  const bool want_cb = opt.callback && opt.callback_type && std::strcmp(opt.callback_type, "NoCallback") != 0;
  if (want_cb && nrhs > 1) return fail(WS_ERR_INVALID_ARGUMENT, "callbacks need a single right-hand side");
  if (s->lay.grid_inner * (long long)nrhs > (1LL << 31) - 1 || s->lay.grid_outer * (long long)nrhs > (1LL << 31) - 1)
    return fail(WS_ERR_INVALID_ARGUMENT, "batch too large for one launch");
  WS_CUDA(use_layout(s, loop_fits(s, nrhs) ? 1 : 0));
  int rc = ensure_batch(s, nrhs);
  if (rc) return rc;
  rc = ensure_partials(s, s->lay.grid_inner * (long long)nrhs * s->nw);
  if (rc) return rc;
  if (s->nrhs != nrhs) free_graph(s);
  s->nrhs = nrhs;
  std::vector<double> src_energy;
  rc = waves ? generate_plane_waves(s, nrhs, waves, src_energy)
             : upload_sources(s, nrhs, counts, src, source_memory, src_energy);
  if (rc) return rc;
  for (int r = 0; r < nrhs; ++r)
    if (!(src_energy[r] > 0)) return fail(WS_ERR_NO_SOURCE, "There is no source inside the grid boundaries");
  // the loop can run at most max_iterations + Nw - 1 iterations
  const long long cap = opt.max_iterations + s->nw;
  rc = ensure_hist(s, cap);
  if (rc) return rc;
  StopRule rule{};
  rule.nw = s->nw;
  rule.fresh = opt.stop_rule == WS_STOP_FRESH;
  rule.nan_stop = opt.stop_on_nonfinite ? 1 : 0;
  rule.interval = (int)std::min<int64_t>(opt.energy_interval, 1 << 30);
  rule.max_iter = opt.max_iterations;
  rule.threshold = opt.energy_threshold;
  const long long hs_stride = 2 * s->hist_cap;
  Hist h{s->d_hist, s->d_hist + s->hist_cap, s->hist_cap, hs_stride};
  s->warm = opt.initial_field != nullptr;
  s->warm_ratio = opt.warm_discard_ratio;
  if (s->warm) {
    const long long fe = (long long)field_elems(s);
    if (!s->d_init) WS_CUDA(cudaMalloc(&s->d_init, fe * s->batch_cap * sizeof(float2)));
    WS_CUDA(cudaMemcpyAsync(s->d_init, opt.initial_field, fe * nrhs * sizeof(float2),
                            opt.initial_memory == WS_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                            s->stream));
    const long long n = fe * nrhs;
    k_warm_scale<<<(unsigned)std::min<long long>((n + 255) / 256, 8 * kNumSms), 256, 0, s->stream>>>(
        s->d_init, s->d_gamma, n, s->g.npts, 1.0f / (float)s->nw, opt.initial_is_eprime ? 1 : 0,
        (long long)field_elems(s), s->n_media > 1 ? (long long)s->g.npts : 0LL);
    WS_CUDA(cudaGetLastError());
  }
  const bool in_one = s->active == 1 && s->fuse;  // the loop as one launch, or one per cycle
  // What comes back with the first wait: the states, the error flag and the
  // first kHead energies of each right-hand side.
  constexpr size_t kHead = 4096;
  const bool head = diff_out && nrhs <= 16;
  const size_t state_bytes = (nrhs * sizeof(DevState) + 15) / 16 * 16;
  HostLease back(state_bytes + 16 + (head ? nrhs * kHead * sizeof(double) : 0));
  if (!back.p) return fail(WS_ERR_OUT_OF_MEMORY, "no memory for the loop's state");
  const DevState* const hs = (const DevState*)back.p;
  const int* const kerr = (const int*)((char*)back.p + state_bytes);
  const double* const hhead = (const double*)((char*)back.p + state_bytes + 16);
  const long long nhead = std::min<long long>((long long)kHead, s->hist_cap);
  auto fetch_state = [&]() -> cudaError_t {
    back.queued(s->stream);
    cudaError_t e = cudaMemcpyAsync((void*)hs, s->d_state, nrhs * sizeof(DevState), cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync((void*)kerr, s->d_err, sizeof(int), cudaMemcpyDeviceToHost, s->stream);
    for (int r = 0; head && r < nrhs && e == cudaSuccess; ++r)
      e = cudaMemcpyAsync((void*)(hhead + r * kHead), s->d_hist + r * hs_stride, nhead * sizeof(double),
                          cudaMemcpyDeviceToHost, s->stream);
    return e;
  };
  auto wait = [&]() -> cudaError_t {
    const cudaError_t e = cudaStreamSynchronize(s->stream);
    if (e == cudaSuccess) back.settled();
    return e;
  };
  auto all_done = [&]() {
    bool all = true;
    for (int r = 0; r < nrhs; ++r) all = all && hs[r].done;
    return all;
  };
  // The fields: E' itself, or E on the roi through k_finalize (in groups of
  // right-hand sides for host memory, so that the device copy stays below 512 MB or
  // one field; smaller groups where that does not fit.  The solver keeps up to 128 MB
  // of it: 96 fields of 960^2 after 20 iterations take 62 ms, 57 with all of it kept,
  // 68 in groups of 128 MB).
  const size_t F = field_elems(s);
  const bool field = opt.output == WS_OUTPUT_FIELD;
  const size_t per = (field ? roi_elems(s->g) : F) * sizeof(float2);  // bytes of a right-hand side
  const bool to_host = E_out && out_memory != WS_DEVICE;
  int group = (int)std::min<size_t>(nrhs, std::max<size_t>(1, (512u << 20) / per));
  if (to_host && field && group * (per / sizeof(float2)) > s->out_cap) {
    if (s->d_out) cudaFree(s->d_out);
    s->d_out = nullptr;
    s->out_cap = 0;
    cudaError_t e;
    group = fitting_group(group, [&](int n) { return cudaMalloc(&s->d_out, n * per); }, &e);
    WS_CUDA(e);
    s->out_cap = group * (per / sizeof(float2));
  }
  bool pageable = false;
  if (to_host) {
    cudaPointerAttributes at{};
    pageable = cudaPointerGetAttributes(&at, E_out) != cudaSuccess || at.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
  }
  // E of right-hand sides r0 .. r1 - 1 where the caller wants it, or in d_out
  auto finalize = [&](int r0, int r1) -> cudaError_t {
    for (int r = r0; r < r1 && field; ++r) {
      const size_t n = per / sizeof(float2);
      const long long blocks = std::min<long long>(((long long)n + 255) / 256, 8 * kNumSms);
      k_finalize<<<(unsigned)blocks, 256, 0, s->stream>>>(
          s->d_E + F * r, s->d_gamma + (s->n_media > 1 ? (long long)r * s->g.npts : 0LL), s->g,
          to_host ? s->d_out + n * (r - r0) : (float2*)E_out + n * r);
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  };
  std::unique_ptr<OutCopy> copy;  // of the first group: its threads touch the caller's pages meanwhile
  auto begin_copy = [&]() -> cudaError_t {
    if (!pageable) return cudaSuccess;
    if (!copy) copy.reset(new OutCopy(E_out, per * group, s->device));
    if (!copy->ok()) return cudaErrorMemoryAllocation;  // no host memory at all
    const cudaError_t e = copy->stage(field ? (const void*)s->d_out : (const void*)s->d_E, s->stream);
    copy->touch();
    return e;
  };
  if (opt.use_graph && !want_cb && in_one) {
    if (s->warm) {
      WS_CUDA(launch_prologue(s, rule, h, CycleGuard{}));
    } else {
      const size_t nbytes = field_elems(s) * nrhs * sizeof(float2);
      WS_CUDA(cudaMemsetAsync(s->d_E, 0, nbytes, s->stream));
      WS_CUDA(cudaMemsetAsync(s->d_dE, 0, nbytes, s->stream));
      k_reset_state<<<1, 256, 0, s->stream>>>(s->d_state, nrhs);
      WS_CUDA(launch_k1(s, 0, true));
    }
    // as many launches as the iteration bound can take, each of a bounded length
    const long long max_cycles = (rule.max_iter + s->nw - 1) / s->nw + 1;
    for (long long cycle = 0; cycle < max_cycles; cycle += kLoopCycles) {
      WS_CUDA(launch_loop(s, rule, h, std::min(kLoopCycles, max_cycles - cycle)));
      if (E_out) WS_CUDA(finalize(0, to_host ? group : nrhs));
      WS_CUDA(fetch_state());
      WS_CUDA(begin_copy());
      WS_CUDA(wait());
      if (all_done() || *kerr) break;
    }
  } else if (opt.use_graph && !want_cb) {
    GraphKey key{rule.threshold, rule.max_iter, rule.interval, opt.stop_rule, rule.nan_stop, nrhs,
                 s->warm ? 1 : 0, s->active, s->warm ? s->warm_ratio : 0.0};
    if (!s->gexec || !(key == s->gkey)) {
      rc = build_graph(s, rule, h);
      if (rc) return rc;
      s->gkey = key;
    }
    WS_CUDA(cudaGraphLaunch(s->gexec, s->stream));
    if (E_out) WS_CUDA(finalize(0, to_host ? group : nrhs));
    WS_CUDA(fetch_state());
    WS_CUDA(begin_copy());
    WS_CUDA(wait());
  } else {
    std::vector<double> hist;
    const long long cb_int = std::max<int64_t>(1, opt.callback_interval);
    const long long max_cycles = (rule.max_iter + s->nw - 1) / s->nw + 1;
    for (long long cycle = 0;; ++cycle) {
      if (cycle >= max_cycles) return fail(WS_ERR_CUDA, "loop did not stop within max_iterations (internal error)");
      if (cycle == 0) {
        WS_CUDA(launch_prologue(s, rule, h, CycleGuard{}));
      } else {
        if (in_one) {
          WS_CUDA(launch_loop(s, rule, h, 1));
        } else {
          for (int i = 0; i < s->nw; ++i) WS_CUDA(launch_steady(s, i));
          WS_CUDA(launch_cycle_end(s, rule, h, CycleGuard{}));
        }
      }
      WS_CUDA(fetch_state());
      WS_CUDA(wait());
      if (want_cb) {
        const long long done_it = hs[0].it - 1;
        hist.resize(done_it);
        WS_CUDA(cudaMemcpy(hist.data(), s->d_hist, done_it * sizeof(double), cudaMemcpyDeviceToHost));
        for (long long k = done_it - s->nw + 1; k <= done_it; ++k)
          if (k >= 1 && (k % cb_int == 0 || (hs[0].done && k == done_it)))
            opt.callback(opt.callback_type, hist.data(), k, opt.energy_threshold, opt.user_data);
      }
      if (all_done() || (in_one && *kerr)) break;
    }
    if (E_out) WS_CUDA(finalize(0, to_host ? group : nrhs));
  }
  if (*kerr) {
    cudaMemset(s->d_err, 0, sizeof(int));
    return fail(WS_ERR_CUDA, "a bounded wait of the FFT kernels (cluster exchange, TMA tile load or the loop's barrier) timed out");
  }
  bool diverged = false;
  for (int r = 0; r < nrhs; ++r) {
    const long long n_iter = hs[r].it - 1;
    if (n_it) n_it[r] = n_iter;
    if (converged) converged[r] = hs[r].converged;
    diverged = diverged || hs[r].status == WS_ERR_DIVERGED;
    const long long nd = std::min<long long>(std::min(n_iter, cap), diff_cap);
    if (!diff_out || nd <= 0) continue;
    if (head && nd <= nhead)
      std::memcpy(diff_out + r * diff_cap, hhead + r * kHead, nd * sizeof(double));
    else
      WS_CUDA(cudaMemcpy(diff_out + r * diff_cap, s->d_hist + r * hs_stride, nd * sizeof(double),
                         cudaMemcpyDeviceToHost));
  }
  if (E_out) {
    for (int r0 = 0; to_host && r0 < nrhs; r0 += group) {
      const int r1 = std::min(nrhs, r0 + group);
      if (r0 > 0) WS_CUDA(finalize(r0, r1));
      char* const dst = (char*)E_out + per * r0;
      const void* const from = field ? (const void*)s->d_out : (const void*)(s->d_E + F * r0);
      if (pageable) {
        if (r0 > 0 || !copy) {
          copy.reset(new OutCopy(dst, per * (r1 - r0), s->device));
          if (!copy->ok()) return fail(WS_ERR_OUT_OF_MEMORY, "no memory for the fields");
          WS_CUDA(copy->stage(from, s->stream));
          WS_CUDA(cudaStreamSynchronize(s->stream));
        }
        WS_CUDA(copy->run());
      } else {
        WS_CUDA(cudaMemcpyAsync(dst, from, per * (r1 - r0), cudaMemcpyDeviceToHost, s->stream));
        WS_CUDA(cudaStreamSynchronize(s->stream));  // d_out takes the next group
      }
    }
    if (!to_host && !field)
      WS_CUDA(cudaMemcpyAsync(E_out, s->d_E, F * nrhs * sizeof(float2), cudaMemcpyDeviceToDevice, s->stream));
    WS_CUDA(cudaStreamSynchronize(s->stream));
    if (s->out_cap * sizeof(float2) > (128u << 20) && group > 1) {
      cudaFree(s->d_out);
      s->d_out = nullptr;
      s->out_cap = 0;
    }
  }
  if (diverged) return fail(WS_ERR_DIVERGED, "residual energy is not finite");
  return WS_OK;
}

static int solve(Solver* s, int64_t n_blocks, const ws_source_block* src, int source_memory,
                 const ws_solve_options* o, ws_complex* E_out, int out_memory, double* diff_out, int64_t* n_it,
                 int* converged) {
  if (n_blocks < 1 || !src) return fail(WS_ERR_NO_SOURCE, "no source blocks");
  const int64_t counts[1] = {n_blocks};
  const int64_t maxit = o ? o->max_iterations : 100000;
  return solve_batch(s, 1, counts, src, source_memory, o, E_out, out_memory, diff_out, maxit + s->nw, n_it,
                     converged);
}

}  // namespace ws

using namespace ws;

// ws_run_algorithm's solver of the previous call, per device
static constexpr int kRunCacheDevices = 64;
static Solver* g_run_cache[kRunCacheDevices] = {};
static std::mutex g_run_mu;

extern "C" {

void ws_default_options(ws_solve_options* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->max_iterations = 100000;
  o->energy_threshold = 1e-2;
  o->energy_interval = 8;
  o->stop_rule = WS_STOP_REFERENCE;
  o->output = WS_OUTPUT_EPRIME;
  o->stop_on_nonfinite = 1;
  o->use_graph = 1;
  o->callback_type = "NoCallback";
  o->callback_interval = 50;
}

const char* ws_version(void) { return "wavesim_b200 0.1.0 (sm_100a)"; }

const char* ws_last_error(void) { return g_last_error.c_str(); }

int ws_size_supported(const int64_t N[4]) {
  if (!N || (N[3] != 1 && N[3] != 3)) return 0;
  Geom g{};
  g.ny = (int)N[0];
  g.nx = (int)N[1];
  g.nz = (int)N[2];
  g.nc = (int)N[3];
  for (int d = 0; d < 3; ++d)
    if (N[d] < 1 || !length_supported((int)N[d])) return 0;
  Layout L;
  std::string why;
  return make_layout(g, L, why) == WS_OK;
}

int ws_solver_create(const int64_t N[4], const ws_complex* gamma, int64_t n_wiggles, const ws_wiggle* wiggles,
                     float epsilon, ws_complex k02e, const int64_t roi[8], int memory, int device, ws_solver* out) {
  if (!out) return fail(WS_ERR_INVALID_ARGUMENT, "null output handle");
  *out = nullptr;
  Solver* s = nullptr;
  const int rc = create_solver(N, gamma, n_wiggles, wiggles, epsilon, k02e, roi, memory, device, &s);
  if (rc) return rc;
  *out = reinterpret_cast<ws_solver>(s);
  return WS_OK;
}

int ws_solver_create_media(const int64_t N[4], int64_t n_media, const ws_complex* gammas, int64_t n_wiggles,
                           const ws_wiggle* wiggles, float epsilon, ws_complex k02e, const int64_t roi[8], int memory,
                           int device, ws_solver* out) {
  if (!out) return fail(WS_ERR_INVALID_ARGUMENT, "null output handle");
  *out = nullptr;
  if (n_media < 1 || n_media > 65536) return fail(WS_ERR_INVALID_ARGUMENT, "n_media must be in [1, 65536]");
  if (!gammas) return fail(WS_ERR_INVALID_ARGUMENT, "null gammas");
  Solver* s = nullptr;
  const int rc = create_solver(N, gammas, n_wiggles, wiggles, epsilon, k02e, roi, memory, device, &s);
  if (rc) return rc;
  if (n_media > 1) {
    const size_t bytes = (size_t)s->g.npts * sizeof(float2);
    cudaFree(s->d_gamma);
    s->d_gamma = nullptr;
    cudaError_t e = cudaMalloc(&s->d_gamma, bytes * (size_t)n_media);
    if (e == cudaSuccess)
      e = cudaMemcpy(s->d_gamma, gammas, bytes * (size_t)n_media,
                     memory == WS_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      destroy_solver(s);
      return fail(e == cudaErrorMemoryAllocation ? WS_ERR_OUT_OF_MEMORY : WS_ERR_CUDA,
                  std::string("media gammas: ") + cudaGetErrorString(e));
    }
    s->n_media = (int)n_media;
  }
  *out = reinterpret_cast<ws_solver>(s);
  return WS_OK;
}

int ws_solver_solve(ws_solver h, int64_t n_blocks, const ws_source_block* source, int source_memory,
                    const ws_solve_options* opts, ws_complex* E_out, int out_memory, double* diff_energy_out,
                    int64_t* n_iterations, int* converged) {
  if (!h) return fail(WS_ERR_INVALID_ARGUMENT, "null solver");
  return solve(reinterpret_cast<Solver*>(h), n_blocks, source, source_memory, opts, E_out, out_memory,
               diff_energy_out, n_iterations, converged);
}

int ws_solver_solve_batch(ws_solver h, int64_t n_rhs, const int64_t* block_counts, const ws_source_block* blocks,
                          int source_memory, const ws_solve_options* opts, ws_complex* E_out, int out_memory,
                          double* diff_energy_out, int64_t diff_capacity, int64_t* n_iterations, int* converged) {
  if (!h) return fail(WS_ERR_INVALID_ARGUMENT, "null solver");
  return solve_batch(reinterpret_cast<Solver*>(h), (int)n_rhs, block_counts, blocks, source_memory, opts, E_out,
                     out_memory, diff_energy_out, diff_capacity, n_iterations, converged);
}

int ws_solver_solve_plane_waves(ws_solver h, int64_t n_rhs, const ws_plane_wave* waves, const ws_solve_options* opts,
                                ws_complex* E_out, int out_memory, double* diff_energy_out, int64_t diff_capacity,
                                int64_t* n_iterations, int* converged) {
  if (!h) return fail(WS_ERR_INVALID_ARGUMENT, "null solver");
  if (!waves) return fail(WS_ERR_NO_SOURCE, "no plane waves");
  return solve_batch(reinterpret_cast<Solver*>(h), (int)n_rhs, nullptr, nullptr, WS_HOST, opts, E_out, out_memory,
                     diff_energy_out, diff_capacity, n_iterations, converged, waves);
}

int ws_solver_buffers(ws_solver h, void** E_prime, void** stream) {
  if (!h) return fail(WS_ERR_INVALID_ARGUMENT, "null solver");
  Solver* s = reinterpret_cast<Solver*>(h);
  if (E_prime) *E_prime = s->d_E;
  if (stream) *stream = s->stream;
  return WS_OK;
}

int ws_solver_set_wait_limit(ws_solver h, int64_t clocks) {
  if (!h) return fail(WS_ERR_INVALID_ARGUMENT, "null solver");
  if (clocks < 0) return fail(WS_ERR_INVALID_ARGUMENT, "clocks must be >= 0");
  Solver* s = reinterpret_cast<Solver*>(h);
  if (s->wait_clocks != (long long)clocks) free_graph(s);  // the graph holds the kernels' arguments
  s->wait_clocks = (long long)clocks;
  return WS_OK;
}

int ws_solver_launches_per_iteration(ws_solver h) {
  if (!h) return 0;
  const Solver* s = reinterpret_cast<Solver*>(h);
  // K2, K3 + next K1 (one kernel, or the split step's three); or K1, K2, K3
  // (the stop rule is one launch per wiggle cycle), of the launched passes
  if (!s->fuses[0]) return 3;
  const Layout& L = s->lays[0];
  if (!L.mode3d) return 2;
  return L.xp || L.uni_in ? 4 : 2;
}

int ws_solver_loop_in_one_launch(ws_solver h) {
  if (!h) return 0;
  const Solver* s = reinterpret_cast<Solver*>(h);
  return loop_fits(s, 1) && s->fuses[1] ? 1 : 0;
}

int ws_solver_fused(ws_solver h) {
  if (!h) return 0;
  return reinterpret_cast<Solver*>(h)->fuses[0] ? 1 : 0;
}

int ws_solver_time_fused(ws_solver h, int n_iterations, float* ms_out, double* bytes_out) {
  if (!h || !ms_out || n_iterations < 1) return fail(WS_ERR_INVALID_ARGUMENT, "bad argument");
  Solver* s = reinterpret_cast<Solver*>(h);
  WS_CUDA(cudaSetDevice(s->device));
  WS_CUDA(use_layout(s, 0));  // the launched passes
  if (!s->fuse) return fail(WS_ERR_UNSUPPORTED, "this solver's loop does not fuse K3 with K1");
  const long long cap = n_iterations + 1;
  if (s->hist_cap < cap) {
    const int rc = ensure_hist(s, cap);
    if (rc) return rc;
  }
  StopRule rule{s->nw, 1, 0, 1, (long long)1 << 62, -1.0};
  Hist hh{s->d_hist, s->d_hist + s->hist_cap, 0, 0};  // cap 0: history untouched
  s->nrhs = 1;
  k_resume_state<<<1, 32, 0, s->stream>>>(s->d_state);
  WS_CUDA(launch_k1(s, 0, false));
  float acc = 0.f;
  for (int i = 0; i < n_iterations; ++i) {
    const int w = i % s->nw;
    WS_CUDA(launch_k2(s, w));
    WS_CUDA(cudaEventRecord(s->ev[0], s->stream));
    WS_CUDA(launch_step(s, w, (i + 1) % s->nw, false));
    WS_CUDA(cudaEventRecord(s->ev[1], s->stream));
    WS_CUDA(launch_finish(s, rule, hh, w, 1));
    WS_CUDA(cudaEventSynchronize(s->ev[1]));
    float t;
    WS_CUDA(cudaEventElapsedTime(&t, s->ev[0], s->ev[1]));
    acc += t;
  }
  *ms_out = acc / n_iterations;
  if (bytes_out) {
    const double n = (double)s->g.npts * s->g.nc;
    // K3's bytes (as ws_solver_time_kernels) plus the write of T for the next
    // iteration; the split step also reads and writes T in each x pass
    *bytes_out = (s->nw % 2 == 0 ? 40.0 : 48.0) * n + 8.0 * (double)s->g.npts + (s->lay.mode3d && (s->lay.xp || s->lay.uni_in) ? 32.0 * n : 0.0);
  }
  return WS_OK;
}

int ws_solver_time_split(ws_solver h, int n_iterations, float ms_out[3], double bytes_out[3]) {
  if (!h || !ms_out || n_iterations < 1) return fail(WS_ERR_INVALID_ARGUMENT, "bad argument");
  Solver* s = reinterpret_cast<Solver*>(h);
  WS_CUDA(cudaSetDevice(s->device));
  WS_CUDA(use_layout(s, 0));
  if (!s->fuse || !s->lay.mode3d || !(s->lay.xp || s->lay.uni_in)) return fail(WS_ERR_UNSUPPORTED, "this solver's loop does not run the split step");
  const long long cap = n_iterations + 1;
  if (s->hist_cap < cap) {
    const int rc = ensure_hist(s, cap);
    if (rc) return rc;
  }
  StopRule rule{s->nw, 1, 0, 1, (long long)1 << 62, -1.0};
  Hist hh{s->d_hist, s->d_hist + s->hist_cap, 0, 0};  // cap 0: history untouched
  s->nrhs = 1;
  k_resume_state<<<1, 32, 0, s->stream>>>(s->d_state);
  WS_CUDA(launch_k1(s, 0, false));
  float acc[3] = {0, 0, 0};
  for (int i = 0; i < n_iterations; ++i) {
    const int w = i % s->nw;
    WS_CUDA(launch_k2(s, w));
    WS_CUDA(cudaEventRecord(s->ev[0], s->stream));
    WS_CUDA(s->lay.uni_in ? launch_uni_x(s, true, s->d_T) : launch_xpencil(s, true));
    WS_CUDA(cudaEventRecord(s->ev[1], s->stream));
    WS_CUDA(s->lay.uni_in ? launch_uni_col(s, uni::kStep, w, (i + 1) % s->nw, nullptr, nullptr, s->d_T, 1.f)
                          : launch_colstep(s, w, (i + 1) % s->nw, false));
    WS_CUDA(cudaEventRecord(s->ev[2], s->stream));
    WS_CUDA(s->lay.uni_in ? launch_uni_x(s, false, s->d_T) : launch_xpencil(s, false));
    WS_CUDA(cudaEventRecord(s->ev[3], s->stream));
    WS_CUDA(launch_finish(s, rule, hh, w, 1));
    WS_CUDA(cudaEventSynchronize(s->ev[3]));
    float t;
    for (int k = 0; k < 3; ++k) {
      WS_CUDA(cudaEventElapsedTime(&t, s->ev[k], s->ev[k + 1]));
      acc[k] += t;
    }
  }
  for (int k = 0; k < 3; ++k) ms_out[k] = acc[k] / n_iterations;
  if (bytes_out) {
    const double n = (double)s->g.npts * s->g.nc;
    bytes_out[0] = 16.0 * n;  // read T, write T
    // read T, dE, gamma, write dE, T; E' read and written after even iterations only (the mean)
    bytes_out[1] = (s->nw % 2 == 0 ? 40.0 : 48.0) * n + 8.0 * (double)s->g.npts;
    bytes_out[2] = 16.0 * n;
  }
  return WS_OK;
}

int ws_solver_time_kernels(ws_solver h, int n_iterations, float ms_out[3], double bytes_out[3]) {
  if (!h || !ms_out || n_iterations < 1) return fail(WS_ERR_INVALID_ARGUMENT, "bad argument");
  Solver* s = reinterpret_cast<Solver*>(h);
  WS_CUDA(cudaSetDevice(s->device));
  WS_CUDA(use_layout(s, 0));
  const long long cap = n_iterations + 1;
  if (s->hist_cap < cap) {
    const int rc = ensure_hist(s, cap);
    if (rc) return rc;
  }
  StopRule rule{s->nw, 1, 0, 1, (long long)1 << 62, -1.0};
  Hist hh{s->d_hist, s->d_hist + s->hist_cap, 0, 0};  // cap 0: history untouched
  s->nrhs = 1;  // time the first right-hand side alone
  k_resume_state<<<1, 32, 0, s->stream>>>(s->d_state);
  float acc[3] = {0, 0, 0};
  for (int i = 0; i < n_iterations; ++i) {
    const int w = i % s->nw;
    WS_CUDA(cudaEventRecord(s->ev[0], s->stream));
    WS_CUDA(launch_k1(s, w, false));
    WS_CUDA(cudaEventRecord(s->ev[1], s->stream));
    WS_CUDA(launch_k2(s, w));
    WS_CUDA(cudaEventRecord(s->ev[2], s->stream));
    WS_CUDA(launch_k3_only(s, w));
    WS_CUDA(cudaEventRecord(s->ev[3], s->stream));
    WS_CUDA(launch_finish(s, rule, hh, w, 1));
    WS_CUDA(cudaEventSynchronize(s->ev[3]));
    float t;
    for (int k = 0; k < 3; ++k) {
      WS_CUDA(cudaEventElapsedTime(&t, s->ev[k], s->ev[k + 1]));
      acc[k] += t;
    }
  }
  for (int k = 0; k < 3; ++k) ms_out[k] = acc[k] / n_iterations;
  if (bytes_out) {
    const double n = (double)s->g.npts * s->g.nc;
    bytes_out[0] = 16.0 * n;                                // read dE, write T
    bytes_out[1] = 16.0 * n;                                // read T, write T
    // read T, dE, gamma, write dE; E read and written every iteration, or
    // every second one when E' takes the increments in pairs (the mean)
    bytes_out[2] = (s->nw % 2 == 0 ? 32.0 : 40.0) * n + 8.0 * (double)s->g.npts;
  }
  return WS_OK;
}

int ws_solver_warm_report(ws_solver h, int64_t rhs, double* cold_first_energy, double* warm_cycle_energy,
                          int* discarded) {
  if (!h) return fail(WS_ERR_INVALID_ARGUMENT, "null solver");
  Solver* s = reinterpret_cast<Solver*>(h);
  if (rhs < 0 || rhs >= s->nrhs) return fail(WS_ERR_INVALID_ARGUMENT, "right-hand side out of range");
  WS_CUDA(cudaSetDevice(s->device));
  DevState st{};
  WS_CUDA(cudaMemcpy(&st, s->d_state + rhs, sizeof(DevState), cudaMemcpyDeviceToHost));
  if (cold_first_energy) *cold_first_energy = st.diff1;
  if (warm_cycle_energy) *warm_cycle_energy = s->warm ? st.warm_e : -1.0;
  if (discarded) *discarded = s->warm ? st.discarded : 0;
  return WS_OK;
}

int ws_solver_warm_residual(ws_solver h, int64_t rhs, double* cold_residual_energy, double* warm_residual_energy) {
  if (!h) return fail(WS_ERR_INVALID_ARGUMENT, "null solver");
  Solver* s = reinterpret_cast<Solver*>(h);
  if (rhs < 0 || rhs >= s->nrhs) return fail(WS_ERR_INVALID_ARGUMENT, "right-hand side out of range");
  WS_CUDA(cudaSetDevice(s->device));
  DevState st{};
  WS_CUDA(cudaMemcpy(&st, s->d_state + rhs, sizeof(DevState), cudaMemcpyDeviceToHost));
  const bool have = s->warm && s->warm_ratio > 0.0;
  if (cold_residual_energy) *cold_residual_energy = have ? (double)s->nw * s->nw * st.diff1 : -1.0;
  if (warm_residual_energy) *warm_residual_energy = have ? st.warm_r : -1.0;
  return WS_OK;
}

// ---------------------------------------------------------------------------
// Autotuner: among the kernel layouts this grid supports (fast power-of-two
// kernels or the generic mixed-radix ones for the inner and the outer pass,
// the generic outer pass's y tile, the 2-D columns per block), keep the
// fastest inner and the fastest outer pass.  Each candidate first runs one
// iteration from a fixed field and must reproduce the current layout's
// increment to 1e-4; only then is it timed.
// ---------------------------------------------------------------------------
}  // extern "C"

namespace ws {
static __global__ void k_fill_pattern(float2* __restrict__ a, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    unsigned h = (unsigned)(i * 2654435761u) ^ (unsigned)(i >> 32) * 2246822519u;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    a[i] = make_float2((float)(h & 0xffff) / 65536.f - 0.5f, (float)(h >> 16) / 65536.f - 0.5f);
  }
}
// out[0] = max |a - b|, out[1] = max |b| (float bits of non-negative values compare as unsigned)
static __global__ void k_max_diff(const float2* __restrict__ a, const float2* __restrict__ b, long long n,
                                  unsigned* __restrict__ out) {
  float d = 0.f, m = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float2 u = a[i], v = b[i];
    d = fmaxf(d, fmaxf(fabsf(u.x - v.x), fabsf(u.y - v.y)));
    m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
  }
  if (!(d == d)) d = __int_as_float(0x7f800000);  // NaN counts as a mismatch
  atomicMax(out, __float_as_uint(d));
  atomicMax(out + 1, __float_as_uint(m));
}

// One iteration (wiggle 0, no source) from the fixed pattern; dE' -> out.
// One iteration of the loop as it runs with the solver's current layout
// (the fused step where there is one), from a fixed pattern; the new
// increment dE' into `out`.
static int tune_probe(Solver* s, const StopRule& rule, const Hist& hh, float2* out) {
  const long long n = (long long)field_elems(s);
  const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 8 * kNumSms);
  k_fill_pattern<<<blocks, 256, 0, s->stream>>>(s->d_dE, n);
  k_resume_state<<<1, 32, 0, s->stream>>>(s->d_state);
  WS_CUDA(cudaGetLastError());
  WS_CUDA(launch_k1(s, 0, false));
  WS_CUDA(launch_k2(s, 0));
  if (s->fuse) {
    WS_CUDA(launch_step(s, 0, 1 % s->nw, false));
  } else {
    WS_CUDA(launch_k3_only(s, 0));
  }
  WS_CUDA(launch_finish(s, rule, hh, 0, 1));
  WS_CUDA(cudaMemcpyAsync(out, s->d_dE, n * sizeof(float2), cudaMemcpyDeviceToDevice, s->stream));
  WS_CUDA(cudaStreamSynchronize(s->stream));
  return WS_OK;
}

// Mean device time of the loop's kernels: K1, K2, K3, or (fused) 0, K2 and
// the step.
static int tune_time(Solver* s, const StopRule& rule, const Hist& hh, int iters, float ms[3]) {
  k_resume_state<<<1, 32, 0, s->stream>>>(s->d_state);
  float acc[3] = {0, 0, 0};
  if (s->fuse) {
    WS_CUDA(launch_k1(s, 0, false));
    for (int i = 0; i < iters; ++i) {
      const int w = i % s->nw;
      WS_CUDA(cudaEventRecord(s->ev[0], s->stream));
      WS_CUDA(launch_k2(s, w));
      WS_CUDA(cudaEventRecord(s->ev[1], s->stream));
      WS_CUDA(launch_step(s, w, (i + 1) % s->nw, false));
      WS_CUDA(cudaEventRecord(s->ev[2], s->stream));
      WS_CUDA(launch_finish(s, rule, hh, w, 1));
      WS_CUDA(cudaEventSynchronize(s->ev[2]));
      float t;
      WS_CUDA(cudaEventElapsedTime(&t, s->ev[0], s->ev[1]));
      acc[1] += t;
      WS_CUDA(cudaEventElapsedTime(&t, s->ev[1], s->ev[2]));
      acc[2] += t;
    }
    for (int k = 0; k < 3; ++k) ms[k] = acc[k] / iters;
    return WS_OK;
  }
  for (int i = 0; i < iters; ++i) {
    const int w = i % s->nw;
    WS_CUDA(cudaEventRecord(s->ev[0], s->stream));
    WS_CUDA(launch_k1(s, w, false));
    WS_CUDA(cudaEventRecord(s->ev[1], s->stream));
    WS_CUDA(launch_k2(s, w));
    WS_CUDA(cudaEventRecord(s->ev[2], s->stream));
    WS_CUDA(launch_k3_only(s, w));
    WS_CUDA(cudaEventRecord(s->ev[3], s->stream));
    WS_CUDA(launch_finish(s, rule, hh, w, 1));
    WS_CUDA(cudaEventSynchronize(s->ev[3]));
    float t;
    for (int k = 0; k < 3; ++k) {
      WS_CUDA(cudaEventElapsedTime(&t, s->ev[k], s->ev[k + 1]));
      acc[k] += t;
    }
  }
  for (int k = 0; k < 3; ++k) ms[k] = acc[k] / iters;
  return WS_OK;
}
// The generic kernels' plans with radix schedule `sched` (same lengths and
// twiddle tables).
static void apply_sched(Solver* s, int sched) {
  std::vector<float2> none;
  FftPlan* plans[3] = {&s->py, &s->pxl, &s->po};
  for (FftPlan* p : plans) {
    const float2* tw = p->tw;
    if (p->n >= 1) build_plan(p->n, none, *p, sched);
    p->tw = tw;
  }
}

// Makes `c` the solver's layout (kernels, plans, fused loop); false if the
// grid does not allow it.
static bool apply_choice(Solver* s, const LayoutChoice& c) {
  Layout L;
  std::string why;
  if (make_layout(s->g, L, why, c, s->pstd != 0) != WS_OK) return false;
  // the generic 3-D kernels transform x-local lines of Nx / csize points with
  // the plan and twiddles made for the solver's first layout: a layout with
  // another cluster size would run them on lines of another length
  if (L.mode3d && !L.fi && !L.uni_in && s->g.nx / L.csize != s->pxl.n) return false;
  if (ensure_partials(s, L.grid_inner * std::max(1, s->batch_cap) * s->nw) != WS_OK) return false;
  s->lays[0] = L;
  if (set_layouts(s) != cudaSuccess || use_layout(s, 0) != cudaSuccess) return false;
  apply_sched(s, c.sched);
  free_graph(s);
  return true;
}
}  // namespace ws

extern "C" {

int ws_solver_autotune(ws_solver h, int n_iterations, int* n_tried, float* ms_before, float* ms_after) {
  if (!h || n_iterations < 1) return fail(WS_ERR_INVALID_ARGUMENT, "bad argument");
  Solver* s = reinterpret_cast<Solver*>(h);
  WS_CUDA(cudaSetDevice(s->device));
  WS_CUDA(use_layout(s, 0));
  if (s->hist_cap < 2) {
    const int rc = ensure_hist(s, 2);
    if (rc) return rc;
  }
  StopRule rule{s->nw, 1, 0, 1, (long long)1 << 62, -1.0};
  Hist hh{s->d_hist, s->d_hist + s->hist_cap, 0, 0};  // cap 0: history untouched
  s->nrhs = 1;
  free_graph(s);
  const long long n = (long long)field_elems(s);
  float2* ref = nullptr;
  float2* got = nullptr;
  unsigned* dmax = nullptr;
  auto cleanup = [&]() {
    if (ref) cudaFree(ref);
    if (got) cudaFree(got);
    if (dmax) cudaFree(dmax);
  };
  if (cudaMalloc(&ref, n * sizeof(float2)) != cudaSuccess || cudaMalloc(&got, n * sizeof(float2)) != cudaSuccess ||
      cudaMalloc(&dmax, 2 * sizeof(unsigned)) != cudaSuccess) {
    cleanup();
    return fail(WS_ERR_OUT_OF_MEMORY, "autotune: no memory for the probe fields");
  }
  const Layout base = s->lay;
  int rc = tune_probe(s, rule, hh, ref);
  float base_ms[3];
  if (!rc) rc = tune_time(s, rule, hh, n_iterations, base_ms);
  if (rc) {
    cleanup();
    return rc;
  }
  // candidates
  std::vector<LayoutChoice> inner_c, outer_c;
  inner_c.push_back(LayoutChoice{1, 0, 0, 0, 0});
  inner_c.push_back(LayoutChoice{2, 0, 0, 0, 0});
  if (base.mode3d)
    for (int c : {8, 16}) inner_c.push_back(LayoutChoice{1, 0, c, 0, 0});  // fast planes on other cluster sizes
  if (!base.mode3d)
    for (int f : {4, 2, -2})
      inner_c.push_back(LayoutChoice{2, 0, 0, f > 0 ? std::max(1, base.ncols / f) : base.ncols * 2, 0});
  for (int k = 1; k < kNumSchedules; ++k) {  // the generic kernels' radix schedules
    LayoutChoice c{2, 0, 0, 0, 0};
    c.sched = k;
    inner_c.push_back(c);
  }
  if (base.mode3d) {  // the split step's x pencils
    const auto& xt = x_pencil_table();
    for (int i = 0; i < (int)xt.size(); ++i)
      if (xt[i].no == s->g.nx && s->g.ny % xt[i].ty == 0) {
        LayoutChoice c{1, 0, 0, 0, 0};
        c.xp = i + 1;
        inner_c.push_back(c);
      }
  }
  outer_c.push_back(LayoutChoice{0, 1, 0, 0, 0});
  outer_c.push_back(LayoutChoice{0, 1, 0, 0, 8});  // fast pencil with 8 y per block, where one exists
  for (int k : {2, 3}) outer_c.push_back(LayoutChoice{0, 3 + k, 0, 0, 0});
  for (int t : {1, 2, 4, 8, 16}) outer_c.push_back(LayoutChoice{0, 2, 0, 0, t});
  int tried = 0;
  LayoutChoice best_in{}, best_out{};
  float t_in = base_ms[0] + base_ms[2], t_out = base_ms[1];
  const LayoutChoice base_choice = s->tuned;
  auto evaluate = [&](const LayoutChoice& c, float ms[3]) -> bool {
    if (!apply_choice(s, c)) {
      apply_choice(s, base_choice);
      return false;
    }
    bool ok = tune_probe(s, rule, hh, got) == WS_OK;
    if (ok) {
      unsigned hmax[2] = {0, 0};
      cudaMemsetAsync(dmax, 0, 2 * sizeof(unsigned), s->stream);
      k_max_diff<<<(unsigned)std::min<long long>((n + 255) / 256, 8 * kNumSms), 256, 0, s->stream>>>(got, ref, n,
                                                                                                  dmax);
      ok = cudaMemcpyAsync(hmax, dmax, sizeof(hmax), cudaMemcpyDeviceToHost, s->stream) == cudaSuccess &&
           cudaStreamSynchronize(s->stream) == cudaSuccess;
      float d, m;
      std::memcpy(&d, &hmax[0], 4);
      std::memcpy(&m, &hmax[1], 4);
      ok = ok && d <= 1e-4f * m;
    }
    if (ok) ok = tune_time(s, rule, hh, n_iterations, ms) == WS_OK;
    apply_choice(s, base_choice);
    cudaGetLastError();  // a launch refused for a candidate must not leak into later calls
    ++tried;
    return ok;
  };
  for (const LayoutChoice& c : inner_c) {
    float ms[3];
    if (evaluate(c, ms) && ms[0] + ms[2] < 0.97f * t_in) {
      t_in = ms[0] + ms[2];
      best_in = c;
    }
  }
  for (const LayoutChoice& c : outer_c) {
    float ms[3];
    if (evaluate(c, ms) && ms[1] < 0.97f * t_out) {
      t_out = ms[1];
      best_out = c;
    }
  }
  LayoutChoice fin = best_in;
  fin.outer = best_out.outer;
  fin.ty = best_out.ty;
  float fin_ms[3] = {base_ms[0], base_ms[1], base_ms[2]};
  if (!(fin == base_choice)) {
    if (!evaluate(fin, fin_ms)) {
      fin = base_choice;
      std::memcpy(fin_ms, base_ms, sizeof(fin_ms));
    }
  }
  apply_choice(s, fin);
  s->tuned = fin;
  cleanup();
  if (n_tried) *n_tried = tried;
  if (ms_before) *ms_before = base_ms[0] + base_ms[1] + base_ms[2];
  if (ms_after) *ms_after = fin_ms[0] + fin_ms[1] + fin_ms[2];
  return WS_OK;
}

int ws_solver_get_layout(ws_solver h, int32_t choice[7]) {
  if (!h || !choice) return fail(WS_ERR_INVALID_ARGUMENT, "bad argument");
  const LayoutChoice& c = reinterpret_cast<Solver*>(h)->tuned;
  const int32_t v[7] = {c.inner, c.outer, c.csize, c.ncols, c.ty, c.sched, c.xp};
  std::memcpy(choice, v, sizeof(v));
  return WS_OK;
}

int ws_solver_set_layout(ws_solver h, const int32_t choice[7]) {
  if (!h || !choice) return fail(WS_ERR_INVALID_ARGUMENT, "bad argument");
  Solver* s = reinterpret_cast<Solver*>(h);
  LayoutChoice c{choice[0], choice[1], choice[2], choice[3], choice[4]};
  c.sched = choice[5];
  c.xp = choice[6];
  if (c.inner < 0 || c.inner > 2 || c.outer < 0 || c.outer > 9 || c.csize < 0 || c.csize > 16 || c.ncols < 0 ||
      c.ty < 0 || c.sched < 0 || c.sched >= kNumSchedules || c.xp < 0 || c.xp > (int)x_pencil_table().size())
    return fail(WS_ERR_INVALID_ARGUMENT, "layout choice out of range");
  WS_CUDA(cudaSetDevice(s->device));
  if (!apply_choice(s, c)) {
    apply_choice(s, s->tuned);
    return fail(WS_ERR_UNSUPPORTED, "this grid does not take that layout");
  }
  s->tuned = c;
  return WS_OK;
}

int ws_solver_destroy(ws_solver h) {
  destroy_solver(reinterpret_cast<Solver*>(h));
  return WS_OK;
}

int ws_run_algorithm(const int64_t N[4], const ws_complex* gamma, int64_t n_wiggles, const ws_wiggle* wiggles,
                     int64_t n_blocks, const ws_source_block* source, float epsilon, ws_complex k02e,
                     const int64_t roi[8], int64_t max_iterations, double energy_threshold,
                     const char* callback_string, int64_t callback_interval, ws_callback_fn callback,
                     void* user_data, int memory, ws_complex* E_out, double* diff_energy_out,
                     int64_t* n_iterations) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kRunCacheDevices) return fail(WS_ERR_INVALID_ARGUMENT, "device ordinal beyond the call cache");
  std::lock_guard<std::mutex> lock(g_run_mu);
  // the solver of the previous call on this device is reused when the grid
  // and the wiggle count match: only the medium is uploaded again
  Solver*& s = g_run_cache[dev];
  int rc = WS_ERR_INVALID_ARGUMENT;
  if (s && N && s->g.ny == N[0] && s->g.nx == N[1] && s->g.nz == N[2] && s->g.nc == N[3] && s->nw == n_wiggles)
    rc = reload_medium(s, N, gamma, n_wiggles, wiggles, epsilon, k02e, roi, memory);
  if (rc) {
    destroy_solver(s);
    s = nullptr;
    rc = create_solver(N, gamma, n_wiggles, wiggles, epsilon, k02e, roi, memory, dev, &s);
    if (rc) {
      s = nullptr;
      return rc;
    }
  }
  ws_solve_options o;
  ws_default_options(&o);
  o.max_iterations = max_iterations;
  o.energy_threshold = energy_threshold;
  o.callback_type = callback_string ? callback_string : "NoCallback";
  o.callback_interval = callback_interval > 0 ? callback_interval : 50;
  o.energy_interval = std::min<int64_t>(8, o.callback_interval);  // Simulation.m:135
  o.callback = callback;
  o.user_data = user_data;
  rc = solve(s, n_blocks, source, memory, &o, E_out, memory, diff_energy_out, n_iterations, nullptr);
  if (rc && rc != WS_ERR_DIVERGED && rc != WS_ERR_NO_SOURCE && rc != WS_ERR_INVALID_ARGUMENT) {
    destroy_solver(s);  // after a CUDA error start afresh next time
    s = nullptr;
  }
  return rc;
}

void ws_run_algorithm_release(void) {
  std::lock_guard<std::mutex> lock(g_run_mu);
  for (Solver*& s : g_run_cache) {
    destroy_solver(s);
    s = nullptr;
  }
  host_pool().trim();
}

}  // extern "C"

// ---------------------------------------------------------------------------
// PSTD (PSTD.m): the reference's pseudo-spectral time-domain comparison
// solver, on the same FFT kernels.  One step (PSTD.m:103-117):
//   Etmp   = ifftn(-(px^2 + py^2 + pz^2) .* fftn(E)) + A(it) S
//   E_next = c2 E + c1 E_prev + c3 Etmp
// runs as K1 (inner FFT of E, unit ramps) -> K2 (outer FFT, Laplacian / N,
// inverse outer FFT, conjugate) -> K1 again (inner FFT of the conjugate, so
// that conj of its output is the inverse inner FFT) -> k_pstd_update (the
// leapfrog, the source, the step energy |E_next - E e^{i(arg A - arg A_prev)}|^2
// on the ROI) -> k_pstd_finish (Simulation.next with can_terminate =
// real(A) > 0.9, energy / |A|^2).  E and E_prev swap buffers every step; the
// source amplitudes A(it) of a chunk of steps come from the host.
// ---------------------------------------------------------------------------
namespace ws {

struct PstdStep {
  Geom g;
  const float2* T2;    // inner FFT of conj(W): conj(T2) = ifftn(k fftn(E))
  const float2* E;
  const float2* Eprev;
  float2* Enext;       // the buffer of Eprev
  const float2* c12;   // (c1, c2) per point
  const float* c3;
  const float2* src;   // dense source field
  const double2* amp;  // amp[k] = A at step it0 - 1 + k
  long long it0;
};

struct PstdRule {
  double threshold;
  long long max_iter;
  int interval;
};

static __global__ void __launch_bounds__(256) k_pstd_update(PstdStep a, const DevState* __restrict__ st,
                                                            double* __restrict__ partials) {
  if (load_done(st)) return;
  const long long k = (long long)__ldcg(&st->it) - a.it0 + 1;
  const double2 A = a.amp[k], Ap = a.amp[k - 1];
  const double dphi = atan2(A.y, A.x) - atan2(Ap.y, Ap.x);
  const float2 ps = make_float2((float)cos(dphi), (float)sin(dphi));
  const float2 Af = make_float2((float)A.x, (float)A.y);
  const Geom& g = a.g;
  float esum = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < g.npts;
       i += (long long)gridDim.x * blockDim.x) {
    float2 t = a.T2[i];
    t.y = -t.y;
    t = cadd(t, cmul(Af, a.src[i]));  // Source.add_to (Source.m:167-169)
    const float2 c12 = a.c12[i];
    const float c3 = a.c3[i];
    const float2 e = a.E[i], ep = a.Eprev[i];
    const float2 en = make_float2(c12.y * e.x + c12.x * ep.x + c3 * t.x, c12.y * e.y + c12.x * ep.y + c3 * t.y);
    a.Enext[i] = en;
    const int y = (int)(i % g.ny);
    const long long r = i / g.ny;
    const int x = (int)(r % g.nx), z = (int)(r / g.nx);
    if (y >= g.r0[0] && y < g.r1[0] && x >= g.r0[1] && x < g.r1[1] && z >= g.r0[2] && z < g.r1[2]) {
      const float2 d = make_float2(en.x - (e.x * ps.x - e.y * ps.y), en.y - (e.x * ps.y + e.y * ps.x));
      esum = fmaf(d.x, d.x, fmaf(d.y, d.y, esum));
    }
  }
  __shared__ float red[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) esum += __shfl_xor_sync(0xffffffffu, esum, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = esum;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < blockDim.x / 32 ? red[threadIdx.x] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) partials[blockIdx.x] = (double)v;
  }
}

// Simulation.next (Simulation.m:193-217) for PSTD.run_algorithm (PSTD.m:108-124)
static __global__ void k_pstd_finish(DevState* st, const double* __restrict__ partials, int nparts,
                                     const double2* __restrict__ amp, long long it0, PstdRule rule,
                                     double* __restrict__ hist, long long hist_cap) {
  __shared__ double red[32];
  if (load_done(st)) return;
  double e = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) e += partials[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x != 0) return;
  e = 0.0;
  for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) e += red[w];
  const int it = st->it;
  const double2 A = amp[it - it0 + 1];
  if (st->calc_energy) st->last_step_energy = e / (A.x * A.x + A.y * A.y);
  const double d = st->last_step_energy;
  if (it - 1 < hist_cap) hist[it - 1] = d;
  if (it == 1) st->diff1 = d;
  const bool can_terminate = A.x > 0.9;  // MATLAB's A > 0.9 compares the real part
  if (can_terminate && d / st->diff1 < rule.threshold) {
    st->done = 1;
    st->converged = 1;
  } else if (can_terminate && it >= rule.max_iter) {
    st->done = 1;
    st->converged = 0;
  }
  st->calc_energy = ((it - 1) % rule.interval) == 0;
  st->it = it + 1;
}

// ROI crop times a phase factor (PSTD.m:126)
static __global__ void k_pstd_output(const float2* __restrict__ E, Geom g, float2 phase, float2* __restrict__ out) {
  const int ry = g.r1[0] - g.r0[0], rx = g.r1[1] - g.r0[1], rz = g.r1[2] - g.r0[2];
  const long long n = (long long)ry * rx * rz;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    long long r = i;
    const int y = (int)(r % ry) + g.r0[0];
    r /= ry;
    const int x = (int)(r % rx) + g.r0[1];
    const int z = (int)(r / rx) + g.r0[2];
    out[i] = cmul(E[y + (long long)g.ny * (x + (long long)g.nx * z)], phase);
  }
}

struct Pstd {
  Solver* s = nullptr;       // layout, twiddles, T, source, state, stream (K2 in Laplacian mode)
  float2* d_Ebuf = nullptr;  // two fields: step it reads E from (it - 1) % 2, writes E_next to it % 2
  float2* d_T2 = nullptr;
  float* d_c3 = nullptr;
  double2* d_amp = nullptr;
  double* d_hist = nullptr;
  long long hist_cap = 0;
  double* d_part = nullptr;
  int nparts = 0;
};

static void pstd_free(Pstd* p) {
  if (!p) return;
  if (p->s) {
    cudaSetDevice(p->s->device);
    void* ptrs[] = {p->d_Ebuf, p->d_T2, p->d_c3, p->d_amp, p->d_hist, p->d_part};
    for (void* q : ptrs)
      if (q) cudaFree(q);
    destroy_solver(p->s);
  }
  delete p;
}

static void pstd_default_amplitude(double ncycle, double* re, double* im, void*) {
  // PSTD.m:130-137
  const double env = 0.5 - 0.5 * std::cos(M_PI * std::min(ncycle / 100.0, 1.0));
  *re = std::cos(-2.0 * M_PI * ncycle) * env;
  *im = std::sin(-2.0 * M_PI * ncycle) * env;
}

constexpr int kPstdChunk = 256;  // steps launched between host checks of the stop flag

}  // namespace ws

extern "C" {

int ws_pstd_create(const int64_t N[3], const float* c1, const float* c2, const float* c3, const float* px,
                   const float* py, const float* pz, const int64_t roi[8], int device, ws_pstd* out) {
  if (!N || !c1 || !c2 || !c3 || !px || !py || !pz || !roi || !out)
    return fail(WS_ERR_INVALID_ARGUMENT, "null argument");
  *out = nullptr;
  const int64_t N4[4] = {N[0], N[1], N[2], 1};
  for (int d = 0; d < 3; ++d)
    if (N[d] < 1) return fail(WS_ERR_INVALID_ARGUMENT, "N must be positive");
  const size_t npts = (size_t)N[0] * N[1] * N[2];
  // the solver's gamma buffer holds (c1, c2); one wiggle with unit ramps and the plain Fourier ranges
  std::vector<float2> c12(npts);
  for (size_t i = 0; i < npts; ++i) c12[i] = make_float2(c1[i], c2[i]);
  std::vector<float2> one((size_t)std::max(N[0], std::max(N[1], N[2])), make_float2(1.f, 0.f));
  ws_wiggle w{px, py, pz, (const ws_complex*)one.data(), (const ws_complex*)one.data(),
              (const ws_complex*)one.data()};
  Pstd* p = new Pstd();
  int rc = create_solver(N4, (const ws_complex*)c12.data(), 1, &w, 1.0f, ws_complex{0.f, 0.f}, roi, WS_HOST, device,
                         &p->s, true);
  if (rc) {
    delete p;
    return rc;
  }
  Solver* s = p->s;
  p->nparts = (int)std::min<long long>(((long long)npts + 255) / 256, 8LL * kNumSms);
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = cudaMalloc(&p->d_Ebuf, 2 * npts * sizeof(float2));
  if (e == cudaSuccess) e = cudaMalloc(&p->d_T2, npts * sizeof(float2));
  if (e == cudaSuccess) e = cudaMalloc(&p->d_c3, npts * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&p->d_amp, (kPstdChunk + 1) * std::max(sizeof(double2), sizeof(uni::PstdStepAmp)));
  if (e == cudaSuccess) e = cudaMalloc(&p->d_part, p->nparts * sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(p->d_c3, c3, npts * sizeof(float), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    pstd_free(p);
    return fail(e == cudaErrorMemoryAllocation ? WS_ERR_OUT_OF_MEMORY : WS_ERR_CUDA, cudaGetErrorString(e));
  }
  *out = reinterpret_cast<ws_pstd>(p);
  return WS_OK;
}

void ws_pstd_default_options(ws_pstd_options* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->max_iterations = 100000;
  o->energy_threshold = 1e-2;
  o->energy_interval = 8;
  o->iterations_per_cycle = 1.0;
}

int ws_pstd_run(ws_pstd h, int64_t n_blocks, const ws_source_block* source, int source_memory,
                const ws_pstd_options* opts, ws_complex* E_out, double* diff_energy_out, int64_t diff_capacity,
                int64_t* n_iterations, int* converged) {
  if (!h || !opts || !E_out) return fail(WS_ERR_INVALID_ARGUMENT, "null argument");
  if (opts->max_iterations < 1 || opts->energy_interval < 1 || !(opts->iterations_per_cycle > 0))
    return fail(WS_ERR_INVALID_ARGUMENT, "bad options");
  Pstd* p = reinterpret_cast<Pstd*>(h);
  Solver* s = p->s;
  WS_CUDA(cudaSetDevice(s->device));
  const Geom& g = s->g;
  if (n_blocks < 1 || !source) return fail(WS_ERR_NO_SOURCE, "There is no source inside the grid boundaries");
  std::vector<double> energy;
  int rc = upload_sources(s, 1, &n_blocks, source, source_memory, energy);
  if (rc) return rc;
  if (!(energy[0] > 0)) return fail(WS_ERR_NO_SOURCE, "There is no source inside the grid boundaries");
  const long long cap = std::max<long long>(0, diff_capacity);
  if (cap > p->hist_cap) {
    if (p->d_hist) cudaFree(p->d_hist);
    p->d_hist = nullptr;
    p->hist_cap = 0;
    WS_CUDA(cudaMalloc(&p->d_hist, cap * sizeof(double)));
    p->hist_cap = cap;
  }
  const size_t npts = (size_t)g.npts;
  WS_CUDA(cudaMemsetAsync(p->d_Ebuf, 0, 2 * npts * sizeof(float2), s->stream));
  DevState st0{};
  st0.it = 1;
  st0.calc_energy = 1;
  st0.last_step_energy = INFINITY;
  WS_CUDA(cudaMemcpyAsync(s->d_state, &st0, sizeof(st0), cudaMemcpyHostToDevice, s->stream));
  ws_amplitude_fn amp = opts->amplitude ? opts->amplitude : pstd_default_amplitude;
  const PstdRule rule{opts->energy_threshold, (long long)opts->max_iterations, (int)opts->energy_interval};
  std::vector<double2> hamp(kPstdChunk + 1);
  double2 a_last = make_double2(1.0, 0.0);  // PSTD.m:83: A = 1 before the first step
  long long it0 = 1;
  DevState hst{};
  const unsigned ublocks = (unsigned)p->nparts;
  // Simulation.next stops at max_iterations only on a step that may terminate
  // (real(A) > 0.9), as the reference does; past max_iterations plus a margin
  // of max(1000, 2 iterations_per_cycle) steps the run ends unconverged.
  const long long hard_stop =
      opts->max_iterations + std::max<long long>(1000, (long long)std::ceil(2 * opts->iterations_per_cycle));
  const bool in_one = s->has_loop;
  std::vector<uni::PstdStepAmp> steps(in_one ? kPstdChunk : 0);
  if (in_one) {
    WS_CUDA(use_layout(s, 1));
    rc = ensure_partials(s, s->lay.grid_inner);
    if (rc) return rc;
    WS_CUDA(cudaMemsetAsync(s->d_T, 0, t_stride(s) * sizeof(float2), s->stream));  // the transform of E = 0
  }
  while (true) {
    const long long K = kPstdChunk;
    hamp[0] = a_last;
    for (long long k = 1; k <= K; ++k)
      amp((double)(it0 - 1 + k) / opts->iterations_per_cycle, &hamp[k].x, &hamp[k].y, opts->user_data);
    if (in_one) {
      for (long long k = 0; k < K; ++k) {
        const double2 A = hamp[k + 1], B = hamp[k];
        const double dphi = std::atan2(A.y, A.x) - std::atan2(B.y, B.x);
        steps[k] = uni::PstdStepAmp{make_float2((float)A.x, (float)A.y),
                                    make_float2((float)std::cos(dphi), (float)std::sin(dphi)), A.x * A.x + A.y * A.y,
                                    A.x > 0.9};  // MATLAB's A > 0.9 compares the real part
      }
      WS_CUDA(cudaMemcpyAsync(p->d_amp, steps.data(), K * sizeof(uni::PstdStepAmp), cudaMemcpyHostToDevice, s->stream));
      uni::PstdLoopArgs a{};
      a.col = uni_col_args(s, 0, 0, nullptr, nullptr, s->d_T, 1.f);
      a.pen = uni_pencil_args(s, 0);
      a.pen.pstd = 2;
      a.c3 = p->d_c3;
      a.src = s->d_src;
      a.fields = p->d_Ebuf;
      a.amp = (const uni::PstdStepAmp*)p->d_amp;
      a.partials = s->d_partials;
      a.st = s->d_state;
      a.hist = p->d_hist;
      a.hist_cap = std::min(p->hist_cap, cap);
      a.max_iter = rule.max_iter;
      a.threshold = rule.threshold;
      a.err = s->d_err;
      a.limit = barrier_limit(s);
      a.steps = (int)K;
      a.interval = rule.interval;
      a.groups = uni_groups(s->lay.ucol);
      const size_t smem = pstd_loop_smem(s->lay, g, &a.tile_elems);
      WS_CUDA(launch_coop(s, uni_kernels(std::max(s->lay.ucol.plan.cls, s->lay.uout.plan.cls)).pstd_loop, smem, 1, &a,
                          &a.arrived));
    } else {
      WS_CUDA(cudaMemcpyAsync(p->d_amp, hamp.data(), (K + 1) * sizeof(double2), cudaMemcpyHostToDevice, s->stream));
    }
    for (long long k = 0; k < K && !in_one; ++k) {
      const long long it = it0 + k;
      float2* E = p->d_Ebuf + (size_t)((it - 1) & 1) * npts;
      float2* Ep = p->d_Ebuf + (size_t)(it & 1) * npts;
      WS_CUDA(launch_k1_io(s, 0, E, nullptr, s->d_T));
      WS_CUDA(launch_k2(s, 0));
      WS_CUDA(launch_k1_io(s, 0, s->d_T, nullptr, p->d_T2));
      PstdStep a{g, p->d_T2, E, Ep, Ep, (const float2*)s->d_gamma, p->d_c3, s->d_src, p->d_amp, it0};
      k_pstd_update<<<ublocks, 256, 0, s->stream>>>(a, s->d_state, p->d_part);
      WS_CUDA(cudaGetLastError());
      k_pstd_finish<<<1, 256, 0, s->stream>>>(s->d_state, p->d_part, p->nparts, p->d_amp, it0, rule, p->d_hist,
                                              p->hist_cap < cap ? p->hist_cap : cap);
      WS_CUDA(cudaGetLastError());
    }
    WS_CUDA(cudaMemcpyAsync(&hst, s->d_state, sizeof(hst), cudaMemcpyDeviceToHost, s->stream));
    int failed = 0;  // a barrier of the loop kernel that gave up
    if (in_one) WS_CUDA(cudaMemcpyAsync(&failed, s->d_err, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    WS_CUDA(cudaStreamSynchronize(s->stream));
    if (hst.done || failed || it0 + K > hard_stop) break;
    a_last = hamp[K];
    it0 += K;
  }
  int kerr = 0;
  WS_CUDA(cudaMemcpy(&kerr, s->d_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (kerr) {
    cudaMemset(s->d_err, 0, sizeof(int));
    return fail(WS_ERR_CUDA, "a bounded wait of the kernels (cluster exchange, TMA tile load or the loop's barrier) timed out");
  }
  const long long last = hst.it - 1;  // the last step run
  double are = 1.0, aim = 0.0;
  amp((double)hst.it / opts->iterations_per_cycle, &are, &aim, opts->user_data);  // PSTD.m:125
  const double ph = -std::atan2(aim, are);
  const float2 phase = make_float2((float)std::cos(ph), (float)std::sin(ph));
  const long long nroi = (long long)(g.r1[0] - g.r0[0]) * (g.r1[1] - g.r0[1]) * (g.r1[2] - g.r0[2]);
  if (s->out_cap < (size_t)nroi) {
    if (s->d_out) cudaFree(s->d_out);
    s->d_out = nullptr;
    s->out_cap = 0;
    WS_CUDA(cudaMalloc(&s->d_out, nroi * sizeof(float2)));
    s->out_cap = nroi;
  }
  k_pstd_output<<<(unsigned)std::min<long long>((nroi + 255) / 256, 8LL * kNumSms), 256, 0, s->stream>>>(
      p->d_Ebuf + (size_t)(last & 1) * npts, g, phase, s->d_out);
  WS_CUDA(cudaGetLastError());
  WS_CUDA(cudaMemcpyAsync(E_out, s->d_out, nroi * sizeof(float2), cudaMemcpyDeviceToHost, s->stream));
  const long long nh = std::min<long long>(last, cap);
  if (diff_energy_out && nh > 0)
    WS_CUDA(cudaMemcpyAsync(diff_energy_out, p->d_hist, nh * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
  WS_CUDA(cudaStreamSynchronize(s->stream));
  if (n_iterations) *n_iterations = last;
  if (converged) *converged = hst.converged;
  return WS_OK;
}

int ws_pstd_set_wait_limit(ws_pstd h, int64_t clocks) {
  if (!h) return fail(WS_ERR_INVALID_ARGUMENT, "null solver");
  return ws_solver_set_wait_limit(reinterpret_cast<ws_solver>(reinterpret_cast<Pstd*>(h)->s), clocks);
}

int ws_pstd_destroy(ws_pstd h) {
  pstd_free(reinterpret_cast<Pstd*>(h));
  return WS_OK;
}

}  // extern "C"
