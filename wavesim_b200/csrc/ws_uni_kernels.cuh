// The kernels of ws_uni.cuh, for radices up to RM (one source file per bound, so
// that they compile side by side).
#pragma once
#include "ws_uni.cuh"

namespace ws {
namespace uni {

// Every kernel is compiled for three bounds RM on its radices: the registers
// of the largest butterfly decide how many blocks an SM holds, and most
// lengths do without the largest ones.
template <int RM>
constexpr int kBlocks = RM <= 8 ? 4 : (RM <= 12 ? 3 : 2);
template <int RM>  // the passes with an epilogue or three components
constexpr int kBlocksHeavy = RM <= 8 ? 3 : 2;

// f<R>() for the radix R <= RM of a stage (uniform over the block)
template <int RM, class F>
__device__ __forceinline__ void with_radix(int R, F f) {
  switch (R) {
#define WS_R(r)                                                            \
  case r:                                                                  \
    if constexpr (r <= RM) f(std::integral_constant<int, r>{});            \
    break;
    WS_R(2) WS_R(3) WS_R(4) WS_R(5) WS_R(6) WS_R(7) WS_R(8) WS_R(9) WS_R(10) WS_R(11) WS_R(12) WS_R(13) WS_R(14)
    WS_R(15) WS_R(16)
#undef WS_R
    default:
      break;
  }
}

// one butterfly of a middle stage, in place on the tile: elements p[r step]
template <int R, bool INV>
__device__ __forceinline__ void middle(float2* p, int step, const float2* tw, int sub) {
  float2 v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = p[r * step];
  if (INV) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul_conj(v[r], tw[r * sub]);
  }
  Dft<R, INV>::run(v);
  if (!INV) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tw[r * sub]);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) p[r * step] = v[r];
}

// n elements of a table into shared memory
template <class V>
__device__ __forceinline__ void copy_table(V* dst, const V* __restrict__ src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(&src[i]);
}

// Column pass --------------------------------------------------------------
// kFwd: K1 (source, ramps, forward y); kInv: K3 (inverse y, f_mix, E' += dE',
// energy); kStep: K3 of an iteration and K1 of the next.
struct ColLine {
  long long goff;  // offset of the column's gamma
  int in;          // x, z and the component inside the roi
};
// What a block needs for its columns, in shared memory (the loads of these
// tables run together; from L2 one after the other they took a third of a
// small pass), and its fields.
struct ColMem {
  float2* tile;
  const float2* tw;          // twiddles
  const float2 *gy, *gy1;    // y ramps of this iteration and of the next
  const float2 *gxz, *gxz1;  // gx gz of each column
  const ColLine* info;
  float* red;                // the energy of each 32 butterflies
  const float2* gamma;
  float2 *dE, *E;            // of the block's first column
  // kPstd: gamma holds (c1, c2), dE the field, E the one before it (then the one after)
  const float* c3 = nullptr;
  const float2* S = nullptr;
  float2 A{}, ps{};
};

// the 16-byte blocks inside n elements from p, into L2
__device__ __forceinline__ void prefetch_columns(const float2* p, int n) {
  const uintptr_t lo = (reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15;
  const uintptr_t hi = reinterpret_cast<uintptr_t>(p + n) & ~(uintptr_t)15;
  if (hi > lo)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((unsigned)(hi - lo)) : "memory");
}

template <int RM, bool INV>
__device__ __forceinline__ void col_middles(const ColArgs& a, float2* tile, const float2* tw, int nl, int tid, int nthr) {
  for (int k = 1; k < a.py.nst - 1; ++k) {
    const Stage& S = a.py.st[INV ? a.py.nst - 1 - k : k];
    with_radix<RM>(S.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int q = tid; q < nl * S.units; q += nthr) {
        const int l = quot(q, S.munits), u = q - l * S.units;
        const int b = quot(u, S.msub), j = u - b * S.sub;
        float2* p = tile + l * a.py.np + b * S.blkp + j + (a.py.pad ? quot(j, a.py.mrl) : 0);
        middle<R, INV>(p, S.subp, tw + S.two + j, S.sub);
      }
    });
    __syncthreads();
  }
}

template <int RM, int MODE, bool D3>
__device__ __forceinline__ void col_body(const ColArgs& a, const ColIter& it, const ColMem& m, int rhs, int bid) {
  const bool acc_now = MODE != kFwd && it.acc != kAccSkip;
  const Geom& g = a.g;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int col0 = bid * a.lines;
  const int nl = min(a.lines, a.total - col0);
  float2* const tile = m.tile;
  float2* const T = a.T + rhs * a.tstride + col0 * a.pitch;
  const long long f0 = rhs * a.fstride + (long long)col0 * g.ny;  // the block's first column
  const Stage& S0 = a.py.st[0];
  const Stage& SL = a.py.st[a.py.nst - 1];
  if (MODE != kFwd) {
    with_radix<RM>(SL.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int q = tid; q < nl * SL.units; q += nthr) {
        const int l = quot(q, SL.munits), u = q - l * SL.units;
        const float2* t = T + l * a.pitch + u;
        float2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = __ldcg(&t[i * SL.units]);
        Dft<R, true>::run(v);
        float2* p = tile + l * a.py.np + u * SL.blkp;
#pragma unroll
        for (int i = 0; i < R; ++i) p[i] = v[i];
      }
    });
    __syncthreads();
    col_middles<RM, true>(a, tile, m.tw, nl, tid, nthr);
  } else {
    __syncthreads();
  }
  with_radix<RM>(S0.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int n0 = nl * S0.units;
    for (int q = tid; q - (tid & 31) < n0; q += nthr) {  // whole warps: the energies are summed across them
      float esum = 0.f;
      if (q < n0) {
        const int l = quot(q, S0.munits), j = q - l * S0.units;
        const ColLine I = m.info[l];
        float2* p = tile + l * a.py.np + j + (a.py.pad ? quot(j, a.py.mrl) : 0);
        const int at = l * g.ny + j;
        const float2* __restrict__ tw0 = m.tw + S0.two + j;
        float2 v[R];
        if (MODE != kFwd) {
          const float2 g0 = MODE == kPstd ? make_float2(1.f, 0.f) : m.gxz[l];
          const float2* __restrict__ gmc = m.gamma + I.goff + j;
          float2* __restrict__ dEc = m.dE + at;
          float2* __restrict__ Ec = m.E + at;
          // the epilogue's loads in groups of H elements, the first group's before the butterfly
          constexpr int H = R <= 5 ? R : (R <= 10 ? (R + 1) / 2 : (R + 2) / 3);
          float2 gm[H], d0[H];
          if (MODE != kPstd) {
#pragma unroll
            for (int r = 0; r < H; ++r) {
              gm[r] = gmc[r * S0.sub];
              d0[r] = dEc[r * S0.sub];
            }
          }
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = p[r * S0.subp];
#pragma unroll
          for (int r = 1; r < R; ++r) v[r] = cmul_conj(v[r], tw0[r * S0.sub]);
          Dft<R, true>::run(v);
          if constexpr (MODE == kPstd) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              // E_next = c2 E + c1 E_prev + c3 (ifftn(k fftn(E)) + A S), PSTD.m:103-107
              const int y = j + r * S0.sub;
              const float2 t = cadd(v[r], cmul(m.A, m.S[at + r * S0.sub]));
              const float2 c12 = gmc[r * S0.sub], e = dEc[r * S0.sub], ep = Ec[r * S0.sub];
              const float c3 = m.c3[at + r * S0.sub];
              const float2 en = make_float2(c12.y * e.x + c12.x * ep.x + c3 * t.x, c12.y * e.y + c12.x * ep.y + c3 * t.y);
              Ec[r * S0.sub] = en;
              if (I.in && y >= g.r0[0] && y < g.r1[0]) {
                const float2 d = make_float2(en.x - (e.x * m.ps.x - e.y * m.ps.y), en.y - (e.x * m.ps.y + e.y * m.ps.x));
                esum = fmaf(d.x, d.x, fmaf(d.y, d.y, esum));
              }
              v[r] = en;
            }
          } else {
#pragma unroll
            for (int h = 0; h < R; h += H) {
              if (h > 0) {
#pragma unroll
                for (int r = 0; r < H; ++r)
                  if (h + r < R) {
                    gm[r] = gmc[(h + r) * S0.sub];
                    d0[r] = dEc[(h + r) * S0.sub];
                  }
              }
              float2 e0[H];
#pragma unroll
              for (int r = 0; r < H; ++r)
                if (h + r < R) e0[r] = acc_now ? Ec[(h + r) * S0.sub] : make_float2(0.f, 0.f);
#pragma unroll
              for (int r = 0; r < H; ++r)
                if (h + r < R) {
                  const int k = h + r, y = j + k * S0.sub;
                  // Eprop after the conjugate ramps (WaveSim.m:55), f_mix (f_mix.m:3-4), E' += dE'
                  const float2 ep = cmul_conj(cmul_conj(v[k], g0), m.gy[y]);
                  float2 dn;
                  if (D3) {
                    // 1 - alpha gamma and gamma^2 first, as the compile-time kernels have it: of a medium of a few
                    // values (spheres) their rounding is the same everywhere, and so the same at every size
                    const float2 one_m = make_float2(1.f - kAlpha * gm[r].x, -kAlpha * gm[r].y);
                    const float2 t = cmul(cmul(gm[r], gm[r]), ep);
                    dn = cadd(cmul(one_m, d0[r]), make_float2(kAlpha * t.y, -kAlpha * t.x));
                  } else {
                    // dE - alpha gamma (dE + i gamma Eprop): nothing is rounded alike in every iteration (81 x 360,
                    // 197 iterations: field 8e-7 from that of 64 bits on the same tables, energies 1.3e-7; as above
                    // 1.5e-6 and 5e-7)
                    const float2 u = cmul(gm[r], ep);
                    const float2 t = cmul(gm[r], make_float2(d0[r].x - u.y, d0[r].y + u.x));
                    dn = make_float2(fmaf(-kAlpha, t.x, d0[r].x), fmaf(-kAlpha, t.y, d0[r].y));
                  }
                  dEc[k * S0.sub] = dn;
                  if (acc_now) Ec[k * S0.sub] = cadd(e0[r], it.acc == kAccPair ? cadd(d0[r], dn) : dn);
                  if (I.in && y >= g.r0[0] && y < g.r1[0]) esum = fmaf(dn.x, dn.x, fmaf(dn.y, dn.y, esum));
                  v[k] = dn;
                }
            }
          }
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = a.dE_in[f0 + at + r * S0.sub];
        }
        if (MODE != kInv) {
          if (MODE != kPstd) {
            const float2 g1 = m.gxz1[l];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              if (it.src) v[r] = cadd(v[r], cmul(a.A, it.src[f0 + at + r * S0.sub]));
              v[r] = cmul(cmul(v[r], g1), m.gy1[j + r * S0.sub]);
            }
          }
          Dft<R, false>::run(v);
#pragma unroll
          for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tw0[r * S0.sub]);
#pragma unroll
          for (int r = 0; r < R; ++r) p[r * S0.subp] = v[r];
        }
      }
      if (MODE != kFwd) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) esum += __shfl_xor_sync(0xffffffffu, esum, o);
        if ((tid & 31) == 0) m.red[q >> 5] = esum;
      }
    }
  });
  if (MODE != kInv) {
    __syncthreads();
    col_middles<RM, false>(a, tile, m.tw, nl, tid, nthr);
    with_radix<RM>(SL.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int q = tid; q < nl * SL.units; q += nthr) {
        const int l = quot(q, SL.munits), u = q - l * SL.units;
        const float2* p = tile + l * a.py.np + u * SL.blkp;
        float2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = p[i];
        Dft<R, false>::run(v);
        float2* t = T + l * a.pitch + u;
#pragma unroll
        for (int i = 0; i < R; ++i) t[i * SL.units] = v[i];
      }
    });
  }
  if (MODE != kFwd) {
    // in order, whatever the number of threads (the barrier above is behind every sum)
    if (MODE == kInv) __syncthreads();
    if (tid == nthr - 1) {
      float v = 0.f;
      for (int w = 0; w < (nl * S0.units + 31) / 32; ++w) v += m.red[w];
      it.partials[rhs * a.bpr + bid] = (double)v;
    }
  }
}

template <int RM, int MODE, bool D3>
__global__ void __launch_bounds__(kMaxThreads, (MODE == kFwd ? kBlocks<RM> : kBlocksHeavy<RM>)) k_col(
    const __grid_constant__ ColArgs a) {
  const int rhs = blockIdx.x / a.bpr, bid = blockIdx.x - rhs * a.bpr;
  if (load_done(a.st + rhs)) return;
  extern __shared__ float2 tile[];
  const Geom& g = a.g;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int col0 = bid * a.lines, nl = min(a.lines, a.total - col0);
  const long long f0 = rhs * a.fstride + (long long)col0 * g.ny;
  float2* const gy = tile + a.lines * a.py.np;
  float2* const gy1 = gy + a.py.n;
  float2* const gxz = gy1 + a.py.n;
  ColLine* const info = reinterpret_cast<ColLine*>(gxz + 2 * a.lines);
  float* const red = reinterpret_cast<float*>(info + a.lines);
  if (MODE != kFwd && tid == 0) {
    // the epilogue's columns are contiguous: into L2 while the transform runs
    const long long g0 = (long long)col0 * g.ny % g.npts;
    prefetch_columns(a.gamma + rhs * a.gstride + g0, (int)min((long long)nl * g.ny, g.npts - g0));
    prefetch_columns(a.dE + f0, nl * g.ny);
    if (a.it.acc != kAccSkip) prefetch_columns(a.E + f0, nl * g.ny);
  }
  if (MODE != kFwd) copy_table(gy, a.it.gy, a.py.n);
  if (MODE != kInv) copy_table(gy1, a.it.gy1, a.py.n);
  for (int l = nthr - 1 - tid; l < nl; l += nthr) {  // from the last warp on: the first ones have a butterfly
    const int col = col0 + l;
    const int zc = col / g.nx, x = col - zc * g.nx;
    const int c = zc / g.nz, z = zc - c * g.nz;
    if (MODE != kFwd) gxz[l] = cmul(a.it.gx[x], a.it.gz[z]);
    if (MODE != kInv) gxz[a.lines + l] = cmul(a.it.gx1[x], a.it.gz1[z]);
    ColLine I;
    I.goff = rhs * a.gstride + (long long)col * g.ny - c * g.npts;
    I.in = x >= g.r0[1] && x < g.r1[1] && z >= g.r0[2] && z < g.r1[2] && c >= g.r0[3] && c < g.r1[3];
    info[l] = I;
  }
  col_body<RM, MODE, D3>(a, a.it, ColMem{tile, a.py.tw, gy, gy1, gxz, gxz + a.lines, info, red, a.gamma, a.dE + f0, a.E + f0}, rhs, bid);
}

// Pencils --------------------------------------------------------------------
// A tile holds ty consecutive y of one line of N rows: element (row, yl) at
// row * ty + yl; thread (w, yl) takes the butterflies w, w + W, ...
template <int RM, bool INV>
__device__ __forceinline__ void row_middles(const Plan& P, float2* tile, const float2* tw, int ty, int yl, int w, int W) {
  for (int k = 1; k < P.nst - 1; ++k) {
    const Stage& S = P.st[INV ? P.nst - 1 - k : k];
    with_radix<RM>(S.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int u = w; u < S.units; u += W) {
        const int b = quot(u, S.msub), j = u - b * S.sub;
        middle<R, INV>(tile + (b * S.R * S.sub + j) * ty + yl, S.sub * ty, tw + S.two + j, S.sub);
      }
    });
    __syncthreads();
  }
}

// first stage of a forward transform, from global rows into the tile
template <int RM>
__device__ __forceinline__ void rows_in(const Stage& S, const float2* tw, const float2* src, long long step,
                                        float2* tile, int ty, int yl, int w, int W, bool live) {
  with_radix<RM>(S.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int j = w; j < S.units; j += W) {
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = live ? __ldcg(&src[(j + r * S.sub) * step]) : make_float2(0.f, 0.f);
      Dft<R, false>::run(v);
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tw[S.two + r * S.sub + j]);
#pragma unroll
      for (int r = 0; r < R; ++r) tile[(j + r * S.sub) * ty + yl] = v[r];
    }
  });
}

// last stage of an inverse transform, from the tile to global rows
template <int RM>
__device__ __forceinline__ void rows_out(const Stage& S, const float2* tw, const float2* tile, float2* dst, long long step,
                                         int ty, int yl, int w, int W, bool live, bool conj) {
  with_radix<RM>(S.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int j = w; j < S.units; j += W) {
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = tile[(j + r * S.sub) * ty + yl];
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul_conj(v[r], tw[S.two + r * S.sub + j]);
      Dft<R, true>::run(v);
      if (live) {
#pragma unroll
        for (int r = 0; r < R; ++r) dst[(j + r * S.sub) * step] = conj ? make_float2(v[r].x, -v[r].y) : v[r];
      }
    }
  });
}

// a + b and what its rounding leaves
__device__ __forceinline__ float2 two_sum(float a, float b) {
  const float s = a + b, t = s - a;
  return make_float2(s, (a - (s - t)) + (b - t));
}

// norm (1 + e) / (dr + i di), for an e below the rounding of norm itself: as a
// float, norm / (dr^2 + di^2) would lose e (always, where norm is a power of
// two), so it is carried in two floats into the products with dr and di,
// whose roundings e then shifts on average.  (81 x 360 with the gains by
// position alone: 5e-7 more on the energies.)
__device__ __forceinline__ float2 green(float dr, float di, float norm, float e) {
  const float d = fmaf(dr, dr, di * di);
  const float r = __frcp_rn(d);
  const float inv = norm * r;
  const float lo = fmaf(inv, fmaf(-r, fminf(d, 3e38f), 1.f) + e, fmaf(norm, r, -inv));
  return make_float2(fmaf(dr, inv, dr * lo), fmaf(-di, inv, -di * lo));
}

// K2: forward transform along the outer dimension, Green's function, inverse.
// po, eo: p and (of the first n / RL elements) the gain's inverse along the outer dimension.
// PSTD: the Laplacian instead (kEither: as a.pstd says)
enum { kGreen = 0, kLaplacian = 1, kEither = 2 };
template <int RM, int NC, int PSTD>
__device__ __forceinline__ void pencil_body(const PencilArgs& a, const Wig& wg, int rhs, int bid, float2* tile, const float2* tw,
                                            const float* po, const float* eo) {
  const Geom& g = a.g;
  const int ty = 1 << a.lty, yl = threadIdx.x & (ty - 1), w = threadIdx.x >> a.lty, W = blockDim.x >> a.lty;
  const int mid = bid / a.nyt, y = (bid - mid * a.nyt) * ty + yl;
  const bool live = y < g.ny;
  const long long step = a.mode3d ? a.pitch * g.nx : a.pitch;
  float2* const base = a.T + rhs * a.tstride + mid * a.pitch + y;
  const int n = a.po.n, tn = n * ty;
  const float py = live ? __ldg(&wg.pye[y]) : 0.f;
  const float pm = a.mode3d ? __ldg(&wg.pxe[mid]) : __ldg(&wg.pze[0]);
  const float e2 = a.norm_e + (live ? __ldg(&a.ey[y]) : 0.f) + (a.mode3d ? __ldg(&a.ex[mid]) : 0.f);
#pragma unroll
  for (int c = 0; c < NC; ++c) rows_in<RM>(a.po.st[0], tw, base + c * a.cstride, step, tile + c * tn, ty, yl, w, W, live);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < NC; ++c) row_middles<RM, false>(a.po, tile + c * tn, tw, ty, yl, w, W);
  const Stage& SL = a.po.st[a.po.nst - 1];
  // |p|^2 - Re k02e: near resonance the difference of two numbers 10 times its size, so
  // what does not depend on the pencil's own p is kept in two floats
  const float py2 = py * py, pm2 = pm * pm;
  const float2 s1 = two_sum(pm2, -a.k02e.x), s2 = two_sum(s1.x, py2);
  const float base2 = s2.x, low2 = (s1.y + s2.y) + (fmaf(pm, pm, -pm2) + fmaf(py, py, -py2));
  const float di = -a.k02e.y;
  with_radix<RM>(SL.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int u = w; u < SL.units; u += W) {
      float2* p = tile + u * R * ty + yl;
      const float eu = e2 + eo[u];
      if constexpr (NC == 1) {
        float2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = p[i * ty];
        Dft<R, false>::run(v);
        // f_g0_scalar with the 1/N of ifftn: E ./ (px^2 + py^2 + (pz^2 - k02e)),
        // or the PSTD Laplacian (k02e = 0)
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float q = po[u + i * SL.units];
          const float dr = fmaf(q, q, base2) + low2;
          const float e = eu - (float)round_trip(0, R, i);
          if (PSTD == kLaplacian || (PSTD == kEither && a.pstd)) {
            const float s = -dr * a.norm, lo = fmaf(s, e, fmaf(-dr, a.norm, -s));
            v[i] = make_float2(fmaf(s, v[i].x, lo * v[i].x), fmaf(s, v[i].y, lo * v[i].y));
          } else {
            v[i] = cmul(v[i], green(dr, di, a.norm, e));
          }
        }
        Dft<R, true>::run(v);
#pragma unroll
        for (int i = 0; i < R; ++i) p[i * ty] = v[i];
      } else {
        // f_g0_vector: div = (p . E) / k02e; E_i <- (E_i - p_i div) / (|p|^2 - k02e); the components
        // one after the other, so that two lines of registers do for three (x, y, z: the pencil's own
        // p is that of z in 3-D, of x in 2-D)
        float2 pe[R];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float2 v[R];
#pragma unroll
          for (int i = 0; i < R; ++i) v[i] = p[c * tn + i * ty];
          Dft<R, false>::run(v);
#pragma unroll
          for (int i = 0; i < R; ++i) {
            p[c * tn + i * ty] = v[i];
            const float pc = c == 1 ? py : ((c == 0) == (a.mode3d != 0) ? pm : po[u + i * SL.units]);
            pe[i] = c == 0 ? cscale(v[i], pc) : make_float2(fmaf(pc, v[i].x, pe[i].x), fmaf(pc, v[i].y, pe[i].y));
          }
        }
#pragma unroll
        for (int i = 0; i < R; ++i) pe[i] = cmul(pe[i], a.ik02e);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float2 v[R];
#pragma unroll
          for (int i = 0; i < R; ++i) {
            const float q = po[u + i * SL.units];
            const float dr = fmaf(q, q, base2) + low2;
            const float pc = c == 1 ? py : ((c == 0) == (a.mode3d != 0) ? pm : q);
            const float2 f = p[c * tn + i * ty];
            v[i] = cmul(make_float2(fmaf(-pc, pe[i].x, f.x), fmaf(-pc, pe[i].y, f.y)),
                        green(dr, di, a.norm, eu - (float)round_trip(0, R, i)));
          }
          Dft<R, true>::run(v);
#pragma unroll
          for (int i = 0; i < R; ++i) p[c * tn + i * ty] = v[i];
        }
      }
    }
  });
  __syncthreads();
#pragma unroll
  for (int c = 0; c < NC; ++c) row_middles<RM, true>(a.po, tile + c * tn, tw, ty, yl, w, W);
#pragma unroll
  for (int c = 0; c < NC; ++c)
    rows_out<RM>(a.po.st[0], tw, tile + c * tn, base + c * a.cstride, step, ty, yl, w, W, live, a.pstd == 1);
}

template <int RM, int NC>
__global__ void __launch_bounds__(kMaxThreads, (NC == 1 ? kBlocks<RM> : kBlocksHeavy<RM>)) k_pencil(
    const __grid_constant__ PencilArgs a) {
  const int rhs = blockIdx.x / a.bpr, bid = blockIdx.x - rhs * a.bpr;
  if (load_done(a.st + rhs)) return;
  extern __shared__ float2 tile[];
  float* const po = reinterpret_cast<float*>(tile + NC * (a.po.n << a.lty));
  float* const eo = po + a.po.n;
  copy_table(po, a.mode3d ? a.w.pze : a.w.pxe, a.po.n);
  copy_table(eo, a.mode3d ? a.ez : a.ex, a.po.st[a.po.nst - 1].units);
  pencil_body<RM, NC, NC == 1 ? kEither : kGreen>(a, a.w, rhs, bid, tile, a.po.tw, po, eo);
}

// The x transforms of a 3-D grid, in place on T
template <int RM, bool INV>
__device__ __forceinline__ void x_body(const XArgs& a, int rhs, int bid, float2* tile) {
  const float2* const tw = a.px.tw;
  const int ty = 1 << a.lty, yl = threadIdx.x & (ty - 1), w = threadIdx.x >> a.lty, W = blockDim.x >> a.lty;
  const int zc = bid / a.nyt, y = (bid - zc * a.nyt) * ty + yl;
  const bool live = y < a.ny;
  float2* const base = a.T + rhs * a.tstride + zc * (a.pitch * a.nx) + y;
  const Stage& SL = a.px.st[a.px.nst - 1];
  if (!INV) {
    rows_in<RM>(a.px.st[0], tw, base, a.pitch, tile, ty, yl, w, W, live);
    __syncthreads();
    row_middles<RM, false>(a.px, tile, tw, ty, yl, w, W);
  }
  with_radix<RM>(SL.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int u = w; u < SL.units; u += W) {
      float2* p = tile + u * R * ty + yl;
      float2 v[R];
      if (INV) {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = live ? __ldcg(&base[(u + i * SL.units) * a.pitch]) : make_float2(0.f, 0.f);
      } else {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = p[i * ty];
      }
      Dft<R, INV>::run(v);
      if (INV) {
#pragma unroll
        for (int i = 0; i < R; ++i) p[i * ty] = v[i];
      } else if (live) {
#pragma unroll
        for (int i = 0; i < R; ++i) base[(u + i * SL.units) * a.pitch] = v[i];
      }
    }
  });
  if (INV) {
    __syncthreads();
    row_middles<RM, true>(a.px, tile, tw, ty, yl, w, W);
    rows_out<RM>(a.px.st[0], tw, tile, base, a.pitch, ty, yl, w, W, live, false);
  }
}

template <int RM, bool INV>
__global__ void __launch_bounds__(kMaxThreads, kBlocks<RM>) k_x(const __grid_constant__ XArgs a) {
  const int rhs = blockIdx.x / a.bpr, bid = blockIdx.x - rhs * a.bpr;
  if (load_done(a.st + rhs)) return;
  extern __shared__ float2 tile[];
  x_body<RM, INV>(a, rhs, bid, tile);
}

// The loop -------------------------------------------------------------------
// What bounds a small 2-D grid is latency: of a launch (64 x 56 and 512^2 spent
// 4-5 of their 6-9 us a pass between kernels and in their first loads), and of
// the loads of everything that a new kernel, or a barrier's acquire, finds
// dropped from L1.  So one launch runs the whole loop; between its barriers
// (1.5-2 us over 148 blocks, less over one cluster) only T goes through L2,
// while the tables of all wiggles and the block's own gamma and dE' (and E') sit
// in shared memory.  Every block steps the stop rule for itself, so that no
// barrier is spent on it.  us an iteration, before (one launch per pass) and
// now: 64 x 56 12.8, 7.5; 160 x 264 21.4, 12.4; 396 x 315 19.7, 11.0; 512^2
// 18.8, 12.7; 1100 x 768 38, 30.  With the fields left in global memory: 9.4,
// 14.5, 14.6, 16.3, 34.  In 3-D (four barriers, more work per point) it lost:
// 96^3 39 against 30, 63 x 77 x 70 x 3 58 against 49, so those stay launched.

// Barrier of all blocks of a cooperative launch; false (in every thread)
// after `limit` clocks, with *err set.  What a block wrote before it is
// visible to loads past L1 (__ldcg) of the others after it.
__device__ __forceinline__ bool grid_barrier(unsigned* arrived, unsigned& target, int* err, long long limit) {
  __shared__ int ok;
  if (!arrived) {  // the grid is one cluster
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    __threadfence();
    atomicAdd(arrived, 1u);
    const long long t0 = clock64();
    int good = 1;
    while (true) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
      if ((int)(v - target) >= 0) break;
      if (clock64() - t0 > limit) {
        atomicExch(err, 1);
        good = 0;
        break;
      }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

template <int RM>
__global__ void __launch_bounds__(kLoopThreads, 1) k_loop(const __grid_constant__ LoopArgs a) {
  extern __shared__ float2 tile[];
  __shared__ DevState st[kLoopRhs];
  __shared__ double energy[kMaxWiggles];
  const int tid = threadIdx.x, nthr = blockDim.x;
  const Geom& g = a.col.g;
  const int nw = a.nw, lines = a.col.lines;
  const int pencils = a.pen.bpr * a.nrhs, columns = a.col.bpr * a.nrhs;
  unsigned target = 0;
  // tables, for every wiggle of the cycle
  float2* const tw_col = tile + a.tile_elems;
  float2* const tw_out = tw_col + a.col.py.ntw;
  float2* const gy = tw_out + a.pen.po.ntw;  // nw ramps
  float2* const gxz = gy + nw * g.ny;        // nw values per column
  float2* const gamma = gxz + nw * lines;    // the block's columns
  float2* const dE = gamma + lines * g.ny;
  float2* const Es = dE + lines * g.ny;
  ColLine* const info = reinterpret_cast<ColLine*>(Es + (a.e_resident ? lines * g.ny : 0));
  float* const red = reinterpret_cast<float*>(info + lines);
  float* const eo = red + a.groups;  // the gain's inverse and nw p tables of the outer dimension
  const int neo = a.pen.po.st[a.pen.po.nst - 1].units;
  float* const po = eo + neo;
  const bool own = blockIdx.x < columns;  // the block's column tile
  const int crhs = own ? blockIdx.x / a.col.bpr : 0, cbid = blockIdx.x - crhs * a.col.bpr;
  const int col0 = cbid * lines, nl = own ? min(lines, a.col.total - col0) : 0;
  const long long f0 = crhs * a.col.fstride + (long long)col0 * g.ny;
  float2* const E = a.e_resident ? Es : a.col.E + f0;
  copy_table(tw_col, a.col.py.tw, a.col.py.ntw);
  copy_table(tw_out, a.pen.po.tw, a.pen.po.ntw);
  copy_table(eo, a.pen.ex, neo);
  for (int i = 0; i < nw; ++i) {
    copy_table(gy + i * g.ny, a.wig[i].gy, g.ny);
    copy_table(po + i * a.pen.po.n, a.wig[i].pxe, a.pen.po.n);
  }
  for (int l = tid; l < nl; l += nthr) {
    const int x = col0 + l;
    for (int i = 0; i < nw; ++i) gxz[i * lines + l] = cmul(a.wig[i].gx[x], a.wig[i].gz[0]);
    info[l] = ColLine{(long long)l * g.ny, x >= g.r0[1] && x < g.r1[1] && g.r0[2] == 0 && g.r0[3] == 0};
  }
  for (int i = tid; i < nl * g.ny; i += nthr) {
    gamma[i] = a.col.gamma[crhs * a.col.gstride + (long long)col0 * g.ny + i];
    dE[i] = a.col.dE[f0 + i];
    if (a.e_resident) Es[i] = a.col.E[f0 + i];
  }
  if (tid < a.nrhs) st[tid] = a.st[tid];
  __syncthreads();
  Hist hist = a.hist;
  if (blockIdx.x != 0) hist.cap = 0;  // every block steps the stop rule, block 0 writes the history
  for (long long cycle = 0; cycle < a.max_cycles; ++cycle) {
    bool first = false, any = false;  // first: the source still enters
    for (int r = 0; r < a.nrhs; ++r) {
      any |= !st[r].done;
      first |= !st[r].done && st[r].it == 1;
    }
    if (!any) break;
    for (int i = 0; i < nw; ++i) {
      const int i1 = i + 1 < nw ? i + 1 : 0;
      for (int t = blockIdx.x; t < pencils; t += gridDim.x) {
        const int rhs = a.nrhs > 1 ? t / a.pen.bpr : 0;
        if (!st[rhs].done)
          pencil_body<RM, 1, kGreen>(a.pen, a.wig[i], rhs, t - rhs * a.pen.bpr, tile, tw_out, po + i * a.pen.po.n, eo);
        __syncthreads();
      }
      if (!grid_barrier(a.arrived, target, a.err, a.limit)) return;
      if (own && !st[crhs].done) {
        ColIter it{};
        it.src = first && i1 > 0 ? a.src : nullptr;
        it.partials = a.partials + (long long)i * columns;
        it.acc = nw % 2 ? kAccEach : (i % 2 ? kAccPair : kAccSkip);
        col_body<RM, kStep, false>(a.col, it,
                            ColMem{tile, tw_col, gy + i * g.ny, gy + i1 * g.ny, gxz + i * lines, gxz + i1 * lines, info,
                                   red, gamma, dE, E},
                            crhs, cbid);
      }
      if (!grid_barrier(a.arrived, target, a.err, a.limit)) return;
    }
    // the stop rule of the cycle, the same in every block
    for (int r = 0; r < a.nrhs; ++r) {
      if (st[r].done) continue;
      for (int k = tid >> 5; k < nw; k += nthr / 32) {
        const double e = sum_partials(a.partials + (long long)k * columns + r * a.col.bpr, a.col.bpr);
        if ((tid & 31) == 0) energy[k] = e;
      }
      __syncthreads();
      if (tid == 0) {
        DevState s = st[r];
        Hist h = hist;
        h.diff += r * h.stride;
        if (h.fresh) h.fresh += r * h.stride;
        for (int k = 0; k < nw && !s.done; ++k) {
          s.e_acc = energy[k];
          finish_iteration(&s, a.rule, h);
        }
        st[r] = s;
      }
      __syncthreads();
    }
  }
  for (int i = tid; i < nl * g.ny; i += nthr) {
    a.col.dE[f0 + i] = dE[i];
    if (a.e_resident) a.col.E[f0 + i] = Es[i];
  }
  if (blockIdx.x == 0 && tid < a.nrhs) a.st[tid] = st[tid];
}

// us a step at 256^2: 11, against 30 of five launches a step (the inner
// transform, the outer pencils, the inner transform again for the inverse, the
// leapfrog, the stop rule), which the host issued one by one.
template <int RM>
__global__ void __launch_bounds__(kLoopThreads, 1) k_pstd_loop(const __grid_constant__ PstdLoopArgs a) {
  extern __shared__ float2 tile[];
  __shared__ DevState st;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const Geom& g = a.col.g;
  const int lines = a.col.lines, elems = lines * g.ny;
  unsigned target = 0;
  float2* const tw_col = tile + a.tile_elems;
  float2* const tw_out = tw_col + a.col.py.ntw;
  float2* const c12 = tw_out + a.pen.po.ntw;  // the block's columns
  float2* const E = c12 + elems;              // two fields
  float2* const S = E + 2 * elems;
  ColLine* const info = reinterpret_cast<ColLine*>(S + elems);
  float* const red = reinterpret_cast<float*>(info + lines);
  float* const po = red + a.groups;
  float* const eo = po + a.pen.po.n;
  const int neo = a.pen.po.st[a.pen.po.nst - 1].units;
  float* const c3 = eo + neo;
  const bool own = blockIdx.x < a.col.bpr;
  const int col0 = blockIdx.x * lines, nl = own ? min(lines, a.col.total - col0) : 0;
  const long long f0 = (long long)col0 * g.ny;
  copy_table(tw_col, a.col.py.tw, a.col.py.ntw);
  copy_table(tw_out, a.pen.po.tw, a.pen.po.ntw);
  copy_table(po, a.pen.w.pxe, a.pen.po.n);
  copy_table(eo, a.pen.ex, neo);
  for (int l = tid; l < nl; l += nthr) {
    const int x = col0 + l;
    info[l] = ColLine{(long long)l * g.ny, x >= g.r0[1] && x < g.r1[1] && g.r0[2] == 0};
  }
  for (int i = tid; i < nl * g.ny; i += nthr) {
    c12[i] = a.col.gamma[f0 + i];
    c3[i] = a.c3[f0 + i];
    S[i] = a.src[f0 + i];
    E[i] = a.fields[f0 + i];
    E[elems + i] = a.fields[g.npts + f0 + i];
  }
  if (tid == 0) st = *a.st;
  __syncthreads();
  for (int k = 0; k < a.steps && !st.done; ++k) {
    const PstdStepAmp amp = a.amp[k];
    for (int t = blockIdx.x; t < a.pen.bpr; t += gridDim.x) {
      pencil_body<RM, 1, kLaplacian>(a.pen, a.pen.w, 0, t, tile, tw_out, po, eo);
      __syncthreads();
    }
    if (!grid_barrier(a.arrived, target, a.err, a.limit)) return;
    const int cur = (st.it - 1) & 1;
    if (own) {
      ColIter it{};
      it.partials = a.partials;
      ColMem m{tile, tw_col, nullptr, nullptr, nullptr, nullptr, info, red, c12, E + cur * elems, E + (1 - cur) * elems};
      m.c3 = c3;
      m.S = S;
      m.A = amp.A;
      m.ps = amp.ps;
      col_body<RM, kPstd, false>(a.col, it, m, 0, blockIdx.x);
    }
    if (!grid_barrier(a.arrived, target, a.err, a.limit)) return;
    // Simulation.next (Simulation.m:193-217) for PSTD.run_algorithm (PSTD.m:108-124), the same in every block
    if (tid < 32) {
      const int calc = st.calc_energy;
      __syncwarp();  // lane 0 changes it below, and without an energy nothing else holds it back
      const double e = calc ? sum_partials(a.partials, a.col.bpr) : 0.0;
      if (tid == 0) {
        if (calc) st.last_step_energy = e / amp.A2;
        const double d = st.last_step_energy;
        const int it = st.it;
        if (blockIdx.x == 0 && it - 1 < a.hist_cap) a.hist[it - 1] = d;
        if (it == 1) st.diff1 = d;
        if (amp.may_end && d / st.diff1 < a.threshold) {
          st.done = 1;
          st.converged = 1;
        } else if (amp.may_end && it >= a.max_iter) {
          st.done = 1;
          st.converged = 0;
        }
        st.calc_energy = ((it - 1) % a.interval) == 0;
        st.it = it + 1;
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < nl * g.ny; i += nthr) {
    a.fields[f0 + i] = E[i];
    a.fields[g.npts + f0 + i] = E[elems + i];
  }
  if (blockIdx.x == 0 && tid == 0) *a.st = st;
}

template <int RM>
Kernels kernels_up_to() {
  const void* const fwd = (const void*)k_col<RM, kFwd, true>;  // the same for both
  return Kernels{{{fwd, (const void*)k_col<RM, kInv, false>, (const void*)k_col<RM, kStep, false>},
                  {fwd, (const void*)k_col<RM, kInv, true>, (const void*)k_col<RM, kStep, true>}},
                 {(const void*)k_x<RM, false>, (const void*)k_x<RM, true>},
                 {(const void*)k_pencil<RM, 1>, (const void*)k_pencil<RM, 3>},
                 (const void*)k_loop<RM>, (const void*)k_pstd_loop<RM>};
}

}  // namespace uni
}  // namespace ws
