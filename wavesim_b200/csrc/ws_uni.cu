// The kernels of ws_uni.cuh.
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
__device__ __forceinline__ void middle(float2* p, int step, const float2* __restrict__ tw, int sub) {
  float2 v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = p[r * step];
  if (INV) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul_conj(v[r], __ldg(&tw[r * sub]));
  }
  Dft<R, INV>::run(v);
  if (!INV) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(&tw[r * sub]));
  }
#pragma unroll
  for (int r = 0; r < R; ++r) p[r * step] = v[r];
}

// Column pass --------------------------------------------------------------
// kFwd: K1 (source, ramps, forward y); kInv: K3 (inverse y, f_mix, E' += dE',
// energy); kStep: K3 of an iteration and K1 of the next.
struct ColLine {
  float2 g0, g1;  // gx gz of this iteration and of the next
  long long goff;  // offset of the column's gamma
  int in;          // x, z and the component inside the roi
};

template <int RM, bool INV>
__device__ __forceinline__ void col_middles(const ColArgs& a, float2* tile, int nl, int tid, int nthr) {
  for (int k = 1; k < a.py.nst - 1; ++k) {
    const Stage& S = a.py.st[INV ? a.py.nst - 1 - k : k];
    with_radix<RM>(S.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int q = tid; q < nl * S.units; q += nthr) {
        const int l = quot(q, S.munits), u = q - l * S.units;
        const int b = quot(u, S.msub), j = u - b * S.sub;
        float2* p = tile + l * a.py.np + b * S.blkp + j + (a.py.pad ? quot(j, a.py.mrl) : 0);
        middle<R, INV>(p, S.subp, S.tw + j, S.sub);
      }
    });
    __syncthreads();
  }
}

template <int RM, int MODE>
__global__ void __launch_bounds__(kMaxThreads, (MODE == kFwd ? kBlocks<RM> : kBlocksHeavy<RM>)) k_col(const __grid_constant__ ColArgs a) {
  const int rhs = blockIdx.x / a.bpr, bid = blockIdx.x - rhs * a.bpr;
  const DevState* st = a.st + rhs;
  if (load_done(st)) return;
  const bool acc_now = MODE != kFwd && a.acc2 != kAccSkip;
  extern __shared__ float2 tile[];
  const Geom& g = a.g;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int col0 = bid * a.lines;
  const int nl = min(a.lines, a.total - col0);
  ColLine* const info = reinterpret_cast<ColLine*>(tile + a.lines * a.py.np);
  float2* const T = a.T + rhs * a.tstride + col0 * a.pitch;
  const long long f0 = rhs * a.fstride + (long long)col0 * g.ny;
  for (int l = tid; l < nl; l += nthr) {
    const int col = col0 + l;
    const int zc = col / g.nx, x = col - zc * g.nx;
    const int c = zc / g.nz, z = zc - c * g.nz;
    ColLine I;
    if (MODE != kFwd) I.g0 = cmul(a.gx[x], a.gz[z]);
    if (MODE != kInv) I.g1 = cmul(a.gx1[x], a.gz1[z]);
    I.goff = rhs * a.gstride + (long long)col * g.ny - c * g.npts;
    I.in = x >= g.r0[1] && x < g.r1[1] && z >= g.r0[2] && z < g.r1[2] && c >= g.r0[3] && c < g.r1[3];
    info[l] = I;
  }
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
        for (int i = 0; i < R; ++i) v[i] = t[i * SL.units];
        Dft<R, true>::run(v);
        float2* p = tile + l * a.py.np + u * SL.blkp;
#pragma unroll
        for (int i = 0; i < R; ++i) p[i] = v[i];
      }
    });
    __syncthreads();
    col_middles<RM, true>(a, tile, nl, tid, nthr);
  } else {
    __syncthreads();
  }
  float esum = 0.f;
  with_radix<RM>(S0.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int q = tid; q < nl * S0.units; q += nthr) {
      const int l = quot(q, S0.munits), j = q - l * S0.units;
      const ColLine I = info[l];
      float2* p = tile + l * a.py.np + j + (a.py.pad ? quot(j, a.py.mrl) : 0);
      const long long at = f0 + (long long)l * g.ny + j;
      float2 v[R];
      if (MODE != kFwd) {
        const float2* __restrict__ gmc = a.gamma + I.goff + j;
        float2* __restrict__ dEc = a.dE + at;
        float2* __restrict__ Ec = a.E + at;
        // the epilogue's loads in groups of H elements, the first group's before the butterfly
        constexpr int H = R <= 5 ? R : (R <= 10 ? (R + 1) / 2 : (R + 2) / 3);
        float2 gm[H], d0[H];
#pragma unroll
        for (int r = 0; r < H; ++r) {
          gm[r] = gmc[r * S0.sub];
          d0[r] = dEc[r * S0.sub];
        }
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = p[r * S0.subp];
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = cmul_conj(v[r], __ldg(&S0.tw[r * S0.sub + j]));
        Dft<R, true>::run(v);
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
              const int m = h + r, y = j + m * S0.sub;
              // Eprop after the conjugate ramps (WaveSim.m:55), f_mix (f_mix.m:3-4), E' += dE'
              const float2 ep = cmul_conj(cmul_conj(v[m], I.g0), __ldg(&a.gy[y]));
              const float2 one_m = make_float2(1.f - kAlpha * gm[r].x, -kAlpha * gm[r].y);
              const float2 t = cmul(cmul(gm[r], gm[r]), ep);
              const float2 dn = cadd(cmul(one_m, d0[r]), make_float2(kAlpha * t.y, -kAlpha * t.x));
              dEc[m * S0.sub] = dn;
              if (acc_now) Ec[m * S0.sub] = cadd(e0[r], a.acc2 ? cadd(d0[r], dn) : dn);
              if (I.in && y >= g.r0[0] && y < g.r1[0]) esum = fmaf(dn.x, dn.x, fmaf(dn.y, dn.y, esum));
              v[m] = dn;
            }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = a.dE_in[at + r * S0.sub];
      }
      if (MODE != kInv) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (a.src) v[r] = cadd(v[r], cmul(a.A, a.src[at + r * S0.sub]));
          v[r] = cmul(cmul(v[r], I.g1), __ldg(&a.gy1[j + r * S0.sub]));
        }
        Dft<R, false>::run(v);
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(&S0.tw[r * S0.sub + j]));
#pragma unroll
        for (int r = 0; r < R; ++r) p[r * S0.subp] = v[r];
      }
    }
  });
  if (MODE != kInv) {
    __syncthreads();
    col_middles<RM, false>(a, tile, nl, tid, nthr);
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
    __shared__ float red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) esum += __shfl_xor_sync(0xffffffffu, esum, o);
    if ((tid & 31) == 0) red[tid >> 5] = esum;
    __syncthreads();
    if (tid == 0) {
      float v = 0.f;
      for (int w = 0; w < nthr / 32; ++w) v += red[w];
      a.partials[blockIdx.x] = (double)v;
    }
  }
}

// Pencils --------------------------------------------------------------------
// A tile holds ty consecutive y of one line of N rows: element (row, yl) at
// row * ty + yl; thread (w, yl) takes the butterflies w, w + W, ...
template <int RM, bool INV>
__device__ __forceinline__ void row_middles(const Plan& P, float2* tile, int ty, int yl, int w, int W) {
  for (int k = 1; k < P.nst - 1; ++k) {
    const Stage& S = P.st[INV ? P.nst - 1 - k : k];
    with_radix<RM>(S.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int u = w; u < S.units; u += W) {
        const int b = quot(u, S.msub), j = u - b * S.sub;
        middle<R, INV>(tile + (b * S.R * S.sub + j) * ty + yl, S.sub * ty, S.tw + j, S.sub);
      }
    });
    __syncthreads();
  }
}

// first stage of a forward transform, from global rows into the tile
template <int RM>
__device__ __forceinline__ void rows_in(const Stage& S, const float2* src, long long step, float2* tile,
                                        int ty, int yl, int w, int W, bool live) {
  with_radix<RM>(S.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int j = w; j < S.units; j += W) {
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = live ? src[(j + r * S.sub) * step] : make_float2(0.f, 0.f);
      Dft<R, false>::run(v);
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(&S.tw[r * S.sub + j]));
#pragma unroll
      for (int r = 0; r < R; ++r) tile[(j + r * S.sub) * ty + yl] = v[r];
    }
  });
}

// last stage of an inverse transform, from the tile to global rows
template <int RM>
__device__ __forceinline__ void rows_out(const Stage& S, const float2* tile, float2* dst, long long step,
                                         int ty, int yl, int w, int W, bool live, bool conj) {
  with_radix<RM>(S.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int j = w; j < S.units; j += W) {
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = tile[(j + r * S.sub) * ty + yl];
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul_conj(v[r], __ldg(&S.tw[r * S.sub + j]));
      Dft<R, true>::run(v);
      if (live) {
#pragma unroll
        for (int r = 0; r < R; ++r) dst[(j + r * S.sub) * step] = conj ? make_float2(v[r].x, -v[r].y) : v[r];
      }
    }
  });
}

// K2: forward transform along the outer dimension, Green's function, inverse
template <int RM, int NC>
__global__ void __launch_bounds__(kMaxThreads, (NC == 1 ? kBlocks<RM> : kBlocksHeavy<RM>)) k_pencil(const __grid_constant__ PencilArgs a) {
  const int rhs = blockIdx.x / a.bpr, bid = blockIdx.x - rhs * a.bpr;
  if (load_done(a.st + rhs)) return;
  extern __shared__ float2 tile[];
  const Geom& g = a.g;
  const int ty = a.ty, yl = threadIdx.x % ty, w = threadIdx.x / ty, W = blockDim.x / ty;
  const int mid = bid / a.nyt, y = (bid - mid * a.nyt) * ty + yl;
  const bool live = y < g.ny;
  const long long step = a.mode3d ? a.pitch * g.nx : a.pitch;
  float2* const base = a.T + rhs * a.tstride + mid * a.pitch + y;
  const int n = a.po.n, tn = n * ty;
#pragma unroll
  for (int c = 0; c < NC; ++c) rows_in<RM>(a.po.st[0], base + c * a.cstride, step, tile + c * tn, ty, yl, w, W, live);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < NC; ++c) row_middles<RM, false>(a.po, tile + c * tn, ty, yl, w, W);
  const Stage& SL = a.po.st[a.po.nst - 1];
  const float py = live ? __ldg(&a.w.pye[y]) : 0.f;
  const float pm = a.mode3d ? __ldg(&a.w.pxe[mid]) : __ldg(&a.w.pze[0]);
  const float* __restrict__ po = a.mode3d ? a.w.pze : a.w.pxe;
  const float base2 = fmaf(pm, pm, py * py);
  const float di = -a.k02e.y;
  with_radix<RM>(SL.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int u = w; u < SL.units; u += W) {
      float2* p = tile + u * R * ty + yl;
      if constexpr (NC == 1) {
        float2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = p[i * ty];
        Dft<R, false>::run(v);
        // f_g0_scalar with the 1/N of ifftn: E ./ (px^2 + py^2 + (pz^2 - k02e)),
        // or the PSTD Laplacian (k02e = 0)
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float q = __ldg(&po[u + i * SL.units]);
          const float dr = fmaf(q, q, base2) - a.k02e.x;
          if (a.pstd) {
            v[i] = make_float2(-dr * a.norm * v[i].x, -dr * a.norm * v[i].y);
          } else {
            const float inv = a.norm / fmaf(dr, dr, di * di);
            v[i] = cmul(v[i], make_float2(dr * inv, -di * inv));
          }
        }
        Dft<R, true>::run(v);
#pragma unroll
        for (int i = 0; i < R; ++i) p[i * ty] = v[i];
      } else {
        // f_g0_vector: div = (p . E) / k02e; E_i <- (E_i - p_i div) / (|p|^2 - k02e); the components
        // one after the other, so that two lines of registers do for three
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
            const float pc = c == 0 ? pm : (c == 1 ? py : __ldg(&po[u + i * SL.units]));
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
            const float q = __ldg(&po[u + i * SL.units]);
            const float dr = fmaf(q, q, base2) - a.k02e.x;
            const float inv = a.norm / fmaf(dr, dr, di * di);
            const float pc = c == 0 ? pm : (c == 1 ? py : q);
            const float2 e = p[c * tn + i * ty];
            v[i] = cmul(make_float2(fmaf(-pc, pe[i].x, e.x), fmaf(-pc, pe[i].y, e.y)),
                        make_float2(dr * inv, -di * inv));
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
  for (int c = 0; c < NC; ++c) row_middles<RM, true>(a.po, tile + c * tn, ty, yl, w, W);
#pragma unroll
  for (int c = 0; c < NC; ++c)
    rows_out<RM>(a.po.st[0], tile + c * tn, base + c * a.cstride, step, ty, yl, w, W, live, a.pstd != 0);
}

// The x transforms of a 3-D grid, in place on T
template <int RM, bool INV>
__global__ void __launch_bounds__(kMaxThreads, kBlocks<RM>) k_x(const __grid_constant__ XArgs a) {
  const int rhs = blockIdx.x / a.bpr, bid = blockIdx.x - rhs * a.bpr;
  if (load_done(a.st + rhs)) return;
  extern __shared__ float2 tile[];
  const int ty = a.ty, yl = threadIdx.x % ty, w = threadIdx.x / ty, W = blockDim.x / ty;
  const int zc = bid / a.nyt, y = (bid - zc * a.nyt) * ty + yl;
  const bool live = y < a.ny;
  float2* const base = a.T + rhs * a.tstride + zc * (a.pitch * a.nx) + y;
  const Stage& SL = a.px.st[a.px.nst - 1];
  if (!INV) {
    rows_in<RM>(a.px.st[0], base, a.pitch, tile, ty, yl, w, W, live);
    __syncthreads();
    row_middles<RM, false>(a.px, tile, ty, yl, w, W);
  }
  with_radix<RM>(SL.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int u = w; u < SL.units; u += W) {
      float2* p = tile + u * R * ty + yl;
      float2 v[R];
      if (INV) {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = live ? base[(u + i * SL.units) * a.pitch] : make_float2(0.f, 0.f);
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
    row_middles<RM, true>(a.px, tile, ty, yl, w, W);
    rows_out<RM>(a.px.st[0], tile, base, a.pitch, ty, yl, w, W, live, false);
  }
}

template <int RM>
static Kernels kernels_of() {
  return Kernels{{(const void*)k_col<RM, kFwd>, (const void*)k_col<RM, kInv>, (const void*)k_col<RM, kStep>},
                 {(const void*)k_x<RM, false>, (const void*)k_x<RM, true>},
                 {(const void*)k_pencil<RM, 1>, (const void*)k_pencil<RM, 3>}};
}
const Kernels& kernels(int cls) {
  static const Kernels t[kClasses] = {kernels_of<kClassRadix[0]>(), kernels_of<kClassRadix[1]>(),
                                      kernels_of<kClassRadix[2]>()};
  return t[cls];
}

}  // namespace uni
}  // namespace ws
