// mks_dslash_fx.cuh -- the FP64 D_eo in integer arithmetic (mks_fixed.cuh).
//
// One thread applies an output site's 16 links to one source (SPLIT = 1), or
// four threads take one direction each and add their integer sums by
// shuffles (SPLIT = 4, for lattices too small to fill the chip: a quarter of
// the serial chain, four times the warps).  Integer sums do not depend on
// their order, so every launch shape gives the same bits.
//
// What bounds it: one source, HBM (32^3x64: 0.391 ms against 0.372 ms for
// its 2.52 GB at the copy rate; the FP64 kernel 0.98 ms, at the FP64 rate);
// 8 sources, latency and the integer pipes (2.43 ms against 7.78 ms; 128
// registers, 16 warps per SM); 8^4, the chain of loads (8 us with four
// threads per site, 14 with one, 30 in FP64).  Lanes are consecutive sites
// and sources go by warps: with the sources in the lanes a quarter warp's
// vector load touched eight arrays, and the L1 data pipe was 80 % busy
// (24^3x48, 8 sources: 0.825 against 0.797 ms).
//
// Inputs are blocks (FxVec) of the other parity; the 16 neighbours are
// aligned to their largest exponent.  The result is written as blocks (the
// first D of D_eo D_oe: the second reads them as they are), as FP64 SoA, or
// in MILC's AoS layout.  A site with an infinity or a NaN among its
// neighbours is done in plain FP64; so is a slot whose links do not suit the
// integer form, by a kernel of its own (k_dslash_raw) on fields that hold
// doubles in the place of the blocks' integers.
#pragma once
#include "mks_fixed.cuh"
#include "mks_dslash.cuh"

namespace mks {

enum { FX_OUT_BLOCK = 0, FX_OUT_F64 = 1, FX_OUT_AOS = 2 };

struct FxArgs {
  Geom g;
  int out_par, nsrc;
  int G;                   // groups of sources: warps that share 32 / SPLIT sites
  int rev;                 // blocks take the sites in reverse order
  FxLinks fat, lng;
  const double2 *fat64, *lng64;   // the same links for sites done in plain FP64
  int EL, dE;                     // exponent of the fat links, and how far the Naik links' is above it
  FxVec in[MAXSRC];        // by source; by output parity in a launch of two grid rows (one source)
  FxVec outq[MAXSRC];
  double2 *out[MAXSRC];    // SoA, or MILC's AoS field
  const double2 *p[MAXSRC], *r[MAXSRC];   // epilogue operands (parity of out)
  double coef[MAXSRC];
  const int *skip;
  RedScratch red;
  double *totals;
};

// one site in plain FP64 (a neighbour is not finite)
static __device__ __noinline__ void fx_site_f64(const Geom &g, const double2 *fat, const double2 *lng, const FxVec &in,
                                                int par, int h, int x, int y, int z, int t, double *out) {
  const LinkF64 F = {fat}, Lg = {lng};
  const int c0[4] = {x, y, z, t}, L[4] = {g.nx, g.ny, g.nz, g.nt};
  auto vec = [&](int n) {
    V3<double> v;
    const int e = in.e[n];
#pragma unroll 1
    for (int c = 0; c < 3; c++) {
      const longlong2 w = in.q[(size_t)c * g.Vh + n];
      if (e == FX_SPECIAL) v.c[c] = {__longlong_as_double(w.x), __longlong_as_double(w.y)};
      else v.c[c] = {e == FX_ZERO ? 0.0 : fx_double(w.x, e), e == FX_ZERO ? 0.0 : fx_double(w.y, e)};
    }
    return v;
  };
  V3<double> acc = {{{0, 0}, {0, 0}, {0, 0}}};
#pragma unroll 1
  for (int mu = 0; mu < 4; mu++) {
    int hf1, hb1, hf3, hb3;
    nbr4(g, c0, L, mu, hf1, hb1, hf3, hb3);
    mv_acc(F.load(par, mu, h, g.Vh), vec(hf1), acc);
    mv_acc(Lg.load(par, mu, h, g.Vh), vec(hf3), acc);
    amv_sub(F.load(1 - par, mu, hb1, g.Vh), vec(hb1), acc);
    amv_sub(Lg.load(1 - par, mu, hb3, g.Vh), vec(hb3), acc);
  }
  for (int c = 0; c < 3; c++) { out[2 * c] = acc.c[c].re; out[2 * c + 1] = acc.c[c].im; }
}

// the epilogue's sums over the block (up to W warps, warp w of source group w
// % G) and the grid, and the finisher
template <int W, int NB, class Fin>
__device__ __forceinline__ void fx_sums(const double (&sums)[NB][3], const FxArgs &a, const Fin &fin) {
  __shared__ double smem[W * NB * 3];
  __shared__ double bt[MAXSRC * 3];
  __shared__ double tot[MAXSRC * 3];
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5, nwarps = (int)blockDim.x >> 5, G = a.G;
#pragma unroll
  for (int s = 0; s < NB; s++)
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double v = warp_sum(sums[s][k]);
      if (lane == 0) smem[(warp * NB + s) * 3 + k] = v;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < G * NB * 3; i += blockDim.x) {   // warp order
    const int g0 = i / (NB * 3), j = i - g0 * NB * 3;
    double v = 0;
    for (int w = g0; w < nwarps; w += G) v += smem[w * NB * 3 + j];
    bt[i] = v;
  }
  __syncthreads();
  if (grid_reduce_last(bt, G * NB * 3, a.red, tot)) {
    if (threadIdx.x == 0)
      for (int i = 0; i < a.nsrc * 3; i++) a.totals[i] = tot[i];
    __syncthreads();
    fin(tot, a.nsrc);
  }
}

// a site's result stored in MILC's AoS field
__device__ __forceinline__ void fx_store_aos(double2 *d, const double (&v)[6]) {
  if (((uintptr_t)d & 15) == 0) {
#pragma unroll
    for (int c = 0; c < 3; c++) d[c] = make_double2(v[2 * c], v[2 * c + 1]);
  } else {  // a caller's field on an 8-byte boundary
#pragma unroll
    for (int k = 0; k < 6; k++) reinterpret_cast<double *>(d)[k] = v[k];
  }
}

template <int SPLIT, bool DENSE, int NB, int OUT, int EPI, class Fin>
__device__ __forceinline__ void dslash_fx_body(const FxArgs &a, const Fin &fin) {
  if (a.skip && *a.skip) return;
  const Geom &g = a.g;
  const int Vh = g.Vh, par = a.out_par ^ (int)blockIdx.y, op = 1 - par, G = a.G;
  const int bid = a.rev ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5, nwarps = (int)blockDim.x >> 5;
  const int grp = warp % G, wsite = (bid * nwarps + warp) / G;   // blocks hold a multiple of G warps
  const int m0 = SPLIT == 1 ? 0 : lane % SPLIT;
  // where the FP64 rate counts, an FP64 tail takes one colour per thread
  constexpr int LANES = DENSE && OUT == FX_OUT_F64 ? 3 : 1, NC = 3 / LANES;
  const int h0 = wsite * (32 / SPLIT) + lane / SPLIT;
  // threads past the last site follow it, so that the shuffles of a warp see all lanes
  const int h = h0 < Vh ? h0 : Vh - 1;
  FxVec in[NB];
  bool live[NB];
#pragma unroll
  for (int s = 0; s < NB; s++) {
    const int S = grp * NB + s;
    live[s] = h0 < Vh && S < a.nsrc && m0 < LANES;
    in[s] = a.in[S < a.nsrc ? S + (int)blockIdx.y : 0];   // blockIdx.y = 1: the second parity of a one-source launch
  }
  int x, y, z, t;
  site_coords(g, par, h, x, y, z, t);
  const int c0[4] = {x, y, z, t}, L[4] = {g.nx, g.ny, g.nz, g.nt};
  int E[NB];
#pragma unroll
  for (int s = 0; s < NB; s++) E[s] = 2 * FX_ZERO;
#pragma unroll
  for (int k = 0; k < 4 / SPLIT; k++) {
    int f1, b1, f3, b3;
    nbr4(g, c0, L, SPLIT == 1 ? k : m0, f1, b1, f3, b3);
#pragma unroll
    for (int s = 0; s < NB; s++)
      E[s] = max(max(E[s], max(__ldg(in[s].e + f1), __ldg(in[s].e + b1))),
                 max(__ldg(in[s].e + f3), __ldg(in[s].e + b3)) + a.dE);
  }
  if (SPLIT > 1) {
#pragma unroll
    for (int s = 0; s < NB; s++)
#pragma unroll
      for (int o = 1; o < SPLIT; o *= 2) E[s] = max(E[s], __shfl_xor_sync(0xffffffffu, E[s], o));
  }
  FxAcc acc[NB];
#pragma unroll
  for (int s = 0; s < NB; s++)
#pragma unroll
    for (int i = 0; i < 3; i++) acc[s].k1[i] = acc[s].k2[i] = acc[s].k3[i] = {0, 0};
#pragma unroll 1
  for (int mu = m0; mu < 4; mu += SPLIT) {
    int nb[4];
    nbr4(g, c0, L, mu, nb[0], nb[1], nb[2], nb[3]);
#pragma unroll
    for (int kind = 0; kind < 2; kind++) {
      const FxLinks &U = kind ? a.lng : a.fat;
      FxOperand o[NB];
      const int nf = nb[2 * kind], nbk = nb[2 * kind + 1];
#pragma unroll
      for (int s = 0; s < NB; s++) {
        s64 q[6];
        fx_load(in[s], nf, Vh, q);
        fx_operand<1>(q, min((kind ? E[s] - a.dE : E[s]) - __ldg(in[s].e + nf), 63), o[s]);
      }
      fx_mv<false, NB>(U, par, mu, h, Vh, o, acc);
#pragma unroll
      for (int s = 0; s < NB; s++) {
        s64 q[6];
        fx_load(in[s], nbk, Vh, q);
        fx_operand<-1>(q, min((kind ? E[s] - a.dE : E[s]) - __ldg(in[s].e + nbk), 63), o[s]);
      }
      fx_mv<true, NB>(U, op, mu, nbk, Vh, o, acc);
    }
  }
  double sums[NB][3];
#pragma unroll
  for (int s = 0; s < NB; s++) {
    const int S = grp * NB + s + (int)blockIdx.y;
    sums[s][0] = sums[s][1] = sums[s][2] = 0;
    // (T + f 2^-28) 2^(E + EL - 56), six components
    s64 T[6];
    unsigned f[6];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      u64 H[2] = {acc[s].k1[i].H - acc[s].k3[i].H, acc[s].k1[i].H + acc[s].k2[i].H};
      u64 M[2] = {acc[s].k1[i].M - acc[s].k3[i].M, acc[s].k1[i].M + acc[s].k2[i].M};
#pragma unroll
      for (int k = 0; k < 2; k++) {
        if (SPLIT > 1) {
#pragma unroll
          for (int o = 1; o < SPLIT; o *= 2) {
            H[k] += __shfl_xor_sync(0xffffffffu, H[k], o);
            M[k] += __shfl_xor_sync(0xffffffffu, M[k], o);
          }
        }
        T[2 * i + k] = (s64)H[k] + ((s64)M[k] >> 28);
        f[2 * i + k] = (unsigned)M[k] & 0xfffffffu;
      }
    }
    if (!live[s]) continue;
    // normalise to |q| < 2^60 (at most the 28 bits of f are shifted in)
    u64 mag = 0;
    unsigned any = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) { mag |= (u64)(T[k] ^ (T[k] >> 63)); any |= f[k]; }
    const int sh = min(28, __clzll((s64)mag) - 4);
    int e = (mag | any) == 0 || E[s] < FX_ZERO / 2 ? FX_ZERO : E[s] + a.EL + 4 - sh;
    s64 q[6];
#pragma unroll
    for (int k = 0; k < 6; k++) q[k] = sh > 0 ? (s64)(((u64)T[k] << sh) + (f[k] >> (28 - sh))) : T[k] >> -sh;
    double v[6];
    if (E[s] > FX_SPECIAL / 2) {
      fx_site_f64(g, a.fat64, a.lng64, in[s], par, h, x, y, z, t, v);
      if (OUT == FX_OUT_BLOCK) fx_encode(v, q, e);
      if (LANES > 1) {
        v[0] = m0 == 0 ? v[0] : m0 == 1 ? v[2] : v[4];
        v[1] = m0 == 0 ? v[1] : m0 == 1 ? v[3] : v[5];
      }
    } else if (OUT != FX_OUT_BLOCK) {
      if (LANES > 1) {
        q[0] = m0 == 0 ? q[0] : m0 == 1 ? q[2] : q[4];
        q[1] = m0 == 0 ? q[1] : m0 == 1 ? q[3] : q[5];
      }
#pragma unroll
      for (int k = 0; k < 2 * NC; k++) v[k] = e == FX_ZERO ? 0.0 : fx_double(q[k], e);
    }
    if (OUT == FX_OUT_BLOCK) {
      fx_store(a.outq[S], h, Vh, q, e);
    } else if (OUT == FX_OUT_AOS) {
      fx_store_aos(a.out[S] + ((size_t)par * Vh + h) * 3, v);
    } else {
      if (EPI == EPI_AXPY) {
        const double cf = a.coef[S];
#pragma unroll
        for (int c = 0; c < NC; c++) {
          const double2 pv = __ldg(a.p[S] + (size_t)(LANES > 1 ? m0 : c) * Vh + h), rv = __ldg(a.r[S] + (size_t)(LANES > 1 ? m0 : c) * Vh + h);
          v[2 * c] = fma(cf, pv.x, v[2 * c]);
          v[2 * c + 1] = fma(cf, pv.y, v[2 * c + 1]);
          sums[s][0] = fma(pv.x, v[2 * c], fma(pv.y, v[2 * c + 1], sums[s][0]));
          sums[s][1] = fma(rv.x, v[2 * c], fma(rv.y, v[2 * c + 1], sums[s][1]));
          sums[s][2] = fma(v[2 * c], v[2 * c], fma(v[2 * c + 1], v[2 * c + 1], sums[s][2]));
        }
      }
#pragma unroll
      for (int c = 0; c < NC; c++) a.out[S][(size_t)(LANES > 1 ? m0 : c) * Vh + h] = make_double2(v[2 * c], v[2 * c + 1]);
    }
  }
  if (EPI == EPI_AXPY) fx_sums<8, NB>(sums, a, fin);
}

template <int SPLIT, int NB, int OUT, int EPI, class Fin>
__global__ void __launch_bounds__(256, NB == 1 ? 2 : 1) k_dslash_fx(const FxArgs a, const Fin fin) {
  dslash_fx_body<SPLIT, false, NB, OUT, EPI, Fin>(a, fin);
}

// Four threads per site in 96 registers: 20 warps per SM instead of 16, for
// launches that 20 hold at once and 16 do not.  On 12^3x24 those left 160 of
// 2592 warps to a second wave, and the FP64 tail of a warp (24 operations of
// 64 clocks, 8 when its threads share the colours) is a good part of an
// epilogue launch: the two D of a multi-shift iteration 55 and 48 us, the
// FP64 trajectory 143 and 135 ms.  On either side it loses: with more warps
// than 20 the registers count (a whole D call on 14x10x18x22, 23 warps: 34.0
// and 38.5 us; on 16^3x32, 54 warps: 52.6 and 55.7), and with 16 or fewer
// sharing colours costs two exchanges (8^4 CG: 1.43 and 1.49 ms).  D into
// MILC's layout, which has no tail to share, keeps the ordinary kernel; within
// the window the dense one would take 1.3 to 2 us off a call (12^3x24 30.5 and
// 29.0 us, 12^3x28 32.4 and 30.4).
template <int OUT, int EPI, class Fin>
__global__ void __launch_bounds__(128, 5) k_dslash_fx_dense(const FxArgs a, const Fin fin) {
  dslash_fx_body<4, true, 1, OUT, EPI, Fin>(a, fin);
}

// D_eo in plain FP64 on links that the integer form does not suit: in[].q and
// out[] hold doubles (a field of blocks keeps its size and its place).  One
// thread per site and source, sources by warps.  Bound by the FP64 rate (576
// fmas a site at 2 lanes per clock and SM): 32^3x64 1.00 ms for one source and
// 7.88 for 8 with the copy of the input.
template <int OUT, int EPI, class Fin>
__global__ void __launch_bounds__(512) k_dslash_raw(const FxArgs a, const Fin fin) {
  if (a.skip && *a.skip) return;
  const Geom &g = a.g;
  const int Vh = g.Vh, par = a.out_par ^ (int)blockIdx.y, G = a.G;
  const int bid = a.rev ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5, nwarps = (int)blockDim.x >> 5;
  const int S = warp % G + (int)blockIdx.y;   // blocks hold a multiple of G = nsrc warps
  const int h = (bid * nwarps + warp) / G * 32 + lane;
  double sums[1][3] = {{0, 0, 0}};
  if (h < Vh) {
    int x, y, z, t;
    site_coords(g, par, h, x, y, z, t);
    const int c0[4] = {x, y, z, t};
    const VecF64 in = {reinterpret_cast<double2 *>(a.in[S].q)};
    V3<double> acc[1] = {{{{0, 0}, {0, 0}, {0, 0}}}};
    site_terms<double, LinkF64, VecF64, 1, false>(LinkF64{a.fat64}, LinkF64{a.lng64}, &in, 1, 0, g, par, h, c0, acc);
    double v[6] = {acc[0].c[0].re, acc[0].c[0].im, acc[0].c[1].re, acc[0].c[1].im, acc[0].c[2].re, acc[0].c[2].im};
    if (EPI == EPI_AXPY) {
      const double cf = a.coef[S];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double2 pv = __ldg(a.p[S] + (size_t)c * Vh + h), rv = __ldg(a.r[S] + (size_t)c * Vh + h);
        v[2 * c] = fma(cf, pv.x, v[2 * c]);
        v[2 * c + 1] = fma(cf, pv.y, v[2 * c + 1]);
        sums[0][0] = fma(pv.x, v[2 * c], fma(pv.y, v[2 * c + 1], sums[0][0]));
        sums[0][1] = fma(rv.x, v[2 * c], fma(rv.y, v[2 * c + 1], sums[0][1]));
        sums[0][2] = fma(v[2 * c], v[2 * c], fma(v[2 * c + 1], v[2 * c + 1], sums[0][2]));
      }
    }
    if (OUT == FX_OUT_AOS) {
      fx_store_aos(a.out[S] + ((size_t)par * Vh + h) * 3, v);
    } else {
#pragma unroll
      for (int c = 0; c < 3; c++) a.out[S][(size_t)c * Vh + h] = make_double2(v[2 * c], v[2 * c + 1]);
    }
  }
  if (EPI == EPI_AXPY) fx_sums<16, 1>(sums, a, fin);
}

}  // namespace mks
