// mks_fixed_mat.cuh -- 3x3 products of FP64 link fields in integer arithmetic,
// and the staple kernels of the link construction and the fermion force on
// them (see mks_fixed.cuh for why: an fma.f64 costs 30 integer multiply-adds).
//
// A matrix is nine complex entries as integers with one exponent: component =
// q 2^(e-60), |q| <= 2^60, cut as q = 4 (h 2^30 + l), |h| <= 2^28, l signed,
// stored as int4 {re h, re l, im h, im l} (the 16 bytes of a double2).  A
// product is K = H 2^60 + M 2^30 by three multiply-adds per real product (the
// low halves' product, 2^-58 of the operands' bounds, is left out) and three
// real products per complex one; six terms of 2^56 leave room in 64 bits, and
// partial sums may wrap around.  q_out = 2 H + M 2^-29 keeps 60 bits of the
// bound 6 * 2^56, e_out = e_a + e_b + 3.  A matrix of zeros has e = FX_ZERO,
// one that holds an infinity or a NaN e = FX_SPECIAL and the doubles' bits; a
// site that meets one is done in plain FP64.
//
// A staple term is a chain L (M R) of three matrices, its adjoint six chains;
// the chains run in a loop whose operands are fetched three ahead into shared
// memory by cp.async (a fetch in flight holds no registers, of which the
// products take about 200).
#pragma once
#include "mks_fixed.cuh"
#include "mks_su3.cuh"

namespace mks {

// one direction of a link field, or a single matrix field
struct FxMat {
  int4 *p;     // [par ps + k Vh + h]
  int *e;      // [par es + h]
  size_t ps, es;
};
__host__ __device__ inline FxMat fx_link_dir(const FxMat &f, int dir, size_t Vh) {
  return {f.p + (size_t)dir * 9 * Vh, f.e + (size_t)dir * Vh, 36 * Vh, 4 * Vh};
}

__device__ __forceinline__ void fxm_split(s64 q, int &h, int &l) {
  const int lo = (int)q;
  h = (int)(q >> 32) + (int)((unsigned)lo >> 31);
  l = lo >> 2;
}

// a matrix of doubles as integers
__device__ __forceinline__ void fxm_encode(const double2 (&v)[9], int4 (&u)[9], int &e) {
  int ex = 0;
  s64 any = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const s64 a = __double_as_longlong(v[k].x), b = __double_as_longlong(v[k].y);
    ex = max(ex, max((int)(a >> 52) & 0x7ff, (int)(b >> 52) & 0x7ff));
    any |= (a | b) << 1;
  }
  if (ex == 0x7ff) {
    e = FX_SPECIAL;
#pragma unroll
    for (int k = 0; k < 9; k++)
      u[k] = make_int4(__double2hiint(v[k].x), __double2loint(v[k].x), __double2hiint(v[k].y), __double2loint(v[k].y));
    return;
  }
  e = max(ex, 1) - 1022;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    fxm_split(fx_scale(v[k].x, e) + 2, u[k].x, u[k].y);   // + 2: rounds the cut at 4
    fxm_split(fx_scale(v[k].y, e) + 2, u[k].z, u[k].w);
  }
  if (!any) e = FX_ZERO;
}

// [2][4][9][Vh] doubles -> integers
static __global__ void __launch_bounds__(128) k_links_to_fxm(const double2 *__restrict__ src, FxMat dst, int Vh) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x, par = blockIdx.y, mu = blockIdx.z;
  if (h >= Vh) return;
  const double2 *s = src + (size_t)(par * 4 + mu) * 9 * Vh + h;
  double2 v[9];
  int4 u[9];
  int e;
#pragma unroll
  for (int k = 0; k < 9; k++) v[k] = s[(size_t)k * Vh];
  fxm_encode(v, u, e);
#pragma unroll
  for (int k = 0; k < 9; k++) dst.p[(size_t)(par * 4 + mu) * 9 * Vh + (size_t)k * Vh + h] = u[k];
  dst.e[(size_t)(par * 4 + mu) * Vh + h] = e;
}

// workspace of `mats` integer matrices per site and parity under `name`
// (p given: the entries go there)
inline int ws_fxm(const char *name, int mats, FxMat *f, void *p = nullptr) {
  const size_t Vh = ctx().Vh;
  if (!p) MKS_TRY(ws(std::string(name) + "_p", (size_t)mats * 2 * 9 * Vh * sizeof(int4), &p));
  f->p = (int4 *)p;
  f->ps = (size_t)mats * 9 * Vh;
  f->es = (size_t)mats * Vh;
  return ws(std::string(name) + "_e", (size_t)mats * 2 * Vh * sizeof(int), (void **)&f->e);
}

// a link field [2][4][9][Vh] as integers in the workspace
inline int ws_links_fxm(const char *name, int family, const double2 *links, FxMat *f) {
  Context &c = ctx();
  MKS_TRY(ws_fxm(name, 4, f));
  timing_begin(family);
  k_links_to_fxm<<<dim3(grid_for(c.Vh, 128), 2, 4), 128, 0, c.stream>>>(links, *f, (int)c.Vh);
  timing_end(family);
  MKS_CUDA(cudaGetLastError());
  return MKS_OK;
}

// an operand of a chain: a site's matrix, as it is or its adjoint
struct FxRef {
  const int4 *p;
  int e, adj;
};
__device__ __forceinline__ FxRef fx_ref(const FxMat &f, int par, int h, int adj) {
  return {f.p + par * f.ps + h, __ldg(f.e + par * f.es + h), adj};
}

constexpr int FXM_BLOCK = 64;   // threads per block of the chain kernels
struct FxRing { int4 v[3][9][FXM_BLOCK]; };

__device__ __forceinline__ void fxm_fetch(FxRing &s, int slot, const FxRef &r, int Vh) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const size_t off = (size_t)(r.adj ? (k % 3) * 3 + k / 3 : k) * Vh;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(&s.v[slot][k][threadIdx.x])),
                 "l"(r.p + off)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void fxm_take(const FxRing &s, int slot, int adj, int4 (&u)[9]) {
  asm volatile("cp.async.wait_group 2;" ::: "memory");   // two younger fetches may be in flight
  const int sg = adj ? -1 : 1;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    u[k] = s.v[slot][k][threadIdx.x];
    u[k].z *= sg;
    u[k].w *= sg;
  }
}

// the right operand of a product with the sums of the three-product form
struct FxRight { int ch[9], cl[9], mh[9], ml[9], ph[9], pl[9]; };
__device__ __forceinline__ void fxm_right(const int4 (&u)[9], FxRight &r) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    r.ch[k] = u[k].x;
    r.cl[k] = u[k].y;
    r.mh[k] = u[k].z - u[k].x;
    r.ml[k] = u[k].w - u[k].y;
    r.ph[k] = u[k].x + u[k].z;
    r.pl[k] = u[k].y + u[k].w;
  }
}
// row i of A B
__device__ __forceinline__ void fxm_row(const int4 (&A)[9], int i, const FxRight &B, s64 (&q)[6]) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    FxSum k1 = {0, 0}, k2 = {0, 0}, k3 = {0, 0};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int4 a = A[3 * i + k];
      const int b = 3 * k + j;
      fx_mac(k1, a.x + a.z, a.y + a.w, B.ch[b], B.cl[b]);
      fx_mac(k2, a.x, a.y, B.mh[b], B.ml[b]);
      fx_mac(k3, a.z, a.w, B.ph[b], B.pl[b]);
    }
    q[2 * j] = (s64)((k1.H - k3.H) << 1) + ((s64)(k1.M - k3.M) >> 29);
    q[2 * j + 1] = (s64)((k1.H + k2.H) << 1) + ((s64)(k1.M + k2.M) >> 29);
  }
}

// a sum of chains: q[18] 2^(E-60)
struct FxSum9 { s64 q[18]; int E; };
__device__ __forceinline__ void fxm_zero(FxSum9 &s) {
#pragma unroll
  for (int k = 0; k < 18; k++) s.q[k] = 0;
  s.E = 4 * FX_ZERO;
}

// s += L (M R), or its adjoint; `right`: M R's right operand R
__device__ __forceinline__ void fxm_add(FxSum9 &s, const int4 (&Lm)[9], const FxRight &X, int e, bool adj) {
  if (e < FX_ZERO / 2) return;   // an operand is zero
  const int up = e > s.E ? min(e - s.E, 63) : 0, dn = e > s.E ? 0 : min(s.E - e, 63);
  s.E = max(e, s.E);
#pragma unroll
  for (int k = 0; k < 18; k++) s.q[k] >>= up;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    s64 q[6];
    fxm_row(Lm, i, X, q);
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const s64 re = q[2 * j] >> dn, im = q[2 * j + 1] >> dn;
      if (adj) {
        s.q[2 * (3 * j + i)] += re;
        s.q[2 * (3 * j + i) + 1] -= im;
      } else {
        s.q[2 * (3 * i + j)] += re;
        s.q[2 * (3 * i + j) + 1] += im;
      }
    }
  }
}

// operand of a chain as doubles
__device__ __forceinline__ M3<double> fxm_f64(const FxRef &r, int Vh) {
  M3<double> m;
  for (int k = 0; k < 9; k++) {
    const int4 w = r.p[(size_t)(r.adj ? (k % 3) * 3 + k / 3 : k) * Vh];
    double re = 0, im = 0;
    if (r.e == FX_SPECIAL) {
      re = __hiloint2double(w.x, w.y);
      im = __hiloint2double(w.z, w.w);
    } else if (r.e != FX_ZERO) {
      re = fx_double(((s64)w.x << 32) + 4 * (s64)w.y, r.e);
      im = fx_double(((s64)w.z << 32) + 4 * (s64)w.w, r.e);
    }
    m.e[k / 3][k % 3] = {re, r.adj ? -im : im};
  }
  return m;
}
// chains [c0, c1) of `get` added up in plain FP64 (an operand is not finite)
template <class Get>
static __device__ __noinline__ void fxm_chains_f64(const Get &get, int c0, int c1, int Vh, M3<double> *out) {
  M3<double> acc;
  for (int k = 0; k < 9; k++) acc.e[k / 3][k % 3] = {0.0, 0.0};
#pragma unroll 1
  for (int c = c0; c < c1; c++) {
    const M3<double> p = tnn<double>(fxm_f64(get(c, 2), Vh), tnn<double>(fxm_f64(get(c, 1), Vh), fxm_f64(get(c, 0), Vh)));
    tacc<double>(acc, get.adjoint(c) ? tadj<double>(p) : p, 1.0);
  }
  *out = acc;
}

// The chains [0, n) of `get`, the first n0 added into s0 and the others into
// s1.  get(c, role): operand R, M, L of chain c for role 0, 1, 2.  Returns
// true when an operand is not finite (the sums are then not to be used).
template <class Get>
__device__ __forceinline__ bool fxm_chains(const Get &get, int n, int n0, int Vh, FxRing &ring, FxSum9 &s0, FxSum9 &s1) {
  FxRef q[3];
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    q[k] = get(0, k);
    fxm_fetch(ring, k, q[k], Vh);
  }
  fxm_zero(s0);
  fxm_zero(s1);
#pragma unroll 1
  for (int c = 0; c < n; c++) {
    const int cn = c + 1 < n ? c + 1 : c;   // past the end: the last chain again, never used
    int4 u[9];
    FxRight X;
    int e = q[0].e;
    bad = bad || q[0].e == FX_SPECIAL || q[1].e == FX_SPECIAL || q[2].e == FX_SPECIAL;
    fxm_take(ring, 0, q[0].adj, u);
    fxm_right(u, X);
    q[0] = get(cn, 0);
    fxm_fetch(ring, 0, q[0], Vh);
    e += q[1].e + 3;
    fxm_take(ring, 1, q[1].adj, u);
    q[1] = get(cn, 1);
    fxm_fetch(ring, 1, q[1], Vh);
    int4 v[9];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      s64 w[6];
      fxm_row(u, i, X, w);
#pragma unroll
      for (int j = 0; j < 3; j++) {
        fxm_split(w[2 * j] + 2, v[3 * i + j].x, v[3 * i + j].y);
        fxm_split(w[2 * j + 1] + 2, v[3 * i + j].z, v[3 * i + j].w);
      }
    }
    fxm_right(v, X);
    e += q[2].e + 3;
    fxm_take(ring, 2, q[2].adj, u);
    q[2] = get(cn, 2);
    fxm_fetch(ring, 2, q[2], Vh);
    if (c < n0) fxm_add(s0, u, X, e, get.adjoint(c));
    else fxm_add(s1, u, X, e, get.adjoint(c));
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  return bad;
}

__device__ __forceinline__ double fxm_component(const FxSum9 &s, int k) {
  return s.E < FX_ZERO / 2 ? 0.0 : fx_double(s.q[k], s.E);
}

// ---- generalised staple (k_staple in FP64) ----
struct FxStapleChains {
  FxMat U, A;
  int par, h, xpnu, xpmu, xmnu, xmnupmu;
  __device__ __forceinline__ FxRef operator()(int c, int role) const {
    const int op = 1 - par;
    if (c == 0)  // U(x) [A(x+nu) U(x+mu)^dag]
      return role == 0 ? fx_ref(U, op, xpmu, 1) : role == 1 ? fx_ref(A, op, xpnu, 0) : fx_ref(U, par, h, 0);
    // U(x-nu)^dag [A(x-nu) U(x-nu+mu)]
    return role == 0 ? fx_ref(U, par, xmnupmu, 0) : role == 1 ? fx_ref(A, op, xmnu, 0) : fx_ref(U, op, xmnu, 1);
  }
  __device__ __forceinline__ bool adjoint(int) const { return false; }
};

// S -> sout (integers) when sout.p, fat += coef S when fat.p
static __global__ void __launch_bounds__(FXM_BLOCK) k_staple_fx(Geom g, int mu, int nu, FxMat U, FxMat A, MatF fat,
                                                               double coef, FxMat sout) {
  __shared__ FxRing ring;
  const int h = blockIdx.x * blockDim.x + threadIdx.x, par = blockIdx.y, Vh = g.Vh;
  if (h >= Vh) return;
  FxStapleChains get;
  get.U = U;
  get.A = A;
  get.par = par;
  get.h = h;
  get.xpnu = nbr(g, par, h, nu, 1);
  get.xpmu = nbr(g, par, h, mu, 1);
  get.xmnu = nbr(g, par, h, nu, -1);
  get.xmnupmu = nbr2(g, par, h, nu, -1, mu, 1);
  FxSum9 s, none;
  const bool bad = fxm_chains(get, 2, 2, Vh, ring, s, none);
  double2 v[9];
  int4 u[9];
  int e = FX_ZERO;
  if (bad) {
    M3<double> m;
    fxm_chains_f64(get, 0, 2, Vh, &m);
#pragma unroll
    for (int k = 0; k < 9; k++) v[k] = make_double2(m.e[k / 3][k % 3].re, m.e[k / 3][k % 3].im);
    if (sout.p) fxm_encode(v, u, e);
  } else {
    if (sout.p) {
      // normalised to |q| < 2^60: the exponents of a chain of three matrices
      // allow for 2^6 more than unitary ones reach, which a staple of a
      // staple would lose again
      u64 mag = 0;
#pragma unroll
      for (int k = 0; k < 18; k++) mag |= (u64)(s.q[k] ^ (s.q[k] >> 63));
      const int sh = __clzll((s64)mag) - 4;   // from -1 on; 60 for zeros and -1
      if (s.E >= FX_ZERO / 2 && mag) e = s.E - sh;
#pragma unroll
      for (int k = 0; k < 18; k++) s.q[k] = sh < 0 ? s.q[k] >> 1 : (s64)((u64)s.q[k] << sh);
#pragma unroll
      for (int k = 0; k < 9; k++) {
        fxm_split(s.q[2 * k] + 2, u[k].x, u[k].y);
        fxm_split(s.q[2 * k + 1] + 2, u[k].z, u[k].w);
      }
      s.E -= sh;
    }
    if (fat.p) {
#pragma unroll
      for (int k = 0; k < 9; k++) v[k] = make_double2(fxm_component(s, 2 * k), fxm_component(s, 2 * k + 1));
    }
  }
  if (sout.p) {
#pragma unroll
    for (int k = 0; k < 9; k++) sout.p[par * sout.ps + (size_t)k * Vh + h] = u[k];
    sout.e[par * sout.es + h] = e;
  }
  if (!fat.p) return;
  double2 *f = fat.p + par * fat.ps + h;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    double2 a = f[(size_t)k * Vh];
    a.x += coef * v[k].x;
    a.y += coef * v[k].y;
    f[(size_t)k * Vh] = a;
  }
}

// ---- reverse of one staple (k_staple_adj in FP64) ----
struct FxStapleAdjChains {
  FxMat U, A, K;
  int par, h, ymnu, ypnu, ypmu, ymmu, ymnupmu, ypnummu;
  __device__ __forceinline__ FxRef operator()(int c, int role) const {
    const int op = 1 - par;
    switch (c) {
    case 0:  // KA: U(y-nu+mu)^dag [K(y-nu) U(y-nu)]
      return role == 0 ? fx_ref(U, op, ymnu, 0) : role == 1 ? fx_ref(K, op, ymnu, 0) : fx_ref(U, par, ymnupmu, 1);
    case 1:  // KA: U(y+mu) [K(y+nu) U(y)^dag]
      return role == 0 ? fx_ref(U, par, h, 1) : role == 1 ? fx_ref(K, op, ypnu, 0) : fx_ref(U, op, ypmu, 0);
    case 2:  // KU: A(y+nu) [U(y+mu)^dag K(y)]
      return role == 0 ? fx_ref(K, par, h, 0) : role == 1 ? fx_ref(U, op, ypmu, 1) : fx_ref(A, op, ypnu, 0);
    case 3:  // KU: A(y-mu+nu)^dag [U(y-mu)^dag K(y-mu)^dag]
      return role == 0 ? fx_ref(K, op, ymmu, 1) : role == 1 ? fx_ref(U, op, ymmu, 1) : fx_ref(A, par, ypnummu, 1);
    case 4:  // KU: (A(y) [U(y+mu) K(y+nu)])^dag
      return role == 0 ? fx_ref(K, op, ypnu, 0) : role == 1 ? fx_ref(U, op, ypmu, 0) : fx_ref(A, par, h, 0);
    default:  // KU: (A(y-mu)^dag [U(y-mu) K(y+nu-mu)^dag])^dag
      return role == 0 ? fx_ref(K, par, ypnummu, 1) : role == 1 ? fx_ref(U, op, ymmu, 0) : fx_ref(A, op, ymmu, 1);
    }
  }
  __device__ __forceinline__ bool adjoint(int c) const { return c >= 4; }
};

// KA <- (init ? cinit init : KA) + f (its chains), KU += f (its chains); with
// kout.p set KA goes there as integers instead of to its FP64 field
static __global__ void __launch_bounds__(FXM_BLOCK) k_staple_adj_fx(Geom g, int mu, int nu, FxMat U, FxMat A, FxMat K,
                                                                   double f, MatF init, double cinit, MatF KA,
                                                                   FxMat kout, MatF KU) {
  __shared__ FxRing ring;
  const int h = blockIdx.x * blockDim.x + threadIdx.x, par = blockIdx.y, Vh = g.Vh;
  if (h >= Vh) return;
  FxStapleAdjChains get;
  get.U = U;
  get.A = A;
  get.K = K;
  get.par = par;
  get.h = h;
  get.ymnu = nbr(g, par, h, nu, -1);
  get.ypnu = nbr(g, par, h, nu, 1);
  get.ypmu = nbr(g, par, h, mu, 1);
  get.ymmu = nbr(g, par, h, mu, -1);
  get.ymnupmu = nbr2(g, par, h, nu, -1, mu, 1);
  get.ypnummu = nbr2(g, par, h, nu, 1, mu, -1);
  FxSum9 ka, ku;
  const bool bad = fxm_chains(get, 6, 2, Vh, ring, ka, ku);
  M3<double> ma, mu_;
  if (bad) {
    fxm_chains_f64(get, 0, 2, Vh, &ma);
    fxm_chains_f64(get, 2, 6, Vh, &mu_);
  }
  double2 v[9];
  const MatF src = init.p ? init : KA;
  const double c0 = init.p ? cinit : 1.0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 o = src.p[par * src.ps + (size_t)k * Vh + h];
    const double re = bad ? ma.e[k / 3][k % 3].re : fxm_component(ka, 2 * k);
    const double im = bad ? ma.e[k / 3][k % 3].im : fxm_component(ka, 2 * k + 1);
    v[k] = make_double2(c0 * o.x + f * re, c0 * o.y + f * im);
  }
  if (kout.p) {
    int4 u[9];
    int e;
    fxm_encode(v, u, e);
#pragma unroll
    for (int k = 0; k < 9; k++) kout.p[par * kout.ps + (size_t)k * Vh + h] = u[k];
    kout.e[par * kout.es + h] = e;
  } else {
#pragma unroll
    for (int k = 0; k < 9; k++) KA.p[par * KA.ps + (size_t)k * Vh + h] = v[k];
  }
  double2 *w = KU.p + par * KU.ps + h;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    double2 o = w[(size_t)k * Vh];
    const double re = bad ? mu_.e[k / 3][k % 3].re : fxm_component(ku, 2 * k);
    const double im = bad ? mu_.e[k / 3][k % 3].im : fxm_component(ku, 2 * k + 1);
    o.x += f * re;
    o.y += f * im;
    w[(size_t)k * Vh] = o;
  }
}

}  // namespace mks
