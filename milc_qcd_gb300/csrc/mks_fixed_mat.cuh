// mks_fixed_mat.cuh -- 3x3 products of FP64 link fields in integer arithmetic,
// and the staple kernels of the link construction and the fermion force on
// them (see mks_fixed.cuh for why: an fma.f64 costs 30 integer multiply-adds).
//
// A matrix is nine complex entries as integers with one exponent: component =
// q 2^(e-60), |q| <= 2^60, cut as q = h 2^32 + l, |h| <= 2^28, |l| < 2^31, stored
// as int4 {re h, re l, im h, im l} (the 16 bytes of a double2) in tiles of 32
// sites, so that an entry is a constant distance from the last.  A product is
// K = H 2^64 + M 2^32 by three multiply-adds per real product (the low halves'
// product, 2^-58 of the operands' bounds, is left out); six terms of 2^56 and
// twelve of 2^59 leave room in 64 bits.  Complex products take four real ones:
// with the three of D_eo the sums of halves, and the narrower l that they
// need, cost more instructions than the multiply-adds they save (the integer
// ALU, half as fast as a multiply-add's issue rate would have it, is what
// bounds these kernels).  The first product of a chain keeps K 2^-64, one add
// of M's high word; the last K 2^-61.  A matrix of zeros has e = FX_ZERO, one
// that holds an infinity or a NaN e = FX_SPECIAL and the doubles' bits; a site
// that meets one is done in plain FP64.  One exponent per matrix bounds a
// product's error by its norm, not entry by entry; links with entries far below
// their largest (FxUneven) are left to the FP64 kernels.
//
// A staple term is a chain L (M R) of three matrices, its adjoint six chains;
// the chains run in a loop whose operands are fetched three ahead into shared
// memory by cp.async (a fetch in flight holds no registers, of which the
// products take up to 200); the FP64 fields that the result is added to come
// the same way behind the last chain.
#pragma once
#include "mks_fixed.cuh"
#include "mks_su3.cuh"

namespace mks {

// a field of nd = 4 matrices per site (a direction each) or nd = 1 (every
// direction uses it), or one direction of it: entry k of site h at
// p[par ps + (9 (h / 32) + k) 32 + h % 32]
struct FxMat {
  int4 *p;
  int *e;      // [par es + h]
  size_t ps, es;
  int nd;
  __host__ __device__ static size_t sites(size_t Vh) { return (Vh + 31) / 32 * 32; }
  __device__ __forceinline__ int4 *at(int par, int h) const {
    return p + par * ps + (size_t)(h >> 5) * 288 + (h & 31);
  }
};
__device__ __forceinline__ FxMat fx_link_dir(const FxMat &f, int dir, size_t Vh) {
  const size_t d = f.nd == 4 ? dir : 0;
  return {f.p + d * 9 * FxMat::sites(Vh), f.e + d * Vh, f.ps, f.es, 1};
}

// l never is -2^31, which has no negative (one unit of 2^-60 off instead)
__device__ __forceinline__ void fxm_split(s64 q, int &h, int &l) {
  const int lo = (int)q;
  h = (int)(q >> 32) + (int)((unsigned)lo >> 31);
  l = max(lo, -0x7fffffff);
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
    fxm_split(fx_scale(v[k].x, e), u[k].x, u[k].y);
    fxm_split(fx_scale(v[k].y, e), u[k].z, u[k].w);
  }
  if (!any) e = FX_ZERO;
}

// [2][4][9][Vh] doubles -> integers; *uneven (where given) counts the matrices
// with entries that one exponent does not hold
static __global__ void __launch_bounds__(128) k_links_to_fxm(const double2 *__restrict__ src, FxMat dst, int Vh,
                                                            FxUneven *uneven) {
  const int h0 = blockIdx.x * blockDim.x + threadIdx.x, par = blockIdx.y, mu = blockIdx.z;
  const int h = h0 < Vh ? h0 : Vh - 1;   // threads past the last site follow it into the warp's counts
  const double2 *s = src + (size_t)(par * 4 + mu) * 9 * Vh + h;
  double2 v[9];
  int4 u[9];
  int e;
#pragma unroll
  for (int k = 0; k < 9; k++) v[k] = s[(size_t)k * Vh];
  fxm_encode(v, u, e);
  if (uneven) {
    const FxShape f(v);
    fx_uneven_add(uneven, f.uneven, h0 < Vh ? f.ents : 0, h0 < Vh ? f.parts : 0);
  }
  if (h0 >= Vh) return;
  int4 *d = fx_link_dir(dst, mu, Vh).at(par, h);
#pragma unroll
  for (int k = 0; k < 9; k++) d[32 * k] = u[k];
  dst.e[(size_t)(par * 4 + mu) * Vh + h] = e;
}

// Runs `once`, which takes its integer fields from the workspace before it
// launches anything that changes a result; true when the caller is to do
// without: the links are uneven, or there was no memory (then it is not to ask
// again on this lattice).  *rc: what `once` returned.
constexpr int FXM_UNEVEN = 1;
template <class F> inline bool fxm_refused(const F &once, int *rc) {
  Context &c = ctx();
  if (c.fxm_off) return true;
  {
    FxBusy busy;
    *rc = once();
  }
  if (*rc == FXM_UNEVEN) {
    *rc = MKS_OK;
    return true;
  }
  if (*rc != MKS_ERR_NOMEM) return false;
  c.fxm_off = true;
  ws_smear_free();
  return true;
}

// workspace of `mats` (1 or 4) integer matrices per site under `name`
inline int ws_fxm(const char *name, int mats, FxMat *f) {
  const size_t Vh = ctx().Vh;
  f->ps = (size_t)mats * 9 * FxMat::sites(Vh);
  f->es = (size_t)mats * Vh;
  f->nd = mats;
  MKS_TRY(ws(std::string("smear_") + name + "_p", 2 * f->ps * sizeof(int4), (void **)&f->p));
  return ws(std::string("smear_") + name + "_e", (size_t)mats * 2 * Vh * sizeof(int), (void **)&f->e);
}

// a field of matrices [2][4][9][Vh] as integers in the workspace
inline int ws_mats_fxm(const char *name, int family, const double2 *mats, FxMat *f, FxUneven *uneven = nullptr) {
  Context &c = ctx();
  MKS_TRY(ws_fxm(name, 4, f));
  timing_begin(family);
  k_links_to_fxm<<<dim3(grid_for(c.Vh, 128), 2, 4), 128, 0, c.stream>>>(mats, *f, (int)c.Vh, uneven);
  timing_end(family);
  MKS_CUDA(cudaGetLastError());
  return MKS_OK;
}
// Links that chains or paths are built of; FXM_UNEVEN when one exponent per
// matrix does not hold them.  (A field between two links, the outer products
// of the force, need not be looked at: even links mix its entries.)
inline int ws_links_fxm(int family, const double2 *links, FxMat *f) {
  Context &c = ctx();
  FxUneven *count, n;
  MKS_TRY(ws("fxm_uneven", sizeof n, (void **)&count));
  MKS_CUDA(cudaMemsetAsync(count, 0, sizeof n, c.stream));
  MKS_TRY(ws_mats_fxm("links", family, links, f, count));
  MKS_CUDA(cudaMemcpyAsync(&n, count, sizeof n, cudaMemcpyDeviceToHost, c.stream));
  MKS_CUDA(cudaStreamSynchronize(c.stream));
  return n.any((size_t)8 * c.Vh) ? FXM_UNEVEN : MKS_OK;
}

// an operand of a chain: a site's matrix, as it is or its adjoint
struct FxRef {
  const int4 *p;
  int e, adj;
};
__device__ __forceinline__ FxRef fx_ref(const FxMat &f, int par, int h, int adj) {
  return {f.at(par, h), __ldg(f.e + par * f.es + h), adj};
}

constexpr int FXM_BLOCK = 64;   // threads per block of the chain kernels
struct FxRing { int4 v[3][9][FXM_BLOCK]; };

__device__ __forceinline__ void fxm_cp(FxRing &s, int slot, int k, const void *p) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(&s.v[slot][k][threadIdx.x])),
               "l"(p)
               : "memory");
}
__device__ __forceinline__ void fxm_fetch(FxRing &s, int slot, const FxRef &r) {
#pragma unroll
  for (int k = 0; k < 9; k++) fxm_cp(s, slot, k, r.p + 32 * k);
  asm volatile("cp.async.commit_group;" ::: "memory");
}
// a matrix of an FP64 field behind the chains (p = nullptr: nothing)
__device__ __forceinline__ void fxm_fetch_f64(FxRing &s, int slot, const double2 *p, int Vh) {
  if (p)
#pragma unroll
    for (int k = 0; k < 9; k++) fxm_cp(s, slot, k, p + (size_t)k * Vh);
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void fxm_take(const FxRing &s, int slot, int adj, int4 (&u)[9]) {
  asm volatile("cp.async.wait_group 2;" ::: "memory");   // two younger fetches may be in flight
  const int sg = adj ? -1 : 1;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    u[k] = s.v[slot][adj ? (k % 3) * 3 + k / 3 : k][threadIdx.x];
    u[k].z *= sg;
    u[k].w *= sg;
  }
}

// element (i, j) of A B as (H, M)
__device__ __forceinline__ void fxm_element(const int4 (&A)[9], int i, const int4 (&B)[9], int j, FxSum &re, FxSum &im) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int4 a = A[3 * i + k], b = B[3 * k + j];
    if (k == 0) {
      re.H = fx_mul(a.x, b.x);
      re.M = fx_mul(a.x, b.y);
      fx_mad(re.M, a.y, b.x);
      im.H = fx_mul(a.x, b.z);
      im.M = fx_mul(a.x, b.w);
      fx_mad(im.M, a.y, b.z);
    } else {
      fx_mac(re, a.x, a.y, b.x, b.y);
      fx_mac(im, a.x, a.y, b.z, b.w);
    }
    fx_mac(re, -a.z, -a.w, b.z, b.w);
    fx_mac(im, a.z, a.w, b.x, b.y);
  }
}

// a sum of chains: q[18] 2^(E-60)
struct FxSum9 { s64 q[18]; int E; };
__device__ __forceinline__ void fxm_zero(FxSum9 &s) {
#pragma unroll
  for (int k = 0; k < 18; k++) s.q[k] = 0;
  s.E = 4 * FX_ZERO;
}
// exponent of a chain L (M R) of operands with these exponents; one with a
// zero among them does not count
__device__ __forceinline__ int fxm_exponent(int er, int em, int el) {
  const int e = er + em + el + 5;
  return e < FX_ZERO / 2 ? 4 * FX_ZERO : e;
}

// s += L X, or its adjoint, of exponent e <= s.E
__device__ __forceinline__ void fxm_add(FxSum9 &s, const int4 (&Lm)[9], const int4 (&X)[9], int e, bool adj) {
  const int dn = min(s.E - e, 63);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      FxSum re, im;
      fxm_element(Lm, i, X, j, re, im);
      const s64 qr = ((s64)(re.H << 3) + ((s64)re.M >> 29)) >> dn;
      const s64 qi = ((s64)(im.H << 3) + ((s64)im.M >> 29)) >> dn;
      if (adj) {
        s.q[2 * (3 * j + i)] += qr;
        s.q[2 * (3 * j + i) + 1] -= qi;
      } else {
        s.q[2 * (3 * i + j)] += qr;
        s.q[2 * (3 * i + j) + 1] += qi;
      }
    }
}

// operand of a chain as doubles
__device__ __forceinline__ M3<double> fxm_f64(const FxRef &r) {
  M3<double> m;
  for (int k = 0; k < 9; k++) {
    const int4 w = r.p[32 * (r.adj ? (k % 3) * 3 + k / 3 : k)];
    double re = 0, im = 0;
    if (r.e == FX_SPECIAL) {
      re = __hiloint2double(w.x, w.y);
      im = __hiloint2double(w.z, w.w);
    } else if (r.e != FX_ZERO) {
      re = fx_double(((s64)w.x << 32) + w.y, r.e);
      im = fx_double(((s64)w.z << 32) + w.w, r.e);
    }
    m.e[k / 3][k % 3] = {re, r.adj ? -im : im};
  }
  return m;
}
// chains [c0, c1) of `get` added up in plain FP64 (an operand is not finite)
template <class Get>
static __device__ __noinline__ void fxm_chains_f64(const Get &get, int c0, int c1, M3<double> *out) {
  M3<double> acc;
  for (int k = 0; k < 9; k++) acc.e[k / 3][k % 3] = {0.0, 0.0};
#pragma unroll 1
  for (int c = c0; c < c1; c++) {
    const M3<double> p = tnn<double>(fxm_f64(get(c, 2)), tnn<double>(fxm_f64(get(c, 1)), fxm_f64(get(c, 0))));
    tacc<double>(acc, get.adjoint(c) ? tadj<double>(p) : p, 1.0);
  }
  *out = acc;
}

// The chains [0, n) of `get`, the first n0 added into s0 and the others into
// s1.  get(c, role): operand R, M, L of chain c for role 0, 1, 2.  On return
// the FP64 matrices at t0 and t1 (where given) are in the ring's slots 0 and
// 1.  True when an operand is not finite (the sums are then not to be used).
template <int n, int n0, class Get>
__device__ __forceinline__ bool fxm_chains(const Get &get, int Vh, FxRing &ring, FxSum9 &s0, FxSum9 &s1,
                                           const double2 *t0, const double2 *t1) {
  FxRef q[3];
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    q[k] = get(0, k);
    fxm_fetch(ring, k, q[k]);
  }
  fxm_zero(s0);
  fxm_zero(s1);
#pragma unroll
  for (int c = 0; c < n; c++) {
    int &E = c < n0 ? s0.E : s1.E;
    E = max(E, fxm_exponent(get(c, 0).e, get(c, 1).e, get(c, 2).e));
  }
#pragma unroll 1
  for (int c = 0; c < n; c++) {
    const bool last = c + 1 == n;
    int4 u[9], X[9], v[9];
    const int e = fxm_exponent(q[0].e, q[1].e, q[2].e);
    bad = bad || q[0].e == FX_SPECIAL || q[1].e == FX_SPECIAL || q[2].e == FX_SPECIAL;
    fxm_take(ring, 0, q[0].adj, X);
    if (!last) {
      q[0] = get(c + 1, 0);
      fxm_fetch(ring, 0, q[0]);
    } else {
      fxm_fetch_f64(ring, 0, t0, Vh);
    }
    fxm_take(ring, 1, q[1].adj, u);
    if (!last) {
      q[1] = get(c + 1, 1);
      fxm_fetch(ring, 1, q[1]);
    } else {
      fxm_fetch_f64(ring, 1, t1, Vh);
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        FxSum re, im;
        fxm_element(u, i, X, j, re, im);
        fxm_split((s64)re.H + ((s64)re.M >> 32), v[3 * i + j].x, v[3 * i + j].y);
        fxm_split((s64)im.H + ((s64)im.M >> 32), v[3 * i + j].z, v[3 * i + j].w);
      }
    fxm_take(ring, 2, q[2].adj, u);
    const bool adj = get.adjoint(c);
    if (!last) {
      q[2] = get(c + 1, 2);
      fxm_fetch(ring, 2, q[2]);
    } else {
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (n0 == n || c < n0) fxm_add(s0, u, v, e, adj);
    else fxm_add(s1, u, v, e, adj);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  return bad;
}
__device__ __forceinline__ double2 fxm_tail(const FxRing &ring, int slot, int k) {
  return *reinterpret_cast<const double2 *>(&ring.v[slot][k][threadIdx.x]);
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

// S -> sout (integers) when sout.p, fat += coef S when fat.p; mu = mu0 +
// blockIdx.z, nu = mu + k
static __global__ void __launch_bounds__(FXM_BLOCK, 5) k_staple_fx(Geom g, int mu0, int k1, FxMat L, FxMat Af,
                                                                  MatD<double> fatf, double coef, FxMat soutf) {
  __shared__ FxRing ring;
  const int h = blockIdx.x * blockDim.x + threadIdx.x, par = blockIdx.y, Vh = g.Vh;
  if (h >= Vh) return;
  const int mu = mu0 + blockIdx.z, nu = (mu + k1) & 3;
  const FxMat U = fx_link_dir(L, nu, Vh), A = fx_link_dir(Af, mu, Vh), sout = fx_link_dir(soutf, mu, Vh);
  const MatF fat = fatf.at(mu);
  const bool keep = soutf.p != nullptr;
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
  double2 *f = fatf.p ? fat.p + par * fat.ps + h : nullptr;
  const bool bad = fxm_chains<2, 2>(get, Vh, ring, s, none, f, nullptr);
  double2 v[9];
  int4 u[9];
  int e = FX_ZERO;
  if (bad) {
    M3<double> m;
    fxm_chains_f64(get, 0, 2, &m);
#pragma unroll
    for (int k = 0; k < 9; k++) v[k] = make_double2(m.e[k / 3][k % 3].re, m.e[k / 3][k % 3].im);
    if (keep) fxm_encode(v, u, e);
  } else {
    if (keep) {
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
        fxm_split(s.q[2 * k], u[k].x, u[k].y);
        fxm_split(s.q[2 * k + 1], u[k].z, u[k].w);
      }
      s.E -= sh;
    }
    if (f) {
#pragma unroll
      for (int k = 0; k < 9; k++) v[k] = make_double2(fxm_component(s, 2 * k), fxm_component(s, 2 * k + 1));
    }
  }
  if (keep) {
    int4 *d = sout.at(par, h);
#pragma unroll
    for (int k = 0; k < 9; k++) d[32 * k] = u[k];
    sout.e[par * sout.es + h] = e;
  }
  if (!f) return;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    double2 a = fxm_tail(ring, 0, k);
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

// KA <- (init ? cinit init : KA) + f (its chains), KU_nu += f (its chains);
// with kout.p set KA goes there as integers instead of to its FP64 field
static __global__ void __launch_bounds__(FXM_BLOCK, 4) k_staple_adj_fx(Geom g, int mu0, int k1, FxMat L, FxMat Af,
                                                                      FxMat Kf, double f, MatD<double> initf,
                                                                      double cinit, MatD<double> KAf, FxMat koutf,
                                                                      MatD<double> KUf) {
  __shared__ FxRing ring;
  const int h = blockIdx.x * blockDim.x + threadIdx.x, par = blockIdx.y, Vh = g.Vh;
  if (h >= Vh) return;
  const int mu = mu0 + blockIdx.z, nu = (mu + k1) & 3;
  const FxMat U = fx_link_dir(L, nu, Vh), A = fx_link_dir(Af, mu, Vh), K = fx_link_dir(Kf, mu, Vh);
  const FxMat kout = fx_link_dir(koutf, mu, Vh);
  const MatF KA = KAf.at(mu), KU = KUf.at(nu), init = initf.at(mu);
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
  const MatF src = initf.p ? init : KA;
  double2 *w = KU.p + par * KU.ps + h;
  const bool bad = fxm_chains<6, 2>(get, Vh, ring, ka, ku, src.p + par * src.ps + h, w);
  M3<double> ma, mu_;
  if (bad) {
    fxm_chains_f64(get, 0, 2, &ma);
    fxm_chains_f64(get, 2, 6, &mu_);
  }
  double2 v[9];
  const double c0 = initf.p ? cinit : 1.0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 o = fxm_tail(ring, 0, k);
    const double re = bad ? ma.e[k / 3][k % 3].re : fxm_component(ka, 2 * k);
    const double im = bad ? ma.e[k / 3][k % 3].im : fxm_component(ka, 2 * k + 1);
    v[k] = make_double2(c0 * o.x + f * re, c0 * o.y + f * im);
  }
  if (koutf.p) {
    int4 u[9];
    int e;
    fxm_encode(v, u, e);
#pragma unroll
    for (int k = 0; k < 9; k++) kout.at(par, h)[32 * k] = u[k];
    kout.e[par * kout.es + h] = e;
  } else {
#pragma unroll
    for (int k = 0; k < 9; k++) KA.p[par * KA.ps + (size_t)k * Vh + h] = v[k];
  }
#pragma unroll
  for (int k = 0; k < 9; k++) {
    double2 o = fxm_tail(ring, 1, k);
    const double re = bad ? mu_.e[k / 3][k % 3].re : fxm_component(ku, 2 * k);
    const double im = bad ? mu_.e[k / 3][k % 3].im : fxm_component(ku, 2 * k + 1);
    o.x += f * re;
    o.y += f * im;
    w[(size_t)k * Vh] = o;
  }
}

// ---- paths of links (gauge force and action in FP64) ----
// a running product as integers, normalised after each step so that a path of
// five links keeps the bits of one
struct FxPath { int4 u[9]; int e; };

// site (par, h)'s matrix of one direction, as it is or its adjoint
__device__ __forceinline__ void fxm_load(const FxMat &f, int par, int h, bool adj, int4 (&u)[9], int &e) {
  const int4 *p = f.at(par, h);
  const int sg = adj ? -1 : 1;
  e = __ldg(f.e + par * f.es + h);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    u[k] = __ldg(p + 32 * (adj ? (k % 3) * 3 + k / 3 : k));
    u[k].z *= sg;
    u[k].w *= sg;
  }
}
// P <- P L
__device__ __forceinline__ void fxm_step(FxPath &P, const int4 (&Lm)[9], int el) {
  s64 q[18];
  u64 mag = 0;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      FxSum re, im;
      fxm_element(P.u, i, Lm, j, re, im);
      const s64 a = (s64)(re.H << 3) + ((s64)re.M >> 29), b = (s64)(im.H << 3) + ((s64)im.M >> 29);
      q[2 * (3 * i + j)] = a;
      q[2 * (3 * i + j) + 1] = b;
      mag |= (u64)(a ^ (a >> 63)) | (u64)(b ^ (b >> 63));
    }
  const int sh = __clzll((s64)mag) - 4;   // from -2 on; 60 for zeros and -1
  P.e += el + 1 - sh;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const s64 a = sh < 0 ? q[2 * k] >> -sh : (s64)((u64)q[2 * k] << sh);
    const s64 b = sh < 0 ? q[2 * k + 1] >> -sh : (s64)((u64)q[2 * k + 1] << sh);
    fxm_split(a, P.u[k].x, P.u[k].y);
    fxm_split(b, P.u[k].z, P.u[k].w);
  }
}
// Re tr(P L)
__device__ __forceinline__ double fxm_trace(const FxPath &P, const int4 (&Lm)[9], int el) {
  s64 t = 0;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    FxSum re = {0, 0};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int4 a = P.u[3 * i + k], b = Lm[3 * k + i];
      fx_mac(re, a.x, a.y, b.x, b.y);
      fx_mac(re, -a.z, -a.w, b.z, b.w);
    }
    t += (s64)(re.H << 1) + ((s64)re.M >> 31);
  }
  const int e = P.e + el + 3;   // t 2^(P.e + el - 57)
  return e < FX_ZERO / 2 ? 0.0 : fx_double(t, e);
}

}  // namespace mks
