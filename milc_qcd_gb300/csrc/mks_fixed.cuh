// mks_fixed.cuh -- 64-bit lattice arithmetic on the integer pipe.
//
// GB300 runs FP64 at 2 lanes per clock and SM (measured 1.9 for fma.f64)
// and a 32 x 32 + 64-bit integer multiply-add at 64 (measured 59), so a
// product of two 57-bit integers built of three such multiply-adds is ten
// times cheaper than one FP64 fma.  The 3x3 products of D_eo are sums of
// bounded terms, which a fixed-point sum represents without any rounding of
// its own.  Its errors are the links' rounding (2^-57 of the largest of their
// kind), the vectors' cut to the largest component among a site's 16
// neighbours (downwards, by up to 2^-56 of it) and the product of the two low
// halves, which is left out (up to 2^-58 of the operands' bounds): bounds on
// the norm of a site's terms, not on each component.
// Measured against a complex128 restatement (which rounds too) on 8^4 ..
// 32^3x64: 1.8e-16 of the result's norm, where the FP64 sums had 3.8e-16.
//
// Format of a colour vector (a "block": one site's six real components):
// component = q 2^(e-60), |q| <= 2^60, one exponent e per site.  A block of
// zeros has e = FX_ZERO; a block that holds an infinity or a NaN has
// e = FX_SPECIAL and q holds the doubles' bits.
//
// For a product, q is cut as q = 16 (h 2^28 + l), |h| <= 2^28, |l| <= 2^27
// (l signed), and K = sum x y is kept as H = sum x_h y_h and
// M = sum (x_h y_l + x_l y_h), K = H 2^56 + M 2^28.  Complex products take
// three real ones: (a + ib)(c + id) has re = c(a+b) - b(c+d) and
// im = c(a+b) + a(d-c).  The sums of the halves are exact in 32 bits (no
// carries between h and l), so re and im are the exact integer sums, which
// stay below 2^63 for the 16 terms of D_eo (96 products of 2^56); the
// partial sums may wrap around, two's complement sums forgive that.
#pragma once
#include "mks_internal.cuh"

namespace mks {

constexpr int FX_ZERO = -(1 << 20), FX_SPECIAL = 1 << 20;

typedef unsigned long long u64;
typedef long long s64;

// a field of blocks of one parity
struct FxVec {
  longlong2 *q;  // [3][Vh]
  int *e;        // [Vh]
};

// |x| 2^(60-e) as an integer, rounded to nearest; |x| < 2^e, x finite
__device__ __forceinline__ s64 fx_scale(double x, int e) {
  const s64 b = __double_as_longlong(x);
  const int f = (int)(b >> 52) & 0x7ff, fe = f ? f : 1;
  u64 a = (((u64)b & 0xfffffffffffffull) | (f ? 0x10000000000000ull : 0)) << 7;
  const int d = e + 1022 - fe;  // >= 0
  if (d > 0) a = d < 62 ? (a + (1ull << (d - 1))) >> d : 0;
  return b < 0 ? -(s64)a : (s64)a;
}

// one site's components into a block
__device__ __forceinline__ void fx_encode(const double (&v)[6], s64 (&q)[6], int &e) {
  int ex = 0;
  s64 any = 0;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const s64 b = __double_as_longlong(v[k]);
    ex = max(ex, (int)(b >> 52) & 0x7ff);
    any |= b << 1;
  }
  if (ex == 0x7ff) {
    e = FX_SPECIAL;
#pragma unroll
    for (int k = 0; k < 6; k++) q[k] = __double_as_longlong(v[k]);
    return;
  }
  const int ev = max(ex, 1) - 1022;
#pragma unroll
  for (int k = 0; k < 6; k++) q[k] = fx_scale(v[k], ev);
  e = any ? ev : FX_ZERO;
}

// q 2^(e-60) as a double, rounded to nearest
__device__ __forceinline__ double fx_double(s64 q, int e) {
  u64 a = q < 0 ? 0 - (u64)q : (u64)q;
  if (a == 0) return 0.0;
  const int lz = __clzll((s64)a);
  int be = 1023 + 3 - lz + e;
  if (be < 1 || be > 2046) return scalbn((double)q, e - 60);
  a <<= lz;
  const u64 r = a + 0x400;   // round at bit 11
  const u64 m = r < a ? (1ull << 53) : r >> 11;   // a carry out of bit 63 leaves 2^53
  const u64 bits = ((u64)(be - 1) << 52) + m;
  return __longlong_as_double((s64)(bits | ((u64)q & 0x8000000000000000ull)));
}

__device__ __forceinline__ void fx_load(const FxVec &v, int h, int Vh, s64 (&q)[6]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const longlong2 w = __ldg(v.q + (size_t)c * Vh + h);
    q[2 * c] = w.x;
    q[2 * c + 1] = w.y;
  }
}
__device__ __forceinline__ void fx_store(const FxVec &v, int h, int Vh, const s64 (&q)[6], int e) {
#pragma unroll
  for (int c = 0; c < 3; c++) v.q[(size_t)c * Vh + h] = make_longlong2(q[2 * c], q[2 * c + 1]);
  v.e[h] = e;
}

// an aligned integer cut into halves
__device__ __forceinline__ void fx_split(s64 q, int &h, int &l) {
  const int lo = (int)q;
  h = (int)(q >> 32) + (int)((unsigned)lo >> 31);
  l = lo >> 4;
}

// sum of products, as (H, M)
struct FxSum { u64 H, M; };
__device__ __forceinline__ void fx_mad(u64 &s, int x, int y) {
  // written out: from s += (s64)x * y the compiler made a slower sequence
  // (8 sources, 24^3x48: 1.33 against 0.83 ms)
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s) : "r"(x), "r"(y));
}
__device__ __forceinline__ u64 fx_mul(int x, int y) {
  u64 s;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(s) : "r"(x), "r"(y));
  return s;
}
__device__ __forceinline__ void fx_mac(FxSum &s, int xh, int xl, int yh, int yl) {
  fx_mad(s.H, xh, yh);
  fx_mad(s.M, xh, yl);
  fx_mad(s.M, xl, yh);
}

// a neighbour's block aligned to exponent E, with the sums and differences
// of the three-product form; SGN = +1: m = d - c, SGN = -1: m = c - d
struct FxOperand { int ch[3], cl[3], mh[3], ml[3], ph[3], pl[3]; };
template <int SGN>
__device__ __forceinline__ void fx_operand(const s64 (&q)[6], int shift, FxOperand &o) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    int dh, dl;
    fx_split(q[2 * j] >> shift, o.ch[j], o.cl[j]);
    fx_split(q[2 * j + 1] >> shift, dh, dl);
    o.mh[j] = SGN > 0 ? dh - o.ch[j] : o.ch[j] - dh;
    o.ml[j] = SGN > 0 ? dl - o.cl[j] : o.cl[j] - dl;
    o.ph[j] = o.ch[j] + dh;
    o.pl[j] = o.cl[j] + dl;
  }
}

// Links: an entry's halves {a_h, a_l, b_h, b_l} (a + ib), value
// (h 2^28 + l) 2^(EL-56), one exponent EL for the slot's fat links and one for
// its Naik links.  A link keeps 2^-57 of the largest of its kind, so the form
// is for links of one size: within FX_SPREAD bits, measured by a matrix's
// largest component, every link keeps the 53 bits of a double.  Smeared links
// lie within 0.2 bits of each other on smooth fields (exp(i 0.3 H)) and within
// 1.7 where the thin links are random; a slot that does not fit is done in
// plain FP64 (k_dslash_raw).
constexpr int FX_SPREAD = 4;

// Components of a vector share an exponent, so a component far below the
// others is as good as a matrix that mixes them makes its part in a result:
// an entry of size 2^-k leaves 56 - k bits.  Links are uneven, and left to
// FP64, when
// - a matrix has an entry more than FX_ENTRY bits, or a real or imaginary part
//   more than FX_PART bits, below its largest component: free, diagonal, real
//   or block matrices, which do not mix some components at all; or
// - one entry in 1024 lies more than FX_ENTRIES bits below, or one part more
//   than FX_PARTS: fields close to such ones, whose typical small entry is
//   under 2^-7 (a generic field has one such entry in 10^7, one such part in
//   10^6).
// Least entry and least part of 262,144 smeared links: 13 and 25 bits below
// for thin links exp(i 0.3 H), 13 and 29 for random ones, 17.5 and 29 for
// exp(i 0.05 H); four times the links bring an entry one bit lower, a part two.
constexpr int FX_ENTRY = 28, FX_PART = 48, FX_ENTRIES = 12, FX_PARTS = 20;
constexpr u64 FX_INF = 0x7ff0000000000000ull;
struct FxShape {
  u64 top;           // bits of the largest component (a NaN does not count)
  bool bad, uneven;  // a component is not finite; the first rule
  int ents, parts;   // entries and parts of the second
  __device__ __forceinline__ FxShape(const double2 (&v)[9]) : top(0), bad(false), uneven(false), ents(0), parts(0) {
    int e[9], p[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
      u64 x = (u64)__double_as_longlong(v[k].x) & ~(1ull << 63), y = (u64)__double_as_longlong(v[k].y) & ~(1ull << 63);
      bad = bad || x >= FX_INF || y >= FX_INF;
      if (x > FX_INF) x = 0;
      if (y > FX_INF) y = 0;
      const u64 hi = x > y ? x : y, lo = x > y ? y : x;
      top = hi > top ? hi : top;
      e[k] = (int)(hi >> 52);
      p[k] = (int)(lo >> 52);
    }
    if (top == 0) return;
    const int t = (int)(top >> 52);
#pragma unroll
    for (int k = 0; k < 9; k++) {
      uneven = uneven || t - e[k] > FX_ENTRY || t - p[k] > FX_PART;
      ents += t - e[k] > FX_ENTRIES;
      parts += t - p[k] > FX_PARTS;
    }
  }
};
// counts of a field's matrices, in global memory and zero at first
struct FxUneven {
  unsigned long long uneven, ents, parts;
  // over `mats` matrices
  bool any(size_t mats) const { return uneven || 1024 * ents > 9 * mats || 1024 * parts > 9 * mats; }
};
// adds a warp's counts (all 32 lanes call)
__device__ __forceinline__ void fx_uneven_add(FxUneven *u, bool uneven, int ents, int parts) {
  uneven = __any_sync(0xffffffffu, uneven);
  ents = __reduce_add_sync(0xffffffffu, ents);
  parts = __reduce_add_sync(0xffffffffu, parts);
  if ((threadIdx.x & 31) != 0) return;
  if (uneven) atomicMax(&u->uneven, 1ull);
  if (ents) atomicAdd(&u->ents, (unsigned long long)ents);
  if (parts) atomicAdd(&u->parts, (unsigned long long)parts);
}
struct FxLinks {
  const int4 *p;  // [par][dir][9][Vh]
};

struct FxAcc { FxSum k1[3], k2[3], k3[3]; };

// acc += U v (ADJ = false) or acc -= U^dag v (ADJ = true) for NB sources
template <bool ADJ, int NB>
__device__ __forceinline__ void fx_mv(const FxLinks &U, int par, int dir, int h, int Vh, const FxOperand (&o)[NB],
                                      FxAcc (&acc)[NB]) {
  const int4 *b = U.p + ((size_t)(par * 4 + dir) * 9) * Vh + h;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int4 u = __ldcs(b + (size_t)(ADJ ? 3 * j + i : 3 * i + j) * Vh);
      const int sh = ADJ ? u.z - u.x : u.x + u.z, sl = ADJ ? u.w - u.y : u.y + u.w;
#pragma unroll
      for (int s = 0; s < NB; s++) {
        fx_mac(acc[s].k1[i], sh, sl, o[s].ch[j], o[s].cl[j]);
        fx_mac(acc[s].k2[i], u.x, u.y, o[s].mh[j], o[s].ml[j]);
        fx_mac(acc[s].k3[i], u.z, u.w, o[s].ph[j], o[s].pl[j]);
      }
    }
}

}  // namespace mks
