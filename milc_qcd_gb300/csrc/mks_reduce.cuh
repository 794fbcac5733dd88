// mks_reduce.cuh -- deterministic in-kernel FP64 reductions.
//
// Every thread contributes NSUM doubles per source.  A block reduces them by
// warp sums (keeping the G thread groups of a site apart) and shared memory,
// and adds its totals to integer accumulators in global memory; integer sums
// do not depend on the order, so results do not depend on block scheduling.
// The block that arrives last reads them and runs a "finisher" that updates
// solver scalars on the device, so the host never waits on a reduction
// inside an iteration.
#pragma once
#include "mks_internal.cuh"

namespace mks {

// x as |x| = m 2^(f - 1075), f >= 1; 0x7ff for an infinity or a NaN
__device__ __forceinline__ void red_split(double x, int &f, unsigned long long &m) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  f = (int)(b >> 52) & 0x7ff;
  m = (b & 0xfffffffffffffull) | (f ? 1ull << 52 : 0);
  if (f == 0) f = 1;
}
// sign q 2^(f - 1075) as a double, rounded to nearest (integer arithmetic but
// for results out of the normal range)
__device__ __forceinline__ double red_double(bool neg, unsigned long long q, int f) {
  if (q == 0) return 0.0;
  const int lz = __clzll((long long)q), be = f + 11 - lz;
  if (be < 1 || be > 2045) {
    const double d = scalbn((double)q, f - 1075);
    return neg ? -d : d;
  }
  const unsigned long long a = q << lz, r = a + 0x400;   // round at bit 11
  const unsigned long long m = r < a ? 1ull << 53 : r >> 11;
  return __longlong_as_double((long long)((((unsigned long long)(be - 1) << 52) + m) | (neg ? 1ull << 63 : 0)));
}

// Sum of x over the 32 lanes of a warp, on every lane.  The lanes' values are
// aligned to the largest exponent (to 53 bits: an FP64 add rounds no later)
// and added by two integer warp sums.  Five FP64 adds by shuffles hold the
// FP64 pipe for 64 clocks each, in every warp of the grid: 1296 blocks of 256
// threads with three sums took 8.7 us for this alone.
__device__ __forceinline__ double warp_sum(double x) {
  int f;
  unsigned long long m;
  red_split(x, f, m);
  const int F = (int)__reduce_max_sync(0xffffffffu, (unsigned)f);
  if (F == 0x7ff) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  }
  const int d = F - f;
  if (d > 0) m = d < 55 ? (m + (1ull << (d - 1))) >> d : 0;
  const long long q = x < 0 ? -(long long)m : (long long)m;
  const long long t = ((long long)__reduce_add_sync(0xffffffffu, (int)(q >> 27)) << 27) +
                      __reduce_add_sync(0xffffffffu, (unsigned)q & 0x7ffffffu);
  return red_double(t < 0, t < 0 ? 0 - (unsigned long long)t : (unsigned long long)t, F);
}

// Block-wide reduction of vals[NV] (per thread) where thread t's values
// belong to slot (t % G)*NB + s for s < NB.  Result: tot[slot*NSUM + k] in
// shared memory on return (valid after the trailing __syncthreads), for
// slots < nslots = G*NB.  smem must hold (blockDim/32) * G*NB*NSUM doubles.
// The per-thread values and the warp-level shuffles use T (float in the
// sloppy solvers: GB300 runs FP64 at a small fraction of the FP32 rate, so
// per-site products and the first 32-way sums stay in FP32); from the warp
// totals on, everything is FP64.
template <typename T, int NB, int NSUM>
__device__ __forceinline__ void block_reduce_grouped(T (&v)[NB][NSUM], int G, double *smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int nslots = G * NB;
#pragma unroll
  for (int s = 0; s < NB; s++)
#pragma unroll
    for (int k = 0; k < NSUM; k++) {
      T x = v[s][k];
      for (int o = 16; o >= G; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      v[s][k] = x;
    }
  if (lane < G) {
#pragma unroll
    for (int s = 0; s < NB; s++)
#pragma unroll
      for (int k = 0; k < NSUM; k++) smem[(warp * nslots + lane * NB + s) * NSUM + k] = (double)v[s][k];
  }
  __syncthreads();
  // sum over warps, in warp order
  for (int i = threadIdx.x; i < nslots * NSUM; i += blockDim.x) {
    double acc = 0;
    for (int w = 0; w < nwarps; w++) acc += smem[w * nslots * NSUM + i];
    smem[nwarps * nslots * NSUM + i] = acc;
  }
  __syncthreads();
}

// ---- sums over the grid ----
// A sum lives in RED_LIMBS 64-bit integers of global memory: limb k counts
// units of 2^(32k - 1074), so a double is three signed 32-bit pieces, and
// blocks add theirs with integer atomics, in any order with the same result
// (up to 2^31 blocks).  The last limb flags infinities and NaN.  One block
// that arrives last reads the limbs; rows summed by a tree in two levels of
// last-to-arrive blocks took 5.3 us more (1296 blocks, three sums).  The limbs
// hold the sum exactly; what is read is its part down to 2^-63 of the largest
// block total (limbs are signed, so the highest may cancel), rounded to FP64.
// Carrying through all limbs first, for the whole of a sum that cancels
// further, costs every reducing kernel registers (k_site with OpUpdate<float>
// 32 to 40; 8-source CG on 32^3x64 368.1 to 370.6 ms).
__device__ __forceinline__ void red_add(unsigned long long *limbs, double x) {
  int f;
  unsigned long long m;
  red_split(x, f, m);
  const bool neg = __double_as_longlong(x) < 0;
  if (f == 0x7ff) {
    atomicOr(limbs + RED_LIMBS - 1, m != 1ull << 52 ? 1ull : neg ? 4ull : 2ull);
    return;
  }
  const int k = (f - 1) >> 5, s = (f - 1) & 31;
  const unsigned long long lo = m << s, c[3] = {lo & 0xffffffffull, lo >> 32, s ? m >> (64 - s) : 0};
#pragma unroll
  for (int i = 0; i < 3; i++)
    if (c[i]) atomicAdd(limbs + k + i, neg ? 0 - c[i] : c[i]);
}
// the sum, on every lane of the calling warp; the limbs are zeroed
__device__ __forceinline__ double red_take(unsigned long long *limbs) {
  const int lane = threadIdx.x & 31;
  constexpr int REST = RED_LIMBS - 64;
  long long v0 = (long long)__ldcg(limbs + lane), v1 = (long long)__ldcg(limbs + 32 + lane);
  long long v2 = lane < REST ? (long long)__ldcg(limbs + 64 + lane) : 0;
  if (v0) limbs[lane] = 0;
  if (v1) limbs[32 + lane] = 0;
  if (v2) limbs[64 + lane] = 0;
  const int flags = (int)__shfl_sync(0xffffffffu, v2, REST - 1);
  if (lane == REST - 1) v2 = 0;
  if (flags) {
    const bool nan = (flags & 1) || (flags & 6) == 6;
    return __longlong_as_double(nan ? 0x7ff8000000000000ll : flags & 4 ? (long long)0xfff0000000000000ull : 0x7ff0000000000000ll);
  }
  const unsigned b0 = __ballot_sync(0xffffffffu, v0 != 0), b1 = __ballot_sync(0xffffffffu, v1 != 0),
                 b2 = __ballot_sync(0xffffffffu, v2 != 0);
  const int top = b2 ? 95 - __clz(b2) : b1 ? 63 - __clz(b1) : 31 - __clz(b0);
  if (top < 0) return 0.0;
  long long w[5];   // the five highest limbs
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const int k = top - i;
    const long long r = __shfl_sync(0xffffffffu, k >= 64 ? v2 : k >= 32 ? v1 : v0, k & 31);
    w[i] = k >= 0 ? r : 0;
  }
  // three limbs with the carry of the two below, in units of limb top - 2; a
  // total with a piece in limb `top` is at least 2^64 of them
  const __int128 a = ((((__int128)w[0] << 32) + w[1]) << 32) + w[2] + ((w[3] + (w[4] >> 32)) >> 32);
  const unsigned __int128 u = a < 0 ? -(unsigned __int128)a : (unsigned __int128)a;
  const unsigned long long hi = (unsigned long long)(u >> 64), lo = (unsigned long long)u;
  const int sh = hi ? 64 - __clzll((long long)hi) : 0;   // bits beyond 64, dropped
  const unsigned long long q = sh == 64 ? hi : sh ? (hi << (64 - sh)) | (lo >> sh) : lo;
  return red_double(a < 0, q, 32 * (top - 2) + 1 + sh);
}

// Grid-wide sum of each block's n totals (`tot`, shared); blocks of whole
// warps.  Returns true in the one block, the last to arrive, that holds the
// grid totals in out[0..n) (shared) on return.  red.limbs: n * RED_LIMBS
// integers, red.count: one counter; zero on entry and zero again when the
// launch ends.
__device__ __forceinline__ bool grid_reduce_last(const double *tot, int n, const RedScratch &red, double *out) {
  __shared__ bool am_last;
  // the host sizes the scratch first (ensure_red); a launch that would not
  // fit writes nothing, flags the error and runs no finisher
  if ((size_t)n > red.max_sums) {
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) atomicExch(red.err, 1);
    return false;
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) red_add(red.limbs + (size_t)i * RED_LIMBS, tot[i]);
  __syncthreads();
  // the fence of the thread that arrives orders the block's adds, which the
  // barrier made visible to it, before the arrival
  if (threadIdx.x == 0) {
    __threadfence();
    am_last = atomicAdd(red.count, 1u) == gridDim.x * gridDim.y - 1;
  }
  __syncthreads();
  if (!am_last) return false;
  __threadfence();
  for (int i = threadIdx.x >> 5; i < n; i += blockDim.x >> 5) {
    const double v = red_take(red.limbs + (size_t)i * RED_LIMBS);
    if ((threadIdx.x & 31) == 0) out[i] = v;
  }
  if (threadIdx.x == 0) *red.count = 0;   // ready for the next launch
  __syncthreads();
  return true;
}

}  // namespace mks
