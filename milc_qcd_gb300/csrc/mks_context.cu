// mks_context.cu -- library context, errors, timing, layout conversion and
// fermion-link residency (the part of the C ABI that replaces MILC's QUDA
// set-up and link cache: generic/milc_to_quda_utilities.c:11-41,
// generic_ks/fermion_links_fn_load_gpu.c:19-78, include/fn_links.h:9-17).
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <string>
#include <unordered_map>
#include "mks_internal.cuh"
#include "mks_fixed.cuh"

namespace mks {

static Context g_ctx;
static char g_errmsg[512] = "";

Context &ctx() { return g_ctx; }

void set_last_error(cudaError_t e, const char *what, const char *file, int line) {
  snprintf(g_errmsg, sizeof g_errmsg, "%s failed: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
}

int check_ready(bool need_lattice) {
  if (!g_ctx.initialised) return MKS_ERR_STATE;
  if (need_lattice && g_ctx.V == 0) return MKS_ERR_STATE;
  return MKS_OK;
}

// MKS_MEM_LIMIT (MiB): the most device memory that the library's own
// allocations may add up to (0 or unset: what the device has)
static size_t mem_limit() {
  static long long v = -1;
  if (v < 0) {
    const char *e = getenv("MKS_MEM_LIMIT");
    v = e && atoll(e) > 0 ? atoll(e) : 0;
  }
  return (size_t)v << 20;
}
static std::unordered_map<void *, size_t> g_sizes;   // with a limit: the live allocations
static size_t g_used = 0;

static cudaError_t try_alloc(void **p, size_t bytes) {
  *p = nullptr;
  const size_t limit = mem_limit();
  if (limit && g_used + bytes > limit) return cudaErrorMemoryAllocation;
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
  } else if (limit) {
    g_sizes[*p] = bytes;
    g_used += bytes;
  }
  return e;
}

int dev_alloc(void **p, size_t bytes) {
  *p = nullptr;
  if (bytes == 0) return MKS_OK;
  cudaError_t e = try_alloc(p, bytes);
  if (e != cudaSuccess && mem_release()) e = try_alloc(p, bytes);
  if (e != cudaSuccess) {
    set_last_error(e, "cudaMalloc", __FILE__, __LINE__);
    return MKS_ERR_NOMEM;
  }
  return MKS_OK;
}

void dev_free(void *p) {
  if (!p) return;
  if (mem_limit()) {
    auto it = g_sizes.find(p);
    if (it != g_sizes.end()) {
      g_used -= it->second;
      g_sizes.erase(it);
    }
  }
  cudaFree(p);
}

void mem_info(size_t *free_bytes, size_t *total) {
  const size_t limit = mem_limit();
  if (cudaMemGetInfo(free_bytes, total) != cudaSuccess) {
    cudaGetLastError();
    *free_bytes = *total = 0;
  }
  if (limit && limit < *total) {
    *total = limit;
    if (limit - g_used < *free_bytes) *free_bytes = limit - g_used;
  }
}

bool mem_release() {
  Context &c = g_ctx;
  if (c.fx_busy || c.capture) return false;
  bool any = false;
  for (auto &s : c.slots) {
    if (s.fat_fx || s.lng_fx) any = c.fx_off = true;
    dev_free(s.fat_fx);
    dev_free(s.lng_fx);
    s.fat_fx = s.lng_fx = nullptr;
    s.fx_made = 0;
  }
  return ws_smear_free() || any;
}

// ---------------- timing ----------------
static const int EV_POOL = 4096;

void timing_begin(int family) {
  Context &c = g_ctx;
  if (c.capture) {
    Capture &k = *c.capture;
    k.family.push_back(family);
    if (k.timed) {
      cudaEvent_t e0, e1;
      cudaEventCreate(&e0);
      cudaEventCreate(&e1);
      k.ev.push_back(e0);
      k.ev.push_back(e1);
      // an external record becomes an event-record node that fires on every replay
      cudaEventRecordWithFlags(e0, c.stream, cudaEventRecordExternal);
    }
    return;
  }
  c.launches++;
  c.kernel_launches[family]++;
  if (!c.timing) return;
  if (c.ev_used >= EV_POOL) timing_flush();
  cudaEventRecord(c.ev_pool[2 * c.ev_used], c.stream);
  c.ev_family[c.ev_used] = family;
}

void timing_end(int family) {
  Context &c = g_ctx;
  (void)family;
  if (c.capture) {
    if (c.capture->timed) cudaEventRecordWithFlags(c.capture->ev.back(), c.stream, cudaEventRecordExternal);
    return;
  }
  if (!c.timing) return;
  cudaEventRecord(c.ev_pool[2 * c.ev_used + 1], c.stream);
  c.ev_used++;
}

int timing_flush() {
  Context &c = g_ctx;
  if (c.ev_used == 0) return MKS_OK;
  MKS_CUDA(cudaStreamSynchronize(c.stream));
  for (int i = 0; i < c.ev_used; i++) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c.ev_pool[2 * i], c.ev_pool[2 * i + 1]);
    c.kernel_ms[c.ev_family[i]] += ms;
  }
  c.ev_used = 0;
  return MKS_OK;
}

void capture_account(const Capture &k) {
  Context &c = g_ctx;
  for (size_t i = 0; i < k.family.size(); i++) {
    c.launches++;
    c.kernel_launches[k.family[i]]++;
    if (k.timed && c.timing) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, k.ev[2 * i], k.ev[2 * i + 1]);
      c.kernel_ms[k.family[i]] += ms;
    }
  }
}

// Scratch for a reduction of nsum sums (grid_reduce_last in mks_reduce.cuh).
// Grown, never shrunk; zeroed when (re)allocated and left at zero by every
// launch.
int ensure_red(int nsum) {
  Context &c = g_ctx;
  if (!c.red.err) {
    MKS_TRY(dev_alloc((void **)&c.red.err, sizeof(int)));
    MKS_CUDA(cudaMemsetAsync(c.red.err, 0, sizeof(int), c.stream));
  }
  if (!c.red.count) {
    MKS_TRY(dev_alloc((void **)&c.red.count, sizeof(unsigned int)));
    MKS_CUDA(cudaMemsetAsync(c.red.count, 0, sizeof(unsigned int), c.stream));
  }
  if (c.red.max_sums < (size_t)nsum) {
    dev_free(c.red.limbs);
    c.red.limbs = nullptr;
    c.red.max_sums = 0;
    const size_t n = nsum < 256 ? 256 : nsum, bytes = n * RED_LIMBS * sizeof(unsigned long long);
    MKS_TRY(dev_alloc((void **)&c.red.limbs, bytes));
    MKS_CUDA(cudaMemsetAsync(c.red.limbs, 0, bytes, c.stream));
    c.red.max_sums = n;
  }
  return MKS_OK;
}

int red_check() {
  Context &c = g_ctx;
  if (!c.red.err) return MKS_OK;
  int e = 0;
  MKS_CUDA(cudaMemcpyAsync(&e, c.red.err, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  MKS_CUDA(cudaStreamSynchronize(c.stream));
  if (!e) return MKS_OK;
  MKS_CUDA(cudaMemsetAsync(c.red.err, 0, sizeof(int), c.stream));
  if (e & 6) {
    // value 2: a TMA-staged D_eo tile gave up waiting for its links (it
    // computed nothing); value 4: its copies were still in flight after the
    // second wait.  The staged kernel is off from now on.
    tma_disable();
    snprintf(g_errmsg, sizeof g_errmsg,
             "TMA-staged D_eo: link staging did not complete within its wait limit (%s); the staged kernel is "
             "switched off for this process",
             (e & 4) ? "copies still in flight" : "tile skipped");
    return MKS_ERR_TIMEOUT;
  }
  snprintf(g_errmsg, sizeof g_errmsg, "reduction scratch too small for a launch (internal sizing error)");
  return MKS_ERR_CUDA;
}

// ---------------- layout conversion kernels ----------------
// full AoS vector field [V][6] -> one parity SoA double2 [3][Vh].  One
// complex number per thread: the parity half of a MILC field is 3*Vh
// consecutive complex numbers, taken in order, so the reads (and in
// k_vec_soa_to_aos the writes) of the AoS side are contiguous across a warp
// -- the AoS side is often a page-locked host array read over the host link.
// 16-byte accesses where the array allows them.
__device__ __forceinline__ double2 aos_get(const double *base, size_t t) {
  if (((uintptr_t)base & 15) == 0) return reinterpret_cast<const double2 *>(base)[t];
  return make_double2(base[2 * t], base[2 * t + 1]);
}
__global__ void k_vec_aos_to_soa(const double *__restrict__ aos, double2 *__restrict__ soa, int par, int Vh) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= 3 * (size_t)Vh) return;
  const size_t h = t / 3;
  const int c = (int)(t - 3 * h);
  soa[(size_t)c * Vh + h] = aos_get(aos + (size_t)par * Vh * 6, t);
}
__global__ void k_vec_soa_to_aos(const double2 *__restrict__ soa, double *__restrict__ aos, int par, int Vh) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= 3 * (size_t)Vh) return;
  const size_t h = t / 3;
  const int c = (int)(t - 3 * h);
  const double2 v = soa[(size_t)c * Vh + h];
  double *base = aos + (size_t)par * Vh * 6;
  if (((uintptr_t)base & 15) == 0) {
    reinterpret_cast<double2 *>(base)[t] = v;
  } else {
    base[2 * t] = v.x;
    base[2 * t + 1] = v.y;
  }
}
// links [V][4][18] -> [2][4][9][Vh]
__global__ void k_links_aos_to_soa(const double *__restrict__ aos, double2 *__restrict__ soa, int Vh) {
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int par = blockIdx.y, dir = blockIdx.z;
  if (h >= Vh) return;
  const double *s = aos + (((size_t)par * Vh + h) * 4 + dir) * 18;
  double2 *d = soa + ((size_t)(par * 4 + dir) * 9) * Vh + h;
#pragma unroll
  for (int k = 0; k < 9; k++) d[(size_t)k * Vh] = make_double2(s[2 * k], s[2 * k + 1]);
}
__global__ void k_links_soa_to_aos(const double2 *__restrict__ soa, double *__restrict__ aos, int Vh) {
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int par = blockIdx.y, dir = blockIdx.z;
  if (h >= Vh) return;
  double *d = aos + (((size_t)par * Vh + h) * 4 + dir) * 18;
  const double2 *s = soa + ((size_t)(par * 4 + dir) * 9) * Vh + h;
#pragma unroll
  for (int k = 0; k < 9; k++) { double2 v = s[(size_t)k * Vh]; d[2 * k] = v.x; d[2 * k + 1] = v.y; }
}
// What the reduced-precision and integer forms need to know of a link field:
// its largest |component|, the smallest of its matrices that are not zero (by
// their largest component), whether one is not finite, and how many are uneven
// (mks_fixed.cuh).  All zero before the launch.
struct LinkStats {
  unsigned long long max, inv_min, bad;   // bits of the doubles; inv_min: of the smallest, complemented
  FxUneven uneven;
};
__global__ void k_links_stats(const double2 *__restrict__ src, int Vh, LinkStats *out) {
  u64 top = 0, low = ~0ull;
  bool bad = false, uneven = false;
  int ents = 0, parts = 0;
  for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < Vh; h += gridDim.x * blockDim.x) {
    const double2 *s = src + (size_t)blockIdx.y * 9 * Vh + h;   // par*4+dir
    double2 v[9];
#pragma unroll
    for (int k = 0; k < 9; k++) v[k] = s[(size_t)k * Vh];
    const FxShape f(v);
    bad = bad || f.bad;
    uneven = uneven || f.uneven;
    ents += f.ents;
    parts += f.parts;
    top = f.top > top ? f.top : top;
    low = f.top != 0 && f.top < low ? f.top : low;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const u64 t = __shfl_xor_sync(0xffffffffu, top, o), l = __shfl_xor_sync(0xffffffffu, low, o);
    top = t > top ? t : top;
    low = l < low ? l : low;
  }
  bad = __any_sync(0xffffffffu, bad);
  fx_uneven_add(&out->uneven, uneven, ents, parts);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&out->max, top);
    if (top > 0) atomicMax(&out->inv_min, ~low);
    if (bad) atomicMax(&out->bad, 1ull);
  }
}
// the FP32, FP16 and, where the slot keeps them, integer forms of a link field
// in one pass over its FP64 entries (a pass each read them three times;
// HBM-bound: 144 B read and 252 B written per link)
__global__ void k_links_lowprec(const double2 *__restrict__ src, float4 *__restrict__ a32, float2 *__restrict__ b32,
                                uint4 *__restrict__ a16, __half2 *__restrict__ b16, int4 *__restrict__ fx, float inv,
                                int fx_exp, int Vh) {
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  int pd = blockIdx.y;  // par*4+dir
  if (h >= Vh) return;
  const double2 *s = src + ((size_t)pd * 9) * Vh + h;
  float2 f[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 u = s[(size_t)k * Vh];
    f[k] = make_float2((float)u.x, (float)u.y);
    if (!fx) continue;   // no integer copies
    int4 w;
    fx_split(fx_scale(u.x, fx_exp) + 8, w.x, w.y);  // + 8: rounds the cut at 16
    fx_split(fx_scale(u.y, fx_exp) + 8, w.z, w.w);
    fx[((size_t)pd * 9 + k) * Vh + h] = w;
  }
#pragma unroll
  for (int k = 0; k < 4; k++)
    a32[((size_t)pd * 4 + k) * Vh + h] = make_float4(f[2 * k].x, f[2 * k].y, f[2 * k + 1].x, f[2 * k + 1].y);
  b32[(size_t)pd * Vh + h] = f[8];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    unsigned w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      __half2 hv = __floats2half2_rn(f[4 * k + j].x * inv, f[4 * k + j].y * inv);
      w[j] = *reinterpret_cast<unsigned *>(&hv);
    }
    a16[((size_t)pd * 2 + k) * Vh + h] = make_uint4(w[0], w[1], w[2], w[3]);
  }
  b16[(size_t)pd * Vh + h] = __floats2half2_rn(f[8].x * inv, f[8].y * inv);
}

int vec_aos_to_soa64(const double *aos_dev, double2 *soa, int par) {
  Context &c = g_ctx;
  int Vh = (int)c.Vh;
  k_vec_aos_to_soa<<<grid_for(3 * Vh, 256), 256, 0, c.stream>>>(aos_dev, soa, par, Vh);
  c.launches++;
  MKS_CUDA(cudaGetLastError());
  return MKS_OK;
}
__global__ void k_vec_aos_to_soa32(const double *__restrict__ aos, float2 *__restrict__ soa, int par, int Vh) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= 3 * (size_t)Vh) return;
  const size_t h = t / 3;
  const int c = (int)(t - 3 * h);
  const double2 v = aos_get(aos + (size_t)par * Vh * 6, t);
  soa[(size_t)c * Vh + h] = make_float2((float)v.x, (float)v.y);
}
int vec_aos_to_soa32(const double *aos_dev, float2 *soa, int par) {
  Context &c = g_ctx;
  int Vh = (int)c.Vh;
  k_vec_aos_to_soa32<<<grid_for(3 * Vh, 256), 256, 0, c.stream>>>(aos_dev, soa, par, Vh);
  c.launches++;
  MKS_CUDA(cudaGetLastError());
  return MKS_OK;
}
int vec_soa64_to_aos(const double2 *soa, double *aos_dev, int par) {
  Context &c = g_ctx;
  int Vh = (int)c.Vh;
  k_vec_soa_to_aos<<<grid_for(3 * Vh, 256), 256, 0, c.stream>>>(soa, aos_dev, par, Vh);
  c.launches++;
  MKS_CUDA(cudaGetLastError());
  return MKS_OK;
}
int links_aos_to_soa64(const double *aos_dev, double2 *soa) {
  Context &c = g_ctx;
  int Vh = (int)c.Vh;
  k_links_aos_to_soa<<<dim3(grid_for(Vh, 128), 2, 4), 128, 0, c.stream>>>(aos_dev, soa, Vh);
  c.launches++;
  MKS_CUDA(cudaGetLastError());
  return MKS_OK;
}
int links_soa64_to_aos(const double2 *soa, double *aos_dev) {
  Context &c = g_ctx;
  int Vh = (int)c.Vh;
  k_links_soa_to_aos<<<dim3(grid_for(Vh, 128), 2, 4), 128, 0, c.stream>>>(soa, aos_dev, Vh);
  c.launches++;
  MKS_CUDA(cudaGetLastError());
  return MKS_OK;
}

static void free_slot(LinkSlot &s) {
  dev_free(s.fat64); dev_free(s.lng64);
  dev_free(s.fat32a); dev_free(s.lng32a); dev_free(s.fat32b); dev_free(s.lng32b);
  dev_free(s.fat16a); dev_free(s.lng16a); dev_free(s.fat16b); dev_free(s.lng16b);
  dev_free(s.fat_fx); dev_free(s.lng_fx);
  s = LinkSlot();
}

// Room for the integer copies of a slot's links, 2304 bytes per site of a
// parity beside the 4032 of its other forms: taken only if eight times as much,
// or an eighth of the memory, stays free for the solves and for other users of
// the device.  D_eo does without them where there is none.
static bool alloc_fx(LinkSlot &s) {
  const size_t bytes = (size_t)8 * 9 * g_ctx.Vh * sizeof(int4), both = 2 * bytes;
  if (s.fat_fx && s.lng_fx) return true;
  if (g_ctx.fx_off) return false;
  size_t avail, total;
  mem_info(&avail, &total);
  if (avail < both + (total / 8 < 8 * both ? total / 8 : 8 * both)) return false;
  if (try_alloc((void **)&s.fat_fx, bytes) == cudaSuccess && try_alloc((void **)&s.lng_fx, bytes) == cudaSuccess)
    return true;
  dev_free(s.fat_fx);
  s.fat_fx = s.lng_fx = nullptr;
  return false;
}

int links_make_lowprec(LinkSlot &s) {
  Context &c = g_ctx;
  int Vh = (int)c.Vh;
  size_t n32a = (size_t)8 * 4 * Vh, n32b = (size_t)8 * Vh;
  s.fx_made = 0;
  auto need = [](auto *&q, size_t n) { return q ? (int)MKS_OK : dev_alloc((void **)&q, n * sizeof *q); };
  MKS_TRY(need(s.fat32a, n32a));
  MKS_TRY(need(s.lng32a, n32a));
  MKS_TRY(need(s.fat32b, n32b));
  MKS_TRY(need(s.lng32b, n32b));
  MKS_TRY(need(s.fat16a, n32a / 2));
  MKS_TRY(need(s.lng16a, n32a / 2));
  MKS_TRY(need(s.fat16b, n32b));
  MKS_TRY(need(s.lng16b, n32b));
  // the FP16 scales, and the integers' exponents if they serve these links
  LinkStats *dst, st[2];
  MKS_TRY(dev_alloc((void **)&dst, sizeof st));
  MKS_CUDA(cudaMemsetAsync(dst, 0, sizeof st, c.stream));
  const dim3 sgrid((c.sm_count + 1) / 2, 8);
  k_links_stats<<<sgrid, 256, 0, c.stream>>>(s.fat64, Vh, dst);
  k_links_stats<<<sgrid, 256, 0, c.stream>>>(s.lng64, Vh, dst + 1);
  MKS_CUDA(cudaMemcpyAsync(st, dst, sizeof st, cudaMemcpyDeviceToHost, c.stream));
  MKS_CUDA(cudaStreamSynchronize(c.stream));
  dev_free(dst);
  double top[2], low[2];
  int ex[2] = {-1021, -1021};
  bool plain = false;
  for (int k = 0; k < 2; k++) {
    memcpy(&top[k], &st[k].max, 8);
    const unsigned long long b = ~st[k].inv_min;
    memcpy(&low[k], &b, 8);
    if (st[k].bad || st[k].uneven.any((size_t)8 * Vh)) plain = true;
    if (st[k].bad || !(top[k] > 0)) continue;
    if (ldexp(low[k], FX_SPREAD) < top[k]) plain = true;
    int e = 0;
    frexp(top[k], &e);
    if (e > ex[k]) ex[k] = e;
  }
  s.fat16scale = (float)top[0];
  s.lng16scale = (float)top[1];
  s.fat_exp = ex[0];
  s.lng_exp = ex[1];
  const float inv[2] = {top[0] > 0 ? (float)(1.0 / top[0]) : 0.f, top[1] > 0 ? (float)(1.0 / top[1]) : 0.f};
  const dim3 grid(grid_for(Vh, 256), 8);
  const bool fx = !plain && alloc_fx(s);
  k_links_lowprec<<<grid, 256, 0, c.stream>>>(s.fat64, s.fat32a, s.fat32b, s.fat16a, s.fat16b,
                                              fx ? s.fat_fx : nullptr, inv[0], ex[0], Vh);
  k_links_lowprec<<<grid, 256, 0, c.stream>>>(s.lng64, s.lng32a, s.lng32b, s.lng16a, s.lng16b,
                                              fx ? s.lng_fx : nullptr, inv[1], ex[1], Vh);
  c.launches += 4;
  MKS_CUDA(cudaGetLastError());
  s.fx_made = fx;
  return MKS_OK;
}

static int load_slot_from_dev(int slot, const double *fat_dev, const double *lng_dev, double eps) {
  Context &c = g_ctx;
  LinkSlot &s = c.slots[slot];
  size_t nsoa = (size_t)8 * 9 * c.Vh;
  if (!s.fat64) {
    MKS_TRY(dev_alloc((void **)&s.fat64, nsoa * sizeof(double2)));
    MKS_TRY(dev_alloc((void **)&s.lng64, nsoa * sizeof(double2)));
  }
  MKS_TRY(links_aos_to_soa64(fat_dev, s.fat64));
  MKS_TRY(links_aos_to_soa64(lng_dev, s.lng64));
  MKS_TRY(links_make_lowprec(s));
  s.eps_naik = eps;
  s.valid = true;
  return MKS_OK;
}

}  // namespace mks

using namespace mks;

extern "C" {

const char *mks_error_string(int status) {
  switch (status) {
  case MKS_OK: return "ok";
  case MKS_ERR_ARG: return "invalid argument";
  case MKS_ERR_CUDA: return g_errmsg[0] ? g_errmsg : "CUDA error";
  case MKS_ERR_NOMEM: return g_errmsg[0] ? g_errmsg : "device allocation failed";
  case MKS_ERR_STATE: return "library not initialised, lattice not set or links not loaded";
  case MKS_ERR_TIMEOUT: return g_errmsg[0] ? g_errmsg : "bounded device wait gave up";
  case MKS_ERR_NUMERIC: return "non-finite value in a solver recurrence";
  case MKS_ERR_UNSUPPORTED: return "unsupported option";
  default: return "unknown status";
  }
}

int mks_init(int device) {
  Context &c = g_ctx;
  if (c.initialised) return MKS_OK;
  int n = 0;
  MKS_CUDA(cudaGetDeviceCount(&n));
  if (device < 0 || device >= n) return MKS_ERR_ARG;
  MKS_CUDA(cudaSetDevice(device));
  cudaDeviceProp prop;
  MKS_CUDA(cudaGetDeviceProperties(&prop, device));
  if (prop.major < 10) {
    snprintf(g_errmsg, sizeof g_errmsg, "device %d is sm_%d%d; the library is compiled for sm_103a", device,
             prop.major, prop.minor);
    return MKS_ERR_UNSUPPORTED;
  }
  c.device = device;
  c.sm_count = prop.multiProcessorCount;
  MKS_CUDA(cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking));
  c.ev_pool.resize(2 * EV_POOL);
  c.ev_family.resize(EV_POOL);
  for (auto &e : c.ev_pool) MKS_CUDA(cudaEventCreate(&e));
  // the allocation-free D_eo takes no device memory after this point: its
  // fixed array and the kernels it launches are loaded now
  cudaFuncAttributes fa;
  MKS_CUDA(cudaFuncGetAttributes(&fa, k_vec_aos_to_soa));
  MKS_CUDA(cudaFuncGetAttributes(&fa, k_vec_soa_to_aos));
  MKS_TRY(noalloc_prepare());
  c.initialised = true;
  return MKS_OK;
}

static void free_lattice_fields() {
  Context &c = g_ctx;
  for (auto &s : c.slots) free_slot(s);
  ws_free_all();
  dev_free(c.auxU); dev_free(c.auxV); dev_free(c.auxW);
  c.auxU = c.auxV = c.auxW = nullptr;
  c.aux_action = 0;
  dev_free(c.mom);
  c.mom = nullptr;
  c.fx_off = c.fxm_off = false;
  gauge_free();
  rhmc_free();
}

int mks_finalize(void) {
  Context &c = g_ctx;
  if (!c.initialised) return MKS_OK;
  cudaStreamSynchronize(c.stream);
  free_lattice_fields();
  dev_free(c.red.limbs); dev_free(c.red.count); dev_free(c.red.err);
  c.red = RedScratch();
  for (auto &e : c.ev_pool) cudaEventDestroy(e);
  c.ev_pool.clear();
  cudaStreamDestroy(c.stream);
  noalloc_forget();
  c = Context();
  return MKS_OK;
}

int mks_set_lattice(const int dims[4]) {
  MKS_TRY(check_ready(false));
  if (!dims) return MKS_ERR_ARG;
  // even extents of at least 4: the Naik term reaches 3 sites, and a hop of
  // 3 must wrap at most once
  for (int d = 0; d < 4; d++)
    if (dims[d] < 4 || (dims[d] & 1)) return MKS_ERR_ARG;
  Context &c = g_ctx;
  size_t V = (size_t)dims[0] * dims[1] * dims[2] * dims[3];
  if (V / 2 > (size_t)0x3fffffff) return MKS_ERR_ARG;  // checkerboard index is 32-bit
  bool same = V == c.V && !memcmp(dims, c.dims, sizeof c.dims);
  if (!same) {
    MKS_CUDA(cudaStreamSynchronize(c.stream));
    free_lattice_fields();
  }
  memcpy(c.dims, dims, sizeof c.dims);
  c.V = V;
  c.Vh = V / 2;
  c.geom.nx = dims[0]; c.geom.ny = dims[1]; c.geom.nz = dims[2]; c.geom.nt = dims[3];
  c.geom.Vh = (int)c.Vh;
  c.geom.sx = 1; c.geom.sy = dims[0]; c.geom.sz = dims[0] * dims[1]; c.geom.st = dims[0] * dims[1] * dims[2];
  // Reduction scratch for the largest reducing launch, so that it is never
  // reallocated while a solver batch is being captured: 32 rows x 3 sums of
  // the BLAS site kernels (D_eo epilogues: 16 sources x 3 sums).
  MKS_TRY(ensure_red(32 * 3));
  return MKS_OK;
}

int mks_load_fn_links_dev(int slot, const double *fat_dev, const double *lng_dev, double eps_naik) {
  MKS_TRY(check_ready());
  if (slot < 0 || slot >= MKS_MAX_SLOTS || !fat_dev || !lng_dev) return MKS_ERR_ARG;
  MKS_TRY(load_slot_from_dev(slot, fat_dev, lng_dev, eps_naik));
  MKS_CUDA(cudaStreamSynchronize(g_ctx.stream));
  return MKS_OK;
}

int mks_load_fn_links(int slot, const double *fat, const double *lng, double eps_naik) {
  MKS_TRY(check_ready());
  if (slot < 0 || slot >= MKS_MAX_SLOTS || !fat || !lng) return MKS_ERR_ARG;
  Context &c = g_ctx;
  size_t bytes = c.V * 4 * 18 * sizeof(double);
  double *tmp;
  MKS_TRY(dev_alloc((void **)&tmp, 2 * bytes));
  MKS_CUDA(cudaMemcpyAsync(tmp, fat, bytes, cudaMemcpyHostToDevice, c.stream));
  MKS_CUDA(cudaMemcpyAsync(tmp + c.V * 72, lng, bytes, cudaMemcpyHostToDevice, c.stream));
  int rc = load_slot_from_dev(slot, tmp, tmp + c.V * 72, eps_naik);
  cudaStreamSynchronize(c.stream);
  dev_free(tmp);
  return rc;
}

int mks_invalidate_fn_links(int slot) {
  MKS_TRY(check_ready(false));
  if (slot < 0 || slot >= MKS_MAX_SLOTS) return MKS_ERR_ARG;
  g_ctx.slots[slot].valid = false;
  return MKS_OK;
}

int mks_get_fn_links(int slot, double *fat, double *lng) {
  MKS_TRY(check_ready());
  if (slot < 0 || slot >= MKS_MAX_SLOTS) return MKS_ERR_ARG;
  Context &c = g_ctx;
  LinkSlot &s = c.slots[slot];
  if (!s.valid) return MKS_ERR_STATE;
  size_t bytes = c.V * 4 * 18 * sizeof(double);
  double *tmp;
  MKS_TRY(dev_alloc((void **)&tmp, bytes));
  int rc = MKS_OK;
  if (fat) {
    MKS_TRY(links_soa64_to_aos(s.fat64, tmp));
    MKS_CUDA(cudaMemcpyAsync(fat, tmp, bytes, cudaMemcpyDeviceToHost, c.stream));
    MKS_CUDA(cudaStreamSynchronize(c.stream));
  }
  if (lng) {
    MKS_TRY(links_soa64_to_aos(s.lng64, tmp));
    MKS_CUDA(cudaMemcpyAsync(lng, tmp, bytes, cudaMemcpyDeviceToHost, c.stream));
    MKS_CUDA(cudaStreamSynchronize(c.stream));
  }
  dev_free(tmp);
  return rc;
}

int mks_timing_enable(int on) {
  MKS_TRY(check_ready(false));
  if (!on) MKS_TRY(timing_flush());
  g_ctx.timing = on != 0;
  return MKS_OK;
}

int mks_timing_reset(void) {
  MKS_TRY(check_ready(false));
  MKS_TRY(timing_flush());
  Context &c = g_ctx;
  for (int k = 0; k < MKS_K_COUNT; k++) { c.kernel_ms[k] = 0; c.kernel_launches[k] = 0; }
  c.launches = 0;
  return MKS_OK;
}

int mks_timing_get(int family, double *total_ms, long long *launches) {
  MKS_TRY(check_ready(false));
  if (family < 0 || family >= MKS_K_COUNT) return MKS_ERR_ARG;
  MKS_TRY(timing_flush());
  if (total_ms) *total_ms = g_ctx.kernel_ms[family];
  if (launches) *launches = g_ctx.kernel_launches[family];
  return MKS_OK;
}

long long mks_launch_count(void) { return g_ctx.launches; }

void *mks_stream(void) { return (void *)g_ctx.stream; }

}  // extern "C"
