// fftoc — C ABI: argument checks, per-device set-up (twiddle tables, kernel
// attributes), engine selection and launch.
//
// Reference behaviour replaced here: the harness of gprabowski/fft_onchip
// (includes/testing.cuh:59-92) sets the dynamic shared-memory attribute,
// launches fft_tester<CT,Exec,N,UPB> with grid (32*SMs)/(UPB*FPU) and block
// (threads, UPB), and aborts the process through gpuErrchk
// (includes/common.cuh:3-13) on any CUDA error.  This library instead returns
// a status, keeps a per-thread message, and sizes the grid from the batch.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include <cuda.h>

#include "../../include/fftoc.h"
#include "fft_core.cuh"
#include "host_range.h"
#include "internal.h"

namespace fftoc {
namespace {

thread_local std::string t_last_error;

fftoc_status fail(fftoc_status st, const std::string& msg) {
  t_last_error = msg;
  return st;
}

fftoc_status cuda_fail(cudaError_t e, const char* what) {
  cudaGetLastError();  // clear a non-sticky error
  return fail(FFTOC_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// cos and sin of 2*pi*k/n in long double, with the angle reduced to
// [0, pi/4] through the exact rational k/n (octant symmetry).
void cos_sin(long long n, long long k, long double* c, long double* s) {
  const long double pi = 3.141592653589793238462643383279502884L;
  k %= n;
  if (k < 0) k += n;
  const long long k8 = 8 * k;
  const long long o = k8 / n;
  const long long r = k8 - o * n;  // angle = (pi/4) * (o + r/n)
  long double cb, sb;
  if (o & 1) {
    const long double phi = (pi / 4.0L) * ((long double)(n - r) / (long double)n);
    cb = cosl(phi);
    sb = sinl(phi);
    switch (((o + 1) / 2) & 3) {  // angle = q*pi/2 - phi
      case 0: *c = cb; *s = -sb; break;
      case 1: *c = sb; *s = cb; break;
      case 2: *c = -cb; *s = sb; break;
      default: *c = -sb; *s = -cb; break;
    }
  } else {
    const long double phi = (pi / 4.0L) * ((long double)r / (long double)n);
    cb = cosl(phi);
    sb = sinl(phi);
    switch ((o / 2) & 3) {  // angle = q*pi/2 + phi
      case 0: *c = cb; *s = sb; break;
      case 1: *c = -sb; *s = cb; break;
      case 2: *c = -cb; *s = -sb; break;
      default: *c = sb; *s = -cb; break;
    }
  }
}

// v * 2^60 as h*2^30 + l with 0 <= l < 2^30 (|v| <= 1 gives |h| <= 2^30)
void fx_limbs(long double v, int* h, int* l) {
  const long long q = llroundl(v * 1152921504606846976.0L);  // 2^60
  *h = (int)(q >> 30);                                       // arithmetic: floor
  *l = (int)(q & ((1LL << 30) - 1));
}

// Device staging for host-buffer calls: three chunk buffers cycled through
// H2D -> transform -> D2H on three streams.
struct Staging {
  static constexpr int kBufs = 3;
  static constexpr size_t kChunkBytes = 64u << 20;
  std::once_flag once;
  fftoc_status status = FFTOC_OK;
  std::string error;
  std::mutex mu;
  cudaStream_t s_h2d = nullptr, s_cmp = nullptr, s_d2h = nullptr;
  void* buf[kBufs] = {};
  cudaEvent_t ev_h2d[kBufs] = {}, ev_cmp[kBufs] = {}, ev_d2h[kBufs] = {};
  cudaEvent_t ev_start = nullptr;
};

struct DeviceState {
  Staging staging;
  std::once_flag once;
  fftoc_status init_status = FFTOC_OK;
  std::string init_error;
  SizeVariants var[2][kNumSizes];                 // [engine: 0 f64, 1 fx][size]
  void* tw[2][kNumSizes][kMaxVariants] = {};      // per-variant twiddle tables
  int* err = nullptr;                             // device error flag (bounded waits that gave up)
  int sms = 0;
  std::atomic<bool> ready{false};                 // set-up done and successful
};

// Plan chosen per (engine, size), plus one: process-wide, set by
// fftoc_plan_select or fftoc_autotune; 0 until then and after
// fftoc_plan_unselect.
std::atomic<int> g_choice[2][kNumSizes];

const SizeVariants* host_variants(int eng_slot) {
  static SizeVariants table[2][kNumSizes];
  static std::once_flag once;
  std::call_once(once, [] {
    describe_f64(table[0]);
    describe_fx(table[1]);
  });
  return table[eng_slot];
}

constexpr int kMaxDevices = 64;
DeviceState g_devices[kMaxDevices];

// v * 2^62 as h*2^32 + l with l signed (|v| <= sqrt 2)
void fxn_limbs(long double v, int* h, int* l) {
  const long long q = llroundl(v * 4611686018427387904.0L);  // 2^62
  *l = (int)(unsigned)q;
  *h = (int)((q - *l) >> 32);
}

// Twiddle table of a plan in each engine's layout.  f64: (cos, -sin) pairs, or
// (d.tangent) those of the upper half of a pass's inputs in EngF64's tangent
// form.
// fx, 4 ints per entry: 30-bit limbs of both parts, or (d.natural) the natural
// limbs of wr and of wi - wr; there, behind all entries, 2 ints per entry: the
// limbs of -(wr + wi).
void build_twiddles(const KernelDesc& d, std::vector<double>& f64, std::vector<int>& fx) {
  f64.assign((size_t)d.tw_entries * 2, 0.0);
  fx.assign((size_t)d.tw_entries * (d.natural ? 6 : 4), 0);
  int off = 0, p = d.radix[0];
  for (int s = 1; s < d.passes; ++s) {
    const int R = d.radix[s];
    for (int m = 1; m < R; ++m)
      for (int k = 0; k < p; ++k) {
        long double c, sn;
        cos_sin((long long)R * p, (long long)k * m, &c, &sn);
        const int e = off + (m - 1) * p + k;
        f64[2 * e] = (double)c;
        f64[2 * e + 1] = (double)(-sn);
        if (d.tangent && m >= R / 2) {
          const bool turned = EngF64::tangent_turned(k * m, R * p);
          f64[2 * e] = (double)(turned ? -sn : c);
          f64[2 * e + 1] = (double)(turned ? c / sn : -sn / c);
        }
        if (d.natural) {
          int* sum = &fx[4 * (size_t)d.tw_entries + 2 * e];
          fxn_limbs(c, &fx[4 * e], &fx[4 * e + 1]);
          fxn_limbs(-sn - c, &fx[4 * e + 2], &fx[4 * e + 3]);
          fxn_limbs(sn - c, &sum[0], &sum[1]);
        } else {
          fx_limbs(c, &fx[4 * e], &fx[4 * e + 1]);
          fx_limbs(-sn, &fx[4 * e + 2], &fx[4 * e + 3]);
        }
      }
    off += (R - 1) * p;
    p *= R;
  }
}

void init_device(DeviceState& ds) {
  for (int eng = 0; eng < 2; ++eng)
    for (int i = 0; i < kNumSizes; ++i) ds.var[eng][i] = host_variants(eng)[i];
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&ds.sms, cudaDevAttrMultiProcessorCount, dev);
  {
    cudaError_t e = cudaMalloc(&ds.err, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(ds.err, 0, sizeof(int));
    if (e != cudaSuccess) {
      cudaGetLastError();
      ds.init_status = FFTOC_ERR_NO_MEMORY;
      ds.init_error = std::string("cudaMalloc(error flag): ") + cudaGetErrorString(e);
      return;
    }
  }
  for (int eng = 0; eng < 2; ++eng)
    for (int i = 0; i < kNumSizes; ++i)
      for (int v = 0; v < ds.var[eng][i].count; ++v) {
        KernelDesc& d = ds.var[eng][i].v[v];
        cudaError_t e = allow_shared(d.fn, d.smem);
        // persistent grids are sized from the resident CTAs per SM
        if (e == cudaSuccess && d.persistent) e = fit_carveout(d.fn, d.threads, d.smem, &d.blocks_per_sm);
        else if (e == cudaSuccess)
          e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.blocks_per_sm, d.fn, d.threads, d.smem);
        if (e != cudaSuccess) {
          cudaGetLastError();
          ds.init_status = FFTOC_ERR_CUDA;
          ds.init_error = std::string("kernel set-up: ") + cudaGetErrorString(e);
          return;
        }
        if (d.blocks_per_sm < 1) d.blocks_per_sm = 1;
        std::vector<double> f64;
        std::vector<int> fx;
        build_twiddles(d, f64, fx);
        const size_t used = eng == 0 ? f64.size() * sizeof(double) : fx.size() * sizeof(int);
        const size_t bytes = used > 0 ? used : 16;
        void* p = nullptr;
        e = cudaMalloc(&p, bytes);
        if (e != cudaSuccess) {
          cudaGetLastError();
          ds.init_status = FFTOC_ERR_NO_MEMORY;
          ds.init_error = std::string("cudaMalloc(twiddles): ") + cudaGetErrorString(e);
          return;
        }
        const void* src = eng == 0 ? (const void*)f64.data() : (const void*)fx.data();
        if (d.tw_entries > 0) e = cudaMemcpy(p, src, used, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
          cudaGetLastError();
          ds.init_status = FFTOC_ERR_CUDA;
          ds.init_error = std::string("cudaMemcpy(twiddles): ") + cudaGetErrorString(e);
          return;
        }
        ds.tw[eng][i][v] = p;
      }
}

fftoc_status device_state(DeviceState** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) return fail(FFTOC_ERR_INVALID_VALUE, "device ordinal out of range");
  DeviceState& ds = g_devices[dev];
  std::call_once(ds.once, [&] {
    init_device(ds);
    if (ds.init_status == FFTOC_OK) ds.ready.store(true, std::memory_order_release);
  });
  if (ds.init_status != FFTOC_OK) return fail(ds.init_status, ds.init_error);
  *out = &ds;
  return FFTOC_OK;
}

void init_staging(Staging& sg) {
  auto bad = [&](cudaError_t e, const char* what) {
    cudaGetLastError();
    sg.status = (e == cudaErrorMemoryAllocation) ? FFTOC_ERR_NO_MEMORY : FFTOC_ERR_CUDA;
    sg.error = std::string(what) + ": " + cudaGetErrorString(e);
  };
  cudaError_t e;
  for (cudaStream_t* st : {&sg.s_h2d, &sg.s_cmp, &sg.s_d2h})
    if ((e = cudaStreamCreateWithFlags(st, cudaStreamNonBlocking)) != cudaSuccess) return bad(e, "cudaStreamCreate");
  for (int b = 0; b < Staging::kBufs; ++b) {
    if ((e = cudaMalloc(&sg.buf[b], Staging::kChunkBytes)) != cudaSuccess) return bad(e, "cudaMalloc(staging)");
    for (cudaEvent_t* ev : {&sg.ev_h2d[b], &sg.ev_cmp[b], &sg.ev_d2h[b]})
      if ((e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming)) != cudaSuccess) return bad(e, "cudaEventCreate");
  }
  if ((e = cudaEventCreateWithFlags(&sg.ev_start, cudaEventDisableTiming)) != cudaSuccess) return bad(e, "cudaEventCreate");
}

int resolve_engine(int n, int engine) {
  (void)n;
  return engine == FFTOC_ENGINE_AUTO ? FFTOC_ENGINE_FX : engine;
}

}  // namespace

// Accessors for other translation units (the allocation-free entry point).
const SizeVariants* compiled_variants(int eng_slot) { return host_variants(eng_slot); }
void twiddle_tables(const KernelDesc& d, std::vector<double>& f64, std::vector<int>& fx) { build_twiddles(d, f64, fx); }
int chosen_variant(int eng_slot, int idx) {
  const int c = g_choice[eng_slot][idx].load(std::memory_order_relaxed);
  return c > 0 ? c - 1 : 0;
}
int resolved_engine(int n, int engine) { return resolve_engine(n, engine); }
fftoc_status set_error(fftoc_status st, const std::string& msg) { return fail(st, msg); }
fftoc_status device_plan_resources(int slot, int idx, int var, const void** tw, int** err, int* sms) {
  DeviceState* ds = nullptr;
  fftoc_status st = device_state(&ds);
  if (st != FFTOC_OK) return st;
  if (var < 0 || var >= ds->var[slot][idx].count) return fail(FFTOC_ERR_INVALID_VALUE, "no such plan variant");
  *tw = ds->tw[slot][idx][var];
  *err = ds->err;
  *sms = ds->sms;
  return FFTOC_OK;
}

// Plan of a batch, on device buffers and on host buffers (which give the same
// bits therefore): the chosen one for every batch, or while none was chosen the SmallBatch<> plan with the lowest limit that takes the
// batch, else variant 0.  The limits are where two neighbours measured equal on
// 152 SMs, or where the larger one's waves first beat the other (back-to-back
// launches, us, variant 0 -> the plans below it, at one transform and at each
// limit):
//          fixed point                                 binary64
//   8      4.0 -> 2.0   7.3 -> 5.9 (77824)             5.4 -> 2.1    6.5 -> 4.9 (29184)
//   16     2.9 -> 2.2   3.5 -> 3.4 (19456)             3.7 -> 2.5    4.3 -> 3.6 (7296)
//   32     4.5 -> 2.3   15.7 -> 15.3 (77824)           8.4 -> 3.1    9.0 -> 7.4 (7296)
//   64     3.0 -> 2.2   3.8 -> 3.7 (4864)             10.1 -> 3.5   10.8 -> 8.8 (3648)
//   128    5.6 -> 2.3   5.5 -> 3.9 (2432), 60.2 -> 55.8 (77824)   12.5 -> 4.1   13.0 -> 10.2 (1824)
//   256    6.2 -> 2.3   6.0 -> 4.1 (1216), 63.6 -> 58.8 (38912)   14.0 -> 4.3   27.1 -> 21.8 (1824)
//   512    3.5 -> 3.3   5.3 -> 5.2 (760)              15.0 -> 7.9   30.2 -> 26.7 (1064)
//   1024   4.2 -> 3.8   6.3 -> 6.2 (456)              33.8 -> 15.8  132 -> 126 (2432)
//   2048   6.8 -> 5.1   18.3 -> 17.4 (912)            radix 8 as fast: none
//   4096   radix 8 in 512 threads 8.7 against 8.6, a barrier more: none; binary64 the same
int batch_variant(int slot, int idx, int64_t batch, int sms) {
  const int c = g_choice[slot][idx].load(std::memory_order_relaxed);
  if (c > 0) return c - 1;
  const SizeVariants& sv = host_variants(slot)[idx];
  int best = 0, limit = INT_MAX;
  for (int v = 0; v < sv.count; ++v) {
    const int s = sv.v[v].small_per_sm;
    if (s > 0 && s < limit && batch <= (int64_t)s * sms) {
      best = v;
      limit = s;
    }
  }
  return best;
}

// `host`: in and out are device addresses of pinned host memory (launch_fwd_host).
fftoc_status launch_fwd(int n, const double* in, double* out, int64_t batch, int engine, cudaStream_t stream,
                        int variant = -1, bool host = false) {
  const int idx = size_index(n);
  if (idx < 0) return fail(FFTOC_ERR_INVALID_SIZE, "n=" + std::to_string(n) + " is not one of 8,16,...,4096");
  if (batch < 0) return fail(FFTOC_ERR_INVALID_VALUE, "batch must be >= 0");
  if (engine < FFTOC_ENGINE_AUTO || engine > kLastEngine) return fail(FFTOC_ERR_INVALID_VALUE, "unknown engine");
  if (batch == 0) return FFTOC_OK;
  if (!in || !out) return fail(FFTOC_ERR_INVALID_VALUE, "null buffer");
  if (((uintptr_t)in & 15) || ((uintptr_t)out & 15)) return fail(FFTOC_ERR_MISALIGNED, "buffers must be 16-byte aligned");
  if (batch > INT64_MAX / ((int64_t)n * 16)) return fail(FFTOC_ERR_INVALID_VALUE, "batch*n overflows");
  const uintptr_t bytes = (uintptr_t)batch * (uintptr_t)n * 16u;
  const uintptr_t a = (uintptr_t)in, b = (uintptr_t)out;
  if (a != b && a < b + bytes && b < a + bytes) return fail(FFTOC_ERR_INVALID_VALUE, "in and out overlap partially");

  const int eng = resolve_engine(n, engine);
  if (eng == FFTOC_ENGINE_DMMA) {
    if (variant > 0) return fail(FFTOC_ERR_INVALID_VALUE, "no such plan variant");
    return launch_dmma(n, in, out, batch, stream);
  }
  if (is_split_engine(eng)) return launch_split(n, in, out, batch, split_kind_of(eng), stream);
  DeviceState* ds = nullptr;
  fftoc_status st = device_state(&ds);
  if (st != FFTOC_OK) return st;
  const int slot = eng == FFTOC_ENGINE_FX ? 1 : 0;
  const int var = variant >= 0 ? variant : batch_variant(slot, idx, batch, ds->sms);
  if (var >= ds->var[slot][idx].count) return fail(FFTOC_ERR_INVALID_VALUE, "no such plan variant");
  const KernelDesc& d = ds->var[slot][idx].v[var];
  const void* tw = ds->tw[slot][idx][var];
  const long long tiles = (batch + d.tpb - 1) / d.tpb;
  // host buffers: as many CTAs per SM as hold 8 KB of tiles (launch_fwd_host)
  int smem = d.smem, per_sm = d.blocks_per_sm;
  if (host) {
    const int want = d.tpb * n * 16 >= 8192 ? 1 : 8192 / (d.tpb * n * 16), alone = direct_smem(want);
    if (alone > smem) smem = alone, per_sm = want;
  }
  const long long cap = (long long)ds->sms * per_sm;
  const long long blocks = d.persistent ? (tiles < cap ? tiles : cap) : tiles;
  if (blocks > 0x7FFFFFFFLL) return fail(FFTOC_ERR_INVALID_VALUE, "batch too large for one launch");
  const double2* in2 = reinterpret_cast<const double2*>(in);
  double2* out2 = reinterpret_cast<double2*>(out);
  long long bl = (long long)batch;
  int* err = ds->err;
  int prefetch = host ? 0 : 1;
  void* args[] = {(void*)&in2, (void*)&out2, (void*)&bl, (void*)&tw, (void*)&err, (void*)&prefetch};
  cudaError_t e = launch_overlapped(d.fn, (unsigned)blocks, cap, d.threads, smem, args, stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaLaunchKernel");
  return FFTOC_OK;
}

// Largest batch that plans which spread a warp's access over many transforms
// (N = 16 and 32, 64- and 128-byte pieces) take straight from host memory: over
// the link the pieces cost more than the copies' own overheads at 1 GB (7.0 and
// 7.6 ms against 6.5 staged), less up to some 200 MB (82 MB: 593 and 666 us
// against 810).
constexpr uintptr_t kDirectIoHostBytes = (uintptr_t)128 << 20;

// cuPointerGetAttributes, or null (a driver without it: host buffers are staged).
using PointerAttributes = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
PointerAttributes pointer_attributes() {
  static const PointerAttributes fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found) != cudaSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return found == cudaDriverEntryPointSuccess ? reinterpret_cast<PointerAttributes>(f) : nullptr;
  }();
  return fn;
}

// The device address of `bytes` of host memory at p if all of it is pinned and
// mapped, else null.  By the registrations' ranges: under unified addressing
// the device addresses of a buffer's two ends say nothing of what lies between.
void* mapped_host(const void* p, size_t bytes) {
  const PointerAttributes get = pointer_attributes();
  if (!get) return nullptr;
  return mapped_range(p, bytes, [&](uintptr_t at) {
    CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                  CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                  CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    unsigned type = 0, managed = 0;
    CUdeviceptr dev = 0, start = 0;
    size_t size = 0;
    void* to[] = {&type, &managed, &dev, &start, &size};
    HostRange r = {};
    if (get(5, what, to, (CUdeviceptr)at) != CUDA_SUCCESS) return r;
    // the range's start is the host's address or the device's
    const ptrdiff_t shift = (ptrdiff_t)(dev - (CUdeviceptr)at);
    if (type != CU_MEMORYTYPE_HOST || managed || !dev || size == 0) return r;
    const uintptr_t host = at - start < size ? (uintptr_t)start : (uintptr_t)start - (uintptr_t)shift;
    r = {true, host, size, shift};
    return r;
  });
}

// Host buffers.  The binary64 and fixed-point engines transform pinned memory
// in place of it: one launch whose CTAs load their tile over the host link and
// store the result over it.  One CTA per SM, or as many as hold 8 KB of tiles
// (direct_smem), keep 1.2 to 10 MB in flight, enough for the link's latency: 82 MB
// take 503 us in tiles of 8 KB (N = 64, 128, 256 and 512; 163 GB/s each way, the
// link's rate in both directions at once), 510 to 600 us in 16 to 64 KB (N = 1024,
// 2048 and 4096).  With full occupancy the first wave only reads and the last
// only writes, 20-80 MB each.  Against staging (which pays the copies' launches,
// and a chunk each way outside the overlap), n = 256: 10 KB 19 us against 33,
// 4 MB 45 against 71, 82 MB 504 against 812, 1 GB 6.0 ms against 6.5.  Pageable
// memory and the other engines are staged.
fftoc_status launch_fwd_host(int n, const double* h_in, double* h_out, int64_t batch, int engine,
                             cudaStream_t stream) {
  const int idx = size_index(n);
  if (idx < 0) return fail(FFTOC_ERR_INVALID_SIZE, "n=" + std::to_string(n) + " is not one of 8,16,...,4096");
  if (batch < 0) return fail(FFTOC_ERR_INVALID_VALUE, "batch must be >= 0");
  if (engine < FFTOC_ENGINE_AUTO || engine > kLastEngine) return fail(FFTOC_ERR_INVALID_VALUE, "unknown engine");
  if (batch == 0) return FFTOC_OK;
  if (!h_in || !h_out) return fail(FFTOC_ERR_INVALID_VALUE, "null buffer");
  if (((uintptr_t)h_in & 15) || ((uintptr_t)h_out & 15)) return fail(FFTOC_ERR_MISALIGNED, "buffers must be 16-byte aligned");
  if (batch > INT64_MAX / ((int64_t)n * 16)) return fail(FFTOC_ERR_INVALID_VALUE, "batch*n overflows");
  const uintptr_t bytes = (uintptr_t)batch * (uintptr_t)n * 16u;
  const uintptr_t a = (uintptr_t)h_in, b = (uintptr_t)h_out;
  if (a != b && a < b + bytes && b < a + bytes) return fail(FFTOC_ERR_INVALID_VALUE, "in and out overlap partially");
  DeviceState* ds = nullptr;
  fftoc_status st = device_state(&ds);
  if (st != FFTOC_OK) return st;
  void *d_in = mapped_host(h_in, bytes), *d_out = d_in;
  if (d_in && h_out != h_in) d_out = mapped_host(h_out, bytes);
  const int eng = resolve_engine(n, engine);
  const int slot = eng == FFTOC_ENGINE_FX ? 1 : 0;
  // the plan of a device batch of this count, for every chunk
  const bool planned = eng == FFTOC_ENGINE_FX || eng == FFTOC_ENGINE_F64;
  const int var = planned ? batch_variant(slot, idx, batch, ds->sms) : -1;
  const KernelDesc& plan = ds->var[slot][idx].v[planned ? var : 0];
  if (d_in && d_out && planned &&
      !plan.persistent &&  // bulk copies stay on device memory
      (!(plan.code_flags & FFTOC_CODE_DIRECT_IO) || bytes <= kDirectIoHostBytes))
    return launch_fwd(n, static_cast<const double*>(d_in), static_cast<double*>(d_out), batch, engine, stream, var, true);
  Staging& sg = ds->staging;
  std::call_once(sg.once, [&] { init_staging(sg); });
  if (sg.status != FFTOC_OK) return fail(sg.status, sg.error);

  std::lock_guard<std::mutex> lock(sg.mu);
  // pinned memory: chunks of 1/6 of the batch (2 to 64 MiB) overlap both
  // directions for most of the call (82 MB: 812 us with 64 MiB chunks, 620-640
  // with 8-16 MiB); pageable copies do not overlap
  size_t chunk_bytes = Staging::kChunkBytes;
  if (d_in && d_out) chunk_bytes = std::min(chunk_bytes, std::max((size_t)bytes / 6, (size_t)2 << 20));
  const int64_t chunk = (int64_t)(chunk_bytes / ((size_t)n * 16));
  cudaError_t e;
  if ((e = cudaEventRecord(sg.ev_start, stream)) != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
  if ((e = cudaStreamWaitEvent(sg.s_h2d, sg.ev_start, 0)) != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent");
  int last = 0;
  for (int64_t off = 0, c = 0; off < batch; off += chunk, ++c) {
    const int bi = (int)(c % Staging::kBufs);
    const int64_t cnt = (batch - off) < chunk ? (batch - off) : chunk;
    const size_t nb = (size_t)cnt * (size_t)n * 16;
    const char* src = reinterpret_cast<const char*>(h_in) + (size_t)off * (size_t)n * 16;
    char* dst = reinterpret_cast<char*>(h_out) + (size_t)off * (size_t)n * 16;
    if ((e = cudaStreamWaitEvent(sg.s_h2d, sg.ev_d2h[bi], 0)) != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent");
    if ((e = cudaMemcpyAsync(sg.buf[bi], src, nb, cudaMemcpyHostToDevice, sg.s_h2d)) != cudaSuccess)
      return cuda_fail(e, "cudaMemcpyAsync(H2D)");
    if ((e = cudaEventRecord(sg.ev_h2d[bi], sg.s_h2d)) != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
    if ((e = cudaStreamWaitEvent(sg.s_cmp, sg.ev_h2d[bi], 0)) != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent");
    st = launch_fwd(n, static_cast<const double*>(sg.buf[bi]), static_cast<double*>(sg.buf[bi]), cnt, engine, sg.s_cmp,
                    var);
    if (st != FFTOC_OK) return st;
    if ((e = cudaEventRecord(sg.ev_cmp[bi], sg.s_cmp)) != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
    if ((e = cudaStreamWaitEvent(sg.s_d2h, sg.ev_cmp[bi], 0)) != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent");
    if ((e = cudaMemcpyAsync(dst, sg.buf[bi], nb, cudaMemcpyDeviceToHost, sg.s_d2h)) != cudaSuccess)
      return cuda_fail(e, "cudaMemcpyAsync(D2H)");
    if ((e = cudaEventRecord(sg.ev_d2h[bi], sg.s_d2h)) != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
    last = bi;
  }
  if ((e = cudaStreamWaitEvent(stream, sg.ev_d2h[last], 0)) != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent");
  return FFTOC_OK;
}

// variant < 0: the plan in use, for a batch of `batch` on `sms` SMs if batch >= 0.
fftoc_status plan_query(int n, int engine, int variant, fftoc_plan_info* info, int64_t batch = -1, int sms = 0) {
  const int idx = size_index(n);
  if (idx < 0) return fail(FFTOC_ERR_INVALID_SIZE, "n=" + std::to_string(n) + " is not one of 8,16,...,4096");
  if (!info) return fail(FFTOC_ERR_INVALID_VALUE, "null info");
  if (engine < FFTOC_ENGINE_AUTO || engine > kLastEngine) return fail(FFTOC_ERR_INVALID_VALUE, "unknown engine");
  const int eng = resolve_engine(n, engine);
  if (eng == FFTOC_ENGINE_DMMA) {
    if (variant > 0) return fail(FFTOC_ERR_INVALID_VALUE, "no such plan variant");
    return dmma_plan_info(n, info);
  }
  if (is_split_engine(eng)) {
    if (variant > 0) return fail(FFTOC_ERR_INVALID_VALUE, "no such plan variant");
    const fftoc_status st = split_plan_info(n, split_kind_of(eng), info);
    if (st == FFTOC_OK) info->uneven_variant = -1;  // the uneven path has no split-form kernels
    return st;
  }
  const int slot = eng == FFTOC_ENGINE_FX ? 1 : 0;
  const SizeVariants& sv = host_variants(slot)[idx];
  const int var = variant >= 0 ? variant : batch >= 0 ? batch_variant(slot, idx, batch, sms) : chosen_variant(slot, idx);
  if (var >= sv.count) return fail(FFTOC_ERR_INVALID_VALUE, "no such plan variant");
  const KernelDesc& d = sv.v[var];
  info->n = n;
  info->engine = eng;
  info->threads_per_transform = d.tpt;
  info->transforms_per_block = d.tpb;
  info->threads_per_block = d.threads;
  info->smem_bytes = d.smem;
  info->passes = d.passes;
  for (int i = 0; i < 4; ++i) info->radix[i] = d.radix[i];
  info->points_per_thread = d.ppt;
  info->variant = var;
  info->variants = sv.count;
  info->persistent = d.persistent;
  info->stages = d.stages;
  info->prefetch = d.prefetch;
  info->code_flags = d.code_flags;
  info->uneven_variant = uneven_variant(slot, idx);
  return FFTOC_OK;
}

// Reads and clears the current device's error flags without allocating:
// the allocation-free entry point's flag (if that path was set up on this
// device) and the other paths' flag (if their device state exists; checking
// does not create it, since nothing could have raised a flag that does not
// exist).
fftoc_status device_error_check() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) return fail(FFTOC_ERR_INVALID_VALUE, "device ordinal out of range");
  int h = 0;
  fftoc_status st = noalloc_take_error(dev, &h);
  if (st != FFTOC_OK) return st;
  DeviceState& ds = g_devices[dev];
  if (ds.ready.load(std::memory_order_acquire)) {
    int d = 0;
    e = cudaMemcpy(&d, ds.err, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpy(error flag)");
    if (d != 0) {
      e = cudaMemset(ds.err, 0, sizeof(int));
      if (e != cudaSuccess) return cuda_fail(e, "cudaMemset(error flag)");
    }
    h |= d;
  }
  if (h & kErrTimeout) return fail(FFTOC_ERR_TIMEOUT, "a kernel's bounded wait for its prefetched tile gave up");
  if (h != 0)
    return fail(FFTOC_ERR_INVALID_VALUE, "an uneven batch skipped entries with an unsupported size or a negative offset");
  return FFTOC_OK;
}

fftoc_status plan_select(int n, int engine, int variant) {
  fftoc_plan_info info;
  fftoc_status st = plan_query(n, engine, variant < 0 ? 0 : variant, &info);
  if (st != FFTOC_OK) return st;
  if (variant < 0) return fail(FFTOC_ERR_INVALID_VALUE, "variant must be >= 0");
  // engines with one plan per size (split forms, DMMA) have no choice to store
  if (info.engine == FFTOC_ENGINE_FX || info.engine == FFTOC_ENGINE_F64)
    g_choice[info.engine == FFTOC_ENGINE_FX ? 1 : 0][size_index(n)].store(variant + 1);
  return FFTOC_OK;
}

// The stored choice of (n, engine), or null for an engine with one plan a size.
fftoc_status plan_choice(int n, int engine, std::atomic<int>** choice) {
  fftoc_plan_info info;
  const fftoc_status st = plan_query(n, engine, 0, &info);
  *choice = nullptr;
  if (st == FFTOC_OK && (info.engine == FFTOC_ENGINE_FX || info.engine == FFTOC_ENGINE_F64))
    *choice = &g_choice[info.engine == FFTOC_ENGINE_FX ? 1 : 0][size_index(n)];
  return st;
}

fftoc_status plan_selected(int n, int engine, int* variant) {
  if (!variant) return fail(FFTOC_ERR_INVALID_VALUE, "null variant");
  std::atomic<int>* c;
  const fftoc_status st = plan_choice(n, engine, &c);
  if (st == FFTOC_OK) *variant = c ? c->load() - 1 : -1;
  return st;
}

fftoc_status plan_unselect(int n, int engine) {
  std::atomic<int>* c;
  const fftoc_status st = plan_choice(n, engine, &c);
  if (c) c->store(0);
  return st;
}

// Time every compiled plan of (n, engine) on a device scratch batch of
// `batch` transforms (3 warm-up + 5 timed launches each, on `stream`), select
// the fastest and report it.  Synchronous; allocates and frees the scratch.
fftoc_status autotune(int n, int engine, int64_t batch, cudaStream_t stream, int* best_variant, float* best_ms) {
  fftoc_plan_info info;
  fftoc_status st = plan_query(n, engine, 0, &info);
  if (st != FFTOC_OK) return st;
  if (batch <= 0) return fail(FFTOC_ERR_INVALID_VALUE, "batch must be > 0");
  if (batch > INT64_MAX / ((int64_t)n * 16)) return fail(FFTOC_ERR_INVALID_VALUE, "batch*n overflows");
  const size_t bytes = (size_t)batch * (size_t)n * 16;
  void *x = nullptr, *y = nullptr;
  cudaError_t e = cudaMalloc(&x, bytes);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(autotune)");
  e = cudaMalloc(&y, bytes);
  if (e != cudaSuccess) {
    cudaFree(x);
    return cuda_fail(e, "cudaMalloc(autotune)");
  }
  cudaEvent_t a = nullptr, b = nullptr;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  float best = 1e30f;
  int bestv = 0;
  // deterministic non-trivial input: bytes 0x3F.. give doubles near 0.5
  e = cudaMemsetAsync(x, 0x3F, bytes, stream);
  for (int v = 0; v < info.variants && e == cudaSuccess && st == FFTOC_OK; ++v) {
    for (int r = 0; r < 3 && st == FFTOC_OK; ++r)
      st = launch_fwd(n, (const double*)x, (double*)y, batch, info.engine, stream, v);
    if (st != FFTOC_OK) break;
    cudaEventRecord(a, stream);
    for (int r = 0; r < 5 && st == FFTOC_OK; ++r)
      st = launch_fwd(n, (const double*)x, (double*)y, batch, info.engine, stream, v);
    cudaEventRecord(b, stream);
    e = cudaEventSynchronize(b);
    float ms = 0;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
    if (e == cudaSuccess && ms / 5 < best) {
      best = ms / 5;
      bestv = v;
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(x);
  cudaFree(y);
  if (st != FFTOC_OK) return st;
  if (e != cudaSuccess) return cuda_fail(e, "autotune");
  if (info.engine == FFTOC_ENGINE_FX || info.engine == FFTOC_ENGINE_F64)
    g_choice[info.engine == FFTOC_ENGINE_FX ? 1 : 0][size_index(n)].store(bestv + 1);
  if (best_variant) *best_variant = bestv;
  if (best_ms) *best_ms = best;
  return FFTOC_OK;
}

}  // namespace fftoc

extern "C" {

#define FFTOC_SIZE_ENTRY(N)                                                                       \
  fftoc_status fftoc_c2c_fwd_n##N(const double* in, double* out, int64_t batch, fftoc_stream s) { \
    return fftoc::launch_fwd(N, in, out, batch, FFTOC_ENGINE_AUTO, (cudaStream_t)s);            \
  }
FFTOC_SIZE_ENTRY(8)
FFTOC_SIZE_ENTRY(16)
FFTOC_SIZE_ENTRY(32)
FFTOC_SIZE_ENTRY(64)
FFTOC_SIZE_ENTRY(128)
FFTOC_SIZE_ENTRY(256)
FFTOC_SIZE_ENTRY(512)
FFTOC_SIZE_ENTRY(1024)
FFTOC_SIZE_ENTRY(2048)
FFTOC_SIZE_ENTRY(4096)
#undef FFTOC_SIZE_ENTRY

fftoc_status fftoc_c2c_fwd(int n, const double* in, double* out, int64_t batch, fftoc_stream s) {
  return fftoc::launch_fwd(n, in, out, batch, FFTOC_ENGINE_AUTO, (cudaStream_t)s);
}

fftoc_status fftoc_c2c_fwd_ex(int n, const double* in, double* out, int64_t batch, int engine, fftoc_stream s) {
  return fftoc::launch_fwd(n, in, out, batch, engine, (cudaStream_t)s);
}

fftoc_status fftoc_c2c_fwd_host(int n, const double* h_in, double* h_out, int64_t batch, int engine, fftoc_stream s) {
  return fftoc::launch_fwd_host(n, h_in, h_out, batch, engine, (cudaStream_t)s);
}

fftoc_status fftoc_plan_query(int n, int engine, fftoc_plan_info* info) { return fftoc::plan_query(n, engine, -1, info); }

fftoc_status fftoc_plan_query_variant(int n, int engine, int variant, fftoc_plan_info* info) {
  return fftoc::plan_query(n, engine, variant, info);
}

fftoc_status fftoc_plan_query_batch(int n, int engine, int64_t batch, int sms, fftoc_plan_info* info) {
  if (batch < 0 || sms < 1) return fftoc::fail(FFTOC_ERR_INVALID_VALUE, "batch must be >= 0 and sms >= 1");
  return fftoc::plan_query(n, engine, -1, info, batch, sms);
}

fftoc_status fftoc_plan_select(int n, int engine, int variant) { return fftoc::plan_select(n, engine, variant); }

fftoc_status fftoc_plan_selected(int n, int engine, int* variant) { return fftoc::plan_selected(n, engine, variant); }

fftoc_status fftoc_plan_unselect(int n, int engine) { return fftoc::plan_unselect(n, engine); }

fftoc_status fftoc_device_error_check(void) { return fftoc::device_error_check(); }

fftoc_status fftoc_autotune(int n, int engine, int64_t batch, fftoc_stream s, int* best_variant, float* best_ms) {
  return fftoc::autotune(n, engine, batch, (cudaStream_t)s, best_variant, best_ms);
}

int fftoc_auto_engine(int n) { return fftoc::size_index(n) < 0 ? -1 : FFTOC_ENGINE_FX; }

const char* fftoc_status_string(fftoc_status s) {
  switch (s) {
    case FFTOC_OK: return "ok";
    case FFTOC_ERR_INVALID_SIZE: return "invalid size";
    case FFTOC_ERR_INVALID_VALUE: return "invalid value";
    case FFTOC_ERR_MISALIGNED: return "misaligned buffer";
    case FFTOC_ERR_NO_MEMORY: return "out of device memory";
    case FFTOC_ERR_CUDA: return "CUDA error";
    case FFTOC_ERR_TIMEOUT: return "device wait timed out";
    case FFTOC_ERR_UNSUPPORTED: return "unsupported";
  }
  return "unknown status";
}

const char* fftoc_last_error_string(void) { return fftoc::t_last_error.c_str(); }

int fftoc_version(void) { return FFTOC_VERSION; }

}  // extern "C"
