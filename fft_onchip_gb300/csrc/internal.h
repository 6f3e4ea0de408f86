// fftoc — declarations shared by the host translation units.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/fftoc.h"

namespace fftoc {

constexpr int kNumSizes = 10;
constexpr int kSizes[kNumSizes] = {8, 16, 32, 64, 128, 256, 512, 1024, 2048, 4096};

inline int size_index(int n) {
  for (int i = 0; i < kNumSizes; ++i)
    if (kSizes[i] == n) return i;
  return -1;
}

// One compiled kernel (an engine x plan instantiation).
struct KernelDesc {
  const void* fn = nullptr;  // __global__ function
  int threads = 0;           // threads per CTA
  int tpb = 0;               // transforms per CTA
  int smem = 0;              // dynamic shared memory bytes
  int tpt = 0;               // threads per transform
  int ppt = 0;               // points per thread
  int passes = 0;
  int radix[4] = {1, 1, 1, 1};
  int tw_entries = 0;        // twiddle table entries
  int natural = 0;           // 1: fixed-point table in the natural-word layout (EngFxN)
  int tangent = 0;           // 1: binary64 table with EngF64's tangent forms
  int persistent = 0;        // 1: grid-stride persistent CTAs with TMA prefetch (extra error-flag argument)
  int stages = 0;            // shared-memory stages of the persistent kernel
  int blocks_per_sm = 0;     // resident CTAs per SM (filled at device set-up)
  int prefetch = 0;          // 1: L2 prefetch one wave ahead (Prefetched<> plans)
  int code_flags = 0;        // FFTOC_CODE_* bits of the plan
  int uneven_default = 0;    // 1: the uneven path's default plan for this size (UnevenDefault<>)
  int small_per_sm = 0;      // > 0: the default plan of batches up to this many transforms per SM (SmallBatch<>)
  // uneven-batch kernel of the same plan (nullptr for TMA-prefetching plans)
  const void* fn_uneven = nullptr;
  int smem_uneven = 0;
  int blocks_per_sm_uneven = 0;
  // on-chip repeat kernel of the same plan (nullptr for TMA-prefetching plans)
  const void* fn_onchip = nullptr;
  int smem_onchip = 0;
};

constexpr int kMaxVariants = 12;
struct SizeVariants {
  int count = 0;
  KernelDesc v[kMaxVariants];
};

// Fill `per_size[kNumSizes]` with the compiled plans of an engine
// (kernels_<engine>.cu); variant 0 is the default choice.
void describe_f64(SizeVariants* per_size);
void describe_fx(SizeVariants* per_size);
// Same walk over the plan list, filling only fn_uneven / smem_uneven
// (kernels_uneven_<engine>.cu).
void describe_uneven_f64(SizeVariants* per_size);
void describe_uneven_fx(SizeVariants* per_size);
void describe_onchip_f64(SizeVariants* per_size);
void describe_onchip_fx(SizeVariants* per_size);

// Split-precision form: one compiled plan per size (fn == nullptr: none).
struct SplitDesc {
  const void* fn = nullptr;          // the kernel of plain launches
  const void* fn_overlap = nullptr;  // and of overlapped ones (launch_overlapped)
  int threads = 0, tpb = 0, smem = 0, passes = 0;
  int radix[4] = {1, 1, 1, 1};
  int tw_entries = 0;  // FP32 twiddles (8 bytes each)
  int b_bytes = 0;     // DFT-matrix operand slices
  int esize = 0, slices = 0;
  int blocks_per_sm = 0;
};
// kernels_split.cu; kind 1 = BF16x3, 2 = TF32x2, 3 = exact slices
void describe_split(int kind, SplitDesc* per_size);
// api_split.cu; kind = fftoc_split_kind
bool split_supported(int n, int kind);
fftoc_status split_plan_info(int n, int kind, fftoc_plan_info* info);
fftoc_status launch_split(int n, const double* in, double* out, int64_t batch, int kind, cudaStream_t stream);
inline bool is_split_engine(int engine) {
  return engine == FFTOC_ENGINE_SPLIT_BF16X3 || engine == FFTOC_ENGINE_SPLIT_TF32X2 ||
         engine == FFTOC_ENGINE_SPLIT_EXACT;
}
inline int split_kind_of(int engine) {
  return engine == FFTOC_ENGINE_SPLIT_BF16X3   ? FFTOC_SPLIT_BF16X3
         : engine == FFTOC_ENGINE_SPLIT_TF32X2 ? FFTOC_SPLIT_TF32X2
                                               : FFTOC_SPLIT_EXACT;
}
constexpr int kLastEngine = FFTOC_ENGINE_SPLIT_EXACT;

// Resident CTAs per SM of a persistent kernel, and the shared-memory carveout
// that holds exactly that many (the rest of the SM's memory stays L1).  The
// occupancy query applies neither a function's carveout preference nor, for
// kernels that use tcgen05 (it returns 1 for them at any size), the actual
// limits, so the CTAs are computed here: the smallest of the register-file
// limit (registers per thread rounded to the 256-register warp allocation
// unit, 64K registers per SM), the thread limit (2048 per SM) and the
// shared-memory limit of the largest carveout.  The carveout is then set to
// the smallest percentage of the SM's shared memory that holds them.
inline cudaError_t fit_carveout(const void* fn, int threads, int smem, int* blocks_per_sm) {
  int dev = 0, smem_sm = 0, reserved = 0, regs_sm = 0, threads_sm = 0;
  cudaFuncAttributes fa;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&threads_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
  if (e != cudaSuccess) return e;
  const int warps = (threads + 31) / 32;
  const int regs_warp = ((fa.numRegs * 32 + 255) / 256) * 256;
  int by_regs = regs_warp > 0 ? regs_sm / (regs_warp * warps) : 32;
  const int by_threads = threads_sm / (warps * 32);
  if (by_threads < by_regs) by_regs = by_threads;
  const int by_smem = smem_sm / (smem + reserved);
  int b = by_regs < by_smem ? by_regs : by_smem;
  if (b < 1) b = 1;
  *blocks_per_sm = b;
  const long long need = (long long)b * (smem + reserved);
  int pct = (int)((100 * need + smem_sm - 1) / smem_sm);
  if (pct > 100) pct = 100;
  return cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
}

// Dynamic shared memory of a launch on host buffers, so large that `per_sm` CTAs
// run per SM and no more (of its 228 KB, 1 KB of them the system's in each CTA).
constexpr int direct_smem(int per_sm) { return (228 << 10) / (per_sm + 1) + 1024; }
constexpr int kDirectSmem = direct_smem(1);
// Dynamic shared-memory limit of a batched kernel: its own and that of its
// launches on host buffers.  Every set-up of such a kernel sets this same
// limit (the attribute belongs to the function, the last call wins).
inline cudaError_t allow_shared(const void* fn, int smem) {
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem > kDirectSmem ? smem : kDirectSmem);
}

// Launch of a kernel that calls after_previous() before it touches the
// caller's buffers: it may be scheduled while the kernel before it in the
// stream drains, which hides the launch and the fill of the first wave: 2-4 us
// a call back to back (N = 64, 64 MiB: 28.6 -> 26.0 us; N = 1024, 82 MB: 41.0
// -> 38.4 us; 1,024 transforms of 512 points: 8.2 -> 5.4 us).
// `wave` is the number of CTAs that fit the device at once.  A grid of 1/2 to
// 2/3 of it is launched without the overlap: two such grids do not fit
// together, so the next one's CTAs crowd on some SMs, and back to back that
// measured up to 14 % slower for the fixed-point plans of N = 256, 512, 1024 and
// 2048 (7-15 % faster at 64, 128 and 4096); below and above the overlap wins at
// every N, by 3-70 %.  The rule goes by the grid alone.  Where it keeps such grids
// of the split kernels and of host buffers from the overlap, they would gain:
// BF16x3 and the exact slices 10 to 30 % (512 points 10.3 against 8.1 us and
// 14.4 against 11.0), TF32x2 at N = 16 and 4096 as much, host buffers 5 to 20 %
// up to N = 1024 and -3 to 4 % above.
inline cudaError_t launch_overlapped(const void* fn, unsigned blocks, long long wave, int threads, int smem,
                                     void** args, cudaStream_t stream, bool overlap = true) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = !overlap || (2LL * blocks > wave && 25LL * blocks <= 17 * wave) ? 0 : 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// Device error-flag bits (the flag is returned by fftoc_device_error_check).
constexpr int kErrTimeout = 1;        // a bounded wait for a prefetched tile gave up
constexpr int kErrUnevenSkipped = 2;  // uneven-batch entries with a bad size or offset were skipped

// api_dmma.cu: FFTOC_ENGINE_DMMA (n = 8)
bool dmma_supported(int n);
fftoc_status dmma_plan_info(int n, fftoc_plan_info* info);
fftoc_status launch_dmma(int n, const double* in, double* out, int64_t batch, cudaStream_t stream);

// api.cu accessors: compiled plans per engine slot (0 F64, 1 FX), twiddle
// tables of a plan (double2, or int32 limbs: build_twiddles), the plan
// currently chosen for (slot, size index), the plan of a batch on a device of
// `sms` SMs, AUTO resolution, and the per-thread error message.
const SizeVariants* compiled_variants(int eng_slot);
void twiddle_tables(const KernelDesc& d, std::vector<double>& f64, std::vector<int>& fx);
int chosen_variant(int eng_slot, int idx);
int batch_variant(int eng_slot, int idx, int64_t batch, int sms);
int resolved_engine(int n, int engine);
// The current device's twiddle table of plan (slot, size index, variant), its
// error flag and SM count (device set-up on first use).
fftoc_status device_plan_resources(int slot, int idx, int var, const void** tw, int** err, int* sms);
fftoc_status set_error(fftoc_status st, const std::string& msg);
// api_noalloc.cu: read (into *flags) and clear the allocation-free entry
// point's device error flag of device `dev`; *flags = 0 if that path has not
// been set up there.  Allocates nothing.
fftoc_status noalloc_take_error(int dev, int* flags);
// Plan variant the uneven-batch path uses for (engine slot, size index), or -1.
int uneven_variant(int slot, int idx);

}  // namespace fftoc
