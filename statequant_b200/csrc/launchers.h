// Launchers of the staged decode-step kernels (one translation unit per recurrence kind, so that they compile in
// parallel) and of the fold kernel.  Return 0: launched; 1: the kernel does not take this shape (the caller falls back);
// < 0: -(1000 + cudaError_t).
#pragma once
#include <atomic>
#include <cuda_runtime.h>
#include "delta_step.cuh"

namespace sqb {
// cudaFuncAttributeMaxDynamicSharedMemorySize is a per-device setting of a kernel: remember, per device, the largest
// size already set, so that the attribute call is made only when a launch needs more on the device it runs on.
struct SmemLimit {
  std::atomic<int> set[64];
  template <class K>
  cudaError_t ensure(K kern, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool cached = dev >= 0 && dev < 64;
    if (cached && bytes <= set[dev].load(std::memory_order_relaxed)) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && cached) set[dev].store(bytes, std::memory_order_relaxed);
    return e;
  }
};
// Launch in plain stream order: the grid's CTAs enter once the kernel in front of it has finished.
template <class... P, class... A>
cudaError_t launch_plain(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}
// Launch with programmatic stream serialisation: the grid's CTAs may be scheduled before the kernel in front of it has
// finished; the kernel itself waits for that (dependency_wait in common.cuh) before it touches memory.
template <class... P, class... A>
cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const A&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}
// CTAs of a kernel that the current device holds at once, asked once per device and shared-memory size.
struct Residency {
  std::atomic<long long> known[64];              // smem << 32 | CTAs
  template <class K>
  long long ctas(K kern, int threads, int smem) {
    int dev = 0, nsm = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    const long long k = known[dev & 63].load(std::memory_order_relaxed);
    if (dev < 64 && k != 0 && (k >> 32) == smem) return k & 0xFFFFFFFFll;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem) != cudaSuccess)
      return 0;
    const long long all = static_cast<long long>(nsm) * n;
    if (dev < 64) known[dev].store(static_cast<long long>(smem) << 32 | all, std::memory_order_relaxed);
    return all;
  }
};
// Whether a step kernel of `grid` CTAs enters early, where the GPU holds `all`: the CTAs of two launches find room side by side up to
// half of it, and from about 0.8 of it on they fill every SM however they come in.  Between the two they crowd on the SMs that are
// free first.  us per layer-step in stream order / early, all slots due together: tensor-core kernel, int4 k/64 (740 at once) 320 CTAs
// 6.4 / 6.0, 384 6.5 / 7.6, 576 7.6 / 7.9, 640 8.3 / 7.9, 1024 12.6 / 12.1; int8 v/32 (592) 288 CTAs 6.7 / 6.2, 304 7.4 / 8.3, 384 7.6 /
// 8.3, 512 8.9 / 8.6; Mamba2 int8 320 6.5 / 6.0, 384 6.5 / 7.7, 640 8.6 / 8.3; register tile, int8 k/32 (592) 288 CTAs 4.3 / 3.9, 320 4.9 /
// 5.2, 416 5.0 / 5.3, 512 5.7 / 5.3; bf16 1024 10.3 / 10.0.  KDA (one head per CTA: the folding ones end the launch) crowds up to a whole
// wave where slots are due one in eight: int4 608 CTAs 11.3 / 12.2, 736 12.1 / 12.7 (all due 7.3 / 7.2, 7.9 / 7.4), 1024 (1036 at once)
// 14.4 / 15.5.
inline bool enters_early(long long grid, long long all, bool kda) { return 2 * grid <= all || (kda ? grid > all : 5 * grid > 4 * all); }

// bf16 activations and output with q and k rows on 8-byte boundaries: the step kernels have instances of their own for these.
inline bool bf16_io(const StepArgs& a) {
  return a.dt_qk == DT_BF16 && a.dt_v == DT_BF16 && a.dt_out == DT_BF16 &&
         ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | static_cast<uintptr_t>(a.sq) | static_cast<uintptr_t>(a.sk)) & 7) == 0;
}

// Shapes the register-tile step takes: d_k 128 and d_v 64 or 128 with bf16 states or (Gated DeltaNet, Mamba2) 8-bit codes in
// key groups of 32 or 4-bit codes in key groups of 64; Gated DeltaNet states of d_k 96 and d_v 64, 128 or 192 with those codes;
// decays per head, int8 buffer of 8, q / k per key head, a CTA's rows of one key head.
inline bool reg_shape_ok(const StepArgs& a, int bits, bool axk, int kind) {
  if (kind == K_KDA || !a.qbuf || a.M != 8 || (!a.per_key_head && a.HV != a.HK)) return false;
  if (bits != 16 && !(axk && ((bits == 8 && a.group == 32) || (bits == 4 && a.group == 64)))) return false;
  const bool wide = a.DK == 128 && (a.DV == 64 || a.DV == 128);
  const bool odd = a.DK == 96 && bits != 16 && kind == K_GDN && (a.DV == 64 || a.DV == 128 || a.DV == 192);
  if (!wide && !odd) return false;
  // a row's scales are one 4- or 8-byte load where there are two or four of them
  const int ng = bits == 16 ? 1 : a.DK == 96 ? (bits == 8 ? 1 : 2) : a.DK / a.group;
  if ((reinterpret_cast<uintptr_t>(a.SC) | static_cast<uintptr_t>(a.sSC)) % (2 * ng)) return false;
  const int hps = a.DV == 64 ? 2 : 1;
  return (a.HV / a.HK) % hps == 0 && a.HV / hps <= 65535;
}
struct GgaArgs;
// the GGA step with the tile in registers (gga_reg.cuh): 0, 1 = shape not taken, -1000 - cudaError
int launch_gga_reg(const GgaArgs& a, long long ctas, cudaStream_t stream);
// the step with the state held in registers (step_reg.cuh), on shapes that reg_shape_ok takes
int launch_reg(int kind, const StepArgs& a, int bits, cudaStream_t stream);
int launch_staged_gdn(const StepArgs& a, int bits, bool axk, cudaStream_t stream);
int launch_staged_m2(const StepArgs& a, int bits, bool axk, cudaStream_t stream);
int launch_staged_kda(const StepArgs& a, int bits, bool axk, cudaStream_t stream);
// the tensor-core kernels (step_mma.cuh); mode 0: the step alone (the fold launch follows), 3: the step with the fold
// of a slot's m-th token inside
int launch_mma_gdn(const StepArgs& a, int bits, int mode, cudaStream_t stream);
int launch_mma_m2(const StepArgs& a, int bits, int mode, cudaStream_t stream);
int launch_mma_kda(const StepArgs& a, int bits, int mode, cudaStream_t stream);
// the fold launch that follows a staged step (that kernel only appends on a slot's m-th token)
int launch_fold(int kind, const StepArgs& a, int bits, bool axk, cudaStream_t stream);
// the fold kernel in its read-out mode: out fp32 [rows, HV, d_v, d_k] = the state advanced across its pending buffer
int launch_read(int kind, const StepArgs& a, int bits, bool axk, float* out, cudaStream_t stream);
// pack canonical fp32 states X [rows, HV, d_v, d_k] into the slots and empty their buffers
int launch_write(int kind, const StepArgs& a, int bits, bool axk, const float* X, cudaStream_t stream);
}  // namespace sqb
