// RMS norm of the activation rows ahead of a projection (reference: MLXFast.rmsNorm in
// DecoderLayer.callAsFunction, Sources/IshizukiKit/Text/TextModel.swift:151-161): the residual
// stream is fp32 (or fp16), the normalised rows leave in fp16, the width the projections read.
//   y[r][i] = fp16( x[r][i] * rsqrt(mean_i x[r][i]^2 + eps) * w[i] ), arithmetic in fp32.
// Its own launch: the norm needs the whole row's sum of squares before the first value can be
// staged, which a product kernel's CTAs (each reads only its column range, or would all have to read
// the whole fp32 row first) cannot get cheaply. Launched with programmatic stream serialization and
// itself releasing its dependents at once, it overlaps the tail of the launch before and the
// prologue of the product after it.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "ishi_kernels.h"

namespace ishi {

namespace {

template <class T>
__device__ __forceinline__ float to_float(T v) { return (float)v; }
template <>
__device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// A row is a cluster of CTAs of 128 threads, eight values per thread in 16-byte loads, held in registers between the
// two passes. Bound by latency alone (a row is 10-20 KB): x and w are hinted into L2 ahead of the wait
// (hints only: either may be the output of the launch before), the rest is one exchange of the warps' sums through
// distributed shared memory and one cluster barrier. The CTAs are as small as the product kernel's leave room for: 4096
// registers (20 warps of 96, 24 of 80, 16 of 120; 16 warps of 128, as Q6_K has at nine to sixteen rows, leave none) and 1280 bytes of
// shared memory of an SM. So most sit beside the products: one CTA of 1024 threads per row kept its SM from the product
// behind it, whose CTA there started 3 us and was ready 1.2 us after the others.
// Two decoder layers of the 27B shape, four norms: Q4_K at eight rows 110.7 -> 109.0 us, at one 103.4 -> 102.2, ternary at four 96.5 -> 95.0.
// Sums: a warp's 256 squares, then the warps' sums, each by a butterfly, whatever the number of CTAs.
constexpr int kNormThreads = 128, kNormPer = 8, kNormWarps = 32;  // threads of a CTA, values of one, most warps of a row

template <class T>
__device__ __forceinline__ void load8_raw(const T *p, T (&v)[kNormPer]) {
  uint4 raw[sizeof(T) / 2];
#pragma unroll
  for (int i = 0; i < (int)(sizeof(T) / 2); ++i) raw[i] = reinterpret_cast<const uint4 *>(p)[i];
  memcpy(v, raw, sizeof(v));
}
template <class T>
__device__ __forceinline__ void load8(const T *p, float (&v)[kNormPer]) {
  T t[kNormPer];
  load8_raw(p, t);
#pragma unroll
  for (int i = 0; i < kNormPer; ++i) v[i] = to_float(t[i]);
}

// WIDE: width a multiple of eight, all pointers 16-byte aligned; else value by value
template <class XT, class WT, bool WIDE>
__global__ void __launch_bounds__(kNormThreads, 16) rms_norm_kernel(const XT *__restrict__ x, const WT *__restrict__ w, long long width, float eps,
                                                                    int ctas, __half *__restrict__ y) {
  __shared__ float part[kNormWarps];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int r = (int)(blockIdx.x / (unsigned)ctas), c = (int)blockIdx.x - r * ctas, lane = (int)threadIdx.x & 31;
  const int i0 = (c * kNormThreads + (int)threadIdx.x) * kNormPer, n = (int)min((long long)kNormPer, width - i0);
  const XT *row = x + (long long)r * width;
  if (n > 0) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(w + i0));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(row + i0));
  }
  if (threadIdx.x < kNormWarps) part[threadIdx.x] = 0.f;  // (of warps that the row does not have)
  // the CTAs of the row run and their sums are cleared (waited for ahead of the first sum)
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // x may be the output of the launch before
  float v[kNormPer] = {};
  if (WIDE) {
    if (n > 0) load8(row + i0, v);
  } else {
#pragma unroll
    for (int j = 0; j < kNormPer; ++j)
      if (j < n) v[j] = to_float(row[i0 + j]);
  }
  WT f[kNormPer];
  if (WIDE) {
    if (n > 0) load8_raw(w + i0, f);
  } else {
#pragma unroll
    for (int j = 0; j < kNormPer; ++j)
      if (j < n) f[j] = w[i0 + j];
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kNormPer; ++j) ss = fmaf(v[j], v[j], ss);
#pragma unroll
  for (int d = 16; d; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (lane < ctas) {  // to every CTA of the row
    uint32_t at = (uint32_t)__cvta_generic_to_shared(part + c * (kNormThreads / 32) + ((int)threadIdx.x >> 5));
    asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(at) : "r"(lane));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(ss) : "memory");
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  float total = part[lane];
#pragma unroll
  for (int d = 16; d; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
  const float s = rsqrtf(total / (float)width + eps);
  __half *out = y + (long long)r * width + i0;
  __half h[kNormPer];
#pragma unroll
  for (int j = 0; j < kNormPer; ++j) h[j] = __float2half_rn(v[j] * s * to_float(f[j]));
  if (WIDE) {
    if (n > 0) {
      uint4 o;
      memcpy(&o, h, sizeof(o));
      *reinterpret_cast<uint4 *>(out) = o;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kNormPer; ++j)
      if (j < n) out[j] = h[j];
  }
}

template <class XT, class WT>
cudaError_t launch_as(const void *x, const void *w, long long rows, long long width, float eps, __half *y, cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  const int ctas = (int)((width + kNormThreads * kNormPer - 1) / (kNormThreads * kNormPer));  // at most 8: rms_norm_max_width()
  cfg.gridDim = dim3((unsigned)(rows * ctas));
  cfg.blockDim = dim3(kNormThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)ctas;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  const bool wide = width % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0;
  return cudaLaunchKernelEx(&cfg, wide ? rms_norm_kernel<XT, WT, true> : rms_norm_kernel<XT, WT, false>, static_cast<const XT *>(x),
                            static_cast<const WT *>(w), width, eps, ctas, y);
}

}  // namespace

namespace {

// The inputs of a host batch, a kernel between two products that copies those of the next few. The copy
// engine takes 4.7 us a copy on top of the bytes and an event between two products, which idles the
// SMs for 2.5 us; this kernel is a link of the chain of programmatic launches and runs beside the
// product before it, whose CTAs leave 4096 registers (most of them, see above) and 1280 bytes of shared memory of an SM free: a CTA
// of this kernel. The copies are one range of 16-byte pieces over all CTAs: one after the other, each
// would add the bus's 2 us of latency. 32 CTAs keep 128 KB on the way; 16 are slower by 8 % of a
// whole batch, more gain nothing. (Outputs stay with the copy engine: written to the host by a
// kernel, they hold up the product's loads, 45 us in a batch of 16 entries.)
constexpr int kCopyThreads = 128, kCopyBlocks = 32;

__global__ void __launch_bounds__(kCopyThreads, 16) host_copy_kernel(const HostCopies c) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (c.wait) asm volatile("griddepcontrol.wait;" ::: "memory");
  constexpr int kStep = kCopyThreads * kCopyBlocks, kBatch = 2;
  int job = 0, base = 0;  // the job the next piece lies in, its first piece
  auto piece = [&](int i) {  // moves on to piece i; false past the end
    while (job < c.count && i >= base + (int)(c.bytes[job] / 16u)) base += (int)(c.bytes[job++] / 16u);
    return job < c.count;
  };
  for (int i0 = (int)(blockIdx.x * kCopyThreads + threadIdx.x); piece(i0); i0 += kStep * kBatch) {
    uint4 v[kBatch], *dst[kBatch];
#pragma unroll
    for (int e = 0; e < kBatch; ++e) {
      const int i = i0 + e * kStep;
      dst[e] = nullptr;
      if (piece(i)) {
        dst[e] = static_cast<uint4 *>(c.dst[job]) + (i - base);
        v[e] = __ldcv(static_cast<const uint4 *>(c.src[job]) + (i - base));
      }
    }
#pragma unroll
    for (int e = 0; e < kBatch; ++e)
      if (dst[e]) *dst[e] = v[e];
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the chain: whoever waits for this kernel waits for all before it
}

}  // namespace

cudaError_t launch_host_copies(const HostCopies &copies, cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(kCopyBlocks);
  cfg.blockDim = dim3(kCopyThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, host_copy_kernel, copies);
}

long long rms_norm_max_width() { return (long long)kNormWarps * 32 * kNormPer; }

// dtypes: 0 fp16, 1 bf16, 2 fp32
cudaError_t launch_rms_norm(const void *x, int x_dtype, const void *w, int w_dtype, long long rows, long long width, float eps,
                            __half *y, cudaStream_t st) {
  if (rows == 0) return cudaSuccess;
  if (x_dtype == 2) {
    if (w_dtype == 2) return launch_as<float, float>(x, w, rows, width, eps, y, st);
    if (w_dtype == 1) return launch_as<float, __nv_bfloat16>(x, w, rows, width, eps, y, st);
    return launch_as<float, __half>(x, w, rows, width, eps, y, st);
  }
  if (x_dtype == 0) {
    if (w_dtype == 2) return launch_as<__half, float>(x, w, rows, width, eps, y, st);
    if (w_dtype == 1) return launch_as<__half, __nv_bfloat16>(x, w, rows, width, eps, y, st);
    return launch_as<__half, __half>(x, w, rows, width, eps, y, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace ishi
