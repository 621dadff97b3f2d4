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

// One CTA of 1024 threads per row, eight values each in 16-byte loads; the row stays in registers
// between the two passes. Bound by latency alone (a row is 10-20 KB): x and w are on their way together
// as soon as the launch before is done, w already hinted into L2 (its values are read after the wait, they
// may be that launch's as well), and the rest is one barrier. Two decoder layers of the 27B shape, four
// norms, in Q4_K: 122.8 us at eight rows and 112.3 at one with 256 threads reading value by value and w
// after the sum, 117.2 and 106.3 this way. The squares add up in another order than with 256 threads,
// which moves a row's factor by its last bit now and then: of 4.1 million values at eight widths 260
// are not the 64-bit result rounded, 288 before.
constexpr int kNormThreads = 1024, kNormPer = 8;

template <class T>
__device__ __forceinline__ void load8(const T *p, float (&v)[kNormPer]) {
  uint4 raw[sizeof(T) / 2];
#pragma unroll
  for (int i = 0; i < (int)(sizeof(T) / 2); ++i) raw[i] = reinterpret_cast<const uint4 *>(p)[i];
  const T *t = reinterpret_cast<const T *>(raw);
#pragma unroll
  for (int i = 0; i < kNormPer; ++i) v[i] = to_float(t[i]);
}

// WIDE: width a multiple of eight, all pointers 16-byte aligned; else value by value
template <class XT, class WT, bool WIDE>
__global__ void __launch_bounds__(kNormThreads) rms_norm_kernel(const XT *__restrict__ x, const WT *__restrict__ w, long long width, float eps,
                                                                __half *__restrict__ y) {
  __shared__ float part[32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int i0 = (int)threadIdx.x * kNormPer, n = (int)min((long long)kNormPer, width - i0);
  if (n > 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + i0));
  asm volatile("griddepcontrol.wait;" ::: "memory");  // x may be the output of the launch before
  const XT *row = x + (long long)blockIdx.x * width;
  float v[kNormPer] = {}, f[kNormPer] = {};
  if (WIDE) {
    if (n > 0) load8(row + i0, v), load8(w + i0, f);
  } else {
#pragma unroll
    for (int j = 0; j < kNormPer; ++j)
      if (j < n) v[j] = to_float(row[i0 + j]), f[j] = to_float(w[i0 + j]);
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kNormPer; ++j) ss = fmaf(v[j], v[j], ss);
#pragma unroll
  for (int d = 16; d; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float total = part[threadIdx.x & 31];
#pragma unroll
  for (int d = 16; d; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
  const float r = rsqrtf(total / (float)width + eps);
  __half *out = y + (long long)blockIdx.x * width + i0;
  __half h[kNormPer];
#pragma unroll
  for (int j = 0; j < kNormPer; ++j) h[j] = __float2half_rn(v[j] * r * f[j]);
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
  cfg.gridDim = dim3((unsigned)rows);
  cfg.blockDim = dim3(kNormThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const bool wide = width % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0;
  return cudaLaunchKernelEx(&cfg, wide ? rms_norm_kernel<XT, WT, true> : rms_norm_kernel<XT, WT, false>, static_cast<const XT *>(x),
                            static_cast<const WT *>(w), width, eps, y);
}

}  // namespace

namespace {

// The inputs of a host batch, a kernel between two products that copies those of the next few. The copy
// engine takes 4.7 us a copy on top of the bytes and an event between two products, which idles the
// SMs for 2.5 us; this kernel is a link of the chain of programmatic launches and runs beside the
// product before it, whose CTAs leave 4096 registers and 1 KB of shared memory of an SM free: a CTA
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

long long rms_norm_max_width() { return (long long)kNormThreads * kNormPer; }

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
