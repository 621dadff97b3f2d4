// Kernels that serve every GGML block format through the shared eight-weight decoders: dense
// decode, embedding-row gather, a one-warp-per-output-row product for the formats without a
// streaming kernel of their own, and the arg-max over a row of logits.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "ggml_decode.cuh"
#include "ishi_kernels.h"

namespace ishi {

namespace {

// Eight consecutive outputs, rounded once: 16-byte stores where the array allows.
__device__ __forceinline__ void store8(float *y, const float (&w)[8], bool wide) {
  if (wide) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(y), "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3]), "f"(w[4]),
                 "f"(w[5]), "f"(w[6]), "f"(w[7])
                 : "memory");
    return;
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) y[e] = w[e];
}
template <class H, class Round>
__device__ __forceinline__ void store8_half(H *y, const float (&w)[8], bool wide, Round &&round) {
  H h[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) h[e] = round(w[e]);
  if (wide) {
    uint4 v;
    memcpy(&v, h, 16);
    __stcs(reinterpret_cast<uint4 *>(y), v);
    return;
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) y[e] = h[e];
}
__device__ __forceinline__ void store8(__half *y, const float (&w)[8], bool wide) {
  store8_half(y, w, wide, [](float v) { return __float2half_rn(v); });
}
__device__ __forceinline__ void store8(__nv_bfloat16 *y, const float (&w)[8], bool wide) {
  store8_half(y, w, wide, [](float v) { return __float2bfloat16_rn(v); });
}

// `bytes` (even) bytes from anywhere into shared memory at a 16-byte boundary, by one warp, in the
// widest pieces the source's alignment allows.
__device__ __forceinline__ void stage_bytes(uint32_t dst, const uint8_t *src, int bytes, int lane) {
  const uint32_t low = (uint32_t)reinterpret_cast<uintptr_t>(src);
  int done = 0;
  if ((low & 15u) == 0) {
    constexpr int kAhead = 4;  // 8 blocks of any type in one batch of loads
    for (int i0 = lane * 16; i0 < (bytes & ~15); i0 += kAhead * 512) {
      uint4 v[kAhead];
#pragma unroll
      for (int e = 0; e < kAhead; ++e)
        if (i0 + e * 512 + 16 <= bytes) v[e] = __ldg(reinterpret_cast<const uint4 *>(src + i0 + e * 512));
#pragma unroll
      for (int e = 0; e < kAhead; ++e)
        if (i0 + e * 512 + 16 <= bytes) sts128u(dst + i0 + e * 512, v[e]);
    }
    done = bytes & ~15;
  } else if ((low & 3u) == 0) {
    constexpr int kAhead = 7;
    for (int i0 = lane * 4; i0 < (bytes & ~3); i0 += kAhead * 128) {
      uint32_t v[kAhead];
#pragma unroll
      for (int e = 0; e < kAhead; ++e)
        if (i0 + e * 128 + 4 <= bytes) v[e] = __ldg(reinterpret_cast<const uint32_t *>(src + i0 + e * 128));
#pragma unroll
      for (int e = 0; e < kAhead; ++e)
        if (i0 + e * 128 + 4 <= bytes) sts32(dst + i0 + e * 128, v[e]);
    }
    done = bytes & ~3;
  }
  for (int i = done + 2 * lane; i < bytes; i += 64) {
    const uint32_t v = (low & 1u) ? (uint32_t)src[i] | ((uint32_t)src[i + 1] << 8) : *reinterpret_cast<const uint16_t *>(src + i);
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + i), "h"((uint16_t)v) : "memory");
  }
}

// Dense decode (Sources/IshizukiKit/Core/GGMLKernels.swift:391-401), and with ids the rows of a
// quantized table (GGMLKernels.swift:102-138, 404-420; an id outside the table gives zeros). A
// warp's work item is a run of up to `chunk` consecutive blocks of a row: their bytes come into
// shared memory in 16-byte pieces (eight blocks of any type are a multiple of 16), are decoded from
// there a lane eight weights, and leave in 16-byte stores.
//
// Bound: HBM on the output. A Q6_K weight of 17408 x 5120 to bf16 takes 43 us (5.8 TB/s), to fp32
// 68 (6.3 TB/s); reading the blocks byte by byte from global memory and storing value by value took
// 129 and 185: the load/store unit was what was busy, with eighteen byte loads and eight stores per
// eight weights against nine and one here.
constexpr int kExpandChunk = 8, kExpandWarps = 8;  // most blocks of an item, warps of a thread block
template <int TYPE>
constexpr int kExpandSlot = (kExpandChunk * ggml_type_bytes(TYPE) + 31) & ~15;  // a reader may look at the words behind a block
template <int TYPE, typename OT, bool ROWS>
__global__ void __launch_bounds__(kExpandWarps * 32) ggml_expand_kernel(const int *__restrict__ ids, long long rows,
                                                                        const uint8_t *__restrict__ blocks, long long table_rows,
                                                                        long long per_row, int chunk_log, OT *__restrict__ y) {
  constexpr int kBytes = ggml_type_bytes(TYPE), kTable = ggml_table_bytes(TYPE);
  __shared__ __align__(16) uint8_t s_blocks[kExpandWarps][kExpandSlot<TYPE>];
  __shared__ __align__(16) uint8_t s_table[kTable ? kTable : 16];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t table = smem_u32(s_table);
  if (kTable) {
    ggml_table_fill<TYPE>(table);
    __syncthreads();
    table = stage_acquire(table);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // ids and blocks may be the launch before's, and y read by it
  const uint32_t slot = smem_u32(s_blocks[warp]);
  const bool wide = (reinterpret_cast<uintptr_t>(y) & (8 * sizeof(OT) - 1)) == 0;
  const int chunk = 1 << chunk_log;
  const long long chunks = (per_row + chunk - 1) >> chunk_log, work = rows * chunks;
  for (long long wi = (long long)blockIdx.x * kExpandWarps + warp; wi < work; wi += (long long)gridDim.x * kExpandWarps) {
    const long long i = !ROWS ? 0 : work >> 32 ? wi / chunks : (long long)((uint32_t)wi / (uint32_t)chunks);
    const long long b0 = (wi - i * chunks) << chunk_log;
    const int nb = (int)(per_row - b0 < chunk ? per_row - b0 : chunk);
    const long long row = ROWS ? ids[i] : 0;
    OT *out = y + (i * per_row + b0) * 256 + 8 * lane;
    float w[8];
    if (ROWS && (row < 0 || row >= table_rows)) {
#pragma unroll
      for (int e = 0; e < 8; ++e) w[e] = 0.f;
      for (int b = 0; b < nb; ++b) store8(out + b * 256, w, wide);
      continue;
    }
    __syncwarp();  // every lane is done with the last item's blocks
    stage_bytes(slot, blocks + (row * per_row + b0) * kBytes, nb * kBytes, lane);
    __syncwarp();
    const uint32_t a = stage_acquire(slot);
#pragma unroll 2
    for (int b = 0; b < nb; ++b) {
      decode8<TYPE>(BlockShared<TYPE>{a + b * kBytes, table}, lane, w);
      store8(out + b * 256, w, wide);
    }
  }
}

// y[m, n] = sum_k x[m, k] * w[n, k]: one warp per output row, every weight decoded once and used
// for all MR activation rows, fp32 accumulation, a warp-shuffle reduction at the end (the shape of
// the reference's ggml_matvec, GGMLKernels.swift:549-565).
template <int TYPE, int MR>
__global__ void __launch_bounds__(256) ggml_rowdot_kernel(const uint8_t *__restrict__ blocks, long long n, long long k,
                                                          const __half *__restrict__ x, int rows, __half *__restrict__ y,
                                                          long long ldy, int transposed) {
  constexpr int kBytes = ggml_type_bytes(TYPE);
  const int lane = threadIdx.x & 31;
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long per_row = k / 256;
  for (long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < n; row += warps) {
    float acc[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[m] = 0.f;
    const uint8_t *b = blocks + row * per_row * kBytes;
    for (long long bi = 0; bi < per_row; ++bi) {
      float w[8];
      decode8<TYPE>(b + bi * kBytes, lane, w);
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        if (m < rows) {
          const uint4 v = __ldg(reinterpret_cast<const uint4 *>(x + (long long)m * k + bi * 256 + 8 * lane));
          const uint32_t p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&p[e]));
            acc[m] = fmaf(w[2 * e], f.x, acc[m]);
            acc[m] = fmaf(w[2 * e + 1], f.y, acc[m]);
          }
        }
      }
    }
#pragma unroll
    for (int m = 0; m < MR; ++m) {
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], d);
      if (lane == 0 && m < rows) {
        if (transposed) y[row * ldy + m] = __float2half_rn(acc[m]);
        else y[(long long)m * ldy + row] = __float2half_rn(acc[m]);
      }
    }
  }
}

// Index of the largest of n fp16 logits per row, the lowest index among equals (MLX argMax as the
// greedy verify uses it, Sources/IshizukiKit/Generate/SpeculativeGeneration.swift:173-177). NaN
// never wins. A row is cut into chunks, one CTA each (grid: chunks x rows): 16-byte loads where the
// row allows, the chunk's best (value, index) goes to `parts`, and the CTA that counts itself last
// for its row reduces the row's parts. Value first, then the lower index: the result does not
// depend on the order in which the CTAs finish. `counters` (one per row) are zero between launches.
struct ArgPart {
  float v;
  int i;
};
__device__ __forceinline__ bool arg_better(float v, int i, float bv, int bi) {
  return i >= 0 && (bi < 0 || v > bv || (v == bv && i < bi));
}
__device__ __forceinline__ void arg_take(float v, int i, float &best, int &at) {
  if (v > best || (at < 0 && v == best)) best = v, at = i;  // indices come in ascending order per thread
}
__global__ void __launch_bounds__(256) argmax_rows_kernel(const __half *__restrict__ y, long long n, long long ldy, int chunk,
                                                          ArgPart *__restrict__ parts, unsigned *__restrict__ counters,
                                                          int *__restrict__ out) {
  __shared__ float s_val[8];
  __shared__ int s_idx[8];
  __shared__ bool s_last;
  const int r = blockIdx.y, c = blockIdx.x, nchunks = gridDim.x;
  const __half *row = y + (long long)r * ldy;
  const long long lo = (long long)c * chunk, hi = lo + chunk < n ? lo + chunk : n;
  float best = -INFINITY;
  int at = -1;
  long long i = lo + (long long)threadIdx.x * 8;
  if ((reinterpret_cast<uintptr_t>(row + lo) & 15u) == 0) {
    for (; i + 8 <= hi; i += 256 * 8) {
      const uint4 q = *reinterpret_cast<const uint4 *>(row + i);
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[e]));
        arg_take(f.x, (int)i + 2 * e, best, at);
        arg_take(f.y, (int)i + 2 * e + 1, best, at);
      }
    }
  }
  // what the 16-byte loads left: a misaligned chunk, the last few values
  for (; i < hi; i += 256 * 8)
    for (long long k = i; k < hi && k < i + 8; ++k) arg_take(__half2float(row[k]), (int)k, best, at);
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, d);
    const int oi = __shfl_xor_sync(0xffffffffu, at, d);
    if (arg_better(ov, oi, best, at)) best = ov, at = oi;
  }
  if ((threadIdx.x & 31) == 0) s_val[threadIdx.x >> 5] = best, s_idx[threadIdx.x >> 5] = at;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w)
      if (arg_better(s_val[w], s_idx[w], best, at)) best = s_val[w], at = s_idx[w];
    parts[(long long)r * nchunks + c] = ArgPart{best, at};
    __threadfence();
    const unsigned before = atomicAdd(counters + r, 1u);
    s_last = before == (unsigned)nchunks - 1;
  }
  __syncthreads();
  if (!s_last || threadIdx.x >= 32) return;
  __threadfence();
  best = -INFINITY, at = -1;
  for (int k = threadIdx.x; k < nchunks; k += 32) {
    const ArgPart *pt = parts + (long long)r * nchunks + k;
    const float pv = __ldcg(&pt->v);  // written by other CTAs of this launch: from L2
    const int pi = __ldcg(&pt->i);
    if (arg_better(pv, pi, best, at)) best = pv, at = pi;
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, d);
    const int oi = __shfl_xor_sync(0xffffffffu, at, d);
    if (arg_better(ov, oi, best, at)) best = ov, at = oi;
  }
  if (threadIdx.x == 0) {
    out[r] = at < 0 ? 0 : at;
    counters[r] = 0;  // for the next launch on this stream
  }
}

template <class F>
cudaError_t with_type(int type, F &&f) {
  switch (type) {
    case 10: f(std::integral_constant<int, 10>()); break;
    case 12: f(std::integral_constant<int, 12>()); break;
    case 14: f(std::integral_constant<int, 14>()); break;
    case 16: f(std::integral_constant<int, 16>()); break;
    case 17: f(std::integral_constant<int, 17>()); break;
    case 18: f(std::integral_constant<int, 18>()); break;
    case 19: f(std::integral_constant<int, 19>()); break;
    case 21: f(std::integral_constant<int, 21>()); break;
    case 22: f(std::integral_constant<int, 22>()); break;
    case 23: f(std::integral_constant<int, 23>()); break;
    case 29: f(std::integral_constant<int, 29>()); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace

int ggml_type_size(int type) { return ggml_type_bytes(type); }

// Blocks per work item (their logarithm): eight where that leaves every SM eight warps or more, fewer
// for small arrays (a warp decodes its blocks one after the other: a short array is done sooner by
// more warps). Measured on 2048 rows of 5120 in Q6_K: eight blocks 7.4 us, four 7.7, two 10.2.
static int expand_chunk_log(long long rows, long long per_row, int sm_count) {
  int log = 3;
  while (log > 0 && rows * ((per_row + (1 << log) - 1) >> log) < (long long)sm_count * 8) --log;
  return log;
}

template <bool ROWS>
static cudaError_t launch_expand(int type, const int *ids, long long rows, const uint8_t *blocks, long long table_rows,
                                 long long per_row, void *out, int out_dtype, int sm_count, cudaStream_t st) {
  const int chunk_log = expand_chunk_log(rows, per_row, sm_count);
  const long long want = (rows * ((per_row + (1 << chunk_log) - 1) >> chunk_log) + kExpandWarps - 1) / kExpandWarps;
  // Two items per warp in long 16-bit arrays: a thread block's start and its codebook are then paid
  // half as often (17408 x 5120 Q6_K to bf16 44.9 -> 43.1 us, IQ2_XS 45.1 -> 41.6); one item in fp32,
  // which is bound by its output (67.8 against 69.8 us). More items leave a longer last wave.
  const int rounds = out_dtype != 2 && want >= (long long)sm_count * 16 ? 2 : 1;
  const long long grid = std::min((want + rounds - 1) / rounds, 0x7fffffffll);
  return with_type(type, [&](auto t) {
    constexpr int T = decltype(t)::value;
    auto launch = [&](auto *y) {
      // may start while the launch before it ends, and waits for that one itself: 2048 rows of 5120 in Q4_K 8.2 -> 7.0 us
      cudaLaunchConfig_t cfg;
      memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3((unsigned)grid);
      cfg.blockDim = dim3(kExpandWarps * 32);
      cfg.stream = st;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[0].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      cudaLaunchKernelEx(&cfg, ggml_expand_kernel<T, std::remove_pointer_t<decltype(y)>, ROWS>, ids, rows, blocks, table_rows, per_row,
                         chunk_log, y);
    };
    if (out_dtype == 0) launch(static_cast<__half *>(out));
    else if (out_dtype == 1) launch(static_cast<__nv_bfloat16 *>(out));
    else launch(static_cast<float *>(out));
  });
}

cudaError_t launch_ggml_dequantize(int type, const uint8_t *blocks, long long n_blocks, void *out, int out_dtype, int sm_count,
                                   cudaStream_t st) {
  return launch_expand<false>(type, nullptr, 1, blocks, 1, n_blocks, out, out_dtype, sm_count, st);
}

cudaError_t launch_ggml_gather(int type, const int *ids, long long count, const uint8_t *blocks, long long table_rows,
                               long long k, void *out, int out_dtype, int sm_count, cudaStream_t st) {
  return launch_expand<true>(type, ids, count, blocks, table_rows, k / 256, out, out_dtype, sm_count, st);
}

cudaError_t launch_ggml_rowdot(int type, const uint8_t *blocks, long long n, long long k, const __half *x, int rows, __half *y,
                               long long ldy, int transposed, int sm_count, cudaStream_t st) {
  const long long want = (n * 32 + 255) / 256;
  const int grid = (int)(want < (long long)sm_count * 16 ? want : (long long)sm_count * 16);
  return with_type(type, [&](auto t) {
    constexpr int T = decltype(t)::value;
    if (rows <= 4) ggml_rowdot_kernel<T, 4><<<grid, 256, 0, st>>>(blocks, n, k, x, rows, y, ldy, transposed);
    else if (rows <= 8) ggml_rowdot_kernel<T, 8><<<grid, 256, 0, st>>>(blocks, n, k, x, rows, y, ldy, transposed);
    else ggml_rowdot_kernel<T, 16><<<grid, 256, 0, st>>>(blocks, n, k, x, rows, y, ldy, transposed);
  });
}

// scratch: ishi::argmax_scratch_bytes() bytes, zero before the first launch
size_t argmax_scratch_bytes() { return (size_t)16 * 1024 * sizeof(ArgPart) + 16 * sizeof(unsigned); }

cudaError_t launch_argmax_rows(const __half *y, int rows, long long n, long long ldy, int *out, void *scratch, cudaStream_t st) {
  if (rows < 1 || rows > 16 || n < 1 || n > 0x7fffffffll) return cudaErrorInvalidValue;
  long long chunk = 8192;
  while ((n + chunk - 1) / chunk > 1024) chunk *= 2;
  const int nchunks = (int)((n + chunk - 1) / chunk);
  ArgPart *parts = static_cast<ArgPart *>(scratch);
  unsigned *counters = reinterpret_cast<unsigned *>(parts + 16 * 1024);
  argmax_rows_kernel<<<dim3(nchunks, rows), 256, 0, st>>>(y, n, ldy, (int)chunk, parts, counters, out);
  return cudaGetLastError();
}

}  // namespace ishi
