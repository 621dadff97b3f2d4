// Instantiates the warp-level kernel for one fragment decoder and wraps its launches in a FragOps
// table (see ishi_kernels.h). Included by the frag_*.cu translation units only.
#pragma once
#include <cstring>

#include "ishi_kernels.h"

namespace ishi {

template <class Fmt>
struct FragOpsOf {
  // the variant that serves a launch: column groups of eight rows, CUDA cores or not, block size, a
  // single row of no exchange (which stores all eight columns).
  // Two column groups keep twice the accumulators and activations: at most Fmt::kManyWarps warps.
  static const void *kernel(int groups, int mode, int warps, bool one) {
    const bool few = warps <= Fmt::kFewWarps;
    if (groups == 2) return warps <= Fmt::kManyWarps ? (const void *)frag_kernel<Fmt, 0, Fmt::kManyWarps, 2> : nullptr;
    if constexpr (Fmt::kRowMode) {
      // (a format without a CUDA-core variant for one activation row runs that row through the MMA path)
      if (mode == 1) return few ? (const void *)frag_kernel<Fmt, 1, Fmt::kFewWarps, 1> : (const void *)frag_kernel<Fmt, 1, kFragMaxWarps, 1>;
    }
    if constexpr (!Fmt::kRows || Fmt::kRowSums)  // (copying one row as it lies in x needs no variant)
      if (one) return few ? (const void *)frag_kernel<Fmt, 0, Fmt::kFewWarps, 1, true> : (const void *)frag_kernel<Fmt, 0, kFragMaxWarps, 1, true>;
    return few ? (const void *)frag_kernel<Fmt, 0, Fmt::kFewWarps, 1> : (const void *)frag_kernel<Fmt, 0, kFragMaxWarps, 1>;
  }

  static cudaError_t configure(int max_smem) {
    for (int groups = 1; groups <= 2; ++groups)
      for (int mode = 0; mode < 2; ++mode)
        for (int warps : {Fmt::kManyWarps, Fmt::kFewWarps, kFragMaxWarps})
          for (bool one : {false, true})
            if (const void *k = kernel(groups, mode, warps, one)) {
              const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
              if (e != cudaSuccess) return e;
            }
    if constexpr (Fmt::kExtraBytes > 0) {
      // on a stream of its own: other threads may be using the default stream
      cudaStream_t st = nullptr;
      cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
      if (e != cudaSuccess) return e;
      fill_table_kernel<Fmt><<<32, 256, 0, st>>>();
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      cudaStreamDestroy(st);
      return e;
    }
    return cudaSuccess;
  }

  static void fill(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *at, int clusters, int split, int warps, size_t smem) {
    memset(cfg, 0, sizeof(*cfg));
    cfg->gridDim = dim3((unsigned)(clusters * split), 1, 1);
    cfg->blockDim = dim3((unsigned)(warps * 32), 1, 1);
    cfg->dynamicSmemBytes = smem;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)split;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
  }

  static int max_clusters(int split, int warps, int groups, size_t smem, int sm_count) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    fill(&cfg, at, sm_count, split, warps, smem);
    int n = 0;
    const void *k = kernel(groups, 0, warps, false);
    const cudaError_t e = k ? cudaOccupancyMaxActiveClusters(&n, k, &cfg) : cudaErrorInvalidValue;
    if (e != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return n;
  }

  static cudaError_t launch(const FragLaunch &l, const FragArgs &args) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    fill(&cfg, at, l.clusters, l.split, l.warps, l.smem);
    cfg.stream = l.stream;
    // Programmatic dependent launch: the kernel may start while the one before it on the stream
    // drains. It prefetches weight tiles, which no earlier kernel writes, and waits for the earlier
    // kernels before it touches x or y.
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = l.early ? 2 : 1;
    void *params[1] = {const_cast<FragArgs *>(&args)};
    return cudaLaunchKernelExC(&cfg, kernel(args.M > 8 ? 2 : 1, l.mode, l.warps, args.M == 1 && args.world == 0), params);
  }

  static cudaError_t prepare(const FragSrc &src, int units, uint8_t *dst, int grid, cudaStream_t stream) {
    prepare_frag_kernel<Fmt><<<grid, 256, 0, stream>>>(src, units, Fmt::kTileBytes, dst);
    return cudaGetLastError();
  }

  static constexpr FragOps ops() {
    return FragOps{Fmt::kTileBytes, Fmt::kXBytes, Fmt::kXFixed, Fmt::kExtraBytes, Fmt::kManyWarps, &configure, &max_clusters, &launch, &prepare};
  }
};

}  // namespace ishi
