// The warp-level verify-matmul kernel: y[m, n] = sum_k x[m, k] * w[n, k] for 1..16 activation rows
// on mma.sync (m16n8k16, weights on the M side, activation rows on the N side), with a CUDA-core
// variant for a single row.
//
// Why not tcgen05 here: eight activation rows fill an m16n8k16 fragment exactly, twenty-odd warps
// per SM decode in registers right beside the MMA, and on the same weights this kernel measures
// about twice as fast as the tcgen05 kernel (ishi_rowstream.cuh: 128 weight rows per instruction,
// four decode warps per CTA feeding tensor memory). That kernel stays for the formats that have
// no fragment decoder and for inputs too wide for this one's shared memory.
//
// Layout. The weight is re-tiled once, when the projection is created, into fragment order: a
// tile is 16 output rows x 256 k (one unit), stored as [16-byte piece][lane] so that every
// warp-wide 128-bit access is one contiguous 512-byte run, followed by a small per-row section
// (block scales). Lane (g = lane / 4, t = lane % 4) owns weight rows g and g + 8 of the tile and,
// in every k-step, the four k positions the format's decoder assigns to t. The raw weight's bits in
// another order (a few formats take some bytes more).
//
// Work. K is cut into S column ranges and the kernel is launched as thread-block clusters of S
// CTAs (S = 1: no cluster): CTA r of a cluster stages the activations of column range r into shared
// memory once, laid out as its format's decoder reads them, and all CTAs of a cluster walk the same
// run of 16-row panels, dealt to the clusters in equal contiguous runs. A CTA's tiles, panel after
// panel and in each its units in order, are one sequence, and every warp takes an equal contiguous
// run of it, whatever panel it begins and ends in: with 14.7 panels per SM (a 27B gate and up pair) 24
// warps walk 12 or 13 tiles each, where whole panels per warp kept 15 of 20 warps busy with 20 tiles.
// A warp streams its run through a private ring in shared memory: its lanes copy a tile with a few
// 16-byte async copies (cp.async), one commit group per tile. What bounds the loop is instruction
// issue, so the copy has to be cheap: a bulk copy per tile on an mbarrier moves the same bytes with
// one instruction, but moving its operands to uniform registers, electing the lane, counting the
// bytes in and polling the barrier made about 100 of the loop's 365 instructions per Q4_K tile. No
// producer warp, no cross-warp wait on the data path.
//
// Reduction, without a CTA-wide barrier. A panel that lies inside one warp's run is complete when
// the warp leaves it. The others (at most two per run: the one it begins in and the one it ends
// in) are parked as partial 16 x 8 tiles, the first in a slot of the warp's, the last in its ring,
// which is empty by then; the warp that arrives last at the panel's counter adds the partials in
// warp order. The tiles' fp32 results are added up in fp64: where a panel is cut depends on where it
// lies in the CTA's sequence, and the sums must not (a gated pair and the same two weights
// stacked give the same products). With S > 1 the CTA's partial panel goes into the
// shared memory of the panel's leader CTA (distributed shared memory, st.async counted on an
// mbarrier there), an inbox slot per panel and rank; when a CTA's warps are through their runs they
// add the S partials of the panels it leads in rank order and write y. Every slot, counter and
// mbarrier is used once per launch: nothing is recycled and nobody waits for room. No global
// scratch, no atomics on values, every y element written once, the summation order fixed by the plan.
//
// Activation rows 9 ... 16 are a second column group: the same A fragments, decoded once, multiply
// a second staged region (NB = 2).
#pragma once
#include "ishi_stream.cuh"

namespace ishi {

constexpr int kFragRows = 16;
#ifndef ISHI_FRAG_MAX_WARPS
#define ISHI_FRAG_MAX_WARPS 24
#endif
// At up to eight rows the kernel is compiled for two block sizes: up to Fmt::kFewWarps warps, and up to
// kFragMaxWarps with 80 registers per thread. The smaller one is 20 warps with 96 registers (the decoders'
// loads then run further ahead of their use), or 16 with 128 in Q2_K and Q6_K (17408 x 5120, eight rows:
// Q2_K 16.4 -> 15.4 us, Q6_K 17.0 -> 16.8 when it was chosen; one row 15.7 -> 14.9, 16.6 -> 16.3). The other formats gain nothing
// by that, and the affine packs lose 2 to 5 % with their 20-warp plans. With two column
// groups it is one block size per format, Fmt::kManyWarps: 16 warps with 128 registers, or 20 with 96
// where the decoder does not use the registers and the smaller tiles want warps. 16 rows, 17408 x 5120
// and 5120 x 17408, 20 -> 16 warps: IQ1_S 25.7 / 31.3 -> 23.6 / 29.5 us, affine 8-bit 23.2 / 26.2 -> 21.3
// / 24.7, affine 4-bit in groups of 32 22.9 / 27.0 -> 21.6 / 25.5, IQ4_XS 23.6 / 26.4 -> 22.8 / 25.9, IQ2_XS,
// Q4_K, ternary and the other affine 4-bit 1 to 2 % less, Q6_K 24.2 / 29.6 -> 23.8 / 28.4; Q2_K 21.2 / 24.3
// -> 21.6 / 26.0, affine 2-bit 19.4 / 21.7 -> 19.5 / 22.4, IQ2_S the same: these stay at 20.
constexpr int kFragMaxWarps = ISHI_FRAG_MAX_WARPS;
constexpr int kFragMaxSplit = 8;  // portable cluster size
constexpr int kFragMaxPeers = 8;  // GPUs of one NVSwitch box

struct FragArgs {
  const uint8_t *tiles;  // [P][units][tile bytes]
  const __half *x;
  __half *y;
  long long ldy;
  int out_transposed;
  int M, N, K;
  int units, S, P, NC;  // NC clusters of S CTAs
  int ring;             // tiles per warp-private ring, two or more: one is decoded while the others are in flight
  int ahead;            // of them, tiles asked for before the dependency wait, 1 ... ring - 1
  int led;              // most panels a CTA leads (S > 1)
  // ceil(2^32 / d) for d = S, NC, warps, umax, umax - 1, or 0 for d = 1: see frag_div()
  unsigned inv_s, inv_nc, inv_w, inv_u, inv_u1;
  int umax;             // most units in a column range
  uint32_t xregion;     // bytes of one staged region: umax * Fmt::kXBytes + Fmt::kXFixed
  int group_size, scale_dtype;
  int *err;             // raised when a bounded wait gives up
  // Block Hadamard rotation of x while it is staged (0: none): xr = WHT_block(x * signs) / sqrt(block)
  int rot_block;           // a power of two, 8 ... 256
  const float *rot_signs;  // [K] or null
  // Gated pair (the weight was tiled with FragSrc::pair_rows): rows g and g + 8 of a panel are the
  // gate and the up row of output row 8 p + g, and the epilogue writes silu(gate) * up, N / 2 rows
  int swiglu;
  // The next kernel of the stream may start at once (0) or only when the launch before this one has
  // completed (1): a kernel that uses what that launch wrote without waiting for this one (HostCopies)
  int release_late;
  // Output exchange between the GPUs of an N-sharded projection (world = 0: none). Every rank holds
  // the whole output as [rows of all shards][8 or 16] fp16 at the same place of its exchange buffer; this
  // launch computes rows row_offset ... row_offset + N - 1 and stores them into every rank's copy
  // over NVLink. When all CTAs have stored, the rank writes seq into its arrival word on every rank.
  int world, rank;
  __half *peer_y[kFragMaxPeers];          // the output array in every rank's buffer ([rank]: the local one)
  int peer_ld;                            // fp16 values between its rows: 8, or 16 when the call has more than 8 rows
  unsigned *peer_flags[kFragMaxPeers];    // every rank's arrival words; this rank writes word [rank] of each
  unsigned *local_flags;                  // this rank's arrival words, one per rank
  unsigned *done;                         // CTAs of this launch that have stored their rows
  // The launches of an exchange are numbered on the device (so that a captured graph can be
  // replayed): *launch_no is the number of the last launch that completed on this rank; all ranks
  // issue the same sequence, so the numbers agree across ranks.
  unsigned *launch_no;
  int wait_previous;                      // first wait until every rank's previous launch has arrived here
  long long row_offset;
  unsigned long long *trace;              // diagnostic builds (-DISHI_TRACE): [CTA][warp][32] timestamps, else unused
};

// Diagnostic builds stamp the global nanosecond timer at the kernel's phase boundaries.
#ifdef ISHI_TRACE
#define ISHI_STAMP(slot)                                                                                   \
  do {                                                                                                     \
    if (a.trace && lane == 0) {                                                                            \
      unsigned long long t_;                                                                               \
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_)::"memory");                                    \
      a.trace[((size_t)blockIdx.x * kFragMaxWarps + warp) * 32 + (slot)] = t_;                             \
    }                                                                                                      \
  } while (0)
// ... and add up the clock cycles a warp spends in each part of its panel loop (slots 16 ... 23)
#define ISHI_CLOCK(var) const long long var = clock64()
#define ISHI_SPENT(slot, from, to)                                                                        \
  do {                                                                                                     \
    if (a.trace && lane == 0) a.trace[((size_t)blockIdx.x * kFragMaxWarps + warp) * 32 + (slot)] += (unsigned long long)((to) - (from)); \
  } while (0)
#else
#define ISHI_STAMP(slot) \
  do {                   \
  } while (0)
#define ISHI_CLOCK(var) \
  do {                  \
  } while (0)
#define ISHI_SPENT(slot, from, to) \
  do {                             \
  } while (0)
#endif

__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
// a tile of BYTES (a multiple of 16) bytes by one warp; src and dst are this lane's: offset by 16 * lane
template <int BYTES>
__device__ __forceinline__ void cp_async_tile(uint32_t dst, const uint8_t *src, int lane) {
#pragma unroll
  for (int i = 0; i < BYTES / 512; ++i) cp_async16(dst + 512u * i, src + 512 * i);
  if (BYTES % 512 && lane < BYTES % 512 / 16) cp_async16(dst + BYTES / 512 * 512u, src + BYTES / 512 * 512);
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void sts128d(uint32_t addr, double a, double b) {
  asm volatile("st.shared.v2.f64 [%0], {%1,%2};" ::"r"(addr), "d"(a), "d"(b) : "memory");
}
// (not volatile: callers tie the address to the barrier that publishes the data)
__device__ __forceinline__ double2 lds128d(uint32_t addr) {
  double2 v;
  asm("ld.shared.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr));
  return v;
}
// One more arrival at a counter in shared memory: returns the arrivals before it. Releases what the warp's lanes
// stored (the caller's __syncwarp orders them ahead of it) and acquires what those who arrived before released.
__device__ __forceinline__ int count_in(uint32_t addr) {
  int old;
  asm volatile("atom.acq_rel.cta.shared::cta.add.s32 %0, [%1], 1;" : "=r"(old) : "r"(addr) : "memory");
  return old;
}
__device__ __forceinline__ float lds32f(uint32_t addr) {
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
// the address of this CTA's shared-memory location addr in CTA rank of the cluster
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// arrival without the release fence, which would wait for every copy and store in flight; the
// data that crosses CTAs here is published by mbarriers instead
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_relaxed() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// n / d through inv = ceil(2^32 / d), exact for n * d < 2^32; inv = 0 stands for d = 1
__device__ __forceinline__ int frag_div(unsigned n, unsigned inv) { return inv ? (int)__umulhi(n, inv) : (int)n; }
__host__ inline unsigned frag_inverse(int d) { return d <= 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d); }

__host__ __device__ inline int frag_column_begin(int c, int units, int S) { return (c * units) / S; }
__host__ __device__ inline int frag_ring_stride(int tile_bytes) { return (tile_bytes + 15) & ~15; }

// shared memory of one CTA, in order: the staged activations (a region per group of eight rows),
// the format's tables, the warps' partial-tile slots, the inbox for the partial panels of the
// cluster's CTAs, a control block, the warps' rings
// control block: arrival counters [warp] @0, abort @96, the activations' mbarrier @104, inbox mbarriers [led] @128
constexpr uint32_t kFragCtrlAbort = 96, kFragCtrlX = 104, kFragCtrlInbox = 128;
static_assert(4 * kFragMaxWarps <= (int)kFragCtrlAbort, "control block");
__host__ __device__ inline uint32_t frag_ctrl_bytes(int led) { return (kFragCtrlInbox + 8u * (uint32_t)led + 127u) & ~127u; }
// x: the staged regions and the format's tables; led: most panels a CTA leads; NB: groups of eight rows
__host__ __device__ inline size_t frag_smem_bytes(size_t x, int W, int led, int S, int NB, int tile_bytes, int ring) {
  return x + (size_t)W * NB * 1024 + (S > 1 ? (size_t)led * S * NB * 512 : 0) + frag_ctrl_bytes(S > 1 ? led : 0) +
         (size_t)W * ring * frag_ring_stride(tile_bytes);
}

__device__ __forceinline__ unsigned ld_acquire_sys(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_sys(unsigned *p, unsigned v) {
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// silu(gate) * up as the reference's MLP computes it on fp16 arrays (downProj(silu(gateProj(x)) *
// upProj(x)), Sources/IshizukiKit/Text/Attention.swift:251): the two products rounded to fp16,
// sigmoid, gate * sigmoid and the product with up each rounded to fp16 (one array per operation),
// the arithmetic itself in fp32. Returns the fp16 value as a float.
__device__ __forceinline__ float frag_swiglu(float gate, float up) {
  const float gf = __half2float(__float2half_rn(gate)), uf = __half2float(__float2half_rn(up));
  const float sig = __half2float(__float2half_rn(1.0f / (1.0f + expf(-gf))));
  const float act = __half2float(__float2half_rn(gf * sig));
  return __half2float(__float2half_rn(act * uf));
}

// One lane's part of panel p's finished 16 x 8 tile, in accumulator-fragment order: lane
// (g = lane / 4, t = lane % 4) holds v.x, v.y = weight row g, activation rows 2t, 2t + 1 and
// v.z, v.w = weight row g + 8, the same activation rows. Called by all 32 lanes of a warp.
// With an output exchange the four lanes of a weight row gather its eight values and one of them
// stores the 16 bytes into every rank's copy.
// m0: the first activation row of the tile's columns.
__device__ __forceinline__ void frag_write(const FragArgs &a, int p, int lane, float4 v, int m0) {
  const int g = lane >> 2, t = lane & 3;
  const long long n0 = (long long)p * kFragRows + g;
  if (a.swiglu) {
    // v.x, v.y: the gate row, v.z, v.w: the up row of output row 8 p + g
    v.x = frag_swiglu(v.x, v.z), v.y = frag_swiglu(v.y, v.w);
    const long long n = (long long)p * 8 + g;
    if (a.world > 0) {
      const __half2 h = __floats2half2_rn(v.x, v.y);
      const uint32_t ph = *reinterpret_cast<const uint32_t *>(&h);
      const int base = lane & ~3;
      uint4 row;
      row.x = __shfl_sync(0xffffffffu, ph, base), row.y = __shfl_sync(0xffffffffu, ph, base + 1);
      row.z = __shfl_sync(0xffffffffu, ph, base + 2), row.w = __shfl_sync(0xffffffffu, ph, base + 3);
      if (n < a.N / 2 && t < 2)  // lanes t = 0, 1 store to the even / odd ranks
        for (int q = t; q < a.world; q += 2) *reinterpret_cast<uint4 *>(a.peer_y[q] + (a.row_offset + n) * a.peer_ld + m0) = row;
      return;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int m = m0 + 2 * t + i;
      if (n < a.N / 2 && m < a.M) {
        const __half h = __float2half_rn(i ? v.y : v.x);
        if (a.out_transposed) a.y[n * a.ldy + m] = h;
        else a.y[(long long)m * a.ldy + n] = h;
      }
    }
    return;
  }
  if (a.world > 0) {
    const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    const uint32_t plo = *reinterpret_cast<const uint32_t *>(&lo), phi = *reinterpret_cast<const uint32_t *>(&hi);
    const int base = lane & ~3;
    uint4 rlo, rhi;
    rlo.x = __shfl_sync(0xffffffffu, plo, base), rlo.y = __shfl_sync(0xffffffffu, plo, base + 1);
    rlo.z = __shfl_sync(0xffffffffu, plo, base + 2), rlo.w = __shfl_sync(0xffffffffu, plo, base + 3);
    rhi.x = __shfl_sync(0xffffffffu, phi, base), rhi.y = __shfl_sync(0xffffffffu, phi, base + 1);
    rhi.z = __shfl_sync(0xffffffffu, phi, base + 2), rhi.w = __shfl_sync(0xffffffffu, phi, base + 3);
    // lanes t = 0, 1 store row g to the even / odd ranks, lanes t = 2, 3 row g + 8
    const long long n = n0 + ((t & 2) ? 8 : 0);
    if (n < a.N) {
      const uint4 row = (t & 2) ? rhi : rlo;
      for (int q = t & 1; q < a.world; q += 2) *reinterpret_cast<uint4 *>(a.peer_y[q] + (a.row_offset + n) * a.peer_ld + m0) = row;
    }
    return;
  }
  const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const long long n = n0 + ((i & 2) ? 8 : 0);
    const int m = m0 + 2 * t + (i & 1);
    if (n < a.N && m < a.M) {
      const __half h = __float2half_rn(e[i]);
      if (a.out_transposed) a.y[n * a.ldy + m] = h;
      else a.y[(long long)m * a.ldy + n] = h;
    }
  }
}

// Eight consecutive activations of one row (this lane's k = 8 * lane ... 8 * lane + 7 of a
// 256-wide unit) through the block Hadamard rotation, all 32 lanes together. fp32 inside, radix-2
// stages h = 1, 2, 4 in the lane and h = 8 ... block / 2 across lanes, in that order and with the
// same roundings as hadamard_rotate_kernel, so the result is bit-identical to rotating first.
__device__ __forceinline__ uint4 frag_rotate8(uint4 v, int block, const float *signs, int lane) {
  float f[8];
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 p = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
    f[2 * i] = p.x;
    f[2 * i + 1] = p.y;
  }
  if (signs) {
    const float4 s0 = __ldg(reinterpret_cast<const float4 *>(signs)), s1 = __ldg(reinterpret_cast<const float4 *>(signs) + 1);
    const float s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __fmul_rn(f[i], s[i]);
  }
#pragma unroll
  for (int h = 1; h < 8; h <<= 1)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (!(j & h)) {
        const float lo = f[j], hi = f[j + h];
        f[j] = __fadd_rn(lo, hi);
        f[j + h] = __fsub_rn(lo, hi);
      }
  for (int d = 1; d < block / 8; d <<= 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float o = __shfl_xor_sync(0xffffffffu, f[j], d);
      f[j] = (lane & d) ? __fsub_rn(o, f[j]) : __fadd_rn(f[j], o);
    }
  }
  const float scale = 1.0f / sqrtf((float)block);
  uint32_t r[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 h2 = __halves2half2(__float2half_rn(__fmul_rn(f[2 * i], scale)), __float2half_rn(__fmul_rn(f[2 * i + 1], scale)));
    r[i] = *reinterpret_cast<const uint32_t *>(&h2);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// 16 bytes into another CTA's shared memory; the bytes count as completed on that CTA's mbarrier
// when they have landed, so the reader needs no fence: it waits for the barrier's phase
__device__ __forceinline__ void st_async128(uint32_t addr, float4 v, uint32_t mbar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(addr),
               "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(mbar)
               : "memory");
}

// The activation rows of a group of eight: `live` rows of x; `staged`, 8 or 1, is known when the kernel is
// compiled. Staged rows past the live ones are zeros, in the single-row variant the other seven are
// whatever the shared memory holds: a row is a column of every MMA from there to y, and columns of no
// row are not written. Staging that is dear (the rotation on the tensor cores) leaves out the rows from
// `stored` on; it is eight where an output exchange stores all columns. (Plain staging loses by the
// extra branch: 1-3 % of a launch.)
struct FragRows {
  const __half *x;
  int live, stored, staged;
  // task i of the staging: (unit, row)
  __device__ __forceinline__ int2 task(int i) const { return staged == 1 ? make_int2(i, 0) : make_int2(i >> 3, i & 7); }
};

// Staging, a warp task per (unit, row): put(unit, row, v) with the values k = 8l .. 8l + 7 of lane l. All
// loads of up to eight tasks go out before the first is used: the staging costs one L2 latency. then() runs
// once, behind the first loads.
template <class Then, class Put>
__device__ __forceinline__ void frag_stage_rows(const FragArgs &a, const FragRows &m, int ub0, int uc, Then then, Put put) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, tasks = uc * m.staged;
  constexpr int kBatch = 8;
  const __half *xl = m.x + (long long)ub0 * 256 + lane * 8;
  int i0 = warp;
  do {
    uint4 v[kBatch];
#pragma unroll
    for (int e = 0; e < kBatch; ++e) {
      const int i = i0 + e * nw;
      const int2 t = m.task(i);
      v[e] = make_uint4(0u, 0u, 0u, 0u);
      if (i < tasks && t.y < m.live) v[e] = __ldg(reinterpret_cast<const uint4 *>(xl + (long long)t.y * a.K + t.x * 256));
    }
    if (i0 == warp) then();
#pragma unroll
    for (int e = 0; e < kBatch; ++e) {
      const int i = i0 + e * nw;
      if (i >= tasks) break;
      const int2 t = m.task(i);
      put(t.x, t.y, v[e]);
    }
    i0 += nw * kBatch;
  } while (i0 < tasks);
}

// How a decoder that copies its activations and adds them up (Fmt::kRows, Fmt::kRowSums) does it, if it says nothing else
struct FragCopying {
  static constexpr int kCopyRows = 8;  // most rows that are copied at up to eight
  static constexpr bool kSumsLater = false;  // do several rows that are not copied leave the sums to row_sums()?
};

// The activations of a decoder that reads them as they lie in x (Fmt::kRows): a bulk copy per row, asked for by
// one warp, all counted on `bar`. No thread's load or store is in the way: alone on the GPU 80 KB are there 1500
// cycles after the request where loads and stores by all warps take 2200 to 2500 (10 KB: 720 against 1150). Launches over weights
// from HBM, in us: Q4_K at eight rows 34816 x 5120 21.5 -> 20.5, 8192 x 5120 unsplit 9.15 -> 8.17, 5120 x 17408 14.55 -> 14.2; IQ2_XS
// 8192 x 5120 11.6 -> 11.2 at sixteen rows, 8.87 -> 8.71 at eight; IQ3_S 5120 x 17408 18.1 -> 17.5.
// An exchange stores all eight columns: there the rows past the live ones are zeros. Elsewhere they are whatever
// the shared memory holds, columns of no row.
template <int NB>
__device__ __forceinline__ void frag_copy_rows(const FragArgs &a, uint32_t xfrag, uint32_t stride, uint32_t bar, int ub0, int uc) {
  auto row_at = [&](int m) { return xfrag + (uint32_t)(m >> 3) * a.xregion + (uint32_t)(m & 7) * stride; };
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) mbar_arrive_expect_tx_u32(bar, (uint32_t)(a.M * uc) * 512u);
    __syncwarp();
    if (a.world > 0) asm volatile("fence.proxy.async;" ::: "memory");  // rows that other GPUs stored, seen by plain loads
    if ((int)threadIdx.x < a.M)
      bulk_g2s_u32(row_at((int)threadIdx.x), a.x + (long long)threadIdx.x * a.K + (long long)ub0 * 256, (uint32_t)uc * 512u, bar);
  }
  if (a.world > 0)
    for (int m = a.M; m < 8 * NB; ++m)
      for (int i = (int)threadIdx.x; i < uc * 32; i += (int)blockDim.x) sts128u(row_at(m) + 16u * (uint32_t)i, make_uint4(0u, 0u, 0u, 0u));
}

// Decoders with a scale per sixteen weights (Q2_K, Q6_K) multiply a group per k-step, and a lane's four values of a group
// are 8 bytes of x. Each 64 bytes of a row (two k-steps) are put in the order that makes its 8 bytes of both one 16-byte
// load: lane t's at 16 t. Where lane l's values k = 8l .. 8l + 7 of a unit go inside a row, the last four 16 bytes further on:
__device__ __forceinline__ uint32_t frag_pair_slot(int lane) { return (uint32_t)((lane >> 2) * 64 + (lane & 1) * 32 + (lane & 2) * 4); }
__device__ __forceinline__ uint32_t frag_times(uint32_t v, uint32_t f) {
  const __half2 r = __hmul2(*reinterpret_cast<const __half2 *>(&v), *reinterpret_cast<const __half2 *>(&f));
  return *reinterpret_cast<const uint32_t *>(&r);
}
// The group sums of x as fp16 high and low parts, the B registers of the MMA over the sixteen groups, whose slots of lane t are groups
// 4t .. 4t + 3: [lane (row, t)][hi hi lo lo].
__device__ __forceinline__ void frag_store_sums16(uint32_t sums, int lane, const float (&s)[4]) {
  uint32_t hi[4], lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half h = __float2half_rn(s[i]), l = __float2half_rn(s[i] - __half2float(h));
    hi[i] = __half_as_ushort(h), lo[i] = __half_as_ushort(l);
  }
  sts128u(sums + (uint32_t)lane * 16u, make_uint4(hi[0] | (hi[1] << 16), hi[2] | (hi[3] << 16), lo[0] | (lo[1] << 16), lo[2] | (lo[3] << 16)));
}
// A pass over copied rows has a warp task per unit and four rows: task i of `halves` (one or two) per unit
struct FragPass {
  int tasks, halves;
  __device__ __forceinline__ FragPass(int rows, int uc) : tasks(uc * (rows > 4 ? 2 : 1)), halves(rows > 4 ? 2 : 1) {}
  __device__ __forceinline__ int unit(int i) const { return halves == 2 ? i >> 1 : i; }
  __device__ __forceinline__ int row(int i) const { return halves == 2 ? (i & 1) * 4 : 0; }  // the first of the four
};
// Both, in place, for the copied rows of a column range. The sums by MMAs whose weight is one for the first
// group of a column's 32 values in rows 0-7 and for the second in rows 8-15. SCALED: the values times `factor` (both halves), the sums without.
template <bool SCALED>
__device__ __forceinline__ void frag_rows_by_16(uint32_t xfrag, uint32_t R, uint32_t sums, uint32_t sum_bytes, int rows, int uc, uint32_t factor) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, g = lane >> 2;
  const uint32_t x = stage_acquire(xfrag), first = lane & 2 ? 0u : 0x3c003c00u, second = lane & 2 ? 0x3c003c00u : 0u;
  const FragPass pass(rows, uc);
  for (int i = warp; i < pass.tasks; i += nw) {
    const int u = pass.unit(i), r0 = pass.row(i);
    const uint32_t at = x + (uint32_t)r0 * R + (uint32_t)u * 512u;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    uint4 v[4];  // (rows past the live ones: whatever is there, for columns of no row)
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = lds128(at + (uint32_t)e * R + (uint32_t)lane * 16u);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float c[4];
      mma16816_first(c, first, second, first, second, v[e].x, v[e].y);
      mma16816(c, first, second, first, second, v[e].z, v[e].w);
      if (g == r0 + e) s[0] = c[0], s[1] = c[2], s[2] = c[1], s[3] = c[3];
    }
    // every lane has its values of the four rows, which other lanes' stores overwrite
#pragma unroll
    for (int e = 0; e < 4; ++e) values_ready(v[e]);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t to = at + (uint32_t)e * R + frag_pair_slot(lane);
      sts64(to, SCALED ? frag_times(v[e].x, factor) : v[e].x, SCALED ? frag_times(v[e].y, factor) : v[e].y);
      sts64(to + 16u, SCALED ? frag_times(v[e].z, factor) : v[e].z, SCALED ? frag_times(v[e].w, factor) : v[e].w);
    }
    if ((g & 4) == r0) frag_store_sums16(sums + (uint32_t)u * sum_bytes, lane, s);
  }
}
// The same for rows that are stored and added up on their way from x: lane l's values v of the unit whose row begins at `row`. By the
// same MMAs: a row has the same sums, and so under one plan the same product bit for bit, whatever rows are beside it.
template <bool SCALED>
__device__ __forceinline__ void frag_put_by_16(uint32_t row, uint32_t sums, int r, uint4 v, uint32_t factor) {
  const int lane = threadIdx.x & 31;
  const uint32_t to = row + frag_pair_slot(lane);
  sts64(to, SCALED ? frag_times(v.x, factor) : v.x, SCALED ? frag_times(v.y, factor) : v.y);
  sts64(to + 16u, SCALED ? frag_times(v.z, factor) : v.z, SCALED ? frag_times(v.w, factor) : v.w);
  const uint32_t first = lane & 2 ? 0u : 0x3c003c00u, second = lane & 2 ? 0x3c003c00u : 0u;
  float c[4];
  mma16816_first(c, first, second, first, second, v.x, v.y);
  mma16816(c, first, second, first, second, v.z, v.w);
  // every lane of a quad's column has its four sums, 4t ... 4t + 3 in c[0], c[2], c[1], c[3]: lane (g, t), g < 4, stores 4t + g (all four
  // by one lane: 17408 x 5120 at eight rows, Q6_K 17.9 -> 17.0 us, Q2_K 14.75 -> 14.15; sums by shuffles 17.05 and 14.35)
  const int g = lane >> 2;
  if (g < 4) {
    const float s = g & 1 ? (g & 2 ? c[3] : c[2]) : (g & 2 ? c[1] : c[0]);
    const __half hi = __float2half_rn(s), lo = __float2half_rn(s - __half2float(hi));
    const uint32_t at = sums + (uint32_t)(r * 64 + (lane & 3) * 16 + g * 2);
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"(__half_as_ushort(hi)) : "memory");
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(at + 8u), "h"(__half_as_ushort(lo)) : "memory");
  }
}

// A decoder's shared-memory tables (kExtraBytes, a multiple of 16), laid out once per device from
// Fmt::table_word; every CTA copies them from here, a few 16-byte async copies per thread that land
// while it waits for the launch before. Building them in place, lookups and conversions ahead of the
// activations, cost a launch 0.8 us more (IQ4_XS, 17408 x 5120).
template <class Fmt>
__device__ __align__(16) uint8_t frag_table[Fmt::kExtraBytes ? Fmt::kExtraBytes : 16];
template <class Fmt>
__global__ void fill_table_kernel() {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < Fmt::kExtraBytes / 4; i += gridDim.x * blockDim.x)
    reinterpret_cast<uint32_t *>(frag_table<Fmt>)[i] = Fmt::table_word(i);
}

// MODE 0: tensor-core (up to eight rows per column group); MODE 1: CUDA-core FMA for a single row.
// MAXW: most warps of a block. NB: column groups of eight activation rows, 1 or 2. ONE: a single activation
// row on the tensor cores, which stages that row alone (17408 x 5120: 0.6 us less in affine 4-bit, 1.5 us
// in ternary, whose staging rotates; a variant of its own because the choice inside one kernel costs
// eight rows 0.5 us).
template <class Fmt, int MODE, int MAXW, int NB, bool ONE = false>
__global__ void __launch_bounds__(MAXW * 32, 1) frag_kernel(const FragArgs a) {
  static_assert(MODE == 0 || NB == 1, "the CUDA-core variant takes one row");
  static_assert(!ONE || (MODE == 0 && NB == 1), "one row is one column group");
  // a single row whose sums the decoder needs is staged by loads and stores, the sums on the way
  constexpr bool kCopied = Fmt::kRows && !(ONE && Fmt::kRowSums), kStaged = !Fmt::kRows || Fmt::kRowSums;
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int kTile = Fmt::kTileBytes;
  constexpr uint32_t kStride = (uint32_t)((kTile + 15) & ~15), kPart = NB * 512u, kPark = NB * 1024u;  // bytes of a partial tile in fp32, fp64
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // (a broadcast: the compiler sees that it is uniform)
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int S = a.S, W = (int)(blockDim.x >> 5);

  const uint32_t xfrag = smem_u32(smem);                                // [NB][a.xregion]
  const uint32_t tables = xfrag + NB * a.xregion;                       // Fmt::kExtraBytes
  const uint32_t red = tables + Fmt::kExtraBytes;                       // [warp][kPark]: the panel this warp's run begins inside of
  const uint32_t inbox = red + (uint32_t)W * kPark;                     // [led][S][kPart]
  const uint32_t ctrl = inbox + (S > 1 ? (uint32_t)(a.led * S) * kPart : 0u);
  const int R = a.ring;  // tiles in this warp's ring
  const uint32_t rings = ctrl + frag_ctrl_bytes(S > 1 ? a.led : 0), ring = rings + (uint32_t)(warp * R) * kStride;
  int *cnt = reinterpret_cast<int *>(smem + (ctrl - xfrag));  // [warp]: arrivals at the panel that begins in this warp's run and goes on
  volatile int *abort_word = reinterpret_cast<volatile int *>(smem + (ctrl - xfrag) + kFragCtrlAbort);

  // (divisions by multiplication: the host checks the ranges)
  const int cid = frag_div(blockIdx.x, a.inv_s);
  const int r = (int)blockIdx.x - cid * S;  // rank in the cluster = column range
  const int ub0 = frag_div((unsigned)(r * a.units), a.inv_s);
  const int uc = frag_div((unsigned)((r + 1) * a.units), a.inv_s) - ub0;
  // the cluster's panels: pa .. pa + np - 1
  const int pa = frag_div((unsigned)cid * (unsigned)a.P, a.inv_nc);
  const int np = frag_div((unsigned)(cid + 1) * (unsigned)a.P, a.inv_nc) - pa;
  const int led = S > 1 ? frag_div((unsigned)(np - 1 - r + S), a.inv_s) : 0;  // panels this CTA leads: r, r + S, ...
  // the CTA's tiles, and this warp's run of them: tiles T w / W ... T (w + 1) / W - 1, or tile w where there are
  // fewer tiles than warps (no division: three of them held up the first copies by 0.2 us)
  const unsigned T = (unsigned)(np * uc);
  auto run_begin = [&](unsigned w) { return T >= (unsigned)W ? frag_div(T * w, a.inv_w) : (int)min(w, T); };
  const int t0 = run_begin((unsigned)warp), t1 = run_begin((unsigned)warp + 1u);
  const int q0 = frag_div((unsigned)t0, uc == a.umax ? a.inv_u : a.inv_u1);  // the run's first panel

  ISHI_STAMP(0);
  // Let the next kernel on the stream start its own prologue as SMs fall free.
  if (!a.release_late) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (threadIdx.x < 32) {  // the control block
    for (int i = threadIdx.x; i < led; i += 32) {
      // each led panel's mbarrier: S partial panels, known now
      mbar_init_u32(ctrl + kFragCtrlInbox + 8u * i, 1);
      mbar_arrive_expect_tx_u32(ctrl + kFragCtrlInbox + 8u * i, (uint32_t)S * kPart);
    }
    if ((int)threadIdx.x < W) cnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
      *abort_word = 0;
      if (kCopied) mbar_init_u32(ctrl + kFragCtrlX, 1);
    }
    mbar_fence_init();
    __syncwarp();
  }
  // Shared memory of another CTA may be written only once that CTA runs and has set up its
  // barriers: every CTA arrives here, and a warp waits before its first partial panel.
  if (S > 1) cluster_arrive_relaxed();  // the init fence above is what the peers need; nothing else to publish yet

  if (Fmt::kExtraBytes) {
    for (int i = threadIdx.x * 16; i < Fmt::kExtraBytes; i += blockDim.x * 16) cp_async16(tables + i, frag_table<Fmt> + i);
    cp_async_commit();
  }

  // This warp's run of tiles. The fetch cursor runs R - 1 tiles ahead of the compute cursor: a tile is
  // fetched into the slot of the tile decoded last. One commit group per tile, empty past the end.
  int f_left = t1 - t0, f_u = t0 - q0 * uc;
  const uint8_t *f_src = a.tiles + ((long long)(pa + q0) * a.units + ub0 + f_u) * (long long)kTile + lane * 16;
  const long long step_panel = (long long)(a.units - uc) * kTile;  // from the end of a panel's column range to the next one's
  auto fetch = [&](uint32_t slot) {
    if (f_left > 0) {
      cp_async_tile<kTile>(slot + (uint32_t)lane * 16u, f_src, lane);
      f_src += kTile;
      if (++f_u == uc) {
        f_u = 0;
        f_src += step_panel;
      }
    }
    --f_left;
    cp_async_commit();
  };
  // Warm L2 and the address translation with this CTA's slice of x. Only a hint: x may still be
  // written by the kernel before this one, its values are read after the wait below, through L2.
  for (int m = warp; m < a.M; m += W) {
    const char *row = reinterpret_cast<const char *>(a.x + (long long)m * a.K + (long long)ub0 * 256);
    for (int c = lane; c < uc * 4; c += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + c * 128));
  }

  // The weight tiles are written by no earlier kernel: the first copies go out at once, no more of them than leave
  // the way free for the activations (a.ahead; the rest of the ring follows the loads of x). Asking the
  // run's next tiles into L2 as well delays the activations too: 60 -> 66 us per layer.
  for (int i = 0; i < a.ahead; ++i) fetch(ring + (uint32_t)i * kStride);

  // x may be the output of the kernel before this one and y may still be read by it: wait for the
  // earlier kernels (returns at once unless this kernel was launched early).
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (a.release_late) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  ISHI_STAMP(1);
  unsigned previous_launch = 0;
  if (a.world > 0) {
    previous_launch = *reinterpret_cast<volatile unsigned *>(a.launch_no);
    if (a.wait_previous && previous_launch != 0) {
      // ... and for the other GPUs: x may be rows they stored into this rank's exchange buffer
      if ((int)threadIdx.x < a.world) {
        bool ok = false;
        for (uint32_t i = 0; i < kWaitSpins && !ok; ++i) {
          ok = (int)(ld_acquire_sys(a.local_flags + threadIdx.x) - previous_launch) >= 0;
          if (!ok) __nanosleep(64);
        }
        if (!ok) *a.err = 2;  // give up: the result is wrong, the error word tells the host
      }
    }
    __syncthreads();  // the other GPUs' rows have arrived, for every warp
  }
  ISHI_STAMP(2);

  auto rest = [&] {  // the ring's other tiles, behind the activations
    for (int i = a.ahead; i < R - 1; ++i) fetch(ring + (uint32_t)i * kStride);
  };
  const bool copied = kCopied && a.rot_block == 0 && (NB == 2 || a.M <= Fmt::kCopyRows);
  if (copied) {
    if constexpr (kCopied) frag_copy_rows<NB>(a, xfrag, Fmt::row_stride(a), ctrl + kFragCtrlX, ub0, uc);
    rest();
  } else if constexpr (kStaged) {
    // activations of the column range into fragment order (all warps)
#pragma unroll
    for (int b = 0; b < NB; ++b)
      Fmt::stage_x(a, FragRows{a.x + (long long)(8 * b) * a.K, ONE ? 1 : a.M - 8 * b, ONE ? 1 : a.world > 0 ? 8 : a.M - 8 * b, ONE ? 1 : 8}, xfrag + b * a.xregion, ub0, uc,
                   [&] { if (b == 0) rest(); });
  }
  ISHI_STAMP(3);
  if (Fmt::kExtraBytes) {  // the tables have landed: all groups but the R - 1 tiles' behind them
    if (R == 2) cp_async_wait<1>();
    else if (R == 3) cp_async_wait<2>();
    else cp_async_wait<3>();
  }
  __syncthreads();  // staged, the tables there, and the control block set up for every warp
  if (copied && !mbar_wait_u32(ctrl + kFragCtrlX, 0u, abort_word)) *a.err = 1;  // (y stays wrong, the error word tells the host)
  if constexpr (kCopied && Fmt::kRowSums) {
    if (copied || Fmt::kSumsLater) {
#pragma unroll
      for (int b = 0; b < NB; ++b) Fmt::row_sums(a, xfrag + b * a.xregion, a.world > 0 ? 8 : min(a.M - 8 * b, 8), uc);
      __syncthreads();
    }
  }
  ISHI_STAMP(4);
  // shared-memory loads are plain asm the compiler may move; tie their addresses to the waits
  const uint32_t xf = stage_acquire(xfrag), tb = stage_acquire(tables);

  bool joined = S == 1;  // this warp has seen every CTA of the cluster arrive
  uint32_t c_slot = ring, f_slot = ring + (uint32_t)(R - 1) * kStride;
  const uint32_t ring_end = ring + (uint32_t)R * kStride;
  int at = t0, u = t0 - q0 * uc;
  for (int q = q0; at < t1; ++q) {
    const int first = at, end = min(t1, (q + 1) * uc);
    double acc[NB][4];
#pragma unroll
    for (int b = 0; b < NB; ++b) acc[b][0] = acc[b][1] = acc[b][2] = acc[b][3] = 0.0;
    for (; at < end; ++at, ++u) {
      ISHI_CLOCK(c0);
      // this tile has landed (all but the last R - 2 groups are complete), for every lane, and every
      // lane is done with the tile before, whose slot is refilled
      if (R == 2) cp_async_wait<0>();
      else if (R == 3) cp_async_wait<1>();
      else cp_async_wait<2>();
      __syncwarp();
      if (at == t0) ISHI_STAMP(6);
      ISHI_CLOCK(c1);
      fetch(f_slot);
      float tile[NB][4];
#pragma unroll
      for (int b = 0; b < NB; ++b) tile[b][0] = tile[b][1] = tile[b][2] = tile[b][3] = 0.f;
      Fmt::template unit<MODE, NB>(tile, a, stage_acquire(c_slot), xf, tb, u, g, t, lane);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        values_ready(tile[b][0], tile[b][1], tile[b][2], tile[b][3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[b][i] += (double)tile[b][i];
      }
      ISHI_CLOCK(c2);
      ISHI_SPENT(16, c0, c1);
      ISHI_SPENT(17, c1, c2);
      f_slot = c_slot;
      c_slot += kStride;
      if (c_slot == ring_end) c_slot = ring;
    }
    u = 0;
    if (MODE == 1) {
      // single activation row: each lane holds partial dot products of rows g (acc[0]) and
      // g + 8 (acc[2]) over its own k positions; add across the four lanes of a row
      double *c = acc[0];
      c[0] += __shfl_xor_sync(0xffffffffu, c[0], 1);
      c[0] += __shfl_xor_sync(0xffffffffu, c[0], 2);
      c[2] += __shfl_xor_sync(0xffffffffu, c[2], 1);
      c[2] += __shfl_xor_sync(0xffffffffu, c[2], 2);
      if (t != 0) c[0] = c[2] = 0.0;  // one copy per row enters the sums below (column m = 0)
      c[1] = c[3] = 0.0;
    }
    if (q == q0) ISHI_STAMP(7);

    ISHI_CLOCK(c3);
    const int begin = q * uc;
    if (first != begin || end != begin + uc) {
      // The panel is shared with other warps: park the partial tile; the warp that arrives last adds
      // the partials in warp order. The panel begins in run wa (parked in that warp's ring, which is
      // drained: the panel's part is the last of the run; the plan leaves it kPark bytes) and ends in run wb (parked in the slots).
      const int begun = run_begin((unsigned)lane);  // lane w: where run w begins
      const unsigned runs = (1u << W) - 1u;
      const int wa = __popc(__ballot_sync(0xffffffffu, begun <= begin) & runs) - 1;
      const int wb = __popc(__ballot_sync(0xffffffffu, begun < begin + uc) & runs) - 1;
      const uint32_t mine = (warp == wa ? ring : red + (uint32_t)warp * kPark) + (uint32_t)lane * 16u;
      __syncwarp();  // every lane is done with the last tile
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        sts128d(mine + b * 1024u, acc[b][0], acc[b][1]);
        sts128d(mine + b * 1024u + 512u, acc[b][2], acc[b][3]);
      }
      __syncwarp();
      int old = 0;
      if (lane == 0) old = count_in(ctrl + 4u * (uint32_t)wa);
      __syncwarp();
      old = __shfl_sync(0xffffffffu, old, 0);
      if (old != wb - wa) continue;
      for (int w = wa; w <= wb; ++w) {
        const uint32_t src = stage_acquire(w == wa ? rings + (uint32_t)(wa * R) * kStride : red + (uint32_t)w * kPark) + (uint32_t)lane * 16u;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const double2 lo = lds128d(src + b * 1024u), hi = lds128d(src + b * 1024u + 512u);
          acc[b][0] = w == wa ? lo.x : acc[b][0] + lo.x, acc[b][1] = w == wa ? lo.y : acc[b][1] + lo.y;
          acc[b][2] = w == wa ? hi.x : acc[b][2] + hi.x, acc[b][3] = w == wa ? hi.y : acc[b][3] + hi.y;
        }
      }
    }
    float4 sum[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      constexpr double kUnit = Fmt::kUnit;  // a power of two: the decoder's unit of a tile's result
      sum[b] = make_float4((float)(acc[b][0] * kUnit), (float)(acc[b][1] * kUnit), (float)(acc[b][2] * kUnit), (float)(acc[b][3] * kUnit));
    }
    ISHI_CLOCK(c4);
    ISHI_SPENT(18, c3, c4);

    if (S == 1) {
#pragma unroll
      for (int b = 0; b < NB; ++b) frag_write(a, pa + q, lane, sum[b], 8 * b);
    } else {
      // the CTA's partial panel goes to the panel's leader, rank q % S, into inbox slot q / S
      if (!joined) cluster_wait_relaxed(), joined = true;
      const int slot = frag_div((unsigned)q, a.inv_s), lead = q - slot * S;
      const uint32_t box = cluster_map(inbox + (uint32_t)(slot * S + r) * kPart + (uint32_t)lane * 16u, (uint32_t)lead);
      const uint32_t bar = cluster_map(ctrl + kFragCtrlInbox + 8u * slot, (uint32_t)lead);
#pragma unroll
      for (int b = 0; b < NB; ++b) st_async128(box + b * 512u, sum[b], bar);
      ISHI_CLOCK(c5);
      ISHI_SPENT(19, c4, c5);
    }
  }
  ISHI_STAMP(24);
  if (S > 1) {
    if (!joined) cluster_wait_relaxed();
    for (int i = warp; i < led; i += W) {
      const uint32_t bar = ctrl + kFragCtrlInbox + 8u * i;
      bool ok = mbar_try_wait_cluster(bar, 0u);
      for (uint32_t spin = 0; spin < kWaitSpins && !ok; ++spin) {
        ok = mbar_try_wait_cluster(bar, 0u);
        if (!ok && *abort_word != 0) break;
      }
      if (!ok) {  // give up: y of this panel stays wrong, the error word tells the host
        *abort_word = 1;
        *a.err = 1;
        break;
      }
      const uint32_t src = stage_acquire(inbox) + (uint32_t)(i * S) * kPart + (uint32_t)lane * 16u;
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float4 total = lds128f(src + b * 512u);
        for (int k = 1; k < S; ++k) {
          const float4 o = lds128f(src + (uint32_t)k * kPart + b * 512u);
          total.x += o.x, total.y += o.y, total.z += o.z, total.w += o.w;
        }
        frag_write(a, pa + i * S + r, lane, total, 8 * b);
      }
    }
    // A CTA that received all it leads may leave: nobody sends to it any more. One that gave up stays
    // until the others have left or given up too, since they may still send to it (a thread that
    // has exited counts as arrived).
    if (__shfl_sync(0xffffffffu, *abort_word, 0) != 0) {
      cluster_arrive_relaxed();
      cluster_wait_relaxed();
    }
  }
  ISHI_STAMP(27);
  if (a.world > 0) {
    // This CTA's rows are on their way to every rank; the last CTA of the launch announces them.
    // One thread fences for the CTA (the barrier orders the other threads' stores before it) at
    // device scope and counts the CTA done; the CTA that counts last has thereby synchronised
    // with every other CTA, so its one system-scope fence covers all their rows (fences are
    // cumulative) before it raises the arrival words. A system-scope fence in every CTA, with its
    // own stores still in flight, measured 1.6 us slower per launch.
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned before = atomicAdd(a.done, 1u);
      if (before == gridDim.x - 1) {
        *reinterpret_cast<volatile unsigned *>(a.done) = 0u;  // for the next launch on this stream
        *reinterpret_cast<volatile unsigned *>(a.launch_no) = previous_launch + 1u;
        __threadfence_system();
        for (int q = 0; q < a.world; ++q) st_relaxed_sys(a.peer_flags[q] + a.rank, previous_launch + 1u);
      }
    }
  }
}
// waits (bounded) until every rank's arrival word has reached this rank's latest launch
static __global__ void peer_wait_kernel(const unsigned *local_flags, int world, const unsigned *launch_no, int *err) {
  if ((int)threadIdx.x < world) {
    const unsigned seq = *reinterpret_cast<const volatile unsigned *>(launch_no);
    bool ok = false;
    for (uint32_t i = 0; i < kWaitSpins && !ok; ++i) {
      ok = (int)(ld_acquire_sys(local_flags + threadIdx.x) - seq) >= 0;
      if (!ok) __nanosleep(64);
    }
    if (!ok) *err = 2;
  }
}

// The exchange for products of the other kernels: rows [first, first + n) of this rank's own
// [.][8] array (just written by the product) go to every other rank's copy, columns past M
// cleared; then the same publication as in frag_kernel (last CTA: one system-scope fence, the
// launch number into this rank's arrival word on every rank).
struct PublishArgs {
  __half *peer_y[kFragMaxPeers];
  unsigned *peer_flags[kFragMaxPeers];
  unsigned *done, *launch_no;
  long long first, n;
  int world, rank, M;
};
static __global__ void __launch_bounds__(256) publish_rows_kernel(const PublishArgs a) {
  const unsigned previous_launch = *reinterpret_cast<volatile unsigned *>(a.launch_no);
  uint4 *mine = reinterpret_cast<uint4 *>(a.peer_y[a.rank]) + a.first;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (long long)gridDim.x * blockDim.x) {
    uint4 v = mine[i];
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (2 * j >= a.M) w[j] = 0u;
      else if (2 * j + 1 >= a.M) w[j] &= 0xffffu;
    }
    v = make_uint4(w[0], w[1], w[2], w[3]);
    for (int q = 0; q < a.world; ++q) (reinterpret_cast<uint4 *>(a.peer_y[q]) + a.first)[i] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned before = atomicAdd(a.done, 1u);
    if (before == gridDim.x - 1) {
      *reinterpret_cast<volatile unsigned *>(a.done) = 0u;
      *reinterpret_cast<volatile unsigned *>(a.launch_no) = previous_launch + 1u;
      __threadfence_system();
      for (int q = 0; q < a.world; ++q) st_relaxed_sys(a.peer_flags[q] + a.rank, previous_launch + 1u);
    }
  }
}

// One-time re-tiling into fragment order: Fmt::tile_halfword says which 2 bytes of the source
// land at halfword hw of tile (p, u). Rows past N read as zero. The source may be several weights
// of the same format and input width stacked along the output rows (projections that share their
// input, fused into one launch): segment i holds rows first_row[i] ... first_row[i + 1] - 1.
constexpr int kFragMaxSegments = 4;
struct FragSrc {
  const uint8_t *w[kFragMaxSegments], *scales[kFragMaxSegments], *biases[kFragMaxSegments];
  long long first_row[kFragMaxSegments + 1];
  int segments;
  long long w_row_bytes, s_row_bytes;  // distance between rows
  long long N;
  int group_size, scale_bytes;
  // Two segments of equal height interleaved by eights instead of stacked: rows 0-7 of panel p are
  // rows 8 p ... 8 p + 7 of segment 0, rows 8-15 the same rows of segment 1, so that one
  // accumulator fragment holds a row of each (see FragArgs::swiglu).
  int pair_rows;
};

// which segment holds output row `row` (< N), and the row's index inside it
__device__ __forceinline__ int frag_segment(const FragSrc &s, long long row, long long *local) {
  if (s.pair_rows) {
    *local = (row >> 4) * 8 + (row & 7);
    return (int)(row >> 3) & 1;
  }
  int i = 0;
  while (i + 1 < s.segments && row >= s.first_row[i + 1]) ++i;
  *local = row - s.first_row[i];
  return i;
}

template <class Fmt>
__global__ void __launch_bounds__(256) prepare_frag_kernel(const FragSrc src, int units, int tile_bytes,
                                                           uint8_t *__restrict__ dst) {
  const long long P = (src.N + kFragRows - 1) / kFragRows;
  const int halfwords = tile_bytes / 2;
  const long long total = P * units * halfwords;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int hw = (int)(i % halfwords);
    const long long pu = i / halfwords;
    const int u = (int)(pu % units);
    const long long p = pu / units;
    reinterpret_cast<uint16_t *>(dst + pu * (long long)tile_bytes)[hw] = Fmt::tile_halfword(src, p, u, hw);
  }
}

}  // namespace ishi
