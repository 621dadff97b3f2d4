// EXL3 trellis-coded weights: decode, rotations and the few-row product that decodes inside the
// matrix multiply (reference: Sources/IshizukiKit/Core/EXL3.swift).
//
// W [k, n] is stored as 16 x 16 tiles, tile (tk, tn) at ((tk * n / 16) + tn) * ring / 32 32-bit
// words; a tile is a ring of 256 * bits bits (half-integer rates: 128 * (2 * whole + 1)), each word
// counted from its top bit. Weight p of a tile is a function (one of three procedural codebooks,
// EXL3.swift:171-182) of the 16 ring bits that end where p's own code ends (EXL3.swift:184-214).
// Weight p = 8 * lane + i lies at row (lane % 4) * 2 + {0, 1, 8, 9}[i % 4], column
// lane / 4 + 8 * (i / 4) (EXL3.swift:286-290): with the weight's output dimension n on the M side of
// mma.sync m16n8k16 (A[n][k]) that is exactly lane's A fragment of one k-step,
//   a0 = (v0, v1), a1 = (v4, v5), a2 = (v2, v3), a3 = (v6, v7),
// so a tile is decoded straight into tensor-core operands and never written anywhere.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>

#include "ishi_kernels.h"
#include "ishi_ptx.cuh"

namespace ishi {

namespace {

// ring bits of a tile
__host__ __device__ constexpr int exl3_ring(int whole, bool half) { return half ? 128 * (2 * whole + 1) : 256 * whole; }

// bit of the ring where weight p's code ends
template <int KA, bool HK>
__device__ __forceinline__ uint32_t exl3_end(uint32_t p) {
  return HK ? (p >> 1) * (2 * KA + 1) + KA + (p & 1) * (KA + 1) : (p + 1) * KA;
}
// the same for weight 8 * lane + i, relative to the start of lane's first 16-bit window
template <int KA, bool HK>
__host__ __device__ constexpr uint32_t exl3_rel(uint32_t i) {
  return HK ? (i >> 1) * (2 * KA + 1) + (i & 1) * (KA + 1) + 16 : i * KA + 16;
}

// Two weights of 16-bit states s0, s1 as one fp16 pair (s0 in the low half).
// Codebooks 3INST and MCG (mul1 == false): x = s * mult + add; the two halves of
// (x & 0x8fff8fff) ^ 0x3b603b60 are fp16 numbers whose fp16 sum is the weight.
// Codebook MUL1: the byte sum of s * 0x83DCD12D as the mantissa of an fp16 in [1024, 2048), then one
// fused multiply-add in fp16.
template <bool MUL1>
__device__ __forceinline__ uint32_t exl3_pair(uint32_t s0, uint32_t s1, uint32_t mult, uint32_t add) {
  if (MUL1) {
    // the byte sums through the four-way byte dot product; the second weight's sum, moved to the
    // upper half, and 1024's bits in both are the addend of the first (one shift-and-add)
    const uint32_t m1 = __dp4a(s1 * 0x83DCD12Du, 0x01010101u, 0u);
    const uint32_t h = __dp4a(s0 * 0x83DCD12Du, 0x01010101u, (m1 << 16) + 0x64006400u);
    const uint32_t m = 0x1eee1eeeu, b = 0xc931c931u;
    const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&h), *reinterpret_cast<const __half2 *>(&m),
                              *reinterpret_cast<const __half2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
  }
  const uint32_t x0 = ((s0 * mult + add) & 0x8fff8fffu) ^ 0x3b603b60u;
  const uint32_t x1 = ((s1 * mult + add) & 0x8fff8fffu) ^ 0x3b603b60u;
  // (the halves of one register added as scalars: one instruction each, then one byte permute; with
  // the operands permuted first it is two permutes, and the permutes' pipe is the busier one)
  const __half2 h0 = *reinterpret_cast<const __half2 *>(&x0), h1 = *reinterpret_cast<const __half2 *>(&x1);
  const __half2 r = __halves2half2(__hadd(__low2half(h0), __high2half(h0)), __hadd(__low2half(h1), __high2half(h1)));
  return *reinterpret_cast<const uint32_t *>(&r);
}

// Which three consecutive ring words (with wrap-around) hold lane's eight 16-bit windows, and the
// bit of the first word where the first window starts. The same for every tile of a rate.
template <int KA, bool HK>
struct Exl3Lane {
  uint32_t j0, j1, j2, sh;
  __device__ __forceinline__ explicit Exl3Lane(int lane) {
    constexpr uint32_t kRing = exl3_ring(KA, HK), kWords = kRing / 32;
    const uint32_t lo = exl3_end<KA, HK>((uint32_t)lane * 8u) + kRing - 16u;  // first bit of the first window
    const uint32_t i0 = lo >> 5;
    sh = lo & 31u;
    j0 = i0 >= kWords ? i0 - kWords : i0;
    j1 = j0 + 1 >= kWords ? j0 + 1 - kWords : j0 + 1;
    j2 = j1 + 1 >= kWords ? j1 + 1 - kWords : j1 + 1;
  }
};

// lane's eight weights of one tile, from its three ring words, as four fp16 pairs (v0 v1 | v2 v3 | v4 v5 | v6 v7)
template <int KA, bool HK, bool MUL1>
__device__ __forceinline__ void exl3_decode8(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t sh, uint32_t mult, uint32_t add,
                                             uint32_t (&v)[4]) {
  uint32_t s[8];
  if constexpr (!HK && KA == 4) {
    // sh is 20 in every lane: windows start at bits 20, 24 ... 48 of w0 w1. Whole-byte positions are one
    // byte permute, those four bits off come from one shifted word (the 16 bits across two words: a
    // shift and a mask)
    const uint32_t b = __funnelshift_l(w1, w0, 20);
    s[0] = b >> 16, s[2] = prmt(b, 0u, 0x4421u), s[4] = prmt(b, 0u, 0x4410u), s[6] = (w1 >> 4) & 0xffffu;
    s[1] = __funnelshift_r(w1, w0, 24) & 0xffffu, s[3] = w1 >> 16, s[5] = prmt(w1, 0u, 0x4421u), s[7] = prmt(w1, 0u, 0x4410u);
  } else if constexpr (!HK && KA == 8) {
    // sh is 24: bits 24, 32 ... 80, whole bytes
    s[0] = __funnelshift_r(w1, w0, 24) & 0xffffu, s[1] = w1 >> 16, s[2] = prmt(w1, 0u, 0x4421u), s[3] = prmt(w1, 0u, 0x4410u);
    s[4] = __funnelshift_r(w2, w1, 24) & 0xffffu, s[5] = w2 >> 16, s[6] = prmt(w2, 0u, 0x4421u), s[7] = prmt(w2, 0u, 0x4410u);
  } else {
    // 96 ring bits from the window's first bit on: b0 (top) b1 b2
    const uint32_t b0 = __funnelshift_l(w1, w0, sh), b1 = __funnelshift_l(w2, w1, sh), b2 = w2 << sh;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t r = exl3_rel<KA, HK>((uint32_t)i);  // the state is bits r - 16 ... r - 1 of the 96
      uint32_t x;
      if (r <= 32) x = b0 >> (32 - r);
      else if (r < 64) x = __funnelshift_l(b1, b0, r - 32);  // bits r - 32 ... r - 1
      else if (r == 64) x = b1;
      else x = __funnelshift_l(b2, b1, r - 64);
      s[i] = x & 0xffffu;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = exl3_pair<MUL1>(s[2 * i], s[2 * i + 1], mult, add);
}

// ---- dequantize: one warp per tile ----------------------------------------------------------------
template <int KA, bool HK, bool MUL1, class OT>
__global__ void __launch_bounds__(256) exl3_dequantize_kernel(const uint32_t *__restrict__ trellis, int tiles_k, int tiles_n,
                                                              uint32_t mult, uint32_t add, OT *__restrict__ w) {
  constexpr uint32_t kWords = exl3_ring(KA, HK) / 32;
  const int lane = threadIdx.x & 31;
  const long long total = (long long)tiles_k * tiles_n;
  const long long N = (long long)tiles_n * 16;
  for (long long tile = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); tile < total; tile += (long long)gridDim.x * 8) {
    uint32_t v[4];
    const Exl3Lane<KA, HK> at(lane);
    const uint32_t *words = trellis + tile * kWords;
    exl3_decode8<KA, HK, MUL1>(__ldg(words + at.j0), __ldg(words + at.j1), __ldg(words + at.j2), at.sh, mult, add, v);
    const long long row = (tile / tiles_n) * 16 + (lane & 3) * 2, col = (tile % tiles_n) * 16 + (lane >> 2);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __half2 pair = *reinterpret_cast<const __half2 *>(&v[i >> 1]);
      const float f = (i & 1) ? __high2float(pair) : __low2float(pair);
      const int dr = (i & 1) + ((i & 2) ? 8 : 0), dc = (i & 4) ? 8 : 0;
      w[(row + dr) * N + col + dc] = (OT)f;
    }
  }
}

// ---- the product: rotated or plain, y [rows][n] = x [rows][k] . W ------------------------------------
// One launch does what EXL3Kernels.apply does in three: the input rotation while the activations
// are staged, the product, the output rotation on the finished sums (or neither: matvec).
//
// Work. A cluster of S CTAs owns 128 outputs (eight tile columns, a block of the output rotation),
// each CTA a contiguous share of the k blocks of 128, one CTA per SM. Its 32 warps are sixteen k phases
// times two column halves: of every two k blocks a warp has one k tile, four adjacent tiles of it,
// which lie one after the other in memory and stream through a private cp.async ring of slices.
//
// Activations are staged a chunk of k blocks at a time, in fragment order (one 8-byte shared-memory
// load per k tile gives the B registers of four MMAs): eight lanes hold a block of 128 values of one
// row, sixteen each, so that the butterflies of stages 1 ... 8 stay in the lane, 16 ... 64 are three
// shuffles, and a lane ends up with all of one k tile of its row. fp32 inside, the order of
// exl3_rotate_kernel, then fp16.
//
// Sums. The k phases are added through shared memory, the CTAs of a cluster through
// distributed shared memory: row m goes to rank m % S, which adds the S partial rows in rank order
// and applies the output rotation, a warp per row.
//
// Bound: the decode's instructions. Per 16 x 16 tile and lane MUL1 takes eight IMAD, eight dp4a, four
// byte permutes and four HFMA2 after the windows are cut out of the ring, all at two cycles per
// issue; at 4 and 8 bits the windows are byte permutes (see exl3_decode8). Gate shape 5120 x 17408,
// 4 bits MUL1, eight rows: 27.8 us with both
// rotations (24.0 at one row, 38.7 at sixteen), where three launches with the decode of before took
// 34.6 and, past eight rows, two products 65. Issue in 73 % of the cycles, the IMAD pipe 56 %.
//
// The trellis is the caller's own memory: nothing of it is read before the launches ahead have
// finished (griddepcontrol.wait), its first slices are only hinted into L2.
constexpr int kExl3Warps = 32, kExl3Phases = 16, kExl3Cols = 4;
constexpr int kExl3OutStride = 132;  // floats between rows of the k phases' sums: conflict-free stores
struct Exl3Args {
  const uint8_t *trellis;
  const __half *x, *su, *sv;  // su, sv null: no rotation
  void *y;                    // fp16 with sv, else fp32
  long long K, N;
  uint32_t mult, add;
  int rows, S, groups, kblocks, chunk;  // chunk: k blocks staged at a time, a multiple of four (two slices of every warp)
  int wide;                             // trellis, x, su: 16-byte aligned
  int *err;
};
template <int KA, bool HK>
constexpr int kExl3Slice = kExl3Cols * exl3_ring(KA, HK) / 8;  // bytes of a warp's four tiles
// slices per ring: about 4 KB
template <int KA, bool HK>
constexpr int kExl3Ring = kExl3Slice<KA, HK> > 512 ? 4 : kExl3Slice<KA, HK> > 256 ? 8 : 16;

__host__ __device__ inline size_t exl3_smem_bytes(int chunk, int rows, int S, int NB, int ring_bytes) {
  const size_t x = (size_t)chunk * 2048 * NB, red = (size_t)kExl3Phases * rows * kExl3OutStride * 4;
  const size_t inbox = S > 1 ? (size_t)((rows + S - 1) / S) * S * 512 : 0, stream = x + (size_t)kExl3Warps * ring_bytes;
  return 128 + inbox + (stream > red ? stream : red);
}

// one block row of the output: the lane's four consecutive values through the rotation
__device__ __forceinline__ float4 exl3_rotate4(float4 v, int lane) {
  const float a0 = __fadd_rn(v.x, v.y), a1 = __fsub_rn(v.x, v.y), a2 = __fadd_rn(v.z, v.w), a3 = __fsub_rn(v.z, v.w);
  float f[4] = {__fadd_rn(a0, a2), __fadd_rn(a1, a3), __fsub_rn(a0, a2), __fsub_rn(a1, a3)};
#pragma unroll
  for (int m = 1; m < 32; m <<= 1) {
    const float sign = (lane & m) ? -1.f : 1.f;  // (a fused multiply-add by +-1 is the sum, rounded once)
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = __fmaf_rn(f[i], sign, __shfl_xor_sync(0xffffffffu, f[i], m));
  }
  return make_float4(f[0], f[1], f[2], f[3]);
}

// two fp32 values in one register pair and the packed operations on them (each half rounded once)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0,%1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// sixteen consecutive halves (values k = 16 * sub ... of a block row) as eight words
__device__ __forceinline__ void exl3_load16(const __half *p, bool wide, uint32_t (&w)[8]) {
  if (wide) {
    const uint4 a = __ldg(reinterpret_cast<const uint4 *>(p)), b = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
    w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w, w[4] = b.x, w[5] = b.y, w[6] = b.z, w[7] = b.w;
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    w[i] = (uint32_t)__half_as_ushort(p[2 * i]) | ((uint32_t)__half_as_ushort(p[2 * i + 1]) << 16);
}
// x * s of one pair of halves, exact in fp32
__device__ __forceinline__ float2 exl3_scaled(uint32_t x, uint32_t s) {
  float2 r = make_float2(0.f, 0.f);
  fma_f32_f16(r.x, (uint16_t)x, (uint16_t)s);
  fma_f32_f16(r.y, (uint16_t)(x >> 16), (uint16_t)(s >> 16));
  return r;
}

// Stages k blocks b0 ... b0 + nb - 1: unit (row, block), eight lanes each, four units per warp task.
// The butterflies run on register pairs (values j and j + 8 of the lane's sixteen) but for the
// stage that crosses the pair. The fragments of k tile `sub` of a block and row r (of its group of
// eight) are 32 bytes at sub * 256 + (r ^ sub) * 32 (the xor spreads the stores over the banks; a
// warp's read of one k tile is one 256-byte run).
__device__ __forceinline__ void exl3_stage_x(const Exl3Args &a, uint32_t xs, int b0, int nb, int NB) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & 7;
  const int units = a.rows * nb;
  for (int u0 = warp * 4; u0 < units; u0 += kExl3Warps * 4) {
    const int u = u0 + (lane >> 3), blk = u / a.rows, row = u - blk * a.rows;
    const bool live = u < units;
    const long long k = (long long)(b0 + blk) * 128 + sub * 16;
    uint32_t p[8] = {};
    if (live) exl3_load16(a.x + (long long)row * a.K + k, a.wide, p);
    if (a.su) {
      uint32_t s[8] = {};
      if (live) exl3_load16(a.su + k, a.wide, s);
      uint64_t f[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 lo = exl3_scaled(p[i], s[i]), hi = exl3_scaled(p[i + 4], s[i + 4]);
        f[2 * i] = pack2(lo.x, hi.x), f[2 * i + 1] = pack2(lo.y, hi.y);
      }
      const uint64_t minus = pack2(-1.f, -1.f);
#pragma unroll
      for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (!(j & h)) {
            const uint64_t lo = f[j], hi = f[j + h];
            f[j] = add2(lo, hi);
            f[j + h] = fma2(hi, minus, lo);
          }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 v = unpack2(f[j]);
        f[j] = pack2(__fadd_rn(v.x, v.y), __fsub_rn(v.x, v.y));
      }
#pragma unroll
      for (int m = 1; m < 8; m <<= 1) {
        const float sign = (sub & m) ? -1.f : 1.f;
        const uint64_t sign2 = pack2(sign, sign);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 v = unpack2(f[j]);
          f[j] = fma2(f[j], sign2, pack2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m)));
        }
      }
      const uint64_t scale = pack2(0.08838834764831845f, 0.08838834764831845f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = unpack2(mul2(f[2 * i], scale)), y = unpack2(mul2(f[2 * i + 1], scale));
        const __half2 lo = __floats2half2_rn(x.x, y.x), hi = __floats2half2_rn(x.y, y.y);
        p[i] = *reinterpret_cast<const uint32_t *>(&lo), p[i + 4] = *reinterpret_cast<const uint32_t *>(&hi);
      }
    }
    if (!live) continue;
    // lane t of the row's quad takes pairs t (inputs 2t, 2t + 1) and t + 4 (2t + 8, 2t + 9)
    const uint32_t at = xs + (uint32_t)(blk * NB + (row >> 3)) * 2048u + (uint32_t)(sub * 256 + (((row & 7) ^ sub) * 32));
    sts128u(at, make_uint4(p[0], p[4], p[1], p[5]));
    sts128u(at + 16u, make_uint4(p[2], p[6], p[3], p[7]));
  }
}

template <int KA, bool HK, bool MUL1, int NB>
__global__ void __launch_bounds__(kExl3Warps * 32, 1) exl3_product_kernel(const Exl3Args a) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr uint32_t kTileBytes = exl3_ring(KA, HK) / 8;
  constexpr int kSlice = kExl3Slice<KA, HK>, R = kExl3Ring<KA, HK>;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int phase = warp >> 1, half = warp & 1;
  const int S = a.S, group = (int)blockIdx.x / S, rank = (int)blockIdx.x - group * S;
  const int kb0 = (int)((long long)rank * a.kblocks / S), kb1 = (int)((long long)(rank + 1) * a.kblocks / S);
  // shared memory: barrier and abort word, the rows this CTA finishes [led][S][512 bytes], the staged
  // activations, the rings; the k phases' sums overlay the last two
  const uint32_t bar = smem_u32(smem), inbox = bar + 128u;
  volatile int *abort_word = reinterpret_cast<volatile int *>(smem + 8);
  const int led = S > 1 ? (a.rows - rank + S - 1) / S : 0;
  const uint32_t xs = inbox + (S > 1 ? (uint32_t)((a.rows + S - 1) / S * S) * 512u : 0u);
  const uint32_t ring = xs + (uint32_t)a.chunk * 2048u * NB + (uint32_t)(warp * R * kSlice);

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    *abort_word = 0;
    if (S > 1) {
      mbar_init_u32(bar, 1);
      mbar_arrive_expect_tx_u32(bar, (uint32_t)(led * S) * 512u);
      mbar_fence_init();
    }
  }
  __syncwarp();
  if (S > 1) cluster_arrive_relaxed();

  // this warp's slices: k tiles 8 kb0 + phase + 16 i
  const long long step = (a.N / 16) * kExl3Phases * (long long)kTileBytes;
  const uint8_t *f_src = a.trellis + ((a.N / 16) * (8ll * kb0 + phase) + 8ll * group + kExl3Cols * half) * kTileBytes;
  int f_left = ((kb1 - kb0) * 8 - phase + kExl3Phases - 1) / kExl3Phases;
  auto fetch = [&](uint32_t slot) {
    if (f_left > 0) {
      if (a.wide) {
#pragma unroll
        for (int i = 0; i < (kSlice + 511) / 512; ++i)
          if (kSlice >= (i + 1) * 512 || lane < (kSlice - i * 512) / 16)
            cp_async16(slot + (uint32_t)(i * 512 + lane * 16), f_src + i * 512 + lane * 16);
      } else {
        for (int i = lane * 4; i < kSlice; i += 128)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(slot + (uint32_t)i), "l"(f_src + i) : "memory");
      }
      f_src += step;
    }
    --f_left;
    cp_async_commit();
  };
  // The first slices into L2 while the launch before this one ends: hints, no value is read before the wait (two gate
  // projections of 17408 x 5120 at eight rows 55.4 -> 54.9 us)
  constexpr int kLines = (kSlice + 127) / 128;
  for (int i = lane; i < min(f_left, R - 2) * kLines; i += 32)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(f_src + (i / kLines) * step + (i % kLines) * 128));
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int i = 0; i < R - 2; ++i) fetch(ring + (uint32_t)(i * kSlice));

  float acc[NB][kExl3Cols][4];
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int c = 0; c < kExl3Cols; ++c) acc[b][c][0] = acc[b][c][1] = acc[b][c][2] = acc[b][c][3] = 0.f;
  const Exl3Lane<KA, HK> at(lane);
  uint32_t c_slot = ring, f_slot = ring + (uint32_t)((R - 2) * kSlice);
  for (int c0 = kb0; c0 < kb1; c0 += a.chunk) {
    const int nb = min(a.chunk, kb1 - c0);
    if (c0 != kb0) __syncthreads();  // every warp is done with the chunk before
    exl3_stage_x(a, xs, c0, nb, NB);
    __syncthreads();
    const uint32_t sub = (uint32_t)phase & 7u;
    uint32_t xf = stage_acquire(xs) + (uint32_t)(phase >> 3) * 2048u * NB + sub * 256u + (((uint32_t)(lane >> 2) ^ sub) * 4u + (uint32_t)(lane & 3)) * 8u;
    auto slice = [&](uint32_t slot, uint32_t xt) {
      const uint32_t *words = reinterpret_cast<const uint32_t *>(smem + (slot - bar));
      const uint32_t *p0 = words + at.j0, *p1 = words + at.j1, *p2 = words + at.j2;
      uint2 b[NB];
#pragma unroll
      for (int n = 0; n < NB; ++n) b[n] = lds64(xt + 2048u * n);
#pragma unroll
      for (int c = 0; c < kExl3Cols; ++c) {
        constexpr int kWords = (int)kTileBytes / 4;
        uint32_t v[4];
        exl3_decode8<KA, HK, MUL1>(p0[c * kWords], p1[c * kWords], p2[c * kWords], at.sh, a.mult, a.add, v);
#pragma unroll
        for (int n = 0; n < NB; ++n) mma16816(acc[n][c], v[0], v[2], v[1], v[3], b[n].x, b[n].y);
      }
    };
    // two slices at a time: the waiting and the cursors once per eight tiles
    for (int i = phase; i < nb * 8; i += 2 * kExl3Phases, xf += 8192u * NB) {
      cp_async_wait<R - 4>();  // both have landed, for every lane ...
      __syncwarp();            // ... and every lane is done with the two before, whose slots are refilled
      fetch(f_slot);
      fetch(f_slot + (uint32_t)kSlice);
      const uint32_t slot = stage_acquire(c_slot);
      slice(slot, xf);
      if (i + kExl3Phases < nb * 8) slice(slot + (uint32_t)kSlice, xf + 4096u * NB);
      f_slot = c_slot;
      c_slot += 2u * kSlice;
      if (c_slot == ring + (uint32_t)(R * kSlice)) c_slot = ring;
    }
  }

  // the k phases' sums: [phase][row][output]
  __syncthreads();
  const uint32_t mine = xs + (uint32_t)(phase * a.rows * kExl3OutStride) * 4u;
#pragma unroll
  for (int n = 0; n < NB; ++n)
#pragma unroll
    for (int c = 0; c < kExl3Cols; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // lane (g, t): c0, c1 = output g, rows 2t, 2t + 1; c2, c3 = output g + 8
        const int m = 8 * n + 2 * (lane & 3) + (i & 1), out = (kExl3Cols * half + c) * 16 + (lane >> 2) + ((i & 2) ? 8 : 0);
        if (m < a.rows) sts32(mine + (uint32_t)(m * kExl3OutStride + out) * 4u, __float_as_uint(acc[n][c][i]));
      }
  __syncthreads();

  auto finish = [&](int m, float4 v) {
    const long long col = (long long)group * 128 + lane * 4;
    if (!a.sv) {
      float *y = static_cast<float *>(a.y) + (long long)m * a.N + col;
      if ((reinterpret_cast<uintptr_t>(a.y) & 15u) == 0) *reinterpret_cast<float4 *>(y) = v;
      else y[0] = v.x, y[1] = v.y, y[2] = v.z, y[3] = v.w;
      return;
    }
    v = exl3_rotate4(v, lane);
    __half h[4] = {a.sv[col], a.sv[col + 1], a.sv[col + 2], a.sv[col + 3]};
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __float2half_rn(__fmul_rn(__fmul_rn(f[i], 0.08838834764831845f), __half2float(h[i])));
    __half *y = static_cast<__half *>(a.y) + (long long)m * a.N + col;
    if ((reinterpret_cast<uintptr_t>(a.y) & 7u) == 0) {
      uint2 w;
      memcpy(&w, h, 8);
      *reinterpret_cast<uint2 *>(y) = w;
    } else {
      for (int i = 0; i < 4; ++i) y[i] = h[i];
    }
  };
  if (S > 1) cluster_wait_relaxed();  // every CTA of the cluster runs and has set its barrier up
  const uint32_t sums = stage_acquire(xs) + (uint32_t)lane * 16u;
  for (int m = warp; m < a.rows; m += kExl3Warps) {
    float4 v = lds128f(sums + (uint32_t)(m * kExl3OutStride) * 4u);
#pragma unroll
    for (int p = 1; p < kExl3Phases; ++p) {
      const float4 o = lds128f(sums + (uint32_t)((p * a.rows + m) * kExl3OutStride) * 4u);
      v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
    }
    if (S == 1) {
      finish(m, v);
    } else {
      const int li = m / S, to = m - li * S;
      st_async128(cluster_map(inbox + (uint32_t)(li * S + rank) * 512u + (uint32_t)lane * 16u, (uint32_t)to), v, cluster_map(bar, (uint32_t)to));
    }
  }
  if (S == 1) return;
  for (int li = warp; li < led; li += kExl3Warps) {
    bool ok = mbar_try_wait_cluster(bar, 0u);
    for (uint32_t spin = 0; spin < kWaitSpins && !ok; ++spin) {
      ok = mbar_try_wait_cluster(bar, 0u);
      if (!ok && *abort_word != 0) break;
    }
    if (!ok) {  // give up: these rows stay wrong, the error word tells the host
      *abort_word = 1;
      *a.err = 1;
      break;
    }
    const uint32_t src = stage_acquire(inbox) + (uint32_t)(li * S) * 512u + (uint32_t)lane * 16u;
    float4 v = lds128f(src);
    for (int q = 1; q < S; ++q) {
      const float4 o = lds128f(src + (uint32_t)q * 512u);
      v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
    }
    finish(li * S + rank, v);
  }
  // A CTA that received its rows may leave: nobody sends to it any more. One without rows, and one
  // that gave up, has nobody waiting for it but may still be sent to: see frag_kernel.
  if (__shfl_sync(0xffffffffu, *abort_word, 0) != 0) {
    cluster_arrive_relaxed();
    cluster_wait_relaxed();
  }
}

// ---- rotation: block Hadamard of 128 with a scale vector before or after (EXL3.swift:219-262) -------
template <class IT, class OT>
__global__ void __launch_bounds__(256) exl3_rotate_kernel(const IT *__restrict__ x, const __half *__restrict__ s, long long blocks,
                                                          int blocks_per_row, int pre, OT *__restrict__ y) {
  const int lane = threadIdx.x & 31;
  for (long long block = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); block < blocks; block += (long long)gridDim.x * 8) {
    const long long base = block * 128 + lane * 4;
    const long long col = (block % blocks_per_row) * 128 + lane * 4;
    float v[4], sc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = (float)x[base + i];
      sc[i] = __half2float(s[col + i]);
      if (pre) v[i] = __fmul_rn(v[i], sc[i]);
    }
    const float a0 = __fadd_rn(v[0], v[1]), a1 = __fsub_rn(v[0], v[1]), a2 = __fadd_rn(v[2], v[3]), a3 = __fsub_rn(v[2], v[3]);
    v[0] = __fadd_rn(a0, a2), v[2] = __fsub_rn(a0, a2), v[1] = __fadd_rn(a1, a3), v[3] = __fsub_rn(a1, a3);
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float p = __shfl_xor_sync(0xffffffffu, v[i], m);
        v[i] = (lane & m) ? __fsub_rn(p, v[i]) : __fadd_rn(v[i], p);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = __fmul_rn(v[i], 0.08838834764831845f);
      if (!pre) v[i] = __fmul_rn(v[i], sc[i]);
      y[base + i] = (OT)v[i];
    }
  }
}

template <int KA, bool HK, bool MUL1>
cudaError_t dequantize_as(const uint32_t *trellis, int tiles_k, int tiles_n, uint32_t mult, uint32_t add, void *out, int out_dtype,
                          int sm_count, cudaStream_t st) {
  const long long total = (long long)tiles_k * tiles_n;
  const int grid = (int)((total + 7) / 8 < (long long)sm_count * 8 ? (total + 7) / 8 : (long long)sm_count * 8);
  if (out_dtype == 2)
    exl3_dequantize_kernel<KA, HK, MUL1, float><<<grid, 256, 0, st>>>(trellis, tiles_k, tiles_n, mult, add, static_cast<float *>(out));
  else
    exl3_dequantize_kernel<KA, HK, MUL1, __half><<<grid, 256, 0, st>>>(trellis, tiles_k, tiles_n, mult, add, static_cast<__half *>(out));
  return cudaGetLastError();
}

// K split S (cluster size) and the chunk of k blocks staged at a time. The cost counts waves of
// clusters, each 1 / S of a group's work (about 4 ns per input: 20 us for 128 outputs of 5120), 3 us per
// wave for start, staging and sums.
template <int KA, bool HK, bool MUL1, int NB>
cudaError_t product_as(Exl3Args a, int sm_count, cudaStream_t st) {
  constexpr int kRingBytes = kExl3Slice<KA, HK> * kExl3Ring<KA, HK>;
  constexpr size_t kMost = 225 * 1024;
  const auto kernel = exl3_product_kernel<KA, HK, MUL1, NB>;
  static std::mutex lock;
  static std::map<int, int> clusters[9];  // per split: of a device, how many clusters run at once
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute at[2];
  cfg.blockDim = dim3(kExl3Warps * 32);
  cfg.attrs = at;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  // programmatic dependent launch: the launch itself overlaps the kernel ahead, whose end is waited for
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  int best = 0;
  double best_cost = 0;
  {
    std::lock_guard<std::mutex> g(lock);
    if (clusters[1].find(device) == clusters[1].end()) {
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost);
      for (int s = 1; s <= 8 && e == cudaSuccess; ++s) {
        cfg.gridDim = dim3(sm_count / s * s);
        cfg.dynamicSmemBytes = kMost;
        at[0].val.clusterDim.x = s;
        cfg.numAttrs = 1;
        int n = 0;
        e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
        clusters[s][device] = n;
      }
      if (e != cudaSuccess) {
        clusters[1].erase(device);
        return e;
      }
    }
    for (int s = 1; s <= 8 && s <= a.kblocks; ++s) {
      const int at_once = clusters[s][device];
      if (at_once < 1) continue;
      const double cost = ((a.groups + at_once - 1) / at_once) * ((double)a.K * 0.004 / s + 3.0) + 0.1 * s;
      if (!best || cost < best_cost) best = s, best_cost = cost;
    }
  }
  if (!best) return cudaErrorInvalidConfiguration;
  a.S = best;
  const int blocks = (a.kblocks + best - 1) / best;
  // the chunk: the CTA's whole share where it fits
  a.chunk = (blocks + 3) & ~3;
  while (a.chunk > 4 && exl3_smem_bytes(a.chunk, a.rows, a.S, NB, kRingBytes) > kMost) a.chunk = (a.chunk / 2 + 3) & ~3;
  cfg.gridDim = dim3((unsigned)(a.groups * a.S));
  cfg.dynamicSmemBytes = exl3_smem_bytes(a.chunk, a.rows, a.S, NB, kRingBytes);
  at[0].val.clusterDim.x = a.S;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

// rate (16-bit words per tile = 16 * bits) and codebook to the template arguments
template <class F>
cudaError_t by_rate(int words16, int codebook, F &&f) {
  const bool half = (words16 & 15) != 0;
  const int whole = words16 >> 4;
  if (codebook < 0 || codebook > 2 || (words16 & 7) || whole < 1 || whole > 8 || (half && (whole > 3 || codebook != 2)))
    return cudaErrorInvalidValue;
#define ISHI_EXL3_CASE(KA)                                                          \
  case KA:                                                                          \
    return codebook == 2 ? f(std::integral_constant<int, KA>(), std::false_type(), std::true_type()) \
                         : f(std::integral_constant<int, KA>(), std::false_type(), std::false_type());
  if (!half) {
    switch (whole) {
      ISHI_EXL3_CASE(1)
      ISHI_EXL3_CASE(2)
      ISHI_EXL3_CASE(3)
      ISHI_EXL3_CASE(4)
      ISHI_EXL3_CASE(5)
      ISHI_EXL3_CASE(6)
      ISHI_EXL3_CASE(7)
      ISHI_EXL3_CASE(8)
    }
  }
#undef ISHI_EXL3_CASE
  switch (whole) {
    case 1: return f(std::integral_constant<int, 1>(), std::true_type(), std::true_type());
    case 2: return f(std::integral_constant<int, 2>(), std::true_type(), std::true_type());
    case 3: return f(std::integral_constant<int, 3>(), std::true_type(), std::true_type());
  }
  return cudaErrorInvalidValue;
}

// multiplier and addend of the two codebooks that share a kernel
void codebook_constants(int codebook, uint32_t *mult, uint32_t *add) {
  *mult = codebook == 1 ? 0xCBAC1FEDu : 89226354u;
  *add = codebook == 1 ? 0u : 64248484u;
}

}  // namespace

bool exl3_rate_supported(int words16, int codebook) {
  const bool half = (words16 & 15) != 0;
  const int whole = words16 >> 4;
  return codebook >= 0 && codebook <= 2 && !(words16 & 7) && whole >= 1 && whole <= 8 && !(half && (whole > 3 || codebook != 2));
}

cudaError_t launch_exl3_dequantize(const int16_t *trellis, int tiles_k, int tiles_n, int words16, int codebook, void *out,
                                   int out_dtype, int sm_count, cudaStream_t st) {
  uint32_t mult, add;
  codebook_constants(codebook, &mult, &add);
  return by_rate(words16, codebook, [&](auto ka, auto hk, auto mul1) {
    return dequantize_as<decltype(ka)::value, decltype(hk)::value, decltype(mul1)::value>(
        reinterpret_cast<const uint32_t *>(trellis), tiles_k, tiles_n, mult, add, out, out_dtype, sm_count, st);
  });
}

cudaError_t launch_exl3_product(const int16_t *trellis, int tiles_k, int tiles_n, int words16, int codebook, const __half *x,
                                const __half *su, const __half *sv, int rows, void *y, int *err, int sm_count, cudaStream_t st) {
  Exl3Args a;
  memset(&a, 0, sizeof(a));
  a.trellis = reinterpret_cast<const uint8_t *>(trellis);
  a.x = x, a.su = su, a.sv = sv, a.y = y;
  a.K = (long long)tiles_k * 16, a.N = (long long)tiles_n * 16;
  a.rows = rows, a.groups = tiles_n / 8, a.kblocks = tiles_k / 8;
  a.wide = ((reinterpret_cast<uintptr_t>(trellis) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(su)) & 15u) == 0;
  a.err = err;
  codebook_constants(codebook, &a.mult, &a.add);
  return by_rate(words16, codebook, [&](auto ka, auto hk, auto mul1) {
    constexpr int KA = decltype(ka)::value;
    constexpr bool HK = decltype(hk)::value, MUL1 = decltype(mul1)::value;
    return rows > 8 ? product_as<KA, HK, MUL1, 2>(a, sm_count, st) : product_as<KA, HK, MUL1, 1>(a, sm_count, st);
  });
}

cudaError_t launch_exl3_rotate(const void *x, int x_dtype, long long rows, long long width, const __half *scales, int before,
                               void *y, int y_dtype, int sm_count, cudaStream_t st) {
  const long long blocks = rows * (width / 128);
  if (blocks == 0) return cudaSuccess;
  const int grid = (int)((blocks + 7) / 8 < (long long)sm_count * 8 ? (blocks + 7) / 8 : (long long)sm_count * 8);
  const int bpr = (int)(width / 128);
  if (x_dtype == 0 && y_dtype == 0)
    exl3_rotate_kernel<__half, __half><<<grid, 256, 0, st>>>(static_cast<const __half *>(x), scales, blocks, bpr, before, static_cast<__half *>(y));
  else if (x_dtype == 0 && y_dtype == 2)
    exl3_rotate_kernel<__half, float><<<grid, 256, 0, st>>>(static_cast<const __half *>(x), scales, blocks, bpr, before, static_cast<float *>(y));
  else if (x_dtype == 2 && y_dtype == 0)
    exl3_rotate_kernel<float, __half><<<grid, 256, 0, st>>>(static_cast<const float *>(x), scales, blocks, bpr, before, static_cast<__half *>(y));
  else if (x_dtype == 2 && y_dtype == 2)
    exl3_rotate_kernel<float, float><<<grid, 256, 0, st>>>(static_cast<const float *>(x), scales, blocks, bpr, before, static_cast<float *>(y));
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace ishi
