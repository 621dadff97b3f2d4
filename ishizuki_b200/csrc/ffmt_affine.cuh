// MLX affine group-quantized packs (8, 4 or 2 bits, fp16 or bf16 scales) for the warp-level kernel.
//
// Layout of the source (reference: Sources/IshizukiKit/Core/VerifyMatmul.swift:282-287 and
// Sources/IshizukiKit/Quantize/WeightedAffineQuantizer.swift:142-161): row n is K*bits/32
// little-endian uint32 words, code i of a word at bit i*bits; w = float(code) * scale + bias with
// one (scale, bias) pair per group of GS inputs.
//
// The product is factored per group as the reference's codes kernel does
// (VerifyMatmul.swift:123-128): y += s_g * sum_k code_k x_k + b_g * sum_k x_k. Codes masked in
// place are fp16 bit patterns of code * 2^-24 times the power of two of their bit position; that
// extra power of two is taken out on the activation side, where x is staged divided by it (exact
// unless |x| is tiny, where it costs at most half a unit in the last place of an fp16
// subnormal). The second sum uses fp32 group sums of x staged beside the fragments.
//
// Fragment mapping (m16n8k16; lane g = lane / 4, t = lane % 4 holds weight rows g and g + 8): of
// every four consecutive words ("quad" q; 8 bits: of every eight) lane t owns word 4q + t of both rows (8 bits: two). A
// word's codes lie where one mask, after at most one shift of the word, makes them A registers:
//   8 bits: k-step q:              a0 = codes (0, 1), a2 = codes (2, 3) of the word
//   4 bits: k-step (q, m), m < 2:  a0 = codes (4m, 4m + 1), a2 = codes (4m + 2, 4m + 3)
//   2 bits: k-step (q, m), m < 4:  a0 = codes (m, m + 8), a2 = codes (m + 4, m + 12)
// so a lane's activations of two k-steps are 16 consecutive bytes of a row: x is copied as it lies in memory and
// then divided by 2^(BITS * m) in place (2 bits: its pairs put in that order too; the order that the rotation on the tensor cores
// gives).
//
// The bias term is a tf32 MMA over the groups: the biases (11 bits at most) are exact in tf32, the fp32 group
// sums of x are three tf32 pieces, so it loses nothing to the operand. One or two instructions (three in groups of 32) and two to four
// conversions per tile, where a lane converted every bias and spent eight multiplications and additions on it. With that,
// the copied rows and the activations of two k-steps in one load, over weights from HBM, best plans, in us:
//   affine 4-bit, groups of 64:  4096 x 4096, sixteen / eight / one row  7.59 / 5.24 / 4.59 -> 7.10 / 5.11 / 4.55
//                                5120 x 17408, eight / one row  13.97 / 12.09 -> 12.22 / 11.43
//   groups of 32:                5120 x 17408, eight / one row  15.83 / 13.84 -> 12.99 / 12.15
//   8-bit, groups of 64:         8192 x 5120, eight / one row  9.41 / 8.94 -> 9.22 / 8.85
//   2-bit, groups of 64:         5120 x 17408, eight / one row  13.77 / 11.33 -> 12.08 / 10.63
//   ternary:                     34816 x 5120, sixteen / eight / one row  28.3 / 17.1 / 15.2 -> 27.1 / 17.1 / 15.1
// Error against 64 bits over six packs, three shapes, one to sixteen rows: outputs that are not the 64-bit result
// rounded 59773 of 8.9 million, 59856 before (groups of 128 7981, 8338 before; groups of 64 7048, 6858 before).
//
// Tile (16 rows x 256 k): BITS pieces of 512 bytes, piece j = [lane][row g: words of quads 2j and
// 2j + 1; row g + 8: the same], then the unit's scales of every row, then its biases.
#pragma once
#include <cuda_bf16.h>

#include "ishi_fragstream.cuh"

namespace ishi {

template <int BITS, int GS, bool BF16>
struct FragAffine : FragCopying {
  static_assert(BITS == 8 || BITS == 4 || BITS == 2, "8-, 4- and 2-bit codes");
  static_assert(GS == 32 || GS == 64 || GS == 128, "group sizes of the reference");
  static_assert(BITS != 2 || GS >= 64, "a 2-bit k-step spans 64 inputs");
  static constexpr int kGroups = 256 / GS;           // per unit
  static constexpr int kQuads = 2 * BITS;            // word quads per unit: 16 (64 words), 8 or 4
  static constexpr int kMasks = 8 / BITS;            // k-steps per quad: 1, 2 or 4
  static constexpr int kQuadK = 256 / kQuads;        // inputs a quad covers: 16, 32 or 64
  static constexpr int kHeader = BITS * 512;         // offset of the scales
  static constexpr int kRowScales = 2 * kGroups;     // bytes per row there, and of the biases behind them
  static constexpr int kBiases = kHeader + 16 * kRowScales;
  static constexpr int kTileBytes = kBiases + 16 * kRowScales;
  static constexpr int kSkew = BITS == 2 ? 16 : 64;  // of the rows against one another: 32 or 16 bytes of a row per lane and load
  static constexpr int kSumBytes = GS == 32 ? 640 : GS == 64 ? 384 : 256;  // per unit: the group sums' pieces, see store_sum()
  static constexpr double kUnit = 16777216.0;  // tile results come in units of 2^24: masked codes are q * 2^-24
  // The activations as they lie in x, then a pass that scales and adds up; a single row and rotated ones by loads and stores. Of
  // the packs that are rotated on the tensor cores all by loads and stores: both ways in one kernel take registers from the loop
  // (34816 x 5120, ternary, eight rows: 17.5 us against 17.1).
  static constexpr bool kRows = !(BITS == 2 && GS == 128), kRowSums = kRows;
  static constexpr bool kSumsLater = true;
  static constexpr int kExtraBytes = 0;  // shared memory per CTA beyond the staged regions
  static constexpr bool kRowMode = true;  // MODE 1: one activation row on CUDA cores
  static constexpr int kFewWarps = 20;  // most warps of the smaller block size at up to eight rows
  // most warps at nine to sixteen rows: a 2-bit pack without rotated inputs gains nothing from the registers
  static constexpr int kManyWarps = BITS == 2 && !BF16 ? 20 : 16;
  static constexpr int kXBytes = 8 * 512 + kSumBytes, kXFixed = 8 * kSkew;  // a staged region: per unit eight rows and the sums; the rows' skews

  static __device__ __forceinline__ uint16_t tile_halfword(const FragSrc &s, long long p, int u, int hw) {
    if (hw < kHeader / 2) {
      const int c = hw >> 8, lane = (hw & 255) >> 3, h = hw & 7;
      const int g = lane >> 2, t = lane & 3, second = (h & 3) >> 1, half = h & 1;
      const long long row = p * kFragRows + g + 8 * (h >> 2);
      if (row >= s.N) return 0;
      const long long word = (long long)u * (8 * BITS) + (BITS == 8 ? 8 * c + 2 * t + second : 4 * (2 * c + second) + t);
      long long local;
      const int seg = frag_segment(s, row, &local);
      const uint16_t *src = reinterpret_cast<const uint16_t *>(s.w[seg] + local * s.w_row_bytes + word * 4);
      const uint32_t w = (uint32_t)src[0] | ((uint32_t)src[1] << 16);
      if (BITS == 8)  // codes half, half + 2
        return (uint16_t)(((w >> (8 * half)) & 0xffu) | (((w >> (8 * half + 16)) & 0xffu) << 8));
      if (BITS == 4)  // codes half, half + 4, half + 2, half + 6
        return (uint16_t)(((w >> (4 * half)) & 15u) | (((w >> (4 * half + 16)) & 15u) << 4) | (((w >> (4 * half + 8)) & 15u) << 8) |
                          (((w >> (4 * half + 24)) & 15u) << 12));
      return src[half];
    }
    const int idx = (hw - kHeader / 2) % (16 * kGroups);
    const long long row = p * kFragRows + idx / kGroups;
    if (row >= s.N) return 0;
    long long local;
    const int seg = frag_segment(s, row, &local);
    const uint8_t *base = hw < kBiases / 2 ? s.scales[seg] : s.biases[seg];
    return *reinterpret_cast<const uint16_t *>(base + local * s.s_row_bytes + ((long long)u * kGroups + idx % kGroups) * 2);
  }

  // x * 2^-e on both halves (exact power-of-two scaling)
  template <int E>
  static __device__ __forceinline__ uint32_t scale_down(uint32_t v) {
    if (E == 0) return v;
    const __half2 f = __float2half2_rn(1.0f / (float)(1 << E));
    const __half2 r = __hmul2(*reinterpret_cast<const __half2 *>(&v), f);
    return *reinterpret_cast<const uint32_t *>(&r);
  }

  static __device__ __forceinline__ uint32_t row_stride(const FragArgs &a) { return (uint32_t)a.umax * 512u + (uint32_t)kSkew; }
  // the sums of unit u: behind the eight rows
  static __device__ __forceinline__ uint32_t sums_of(const FragArgs &a, uint32_t xfrag, int u) {
    return xfrag + 8u * row_stride(a) + (uint32_t)(u * kSumBytes);
  }

  // lane l's eight activations k = 8l .. 8l + 7 of a unit as the product reads them
  static __device__ __forceinline__ uint4 arranged(uint4 v, int lane) {
    if (BITS == 8) return v;
    if (BITS == 4) return make_uint4(v.x, v.y, scale_down<4>(v.z), scale_down<4>(v.w));
    // half of word l / 2 (codes 0..7 when l is even, 8..15 when odd): the even lane builds m = 0, 1 and the odd
    // lane m = 2, 3, each with the other's half of the word
    const bool odd = lane & 1;
    const uint32_t ox = __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 1), oz = __shfl_xor_sync(0xffffffffu, odd ? v.z : v.w, 1);
    // codes (0, 1) or (2, 3), (4, 5) or (6, 7) of the word, and the eight codes further on
    const uint32_t la = odd ? ox : v.x, lb = odd ? oz : v.z, ha = odd ? v.y : ox, hb = odd ? v.w : oz;
    const uint4 r = make_uint4(prmt(la, ha, 0x5410u), prmt(lb, hb, 0x5410u), prmt(la, ha, 0x7632u), prmt(lb, hb, 0x7632u));
    const uint32_t s0 = odd ? 0x2c002c00u : 0x3c003c00u, s1 = odd ? 0x24002400u : 0x34003400u;  // 1 / 16, 1; 1 / 64, 1 / 4
    return make_uint4(times(r.x, s0), times(r.y, s0), times(r.z, s1), times(r.w, s1));
  }
  static __device__ __forceinline__ uint32_t times(uint32_t v, uint32_t f) {
    const __half2 r = __hmul2(*reinterpret_cast<const __half2 *>(&v), *reinterpret_cast<const __half2 *>(&f));
    return *reinterpret_cast<const uint32_t *>(&r);
  }

  // The sum of x over a group of activation row r, in the codes' unit, as three tf32 pieces where the B registers of lane
  // (r, t) find them: groups of 64: group t = j, [lane][hi mid] and behind them [lane][lo]; of 32: groups 2t and 2t + 1,
  // [hi hi], [mid mid], [lo lo]; of 128: group t / 2, [hi lo] in the even lane, [mid 0] in the odd one.
  // hi and mid take eleven bits each of the 24, lo has two at most: it is exact in a bf16, as which it is kept for
  // groups of 32 (the widest inputs have no room for more).
  struct Pieces {
    uint32_t hi, mid, lo;
  };
  static __device__ __forceinline__ void store_lo(uint32_t addr, uint32_t lo) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((uint16_t)(lo >> 16)) : "memory");
  }
  static __device__ __forceinline__ Pieces pieces_of(float sum) {
    const float s = sum * (1.f / 16777216.f);
    Pieces p;
    p.hi = __float_as_uint(s) & 0xffffe000u;
    const float rest = __uint_as_float(p.hi) == s ? 0.f : s - __uint_as_float(p.hi);  // (an infinite sum has one piece)
    p.mid = __float_as_uint(rest) & 0xffffe000u;
    p.lo = __float_as_uint(rest - __uint_as_float(p.mid));
    return p;
  }
  static __device__ __forceinline__ void store_sum(uint32_t base, int r, int j, float sum) {
    const Pieces p = pieces_of(sum);
    if (GS == 64) {
      sts64(base + (uint32_t)((r * 4 + j) * 8), p.hi, p.mid);
      sts32(base + 256u + (uint32_t)((r * 4 + j) * 4), p.lo);
    } else if (GS == 32) {
      const uint32_t at = base + (uint32_t)((r * 4 + (j >> 1)) * 8 + (j & 1) * 4);
      sts32(at, p.hi), sts32(at + 256u, p.mid);
      store_lo(base + 512u + (uint32_t)(r * 16 + j * 2), p.lo);
    } else {
      sts64(base + (uint32_t)((r * 4 + 2 * j) * 8), p.hi, p.lo);
      sts64(base + (uint32_t)((r * 4 + 2 * j + 1) * 8), p.mid, 0u);
    }
  }

  // The sums of activation row g's groups from those of its inputs 64 t ... + 31 (s0) and + 32 ... + 63 (s1), if the row is `mine`
  static __device__ __forceinline__ void store_sums(uint32_t base, int lane, float s0, float s1, bool mine) {
    const int g = lane >> 2, t = lane & 3;
    if (GS == 128) s0 += s1, s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    if (!mine) return;
    if (GS == 32) {
      store_sum(base, g, 2 * t, s0), store_sum(base, g, 2 * t + 1, s1);
    } else {
      if (GS == 64) s0 += s1;
      if (GS == 64 || !(t & 1)) store_sum(base, g, GS == 64 ? t : t >> 1, s0);
    }
  }

  // After the copies: a warp task per unit and four rows. The sums by MMAs with a weight of ones, as in ffmt_q4k.cuh: lane (g, t) gets those of
  // inputs 64 t ... + 31 and + 32 ... + 63 of activation row g.
  static __device__ __forceinline__ void row_sums(const FragArgs &a, uint32_t xfrag, int rows, int uc) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t R = row_stride(a), x = stage_acquire(xfrag);
    constexpr uint32_t kOnes = 0x3c003c00u;
    const FragPass pass(rows, uc);
    for (int i = warp; i < pass.tasks; i += nw) {
      const int u = pass.unit(i), r0 = pass.row(i);
      float s0 = 0.f, s1 = 0.f;
      uint4 v[4];  // (rows past the live ones: whatever is there, for columns of no row)
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = lds128(x + (uint32_t)(r0 + e) * R + (uint32_t)u * 512u + (uint32_t)lane * 16u);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t at = x + (uint32_t)(r0 + e) * R + (uint32_t)u * 512u + (uint32_t)lane * 16u;
        const uint4 w = arranged(v[e], lane);
        if (BITS == 4) sts64(at + 8u, w.z, w.w);
        if (BITS == 2) sts128u(at, w);
        float c[4];
        mma16816_first(c, kOnes, kOnes, kOnes, kOnes, v[e].x, v[e].y);
        mma16816(c, kOnes, kOnes, kOnes, kOnes, v[e].z, v[e].w);
        if (g == r0 + e) s0 = c[0], s1 = c[1];
      }
      store_sums(sums_of(a, x, u), lane, s0, s1, (g & 4) == r0);
    }
  }

  // is the input rotated on the tensor cores, by stage_x_rot128()?
  static __device__ __forceinline__ bool rotated_128(const FragArgs &a) { return BITS == 2 && GS == 128 && a.rot_block == 128 && !a.rot_signs; }
  // Rotated activations, on their way from x, and a single row, which is added up on the way too. A warp task is (unit,
  // activation row): lane l loads the eight values k = 8l .. 8l + 7. (Several rotated rows leave the sums to row_sums() as copied ones do:
  // the same bits as from an input rotated before.)
  template <class Then>
  static __device__ __forceinline__ void stage_x(const FragArgs &a, const FragRows &m, uint32_t xfrag, int ub0, int uc, Then then) {
    if (rotated_128(a)) {
      stage_x_rot128(a, m, xfrag, ub0, uc, then);
      return;
    }
    const int lane = threadIdx.x & 31;
    const uint32_t R = row_stride(a);
    frag_stage_rows(a, m, ub0, uc, then, [&](int u, int r, uint4 v) {
      if (a.rot_block)
        v = frag_rotate8(v, a.rot_block,
                            a.rot_signs ? a.rot_signs + (long long)(ub0 + u) * 256 + lane * 8 : nullptr, lane);
      sts128u(xfrag + (uint32_t)r * R + (uint32_t)u * 512u + (uint32_t)lane * 16u, kRows && m.staged != 1 ? v : arranged(v, lane));
      if (kRows && m.staged != 1) return;
      if (kRows) {  // as row_sums() has them: a row's product has the same bits alone and beside others
        constexpr uint32_t kOnes = 0x3c003c00u;
        float c[4];
        mma16816_first(c, kOnes, kOnes, kOnes, kOnes, v.x, v.y);
        mma16816(c, kOnes, kOnes, kOnes, kOnes, v.z, v.w);
        store_sums(sums_of(a, xfrag, u), lane, c[0], c[1], (lane >> 2) == r);
        return;
      }
      const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&v.x));
      const float2 f1 = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
      const float2 f2 = __half22float2(*reinterpret_cast<const __half2 *>(&v.z));
      const float2 f3 = __half22float2(*reinterpret_cast<const __half2 *>(&v.w));
      float s = ((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y));
#pragma unroll
      for (int d = 1; d < GS / 8; d *= 2) s += __shfl_xor_sync(0xffffffffu, s, d);
      if ((lane & (GS / 8 - 1)) == 0) store_sum(sums_of(a, xfrag, u), r, lane / (GS / 8), s);
    });
  }

  // +1 or -1 in fp16 by the parity of v
  static __device__ __forceinline__ uint32_t sign_half(int v) { return 0x3c00u | ((uint32_t)(__popc(v) & 1) << 15); }
  static __device__ __forceinline__ uint32_t pack_rn(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
  }

  // The 2-bit staging with the block Hadamard rotation of 128 (no sign vector) on the tensor
  // cores. With k = 8 i + j inside a block (i < 16, j < 8) the natural-order transform factors as
  // H128 = H16 (x) H8, so the rotated block, seen as the matrix Y[j'][i'], is H8 * X^T * H16:
  //   stage 1: Z[j'][i] = sum_j H8[j'][j] x[8 i + j]. One m16n8k16 takes both blocks of a unit:
  //     A = [H8 0; 0 H8] (rows j' of the first block, then of the second), B rows k = j of the
  //     first block then of the second, columns i of one half (eight of the sixteen): lane
  //     (g, t) supplies the 32-bit word g * 4 + t of that half, a coalesced load.
  //   stage 2: Y[j'][i'] = sum_i Z[j'][i] H16[i][i'], A = Z of both blocks (the fp32 sums of
  //     stage 1 as fp16 high and low parts, two MMAs, so nothing is lost to the fp16 operand),
  //     B = H16, columns i' of one half.
  // The fp32 result times 1 / sqrt(128) is rounded to fp16 as the butterfly's is; the two agree
  // to fp32 rounding. Lane (g, t) ends up with the values k' = 16 (4 h + t) + g and + 8 of each
  // block: the codes g and g + 8 of the block's word 4 h + t, which are one B register of the
  // product's k-step (quad 2 block + h, mask g % 4), low register when g < 4: word 2 (g % 4) + g / 4 of the eight that
  // lane t reads (a warp's stores meet all banks).
  template <class Then>
  static __device__ __forceinline__ void stage_x_rot128(const FragArgs &a, const FragRows &rows, uint32_t xfrag, int ub0, int uc, Then then) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    constexpr int kBatch = 8;
    constexpr uint32_t kOnes = 0x3c003c00u;
    const uint32_t R = row_stride(a);
    const uint32_t h8 = sign_half(g & (2 * t)) | (sign_half(g & (2 * t + 1)) << 16);
    uint32_t h16[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = 8 * h + g;
      h16[h][0] = sign_half(n & (2 * t)) | (sign_half(n & (2 * t + 1)) << 16);
      h16[h][1] = sign_half(n & (2 * t + 8)) | (sign_half(n & (2 * t + 9)) << 16);
    }
    const int m = g & 3;
    const uint32_t down1 = (uint32_t)(15 - 2 * m) << 10;  // 2^-(2 m) in fp16
    const uint32_t down = down1 | (down1 << 16);
    const float scale = 1.0f / sqrtf(128.f);
    const uint32_t *xl = reinterpret_cast<const uint32_t *>(rows.x + (long long)ub0 * 256) + lane;
    const int tasks = uc * rows.staged;
    int i0 = warp;
    do {
      uint32_t v[kBatch][4];  // [block * 2 + half]
#pragma unroll
      for (int e = 0; e < kBatch; ++e) {
        const int i = i0 + e * nw;
        const int2 task = rows.task(i);
        const bool live = i < tasks && task.y < rows.live;
        const uint32_t *src = xl + (long long)task.y * (a.K >> 1) + task.x * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c) v[e][c] = live ? __ldg(src + 32 * c) : 0u;
      }
      if (i0 == warp) then();
#pragma unroll
      for (int e = 0; e < kBatch; ++e) {
        const int i = i0 + e * nw;
        if (i >= tasks) break;
        const int2 task = rows.task(i);
        const int r = task.y;
        if (r >= rows.stored) continue;  // two 27B layers in ternary at four rows: 106.2 -> 102.3 us
        const uint32_t base = xfrag + (uint32_t)r * R + (uint32_t)task.x * 512u + (uint32_t)(t * 32 + (g & 3) * 8 + (g >> 2) * 4);
        uint32_t zh[4], zl[4];  // stage 2's A registers: (block 0, half 0), (block 1, half 0), (block 0, half 1), (block 1, half 1)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float z[4];
          mma16816_first(z, h8, 0u, 0u, h8, v[e][h], v[e][2 + h]);
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const uint32_t hi = pack_rn(z[2 * b], z[2 * b + 1]);
            const float2 hf = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
            zh[2 * h + b] = hi;
            zl[2 * h + b] = pack_rn(z[2 * b] - hf.x, z[2 * b + 1] - hf.y);
          }
        }
        uint32_t pr[2][2];  // [block][half]: two rotated values
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float y[4];
          mma16816_first(y, zh[0], zh[1], zh[2], zh[3], h16[h][0], h16[h][1]);
          mma16816(y, zl[0], zl[1], zl[2], zl[3], h16[h][0], h16[h][1]);
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            pr[b][h] = pack_rn(__fmul_rn(y[2 * b], scale), __fmul_rn(y[2 * b + 1], scale));
            const __half2 sc = __hmul2(*reinterpret_cast<const __half2 *>(&pr[b][h]), *reinterpret_cast<const __half2 *>(&down));
            const int q = 2 * b + h;
            sts32(base + (uint32_t)q * 128u, *reinterpret_cast<const uint32_t *>(&sc));
          }
        }
        // fp32 sums of the rounded values over each block (the group of the bias term), again by an MMA with ones: over the
        // lanes of a column, then over the columns. Lanes 0 to 3 store the blocks' pieces (see store_sum()).
        float sum[2];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          float c[4];
          mma16816_first(c, kOnes, kOnes, kOnes, kOnes, pr[b][0], pr[b][1]);
          sum[b] = c[0] + c[1];
          sum[b] += __shfl_xor_sync(0xffffffffu, sum[b], 1);
          sum[b] += __shfl_xor_sync(0xffffffffu, sum[b], 2);
        }
        const Pieces p = pieces_of(lane & 2 ? sum[1] : sum[0]);
        if (lane < 4) sts64(sums_of(a, xfrag, task.x) + (uint32_t)((r * 4 + lane) * 8), lane & 1 ? p.mid : p.hi, lane & 1 ? 0u : p.lo);
      }
      i0 += nw * kBatch;
    } while (i0 < tasks);
  }

  static __device__ __forceinline__ float param(uint32_t pair, int hi) {
    if (BF16) return hi ? __uint_as_float(pair & 0xffff0000u) : __uint_as_float(pair << 16);
    return half_bits_to_float(hi ? pair >> 16 : pair & 0xffffu);
  }
  static __device__ __forceinline__ float half_lo(uint32_t pair) { return __half2float(__ushort_as_half((unsigned short)(pair & 0xffffu))); }
  static __device__ __forceinline__ float half_hi(uint32_t pair) { return __half2float(__ushort_as_half((unsigned short)(pair >> 16))); }

  // One tile against the activations of its unit. acc: the warp's C fragment (MODE 0) or this
  // lane's partial dot products of rows g (acc[0]) and g + 8 (acc[2]) (MODE 1).
  template <int MODE, int NB>
  static __device__ __forceinline__ void unit(float (&acc)[NB][4], const FragArgs &a, uint32_t tile, uint32_t xbase,
                                              uint32_t tables, int uq, int g, int t, int lane) {
    // the scales of the two rows, halfwords in pairs
    constexpr int kWords = kGroups > 2 ? kGroups / 2 : 1;
    uint32_t sc0[kWords], sc1[kWords];
    if (kGroups == 8) {
      const uint4 p0 = lds128(tile + kHeader + (uint32_t)g * 16u), p1 = lds128(tile + kHeader + (uint32_t)(g + 8) * 16u);
      sc0[0] = p0.x, sc0[1 % kWords] = p0.y, sc0[2 % kWords] = p0.z, sc0[3 % kWords] = p0.w;
      sc1[0] = p1.x, sc1[1 % kWords] = p1.y, sc1[2 % kWords] = p1.z, sc1[3 % kWords] = p1.w;
    } else if (kGroups == 4) {
      const uint2 p0 = lds64(tile + kHeader + (uint32_t)g * 8u), p1 = lds64(tile + kHeader + (uint32_t)(g + 8) * 8u);
      sc0[0] = p0.x, sc0[1 % kWords] = p0.y, sc1[0] = p1.x, sc1[1 % kWords] = p1.y;
    } else {
      sc0[0] = lds32(tile + kHeader + (uint32_t)g * 4u), sc1[0] = lds32(tile + kHeader + (uint32_t)(g + 8) * 4u);
    }
    // The bias term: this lane's groups (see store_sum()) of rows g and g + 8, the smallest pieces first (an MMA cuts its
    // sum off, so the large ones enter once). First, so that its latency is covered; last in the
    // packs rotated on the tensor cores, whose loop has no registers to spare (34816 x 5120, ternary, four rows: 16.5 us first,
    // 16.4 last; affine 4-bit 5120 x 17408, eight rows: 12.25 and 12.5).
    constexpr bool kBiasLast = BITS == 2 && GS == 128;
    auto bias_term = [&] {
      float b0, b1, b2 = 0.f, b3 = 0.f;
      if (GS == 32) {
        const uint32_t p0 = lds32(tile + kBiases + (uint32_t)(g * 16 + t * 4)), p1 = lds32(tile + kBiases + (uint32_t)((g + 8) * 16 + t * 4));
        b0 = param(p0, 0), b2 = param(p0, 1), b1 = param(p1, 0), b3 = param(p1, 1);
      } else {
        const uint32_t at = tile + kBiases + (uint32_t)(g * kRowScales) + (uint32_t)((GS == 64 ? t : t >> 1) * 2);
        b0 = param(lds16(at), 0), b1 = param(lds16(at + 8 * kRowScales), 0);
      }
      const uint32_t sums = sums_of(a, xbase, uq) + (uint32_t)lane * 8u;
      if (MODE == 0) {
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          const uint32_t xs = sums + nb * a.xregion;
          if (GS == 32) {
            const uint32_t lo = lds32(xs + 512u - (uint32_t)lane * 4u);
            mma1688_tf32(acc[nb], b0, b1, b2, b3, lo << 16, lo & 0xffff0000u);
#pragma unroll
            for (int i = 1; i >= 0; --i) {
              const uint2 p = lds64(xs + 256u * i);
              mma1688_tf32(acc[nb], b0, b1, b2, b3, p.x, p.y);
            }
          } else {
            const uint2 p = lds64(xs);
            if (GS == 64) mma1684_tf32(acc[nb], b0, b1, lds32(xs + 256u - (uint32_t)lane * 4u));
            mma1688_tf32(acc[nb], b0, b1, b0, b1, p.x, p.y);
          }
        }
      } else {  // the lane's share of the bias terms of activation row 0, its groups' pieces
        const uint32_t xs = sums - (uint32_t)g * 32u;
        if (GS == 32) {
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            float2 p;
            if (i < 2) {
              p = lds64f(xs + 256u * i);
            } else {
              const uint32_t lo = lds32(xs + 512u - (uint32_t)t * 4u);
              p = make_float2(__uint_as_float(lo << 16), __uint_as_float(lo & 0xffff0000u));
            }
            acc[0][0] += b0 * p.x + b2 * p.y, acc[0][2] += b1 * p.x + b3 * p.y;
          }
        } else {
          const float2 p = lds64f(xs);
          float s = p.x + p.y;
          if (GS == 64) s += lds32f(xs + 256u - (uint32_t)t * 4u);
          acc[0][0] += b0 * s, acc[0][2] += b1 * s;
        }
      }
    };
    if (!kBiasLast) bias_term();

    const uint32_t R = row_stride(a);
    const uint32_t xrow = xbase + (uint32_t)(MODE == 0 ? g : 0) * R + (uint32_t)uq * 512u + (uint32_t)t * (BITS == 2 ? 32u : 16u);
    float part[NB][4];
#pragma unroll
    for (int j = 0; j < BITS; ++j) {
      const uint4 w = lds128(tile + (uint32_t)j * 512u + (uint32_t)lane * 16u);  // row g: w.x, w.y; row g + 8: w.z, w.w
      uint4 b[NB];  // two k-steps' activations
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int q = 2 * j + s;
        const uint32_t x0 = s ? w.y : w.x, x1 = s ? w.w : w.z;
        const uint32_t y0 = x0 >> 8, y1 = x1 >> 8;
#pragma unroll
        for (int m = 0; m < kMasks; ++m) {
          const int step = kMasks * q + m;  // k-step of the unit
          if (!(step & 1))
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
              b[nb] = lds128(xrow + nb * a.xregion + (BITS == 2 ? (uint32_t)(step >> 2) * 128u + (uint32_t)((step >> 1) & 1) * 16u : (uint32_t)(step >> 1) * 64u));
          const uint32_t mask = (BITS == 8 ? 0x00ff00ffu : BITS == 4 ? 0x000f000fu : 0x00030003u) << (BITS * m);
          const uint32_t a0 = x0 & mask, a1 = x1 & mask, a2 = y0 & mask, a3 = y1 & mask;
          const bool first = (step * 16) % GS == 0;  // first k-step of a group
          if (MODE == 0) {
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
              const uint32_t e0 = step & 1 ? b[nb].z : b[nb].x, e1 = step & 1 ? b[nb].w : b[nb].y;
              if (first) mma16816_first(part[nb], a0, a1, a2, a3, e0, e1);
              else mma16816(part[nb], a0, a1, a2, a3, e0, e1);
            }
          } else {
            const uint32_t e0 = step & 1 ? b[0].z : b[0].x, e1 = step & 1 ? b[0].w : b[0].y;
            float(&d)[4] = part[0];
            if (first) d[0] = d[1] = d[2] = d[3] = 0.f;
            d[0] = fmaf(half_lo(a0), half_lo(e0), d[0]);
            d[0] = fmaf(half_hi(a0), half_hi(e0), d[0]);
            d[0] = fmaf(half_lo(a2), half_lo(e1), d[0]);
            d[0] = fmaf(half_hi(a2), half_hi(e1), d[0]);
            d[2] = fmaf(half_lo(a1), half_lo(e0), d[2]);
            d[2] = fmaf(half_hi(a1), half_hi(e0), d[2]);
            d[2] = fmaf(half_lo(a3), half_lo(e1), d[2]);
            d[2] = fmaf(half_hi(a3), half_hi(e1), d[2]);
          }
          if (((step + 1) * 16) % GS == 0) {  // the group is complete: scale its code sum
            const int grp = step * 16 / GS;
            const float s0 = param(sc0[grp >> 1], grp & 1), s1 = param(sc1[grp >> 1], grp & 1);
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
              acc[nb][0] = fmaf(s0, part[nb][0], acc[nb][0]);
              if (MODE == 0) acc[nb][1] = fmaf(s0, part[nb][1], acc[nb][1]);
              acc[nb][2] = fmaf(s1, part[nb][2], acc[nb][2]);
              if (MODE == 0) acc[nb][3] = fmaf(s1, part[nb][3], acc[nb][3]);
            }
          }
        }
      }
    }
    if (kBiasLast) bias_term();
  }
};

}  // namespace ishi
