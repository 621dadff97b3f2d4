// GGUF Q6_K for the warp-level kernel (mma.sync fragments).
//
// Block layout (210 bytes per 256 weights; reference: Sources/IshizukiKit/Core/GGMLDequant.swift,
// the Q6_K decoder, and the matvec body in Sources/IshizukiKit/Core/GGMLKernels.swift):
//   ql[128] low nibbles @0, qh[64] high bit pairs @128, sixteen int8 scales @192, d f16 @208.
//   Weight k = 128n + 32c + l (half n, quarter c, l < 32) has its low nibble in ql[64n + 32(c&1) + l]
//   (the high nibble of that byte when c >= 2) and its two high bits at bit 2c of qh[32n + l];
//   w = d * scale[k / 16] * (q - 32).
//
// The product is factored as
//   y += d * (sum_g scale_g * sum_{k in g} q_k x_k  -  32 * sum_g scale_g * sum_{k in g} x_k),
// g running over the sixteen groups of 16 weights. A group is exactly one k-step of the MMA, so
// every k-step's accumulator takes its (exact, fp32) scale afterwards; the second sum is one more
// MMA whose k index runs over the groups, against the group sums of x.
//
// A 6-bit value at bits 4..9 of each half of a register is the bit pattern of the fp16 number
// q * 2^-20 (subnormal, hence linear in q). A pair of k-steps (2i, 2i + 1) takes eight A registers per
// lane, sixteen values, and they lie in three words: each half of a word has one value at bits 4..9 (a
// register for one mask), one at bits 10..15 (a shift and a mask) and four bits below; the low nibbles of
// the first k-step's row g are those of words 0 and 1, their high bit pairs bits 0..1 and 2..3 of word 2.
// These two are put together at bits 0..5, q * 2^-24, and multiplied by sixteen as half2. That is
// fifteen bit operations and two multiplies for eight registers, where nibbles and bit pairs in words of
// their own take twenty-one.
// All registers hold one unit, and both rows of a lane add up their k-steps in the same order, because a
// weight row's product must not depend on which half of a panel it lies in (or a gated pair and the same
// two weights stacked differ) and the MMA's rounding depends on the unit: codes at bits 0..5 lose more
// low bits of a product. With row g's first k-steps left at 2^-24 and in sums of their own 112 of 65536
// products of a weight turned by eight rows changed. Of 393216 products (8192 x 5120) 522 are not the
// 64-bit result rounded to fp16, 617 with that, 683 with both rows' first k-steps at 2^-24, 750 with one
// sum besides. The half2 multiplies cost 1 to 2 %, shifts in their place 2 %.
// The loop is bound by the integer pipe and by memory in equal parts: 17408 x 5120 at eight rows 19.1
// -> 17.1 us (23.5 at sixteen); 248320 x 5120 at eight rows 213 -> 177 us in short runs, 5.9 TB/s (a
// loop of seconds runs into the power cap: 219).
// Inside a k-step the lane t holds the weights 4t .. 4t + 3 of the group: slots (2t, 2t + 1) are
// 4t, 4t + 1 and slots (2t + 8, 2t + 9) are 4t + 2, 4t + 3; the activations are copied as they lie in x and put in that
// order in place (frag_rows_by_16()), so that a lane reads the B registers of two k-steps with one 16-byte load. Over weights
// from HBM, best plans, 17408 x 5120 at four / one row 16.5 / 16.1 -> 16.3 / 15.2 us, 5120 x 17408 18.6 / 17.5 -> 18.1 / 16.9.
//
// Tile (16 rows x 256 k, 3360 bytes = 16 * 210): [6][lane][16 bytes] = the lane's words 3 i + w of
// pair i, four at a time; per row the sixteen scales + 128 @3072 (a lane's A registers of the group-sum MMA, groups 4t .. 4t + 3,
// are one word), and d of rows (g, g + 8) side by side @3328.
#pragma once
#include "ishi_fragstream.cuh"

namespace ishi {

struct FragQ6K : FragCopying {
  static constexpr int kTileBytes = 16 * 210;
  static constexpr int kSumBytes = 512;           // per unit: [lane][hi hi | lo lo] group sums
  static constexpr int kXBytes = 8 * 512 + kSumBytes, kXFixed = 8 * 64;  // a staged region: per unit eight rows and the sums; the rows' skews
  static constexpr double kUnit = 16777216.0;  // tile results come in units of 2^24: masked codes are q * 2^-24
  static constexpr bool kRows = true, kRowSums = true;  // the activations as they lie in x, then put in order and added up
  // five to eight rows by loads and stores, which arrange and add up on the way (4096 x 4096 at eight rows, copied: 6.36 us against 6.28)
  static constexpr int kCopyRows = 4;
  static constexpr int kExtraBytes = 0;  // shared memory per CTA beyond the staged regions
  static constexpr bool kRowMode = false;         // one activation row runs through the MMA path as well
  static constexpr int kFewWarps = 16;  // most warps of the smaller block size at up to eight rows
  static constexpr int kManyWarps = 16;  // most warps at nine to sixteen rows

  // the low four and the high two bits of weight k of a block
  static __device__ __forceinline__ uint32_t low4(const uint8_t *blk, int k) {
    const int n = k >> 7, c = (k >> 5) & 3, l = k & 31;
    return ((uint32_t)blk[64 * n + 32 * (c & 1) + l] >> (c >= 2 ? 4 : 0)) & 15u;
  }
  static __device__ __forceinline__ uint32_t high2(const uint8_t *blk, int k) {
    const int n = k >> 7, c = (k >> 5) & 3, l = k & 31;
    return ((uint32_t)blk[128 + 32 * n + l] >> (2 * c)) & 3u;
  }
  static __device__ __forceinline__ uint32_t code(const uint8_t *blk, int k) { return low4(blk, k) | (high2(blk, k) << 4); }

  static __device__ __forceinline__ const uint8_t *block(const FragSrc &s, long long row, int u) {
    long long local;
    const int seg = frag_segment(s, row, &local);
    return s.w[seg] + local * s.w_row_bytes + (long long)u * 210;
  }

  static __device__ __forceinline__ uint16_t tile_halfword(const FragSrc &s, long long p, int u, int hw) {
    const int h = hw & 1;  // half of a word
    if (hw < 1536) {
      const int lane = (hw & 255) >> 3, word = 4 * (hw >> 8) + ((hw & 7) >> 1), pi = word / 3, w = word - 3 * pi;
      const int g = lane >> 2, t = lane & 3;
      const long long row = p * kFragRows + g;
      const uint8_t *top = row < s.N ? block(s, row, u) : nullptr, *low = row + 8 < s.N ? block(s, row + 8, u) : nullptr;
      // weights of k-steps 2 pi (k0) and 2 pi + 1, slots (2t, 2t + 1); two further on: slots (2t + 8, 2t + 9)
      const int k0 = 32 * pi + 4 * t + h, k1 = k0 + 16;
      uint32_t out = 0;
      if (w == 0) {
        if (top) out = low4(top, k0) | (code(top, k1) << 4);
        if (low) out |= code(low, k0) << 10;
      } else if (w == 1) {
        if (top) out = low4(top, k0 + 2);
        if (low) out |= (code(low, k1) << 4) | (code(low, k0 + 2) << 10);
      } else {
        if (top) out = high2(top, k0) | (high2(top, k0 + 2) << 2) | (code(top, k1 + 2) << 4);
        if (low) out |= code(low, k1 + 2) << 10;
      }
      return (uint16_t)out;
    }
    if (hw < 1664) {
      const int row16 = (hw - 1536) >> 3, pair = (hw - 1536) & 7;
      const long long row = p * kFragRows + row16;
      if (row >= s.N) return 0;
      const uint8_t *sc = block(s, row, u) + 192 + 2 * pair;
      return (uint16_t)(((uint32_t)sc[0] | ((uint32_t)sc[1] << 8)) ^ 0x8080u);
    }
    const long long row = p * kFragRows + ((hw - 1664) >> 1) + 8 * h;
    if (row >= s.N) return 0;
    const uint8_t *blk = block(s, row, u);
    return (uint16_t)((uint32_t)blk[208] | ((uint32_t)blk[209] << 8));
  }

  static __device__ __forceinline__ uint32_t row_stride(const FragArgs &a) { return (uint32_t)a.umax * 512u + 64u; }

  static __device__ __forceinline__ void row_sums(const FragArgs &a, uint32_t xfrag, int rows, int uc) {
    frag_rows_by_16<false>(xfrag, row_stride(a), xfrag + 8u * row_stride(a), kSumBytes, rows, uc, 0u);
  }
  // Rows on their way from x. A warp task is (unit, row): lane l loads k = 8l .. 8l + 7.
  template <class Then>
  static __device__ __forceinline__ void stage_x(const FragArgs &a, const FragRows &m, uint32_t xfrag, int ub0, int uc, Then then) {
    const uint32_t R = row_stride(a);
    frag_stage_rows(a, m, ub0, uc, then, [&](int u, int r, uint4 v) {
      frag_put_by_16<false>(xfrag + (uint32_t)r * R + (uint32_t)u * 512u, xfrag + 8u * R + (uint32_t)(u * kSumBytes), r, v, 0u);
    });
  }

  // byte `byte` of a word of scales + 128 as the scale: the low mantissa bits of 2^23
  static __device__ __forceinline__ float scale_of(uint32_t word, int byte) {
    return __uint_as_float(prmt(word, 0x4b000000u, 0x7650u + (uint32_t)byte)) - 8388736.f;
  }
  // both halves times sixteen, exact
  static __device__ __forceinline__ uint32_t times16(uint32_t v) {
    const __half2 r = __hmul2(*reinterpret_cast<const __half2 *>(&v), __float2half2_rn(16.f));
    return *reinterpret_cast<const uint32_t *>(&r);
  }
  // two of its bytes as a half2: the low mantissa bits of 1024
  static __device__ __forceinline__ uint32_t scale_pair(uint32_t word, uint32_t selector) {
    const uint32_t bits = prmt(word, 0x64646464u, selector);
    const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&bits), __float2half2_rn(1152.f));
    return *reinterpret_cast<const uint32_t *>(&v);
  }

  // One tile against the activations of its unit; acc is the warp's C fragment.
  template <int MODE, int NB>
  static __device__ __forceinline__ void unit(float (&acc)[NB][4], const FragArgs &a, uint32_t tile, uint32_t xbase,
                                              uint32_t tables, int uq, int g, int t, int lane) {
    const uint32_t R = row_stride(a), xrow = xbase + (uint32_t)g * R + (uint32_t)uq * 512u + (uint32_t)t * 16u;
    const uint32_t sums = xbase + 8u * R + (uint32_t)(uq * kSumBytes) + (uint32_t)lane * 16u;
    const uint4 h0 = lds128(tile + 3072u + (uint32_t)g * 16u), h1 = lds128(tile + 3072u + (uint32_t)(g + 8) * 16u);
    const uint32_t hw0[4] = {h0.x, h0.y, h0.z, h0.w}, hw1[4] = {h1.x, h1.y, h1.z, h1.w};
    // The first k-steps of the pairs are added up in su, the second in sv: shorter chains. Two column groups
    // have too few registers for both (sixteen rows: 2 % slower than with one sum).
    constexpr bool kOneSum = NB == 2;
    float su[NB][4], sv[NB][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int i = 0; i < 4; ++i) su[nb][i] = sv[nb][i] = 0.f;
    uint32_t qw[12];  // the words of four pairs
#pragma unroll
    for (int pi = 0; pi < 8; ++pi) {
      if ((pi & 3) == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const uint4 q = lds128(tile + (uint32_t)(3 * (pi >> 2) + i) * 512u + (uint32_t)lane * 16u);
          qw[4 * i] = q.x, qw[4 * i + 1] = q.y, qw[4 * i + 2] = q.z, qw[4 * i + 3] = q.w;
        }
      }
      const uint32_t w0 = qw[3 * (pi & 3)], w1 = qw[3 * (pi & 3) + 1], w2 = qw[3 * (pi & 3) + 2];
      const uint32_t a0 = times16((w0 & 0x000f000fu) | ((w2 << 4) & 0x00300030u)), a2 = times16((w1 & 0x000f000fu) | ((w2 << 2) & 0x00300030u));
      const uint32_t a1 = (w0 >> 6) & 0x03f003f0u, a3 = (w1 >> 6) & 0x03f003f0u;
      const uint32_t e0 = w0 & 0x03f003f0u, e1 = w1 & 0x03f003f0u;
      const uint32_t e2 = w2 & 0x03f003f0u, e3 = (w2 >> 6) & 0x03f003f0u;
      // scales of groups 2 pi and 2 pi + 1
      const float s00 = scale_of(hw0[pi >> 1], 2 * (pi & 1)), s01 = scale_of(hw0[pi >> 1], 2 * (pi & 1) + 1);
      const float s10 = scale_of(hw1[pi >> 1], 2 * (pi & 1)), s11 = scale_of(hw1[pi >> 1], 2 * (pi & 1) + 1);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const uint4 b = lds128(xrow + nb * a.xregion + (uint32_t)pi * 64u);
        float c0[4], c1[4];
        mma16816_first(c0, a0, a1, a2, a3, b.x, b.y);
        mma16816_first(c1, e0, e1, e2, e3, b.z, b.w);
        float(&sw)[4] = kOneSum ? su[nb] : sv[nb];
        su[nb][0] = fmaf(s00, c0[0], su[nb][0]), su[nb][1] = fmaf(s00, c0[1], su[nb][1]);
        su[nb][2] = fmaf(s10, c0[2], su[nb][2]), su[nb][3] = fmaf(s10, c0[3], su[nb][3]);
        sw[0] = fmaf(s01, c1[0], sw[0]), sw[1] = fmaf(s01, c1[1], sw[1]);
        sw[2] = fmaf(s11, c1[2], sw[2]), sw[3] = fmaf(s11, c1[3], sw[3]);
      }
    }
    // sum_g scale_g * (sum of x over group g): the MMA over groups; this lane's slots are groups
    // 4t .. 4t + 3, the word t of each row's scales
    const uint32_t w0 = (t == 0 ? h0.x : t == 1 ? h0.y : t == 2 ? h0.z : h0.w);
    const uint32_t w1 = (t == 0 ? h1.x : t == 1 ? h1.y : t == 2 ? h1.z : h1.w);
    const uint32_t a0 = scale_pair(w0, 0x4140u), a1 = scale_pair(w1, 0x4140u);
    const uint32_t a2 = scale_pair(w0, 0x4342u), a3 = scale_pair(w1, 0x4342u);
    const uint32_t dd = lds32(tile + 3328u + (uint32_t)g * 4u);
    const float d0 = half_bits_to_float(dd & 0xffffu), d1 = half_bits_to_float(dd >> 16);
    const float dl0 = d0 * 0.0625f, dl1 = d1 * 0.0625f, dm0 = d0 * (-32.f / 16777216.f), dm1 = d1 * (-32.f / 16777216.f);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const uint4 bs = lds128(sums + nb * a.xregion);
      float cm[4];
      mma16816_first(cm, a0, a1, a2, a3, bs.x, bs.y);
      mma16816(cm, a0, a1, a2, a3, bs.z, bs.w);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float sum = kOneSum ? su[nb][i] : su[nb][i] + sv[nb][i];
        acc[nb][i] = fmaf(i < 2 ? dl0 : dl1, sum, fmaf(i < 2 ? dm0 : dm1, cm[i], acc[nb][i]));
      }
    }
  }
};

}  // namespace ishi
