// GGUF Q2_K for the warp-level kernel (mma.sync fragments).
//
// Block layout (84 bytes per 256 weights; reference: Sources/IshizukiKit/Core/GGMLDequant.swift:125-150):
//   sixteen bytes (scale | min << 4) @0, 64 code bytes @16, d f16 @80, dmin f16 @82. Weight
//   k = 128 n + 32 j + l (half n, shift j < 4, l < 32) has its two bits at bit 2j of code byte
//   32 n + l and belongs to sub-block is = 8 n + 2 j + l / 16;  w = d * scale_is * q - dmin * min_is.
//
// The product is factored as
//   y += d * sum_is scale_is * sum_{k in is} q_k x_k  -  dmin * sum_is min_is * sum_{k in is} x_k.
// A sub-block is exactly one k-step of the MMA, so every k-step's accumulator takes its (integer)
// scale afterwards; the second sum is one more MMA whose k index runs over the sub-blocks, against
// the sub-block sums of x (fp16 high and low parts).
//
// A 2-bit code masked in place at bits 2j, 2j + 1 of each half of a register is the bit pattern of
// the fp16 number q * 4^j * 2^-24 (subnormal, hence linear in q); the activations of shift j are
// divided by 4^j (exact unless |x| is tiny). A lane t owns, per weight row, the 32-bit word
// of code bytes 32 n + 16 h + 4t + {0, 2, 1, 3} (h = l / 16): masked at shift j it gives the weights
// l % 16 = 4t, 4t + 1 of sub-block 8 n + 2 j + h, shifted right by 8 and masked the weights 4t + 2,
// 4t + 3: the MMA's k columns (2t, 2t + 1) and (2t + 8, 2t + 9). The activations are copied as they lie in x and divided and put
// in the order of one 16-byte load per two sub-blocks in place (frag_rows_by_16()). Over weights from HBM, best plans,
// 17408 x 5120 at sixteen / four / one row 21.9 / 14.3 / 13.8 -> 20.1 / 13.95 / 13.4 us, 4096 x 4096 at sixteen 8.3 -> 7.8.
//
// Tile (16 rows x 256 k, 1344 bytes = 16 * 84): code words [2][lane][row g: h = 0, 1; row g + 8:
// h = 0, 1] @0, per row the sixteen scale bytes @1024 (a lane's A registers of the MMA over sub-blocks, 4t .. 4t + 3, are
// one word), d of rows (g, g + 8) side by side @1280, dmin the same @1312.
#pragma once
#include "ishi_fragstream.cuh"

namespace ishi {

struct FragQ2K : FragCopying {
  static constexpr int kTileBytes = 16 * 84;
  static constexpr int kSumBytes = 512;         // per unit: [lane][hi hi | lo lo] sub-block sums
  static constexpr int kXBytes = 8 * 512 + kSumBytes, kXFixed = 8 * 64;  // a staged region: per unit eight rows and the sums; the rows' skews
  static constexpr double kUnit = 16777216.0;  // tile results come in units of 2^24: masked codes are q * 2^-24
  static constexpr bool kRows = true, kRowSums = true;  // the activations as they lie in x, then put in order and added up
  // five to eight rows by loads and stores, which arrange and add up on the way (4096 x 4096 at eight rows, copied: 5.48 us against 5.39)
  static constexpr int kCopyRows = 4;
  static constexpr int kExtraBytes = 0;
  static constexpr bool kRowMode = false;       // one activation row runs through the MMA path as well
  static constexpr int kFewWarps = 16;  // most warps of the smaller block size at up to eight rows
  static constexpr int kManyWarps = 20;  // most warps at nine to sixteen rows

  static __device__ __forceinline__ const uint8_t *block(const FragSrc &s, long long row, int u) {
    long long local;
    const int seg = frag_segment(s, row, &local);
    return s.w[seg] + local * s.w_row_bytes + (long long)u * 84;
  }

  static __device__ __forceinline__ uint8_t tile_byte(const FragSrc &s, long long p, int u, int b) {
    if (b < 1024) {
      const int n = b >> 9, lane = (b & 511) >> 4, i = b & 15;
      const int g = lane >> 2, t = lane & 3, wi = i >> 2, bi = i & 3;
      const long long row = p * kFragRows + g + 8 * (wi >> 1);
      if (row >= s.N) return 0;
      const int k = bi == 1 ? 2 : bi == 2 ? 1 : bi;
      return block(s, row, u)[16 + 32 * n + 16 * (wi & 1) + 4 * t + k];
    }
    if (b < 1280) {
      const int idx = b - 1024, pos = idx & 15;
      const long long row = p * kFragRows + (idx >> 4);
      if (row >= s.N) return 0;
      return block(s, row, u)[pos];
    }
    const int idx = (b - 1280) & 31;
    const long long row = p * kFragRows + (idx >> 2) + 8 * ((idx >> 1) & 1);
    if (row >= s.N) return 0;
    return block(s, row, u)[(b < 1312 ? 80 : 82) + (idx & 1)];
  }

  static __device__ __forceinline__ uint16_t tile_halfword(const FragSrc &s, long long p, int u, int hw) {
    return (uint16_t)(tile_byte(s, p, u, 2 * hw) | ((uint32_t)tile_byte(s, p, u, 2 * hw + 1) << 8));
  }

  static __device__ __forceinline__ uint32_t row_stride(const FragArgs &a) { return (uint32_t)a.umax * 512u + 64u; }
  // 4^-j in both halves for lane l's values k = 8l .. 8l + 7 of a unit
  static __device__ __forceinline__ uint32_t factor() { return (uint32_t)(15 - 2 * ((threadIdx.x >> 2) & 3)) * 0x04000400u; }

  static __device__ __forceinline__ void row_sums(const FragArgs &a, uint32_t xfrag, int rows, int uc) {
    frag_rows_by_16<true>(xfrag, row_stride(a), xfrag + 8u * row_stride(a), kSumBytes, rows, uc, factor());
  }
  // Rows on their way from x. A warp task is (unit, row): lane l loads k = 8l .. 8l + 7.
  template <class Then>
  static __device__ __forceinline__ void stage_x(const FragArgs &a, const FragRows &m, uint32_t xfrag, int ub0, int uc, Then then) {
    const uint32_t R = row_stride(a), f = factor();
    frag_stage_rows(a, m, ub0, uc, then, [&](int u, int r, uint4 v) {
      frag_put_by_16<true>(xfrag + (uint32_t)r * R + (uint32_t)u * 512u, xfrag + 8u * R + (uint32_t)(u * kSumBytes), r, v, f);
    });
  }

  // 8388608 + byte `byte` of word w, as a float
  static __device__ __forceinline__ float byte_float(uint32_t w, int byte) {
    return __uint_as_float(prmt(w, 0x4b000000u, 0x7440u | (uint32_t)byte));
  }
  // One tile against the activations of its unit; acc is the warp's C fragment.
  template <int MODE, int NB>
  static __device__ __forceinline__ void unit(float (&acc)[NB][4], const FragArgs &a, uint32_t tile, uint32_t xbase,
                                              uint32_t tables, int uq, int g, int t, int lane) {
    const uint32_t R = row_stride(a), xrow = xbase + (uint32_t)g * R + (uint32_t)uq * 512u + (uint32_t)t * 16u;
    const uint32_t sums = xbase + 8u * R + (uint32_t)(uq * kSumBytes) + (uint32_t)lane * 16u;
    const uint4 h0 = lds128(tile + 1024u + (uint32_t)g * 16u), h1 = lds128(tile + 1024u + (uint32_t)(g + 8) * 16u);
    // the scales (low nibbles)
    const uint32_t sl0[4] = {h0.x & 0x0f0f0f0fu, h0.y & 0x0f0f0f0fu, h0.z & 0x0f0f0f0fu, h0.w & 0x0f0f0f0fu};
    const uint32_t sl1[4] = {h1.x & 0x0f0f0f0fu, h1.y & 0x0f0f0f0fu, h1.z & 0x0f0f0f0fu, h1.w & 0x0f0f0f0fu};
    float su[NB][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) su[nb][0] = su[nb][1] = su[nb][2] = su[nb][3] = 0.f;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const uint4 q = lds128(tile + (uint32_t)n * 512u + (uint32_t)lane * 16u);
      const uint32_t y[4] = {q.x >> 8, q.y >> 8, q.z >> 8, q.w >> 8};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t mask = 0x00030003u << (2 * j);
        uint4 b[NB];  // both sub-blocks' activations
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) b[nb] = lds128(xrow + nb * a.xregion + (uint32_t)(4 * n + j) * 64u);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int is = 8 * n + 2 * j + h;
          const uint32_t w0 = h ? q.y : q.x, w1 = h ? q.w : q.z, y0 = h ? y[1] : y[0], y1 = h ? y[3] : y[2];
          const float f0 = byte_float(sl0[is >> 2], is & 3) - 8388608.f, f1 = byte_float(sl1[is >> 2], is & 3) - 8388608.f;
#pragma unroll
          for (int nb = 0; nb < NB; ++nb) {
            float part[4];
            mma16816_first(part, w0 & mask, w1 & mask, y0 & mask, y1 & mask, h ? b[nb].z : b[nb].x, h ? b[nb].w : b[nb].y);
            su[nb][0] = fmaf(f0, part[0], su[nb][0]), su[nb][1] = fmaf(f0, part[1], su[nb][1]);
            su[nb][2] = fmaf(f1, part[2], su[nb][2]), su[nb][3] = fmaf(f1, part[3], su[nb][3]);
          }
        }
      }
    }
    // sum_is min_is * (sum of x over sub-block is): the MMA over sub-blocks; this lane's slots are
    // sub-blocks 4t .. 4t + 3, the word t of each row's sixteen bytes, high nibbles
    const uint32_t m0 = ((t == 0 ? h0.x : t == 1 ? h0.y : t == 2 ? h0.z : h0.w) >> 4) & 0x0f0f0f0fu;
    const uint32_t m1 = ((t == 0 ? h1.x : t == 1 ? h1.y : t == 2 ? h1.z : h1.w) >> 4) & 0x0f0f0f0fu;
    // (a byte as the low bits of an fp16 is the subnormal number m * 2^-24, as the codes are)
    const uint32_t a0 = prmt(m0, 0u, 0x4140u), a1 = prmt(m1, 0u, 0x4140u);
    const uint32_t a2 = prmt(m0, 0u, 0x4342u), a3 = prmt(m1, 0u, 0x4342u);
    const uint32_t dd = lds32(tile + 1280u + (uint32_t)g * 4u), mm = lds32(tile + 1312u + (uint32_t)g * 4u);
    const float d0 = half_bits_to_float(dd & 0xffffu), d1 = half_bits_to_float(dd >> 16);
    const float n0 = -half_bits_to_float(mm & 0xffffu), n1 = -half_bits_to_float(mm >> 16);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const uint4 bs = lds128(sums + nb * a.xregion);
      float cm[4];
      mma16816_first(cm, a0, a1, a2, a3, bs.x, bs.y);
      mma16816(cm, a0, a1, a2, a3, bs.z, bs.w);
      acc[nb][0] = fmaf(d0, su[nb][0], fmaf(n0, cm[0], acc[nb][0]));
      acc[nb][1] = fmaf(d0, su[nb][1], fmaf(n0, cm[1], acc[nb][1]));
      acc[nb][2] = fmaf(d1, su[nb][2], fmaf(n1, cm[2], acc[nb][2]));
      acc[nb][3] = fmaf(d1, su[nb][3], fmaf(n1, cm[3], acc[nb][3]));
    }
  }
};

}  // namespace ishi
