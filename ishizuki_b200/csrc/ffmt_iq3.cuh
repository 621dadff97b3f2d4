// GGUF IQ3_XXS and IQ3_S for the warp-level kernel (mma.sync fragments).
//
// Block layouts (reference: Sources/IshizukiKit/Core/GGMLDequant.swift:313-374):
//   IQ3_XXS (98 bytes per 256 weights): d f16 @0, 64 index bytes @2 (each: four magnitudes out of a
//     256-entry grid), eight words @66: four 7-bit sign indices (eighth sign = parity) and the
//     four-bit scale s of 32 weights; w = d * (2 s + 1) / 4 * magnitude * sign.
//   IQ3_S (110 bytes): d @0, 64 index bytes @2, qh @66 (a ninth index bit each; 512-entry grid), 32
//     sign bytes @74 (all eight signs), scale nibbles @106 (per 32 weights); w = d * (2 s + 1) *
//     magnitude * sign.
//
// The decoder is the one of IQ2_XS with two lookups per eight weights: the grid lives in shared
// memory as fp16 (an entry = four magnitudes = 8 bytes = two A registers), in sixteen copies, copy
// c of entry i at i * 128 + c * 8: an 8-byte load is served sixteen lanes at a time, lane l reads
// copy l % 16. Scales (magnitude * (2 s + 1) <= 1922, an exact fp16 integer) and signs as there.
// Fragment mapping and activations as for IQ2_XS: a lane owns the sub-blocks (sixteen weights = four
// indices) 4 j + t, j = 0..3, of rows g and g + 8.
//
// Tile (16 rows x 256 k, 2080 bytes; blocks: IQ3_XXS 1568, IQ3_S 1760): [4][lane][16 bytes] = for
// sub-block 4 j + t the words of its two entries (eight weights each) of row g, then of row g + 8;
// then d of rows (g, g + 8) side by side. A word has the entry's first index in its low half and the
// second in its high half, from bit 7 up, where a mask makes it a byte offset into the grid. The bits
// below hold the signs, register r's pair at p and p + 16 (p = 3 ... 6 in a first word, 2, 4, 5, 6 in a
// second), and in both halves the scale s: its low three bits at 0 ... 2 of the first word, the fourth
// at bit 3 of the second. The loop is bound by instruction issue: 17408 x 5120 at eight rows, one
// weight repeated out of L2, took 19.2 us and 640 warp instructions a tile with index bytes, ninth bits,
// signs and scales in words of their own (1824 bytes), 16.5 us and 519 with this layout (17.7 us with
// weights of their own in HBM).
#pragma once
#include "ffmt_iq2xs.cuh"

namespace ishi {

// TYPE: the GGML type number, 18 IQ3_XXS, 21 IQ3_S
template <int TYPE>
struct FragIQ3 : FragCopying {
  static_assert(TYPE == 18 || TYPE == 21, "IQ3_XXS or IQ3_S");
  static constexpr bool kNine = TYPE == 21;  // nine index bits, explicit signs
  static constexpr int kBlock = kNine ? 110 : 98;
  static constexpr int kEntries = kNine ? 512 : 256;
  static constexpr int kD = 2048;  // offset of d
  static constexpr int kTileBytes = kD + 32;
  static constexpr uint32_t kMask = (uint32_t)(kEntries - 1) << 7;
  static constexpr int kXBytes = FragIQ2<17>::kXBytes, kXFixed = FragIQ2<17>::kXFixed;
  static constexpr double kUnit = kNine ? 1.0 : 0.25;  // unit of the tile results
  static constexpr bool kRows = true, kRowSums = false;  // the activations as they lie in x
  static constexpr int kExtraBytes = kEntries * 128;  // the grid as fp16, sixteen copies interleaved
  static constexpr bool kRowMode = false;  // one activation row runs through the MMA path as well
  static constexpr int kFewWarps = 20;  // most warps of the smaller block size at up to eight rows
  static constexpr int kManyWarps = 16;  // most warps at nine to sixteen rows

  static __device__ __forceinline__ const uint8_t *block(const FragSrc &s, long long row, int u) {
    long long local;
    const int seg = frag_segment(s, row, &local);
    return s.w[seg] + local * s.w_row_bytes + (long long)u * kBlock;
  }

  // position of register r's sign pair in the first or second word of a sub-block
  static __device__ __forceinline__ constexpr int pair_at(int second, int r) { return second && r == 0 ? 2 : 3 + r; }

  static __device__ __forceinline__ uint16_t tile_halfword(const FragSrc &s, long long p, int u, int hw) {
    const int h = hw & 1;  // half of a word
    if (hw < kD / 2) {
      const int j = hw >> 8, lane = (hw & 255) >> 3, i = (hw & 7) >> 1, second = i & 1;
      const long long row = p * kFragRows + (lane >> 2) + 8 * (i >> 1);
      if (row >= s.N) return 0;
      const uint8_t *blk = block(s, row, u);
      const int sb = 4 * j + (lane & 3), E = 2 * sb + second, b = 2 * E + h;  // sub-block, entry, index byte
      uint32_t index = blk[2 + b], signs, scale;
      if (kNine) {
        index |= (((uint32_t)blk[66 + (b >> 3)] >> (b & 7)) & 1u) << 8;
        signs = blk[74 + E];
        scale = ((uint32_t)blk[106 + (sb >> 2)] >> (4 * ((sb >> 1) & 1))) & 15u;
      } else {
        const uint8_t *aux = blk + 66 + 4 * (E >> 2);
        const uint32_t word = (uint32_t)aux[0] | ((uint32_t)aux[1] << 8) | ((uint32_t)aux[2] << 16) | ((uint32_t)aux[3] << 24);
        const uint32_t s7 = (word >> (7 * (E & 3))) & 127u;
        signs = s7 | ((uint32_t)(__popc(s7) & 1) << 7);
        scale = word >> 28;
      }
      uint32_t out = (index << 7) | (second ? scale & 8u : scale & 7u);
      for (int r = 0; r < 4; ++r) out |= ((signs >> (2 * r + h)) & 1u) << pair_at(second, r);
      return (uint16_t)out;
    }
    const long long row = p * kFragRows + ((hw - kD / 2) >> 1) + 8 * h;
    if (row >= s.N) return 0;
    const uint8_t *blk = block(s, row, u);
    return (uint16_t)((uint32_t)blk[0] | ((uint32_t)blk[1] << 8));
  }

  static __device__ __forceinline__ uint32_t row_stride(const FragArgs &a) { return (uint32_t)a.umax * 512u + 16u; }

  // word i of the grid: entry i / 32's four magnitudes as fp16, in sixteen copies side by side
  static __device__ __forceinline__ uint32_t table_word(int i) {
    const uint32_t bytes = (kNine ? d_iq3s_grid[i >> 5] : d_iq3xxs_grid[i >> 5]) >> (16 * (i & 1));
    const __half2 h = __halves2half2(__int2half_rn((int)(bytes & 0xffu)), __int2half_rn((int)((bytes >> 8) & 0xffu)));
    return *reinterpret_cast<const uint32_t *>(&h);
  }

  // a sub-block's sixteen weights (two words) as eight A registers; `copy`: byte offset of this lane's copy
  static __device__ __forceinline__ void sub_block(uint32_t (&r)[8], uint32_t w0, uint32_t w1, uint32_t grid, uint32_t copy) {
    // 2 s + 1: the bits of s in the low mantissa bits of 1024, in both halves
    const uint32_t bits = ((w0 & 0x00070007u) | 0x64006400u) | (w1 & 0x00080008u);
    const __half2 scale = __hfma2(*reinterpret_cast<const __half2 *>(&bits), __float2half2_rn(2.f), __float2half2_rn(-2047.f));
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const uint32_t w = e ? w1 : w0;
      const uint2 m = lds64(grid + ((w & kMask) | copy)), n = lds64(grid + (((w >> 16) & kMask) | copy));
      const uint32_t mag[4] = {m.x, m.y, n.x, n.y};
#pragma unroll
      for (int k = 0; k < 4; ++k) r[4 * e + k] = FragIQ2<17>::signed_scaled(mag[k], scale, w, pair_at(e, k));
    }
  }

  // One tile against the activations of its unit; acc is the warp's C fragment.
  template <int MODE, int NB>
  static __device__ __forceinline__ void unit(float (&acc)[NB][4], const FragArgs &a, uint32_t tile, uint32_t xbase,
                                              uint32_t tables, int uq, int g, int t, int lane) {
    const uint32_t R = row_stride(a);
    const uint32_t copy = (uint32_t)(lane & 15) * 8u;
    const uint32_t xrow = xbase + (uint32_t)g * R + (uint32_t)uq * 512u + (uint32_t)t * 32u;
    float c[NB][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 w = lds128(tile + (uint32_t)j * 512u + (uint32_t)lane * 16u);
      uint32_t r0[8], r1[8];  // sub-block 4 j + t of row g, of row g + 8
      sub_block(r0, w.x, w.y, tables, copy);
      sub_block(r1, w.z, w.w, tables, copy);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const uint32_t xj = xrow + nb * a.xregion + (uint32_t)j * 128u;
        const uint4 x0 = lds128(xj), x1 = lds128(xj + 16u);
        if (j == 0)
          mma16816_first(c[nb], r0[0], r1[0], r0[1], r1[1], x0.x, x0.y);
        else
          mma16816(c[nb], r0[0], r1[0], r0[1], r1[1], x0.x, x0.y);
        mma16816(c[nb], r0[2], r1[2], r0[3], r1[3], x0.z, x0.w);
        mma16816(c[nb], r0[4], r1[4], r0[5], r1[5], x1.x, x1.y);
        mma16816(c[nb], r0[6], r1[6], r0[7], r1[7], x1.z, x1.w);
      }
    }
    const uint32_t dd = lds32(tile + (uint32_t)kD + (uint32_t)g * 4u);
    const float d0 = half_bits_to_float(dd & 0xffffu), d1 = half_bits_to_float(dd >> 16);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      acc[nb][0] = fmaf(d0, c[nb][0], acc[nb][0]);
      acc[nb][1] = fmaf(d0, c[nb][1], acc[nb][1]);
      acc[nb][2] = fmaf(d1, c[nb][2], acc[nb][2]);
      acc[nb][3] = fmaf(d1, c[nb][3], acc[nb][3]);
    }
  }
};

}  // namespace ishi
