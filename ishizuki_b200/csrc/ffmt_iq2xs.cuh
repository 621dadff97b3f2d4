// GGUF IQ2_XS for the warp-level kernel (mma.sync fragments).
//
// Block layout (74 bytes per 256 weights; reference: Sources/IshizukiKit/Core/GGMLDequant.swift
// :264-285 and the kernel body at Sources/IshizukiKit/Core/GGMLKernels.swift:664-676):
//   d f16 @0, thirty-two u16 @2 (bits 0-8: index into the 512-entry grid of eight magnitudes out of
//   {8, 25, 43}; bits 9-15: index into the 128 sign patterns, whose eighth sign is the parity of
//   the seven), eight scale bytes @66 (low nibble: first sixteen weights of a 32-group, high
//   nibble: the second sixteen);  w = d * (2 s + 1) / 8 * magnitude * sign.
//
// Decode: the grid lives in shared memory as fp16 (512 entries x 16 bytes = one 16-byte load per
// eight weights = four A registers), in eight copies, copy c of entry i at i * 128 + c * 16: a
// 16-byte load is served eight lanes at a time, lane l reads copy l % 8, so the eight lanes of a
// pass always hit eight different bank groups whatever their indices are (one copy alone measured
// 2.2 million bank conflicts per launch and warps stalled on shared memory 3.7 cycles per issue).
// The loop is bound by instruction issue, so the tile keeps indices and signs where an instruction
// finds them (below): an index masked in place is its byte offset into the grid; a register takes
// its scale by a half2 multiply with 2 s + 1 (magnitude * (2 s + 1) <= 1333 is an exact fp16
// integer) and its two signs by one shift, which brings its sign pair to bits 15 and 31, and a
// mask-and-xor. With the scale inside the fragments a whole tile accumulates in one MMA chain; d / 8
// remains for fp32. A 17408 x 5120 projection
// of eight rows, one weight repeated out of L2, took 18.7 us and 587 warp instructions a tile with index and
// seven sign bits packed as the block has them and the parity recomputed, 14.9 us and 473 with this layout
// (16.0 us with weights of their own in HBM).
//
// Fragment mapping (m16n8k16; lane g = lane / 4, t = lane % 4 holds weight rows g and g + 8): a
// lane owns the sub-blocks (sixteen weights = two u16 = one scale) 4 j + t, j = 0..3, of both rows.
// The eight registers of a sub-block feed four k-steps m = 0..3: slots (2t, 2t + 1) are weights
// 4m, 4m + 1 and slots (2t + 8, 2t + 9) weights 4m + 2, 4m + 3 of the sub-block, so that the
// activations are used as they lie in memory: 32 contiguous bytes of x per lane and sub-block.
//
// Tile (16 rows x 256 k, 1312 bytes for 1184 of blocks): [2][lane][16 bytes] = for j = 2p, 2p + 1: a
// word of sub-block 4j + t of row g, then of row g + 8. A word's low half is the first entry (eight
// weights), its high half the second: the index from bit 7 up, and below it bits of sign pairs. Pair
// k = 4 e + r (register r of entry e) is bits p and p + 16 of the word, the signs of weights 2r and
// 2r + 1; pairs 0 ... 6 have p = k, which leaves the last pair for a word of its own: [lane][8 bytes]
// = the lane's four scale nibbles of row g (16 bits, nibble j), then of row g + 8, and the eight last
// pairs, p = 2 j (row g), 2 j + 1 (row g + 8). Then d of rows (g, g + 8) side by side.
//
// Activations of a unit in shared memory: eight rows of 256 fp16 as they lie in x, the rows
// umax * 512 + 16 bytes apart (a quarter warp's 16-byte loads then sweep all banks).
//
// The same decoder serves the two sibling formats, which differ in where a block keeps the same
// three things (a grid index and eight signs per eight weights, a four-bit scale):
//   IQ2_XXS (66 bytes; GGMLDequant.swift:243-262): per 32 weights four index bytes into a 256-entry
//     grid and one word of four 7-bit sign indices and the scale of all 32. Bit 15 of each half is
//     free and holds the last pair: no word of last pairs, 1184 bytes for 1056 of blocks.
//   IQ2_S (82 bytes; GGMLDequant.swift:287-311): index bytes, sign bytes (all eight signs, no
//     parity), two more index bits per eight weights, scales as IQ2_XS; 1024-entry grid. Its grid has
//     four copies (64 KB), two lanes of a pass share one. Its index starts at bit 6, so pairs 6 and 7
//     both go to the word of last pairs, p = 4 j + (row g + 8) * 2 + (k - 6); 1312 bytes = 16 * 82.
#pragma once
#include "ggml_decode.cuh"
#include "ishi_fragstream.cuh"
#include "iq2xs_tables.h"

namespace ishi {

static __device__ const uint16_t g_iq2xs_frag_codes[512] = {ISHI_IQ2XS_CODES_LIST};

// TYPE: the GGML type number, 17 IQ2_XS, 16 IQ2_XXS, 22 IQ2_S
template <int TYPE>
struct FragIQ2 : FragCopying {
  static_assert(TYPE == 17 || TYPE == 16 || TYPE == 22, "IQ2_XS, IQ2_XXS or IQ2_S");
  static constexpr bool kWide = TYPE == 22;                  // IQ2_S: ten index bits, eight explicit signs
  static constexpr int kBlock = TYPE == 17 ? 74 : TYPE == 16 ? 66 : 82;
  static constexpr int kEntries = TYPE == 17 ? 512 : TYPE == 16 ? 256 : 1024;
  static constexpr int kCopies = kWide ? 4 : 8;              // of the grid
  static constexpr int kShift = kWide ? 6 : 7;               // an index times the bytes of an entry's copies
  static constexpr uint32_t kMask = (uint32_t)(kEntries - 1) << kShift;
  static constexpr int kInline = TYPE == 16 ? 8 : kShift;    // sign pairs inside the words
  static constexpr int kScales = 1024;                       // offset of the per-lane scales (and last pairs)
  static constexpr int kLane = kInline == 8 ? 4 : 8;
  static constexpr int kD = kScales + 32 * kLane;            // offset of d
  static constexpr int kTileBytes = kD + 32;
  static constexpr int kXBytes = 8 * 512, kXFixed = 8 * 16;    // a staged region: per unit eight rows of 512 bytes; the rows' skews
  static constexpr double kUnit = 0.125;         // tile results come in units of 1/8
  static constexpr bool kRows = true, kRowSums = false;  // the activations as they lie in x
  static constexpr int kExtraBytes = kEntries * kCopies * 16;  // the grid as fp16, its copies interleaved
  static constexpr bool kRowMode = false;        // one activation row runs through the MMA path as well
  static constexpr int kFewWarps = 20;  // most warps of the smaller block size at up to eight rows
  static constexpr int kManyWarps = kWide ? 20 : 16;  // most warps at nine to sixteen rows

  static __device__ __forceinline__ const uint8_t *block(const FragSrc &s, long long row, int u) {
    long long local;
    const int seg = frag_segment(s, row, &local);
    return s.w[seg] + local * s.w_row_bytes + (long long)u * kBlock;
  }

  // the four bytes of IQ2_XXS with the sign indices and the scale of entry E's 32 weights
  static __device__ __forceinline__ uint32_t aux(const uint8_t *blk, int E) {
    const uint8_t *q = blk + 6 + 8 * (E >> 2);
    return (uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16) | ((uint32_t)q[3] << 24);
  }
  // grid index of entry E (eight weights) of a block
  static __device__ __forceinline__ uint32_t index_of(const uint8_t *blk, int E) {
    if (TYPE == 17) return (uint32_t)blk[2 + 2 * E] | (((uint32_t)blk[3 + 2 * E] & 1u) << 8);
    if (TYPE == 16) return blk[2 + 8 * (E >> 2) + (E & 3)];
    return (uint32_t)blk[2 + E] | ((((uint32_t)blk[66 + (E >> 2)] >> (2 * (E & 3))) & 3u) << 8);
  }
  // its eight signs
  static __device__ __forceinline__ uint32_t signs_of(const uint8_t *blk, int E) {
    if (kWide) return blk[34 + E];
    const uint32_t s7 = TYPE == 17 ? (uint32_t)blk[3 + 2 * E] >> 1 : (aux(blk, E) >> (7 * (E & 3))) & 127u;
    return s7 | ((uint32_t)(__popc(s7) & 1) << 7);
  }
  // the four-bit scale of sub-block sb (sixteen weights)
  static __device__ __forceinline__ uint32_t scale4(const uint8_t *blk, int sb) {
    if (TYPE == 16) return aux(blk, 2 * sb) >> 28;
    return ((uint32_t)blk[(TYPE == 17 ? 66 : 74) + (sb >> 1)] >> (4 * (sb & 1))) & 15u;
  }
  // position of sign pair k in its word: word j of row g (r = 0) or g + 8 (r = 1), or the last pairs' word
  static __device__ __forceinline__ constexpr int pair_at(int k, int j, int r) {
    return k < kShift ? k : TYPE == 16 ? 15 : (2 * j + r) * (8 - kInline) + k - kInline;
  }

  static __device__ __forceinline__ uint16_t tile_halfword(const FragSrc &s, long long p, int u, int hw) {
    const int h = hw & 1;  // half of a word
    uint32_t out = 0;
    if (hw < kScales / 2) {
      const int j = 2 * (hw >> 8) + ((hw >> 2) & 1), lane = (hw & 255) >> 3, r = (hw >> 1) & 1;
      const long long row = p * kFragRows + (lane >> 2) + 8 * r;
      if (row >= s.N) return 0;
      const uint8_t *blk = block(s, row, u);
      const int sb = 4 * j + (lane & 3);
      out = index_of(blk, 2 * sb + h) << kShift;
      for (int k = 0; k < kInline; ++k)
        out |= ((signs_of(blk, 2 * sb + (k >> 2)) >> (2 * (k & 3) + h)) & 1u) << pair_at(k, j, r);
      return (uint16_t)out;
    }
    if (hw < kD / 2) {
      const int lane = (hw - kScales / 2) / (kLane / 2), i = (hw - kScales / 2) % (kLane / 2);
      for (int j = 0; j < 4; ++j)
        for (int r = 0; r < 2; ++r) {
          const long long row = p * kFragRows + (lane >> 2) + 8 * r;
          if (row >= s.N || (i < 2 && r != h)) continue;
          const uint8_t *blk = block(s, row, u);
          const int sb = 4 * j + (lane & 3);
          if (i < 2) out |= scale4(blk, sb) << (4 * j);
          else
            for (int k = kInline; k < 8; ++k)
              out |= ((signs_of(blk, 2 * sb + 1) >> (2 * (k & 3) + h)) & 1u) << pair_at(k, j, r);
        }
      return (uint16_t)out;
    }
    const long long row = p * kFragRows + ((hw - kD / 2) >> 1) + 8 * h;
    if (row >= s.N) return 0;
    const uint8_t *blk = block(s, row, u);
    return (uint16_t)((uint32_t)blk[0] | ((uint32_t)blk[1] << 8));
  }

  static __device__ __forceinline__ uint32_t row_stride(const FragArgs &a) { return (uint32_t)a.umax * 512u + 16u; }

  // word i of the grid: two of an entry's eight magnitudes as fp16 (an entry is four words, its
  // copies lie side by side)
  static __device__ __forceinline__ uint32_t table_word(int i) {
    const int entry = i / (4 * kCopies), r = i & 3;
    uint32_t m0, m1;
    if (TYPE == 17) {  // the codes are two bits each: 0, 1, 2 -> 8, 25, 43
      const uint32_t c0 = ((uint32_t)g_iq2xs_frag_codes[entry] >> (4 * r)) & 3u, c1 = ((uint32_t)g_iq2xs_frag_codes[entry] >> (4 * r + 2)) & 3u;
      m0 = c0 == 0 ? 8u : c0 == 1 ? 25u : 43u, m1 = c1 == 0 ? 8u : c1 == 1 ? 25u : 43u;
    } else {
      const uint32_t bytes = (uint32_t)((TYPE == 16 ? d_iq2xxs_grid[entry] : d_iq2s_grid[entry]) >> (16 * r));
      m0 = bytes & 0xffu, m1 = (bytes >> 8) & 0xffu;
    }
    const __half2 h = __halves2half2(__int2half_rn((int)m0), __int2half_rn((int)m1));
    return *reinterpret_cast<const uint32_t *>(&h);
  }

  // 2 s + 1 of scale nibble j, in both halves, from the nibbles of a row in both halves: the nibble
  // in the low mantissa bits of 1024 is 1024 + s, four bits up 1024 + 16 s
  static __device__ __forceinline__ __half2 scale_of(uint32_t twice, int j) {
    const uint32_t v = j < 2 ? twice : twice >> 8;
    const uint32_t bits = (v & (j & 1 ? 0x00f000f0u : 0x000f000fu)) | 0x64006400u;
    const __half2 h = *reinterpret_cast<const __half2 *>(&bits);
    return j & 1 ? __hfma2(h, __float2half2_rn(0.125f), __float2half2_rn(-127.f))
                 : __hfma2(h, __float2half2_rn(2.f), __float2half2_rn(-2047.f));
  }

  // two magnitudes of the grid as an A register: times the scale, and its sign pair (bits p and
  // p + 16 of `word`) xor-ed in
  static __device__ __forceinline__ uint32_t signed_scaled(uint32_t mag, __half2 scale, uint32_t word, int p) {
    const __half2 v = __hmul2(*reinterpret_cast<const __half2 *>(&mag), scale);
    return *reinterpret_cast<const uint32_t *>(&v) ^ ((word << (15 - p)) & 0x80008000u);
  }
  // a word's sixteen weights as eight A registers; `copy`: byte offset of this lane's copy
  static __device__ __forceinline__ void sub_block(uint32_t (&r)[8], uint32_t word, uint32_t last, int j, int row, uint32_t grid,
                                                   uint32_t copy, __half2 scale) {
    const uint4 m = lds128(grid + ((word & kMask) | copy)), n = lds128(grid + (((word >> 16) & kMask) | copy));
    const uint32_t mag[8] = {m.x, m.y, m.z, m.w, n.x, n.y, n.z, n.w};
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = signed_scaled(mag[k], scale, k < kInline ? word : last, pair_at(k, j, row));
  }

  // One tile against the activations of its unit; acc is the warp's C fragment.
  template <int MODE, int NB>
  static __device__ __forceinline__ void unit(float (&acc)[NB][4], const FragArgs &a, uint32_t tile, uint32_t xbase,
                                              uint32_t tables, int uq, int g, int t, int lane) {
    const uint32_t R = row_stride(a);
    const uint32_t copy = (uint32_t)(lane & (kCopies - 1)) * 16u;
    const uint32_t xrow = xbase + (uint32_t)g * R + (uint32_t)uq * 512u + (uint32_t)t * 32u;
    uint2 sn = make_uint2(0u, 0u);  // scale nibbles; the last sign pairs
    if (kLane == 8) sn = lds64(tile + kScales + (uint32_t)lane * 8u);
    else sn.x = lds32(tile + kScales + (uint32_t)lane * 4u);
    const uint32_t sn0 = prmt(sn.x, 0u, 0x1010u), sn1 = prmt(sn.x, 0u, 0x3232u);  // row g's, row g + 8's in both halves
    float c[NB][4];
#pragma unroll
    for (int pc = 0; pc < 2; ++pc) {
      const uint4 w = lds128(tile + (uint32_t)pc * 512u + (uint32_t)lane * 16u);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = 2 * pc + e;
        uint32_t r0[8], r1[8];  // sub-block 4 j + t of row g, of row g + 8
        sub_block(r0, e ? w.z : w.x, sn.y, j, 0, tables, copy, scale_of(sn0, j));
        sub_block(r1, e ? w.w : w.y, sn.y, j, 1, tables, copy, scale_of(sn1, j));
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

using FragIQ2XS = FragIQ2<17>;

}  // namespace ishi
