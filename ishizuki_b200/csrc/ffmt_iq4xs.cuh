// GGUF IQ4_XS for the warp-level kernel (mma.sync fragments).
//
// Block layout (136 bytes per 256 weights; reference: Sources/IshizukiKit/Core/GGMLDequant.swift:222-241):
//   d f16 @0, scales_h u16 @2, scales_l[4] @4, qs[128] @8. Sub-block ib (32 weights) has the six-bit
//   scale ls = (scales_l[ib / 2] >> 4 (ib % 2)) & 15 | ((scales_h >> 2 ib) & 3) << 4 and sixteen
//   bytes qs[16 ib + j]: weight j takes the low nibble, weight j + 16 the high nibble, as indices
//   into the sixteen non-uniform values kvalues_iq4nl; w = d * (ls - 32) * value.
//
// The tile holds the nibbles in the weights' order: a byte is two neighbours, exactly one A register (an fp16
// pair), looked up whole in a 256-entry table of value pairs in shared memory (one copy per lane, so that the 32
// lookups of a warp never meet in a bank). Lane t owns weights 8t ... 8t + 7 of every sub-block of its two rows, a 32-bit word: in
// k-step s (0, 1) its bytes 2s and 2s + 1 are the MMA's k columns (2t, 2t + 1) and (2t + 8, 2t + 9). The activations of both k-steps
// are then 16 bytes of x as it lies in memory: copied, not staged, and one load (with bytes as the block has them, two
// weights 16 apart, x was staged in that order by shuffles and read in two; over weights from HBM, best plans, 17408 x 5120 at sixteen / eight / one row
// 22.8 / 16.1 / 15.5 -> 21.9 / 15.0 / 14.9 us, 5120 x 17408 at eight 18.6 -> 16.8, 4096 x 4096 6.21 -> 5.78). The table values are small
// integers, exact in fp16; a sub-block's two k-steps accumulate in fp32 inside the MMA and take the integer ls - 32
// afterwards, the block's d at the end of the tile.
//
// Tile (16 rows x 256 k, 2208 bytes): words [4][lane][row g: sub-blocks 2j, 2j + 1; row g + 8: the
// same] @0, per row the eight scales ls as bytes @2048, d of rows (g, g + 8) side by side @2176.
#pragma once
#include "ggml_decode.cuh"
#include "ishi_fragstream.cuh"

namespace ishi {

struct FragIQ4XS : FragCopying {
  static constexpr int kTileBytes = 2048 + 128 + 32;
  static constexpr int kXBytes = 8 * 512, kXFixed = 8 * 64;  // a staged region: per unit eight rows of 512 bytes; the rows' skews
  static constexpr double kUnit = 1.0;  // unit of the tile results
  static constexpr bool kRows = true, kRowSums = false;  // the activations as they lie in x
  static constexpr int kExtraBytes = 256 * 128;       // the pair table: entry e of lane l's copy at e * 128 + l * 4
  static constexpr bool kRowMode = false;             // one activation row runs through the MMA path as well
  static constexpr int kFewWarps = 20;  // most warps of the smaller block size at up to eight rows
  static constexpr int kManyWarps = 16;  // most warps at nine to sixteen rows

  static __device__ __forceinline__ const uint8_t *block(const FragSrc &s, long long row, int u) {
    long long local;
    const int seg = frag_segment(s, row, &local);
    return s.w[seg] + local * s.w_row_bytes + (long long)u * 136;
  }

  static __device__ __forceinline__ uint8_t tile_byte(const FragSrc &s, long long p, int u, int b) {
    if (b < 2048) {
      const int j = b >> 9, lane = (b & 511) >> 4, i = b & 15;
      const int g = lane >> 2, t = lane & 3, wi = i >> 2, bi = i & 3;
      const long long row = p * kFragRows + g + 8 * (wi >> 1);
      if (row >= s.N) return 0;
      const int sb = 2 * j + (wi & 1);
      // weights 8 t + 2 bi and the next: the low or the high nibbles of two bytes
      const uint8_t *q = block(s, row, u) + 8 + 16 * sb + 8 * (t & 1) + 2 * bi;
      return (uint8_t)(t < 2 ? (q[0] & 15) | (q[1] << 4) : (q[0] >> 4) | (q[1] & 0xf0));
    }
    if (b < 2176) {
      const int idx = b - 2048, sb = idx & 7;
      const long long row = p * kFragRows + (idx >> 3);
      if (row >= s.N) return 32;  // d = 0 there as well
      const uint8_t *blk = block(s, row, u);
      const uint32_t low = (blk[4 + sb / 2] >> (4 * (sb % 2))) & 0xfu;
      const uint32_t high = (((uint32_t)blk[2] | ((uint32_t)blk[3] << 8)) >> (2 * sb)) & 3u;
      return (uint8_t)(low | (high << 4));
    }
    const int idx = b - 2176;
    const long long row = p * kFragRows + (idx >> 2) + 8 * ((idx >> 1) & 1);
    if (row >= s.N) return 0;
    return block(s, row, u)[idx & 1];
  }

  static __device__ __forceinline__ uint16_t tile_halfword(const FragSrc &s, long long p, int u, int hw) {
    return (uint16_t)(tile_byte(s, p, u, 2 * hw) | ((uint32_t)tile_byte(s, p, u, 2 * hw + 1) << 8));
  }

  // word i of the pair table: byte i / 32's two values as fp16, a copy per lane
  static __device__ __forceinline__ uint32_t table_word(int i) {
    const int e = i >> 5;
    const __half2 pair = __halves2half2(__int2half_rn((int)d_kvalues_iq4nl[e & 15]), __int2half_rn((int)d_kvalues_iq4nl[e >> 4]));
    return *reinterpret_cast<const uint32_t *>(&pair);
  }

  static __device__ __forceinline__ uint32_t row_stride(const FragArgs &a) { return (uint32_t)a.umax * 512u + 64u; }

  // the value pair of byte `byte` of word w
  static __device__ __forceinline__ uint32_t pair_of(uint32_t w, int byte, uint32_t table) {
    return lds32(prmt(w, 0u, 0x4440u | (uint32_t)byte) * 128u + table);
  }
  // 8388608 + byte `byte` of word w, as a float
  static __device__ __forceinline__ float byte_float(uint32_t w, int byte) {
    return __uint_as_float(prmt(w, 0x4b000000u, 0x7440u | (uint32_t)byte));
  }

  // One tile against the activations of its unit; acc is the warp's C fragment.
  template <int MODE, int NB>
  static __device__ __forceinline__ void unit(float (&acc)[NB][4], const FragArgs &a, uint32_t tile, uint32_t xbase,
                                              uint32_t tables, int uq, int g, int t, int lane) {
    const uint32_t xrow = xbase + (uint32_t)g * row_stride(a) + (uint32_t)uq * 512u + (uint32_t)t * 16u;
    const uint32_t table = tables + (uint32_t)lane * 4u;
    const uint2 sc0 = lds64(tile + 2048u + (uint32_t)g * 8u), sc1 = lds64(tile + 2048u + (uint32_t)(g + 8) * 8u);
    float su[NB][4];  // sum over the sub-blocks of (ls - 32) * (sum of value * x), d follows at the end
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) su[nb][0] = su[nb][1] = su[nb][2] = su[nb][3] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 q = lds128(tile + (uint32_t)j * 512u + (uint32_t)lane * 16u);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int sb = 2 * j + e;
        const uint32_t w0 = e ? q.y : q.x, w1 = e ? q.w : q.z;
        float part[NB][4];
        uint4 x[NB];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) x[nb] = lds128(xrow + nb * a.xregion + (uint32_t)sb * 64u);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const uint32_t a0 = pair_of(w0, 2 * s, table), a2 = pair_of(w0, 2 * s + 1, table);
          const uint32_t a1 = pair_of(w1, 2 * s, table), a3 = pair_of(w1, 2 * s + 1, table);
#pragma unroll
          for (int nb = 0; nb < NB; ++nb) {
            if (s == 0) mma16816_first(part[nb], a0, a1, a2, a3, x[nb].x, x[nb].y);
            else mma16816(part[nb], a0, a1, a2, a3, x[nb].z, x[nb].w);
          }
        }
        const float f0 = byte_float(sb < 4 ? sc0.x : sc0.y, sb & 3) - 8388640.f;  // ls - 32, exact
        const float f1 = byte_float(sb < 4 ? sc1.x : sc1.y, sb & 3) - 8388640.f;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          su[nb][0] = fmaf(f0, part[nb][0], su[nb][0]), su[nb][1] = fmaf(f0, part[nb][1], su[nb][1]);
          su[nb][2] = fmaf(f1, part[nb][2], su[nb][2]), su[nb][3] = fmaf(f1, part[nb][3], su[nb][3]);
        }
      }
    }
    const uint32_t dd = lds32(tile + 2176u + (uint32_t)g * 4u);
    const float d0 = half_bits_to_float(dd & 0xffffu), d1 = half_bits_to_float(dd >> 16);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      acc[nb][0] = fmaf(d0, su[nb][0], acc[nb][0]), acc[nb][1] = fmaf(d0, su[nb][1], acc[nb][1]);
      acc[nb][2] = fmaf(d1, su[nb][2], acc[nb][2]), acc[nb][3] = fmaf(d1, su[nb][3], acc[nb][3]);
    }
  }
};

}  // namespace ishi
