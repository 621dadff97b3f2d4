// GGUF IQ1_S and IQ1_M for the warp-level kernel (mma.sync fragments).
//
// Block layouts (reference: Sources/IshizukiKit/Core/GGMLDequant.swift:376-428). Eight weights are
// one entry of a 2048-entry grid of values out of {-1, 0, 1}, plus a common delta of +-1/8:
//   w = d * (2 s + 1) * (grid value + delta).
//   IQ1_S (50 bytes per 256 weights): d f16 @0, 32 index bytes @2, eight words @34 per 32 weights:
//     three more index bits for each of the four entries, the scale s (3 bits), the delta's sign.
//   IQ1_M (56 bytes): 32 index bytes @0, 16 bytes @32 (per entry a nibble: three index bits and the
//     delta's sign), four words @48: 3-bit scales per sixteen weights, and in their top nibbles the
//     fp16 d.
//
// The product is factored as
//   y += d * (sum_k (2 s + 1) g_k x_k  +  1/8 * sum_E (+-(2 s + 1))_E * sum_{k in E} x_k),
// E running over the 32 entries of a unit. The first sum is the IQ2_XS scheme: the grid lives in
// shared memory (an entry = eight bytes value + 128, four copies, copy c of entry i at
// i * 32 + c * 8), two bytes become an fp16 pair by a byte permute (the bits of 1152 + v) and one
// fused multiply-add, (1152 + v) * (2 s + 1) - 1152 * (2 s + 1), exact. The second sum is two more
// k-steps of MMA over the entries, against the entries' sums of x (fp16 high and low parts): a
// lane's eight entries per row are exactly its A registers of those two k-steps.
//
// Fragment mapping as for IQ2_XS: a lane owns the sub-blocks (sixteen weights = two entries)
// 4 j + t, j = 0..3, of rows g and g + 8. Both formats are tiled into one form, a word per sub-block
// and row, a half for each of its two entries: the index from bit 5 up, where a mask makes it a byte
// offset into the grid, the delta's sign at bit 3 (one shift brings both to bits 15 and 31) and the
// scale at bits 0 ... 2 of both halves. Tile (16 rows x 256 k, 1056 bytes; the blocks are 800 and 896):
// [2][lane][16 bytes] = for j = 2p, 2p + 1: the word of row g, of row g + 8; then d of rows (g, g + 8)
// side by side. The loop is bound by instruction issue: 17408 x 5120 at eight rows, one weight repeated
// out of L2, 17.4 us with index bytes, high bits and scale in fields of their own, 16.5 us with this
// layout (17.9 us with weights of their own in HBM).
//
// Activations of a unit in shared memory: eight rows of 256 fp16 as they lie in x, the rows
// umax * 512 + 16 bytes apart; behind all rows, per unit, the entry sums: [k-step][lane][hi hi | lo lo].
#pragma once
#include "ggml_decode.cuh"
#include "ishi_fragstream.cuh"

namespace ishi {

// TYPE: the GGML type number, 19 IQ1_S, 29 IQ1_M
template <int TYPE>
struct FragIQ1 : FragCopying {
  static_assert(TYPE == 19 || TYPE == 29, "IQ1_S or IQ1_M");
  static constexpr int kBlock = TYPE == 19 ? 50 : 56;
  static constexpr int kD = 1024;
  static constexpr int kTileBytes = kD + 32;
  // a staged region: per unit eight rows of 512 bytes and the entry sums; the rows' 16-byte skews
  static constexpr int kXBytes = 8 * 512 + 1024, kXFixed = 8 * 16;
  static constexpr double kUnit = 1.0;  // unit of the tile results
  static constexpr bool kRows = false, kRowSums = false;  // staged by loads and stores: the entry sums come from the registers (a pass over copied rows: 0.4 us a launch more)
  static constexpr int kExtraBytes = 2048 * 32;  // the grid, four copies interleaved
  static constexpr bool kRowMode = false;         // one activation row runs through the MMA path as well
  static constexpr int kFewWarps = 20;  // most warps of the smaller block size at up to eight rows
  static constexpr int kManyWarps = 16;  // most warps at nine to sixteen rows

  static __device__ __forceinline__ const uint8_t *block(const FragSrc &s, long long row, int u) {
    long long local;
    const int seg = frag_segment(s, row, &local);
    return s.w[seg] + local * s.w_row_bytes + (long long)u * kBlock;
  }
  static __device__ __forceinline__ uint32_t u16_at(const uint8_t *p) { return (uint32_t)p[0] | ((uint32_t)p[1] << 8); }

  // half e (entry e) of the word of sub-block sb of a block (see above)
  static __device__ __forceinline__ uint16_t word_half(const uint8_t *blk, int sb, int e) {
    const int ib = sb >> 1, l = 2 * (sb & 1) + e;  // the 32-group, the entry in it
    if (TYPE == 19) {
      const uint32_t qh = u16_at(blk + 34 + 2 * ib);
      return (uint16_t)((((uint32_t)blk[2 + 4 * ib + l] | (((qh >> (3 * l)) & 7u) << 8)) << 5) | ((qh >> 15) << 3) | ((qh >> 12) & 7u));
    }
    const uint32_t nibble = ((uint32_t)blk[32 + 2 * ib + (l >> 1)] >> (4 * (l & 1))) & 15u;
    const uint32_t scale = (u16_at(blk + 48 + 2 * (ib >> 1)) >> (6 * (ib & 1) + 3 * (sb & 1))) & 7u;
    return (uint16_t)((((uint32_t)blk[4 * ib + l] | ((nibble & 7u) << 8)) << 5) | (nibble & 8u) | scale);
  }

  static __device__ __forceinline__ uint16_t tile_halfword(const FragSrc &s, long long p, int u, int hw) {
    const int h = hw & 1;  // half of a word
    if (hw < kD / 2) {
      const int j = 2 * (hw >> 8) + ((hw >> 2) & 1), lane = (hw & 255) >> 3;
      const long long row = p * kFragRows + (lane >> 2) + 8 * ((hw >> 1) & 1);
      return row < s.N ? word_half(block(s, row, u), 4 * j + (lane & 3), h) : (uint16_t)0;
    }
    const long long row = p * kFragRows + ((hw - kD / 2) >> 1) + 8 * h;
    if (row >= s.N) return 0;
    const uint8_t *blk = block(s, row, u);
    if (TYPE == 19) return (uint16_t)u16_at(blk);
    const uint32_t s0 = u16_at(blk + 48), s1 = u16_at(blk + 50), s2 = u16_at(blk + 52), s3 = u16_at(blk + 54);
    return (uint16_t)((s0 >> 12) | ((s1 >> 8) & 0x00f0u) | ((s2 >> 4) & 0x0f00u) | (s3 & 0xf000u));
  }

  static __device__ __forceinline__ uint32_t row_stride(const FragArgs &a) { return (uint32_t)a.umax * 512u + 16u; }
  // the entry sums of unit u: behind the eight rows
  static __device__ __forceinline__ uint32_t sums_of(const FragArgs &a, uint32_t xfrag, int u) {
    return xfrag + (uint32_t)a.umax * 4096u + 128u + (uint32_t)u * 1024u;
  }

  // word i of the grid: entry i / 8's eight values, each + 128, in four copies side by side
  static __device__ __forceinline__ uint32_t table_word(int i) {
    return (uint32_t)((d_iq1s_grid[i >> 3] ^ 0x8080808080808080ull) >> (32 * (i & 1)));
  }

  // Activations of the CTA's column range as they lie in x (rows past M as zeros), and per entry
  // (the eight values of one lane) their sum as fp16 high and low parts, where the MMA over the
  // entries reads them: entry E = 2 (4 j + t) + e is slot 2t + e + 8 (j % 2) of k-step j / 2, i.e.
  // register j % 2, half e, of lane (r, t). No rotation here.
  template <class Then>
  static __device__ __forceinline__ void stage_x(const FragArgs &a, const FragRows &m, uint32_t xfrag, int ub0, int uc, Then then) {
    const int lane = threadIdx.x & 31;
    const uint32_t R = row_stride(a);
    const int sb = lane >> 1, j = sb >> 2, t = sb & 3;
    const uint32_t slot = (uint32_t)((j >> 1) * 512 + t * 16 + (j & 1) * 4 + (lane & 1) * 2);
    frag_stage_rows(a, m, ub0, uc, then, [&](int u, int r, uint4 v) {
      sts128u(xfrag + (uint32_t)r * R + (uint32_t)u * 512u + (uint32_t)lane * 16u, v);
      const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&v.x));
      const float2 f1 = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
      const float2 f2 = __half22float2(*reinterpret_cast<const __half2 *>(&v.z));
      const float2 f3 = __half22float2(*reinterpret_cast<const __half2 *>(&v.w));
      const float s = ((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y));
      const __half hi = __float2half_rn(s), lo = __float2half_rn(s - __half2float(hi));
      const uint32_t at = sums_of(a, xfrag, u) + (uint32_t)r * 64u + slot;
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"(__half_as_ushort(hi)) : "memory");
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(at + 8u), "h"(__half_as_ushort(lo)) : "memory");
    });
  }

  // eight weights as four A registers, value * (2 s + 1): address of the grid entry (this lane's
  // copy), scale = 2 s + 1 and offset = -1152 * (2 s + 1) in both halves
  static __device__ __forceinline__ void entry(uint32_t *r, uint32_t at, __half2 scale, __half2 offset) {
    const uint2 m = lds64(at);
    const uint32_t bits[4] = {prmt(m.x, 0x64646464u, 0x4140u), prmt(m.x, 0x64646464u, 0x4342u), prmt(m.y, 0x64646464u, 0x4140u),
                              prmt(m.y, 0x64646464u, 0x4342u)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 v = __hfma2(*reinterpret_cast<const __half2 *>(&bits[i]), scale, offset);
      r[i] = *reinterpret_cast<const uint32_t *>(&v);
    }
  }
  // a word's sixteen weights as eight A registers (`copy`: byte offset of this lane's copy of the
  // grid), and its entries' +-(2 s + 1)
  static __device__ __forceinline__ uint32_t sub_block(uint32_t (&r)[8], uint32_t w, uint32_t grid, uint32_t copy) {
    const uint32_t bits = (w & 0x00070007u) | 0x64006400u;  // 1024 + s
    const __half2 scale = __hfma2(*reinterpret_cast<const __half2 *>(&bits), __float2half2_rn(2.f), __float2half2_rn(-2047.f));
    const __half2 offset = __hmul2(scale, __float2half2_rn(-1152.f));
    entry(r, grid + ((w & 0xffe0u) | copy), scale, offset);
    entry(r + 4, grid + (((w >> 16) & 0xffe0u) | copy), scale, offset);
    return *reinterpret_cast<const uint32_t *>(&scale) ^ ((w << 12) & 0x80008000u);
  }

  // One tile against the activations of its unit; acc is the warp's C fragment.
  template <int MODE, int NB>
  static __device__ __forceinline__ void unit(float (&acc)[NB][4], const FragArgs &a, uint32_t tile, uint32_t xbase,
                                              uint32_t tables, int uq, int g, int t, int lane) {
    const uint32_t R = row_stride(a);
    const uint32_t copy = (uint32_t)(lane & 3) * 8u;
    const uint32_t xrow = xbase + (uint32_t)g * R + (uint32_t)uq * 512u + (uint32_t)t * 32u;
    float c[NB][4];
    uint32_t da[2][4];  // the A registers of the two k-steps over the entries: +-(2 s + 1)
#pragma unroll
    for (int pc = 0; pc < 2; ++pc) {
      const uint4 w = lds128(tile + (uint32_t)pc * 512u + (uint32_t)lane * 16u);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = 2 * pc + e;
        uint32_t r0[8], r1[8];  // sub-block 4 j + t of row g, of row g + 8
        da[j >> 1][(j & 1) * 2] = sub_block(r0, e ? w.z : w.x, tables, copy);
        da[j >> 1][(j & 1) * 2 + 1] = sub_block(r1, e ? w.w : w.y, tables, copy);
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
    // sum_E +-(2 s + 1) * (sum of x over entry E): da[ks] = {row g: j = 2 ks, row g + 8: j = 2 ks,
    // row g: j = 2 ks + 1, row g + 8: j = 2 ks + 1} = the registers a0, a1, a2, a3 of k-step ks
    const uint32_t sums = sums_of(a, xbase, uq) + (uint32_t)lane * 16u;
    const uint32_t dd = lds32(tile + (uint32_t)kD + (uint32_t)g * 4u);
    const float d0 = half_bits_to_float(dd & 0xffffu), d1 = half_bits_to_float(dd >> 16);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      float cm[4];
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        const uint4 bs = lds128(sums + nb * a.xregion + (uint32_t)ks * 512u);
        if (ks == 0) mma16816_first(cm, da[ks][0], da[ks][1], da[ks][2], da[ks][3], bs.x, bs.y);
        else mma16816(cm, da[ks][0], da[ks][1], da[ks][2], da[ks][3], bs.x, bs.y);
        mma16816(cm, da[ks][0], da[ks][1], da[ks][2], da[ks][3], bs.z, bs.w);
      }
      acc[nb][0] = fmaf(d0, fmaf(0.125f, cm[0], c[nb][0]), acc[nb][0]);
      acc[nb][1] = fmaf(d0, fmaf(0.125f, cm[1], c[nb][1]), acc[nb][1]);
      acc[nb][2] = fmaf(d1, fmaf(0.125f, cm[2], c[nb][2]), acc[nb][2]);
      acc[nb][3] = fmaf(d1, fmaf(0.125f, cm[3], c[nb][3]), acc[nb][3]);
    }
  }
};

}  // namespace ishi
