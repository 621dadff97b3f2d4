// Decoders of the GGML block formats, eight weights at a time: lane L of a warp decodes weights
// 8L .. 8L+7 of one 256-weight block, as the reference's Metal decoder does
// (Sources/IshizukiKit/Core/GGMLKernels.swift:391-401, bodies :568-761). These define "the decoded
// weight values": they must equal ggml's to_float (restated in
// Sources/IshizukiKit/Core/GGMLDequant.swift:125-428) bit for bit, so every product is written
// with explicit single-rounding intrinsics in the reference's order of operations and nothing
// here may be compiled with fast-math.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "ggml_tables.h"
#include "iq2xs_tables.h"
#include "ishi_ptx.cuh"

namespace ishi {

// codebooks (Sources/IshizukiKit/Core/GGMLTables.swift:26-1137), byte j of an entry = value j
static __device__ const uint64_t d_iq2xxs_grid[256] = {ISHI_IQ2_XXS_GRID_LIST};
static __device__ const uint16_t d_iq2xs_codes[512] = {ISHI_IQ2XS_CODES_LIST};
static __device__ const uint64_t d_iq2s_grid[1024] = {ISHI_IQ2_S_GRID_LIST};
static __device__ const uint32_t d_iq3xxs_grid[256] = {ISHI_IQ3_XXS_GRID_LIST};
static __device__ const uint32_t d_iq3s_grid[512] = {ISHI_IQ3_S_GRID_LIST};
static __device__ const uint64_t d_iq1s_grid[2048] = {ISHI_IQ1_S_GRID_LIST};
static __device__ const int8_t d_kvalues_iq4nl[16] = {ISHI_IQ4NL_VALUES_LIST};

// GGMLType.typeSize (Sources/IshizukiKit/Config/GGUFFile.swift:44-80); 0: no decoder here
__host__ __device__ constexpr int ggml_type_bytes(int type) {
  return type == 10 ? 84 : type == 12 ? 144 : type == 14 ? 210 : type == 16 ? 66 : type == 17 ? 74 : type == 18 ? 98
       : type == 19 ? 50 : type == 21 ? 110 : type == 22 ? 82 : type == 23 ? 136 : type == 29 ? 56 : 0;
}

// an entry of a type's codebook of eight values
template <int TYPE>
__device__ __forceinline__ uint64_t ggml_grid8(uint32_t i) {
  if (TYPE == 16) return d_iq2xxs_grid[i];
  if (TYPE == 22) return d_iq2s_grid[i];
  if (TYPE == 17) {  // kept as 2-bit codes
    const uint32_t codes = d_iq2xs_codes[i];
    uint64_t e = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t c = (codes >> (2 * j)) & 3u;
      e |= (uint64_t)(c == 0 ? ISHI_IQ2XS_VALUE0 : c == 1 ? ISHI_IQ2XS_VALUE1 : ISHI_IQ2XS_VALUE2) << (8 * j);
    }
    return e;
  }
  return d_iq1s_grid[i];
}

// Where a block's bytes come from. Both readers give bytes, little-endian 16- and 32-bit words, a
// run of eight bytes, and the codebooks' entries.
//
// BlockBytes: any pointer, a byte at a time (no alignment is assumed).
struct BlockBytes {
  const uint8_t *p;
  __device__ __forceinline__ uint32_t u8(int i) const { return p[i]; }
  __device__ __forceinline__ uint32_t u16(int i) const { return (uint32_t)p[i] | ((uint32_t)p[i + 1] << 8); }
  __device__ __forceinline__ uint32_t u32(int i) const { return u16(i) | (u16(i + 2) << 16); }
  __device__ __forceinline__ uint2 eight(int i) const { return make_uint2(u32(i), u32(i + 4)); }
  // eight magnitudes (IQ1: signed values), a byte each
  template <int TYPE>
  __device__ __forceinline__ uint2 entry8(uint32_t i) const {
    const uint64_t e = ggml_grid8<TYPE>(i);
    return make_uint2((uint32_t)e, (uint32_t)(e >> 32));
  }
  template <int TYPE>
  __device__ __forceinline__ uint32_t entry4(uint32_t i) const { return TYPE == 18 ? d_iq3xxs_grid[i] : d_iq3s_grid[i]; }
  __device__ __forceinline__ float iq4_value(uint32_t q) const { return (float)d_kvalues_iq4nl[q]; }
};
// BlockShared: a block staged in shared memory at an even address, the codebook beside it (see
// ggml_table_fill). Words are loaded whole; types whose size is no multiple of four put every other
// block half a word off, where a run of n words is n + 1 aligned loads and a byte permute each.
template <int TYPE>
struct BlockShared {
  uint32_t a, table;
  static constexpr bool kWords = ggml_type_bytes(TYPE) % 4 == 0;
  __device__ __forceinline__ uint32_t u8(int i) const { return lds8(a + i); }
  __device__ __forceinline__ uint32_t u16(int i) const { return lds16(a + i); }
  __device__ __forceinline__ uint32_t u32(int i) const {  // (i even)
    const uint32_t x = a + i, al = x & ~3u;
    const uint32_t w0 = lds32(al);
    return kWords && (i & 3) == 0 ? w0 : prmt(w0, lds32(al + 4), (x & 2u) ? 0x5432u : 0x3210u);
  }
  __device__ __forceinline__ uint2 eight(int i) const {
    const uint32_t x = a + i, al = x & ~3u;
    const uint32_t w0 = lds32(al), w1 = lds32(al + 4);
    if (kWords) return make_uint2(w0, w1);
    const uint32_t w2 = lds32(al + 8), sel = (x & 2u) ? 0x5432u : 0x3210u;
    return make_uint2(prmt(w0, w1, sel), prmt(w1, w2, sel));
  }
  template <int>
  __device__ __forceinline__ uint2 entry8(uint32_t i) const { return lds64(table + i * 8u); }
  template <int>
  __device__ __forceinline__ uint32_t entry4(uint32_t i) const { return lds32(table + i * 4u); }
  __device__ __forceinline__ float iq4_value(uint32_t q) const { return __uint_as_float(lds32(table + q * 4u)); }
};
// bytes of the codebook a BlockShared reader wants at `table`
__host__ __device__ constexpr int ggml_table_bytes(int type) {
  return type == 16 ? 256 * 8 : type == 17 ? 512 * 8 : type == 22 ? 1024 * 8 : type == 18 ? 256 * 4 : type == 21 ? 512 * 4
       : type == 19 || type == 29 ? 2048 * 8 : type == 23 ? 16 * 4 : 0;
}
// ... and its filling by a whole thread block
template <int TYPE>
__device__ __forceinline__ void ggml_table_fill(uint32_t table) {
  const BlockBytes g{nullptr};
  constexpr bool four = TYPE == 18 || TYPE == 21 || TYPE == 23;
  for (int i = threadIdx.x; i < ggml_table_bytes(TYPE) / (four ? 4 : 8); i += blockDim.x) {
    if (TYPE == 23) sts32(table + 4u * i, __float_as_uint(g.iq4_value(i)));
    else if (four) sts32(table + 4u * i, g.entry4<TYPE>(i));
    else {
      const uint2 e = g.entry8<TYPE>(i);
      sts64(table + 8u * i, e.x, e.y);
    }
  }
}

template <class R>
__device__ __forceinline__ float rd_half(const R &b, int i) { return half_bits_to_float(b.u16(i)); }
// the i-quants' sign byte of 7-bit index i: i with bit 7 = parity(i) (GGMLTables.swift:15-24)
__device__ __forceinline__ uint32_t ksigns(uint32_t i) { return i | ((__popc(i) & 1u) << 7); }
// v or -v by sign bit j
__device__ __forceinline__ float with_sign(float v, uint32_t signs, int j) {
  return __uint_as_float(__float_as_uint(v) ^ ((signs << (31 - j)) & 0x80000000u));
}
// byte j of a word as a float, less `off` (an integer): the bits of 2^23 + byte, then one exact
// subtraction. A conversion instruction does it in one, at a quarter of the rate.
__device__ __forceinline__ float byte_value(uint32_t w, int j, int off = 0) {
  return __fsub_rn(__uint_as_float(prmt(w, 0x4b000000u, 0x7540u | (uint32_t)j)), 8388608.f + (float)off);
}
__device__ __forceinline__ float byte_value(uint2 w, int j, int off = 0) { return byte_value(j < 4 ? w.x : w.y, j & 3, off); }
__device__ __forceinline__ uint2 shifted(uint2 w, int sh, uint32_t mask) { return make_uint2((w.x >> sh) & mask, (w.y >> sh) & mask); }

// Q2_K (GGMLDequant.swift:125-150): scale | min << 4 bytes @0, 2-bit codes @16, d @80, dmin @82
template <class R>
__device__ __forceinline__ void decode8_q2k(const R &b, int lane, float (&w)[8]) {
  const int half = lane >> 4, sh = (lane >> 2) & 3, l16 = (lane >> 1) & 1, l0 = 8 * (lane & 1);
  const uint32_t sc = b.u8(half * 8 + sh * 2 + l16);
  const float dl = __fmul_rn(rd_half(b, 80), (float)(sc & 0xfu)), ml = __fmul_rn(rd_half(b, 82), (float)(sc >> 4));
  const uint2 q = shifted(b.eight(16 + half * 32 + l16 * 16 + l0), 2 * sh, 0x03030303u);
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = __fsub_rn(__fmul_rn(dl, byte_value(q, e)), ml);
}

// Q4_K (GGMLDequant.swift:187-220)
template <class R>
__device__ __forceinline__ void decode8_q4k(const R &b, int lane, float (&w)[8]) {
  const int j = lane >> 3;           // 64-weight chunk
  const int hi = (lane >> 2) & 1;    // second 32 of the chunk: high nibbles
  const int i = 2 * j + hi;          // sub-block
  // ggml's get_scale_min_k4: sub-blocks 4 ... 7 have their low four bits in the third four bytes
  const uint32_t v0 = b.u8(4 + (i & 3)), v1 = b.u8(8 + (i & 3)), v2 = b.u8(12 + (i & 3));
  const uint32_t sc = i < 4 ? v0 & 63u : (v2 & 0xfu) | ((v0 >> 6) << 4);
  const uint32_t m = i < 4 ? v1 & 63u : (v2 >> 4) | ((v1 >> 6) << 4);
  const float dl = __fmul_rn(rd_half(b, 0), (float)sc);
  const float ml = __fmul_rn(rd_half(b, 2), (float)m);
  const uint2 q = shifted(b.eight(16 + 32 * j + 8 * (lane & 3)), 4 * hi, 0x0f0f0f0fu);
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = __fsub_rn(__fmul_rn(dl, byte_value(q, e)), ml);
}

// Q6_K (GGMLDequant.swift:154-185)
template <class R>
__device__ __forceinline__ void decode8_q6k(const R &b, int lane, float (&w)[8]) {
  const int half = lane >> 4;          // 128-weight half
  const int run = (lane >> 2) & 3;     // which of the four 32-weight runs of the half
  const int l0 = 8 * (lane & 3);       // offset inside the run
  const int scale = (int)(int8_t)b.u8(192 + 8 * half + 2 * run + l0 / 16);
  const float dl = __fmul_rn(rd_half(b, 208), (float)scale);
  const uint2 nib = shifted(b.eight(64 * half + 32 * (run & 1) + l0), run < 2 ? 0 : 4, 0x0f0f0f0fu);
  const uint2 top = shifted(b.eight(128 + 32 * half + l0), 2 * run, 0x03030303u);
  const uint2 q = make_uint2(nib.x | (top.x << 4), nib.y | (top.y << 4));
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = __fmul_rn(dl, byte_value(q, e, 32));
}

// IQ4_XS (GGMLDequant.swift:222-241): d @0, scales_h @2, scales_l @4, nibbles @8
template <class R>
__device__ __forceinline__ void decode8_iq4xs(const R &b, int lane, float (&w)[8]) {
  const int ib = lane >> 2, pos = 8 * (lane & 3);
  const int low = (b.u8(4 + ib / 2) >> (4 * (ib % 2))) & 0xf;
  const int high = (int)((b.u16(2) >> (2 * ib)) & 3u) << 4;
  const float dl = __fmul_rn(rd_half(b, 0), (float)((low | high) - 32));
  const uint2 q = shifted(b.eight(8 + 16 * ib + (pos & 15)), pos < 16 ? 0 : 4, 0x0f0f0f0fu);
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = __fmul_rn(dl, b.iq4_value(((e < 4 ? q.x : q.y) >> (8 * (e & 3))) & 0xffu));
}

// eight magnitudes times the sub-block's scale, signs by the bits of `signs`
__device__ __forceinline__ void signed8(float db, uint2 mag, uint32_t signs, float (&w)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = with_sign(__fmul_rn(db, byte_value(mag, e)), signs, e);
}

// IQ2_XXS (GGMLDequant.swift:243-262)
template <class R>
__device__ __forceinline__ void decode8_iq2xxs(const R &b, int lane, float (&w)[8]) {
  const int ib = lane >> 2, l = lane & 3;
  const uint32_t aux2 = b.u32(6 + 8 * ib);
  const float db = __fmul_rn(__fmul_rn(rd_half(b, 0), 0.5f + (float)(aux2 >> 28)), 0.25f);
  signed8(db, b.template entry8<16>(b.u8(2 + 8 * ib + l)), ksigns((aux2 >> (7 * l)) & 127u), w);
}

// IQ2_XS (GGMLDequant.swift:264-285)
template <class R>
__device__ __forceinline__ void decode8_iq2xs(const R &b, int lane, float (&w)[8]) {
  const int ib = lane >> 2, l = lane & 3;
  const uint32_t sbyte = b.u8(66 + ib);
  const uint32_t s = l < 2 ? (sbyte & 0xfu) : (sbyte >> 4);
  const float db = __fmul_rn(__fmul_rn(rd_half(b, 0), 0.5f + (float)s), 0.25f);
  const uint32_t q = b.u16(2 + 2 * lane);
  signed8(db, b.template entry8<17>(q & 511u), ksigns(q >> 9), w);
}

// IQ2_S (GGMLDequant.swift:287-311): d @0, index bytes @2, sign bytes @34, qh @66, scales @74
template <class R>
__device__ __forceinline__ void decode8_iq2s(const R &b, int lane, float (&w)[8]) {
  const int ib = lane >> 2, l = lane & 3;
  const uint32_t scale = b.u8(74 + ib);
  const float db = __fmul_rn(__fmul_rn(rd_half(b, 0), 0.5f + (float)(l < 2 ? (scale & 0xfu) : (scale >> 4))), 0.25f);
  const uint32_t idx = b.u8(2 + 4 * ib + l) | ((b.u8(66 + ib) << (8 - 2 * l)) & 0x300u);
  signed8(db, b.template entry8<22>(idx), b.u8(34 + 4 * ib + l), w);
}

// IQ3_XXS (GGMLDequant.swift:313-335): d @0, index bytes @2, signs and scales @66
template <class R>
__device__ __forceinline__ void decode8_iq3xxs(const R &b, int lane, float (&w)[8]) {
  const int ib = lane >> 2, l = lane & 3;
  const uint32_t aux = b.u32(66 + 4 * ib);
  const float db = __fmul_rn(__fmul_rn(rd_half(b, 0), 0.5f + (float)(aux >> 28)), 0.5f);
  const uint32_t q = b.u16(2 + 8 * ib + 2 * l);
  signed8(db, make_uint2(b.template entry4<18>(q & 0xffu), b.template entry4<18>(q >> 8)), ksigns((aux >> (7 * l)) & 127u), w);
}

// IQ3_S (GGMLDequant.swift:337-374): d @0, index bytes @2, qh @66, sign bytes @74, scales @106
template <class R>
__device__ __forceinline__ void decode8_iq3s(const R &b, int lane, float (&w)[8]) {
  const int ib = lane >> 2, l = lane & 3;
  const uint32_t scale = b.u8(106 + ib / 2);
  const float db = __fmul_rn(rd_half(b, 0), (float)(1 + 2 * (int)((ib & 1) ? (scale >> 4) : (scale & 0xfu))));
  const uint32_t qh = b.u8(66 + ib), q = b.u16(2 + 8 * ib + 2 * l);
  const uint32_t i1 = (q & 0xffu) | ((qh << (8 - 2 * l)) & 256u), i2 = (q >> 8) | ((qh << (7 - 2 * l)) & 256u);
  signed8(db, make_uint2(b.template entry4<21>(i1), b.template entry4<21>(i2)), b.u8(74 + 4 * ib + l), w);
}

// eight values out of {-1, 0, 1} (signed bytes) of the 2048-entry grid of IQ1_S and IQ1_M
__device__ __forceinline__ void iq1_values(float dl, uint2 g, float delta, float (&w)[8]) {
  g.x ^= 0x80808080u, g.y ^= 0x80808080u;  // value + 128, unsigned
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = __fmul_rn(dl, __fadd_rn(byte_value(g, e, 128), delta));
}

// IQ1_S (GGMLDequant.swift:376-395): d @0, index bytes @2, qh words @34
template <class R>
__device__ __forceinline__ void decode8_iq1s(const R &b, int lane, float (&w)[8]) {
  const int ib = lane >> 2, l = lane & 3;
  const uint32_t qh = b.u16(34 + 2 * ib);
  const float dl = __fmul_rn(rd_half(b, 0), (float)(2 * (int)((qh >> 12) & 7u) + 1));
  const float delta = (qh & 0x8000u) ? -0.125f : 0.125f;
  iq1_values(dl, b.template entry8<19>(b.u8(2 + 4 * ib + l) | (((qh >> (3 * l)) & 7u) << 8)), delta, w);
}

// IQ1_M (GGMLDequant.swift:397-428): index bytes @0, qh @32, four scale words @48 whose top
// nibbles spell the fp16 block scale
template <class R>
__device__ __forceinline__ void decode8_iq1m(const R &b, int lane, float (&w)[8]) {
  const int ib = lane >> 2, l = lane & 3;
  const uint2 s = b.eight(48);
  const float d = half_bits_to_float(((s.x >> 12) & 0xfu) | ((s.x >> 24) & 0x00f0u) | ((s.y >> 4) & 0x0f00u) | ((s.y >> 16) & 0xf000u));
  const uint32_t word = (ib & 4 ? s.y : s.x) >> (ib & 2 ? 16 : 0);
  const int shift = 6 * (ib % 2) + (l < 2 ? 0 : 3);
  const float dl = __fmul_rn(d, (float)(2 * (int)((word >> shift) & 7u) + 1));
  const uint32_t qh = b.u8(32 + 2 * ib + (l >> 1));
  const uint32_t idx = b.u8(4 * ib + l) | (((l & 1) ? (qh << 4) : (qh << 8)) & 0x700u);
  const float delta = (qh & ((l & 1) ? 0x80u : 0x08u)) ? -0.125f : 0.125f;
  iq1_values(dl, b.template entry8<29>(idx), delta, w);
}

template <int TYPE, class R>
__device__ __forceinline__ void decode8(const R &b, int lane, float (&w)[8]) {
  if (TYPE == 10) decode8_q2k(b, lane, w);
  else if (TYPE == 12) decode8_q4k(b, lane, w);
  else if (TYPE == 14) decode8_q6k(b, lane, w);
  else if (TYPE == 16) decode8_iq2xxs(b, lane, w);
  else if (TYPE == 17) decode8_iq2xs(b, lane, w);
  else if (TYPE == 18) decode8_iq3xxs(b, lane, w);
  else if (TYPE == 19) decode8_iq1s(b, lane, w);
  else if (TYPE == 21) decode8_iq3s(b, lane, w);
  else if (TYPE == 22) decode8_iq2s(b, lane, w);
  else if (TYPE == 23) decode8_iq4xs(b, lane, w);
  else decode8_iq1m(b, lane, w);
}
template <int TYPE>
__device__ __forceinline__ void decode8(const uint8_t *b, int lane, float (&w)[8]) { decode8<TYPE>(BlockBytes{b}, lane, w); }

}  // namespace ishi
