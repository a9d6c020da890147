// GGUF block formats on the device: one 32-weight chunk of a packed row as fp32 values (decode32), and as tensor-core operands
// (frag: the block's small integers, which bf16 holds exactly, with their scales beside them in fp32).
#pragma once
#include "common.cuh"

namespace ve {

enum GgmlType { kQ4_0 = 2, kQ4_1 = 3, kQ5_0 = 6, kQ5_1 = 7, kQ8_0 = 8, kQ2_K = 10, kQ3_K = 11, kQ4_K = 12, kQ5_K = 13,
                kQ6_K = 14, kIQ2_XXS = 16, kIQ2_XS = 17, kIQ3_XXS = 18, kIQ1_S = 19, kIQ4_NL = 20, kIQ3_S = 21, kIQ2_S = 22,
                kIQ4_XS = 23, kIQ1_M = 29 };

// Codebook formats (IQ1 / IQ2 / IQ3): one table of grid vectors and sign bytes in device memory, uploaded once per device
// by the host (ve_gguf_set_iq_grids). Byte offsets of the parts, as in quant/gguf_iq.py:
//   0 sign bytes [128] | 128 iq2xxs [256][8] | 2176 iq2xs [512][8] | 6272 iq2s [1024][8] | 14464 iq3xxs [256][4]
//   | 15488 iq3s [512][4] | 17536 iq1s [2048][8] (int8)
static __constant__ const uint8_t* kIqGrids;
constexpr int kOffSigns = 0, kOff2xxs = 128, kOff2xs = 2176, kOff2s = 6272, kOff3xxs = 14464, kOff3s = 15488, kOff1s = 17536;

// 8 grid bytes times a scale with the signs of `sb` (bit j set = element j negative)
VE_DEVINL void put8(const uint8_t* __restrict__ g, uint32_t sb, float db, float* w) {
  const uint2 v = *reinterpret_cast<const uint2*>(g);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w[j] = ((sb >> j) & 1 ? -db : db) * (float)((v.x >> (8 * j)) & 255);
    w[j + 4] = ((sb >> (j + 4)) & 1 ? -db : db) * (float)((v.y >> (8 * j)) & 255);
  }
}
VE_DEVINL void put4(const uint8_t* __restrict__ g, uint32_t sb, float db, float* w) {
  const uint32_t v = *reinterpret_cast<const uint32_t*>(g);
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = ((sb >> j) & 1 ? -db : db) * (float)((v >> (8 * j)) & 255);
}
// 8 ternary grid values (int8) plus a shift, times a scale
VE_DEVINL void put8_shift(const uint8_t* __restrict__ g, float delta, float dl, float* w) {
  const uint2 v = *reinterpret_cast<const uint2*>(g);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w[j] = dl * ((float)(int8_t)((v.x >> (8 * j)) & 255) + delta);
    w[j + 4] = dl * ((float)(int8_t)((v.y >> (8 * j)) & 255) + delta);
  }
}

// the 16 non-uniform levels of the IQ4 formats
static __constant__ int8_t kIq4Levels[16] = {-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113};

VE_DEVINL void scale_min_k4(const uint8_t* s, int sb, int& sc, int& mn) {
  if (sb < 4) { sc = s[sb] & 63; mn = s[sb + 4] & 63; }
  else { sc = (s[sb + 4] & 15) | ((s[sb - 4] >> 6) << 4); mn = (s[sb + 4] >> 4) | ((s[sb] >> 6) << 4); }
}

VE_DEVINL float h2f(const uint8_t* p) {
  return __half2float(__ushort_as_half((unsigned short)(p[0] | (p[1] << 8))));
}

// Decode the 32 weights of chunk `c` of a packed row into w[32].
template <int TYPE>
VE_DEVINL void decode32(const uint8_t* __restrict__ row, int c, float* w) {
  if (TYPE == kQ8_0) {
    const uint8_t* b = row + (size_t)c * 34;
    const float d = h2f(b);
#pragma unroll
    for (int j = 0; j < 32; ++j) w[j] = d * (float)(int8_t)b[2 + j];
  } else if (TYPE == kQ4_0) {
    const uint8_t* b = row + (size_t)c * 18;
    const float d = h2f(b);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      w[j] = d * (float)((int)(b[2 + j] & 15) - 8);
      w[j + 16] = d * (float)((int)(b[2 + j] >> 4) - 8);
    }
  } else if (TYPE == kQ4_K) {
    const uint8_t* b = row + (size_t)(c >> 3) * 144;
    const int sb = c & 7;                       // sub-block 0..7
    const float d = h2f(b), dmin = h2f(b + 2);
    const uint8_t* s = b + 4;
    int sc, mn;
    scale_min_k4(s, sb, sc, mn);
    const float d1 = d * (float)sc, m1 = dmin * (float)mn;
    const uint8_t* q = b + 16 + (sb >> 1) * 32;
    const int shift = (sb & 1) * 4;
#pragma unroll
    for (int j = 0; j < 32; ++j) w[j] = d1 * (float)((q[j] >> shift) & 15) - m1;
  } else if (TYPE == kQ4_1) {
    const uint8_t* b = row + (size_t)c * 20;
    const float d = h2f(b), m = h2f(b + 2);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      w[j] = fmaf(d, (float)(b[4 + j] & 15), m);
      w[j + 16] = fmaf(d, (float)(b[4 + j] >> 4), m);
    }
  } else if (TYPE == kQ5_0 || TYPE == kQ5_1) {
    const int hdr = TYPE == kQ5_0 ? 2 : 4;
    const uint8_t* b = row + (size_t)c * (TYPE == kQ5_0 ? 22 : 24);
    const float d = h2f(b), m = TYPE == kQ5_0 ? 0.f : h2f(b + 2);
    const uint32_t qh = b[hdr] | (b[hdr + 1] << 8) | (b[hdr + 2] << 16) | ((uint32_t)b[hdr + 3] << 24);
    const int off = TYPE == kQ5_0 ? 16 : 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int q0 = (b[hdr + 4 + j] & 15) | (((qh >> j) & 1) << 4);
      const int q1 = (b[hdr + 4 + j] >> 4) | (((qh >> (j + 16)) & 1) << 4);
      w[j] = fmaf(d, (float)(q0 - off), m);
      w[j + 16] = fmaf(d, (float)(q1 - off), m);
    }
  } else if (TYPE == kIQ4_NL) {
    const uint8_t* b = row + (size_t)c * 18;
    const float d = h2f(b);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      w[j] = d * (float)kIq4Levels[b[2 + j] & 15];
      w[j + 16] = d * (float)kIq4Levels[b[2 + j] >> 4];
    }
  } else if (TYPE == kIQ4_XS) {
    const uint8_t* b = row + (size_t)(c >> 3) * 136;
    const int ib = c & 7;
    const int sh = b[2] | (b[3] << 8);
    const int ls = ((b[4 + (ib >> 1)] >> (4 * (ib & 1))) & 15) | (((sh >> (2 * ib)) & 3) << 4);
    const float dl = h2f(b) * (float)(ls - 32);
    const uint8_t* q = b + 8 + ib * 16;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      w[j] = dl * (float)kIq4Levels[q[j] & 15];
      w[j + 16] = dl * (float)kIq4Levels[q[j] >> 4];
    }
  } else if (TYPE == kIQ2_XXS) {
    const uint8_t* b = row + (size_t)(c >> 3) * 66;
    const uint8_t* q = b + 2 + (c & 7) * 8;
    const uint32_t aux = q[4] | (q[5] << 8) | (q[6] << 16) | ((uint32_t)q[7] << 24);
    const float db = h2f(b) * (0.5f + (float)(aux >> 28)) * 0.25f;
#pragma unroll
    for (int l = 0; l < 4; ++l)
      put8(kIqGrids + kOff2xxs + q[l] * 8, kIqGrids[kOffSigns + ((aux >> (7 * l)) & 127)], db, w + 8 * l);
  } else if (TYPE == kIQ2_XS) {
    const uint8_t* b = row + (size_t)(c >> 3) * 74;
    const int ib = c & 7;
    const uint8_t* q = b + 2 + ib * 8;
    const int sc = b[66 + ib];
    const float d = h2f(b);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const int v = q[2 * l] | (q[2 * l + 1] << 8);
      const float db = d * (0.5f + (float)(l < 2 ? (sc & 15) : (sc >> 4))) * 0.25f;
      put8(kIqGrids + kOff2xs + (v & 511) * 8, kIqGrids[kOffSigns + (v >> 9)], db, w + 8 * l);
    }
  } else if (TYPE == kIQ2_S) {
    const uint8_t* b = row + (size_t)(c >> 3) * 82;
    const int ib = c & 7;
    const uint8_t* q = b + 2 + ib * 4;
    const uint8_t* sg = b + 34 + ib * 4;
    const int qh = b[66 + ib], sc = b[74 + ib];
    const float d = h2f(b);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const float db = d * (0.5f + (float)(l < 2 ? (sc & 15) : (sc >> 4))) * 0.25f;
      put8(kIqGrids + kOff2s + (q[l] | ((qh << (8 - 2 * l)) & 0x300)) * 8, sg[l], db, w + 8 * l);
    }
  } else if (TYPE == kIQ3_XXS) {
    const uint8_t* b = row + (size_t)(c >> 3) * 98;
    const int ib = c & 7;
    const uint8_t* q = b + 2 + ib * 8;
    const uint8_t* a = b + 66 + ib * 4;
    const uint32_t aux = a[0] | (a[1] << 8) | (a[2] << 16) | ((uint32_t)a[3] << 24);
    const float db = h2f(b) * (0.5f + (float)(aux >> 28)) * 0.5f;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t sb = kIqGrids[kOffSigns + ((aux >> (7 * l)) & 127)];
      put4(kIqGrids + kOff3xxs + q[2 * l] * 4, sb, db, w + 8 * l);
      put4(kIqGrids + kOff3xxs + q[2 * l + 1] * 4, sb >> 4, db, w + 8 * l + 4);
    }
  } else if (TYPE == kIQ3_S) {
    const uint8_t* b = row + (size_t)(c >> 3) * 110;
    const int ib = c & 7;
    const uint8_t* q = b + 2 + ib * 8;
    const int qh = b[66 + ib];
    const uint8_t* sg = b + 74 + ib * 4;
    const int nib = (b[106 + (ib >> 1)] >> (4 * (ib & 1))) & 15;
    const float db = h2f(b) * (float)(1 + 2 * nib);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      put4(kIqGrids + kOff3s + (q[2 * l] | ((qh << (8 - 2 * l)) & 256)) * 4, sg[l], db, w + 8 * l);
      put4(kIqGrids + kOff3s + (q[2 * l + 1] | ((qh << (7 - 2 * l)) & 256)) * 4, sg[l] >> 4, db, w + 8 * l + 4);
    }
  } else if (TYPE == kIQ1_S) {
    const uint8_t* b = row + (size_t)(c >> 3) * 50;
    const int ib = c & 7;
    const uint8_t* q = b + 2 + ib * 4;
    const int qh = b[34 + 2 * ib] | (b[35 + 2 * ib] << 8);
    const float dl = h2f(b) * (float)(2 * ((qh >> 12) & 7) + 1);
    const float delta = (qh & 0x8000) ? -0.125f : 0.125f;
#pragma unroll
    for (int l = 0; l < 4; ++l)
      put8_shift(kIqGrids + kOff1s + (q[l] | (((qh >> (3 * l)) & 7) << 8)) * 8, delta, dl, w + 8 * l);
  } else if (TYPE == kIQ1_M) {
    const uint8_t* b = row + (size_t)(c >> 3) * 56;
    const int ib = c & 7;
    const uint8_t* q = b + ib * 4;
    const int q0 = b[32 + 2 * ib], q1 = b[33 + 2 * ib];
    const uint8_t* s8 = b + 48;
    const int s0 = s8[0] | (s8[1] << 8), s1 = s8[2] | (s8[3] << 8), s2 = s8[4] | (s8[5] << 8), s3 = s8[6] | (s8[7] << 8);
    const unsigned short bits = (unsigned short)((s0 >> 12) | ((s1 >> 8) & 0x00f0) | ((s2 >> 4) & 0x0f00) | (s3 & 0xf000));
    const float d = __half2float(__ushort_as_half(bits));
    const int sw = (ib >> 1) == 0 ? s0 : (ib >> 1) == 1 ? s1 : (ib >> 1) == 2 ? s2 : s3;
    const float dl1 = d * (float)(2 * ((sw >> (6 * (ib & 1))) & 7) + 1);
    const float dl2 = d * (float)(2 * ((sw >> (6 * (ib & 1) + 3)) & 7) + 1);
    put8_shift(kIqGrids + kOff1s + (q[0] | ((q0 << 8) & 0x700)) * 8, (q0 & 0x08) ? -0.125f : 0.125f, dl1, w);
    put8_shift(kIqGrids + kOff1s + (q[1] | ((q0 << 4) & 0x700)) * 8, (q0 & 0x80) ? -0.125f : 0.125f, dl1, w + 8);
    put8_shift(kIqGrids + kOff1s + (q[2] | ((q1 << 8) & 0x700)) * 8, (q1 & 0x08) ? -0.125f : 0.125f, dl2, w + 16);
    put8_shift(kIqGrids + kOff1s + (q[3] | ((q1 << 4) & 0x700)) * 8, (q1 & 0x80) ? -0.125f : 0.125f, dl2, w + 24);
  } else if (TYPE == kQ2_K) {
    const uint8_t* b = row + (size_t)(c >> 3) * 84;
    const int half = (c >> 2) & 1, sft = (c & 3) * 2;
    const float d = h2f(b + 80), dmin = h2f(b + 82);
    const uint8_t* q = b + 16 + half * 32;
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      const int s = b[half * 8 + (c & 3) * 2 + part];
      const float dl = d * (float)(s & 15), ml = dmin * (float)(s >> 4);
#pragma unroll
      for (int l = 0; l < 16; ++l) w[part * 16 + l] = dl * (float)((q[part * 16 + l] >> sft) & 3) - ml;
    }
  } else if (TYPE == kQ3_K) {
    const uint8_t* b = row + (size_t)(c >> 3) * 110;
    const int half = (c >> 2) & 1, j4 = c & 3, sft = j4 * 2, bit = half * 4 + j4;
    const float d = h2f(b + 108);
    const uint8_t* hm = b;
    const uint8_t* q = b + 32 + half * 32;
    const uint8_t* s12 = b + 96;
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      const int i = half * 8 + j4 * 2 + part;                 // scale index 0..15
      const int lo = i < 8 ? (s12[i] & 15) : (s12[i - 8] >> 4);
      const int hi = (s12[8 + (i & 3)] >> (2 * (i >> 2))) & 3;
      const float dl = d * (float)((lo | (hi << 4)) - 32);
#pragma unroll
      for (int l = 0; l < 16; ++l) {
        const int e = part * 16 + l;
        w[e] = dl * (float)((int)((q[e] >> sft) & 3) - (((hm[e] >> bit) & 1) ? 0 : 4));
      }
    }
  } else if (TYPE == kQ5_K) {
    const uint8_t* b = row + (size_t)(c >> 3) * 176;
    const int sb = c & 7;
    const float d = h2f(b), dmin = h2f(b + 2);
    int sc, mn;
    scale_min_k4(b + 4, sb, sc, mn);
    const float d1 = d * (float)sc, m1 = dmin * (float)mn;
    const uint8_t* qh = b + 16;
    const uint8_t* q = b + 48 + (sb >> 1) * 32;
    const int shift = (sb & 1) * 4;
#pragma unroll
    for (int j = 0; j < 32; ++j) w[j] = d1 * (float)(((q[j] >> shift) & 15) | (((qh[j] >> sb) & 1) << 4)) - m1;
  } else {  // Q6_K
    const uint8_t* b = row + (size_t)(c >> 3) * 210;
    const int sub = c & 7, half = sub >> 2, qtr = sub & 3;
    const uint8_t* ql = b + half * 64 + (qtr & 1) * 32;
    const uint8_t* qh = b + 128 + half * 32;
    const int8_t* sc = reinterpret_cast<const int8_t*>(b + 192) + half * 8 + qtr * 2;
    const float d = h2f(b + 208);
    const int lshift = (qtr >> 1) * 4, hshift = qtr * 2;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int q = (int)(((ql[j] >> lshift) & 15) | (((qh[j] >> hshift) & 3) << 4)) - 32;
      w[j] = d * (float)sc[j >> 4] * (float)q;
    }
  }
}


// ---------------------------------------------------------------------------------------------------------------------------
// Operand fragments. Every format is   w = s * q - m   with q an integer of at most 8 significant bits (or a codebook value plus an
// eighth), s one scale per 16 or 32 weights, m a minimum for some formats: q goes to the tensor cores as bf16, exactly, and s and m
// are applied in fp32 to the sums of 16 or 32 products, so nothing is rounded that decode32 does not round.
template <int TYPE>
struct Fmt {
  static constexpr bool kBig = TYPE >= kQ2_K && TYPE != kIQ4_NL;       // 256-weight blocks
  static constexpr int kBytes = TYPE == kQ8_0 ? 34 : TYPE == kQ4_0 || TYPE == kIQ4_NL ? 18 : TYPE == kQ4_1 ? 20 : TYPE == kQ5_0 ? 22
      : TYPE == kQ5_1 ? 24 : TYPE == kQ2_K ? 84 : TYPE == kQ3_K ? 110 : TYPE == kQ4_K ? 144 : TYPE == kQ5_K ? 176 : TYPE == kQ6_K ? 210
      : TYPE == kIQ2_XXS ? 66 : TYPE == kIQ2_XS ? 74 : TYPE == kIQ3_XXS ? 98 : TYPE == kIQ1_S ? 50 : TYPE == kIQ3_S ? 110
      : TYPE == kIQ2_S ? 82 : TYPE == kIQ4_XS ? 136 : 56;
  // chunks of 32 weights that a warp stages at a time, and their bytes
  static constexpr int kChunks = TYPE == kQ8_0 ? 4 : 8;
  static constexpr int kUnit = kBig ? kBytes : kBytes * kChunks;
  static constexpr bool kWords = kBytes % 4 == 0;                       // fields lie on 4-byte boundaries (where the rows do)
  static constexpr bool kScale16 = TYPE == kQ2_K || TYPE == kQ3_K || TYPE == kQ6_K || TYPE == kIQ2_XS || TYPE == kIQ2_S;
  static constexpr int kMin = TYPE == kQ2_K ? 2 : (TYPE == kQ4_K || TYPE == kQ5_K || TYPE == kQ4_1 || TYPE == kQ5_1) ? 1 : 0;
  // codebook in shared memory
  // IQ1: a lane takes a whole codebook vector, 8 weights, and the odd scale factors 1..15 are part of the integers
  static constexpr bool kVec8 = TYPE == kIQ1_S || TYPE == kIQ1_M;
  static constexpr int kTable = TYPE == kIQ2_XXS ? 2048 : TYPE == kIQ2_XS ? 4096 : TYPE == kIQ2_S ? 8192 : TYPE == kIQ3_XXS ? 1024
      : TYPE == kIQ3_S ? 2048 : TYPE == kIQ1_S || TYPE == kIQ1_M ? 8192 + 128 : TYPE == kIQ4_NL || TYPE == kIQ4_XS ? 1024 : 0;
  static constexpr bool kSigns = TYPE == kIQ2_XXS || TYPE == kIQ2_XS || TYPE == kIQ3_XXS;
  static constexpr int kTabBytes = kTable + (kSigns ? 128 : 0);
};

// The block's threads copy the format's codebook to `tab` (16-byte aligned): grid bytes as they are with the sign table behind them;
// IQ1: 32 bits per vector, four per value (value + 1: a byte-permute selector), and behind them, for scale s and sign of the shift
// (index s + 8 * negative), the low and the high bytes of the bf16 values (2 s + 1) * (value +- 1/8); IQ4: the bf16 levels of two nibbles.
template <int TYPE>
VE_DEVINL void load_table(uint8_t* tab) {
  if (TYPE == kIQ4_NL || TYPE == kIQ4_XS) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
      const __nv_bfloat162 v = __floats2bfloat162_rn((float)kIq4Levels[i & 15], (float)kIq4Levels[i >> 4]);
      reinterpret_cast<uint32_t*>(tab)[i] = *reinterpret_cast<const uint32_t*>(&v);
    }
  } else if (TYPE == kIQ1_S || TYPE == kIQ1_M) {
    for (int i = threadIdx.x; i < 2048; i += blockDim.x) {
      const uint2 g = *reinterpret_cast<const uint2*>(kIqGrids + kOff1s + i * 8);
      uint32_t v = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) v |= ((((j < 4 ? g.x : g.y) >> (8 * (j & 3))) + 1) & 3) << (4 * j);      // -1, 0, 1 as 0, 1, 2
      reinterpret_cast<uint32_t*>(tab)[i] = v;
    }
    if (threadIdx.x < 16) {
      const float m = (float)(2 * (threadIdx.x & 7) + 1), dl = threadIdx.x & 8 ? -0.125f : 0.125f;
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const uint32_t v = __bfloat16_as_ushort(__float2bfloat16_rn(m * ((float)(j - 1) + dl)));              // at most 8 bits: exact
        lo |= (v & 255) << (8 * j);
        hi |= (v >> 8) << (8 * j);
      }
      reinterpret_cast<uint2*>(tab + 8192)[threadIdx.x] = make_uint2(lo, hi);
    }
  } else if (Fmt<TYPE>::kTable > 0) {
    constexpr int off = TYPE == kIQ2_XXS ? kOff2xxs : TYPE == kIQ2_XS ? kOff2xs : TYPE == kIQ2_S ? kOff2s : TYPE == kIQ3_XXS ? kOff3xxs : kOff3s;
    for (int i = threadIdx.x; i < Fmt<TYPE>::kTable / 4; i += blockDim.x)
      reinterpret_cast<uint32_t*>(tab)[i] = reinterpret_cast<const uint32_t*>(kIqGrids + off)[i];
    if (Fmt<TYPE>::kSigns)
      for (int i = threadIdx.x; i < 32; i += blockDim.x)
        reinterpret_cast<uint32_t*>(tab + Fmt<TYPE>::kTable)[i] = reinterpret_cast<const uint32_t*>(kIqGrids + kOffSigns)[i];
  }
}

VE_DEVINL float u2f(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.f; }       // v < 2^23
VE_DEVINL uint32_t ld16(const uint8_t* p) { return *reinterpret_cast<const unsigned short*>(p); }
template <bool WORDS>
VE_DEVINL uint32_t ld32(const uint8_t* p) {
  if (WORDS) return *reinterpret_cast<const uint32_t*>(p);
  return ld16(p) | (ld16(p + 2) << 16);
}
VE_DEVINL float half_at(const uint8_t* p) { return __half2float(__ushort_as_half((unsigned short)ld16(p))); }
VE_DEVINL uint32_t bsub2(uint32_t a, uint32_t b) {            // exact differences of small integers
  const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// Bytes 0, 1 (2, 3) of a word, as two 16-bit fields.
VE_DEVINL uint32_t b01(uint32_t w) { return __byte_perm(w, 0u, 0x4140); }
VE_DEVINL uint32_t b23(uint32_t w) { return __byte_perm(w, 0u, 0x4342); }
// Two int8 values in 16-bit fields -> bf16: 128 + low seven bits, less 128 or (sign bit set) 256. bf16 128.0 is 0x4300 with an ulp of
// one, and the sign bit falls on the exponent's lowest bit.
VE_DEVINL uint32_t s8_bf16(uint32_t p) { return bsub2((p & 0x007f007fu) | 0x43004300u, (p & 0x00800080u) | 0x43004300u); }
// Two unsigned fields below 128 -> bf16, less `off` (128 + offset as bf16 in both halves).
VE_DEVINL uint32_t u7_bf16(uint32_t p, uint32_t off) { return bsub2(p | 0x43004300u, off); }
// bits 0..3 of v to the signs of (a[0] lo, a[0] hi, a[1] lo, a[1] hi)
VE_DEVINL void flip4(uint32_t v, uint32_t* a) {
  a[0] ^= ((v << 15) & 0x8000u) | ((v << 30) & 0x80000000u);
  a[1] ^= ((v << 13) & 0x8000u) | ((v << 28) & 0x80000000u);
}

// Lane t (0..3) of a quad takes weights 16 i + 4 t .. + 3 of chunk c of the unit at `u`, for the groups i = 0, 1 of 16 weights:
// a[2 i], a[2 i + 1] = their bf16 pairs; s[i], m[i] the group's scale and minimum (only s[0], m[0] where they hold for the chunk).
template <int TYPE>
VE_DEVINL void frag(const uint8_t* u, int c, int t, const uint8_t* tab, uint32_t* a, float* s, float* m) {
  constexpr bool W = Fmt<TYPE>::kWords;
  if (TYPE == kQ8_0) {
    const uint8_t* b = u + c * 34;
    s[0] = half_at(b);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a[2 * i] = s8_bf16(b01(ld16(b + 2 + 16 * i + 4 * t)));
      a[2 * i + 1] = s8_bf16(b01(ld16(b + 4 + 16 * i + 4 * t)));
    }
  } else if (TYPE == kQ4_0 || TYPE == kQ4_1 || TYPE == kQ5_0 || TYPE == kQ5_1 || TYPE == kIQ4_NL || TYPE == kIQ4_XS) {
    const uint8_t* q;                                   // 16 bytes: weights j (low nibbles) and 16 + j
    uint32_t h = 0;
    if (TYPE == kIQ4_XS) {
      const uint32_t sh = ld16(u + 2);
      const uint32_t ls = ((u[4 + (c >> 1)] >> (4 * (c & 1))) & 15) | (((sh >> (2 * c)) & 3) << 4);
      s[0] = half_at(u) * (u2f(ls) - 32.f);
      q = u + 8 + c * 16;
    } else {
      const uint8_t* b = u + c * Fmt<TYPE>::kBytes;
      s[0] = half_at(b);
      if (TYPE == kQ4_1 || TYPE == kQ5_1) m[0] = -half_at(b + 2);
      const int hdr = TYPE == kQ4_1 || TYPE == kQ5_1 ? 4 : 2;
      if (TYPE == kQ5_0 || TYPE == kQ5_1) h = ld32<W>(b + hdr) >> (4 * t);
      q = b + hdr + (TYPE == kQ5_0 || TYPE == kQ5_1 ? 4 : 0);
    }
    const uint32_t w = ld32<W>(q + 4 * t);
    const uint32_t p[2] = {b01(w), b23(w)};
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (TYPE == kIQ4_NL || TYPE == kIQ4_XS) {
          const uint32_t v = p[j] >> (4 * i);
          a[2 * i + j] = reinterpret_cast<const uint32_t*>(tab)[(v & 15) | ((v >> 12) & 0xf0)];
        } else {
          uint32_t v = (p[j] >> (4 * i)) & 0x000f000fu;
          if (TYPE == kQ5_0 || TYPE == kQ5_1) {
            const uint32_t hb = h >> (16 * i + 2 * j);
            v |= ((hb << 4) & 0x10u) | ((hb << 19) & 0x100000u);
          }
          a[2 * i + j] = u7_bf16(v, TYPE == kQ4_0 ? 0x43084308u : TYPE == kQ5_0 ? 0x43104310u : 0x43004300u);
        }
      }
  } else if (TYPE == kQ4_K || TYPE == kQ5_K) {
    const uint32_t w0 = ld32<W>(u + 4), w1 = ld32<W>(u + 8), w2 = ld32<W>(u + 12);
    // four scales (minima) of six bits in the bytes of a word, for chunks 0..3 and 4..7
    const uint32_t sw = c < 4 ? w0 & 0x3f3f3f3fu : (w2 & 0x0f0f0f0fu) | ((w0 >> 2) & 0x30303030u);
    const uint32_t mw = c < 4 ? w1 & 0x3f3f3f3fu : ((w2 >> 4) & 0x0f0f0f0fu) | ((w1 >> 2) & 0x30303030u);
    // d * byte: the byte as 2^23 + byte, the 2^23 taken off inside the FMA (d * 2^23 is exact)
    const float d = half_at(u), dmin = half_at(u + 2);
    s[0] = fmaf(d, __uint_as_float(__byte_perm(sw, 0x4B000000u, 0x7440u | (c & 3))), -8388608.f * d);
    m[0] = fmaf(dmin, __uint_as_float(__byte_perm(mw, 0x4B000000u, 0x7440u | (c & 3))), -8388608.f * dmin);
    const uint8_t* q = u + (TYPE == kQ4_K ? 16 : 48) + (c >> 1) * 32;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t w = (ld32<W>(q + 16 * i + 4 * t) >> (4 * (c & 1))) & 0x0f0f0f0fu;
      if (TYPE == kQ5_K) w |= ((ld32<W>(u + 16 + 16 * i + 4 * t) >> c) & 0x01010101u) << 4;
      a[2 * i] = u7_bf16(b01(w), 0x43004300u);
      a[2 * i + 1] = u7_bf16(b23(w), 0x43004300u);
    }
  } else if (TYPE == kQ6_K) {
    const int half = c >> 2, qtr = c & 3;
    const float d = half_at(u + 208);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t lo = ld32<W>(u + half * 64 + (qtr & 1) * 32 + 16 * i + 4 * t) >> ((qtr >> 1) * 4);
      const uint32_t hi = ld32<W>(u + 128 + half * 32 + 16 * i + 4 * t) >> (2 * qtr);
      const uint32_t w = (lo & 0x0f0f0f0fu) | ((hi & 0x03030303u) << 4);
      s[i] = d * (float)(int8_t)u[192 + half * 8 + qtr * 2 + i];
      a[2 * i] = u7_bf16(b01(w), 0x43204320u);
      a[2 * i + 1] = u7_bf16(b23(w), 0x43204320u);
    }
  } else if (TYPE == kQ2_K) {
    const int half = (c >> 2) & 1, sft = (c & 3) * 2;
    const float d = half_at(u + 80), dmin = half_at(u + 82);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t sc = u[half * 8 + (c & 3) * 2 + i];
      s[i] = d * u2f(sc & 15);
      m[i] = dmin * u2f(sc >> 4);
      const uint32_t w = (ld32<W>(u + 16 + half * 32 + 16 * i + 4 * t) >> sft) & 0x03030303u;
      a[2 * i] = u7_bf16(b01(w), 0x43004300u);
      a[2 * i + 1] = u7_bf16(b23(w), 0x43004300u);
    }
  } else if (TYPE == kQ3_K) {
    const int half = (c >> 2) & 1, j4 = c & 3, sft = j4 * 2, bit = half * 4 + j4;
    const float d = half_at(u + 108);
    const uint8_t* s12 = u + 96;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = half * 8 + j4 * 2 + i;
      const uint32_t lo = k < 8 ? (s12[k] & 15) : (s12[k - 8] >> 4);
      const uint32_t hi = (s12[8 + (k & 3)] >> (2 * (k >> 2))) & 3;
      s[i] = d * (u2f(lo | (hi << 4)) - 32.f);
      const uint32_t w = ((ld32<W>(u + 32 + half * 32 + 16 * i + 4 * t) >> sft) & 0x03030303u) |
                         (((ld32<W>(u + 16 * i + 4 * t) >> bit) & 0x01010101u) << 2);
      a[2 * i] = u7_bf16(b01(w), 0x43044304u);
      a[2 * i + 1] = u7_bf16(b23(w), 0x43044304u);
    }
  } else {                                              // IQ2 / IQ3: grid bytes (below 128) with signs
    const int v = t >> 1;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int l = 2 * i + v;                          // vector of 8 weights that holds this lane's four
      uint32_t g, sg;                                   // four grid bytes, sign bits
      if (TYPE == kIQ2_XXS) {
        const uint8_t* q = u + 2 + c * 8;
        const uint32_t aux = ld32<W>(q + 4);
        s[0] = half_at(u) * (0.5f + u2f(aux >> 28)) * 0.25f;
        g = reinterpret_cast<const uint32_t*>(tab)[q[l] * 2 + (t & 1)];
        sg = tab[Fmt<TYPE>::kTable + ((aux >> (7 * l)) & 127)];
      } else if (TYPE == kIQ2_XS) {
        const uint32_t w = ld16(u + 2 + c * 8 + 2 * l);
        const uint32_t sc = u[66 + c];
        s[i] = half_at(u) * (0.5f + u2f(i ? sc >> 4 : sc & 15)) * 0.25f;
        g = reinterpret_cast<const uint32_t*>(tab)[(w & 511) * 2 + (t & 1)];
        sg = tab[Fmt<TYPE>::kTable + (w >> 9)];
      } else if (TYPE == kIQ2_S) {
        const uint32_t qh = u[66 + c], sc = u[74 + c];
        s[i] = half_at(u) * (0.5f + u2f(i ? sc >> 4 : sc & 15)) * 0.25f;
        g = reinterpret_cast<const uint32_t*>(tab)[(u[2 + c * 4 + l] | ((qh << (8 - 2 * l)) & 0x300)) * 2 + (t & 1)];
        sg = u[34 + c * 4 + l];
      } else if (TYPE == kIQ3_XXS) {
        const uint32_t aux = ld32<W>(u + 66 + c * 4);
        s[0] = half_at(u) * (0.5f + u2f(aux >> 28)) * 0.5f;
        g = reinterpret_cast<const uint32_t*>(tab)[u[2 + c * 8 + 4 * i + t]];
        sg = tab[Fmt<TYPE>::kTable + ((aux >> (7 * l)) & 127)];
      } else {                                          // IQ3_S
        const uint32_t qh = u[66 + c];
        const uint32_t nib = (u[106 + (c >> 1)] >> (4 * (c & 1))) & 15;
        s[0] = half_at(u) * u2f(1 + 2 * nib);
        g = reinterpret_cast<const uint32_t*>(tab)[u[2 + c * 8 + 4 * i + t] | ((qh << (8 - 4 * i - t)) & 256)];
        sg = u[74 + c * 4 + l];
      }
      a[2 * i] = u7_bf16(b01(g), 0x43004300u);
      a[2 * i + 1] = u7_bf16(b23(g), 0x43004300u);
      flip4(sg >> (4 * (t & 1)), a + 2 * i);
    }
  }
}

// IQ1: lane t takes weights 8 t .. 8 t + 7 of chunk c, one vector. vec8_codes: its selector word; `lut` = scale s (bits 0..2) and sign of the
// shift (bit 3) of the vector. vec8_scale: the block's scale, w = d * (2 s + 1) * (value +- 1/8).
template <int TYPE>
VE_DEVINL uint32_t vec8_codes(const uint8_t* u, int c, int t, const uint8_t* tab, uint32_t& lut) {
  uint32_t idx;
  if (TYPE == kIQ1_M) {
    const uint32_t h = (uint32_t)u[32 + 2 * c + (t >> 1)] >> (4 * (t & 1));
    const uint32_t sw = ld32<Fmt<TYPE>::kWords>(u + (c < 4 ? 48 : 52)) >> (3 * (t >> 1));
    lut = ((sw >> (16 * ((c >> 1) & 1) + 6 * (c & 1))) & 7) | (h & 8);
    idx = u[c * 4 + t] | ((h & 7) << 8);
  } else {
    const uint32_t qh = ld16(u + 34 + 2 * c);
    lut = ((qh >> 12) & 15);
    idx = u[2 + c * 4 + t] | (((qh >> (3 * t)) & 7) << 8);
  }
  return reinterpret_cast<const uint32_t*>(tab)[idx];
}
template <int TYPE>
VE_DEVINL float vec8_scale(const uint8_t* u) {
  if (TYPE == kIQ1_S) return half_at(u);
  const uint32_t s01 = ld32<Fmt<TYPE>::kWords>(u + 48), s23 = ld32<Fmt<TYPE>::kWords>(u + 52);
  return __half2float(__ushort_as_half((unsigned short)(((s01 >> 12) & 0xf) | ((s01 >> 24) & 0xf0) | ((s23 >> 4) & 0xf00) | ((s23 >> 16) & 0xf000))));
}
// Eight selectors -> four bf16 pairs, from the low and the high bytes of the three values.
VE_DEVINL void vec8_expand(uint32_t codes, uint32_t lo, uint32_t hi, uint32_t* a) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t l = __byte_perm(lo, 0u, codes >> (16 * i)), h = __byte_perm(hi, 0u, codes >> (16 * i));
    a[2 * i] = __byte_perm(l, h, 0x5140);
    a[2 * i + 1] = __byte_perm(l, h, 0x7362);
  }
}

}  // namespace ve

// CALL(type) for the block type of a launch
#define VE_GGUF_TYPES(ggml_type, CALL)      \
  switch (ggml_type) {                      \
    case kQ8_0: return CALL(kQ8_0);         \
    case kQ4_0: return CALL(kQ4_0);         \
    case kQ4_K: return CALL(kQ4_K);         \
    case kQ6_K: return CALL(kQ6_K);         \
    case kQ4_1: return CALL(kQ4_1);         \
    case kQ5_0: return CALL(kQ5_0);         \
    case kQ5_1: return CALL(kQ5_1);         \
    case kQ2_K: return CALL(kQ2_K);         \
    case kQ3_K: return CALL(kQ3_K);         \
    case kQ5_K: return CALL(kQ5_K);         \
    case kIQ4_NL: return CALL(kIQ4_NL);     \
    case kIQ4_XS: return CALL(kIQ4_XS);     \
    case kIQ2_XXS: return CALL(kIQ2_XXS);   \
    case kIQ2_XS: return CALL(kIQ2_XS);     \
    case kIQ2_S: return CALL(kIQ2_S);       \
    case kIQ3_XXS: return CALL(kIQ3_XXS);   \
    case kIQ3_S: return CALL(kIQ3_S);       \
    case kIQ1_S: return CALL(kIQ1_S);       \
    case kIQ1_M: return CALL(kIQ1_M);       \
    default: return cudaErrorInvalidValue;  \
  }

namespace ve {
// false: a codebook format whose grid table has not been set on the current device (gguf_gemv.cu)
bool iq_grids_ready(int ggml_type);
int set_iq_grids_gemm(const void* table);                   // gemm_blocks.cu
}  // namespace ve
