// EXL3 tiles on the device: the eight 16-bit windows of a lane and their codebook values. A 16 x 16 tile is a cyclic stream of
// 256 * bits bits; lane `lane` of a warp holds the values k = 2t + (i&1) + 8*((i>>1)&1), n = g + 8*(i>>2) (g = lane>>2, t = lane&3).
#pragma once
#include "common.cuh"
#include <cuda_fp16.h>

namespace ve {

// Two windows -> packed half2 bits of the two decoded values (low half = first window).
template <int CB>
VE_DEVINL uint32_t exl3_decode2(uint32_t w0, uint32_t w1) {
  if (CB == 2) {
    const uint32_t h0 = __dp4a(w0 * 0x83DCD12Du, 0x01010101u, 0x6400u);   // fp16 bits of 1024 + s
    const uint32_t h1 = __dp4a(w1 * 0x83DCD12Du, 0x01010101u, 0x6400u);
    const uint32_t pk = __byte_perm(h0, h1, 0x5410);                       // low halves of h0, h1 (their high halves are 0)
    const __half2 a = __half2half2(__ushort_as_half((unsigned short)0x1eee));
    const __half2 b = __half2half2(__ushort_as_half((unsigned short)0xc931));
    const __half2 v = __hfma2(*reinterpret_cast<const __half2*>(&pk), a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    uint32_t x0, x1;
    if (CB == 0) { x0 = w0 * 89226354u + 64248484u; x1 = w1 * 89226354u + 64248484u; }
    else { x0 = w0 * 0xCBAC1FEDu; x1 = w1 * 0xCBAC1FEDu; }
    x0 = (x0 & 0x8fff8fffu) ^ 0x3b603b60u;
    x1 = (x1 & 0x8fff8fffu) ^ 0x3b603b60u;
    const uint32_t lo = __byte_perm(x0, x1, 0x5410), hi = __byte_perm(x0, x1, 0x7632);
    const __half2 v = __hadd2(*reinterpret_cast<const __half2*>(&lo), *reinterpret_cast<const __half2*>(&hi));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

// Words a lane needs from its tile and the bit offset of its first window inside them.
template <int BITS> struct Exl3Lane {
  static constexpr int NW = BITS <= 4 ? 2 : 3;
  int w0, off;
  VE_DEVINL explicit Exl3Lane(int lane) {
    const int total = 256 * BITS;
    const int s0 = (8 * lane * BITS + BITS - 16 + total) % total;
    w0 = s0 >> 5; off = s0 & 31;
  }
  VE_DEVINL void load(const uint32_t* __restrict__ tile, uint32_t* w) const {
#pragma unroll
    for (int j = 0; j < NW; ++j) { int idx = w0 + j; if (idx >= 8 * BITS) idx -= 8 * BITS; w[j] = __ldg(tile + idx); }
  }
  VE_DEVINL void load_shared(const uint32_t* tile, uint32_t* w) const {
#pragma unroll
    for (int j = 0; j < NW; ++j) { int idx = w0 + j; if (idx >= 8 * BITS) idx -= 8 * BITS; w[j] = tile[idx]; }
  }
  // The lane's 8 windows -> four packed half2 (B fragments b0,b1 of column block 0, then of block 1).
  template <int CB> VE_DEVINL void decode(const uint32_t* w, uint32_t* frag) const {
    uint32_t q[3];
    q[0] = __funnelshift_l(w[1], w[0], off);
    q[1] = __funnelshift_l(NW > 2 ? w[2] : 0u, w[1], off);
    q[2] = NW > 2 ? (w[2] << off) : 0u;
    uint32_t win[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = i * BITS, j = t >> 5, sh = t & 31;          // window i = bits [sh, sh + 16) below the top of q[j] : q[j + 1]
      if (sh <= 16) {
        win[i] = (q[j] >> (16 - sh)) & 0xffffu;                 // inside one word: a single bit-field extract
      } else {
        win[i] = __funnelshift_r(q[j + 1 > 2 ? 2 : j + 1], q[j], 48 - sh) & 0xffffu;
      }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) frag[p] = exl3_decode2<CB>(win[2 * p], win[2 * p + 1]);
  }
};

}  // namespace ve
