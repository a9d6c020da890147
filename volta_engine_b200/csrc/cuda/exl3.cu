// EXL3 (trellis-coded) weights: fused decode + mat-vec for decode / verify rows, 128-point Hadamard rotation,
// and a reconstruct-to-bf16 kernel that feeds the tcgen05 GEMM for prefill chunks.
//
// Format: codes uint16 [K/16, N/16, 16*bits]; one 16x16 tile is a cyclic stream of 256*bits bits (uint16 pairs
// = little-endian words, MSB first); position p = 8*lane + i owns the 16-bit window that starts at bit
// p*bits + bits - 16. In that order lane `lane` of a warp holds exactly the two B fragments of
// mma.m16n8k16 for the tile (k = 2t + (i&1) + 8*((i>>1)&1), n = g + 8*(i>>2), g = lane>>2, t = lane&3), so the
// decoded fp16 pairs go to the tensor core without any shuffle; the activations (<= 16 rows, fp16, already
// rotated) are the A operand, read through L1. A CTA's 8 warps split K
// in a fixed order, and the cross-warp sum is a fixed tree: results do not depend on M or on the grid.
// Codebooks: 2 = MUL1 (x = w*0x83DCD12D, byte sum s, value = fma(1024+s, h(0x1eee), h(0xc931)) in fp16),
// 0 = 3INST (x = w*89226354+64248484), 1 = MCG (x = w*0xCBAC1FED), both y = (x & 0x8fff8fff) ^ 0x3b603b60,
// value = lo half + hi half.
// Reference counterparts: src/kernels/slang/ref_trellis.slang:1-130 (format statement),
// src/kernels/cuda/trellis/ (decode GEMV / GEMM), src/backend/cpu/linear_trellis.cpp:129-239.
#include "exl3_blocks.cuh"

namespace ve {

VE_DEVINL void mma_f16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kExl3Warps = 8;

// Few groups (a dense matrix, the routes of a few rows): see exl3_gemv_launch.
// x: fp16 [groups][M][K] rotated activations (read through L1: at most 16 x K halves, re-used by every warp);
// y: fp32 [groups][M][N]; group = blockIdx.y, its weights start at codes + expert[group] * expert_stride
// (expert == nullptr: one shared matrix). The column tiles of a group are split evenly over gridDim.x CTAs (the host
// sizes the grid to the number of CTAs that are resident at once, so every CTA gets the same work to within one tile
// and there is no partial last wave); a CTA walks its range in units of 4, 2 or 1 adjacent column tiles. In a unit every
// warp walks its share of K and reads NTW * 32 * BITS contiguous bytes per k-tile.
template <int BITS, int CB, int MH, int NTW>   // MH: 8 or 16 activation rows held by the A fragment
VE_DEVINL void exl3_gemv_unit(const uint32_t* __restrict__ base, size_t tstride, const __half* __restrict__ xlo,
                              const __half* __restrict__ xhi, bool row_lo, bool row_hi, float* __restrict__ y, float* red,
                              int M, int KT, int N, int nt0) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int per = (KT + kExl3Warps - 1) / kExl3Warps;
  const int kt0 = warp * per, kt1 = min(KT, kt0 + per);
  const Exl3Lane<BITS> L(lane);
  constexpr int NW = Exl3Lane<BITS>::NW;
  base += (size_t)nt0 * (8 * BITS);
  float acc[NTW][2][4];
#pragma unroll
  for (int j = 0; j < NTW; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][h][i] = 0.f;
  constexpr int UK = (NW == 2 ? 4 : 2) / NTW > 0 ? (NW == 2 ? 4 : 2) / NTW : 1;   // k-tiles per step of a warp
  // Two register buffers: the words of step i + 1 are requested before step i is decoded, so a warp's memory latency
  // overlaps its own arithmetic (the warps of a CTA run in lock-step and would otherwise all wait at the same time).
  uint32_t wn[UK][NTW][NW], an[UK][4];
  auto fetch = [&](int kt) {
#pragma unroll
    for (int u = 0; u < UK; ++u) {
      const int k = min(kt + u, kt1 - 1);                           // tail: re-read the last tile, its math is skipped
#pragma unroll
      for (int j = 0; j < NTW; ++j) L.load(base + (size_t)k * tstride + j * (8 * BITS), wn[u][j]);
      const int ko = k * 16;                                        // the A fragment of the same k-tile (L1 resident)
      an[u][0] = row_lo ? __ldg(reinterpret_cast<const uint32_t*>(xlo + ko)) : 0u;
      an[u][2] = row_lo ? __ldg(reinterpret_cast<const uint32_t*>(xlo + ko + 8)) : 0u;
      an[u][1] = row_hi ? __ldg(reinterpret_cast<const uint32_t*>(xhi + ko)) : 0u;
      an[u][3] = row_hi ? __ldg(reinterpret_cast<const uint32_t*>(xhi + ko + 8)) : 0u;
    }
  };
  if (kt0 < kt1) fetch(kt0);
  for (int kt = kt0; kt < kt1; kt += UK) {
    uint32_t w[UK][NTW][NW], a[UK][4];
#pragma unroll
    for (int u = 0; u < UK; ++u) {
#pragma unroll
      for (int j = 0; j < NTW; ++j)
#pragma unroll
        for (int i = 0; i < NW; ++i) w[u][j][i] = wn[u][j][i];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[u][i] = an[u][i];
    }
    if (kt + UK < kt1) fetch(kt + UK);
#pragma unroll
    for (int u = 0; u < UK; ++u) {
      if (kt + u < kt1) {
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
          uint32_t f[4];
          L.template decode<CB>(w[u][j], f);
          mma_f16(acc[j][0], a[u], f[0], f[1]);
          mma_f16(acc[j][1], a[u], f[2], f[3]);
        }
      }
    }
  }
  // C fragment: c[0],c[1] -> row g, cols 2t,2t+1; c[2],c[3] -> row g+8.
  constexpr int W = 16 * NTW;
  __syncthreads();                                                  // the previous unit's sums have been read
  float* r = red + warp * 16 * W;
#pragma unroll
  for (int j = 0; j < NTW; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = j * 16 + h * 8 + 2 * t;
      r[g * W + c] = acc[j][h][0]; r[g * W + c + 1] = acc[j][h][1];
      r[(g + 8) * W + c] = acc[j][h][2]; r[(g + 8) * W + c + 1] = acc[j][h][3];
    }
  __syncthreads();
  for (int i = tid; i < M * W; i += blockDim.x) {
    const int m = i / W, n = i % W;
    float s = 0.f;
#pragma unroll
    for (int wv = 0; wv < kExl3Warps; ++wv) s += red[wv * 16 * W + m * W + n];
    y[(size_t)m * N + nt0 * 16 + n] = s;
  }
}

template <int BITS, int CB, int MH>
__global__ void __launch_bounds__(kExl3Warps * 32, 2)
exl3_gemv_few_kernel(const uint16_t* __restrict__ codes, const __half* __restrict__ x, float* __restrict__ y,
                 int M, int K, int N, const int* __restrict__ expert, long expert_stride) {
  __shared__ float red[kExl3Warps * 256 * 4];                       // [warps][16 rows][16 * NTW cols], NTW <= 4
  const int grp = blockIdx.y;
  if (expert) { const int e = expert[grp]; if (e < 0) return; codes += (size_t)e * expert_stride; }
  x += (size_t)grp * M * K; y += (size_t)grp * M * N;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bool row_lo = g < M, row_hi = MH == 16 && g + 8 < M;
  const __half* xlo = x + (size_t)(row_lo ? g : 0) * K + 2 * t;
  const __half* xhi = x + (size_t)(row_hi ? g + 8 : 0) * K + 2 * t;
  const int KT = K >> 4, NT = N >> 4;
  const uint32_t* base = reinterpret_cast<const uint32_t*>(codes);
  const size_t tstride = (size_t)NT * (8 * BITS);
  int nt = (int)((long)NT * blockIdx.x / gridDim.x);
  const int nt_end = (int)((long)NT * (blockIdx.x + 1) / gridDim.x);
  while (nt < nt_end) {
    const int left = nt_end - nt;
    if (left >= 4) { exl3_gemv_unit<BITS, CB, MH, 4>(base, tstride, xlo, xhi, row_lo, row_hi, y, red, M, KT, N, nt); nt += 4; }
    else if (left >= 2) { exl3_gemv_unit<BITS, CB, MH, 2>(base, tstride, xlo, xhi, row_lo, row_hi, y, red, M, KT, N, nt); nt += 2; }
    else { exl3_gemv_unit<BITS, CB, MH, 1>(base, tstride, xlo, xhi, row_lo, row_hi, y, red, M, KT, N, nt); nt += 1; }
  }
}

// Many groups. x: fp16 [groups][M][K] rotated activations (read through L1: at most 16 x K halves, re-used by every warp);
// y: fp32 [groups][M][N]; the weights of a group start at codes + expert[group] * expert_stride (expert == nullptr: one shared matrix; a
// negative expert: nothing is written).
//
// A unit is UT = 4, 2 or 1 adjacent column tiles of one group, as wide as still gives every block two units; the units of all groups are
// split evenly over the blocks that are resident at once, so every block gets the same work to within one unit whatever the number of
// groups is. In a unit the eight warps split K, and each brings its k-tiles, 4 / UT at a time, through a cp.async ring of its own that runs
// several stages ahead and on into the next unit. One k-tile ahead in registers (and a grid of groups x columns) a unit cost sixteen memory
// latencies in a row: 108 us for 160 routes of 2048 x 512 weights at 4 bits, now 70 us; their bytes take 13 us. What bounds it now is
// issuing: 8.7 instructions a weight, 72 % of the issue slots of 16 warps an SM.
template <int BITS, int MH>
struct Exl3Gemv {
  static constexpr int kStage = 4 * 32 * BITS, kStages = BITS <= 4 ? 8 : 4;      // bytes of four tiles; stages of the ring
  static constexpr int kRed = kExl3Warps * MH * 64;                               // floats, one of two buffers (units of four tiles)
  static constexpr int kSmem = 2 * kRed * 4 + kExl3Warps * kStages * kStage;
};

template <int BITS, int CB, int MH, int UT>   // MH: 8 or 16 activation rows held by the A fragment
__global__ void __launch_bounds__(kExl3Warps * 32, 2)
exl3_gemv_kernel(const uint16_t* __restrict__ codes, const __half* __restrict__ x, float* __restrict__ y,
                 int M, int K, int N, const int* __restrict__ expert, long expert_stride, int groups) {
  using C = Exl3Gemv<BITS, MH>;
  constexpr int KU = 4 / UT, W = 16 * UT;                           // k-tiles of a stage, columns of a unit
  extern __shared__ __align__(16) uint8_t exl3_smem[];
  float* const red = reinterpret_cast<float*>(exl3_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  uint8_t* const ring = exl3_smem + 2 * C::kRed * 4 + warp * C::kStages * C::kStage;
  const bool row_lo = g < M, row_hi = MH == 16 && g + 8 < M;
  const int KT = K >> 4, NT = N >> 4, per_group = (NT + UT - 1) / UT;
  const long total = (long)groups * per_group;
  const int u0 = (int)(total * blockIdx.x / gridDim.x), u1 = (int)(total * (blockIdx.x + 1) / gridDim.x);
  const int per = (KT + kExl3Warps - 1) / kExl3Warps;
  const int kt0 = min(KT, warp * per), kt1 = min(KT, kt0 + per);
  const size_t tstride = (size_t)NT * (32 * BITS);                  // bytes from one k-tile to the next

  int l_unit = u0, l_kt = kt0, l_slot = 0, l_live = 0;             // what is loaded next
  const uint8_t* l_base = nullptr;
  auto load = [&]() {
    if (l_unit < u1 && kt0 < kt1) {
      if (l_kt == kt0) {
        const int grp = l_unit / per_group, nt0 = (l_unit - grp * per_group) * UT;
        const int e = expert ? expert[grp] : 0;
        l_live = e < 0 ? 0 : min(UT, NT - nt0) * 2 * BITS;          // 16-byte pieces of a k-tile
        l_base = reinterpret_cast<const uint8_t*>(codes + (size_t)max(e, 0) * expert_stride) + (size_t)nt0 * (32 * BITS);
      }
      const uint8_t* src = l_base + (size_t)l_kt * tstride;
      uint8_t* dst = ring + l_slot * C::kStage;
      constexpr int P = 2 * BITS * UT;
      if (!((uintptr_t)src & 15)) {
#pragma unroll
        for (int i = 0; i < (8 * BITS + 31) / 32; ++i) {
          const int j = lane + 32 * i, ku = j / P, piece = j % P;
          if (ku < KU && piece < l_live && l_kt + ku < kt1)
            cp_async16(dst + j * 16, src + ku * tstride + piece * 16);
        }
      } else {                                                       // codes that start between 16-byte boundaries: word by word
        for (int j = lane; j < 4 * 8 * BITS; j += 32) {
          const int ku = j / (4 * P), word = j % (4 * P);
          if (word < 4 * l_live && l_kt + ku < kt1)
            cp_async4(dst + j * 4, src + ku * tstride + word * 4);
        }
      }
      l_slot = l_slot + 1 == C::kStages ? 0 : l_slot + 1;
      l_kt += KU;
      if (l_kt >= kt1) { l_kt = kt0; ++l_unit; }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < C::kStages - 1; ++i) load();

  const Exl3Lane<BITS> L(lane);
  constexpr int NW = Exl3Lane<BITS>::NW;
  int slot = 0, buf = 0;
  for (int unit = u0; unit < u1; ++unit) {
    const int grp = unit / per_group, nt0 = (unit - grp * per_group) * UT;
    const bool here = !expert || expert[grp] >= 0;
    const __half* xlo = x + ((size_t)grp * M + (row_lo ? g : 0)) * K + 2 * t;
    const __half* xhi = x + ((size_t)grp * M + (row_hi ? g + 8 : 0)) * K + 2 * t;
    float acc[UT][2][4];
#pragma unroll
    for (int j = 0; j < UT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][h][i] = 0.f;
    uint32_t an[KU][4];
    auto fetch = [&](int kt) {                                      // the A fragments of a stage, one ahead
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        const int ko = min(kt + u, kt1 - 1) * 16;
        an[u][0] = row_lo ? __ldg(reinterpret_cast<const uint32_t*>(xlo + ko)) : 0u;
        an[u][2] = row_lo ? __ldg(reinterpret_cast<const uint32_t*>(xlo + ko + 8)) : 0u;
        an[u][1] = row_hi ? __ldg(reinterpret_cast<const uint32_t*>(xhi + ko)) : 0u;
        an[u][3] = row_hi ? __ldg(reinterpret_cast<const uint32_t*>(xhi + ko + 8)) : 0u;
      }
    };
    if (kt0 < kt1 && here) fetch(kt0);
    for (int kt = kt0; kt < kt1; kt += KU) {
      asm volatile("cp.async.wait_group %0;" ::"n"(C::kStages - 2) : "memory");
      __syncwarp();                                                  // the stage is here for every lane, the slot in front of it is free
      load();
      const uint32_t* st = reinterpret_cast<const uint32_t*>(ring + slot * C::kStage);
      slot = slot + 1 == C::kStages ? 0 : slot + 1;
      if (!here) continue;
      uint32_t a[KU][4];
#pragma unroll
      for (int u = 0; u < KU; ++u)
#pragma unroll
        for (int i = 0; i < 4; ++i) a[u][i] = an[u][i];
      if (kt + KU < kt1) fetch(kt + KU);
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        if (kt + u >= kt1) break;
#pragma unroll
        for (int j = 0; j < UT; ++j) {                               // (tiles behind the matrix: old bytes of the ring, not stored)
          uint32_t w[NW], f[4];
          L.load_shared(st + (u * UT + j) * (8 * BITS), w);
          L.template decode<CB>(w, f);
          mma_f16(acc[j][0], a[u], f[0], f[1]);
          mma_f16(acc[j][1], a[u], f[2], f[3]);
        }
      }
    }
    if (!here) continue;                                             // (the same answer in every warp of the block)
    // C fragment: c[0],c[1] -> row g, cols 2t,2t+1; c[2],c[3] -> row g+8. Warp sums are added in warp order.
    float* rb = red + buf * C::kRed;                                 // (sums of the unit in front were read, or are, from the other)
    buf ^= 1;
    float* r = rb + warp * MH * W;
#pragma unroll
    for (int j = 0; j < UT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = j * 16 + h * 8 + 2 * t;
        *reinterpret_cast<float2*>(r + g * W + c) = make_float2(acc[j][h][0], acc[j][h][1]);
        if (MH == 16) *reinterpret_cast<float2*>(r + (g + 8) * W + c) = make_float2(acc[j][h][2], acc[j][h][3]);
      }
    __syncthreads();
    for (int i = tid; i < M * W; i += kExl3Warps * 32) {
      const int m = i / W, n = i % W;
      if (nt0 * 16 + n >= N) continue;
      float s = 0.f;
#pragma unroll
      for (int wv = 0; wv < kExl3Warps; ++wv) s += rb[wv * MH * W + m * W + n];
      y[((size_t)grp * M + m) * N + nt0 * 16 + n] = s;
    }
  }
}

// ------------------------------------------------------------------------------------------------ Hadamard
// dtype codes: 0 bf16, 1 fp32, 2 fp16.
template <int DT> VE_DEVINL void had_load4(const void* p, size_t i, float* v) {
  if (DT == 1) { const float4 f = *reinterpret_cast<const float4*>((const float*)p + i); v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; }
  else if (DT == 0) {
    const uint2 u = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)p + i);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>((const __half*)p + i);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}
template <int DT> VE_DEVINL void had_store4(void* p, size_t i, const float* v) {
  if (DT == 1) *reinterpret_cast<float4*>((float*)p + i) = make_float4(v[0], v[1], v[2], v[3]);
  else if (DT == 0) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    uint2 u; u.x = *reinterpret_cast<uint32_t*>(&a); u.y = *reinterpret_cast<uint32_t*>(&b);
    *reinterpret_cast<uint2*>((__nv_bfloat16*)p + i) = u;
  } else {
    __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    uint2 u; u.x = *reinterpret_cast<uint32_t*>(&a); u.y = *reinterpret_cast<uint32_t*>(&b);
    *reinterpret_cast<uint2*>((__half*)p + i) = u;
  }
}

// 16 consecutive values; vec: the address is 16-byte aligned (else 8 bytes, fp32 16).
template <int DT> VE_DEVINL void had_load16(const void* p, size_t i, bool vec, float* v) {
  if (DT == 1 || !vec) {
#pragma unroll
    for (int j = 0; j < 16; j += 4) had_load4<DT>(p, i + j, v + j);
  } else {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p) + i);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 u = src[h];
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = DT == 0 ? __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]))
                                 : __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
        v[h * 8 + 2 * j] = f.x; v[h * 8 + 2 * j + 1] = f.y;
      }
    }
  }
}
template <int DT> VE_DEVINL void had_store16(void* p, size_t i, bool vec, const float* v) {
  if (DT == 1 || !vec) {
#pragma unroll
    for (int j = 0; j < 16; j += 4) had_store4<DT>(p, i + j, v + j);
  } else {
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(p) + i);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (DT == 0) { const __nv_bfloat162 r = __floats2bfloat162_rn(v[h * 8 + 2 * j], v[h * 8 + 2 * j + 1]); w[j] = *reinterpret_cast<const uint32_t*>(&r); }
        else { const __half2 r = __floats2half2_rn(v[h * 8 + 2 * j], v[h * 8 + 2 * j + 1]); w[j] = *reinterpret_cast<const uint32_t*>(&r); }
      }
      dst[h] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

template <int DT, int V> VE_DEVINL void had_load(const void* p, size_t i, bool vec, float* v) {
  if (V == 16) had_load16<DT>(p, i, vec, v);
  else had_load4<DT>(p, i, v);
}
template <int DT, int V> VE_DEVINL void had_store(void* p, size_t i, bool vec, const float* v) {
  if (V == 16) had_store16<DT>(p, i, vec, v);
  else had_store4<DT>(p, i, v);
}

// 128-point Walsh-Hadamard transform (natural order, scaled by 1/sqrt(128)) over 128 / V lanes of V consecutive values each: strides
// below V inside the lane, the others by shuffles, in rising order.
template <int V>
VE_DEVINL void wht128(float* v, int lane) {
#pragma unroll
  for (int m = 1; m < V; m <<= 1)
#pragma unroll
    for (int j = 0; j < V; ++j)
      if (!(j & m)) {
        const float a = v[j], b = v[j | m];
        v[j] = a + b;
        v[j | m] = a - b;
      }
#pragma unroll
  for (int m = 1; m < 128 / V; m <<= 1) {
    const bool up = lane & m;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float o = __shfl_xor_sync(0xffffffffu, v[j], m);
      v[j] = up ? o - v[j] : v[j] + o;
    }
  }
  const float s = 0.08838834764831845f;
#pragma unroll
  for (int j = 0; j < V; ++j) v[j] *= s;
}

struct HadArgs {
  const void* in; const void* in2; void* out;
  const __half* scale; const __half* scale2;
  const int* expert; long scale_stride;
  const int* src;                // null: input row = row / in_div; else src[row] / in_div
  int rows, C, post, in_div, rows_per_group, act;
  bool vec;                      // every row of 16-bit values starts on a 16-byte boundary
};

VE_DEVINL float act_apply(float x, int act) {
  if (act == 1) { const float t = tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)); return 0.5f * x * (1.f + t); }
  return x / (1.f + __expf(-x));
}

// 128 / V lanes per 128-block. post == 0: out = had(in * scale); post == 1: out = had(in) * scale; with in2:
// out = act(had(in) * scale) * (had(in2) * scale2).
// Many rows are bound by what is read and written, and by the shuffles: four values a lane take 20 a block, 16 values 12, for the same sums in
// the same order (2000 rows of 2048 columns 9.1 to 6.9 us, of 5120 18.6 to 13.8 us). A few rows are bound by latency, which four values a
// lane keep shorter (1 to 16 rows of 2048 columns 1.9 us against 2.5 us, 160 rows 2.5 against 2.9 us).
template <int DI, int DO, int V>
__global__ void __launch_bounds__(256) had128_kernel(HadArgs a) {
  const int lane = threadIdx.x & 31;
  const int nb = a.C >> 7;
  const long total = (long)a.rows * nb;
  constexpr int LANES = 128 / V, PER = 32 / LANES;          // of a block; blocks of a warp
  for (long b0 = ((long)blockIdx.x * 8 + (threadIdx.x >> 5)) * PER; b0 < total; b0 += (long)gridDim.x * 8 * PER) {
    const long blk = b0 + lane / LANES;
    const bool in = blk < total;                          // (every lane takes part in the shuffles)
    const int row = in ? (int)(blk / nb) : 0, cb = in ? (int)(blk % nb) : 0;
    const int col = cb * 128 + (lane % LANES) * V;
    long soff = col;
    int e = 0;
    if (a.expert) {
      e = a.expert[row / a.rows_per_group];
      if (e > 0) soff += (long)e * a.scale_stride;
    }
    const bool live = in && e >= 0;
    float s[V], v[V];
#pragma unroll
    for (int j = 0; j < V; ++j) { s[j] = 1.f; v[j] = 0.f; }
    size_t in_row = 0;
    if (live) {
      in_row = (size_t)((a.src ? a.src[row] : row) / a.in_div) * a.C;
      if (a.scale) had_load<2, V>(a.scale, soff, a.vec, s);
      had_load<DI, V>(a.in, in_row + col, a.vec, v);
    }
    if (!a.post) {
#pragma unroll
      for (int j = 0; j < V; ++j) v[j] *= s[j];
    }
    wht128<V>(v, lane);
    if (a.post) {
#pragma unroll
      for (int j = 0; j < V; ++j) v[j] *= s[j];
    }
    if (a.in2) {
      float u[V];
#pragma unroll
      for (int j = 0; j < V; ++j) { s[j] = 1.f; u[j] = 0.f; }
      if (live) {
        if (a.scale2) had_load<2, V>(a.scale2, soff, a.vec, s);
        had_load<DI, V>(a.in2, in_row + col, a.vec, u);
      }
      wht128<V>(u, lane);
#pragma unroll
      for (int j = 0; j < V; ++j) v[j] = act_apply(v[j], a.act) * (u[j] * s[j]);
    }
    if (in && e < 0) {                                    // another rank's route: zeros (rows behind the sorted routes stay unwritten)
#pragma unroll
      for (int j = 0; j < V; ++j) v[j] = 0.f;
    }
    if (live || (in && !a.src)) had_store<DO, V>(a.out, (size_t)row * a.C + col, a.vec, v);
  }
}

// ------------------------------------------------------------------------------------------------ reconstruct
// codes -> bf16 [N][K] (output features major, K contiguous): the A operand layout of the tcgen05 GEMM.
// batch > 1: `batch` matrices back to back (the experts of a bank) -> [batch * N][K].
template <int BITS, int CB>
__global__ void __launch_bounds__(256) exl3_reconstruct_kernel(const uint16_t* __restrict__ codes,
                                                               __nv_bfloat16* __restrict__ out, int K, int N, int batch) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int KT = K >> 4, NT = N >> 4;
  const Exl3Lane<BITS> L(lane);
  const long per = (long)KT * NT, total = per * batch;
  // consecutive warps walk kt for a fixed nt so that a CTA writes runs of 128 contiguous k per output row
  for (long gid = (long)blockIdx.x * 8 + (threadIdx.x >> 5); gid < total; gid += (long)gridDim.x * 8) {
    const long b = gid / per, id = gid % per;
    const int nt = (int)(id / KT), kt = (int)(id % KT);
    uint32_t w[3], f[4];
    L.load(reinterpret_cast<const uint32_t*>(codes) + ((size_t)b * per + (size_t)kt * NT + nt) * (8 * BITS), w);
    L.template decode<CB>(w, f);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&f[p]));
      const int n = nt * 16 + g + 8 * (p >> 1), k = kt * 16 + 2 * t + 8 * (p & 1);
      *reinterpret_cast<__nv_bfloat162*>(out + ((size_t)b * N + n) * K + k) = __floats2bfloat162_rn(v.x, v.y);
    }
  }
}

}  // namespace ve

using namespace ve;

template <int BITS, int CB, int MH, int UT>
static int exl3_gemv_blocks(int* blocks) {                           // blocks that are resident at once, found on the first call
  static int ctas = 0;
  constexpr int smem = Exl3Gemv<BITS, MH>::kSmem;
  const cudaError_t e = allow_smem<exl3_gemv_kernel<BITS, CB, MH, UT>>(smem);
  if (e != cudaSuccess) return (int)e;
  if (!ctas) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, exl3_gemv_kernel<BITS, CB, MH, UT>, kExl3Warps * 32, smem) != cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
    ctas = per_sm * 148;
  }
  *blocks = ctas;
  return 0;
}

template <int BITS, int CB, int MH>
static int exl3_gemv_run(const void* codes, const void* x, void* y, int M, int K, int N, const int* expert, long stride, int groups,
                         cudaStream_t st) {
  int n = 0, rc = exl3_gemv_blocks<BITS, CB, MH, 4>(&n);
  if (rc) return rc;
  const int NT = N / 16;
  // units of four tiles decode with the fewest loads and barriers a weight; fewer than two a block leave blocks idle in the last round
  const long four = (long)groups * ((NT + 3) / 4), two = (long)groups * ((NT + 1) / 2), one = (long)groups * NT;
#define VE_UNITS(UT, TOTAL)                                                                                                      \
  do {                                                                                                                           \
    if ((rc = exl3_gemv_blocks<BITS, CB, MH, UT>(&n))) return rc;                                                                \
    exl3_gemv_kernel<BITS, CB, MH, UT><<<(unsigned)(TOTAL < n ? TOTAL : n), kExl3Warps * 32, Exl3Gemv<BITS, MH>::kSmem, st>>>(   \
        (const uint16_t*)codes, (const __half*)x, (float*)y, M, K, N, expert, stride, groups);                                   \
  } while (0)
  if (four >= 2 * n) VE_UNITS(4, four);
  else if (two >= 2 * n) VE_UNITS(2, two);
  else VE_UNITS(1, one);
#undef VE_UNITS
  VE_CHECK_LAUNCH();
}

template <int BITS, int CB, int MH>
static int exl3_gemv_few(const void* codes, const void* x, void* y, int M, int K, int N, const int* expert, long stride, int groups,
                         cudaStream_t st) {
  static int ctas = 0;                                             // blocks that are resident at once
  if (!ctas) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, exl3_gemv_few_kernel<BITS, CB, MH>, kExl3Warps * 32, 0) != cudaSuccess || per_sm < 1)
      per_sm = 1;
    ctas = per_sm * 148;
  }
  const int gx = max(1, min(N / 16, ctas / groups));
  exl3_gemv_few_kernel<BITS, CB, MH><<<dim3(gx, groups), kExl3Warps * 32, 0, st>>>((const uint16_t*)codes, (const __half*)x, (float*)y, M, K, N,
                                                                                    expert, stride);
  VE_CHECK_LAUNCH();
}

// Both kernels add in the same order and give the same bits. A group of blocks for each group of routes has the shorter path from memory to
// the tensor core and is faster as long as the resident blocks divide among the groups: 5120 x 5120 at 4 bits 18 us (ring 22), 5120 x 34816 61 us
// (69), ten routes of 2048 x 512 7.8 us (11.0), 32 of 4096 x 1408 at 3 bits 63 us (84). With many groups most of its blocks have no second column
// tile to take or none at all: 80 routes of 4096 x 1408 195 us (166), 160 of 2048 x 512 100 us (68). At 40 routes the two are level.
constexpr int kExl3FewGroups = 48;

template <int BITS, int CB>
static int exl3_gemv_launch(const void* codes, const void* x, void* y, int M, int K, int N, const int* expert,
                            long stride, int groups, cudaStream_t st) {
  if (groups < kExl3FewGroups)
    return M <= 8 ? exl3_gemv_few<BITS, CB, 8>(codes, x, y, M, K, N, expert, stride, groups, st)
                  : exl3_gemv_few<BITS, CB, 16>(codes, x, y, M, K, N, expert, stride, groups, st);
  return M <= 8 ? exl3_gemv_run<BITS, CB, 8>(codes, x, y, M, K, N, expert, stride, groups, st)
                : exl3_gemv_run<BITS, CB, 16>(codes, x, y, M, K, N, expert, stride, groups, st);
}

extern "C" {

int ve_exl3_gemv(const void* codes, const void* x, void* y, int M, int K, int N, int bits, int cb,
                 const void* expert, long expert_stride, int groups, cudaStream_t st) {
  if (M < 1 || M > 16 || K % 16 || N % 16 || groups < 1 || cb < 0 || cb > 2) return cudaErrorInvalidValue;
#define VE_EX(B)                                                                                             \
  case B:                                                                                                    \
    return cb == 2 ? exl3_gemv_launch<B, 2>(codes, x, y, M, K, N, (const int*)expert, expert_stride, groups, st) \
         : cb == 1 ? exl3_gemv_launch<B, 1>(codes, x, y, M, K, N, (const int*)expert, expert_stride, groups, st) \
                   : exl3_gemv_launch<B, 0>(codes, x, y, M, K, N, (const int*)expert, expert_stride, groups, st);
  switch (bits) {
    VE_EX(1) VE_EX(2) VE_EX(3) VE_EX(4) VE_EX(5) VE_EX(6) VE_EX(7) VE_EX(8)
    default: return cudaErrorInvalidValue;
  }
#undef VE_EX
}

static int exl3_reconstruct_n(const void* codes, void* out, int K, int N, int bits, int cb, int batch, cudaStream_t st);

int ve_exl3_reconstruct(const void* codes, void* out, int K, int N, int bits, int cb, cudaStream_t st) {
  return exl3_reconstruct_n(codes, out, K, N, bits, cb, 1, st);
}

// `batch` matrices back to back ([batch][K/16][N/16][16 * bits]) -> bf16 [batch * N][K]: the stacked A operand of the
// grouped GEMM for a slab of routed experts.
int ve_exl3_reconstruct_batch(const void* codes, void* out, int K, int N, int bits, int cb, int batch, cudaStream_t st) {
  return exl3_reconstruct_n(codes, out, K, N, bits, cb, batch, st);
}

}  // extern "C"

static int exl3_reconstruct_n(const void* codes, void* out, int K, int N, int bits, int cb, int batch, cudaStream_t st) {
  if (K % 16 || N % 16 || cb < 0 || cb > 2 || batch < 1) return cudaErrorInvalidValue;
  const long tiles = (long)(K / 16) * (N / 16) * batch;
  const int blocks = (int)((tiles + 7) / 8 < 148 * 8 ? (tiles + 7) / 8 : 148 * 8);
#define VE_RC(B)                                                                                                           \
  case B:                                                                                                                  \
    if (cb == 2) exl3_reconstruct_kernel<B, 2><<<blocks, 256, 0, st>>>((const uint16_t*)codes, (__nv_bfloat16*)out, K, N, batch); \
    else if (cb == 1) exl3_reconstruct_kernel<B, 1><<<blocks, 256, 0, st>>>((const uint16_t*)codes, (__nv_bfloat16*)out, K, N, batch); \
    else exl3_reconstruct_kernel<B, 0><<<blocks, 256, 0, st>>>((const uint16_t*)codes, (__nv_bfloat16*)out, K, N, batch);         \
    break;
  switch (bits) {
    VE_RC(1) VE_RC(2) VE_RC(3) VE_RC(4) VE_RC(5) VE_RC(6) VE_RC(7) VE_RC(8)
    default: return cudaErrorInvalidValue;
  }
#undef VE_RC
  VE_CHECK_LAUNCH();
}

extern "C" {

// dt codes: 0 bf16, 1 fp32, 2 fp16. Supported (in -> out): bf16->fp16, fp32->bf16, fp32->fp16, fp16->fp16, bf16->bf16.
// expert: scale row of every output row (negative: zeros are written); src: input row times in_div of every output row.
int ve_had128(const void* in, const void* in2, void* out, const void* scale, const void* scale2, const void* expert,
              const void* src, long scale_stride, int rows, int C, int post, int in_div, int rows_per_group, int act, int dt_in,
              int dt_out, cudaStream_t st) {
  if (rows < 1 || C % 128 || in_div < 1 || rows_per_group < 1) return cudaErrorInvalidValue;
  HadArgs a{in, in2, out, (const __half*)scale, (const __half*)scale2, (const int*)expert, scale_stride,
            (const int*)src, rows, C, post, in_div, rows_per_group, act};
  a.vec = !(((uintptr_t)in | (uintptr_t)in2 | (uintptr_t)out | (uintptr_t)scale | (uintptr_t)scale2) & 15) && scale_stride % 8 == 0;
  const long n = (long)rows * (C / 128);
  // 16 values a lane once they still give every SM 32 blocks of 128 (at 4700 the two are level)
  const int per = n < 148 * 32 ? 8 : 32;                            // blocks of 128 a thread block
  const int blocks = (int)((n + per - 1) / per < 148 * 8 ? (n + per - 1) / per : 148 * 8);
#define VE_HAD(DI, DO)                                                         \
  do {                                                                          \
    if (per == 8) had128_kernel<DI, DO, 4><<<blocks, 256, 0, st>>>(a);        \
    else had128_kernel<DI, DO, 16><<<blocks, 256, 0, st>>>(a);                \
  } while (0)
  if (dt_in == 0 && dt_out == 2) VE_HAD(0, 2);
  else if (dt_in == 1 && dt_out == 0) VE_HAD(1, 0);
  else if (dt_in == 1 && dt_out == 1) VE_HAD(1, 1);
  else if (dt_in == 1 && dt_out == 2) VE_HAD(1, 2);
  else if (dt_in == 2 && dt_out == 2) VE_HAD(2, 2);
  else if (dt_in == 0 && dt_out == 0) VE_HAD(0, 0);
  else return cudaErrorInvalidValue;
#undef VE_HAD
  VE_CHECK_LAUNCH();
}

}  // extern "C"
