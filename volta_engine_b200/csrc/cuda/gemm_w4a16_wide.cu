// Prefill linear with NVFP4 weights and bf16 activations, two shapes of output tile:
//   out[t, n] = alpha * sum_k W[n, k] * X[t, k],   W dequantised to bf16 inside the tile loader (exact products).
//
// The form in front of this one (256 features x 256 tokens, dequantised weights in shared memory) was bound by shared memory: per 64-wide k
// step both weight sub-tiles were written to it as bf16 (32 KB) and read back (32 KB) beside two reads of the activation tile (64 KB) and the
// loads (41 KB): 180 KB, 1400 cycles at 128 B a cycle for 1024 cycles of tensor work. Here the dequantised weights go to tensor memory, from
// where the MMA takes its A operand, and the blocks are persistent. Two shapes of tile, which differ in how they fill the last wave:
//   * two 128-feature sub-tiles x 192 tokens: accumulators of 2 x 192 columns and two buffers of 2 x 32 columns of weights fill the 512
//     columns. 92 KB of shared memory a step, 720 cycles for 768 of tensor work; measured 0.75 us a step: the dequantising, one weight row of
//     64 a thread and step, takes most of it (shorter tiles are no faster).
//   * one sub-tile x 256 tokens: half a weight row a thread and step, four buffers; 0.52 us a step for two thirds of the products (34816 x
//     5120 at 2048 tokens: tensor pipe 61 % busy, issue slots 54 %).
// The shape that needs less time for its waves of 148 tiles is taken (0.75 : 0.52 is 10 : 7). Times in us of the former kernel, of one
// sub-tile and of two: 5120 x 5120 600 tokens 84 51 61, 953 tokens 85 98 63, 2048 tokens 166 145 122; 34816 x 5120 256 tokens 90 84 125,
// 2048 tokens 699 620 657, 8192 tokens 2919 2745 2944; 5120 x 17408 150 tokens 260 164 234, 1500 tokens 262 283 378, 2048 tokens 511 381
// 379. Where 256 x 256 tiles happened to fill whole waves the former kernel was faster (16384 x 5120 at 452 tokens 90 us against 95,
// 5120 x 5120 at 3001 tokens 180 against 210).
//
// A result depends on its own row of X alone: every tile runs over K in one chain, whatever T and the shape are. (Tiles of a partial last
// wave cut along K, with fp32 partial sums, would give 5120 x 17408 116 to 140 us at 129 to 256 tokens in place of 162 to 171, but rows that
// change with the number of rows beside them.)
//
// Warp roles (320 threads): warp 0 TMA producer, warp 1 TMEM owner + MMA issuer, warps 2..9 dequantise and run the epilogue. Every wait is
// bounded.
// Reference kernel family this replaces: src/kernels/cuda/nvfp4/skinny_kernels.cu:531-558 (fused WMMA GEMM / dequant + HGEMM).
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "tmap.h"

namespace ve {

constexpr int W_KT = 64, W_RAW = 128 * 32, W_SF = 1024, W_STAGES = 5, W_GRID = 148;
constexpr int W_STORE = 32 * 528;                                   // 32 tokens of an output sub-tile at a time

// SUBS: 128-feature sub-tiles of a tile.
template <int SUBS>
struct Wide {
  static constexpr int kT = SUBS == 2 ? 192 : 256;                   // tokens of a tile at most
  static constexpr int kB = kT * 128, kStage = kB + SUBS * (W_RAW + W_SF);
  static constexpr int kSmem = W_STAGES * kStage + 2 * W_STORE + 1024;
  static constexpr int kBufs = SUBS == 2 ? 2 : 4;                    // buffers of dequantised weights, SUBS * 32 TMEM columns each
  static constexpr int kW = SUBS * kT;                               // their first column, behind the accumulators
  static_assert(kW + kBufs * SUBS * 32 <= 512 && kStage % 1024 == 0 && kSmem <= 227 * 1024, "TMEM, swizzle atoms, shared memory");
};

struct WidePlan {
  int tile_t;                     // tokens of a tile, a multiple of 16
  int tiles_t, tiles, grid;
};
template <int SUBS>
static inline WidePlan wide_plan(int T, int N) {
  WidePlan p;
  p.tiles_t = (T + Wide<SUBS>::kT - 1) / Wide<SUBS>::kT;
  p.tiles = (N + 128 * SUBS - 1) / (128 * SUBS) * p.tiles_t;
  p.tile_t = ((T + p.tiles_t - 1) / p.tiles_t + 15) / 16 * 16;          // (no taller than the tokens ask for: 452 are 3 x 160)
  p.grid = p.tiles < W_GRID ? p.tiles : W_GRID;
  return p;
}

struct WideParams {
  WidePlan plan;
  int N, T, K;
  float alpha;
  __nv_bfloat16* out;
  long ldo;
  const __nv_bfloat16* residual;
  long ldr;
  const uint8_t* sfa;     // [N/128][K/128][128][8] E4M3 scales
  int* status;
};

VE_DEVINL void w_e2m1x8_to_bf16x8(uint32_t w, uint32_t* o) {
  // table lookup on the byte-permute unit: bf16 patterns of {0, .5, 1, 1.5, 2, 3, 4, 6}
  const uint32_t mags = w & 0x77777777u, sg = (w >> 3) & 0x11111111u;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t sel = mags >> (16 * h), ssel = sg >> (16 * h);
    const uint32_t lo4 = __byte_perm(0xC0800000u, 0xC0804000u, sel);
    const uint32_t hi4 = __byte_perm(0x3F3F3F00u, 0x40404040u, sel) | __byte_perm(0x00008000u, 0u, ssel);
    o[2 * h] = __byte_perm(lo4, hi4, 0x5140);
    o[2 * h + 1] = __byte_perm(lo4, hi4, 0x7362);
  }
}
VE_DEVINL uint32_t w_e4m3_to_bf16x2_dup(uint32_t byte) {
  uint32_t r;
  asm("{ .reg .b16 t; cvt.u16.u32 t, %1; cvt.rn.f16x2.e4m3x2 %0, t; }" : "=r"(r) : "r"(byte | (byte << 8)));
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&r));
  const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&b);
}


template <int SUBS>
__global__ void __launch_bounds__(320, 1)
gemm_w4a16_wide_kernel(const WideParams p, const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap) {
  using C = Wide<SUBS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[W_STAGES], empty[W_STAGES], wfull[C::kBufs], wempty[C::kBufs], acc_full, acc_free;
  __shared__ uint32_t tmem_holder;
  __shared__ int s_fail;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < W_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < C::kBufs; ++s) { mbar_init(&wfull[s], 8); mbar_init(&wempty[s], 1); }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_free, 8);
    s_fail = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&tmem_holder, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  auto stage_ptr = [&](int s) { return smem + (size_t)s * C::kStage; };   // [B][RAW x SUBS][SF x SUBS]
  constexpr int OFF_RAW = C::kB, OFF_SF = C::kB + SUBS * W_RAW;
  const int nkt = p.K / W_KT;

  if (warp == 0) {
    if (elect_one()) {
      prefetch_tmap(&amap);
      prefetch_tmap(&bmap);
      const size_t blk = (size_t)(p.K / 128);
      int i = 0;                                   // steps so far, over all tiles
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.plan.tiles && ok; tile += p.plan.grid) {
        const int tn = tile / p.plan.tiles_t, t0 = (tile - tn * p.plan.tiles_t) * p.plan.tile_t, n0 = tn * 128 * SUBS;
        for (int kt = 0; kt < nkt; ++kt, ++i) {
          const int s = i % W_STAGES;
          ok = mbar_wait(&empty[s], ((i / W_STAGES) & 1) ^ 1);
          if (!ok) break;
          uint8_t* st = stage_ptr(s);
          mbar_expect_tx(&full[s], SUBS * (W_RAW + W_SF) + p.plan.tile_t * 128);
          tma_load_2d(st, &bmap, &full[s], kt * W_KT, t0);
#pragma unroll
          for (int sub = 0; sub < SUBS; ++sub) {
            // (a matrix of an odd number of 128-feature tiles: the second one's codes read as zero, its scales are the first one's)
            const int sf = n0 + sub * 128 < p.N ? SUBS * tn + sub : SUBS * tn;
            tma_load_2d(st + OFF_RAW + sub * W_RAW, &amap, &full[s], kt * 32, n0 + sub * 128);
            bulk_load(st + OFF_SF + sub * W_SF, p.sfa + ((size_t)sf * blk + (kt >> 1)) * 1024, W_SF, &full[s]);
          }
        }
      }
      if (!ok) atomicExch(&s_fail, 1);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_f16(1, 1, 128, p.plan.tile_t);
      int i = 0, item = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.plan.tiles && ok; tile += p.plan.grid, ++item) {
        ok = mbar_wait(&acc_free, (item & 1) ^ 1);          // the epilogue has read the tile in front
        tc_fence_after();
        for (int kt = 0; kt < nkt && ok; ++kt, ++i) {
          const int s = i % W_STAGES, w = i % C::kBufs;
          ok = mbar_wait(&full[s], (i / W_STAGES) & 1) && mbar_wait(&wfull[w], (i / C::kBufs) & 1);
          if (!ok) break;
          tc_fence_after();
          const uint64_t bd = make_desc_sw128(smem_u32(stage_ptr(s)));
#pragma unroll
          for (int sub = 0; sub < SUBS; ++sub)
#pragma unroll
            for (int kb = 0; kb < 4; ++kb)
              tc_mma_f16_ta(tmem_base + sub * C::kT, tmem_base + C::kW + (w * SUBS + sub) * 32 + kb * 8, bd + kb * 2, idesc, (kt | kb) ? 1u : 0u);
          tc_commit(&empty[s]);
          tc_commit(&wempty[w]);
        }
        tc_commit(&acc_full);
      }
      if (!ok) atomicExch(&s_fail, 1);
    }
  } else {
    const int grp = (warp - 2) >> 2, quarter = warp & 3, row = quarter * 32 + lane, etid = ((warp - 2) & 3) * 32 + lane;
    const int sub = SUBS == 2 ? grp : 0;
    constexpr int WORDS = SUBS == 2 ? 8 : 4;                  // of eight codes each: the thread's share of a row's 64 weights
    const int w0 = SUBS == 2 ? 0 : grp * 4;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    uint8_t* const staging = smem + W_STAGES * C::kStage + grp * W_STORE;
    int i = 0, item = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.plan.tiles && ok; tile += p.plan.grid, ++item) {
      for (int kt = 0; kt < nkt; ++kt, ++i) {
        const int s = i % W_STAGES, w = i % C::kBufs;
        ok = mbar_wait(&full[s], (i / W_STAGES) & 1);
        if (!ok) break;
        const uint8_t* st = stage_ptr(s);
        const uint4* raw = reinterpret_cast<const uint4*>(st + OFF_RAW + sub * W_RAW + row * 32 + w0 * 4);
        uint32_t words[WORDS];
#pragma unroll
        for (int j = 0; j < WORDS / 4; ++j) { const uint4 c = raw[j]; words[4 * j] = c.x; words[4 * j + 1] = c.y; words[4 * j + 2] = c.z; words[4 * j + 3] = c.w; }
        const uint32_t sc = *reinterpret_cast<const uint32_t*>(st + OFF_SF + sub * W_SF + row * 8 + (kt & 1) * 4) >> (4 * w0);
        uint32_t r[4 * WORDS];
#pragma unroll
        for (int j = 0; j < WORDS; ++j) {                    // 8 weights -> 4 columns
          const uint32_t scale = w_e4m3_to_bf16x2_dup((sc >> (8 * (j >> 1))) & 0xffu);
          w_e2m1x8_to_bf16x8(words[j], r + 4 * j);
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            // code x scale has <= 6 significant bits: the bf16 product is exact
            const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&r[4 * j + b]),
                                             *reinterpret_cast<const __nv_bfloat162*>(&scale));
            r[4 * j + b] = *reinterpret_cast<const uint32_t*>(&v);
          }
        }
        ok = mbar_wait(&wempty[w], ((i / C::kBufs) & 1) ^ 1);
        if (!ok) break;
        tc_fence_after();
        if (SUBS == 2) tmem_st32(lane_base + C::kW + (w * 2 + sub) * 32, r);
        else tmem_st16(lane_base + C::kW + w * 32 + w0 * 4, r);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&wfull[w]);
      }
      // epilogue: TMEM lane = output feature, column = token. Two sub-tiles: a group of four warps each; one: half of the tokens each
      if (ok) ok = mbar_wait(&acc_full, item & 1);
      ok = !__any_sync(0xffffffffu, !ok);
      if (!ok) atomicExch(&s_fail, 1);
      tc_fence_after();
      asm volatile("bar.sync 3, 256;" ::: "memory");          // one answer for the eight warps: they meet at barriers below
      ok = !*(volatile int*)&s_fail;
      if (!ok) break;
      const int tn = tile / p.plan.tiles_t, t0 = (tile - tn * p.plan.tiles_t) * p.plan.tile_t, n0 = tn * 128 * SUBS + sub * 128;
      const int rows = min(p.plan.tile_t, p.T - t0);
      const int c0 = SUBS == 2 ? 0 : grp * 128, c1 = SUBS == 2 ? rows : min(rows, c0 + 128);
      if (n0 < p.N)
        for (int t = c0; t < c1; t += 32)
          store_tile<32>(staging, tmem_base + sub * C::kT + t, quarter, etid, n0, t0 + t,
                         TileOut{p.N, t0 + c1, p.alpha, p.out, nullptr, p.ldo, p.residual, p.ldr}, 1 + grp);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_free);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
  if (threadIdx.x == 0 && s_fail && p.status) atomicExch(p.status, (int)kErrMbarTimeout);
}

template <int SUBS>
static int launch_wide(WideParams p, const void* Wp, const void* X, long ldx, cudaStream_t st) {
  p.plan = wide_plan<SUBS>(p.T, p.N);
  CUtensorMap amap, bmap;
  int rc = make_tmap_2d(&amap, Wp, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.N, p.K / 2, (uint64_t)p.K / 2, 128, 32, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (rc) return rc;
  rc = make_tmap_2d(&bmap, X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.T, p.K, (uint64_t)ldx * 2, p.plan.tile_t, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_w4a16_wide_kernel<SUBS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Wide<SUBS>::kSmem);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  gemm_w4a16_wide_kernel<SUBS><<<p.plan.grid, 320, Wide<SUBS>::kSmem, st>>>(p, amap, bmap);
  return (int)cudaGetLastError();
}

}  // namespace ve

using namespace ve;

extern "C" {

// Wp [N, K/2] bytes, sfa [N/128][K/128][128][8], X [T, K] bf16 (pitch ldx). N % 128 == 0, K % 128 == 0.
int ve_gemm_w4a16_wide(const void* Wp, const void* sfa, const void* X, long ldx, void* out, long ldo, const void* residual,
                       long ldr, int T, int N, int K, float alpha, void* status, cudaStream_t st) {
  if (T <= 0 || N <= 0) return 0;
  if (N % 128 || K % 128 || K <= 0) return cudaErrorInvalidValue;
  const WideParams p{{}, N, T, K, alpha, (__nv_bfloat16*)out, ldo, (const __nv_bfloat16*)residual, ldr, (const uint8_t*)sfa, (int*)status};
  const WidePlan one = wide_plan<1>(T, N), two = wide_plan<2>(T, N);
  const long waves1 = (one.tiles + W_GRID - 1) / W_GRID, waves2 = (two.tiles + W_GRID - 1) / W_GRID;
  return 10 * waves2 <= 7 * waves1 ? launch_wide<2>(p, Wp, X, ldx, st) : launch_wide<1>(p, Wp, X, ldx, st);
}

}  // extern "C"
