// Prefill linear with NVFP4 weights and bf16 activations on 256-feature x 192-token (or shorter) output tiles:
//   out[t, n] = alpha * sum_k W[n, k] * X[t, k],   W dequantised to bf16 inside the tile loader (exact products).
//
// Two things bounded the form in front of this one (256 x 256 tiles, dequantised weights in shared memory, a block per tile):
//  * shared memory: per 64-wide k step both weight sub-tiles were written to it as bf16 (32 KB) and read back (32 KB) beside two reads of the
//    activation tile (64 KB) and the loads (41 KB): 180 KB, 1400 cycles at 128 B a cycle for 1024 cycles of tensor work. Here the dequantised
//    weights go to tensor memory, from where the MMA takes its A operand: 92 KB, 720 cycles for 768 cycles of tensor work. Two accumulators
//    of 192 columns and two buffers of 2 x 32 columns of weights fill the 512 columns, hence the 192 tokens.
//  * the last wave: 2048 tokens x 5120 features are 160 tiles of 256 x 256 on 148 SMs. Here the blocks are persistent, and the tiles of the
//    partial last wave (or of the last two) are dealt to the blocks by k steps where that is shorter: a cut tile leaves fp32 partial
//    sums in a workspace, and the block that arrives last adds them up in the order of k and stores. No block waits for another.
//
// Warp roles (320 threads): warp 0 TMA producer, warp 1 TMEM owner + MMA issuer, warps 2..9 dequantise (one weight row of 64 a thread and step,
// warps 2..5 and 6..9 a 128-feature sub-tile each) and run the epilogue. Every wait is bounded.
// Reference kernel family this replaces: src/kernels/cuda/nvfp4/skinny_kernels.cu:531-558 (fused WMMA GEMM / dequant + HGEMM).
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "tmap.h"

namespace ve {

constexpr int W_KT = 64, W_T = 192, W_RAW = 128 * 32, W_B = W_T * 128, W_SF = 1024;
constexpr int W_STAGE = W_B + 2 * W_RAW + 2 * W_SF;                  // 34816
constexpr int W_STAGES = 5, W_STORE = 32 * 528;                       // 32 tokens of an output sub-tile at a time
constexpr int W_SMEM = W_STAGES * W_STAGE + 2 * W_STORE + 1024;
constexpr int W_ACC = 2 * W_T;                                         // first TMEM column of the weight buffers
constexpr int W_GRID = 148;

// How the output tiles are dealt: the first `cut` tiles by k steps (multiples of `quantum`) to the first `cutters` blocks, the others whole.
struct WidePlan {
  int tile_t;                     // tokens of a tile, a multiple of 16
  int tiles_n, tiles_t, tiles, nkt, grid, cut, cutters, quantum;
  // first of block c's steps of the cut tiles
  __host__ __device__ int begin(int c) const {
    const long q = (long)cut * (nkt / quantum);                        // quanta in all
    return c >= cutters ? cut * nkt : (int)(q * c / cutters) * quantum;
  }
};
// Costs in k steps of a 192-token tile (0.5 to 0.8 us): a block that leaves a piece of a tile spends about eight on writing it, and the block that
// adds a tile up about six for each of its pieces (2048 tokens, 5120 x 5120: 44 us for two pieces a block and 2.5 a tile). So tiles are
// cut where that is less than what the last, partly filled wave wastes: the remainder alone, in at most eight pieces a tile (220 tiles:
// 148 whole and 72 in two), or with one whole wave (160 tiles), whichever is shorter; a short K or a handful of tiles stay whole
// (44 tiles of 32 steps: 39 us whole, 68 us cut).
static inline WidePlan wide_plan(int T, int N, int K) {
  WidePlan p;
  p.tiles_n = (N + 255) / 256; p.tiles_t = (T + W_T - 1) / W_T; p.tiles = p.tiles_n * p.tiles_t; p.nkt = K / W_KT;
  p.tile_t = ((T + p.tiles_t - 1) / p.tiles_t + 15) / 16 * 16;          // (no taller than the tokens ask for: 452 are 3 x 160)
  p.quantum = 1;
  for (int q = p.nkt / 16; q > 1; --q)
    if (p.nkt % q == 0) { p.quantum = q; break; }
  const int waves = (p.tiles + W_GRID - 1) / W_GRID, rest = p.tiles % W_GRID;
  p.grid = p.tiles < W_GRID ? p.tiles : W_GRID;
  p.cut = 0;
  p.cutters = 1;
  long best = (long)waves * p.nkt;
  if (rest) {
    for (int n = 2; n <= 8 && rest * n <= W_GRID + rest; ++n) {           // n pieces a tile, as far as there are blocks
      const int blocks = rest * n < W_GRID ? rest * n : W_GRID;
      const long cost = (long)(waves - 1) * p.nkt + ((long)rest * p.nkt + blocks - 1) / blocks + 8 + 6 * (n + (blocks < rest * n));
      if (cost < best) { best = cost; p.cut = rest; p.cutters = blocks; }
    }
    const long cost = ((long)p.tiles * p.nkt + W_GRID - 1) / W_GRID + 16 + 6 * 3;
    if (waves > 1 && cost < best) { best = cost; p.cut = rest + W_GRID; p.cutters = W_GRID; }
    if (p.cut && p.grid < p.cutters) p.grid = p.cutters;
  }
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
  float* partial;         // [2 * cutters][W_T][256]: a block's first and last piece of a cut tile
  int* arrived;           // [cut] zeros
  int* status;
};

// The pieces of work of a block, in order: its share of the cut tiles, then whole tiles.
struct WideItems {
  const WidePlan& p;
  int c, pos, end, whole, tile, k0, k1, first;
  __device__ WideItems(const WidePlan& plan, int block) : p(plan), c(block), whole(plan.cut + block), first(1) {
    pos = p.cut ? p.begin(c) : 0;
    end = p.cut ? p.begin(c + 1) : 0;
  }
  __device__ bool next() {
    if (pos < end) {
      tile = pos / p.nkt;
      k0 = pos - tile * p.nkt;
      k1 = min(p.nkt, k0 + end - pos);
      first = pos == p.begin(c);
      pos += k1 - k0;
      return true;
    }
    if (whole >= p.tiles) return false;
    tile = whole; k0 = 0; k1 = p.nkt;
    whole += p.grid;
    return true;
  }
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


__global__ void __launch_bounds__(320, 1)
gemm_w4a16_wide_kernel(const WideParams p, const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap) {
  static_assert(W_STAGE % 1024 == 0, "stage must keep 1024 B alignment");
  static_assert(W_SMEM <= 227 * 1024, "shared memory budget");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[W_STAGES], empty[W_STAGES], wfull[2], wempty[2], acc_full, acc_free;
  __shared__ uint32_t tmem_holder;
  __shared__ int s_fail, s_last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < W_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&wfull[s], 8); mbar_init(&wempty[s], 1); }
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
  auto stage_ptr = [&](int s) { return smem + (size_t)s * W_STAGE; };   // [B][RAW0][RAW1][SF0][SF1]
  constexpr int OFF_RAW = W_B, OFF_SF = W_B + 2 * W_RAW;
  WideItems it(p.plan, blockIdx.x);

  if (warp == 0) {
    if (elect_one()) {
      prefetch_tmap(&amap);
      prefetch_tmap(&bmap);
      const size_t blk = (size_t)(p.K / 128);
      int i = 0;                                   // steps so far, over all items
      bool ok = true;
      while (ok && it.next()) {
        const int tn = it.tile / p.plan.tiles_t, t0 = (it.tile - tn * p.plan.tiles_t) * p.plan.tile_t, n0 = tn * 256;
        // (a matrix of an odd number of 128-feature tiles: the second one's codes read as zero, its scales are the first one's)
        const int sf1 = n0 + 128 < p.N ? 2 * tn + 1 : 2 * tn;
        for (int kt = it.k0; kt < it.k1; ++kt, ++i) {
          const int s = i % W_STAGES;
          ok = mbar_wait(&empty[s], ((i / W_STAGES) & 1) ^ 1);
          if (!ok) break;
          uint8_t* st = stage_ptr(s);
          mbar_expect_tx(&full[s], 2 * W_RAW + p.plan.tile_t * 128 + 2 * W_SF);
          tma_load_2d(st + OFF_RAW, &amap, &full[s], kt * 32, n0);
          tma_load_2d(st + OFF_RAW + W_RAW, &amap, &full[s], kt * 32, n0 + 128);
          tma_load_2d(st, &bmap, &full[s], kt * W_KT, t0);
          bulk_load(st + OFF_SF, p.sfa + ((size_t)(2 * tn) * blk + (kt >> 1)) * 1024, W_SF, &full[s]);
          bulk_load(st + OFF_SF + W_SF, p.sfa + ((size_t)sf1 * blk + (kt >> 1)) * 1024, W_SF, &full[s]);
        }
      }
      if (!ok) atomicExch(&s_fail, 1);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_f16(1, 1, 128, p.plan.tile_t);
      int i = 0, item = 0;
      bool ok = true;
      while (ok && it.next()) {
        ok = mbar_wait(&acc_free, (item & 1) ^ 1);          // the epilogue has read the item in front
        tc_fence_after();
        for (int kt = it.k0; kt < it.k1 && ok; ++kt, ++i) {
          const int s = i % W_STAGES, w = i & 1;
          ok = mbar_wait(&full[s], (i / W_STAGES) & 1) && mbar_wait(&wfull[w], (i >> 1) & 1);
          if (!ok) break;
          tc_fence_after();
          const uint64_t bd = make_desc_sw128(smem_u32(stage_ptr(s)));
#pragma unroll
          for (int sub = 0; sub < 2; ++sub)
#pragma unroll
            for (int kb = 0; kb < 4; ++kb)
              tc_mma_f16_ta(tmem_base + sub * W_T, tmem_base + W_ACC + w * 64 + sub * 32 + kb * 8, bd + kb * 2, idesc,
                            (kt > it.k0 || kb) ? 1u : 0u);
          tc_commit(&empty[s]);
          tc_commit(&wempty[w]);
        }
        tc_commit(&acc_full);
        ++item;
      }
      if (!ok) atomicExch(&s_fail, 1);
    }
  } else {
    const int dw = warp - 2, sub = dw >> 2, quarter = warp & 3, row = quarter * 32 + lane, etid = (dw & 3) * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    uint8_t* const staging = smem + W_STAGES * W_STAGE + sub * W_STORE;
    int i = 0, item = 0;
    bool ok = true;
    while (ok && it.next()) {
      for (int kt = it.k0; kt < it.k1; ++kt, ++i) {
        const int s = i % W_STAGES, w = i & 1;
        ok = mbar_wait(&full[s], (i / W_STAGES) & 1);
        if (!ok) break;
        const uint8_t* st = stage_ptr(s);
        const uint4* raw = reinterpret_cast<const uint4*>(st + OFF_RAW + sub * W_RAW + row * 32);
        const uint4 c0 = raw[0], c1 = raw[1];
        const uint32_t words[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        const uint32_t sc = *reinterpret_cast<const uint32_t*>(st + OFF_SF + sub * W_SF + row * 8 + (kt & 1) * 4);
        uint32_t r[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {                        // 8 weights -> 4 columns
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
        ok = mbar_wait(&wempty[w], ((i >> 1) & 1) ^ 1);
        if (!ok) break;
        tc_fence_after();
        tmem_st32(lane_base + W_ACC + w * 64 + sub * 32, r);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&wfull[w]);
      }
      // epilogue: TMEM lane = output feature, column = token
      if (ok) ok = mbar_wait(&acc_full, item & 1);
      ok = !__any_sync(0xffffffffu, !ok);
      if (!ok) atomicExch(&s_fail, 1);
      tc_fence_after();
      asm volatile("bar.sync 3, 256;" ::: "memory");          // one answer for the eight warps: they meet at barriers below
      ok = !*(volatile int*)&s_fail;
      if (!ok) break;
      const int tn = it.tile / p.plan.tiles_t, t0 = (it.tile - tn * p.plan.tiles_t) * p.plan.tile_t, n0 = tn * 256;
      const int rows = min(p.plan.tile_t, p.T - t0);
      const bool piece = it.k0 > 0 || it.k1 < p.plan.nkt;
      if (!piece) {
        if (n0 + sub * 128 < p.N)
          for (int t = 0; t < rows; t += 32)
            store_tile<32>(staging, tmem_base + sub * W_T + t, quarter, etid, n0 + sub * 128, t0 + t,
                           TileOut{p.N, t0 + rows, p.alpha, p.out, nullptr, p.ldo, p.residual, p.ldr}, 1 + sub);
      } else {
        float* mine = p.partial + (size_t)(2 * blockIdx.x + (it.first ? 0 : 1)) * (W_T * 256) + sub * 128 + row;
#pragma unroll 1
        for (int t = 0; t < rows; t += 16) {
          uint32_t r[16];
          tmem_ld16(lane_base + sub * W_T + t, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) __stcg(mine + (size_t)(t + j) * 256, __uint_as_float(r[j]));
        }
        __threadfence();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_free);
      if (piece) {
        // the tile's pieces: blocks c_lo .. c_hi; the last one to arrive adds all of them in the order of k
        const int begin = it.tile * p.plan.nkt, end = begin + p.plan.nkt;
        int c_lo = blockIdx.x, c_hi = blockIdx.x;
        while (p.plan.begin(c_lo) > begin) --c_lo;
        while (p.plan.begin(c_hi + 1) < end) ++c_hi;
        asm volatile("bar.sync 3, 256;" ::: "memory");
        if (threadIdx.x == 64) {
          int pieces = 0;
          for (int c = c_lo; c <= c_hi; ++c) pieces += p.plan.begin(c + 1) > p.plan.begin(c);
          s_last = atomicAdd(p.arrived + it.tile, 1) == pieces - 1;
        }
        asm volatile("bar.sync 3, 256;" ::: "memory");
        if (s_last) {
          __threadfence();
          const int f = ((threadIdx.x - 64) & 63) * 4, n = n0 + f;
          const bool vec = !((uintptr_t)p.out & 7) && p.ldo % 4 == 0 && (!p.residual || (!((uintptr_t)p.residual & 7) && p.ldr % 4 == 0));
          if (n < p.N)
            for (int t = (threadIdx.x - 64) >> 6; t < rows; t += 64) {
              float4 sum[16];                        // (sixteen loads in flight a thread)
#pragma unroll
              for (int j = 0; j < 16; ++j) sum[j] = make_float4(0.f, 0.f, 0.f, 0.f);
              for (int c = c_lo; c <= c_hi; ++c) {
                const int b0 = p.plan.begin(c);
                if (p.plan.begin(c + 1) == b0) continue;
                const float* src = p.partial + (size_t)(2 * c + (b0 >= begin ? 0 : 1)) * (W_T * 256) + f;
#pragma unroll
                for (int j = 0; j < 16; ++j)
                  if (t + 4 * j < rows) {
                    const float4 v = __ldcg(reinterpret_cast<const float4*>(src + (size_t)(t + 4 * j) * 256));
                    sum[j].x += v.x; sum[j].y += v.y; sum[j].z += v.z; sum[j].w += v.w;
                  }
              }
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                if (t + 4 * j >= rows) continue;
                float o[4] = {sum[j].x * p.alpha, sum[j].y * p.alpha, sum[j].z * p.alpha, sum[j].w * p.alpha};
                __nv_bfloat16* dst = p.out + (long)(t0 + t + 4 * j) * p.ldo + n;
                const __nv_bfloat16* res = p.residual ? p.residual + (long)(t0 + t + 4 * j) * p.ldr + n : nullptr;
                if (vec) {
                  if (res) {
                    const uint2 b = *reinterpret_cast<const uint2*>(res);
                    o[0] += __uint_as_float(b.x << 16); o[1] += __uint_as_float(b.x & 0xffff0000u);
                    o[2] += __uint_as_float(b.y << 16); o[3] += __uint_as_float(b.y & 0xffff0000u);
                  }
                  const __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]), hi = __floats2bfloat162_rn(o[2], o[3]);
                  *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                } else {
                  for (int e = 0; e < 4; ++e) dst[e] = f2bf(o[e] + (res ? bf2f(res[e]) : 0.f));
                }
              }
            }
        }
      }
      ++item;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
  if (threadIdx.x == 0 && s_fail && p.status) atomicExch(p.status, (int)kErrMbarTimeout);
}

}  // namespace ve

using namespace ve;

extern "C" {

// Bytes of workspace that a call of these sizes wants (0: none).
long ve_gemm_w4a16_wide_scratch(int T, int N, int K) {
  if (T <= 0 || N <= 0 || K < W_KT) return 0;
  const WidePlan pl = wide_plan(T, N, K);
  return pl.cut ? (long)2 * pl.cutters * W_T * 256 * 4 + (long)pl.cut * 4 : 0;
}

// Wp [N, K/2] bytes, sfa [N/128][K/128][128][8], X [T, K] bf16 (pitch ldx). N % 128 == 0, K % 128 == 0. scratch: 16-byte aligned,
// ve_gemm_w4a16_wide_scratch bytes, this call's alone until it has run.
int ve_gemm_w4a16_wide(const void* Wp, const void* sfa, const void* X, long ldx, void* out, long ldo, const void* residual,
                       long ldr, int T, int N, int K, float alpha, void* status, void* scratch, cudaStream_t st) {
  if (T <= 0 || N <= 0) return 0;
  if (N % 128 || K % 128 || K <= 0) return cudaErrorInvalidValue;
  const WidePlan pl = wide_plan(T, N, K);
  if (pl.cut && !scratch) return cudaErrorInvalidValue;
  CUtensorMap amap, bmap;
  int rc = make_tmap_2d(&amap, Wp, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K / 2, (uint64_t)K / 2, 128, 32, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (rc) return rc;
  rc = make_tmap_2d(&bmap, X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, T, K, (uint64_t)ldx * 2, pl.tile_t, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_w4a16_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, W_SMEM);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  float* partial = (float*)scratch;
  int* arrived = pl.cut ? (int*)(partial + (size_t)2 * pl.cutters * W_T * 256) : nullptr;
  if (pl.cut) {
    const cudaError_t e = cudaMemsetAsync(arrived, 0, (size_t)pl.cut * 4, st);
    if (e != cudaSuccess) return (int)e;
  }
  WideParams p{pl, N, T, K, alpha, (__nv_bfloat16*)out, ldo, (const __nv_bfloat16*)residual, ldr, (const uint8_t*)sfa, partial, arrived, (int*)status};
  gemm_w4a16_wide_kernel<<<pl.grid, 320, W_SMEM, st>>>(p, amap, bmap);
  return (int)cudaGetLastError();
}

}  // extern "C"
