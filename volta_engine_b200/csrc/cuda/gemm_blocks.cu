// Grouped (mixture-of-experts) GEMM over block-quantised expert weights, decoded in the tile loader:
//   out[r, n] = sum_k W[expert(r)][n, k] * X[r, k]       rows r sorted by expert, W as GGUF blocks or EXL3 tiles
// The weights are decoded to bf16 straight into the swizzled operand tile of a tcgen05 MMA, with the same rounding as decoding the whole
// bank to bf16 first and multiplying it with the bf16 grouped GEMM. That way wrote and read 2 bytes a weight for 0.2 to 0.5 stored: for
// 256 experts of 3 x 7168 x 2048 weights (IQ1_M) 45 GB each way and layer pair, 47.7 ms of decoding and 12.0 ms of GEMM per 1900 rows.
//
// One CTA: 128 output features x one tile of at most 128 rows of one expert. Warp 0: TMA of the rows' bf16 tiles (boxes of 32 rows, as many
// as the tile has); warp 1: TMEM and MMA; warps 2..9 decode: each copies the raw blocks of its 16 features (EXL3: its 16-column tiles) with
// cp.async through a ring of its own, 256 weights of K ahead, and writes bf16 into the stage; warps 2..5 store the tile. Two CTAs share an
// SM, so one decodes while the other multiplies or stores. What bounds it is issuing the decoding: 9.7 instructions a
// weight and tile for IQ1_M, 10.7 for trellis codes of 4 bits, 61 and 72 % of the issue slots of 20 warps an SM; next come waits for a stage. So a
// tile is as tall as two CTAs' shared memory allows.
// Every wait is bounded; on expiry the kernel records a status code and drains.
#include "common.cuh"
#include "exl3_blocks.cuh"
#include "gemm_epilogue.cuh"
#include "gguf_blocks.cuh"
#include "tmap.h"

namespace ve {

struct BlockGemmParams {
  int N, K;
  const uint8_t* W; long row_bytes; const uint8_t* W_end;    // experts back to back (EXL3: row_bytes = bytes of one expert)
  __nv_bfloat16* out; long ldo;
  const int* tile_tab;          // [tiles] {expert, first row, rows, 0}
  int* status;
};

constexpr int kBgRows = 128, kBgStages = 2, kBgA = 128 * 128, kBgB = kBgRows * 128, kBgStage = kBgA + kBgB, kBgWarps = 8;
constexpr int kBgTwo = 113 * 1024;      // shared memory of a CTA that lets two share an SM

VE_DEVINL uint32_t scaled_pair(uint32_t q, float s, float m, bool has_min) {
  const float lo = __uint_as_float(q << 16), hi = __uint_as_float(q & 0xffff0000u);
  const __nv_bfloat162 r = has_min ? __floats2bfloat162_rn(fmaf(s, lo, -m), fmaf(s, hi, -m)) : __floats2bfloat162_rn(s * lo, s * hi);
  return *reinterpret_cast<const uint32_t*>(&r);
}

// 16 features of GGUF rows: lane quad g, lane t takes features row and row + 8, weights 16 i + 4 t .. + 3 of each chunk (see frag).
template <int TYPE>
struct GgufTile {
  using F = Fmt<TYPE>;
  static constexpr int kPitch = ((F::kUnit + 14 + 15) / 16 | 1) * 16;
  static constexpr int kRaw = 16 * kPitch;                   // a warp's raw bytes of one unit
  static constexpr int kSub = F::kChunks / 2;                 // 64-wide k steps of a unit
  static constexpr int kTab = (F::kTabBytes + 15) / 16 * 16;
  const uint8_t* rp[2];
  const uint8_t* end;
  int chunks, row, t, g;
  VE_DEVINL void init(const BlockGemmParams& p, int expert, int n0, int warp, int lane) {
    g = lane >> 2; t = lane & 3;
    // rows of an octet go to quads 0, 2, 4, 6, 1, 3, 5, 7: the 8-byte stores of half a warp then meet all eight 16-byte slots of the swizzle
    // (16-byte stores of a quarter warp: rows 0 and 4, 1 and 5, ...)
    row = warp * 16 + (F::kVec8 ? ((g & 1) << 2) | (g >> 1) : ((g & 3) << 1) | (g >> 2));
    end = p.W_end;
    chunks = p.K >> 5;
#pragma unroll
    for (int r = 0; r < 2; ++r)                                // (features behind the matrix repeat its last row; they are not stored)
      rp[r] = p.W + ((size_t)expert * p.N + min(n0 + row + 8 * r, p.N - 1)) * p.row_bytes;
  }
  VE_DEVINL void load(int unit, uint8_t* dst) const {
    if (unit * F::kChunks >= chunks) return;
    const int bytes = F::kBig ? F::kBytes : min(F::kChunks, chunks - unit * F::kChunks) * F::kBytes;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint8_t* src = rp[r] + (size_t)unit * F::kUnit;
      const int off = (int)((uintptr_t)src & 15);              // whole 16-byte pieces: inside the allocation, but for the one the bank ends in
      src -= off;
      const int n16 = (off + bytes + 15) >> 4;
      for (int j = t; j < n16; j += 4) {
        const long left = end - (src + j * 16);
        cp_async16(dst + (r * 8 + g) * kPitch + j * 16, src + j * 16, left < 16 ? (int)left : 16);
      }
    }
  }
  VE_DEVINL void decode(const uint8_t* raw, int unit, int sub, uint8_t* a, const uint8_t* tab) const {
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
      const int c = sub * 2 + cc;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if constexpr (F::kVec8) {                              // three values a vector, rounded once each and picked by the codes
          const uint8_t* u = raw + (r * 8 + g) * kPitch + (int)((uintptr_t)(rp[r] + (size_t)unit * F::kUnit) & 15);
          uint32_t lut, f[4];
          const uint32_t codes = vec8_codes<TYPE>(u, c, t, tab, lut);
          const float dl = vec8_scale<TYPE>(u) * u2f(2 * (lut & 7) + 1), sh = lut & 8 ? -0.125f : 0.125f;
          const __nv_bfloat162 v01 = __floats2bfloat162_rn(dl * (-1.f + sh), dl * sh), v2 = __floats2bfloat162_rn(dl * (1.f + sh), 0.f);
          const uint32_t p01 = *reinterpret_cast<const uint32_t*>(&v01), p2 = *reinterpret_cast<const uint32_t*>(&v2);
          vec8_expand(codes, __byte_perm(p01, p2, 0x6420), __byte_perm(p01, p2, 0x7531), f);
          *reinterpret_cast<uint4*>(a + (row + 8 * r) * 128 + (((cc * 4 + t) ^ (row & 7)) << 4)) = make_uint4(f[0], f[1], f[2], f[3]);
          continue;
        }
        uint32_t q[4] = {0u, 0u, 0u, 0u};
        float s[2] = {0.f, 0.f}, m[2] = {0.f, 0.f};
        if (F::kBig || unit * F::kChunks + c < chunks) {
          const uint8_t* u = raw + (r * 8 + g) * kPitch + (int)((uintptr_t)(rp[r] + (size_t)unit * F::kUnit) & 15);
          if constexpr (!F::kVec8) frag<TYPE>(u, c, t, tab, q, s, m);
        }
        if (!F::kScale16) s[1] = s[0];
        if (F::kMin == 1) m[1] = m[0];
        uint8_t* dst = a + (row + 8 * r) * 128 + (t & 1) * 8;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *reinterpret_cast<uint2*>(dst + (((cc * 4 + 2 * i + (t >> 1)) ^ (row & 7)) << 4)) =
              make_uint2(scaled_pair(q[2 * i], s[i], m[i], F::kMin != 0), scaled_pair(q[2 * i + 1], s[i], m[i], F::kMin != 0));
      }
    }
  }
};

// 16 features of EXL3 tiles: one column of tiles, 16 k-tiles a unit.
template <int BITS, int CB>
struct Exl3Tile {
  static constexpr int kRaw = 16 * 32 * BITS, kSub = 4, kTab = 0;
  const uint8_t* base;
  size_t kstride;
  int kt_all, warp, lane;
  VE_DEVINL void init(const BlockGemmParams& p, int expert, int n0, int warp_, int lane_) {
    warp = warp_; lane = lane_;
    kt_all = p.K >> 4;
    kstride = (size_t)(p.N >> 4) * 32 * BITS;
    base = p.W + (size_t)expert * p.row_bytes + (size_t)((n0 >> 4) + warp) * 32 * BITS;
  }
  VE_DEVINL void load(int unit, uint8_t* dst) const {
#pragma unroll
    for (int i = 0; i < BITS; ++i) {
      const int j = lane + 32 * i, tile = j / (2 * BITS), piece = j % (2 * BITS), kt = unit * 16 + tile;
      if (kt < kt_all)
        cp_async16(dst + j * 16, base + (size_t)kt * kstride + piece * 16);
    }
  }
  VE_DEVINL void decode(const uint8_t* raw, int unit, int sub, uint8_t* a, const uint8_t*) const {
    const Exl3Lane<BITS> L(lane);
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t w[3] = {0u, 0u, 0u}, f[4];
      L.load_shared(reinterpret_cast<const uint32_t*>(raw + (sub * 4 + j) * 32 * BITS), w);
      L.template decode<CB>(w, f);
      const bool live = unit * 16 + sub * 4 + j < kt_all;
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&f[p]));
        const __nv_bfloat162 r = __floats2bfloat162_rn(v.x, v.y);
        const int row = warp * 16 + g + 8 * (p >> 1);
        *reinterpret_cast<uint32_t*>(a + row * 128 + (((j * 2 + (p & 1)) ^ (row & 7)) << 4) + t * 4) =
            live ? *reinterpret_cast<const uint32_t*>(&r) : 0u;
      }
    }
  }
};

template <class D>
struct BgCfg {
  // raw units in flight: as many as leave room for two CTAs, two at least
  static constexpr int fits(int n) { return kBgStages * kBgStage + n * kBgWarps * D::kRaw + D::kTab + 1024 + 256; }
  static constexpr int kRing = fits(3) <= kBgTwo ? 3 : 2;
  static constexpr int kSmem = kBgStages * kBgStage + kRing * kBgWarps * D::kRaw + D::kTab + 1024;
};

template <class D> struct TableOf { static VE_DEVINL void load(uint8_t*) {} };
template <int TYPE> struct TableOf<GgufTile<TYPE>> { static VE_DEVINL void load(uint8_t* tab) { if (GgufTile<TYPE>::kTab) load_table<TYPE>(tab); } };

template <class D>
__global__ void __launch_bounds__(64 + 32 * kBgWarps, 2) gemm_blocks_kernel(const BlockGemmParams p, const __grid_constant__ CUtensorMap bmap) {
  static_assert(kBgStages * kBgStage + BgCfg<D>::kRing * kBgWarps * D::kRaw >= 128 * 528, "the output tile is staged in the operand memory");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* const ring = smem + kBgStages * kBgStage;
  uint8_t* const tab = ring + BgCfg<D>::kRing * kBgWarps * D::kRaw;
  __shared__ uint64_t full[kBgStages], empty[kBgStages], deq[kBgStages], acc_full;
  __shared__ uint32_t tmem_holder;
  __shared__ int s_fail;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int4 tt = reinterpret_cast<const int4*>(p.tile_tab)[blockIdx.y];
  if (tt.z <= 0) return;                        // idle tile: uniform exit before any barrier or TMEM use
  const int n0 = blockIdx.x * 128, boxes = (min(tt.z, kBgRows) + 31) / 32;
  const int nkt = (p.K + 63) / 64;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kBgStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); mbar_init(&deq[s], kBgWarps); }
    mbar_init(&acc_full, 1);
    s_fail = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&tmem_holder, 128); tmem_relinquish(); }
  TableOf<D>::load(tab);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_holder;

  if (warp == 0) {
    if (elect_one()) {
      prefetch_tmap(&bmap);
      for (int kt = 0; kt < nkt; ++kt) {
        const int s = kt % kBgStages;
        if (!mbar_wait(&empty[s], ((kt / kBgStages) & 1) ^ 1)) { atomicExch(&s_fail, 1); break; }
        mbar_expect_tx(&full[s], boxes * 4096);
        for (int b = 0; b < boxes; ++b) tma_load_2d(smem + s * kBgStage + kBgA + b * 4096, &bmap, &full[s], kt * 64, tt.y + b * 32);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_f16(1, 1, 128, boxes * 32);
      bool ok = true;
      for (int kt = 0; kt < nkt && ok; ++kt) {
        const int s = kt % kBgStages;
        const uint32_t par = (kt / kBgStages) & 1;
        ok = mbar_wait(&full[s], par) && mbar_wait(&deq[s], par);
        if (!ok) break;
        tc_fence_after();
        const uint64_t ad = make_desc_sw128(smem_u32(smem + s * kBgStage)), bd = make_desc_sw128(smem_u32(smem + s * kBgStage + kBgA));
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) tc_mma_f16(tmem, ad + kb * 2, bd + kb * 2, idesc, (kt | kb) ? 1u : 0u);
        tc_commit(&empty[s]);
      }
      if (!ok) atomicExch(&s_fail, 1);
      tc_commit(&acc_full);
    }
  } else {
    constexpr int R = BgCfg<D>::kRing;
    D d;
    d.init(p, tt.x, n0, warp - 2, lane);
    uint8_t* const mine = ring + (warp - 2) * R * D::kRaw;
    const int units = (nkt + D::kSub - 1) / D::kSub;
#pragma unroll
    for (int u = 0; u < R - 1; ++u) {
      if (u < units) d.load(u, mine + u * D::kRaw);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    bool ok = true;
    for (int u = 0; u < units && ok; ++u) {
      asm volatile("cp.async.wait_group %0;" ::"n"(R - 2) : "memory");
      __syncwarp();                                // the unit is here for every lane, and the slot in front of it is free
      if (u + R - 1 < units) d.load(u + R - 1, mine + (u + R - 1) % R * D::kRaw);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const uint8_t* raw = mine + u % R * D::kRaw;
#pragma unroll
      for (int sub = 0; sub < D::kSub; ++sub) {
        const int kt = u * D::kSub + sub;
        if (kt < nkt && ok) {
          const int s = kt % kBgStages;
          ok = mbar_wait(&empty[s], ((kt / kBgStages) & 1) ^ 1);
          if (ok) {
            d.decode(raw, u, sub, smem + s * kBgStage, tab);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&deq[s]);
          }
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok) atomicExch(&s_fail, 1);
    if (warp < 6) {
      // epilogue: TMEM lane = output feature, column = row of the tile
      if (!mbar_wait(&acc_full, 0)) atomicExch(&s_fail, 1);
      tc_fence_after();
      asm volatile("bar.sync 1, 128;" ::: "memory");        // one answer for the four warps: they meet at barriers below
      if (!*(volatile int*)&s_fail)
        store_tile<128>(smem, tmem, warp & 3, threadIdx.x - 64, n0, tt.y, TileOut{p.N, tt.y + min(tt.z, kBgRows), 1.f, p.out, nullptr, p.ldo, nullptr, 0});
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 128); }
  if (threadIdx.x == 0 && s_fail && p.status) atomicExch(p.status, (int)kErrMbarTimeout);
}

template <class D>
static int launch_blocks(const BlockGemmParams& p, const CUtensorMap& bmap, int n_tiles, cudaStream_t st) {
  const cudaError_t e = allow_smem<gemm_blocks_kernel<D>>(BgCfg<D>::kSmem);
  if (e != cudaSuccess) return (int)e;
  gemm_blocks_kernel<D><<<dim3((p.N + 127) / 128, n_tiles), 64 + 32 * kBgWarps, BgCfg<D>::kSmem, st>>>(p, bmap);
  return (int)cudaGetLastError();
}

template <int TYPE>
static int launch_gguf_blocks(const BlockGemmParams& p, const CUtensorMap& bmap, int n_tiles, cudaStream_t st) {
  // (fields are read in words of their natural alignment)
  if (((uintptr_t)p.W | (uintptr_t)p.row_bytes) & (Fmt<TYPE>::kWords ? 3 : 1)) return cudaErrorMisalignedAddress;
  return launch_blocks<GgufTile<TYPE>>(p, bmap, n_tiles, st);
}

// The codebook table of this translation unit (gguf_gemv.cu holds its own copy of the pointer).
int set_iq_grids_gemm(const void* table) { return (int)cudaMemcpyToSymbol(kIqGrids, &table, sizeof(table)); }

}  // namespace ve

using namespace ve;

extern "C" {

// W: E experts of [N, row_bytes] GGUF rows back to back (16-bit aligned, formats with 4-byte fields 4-byte aligned); X [R, K] bf16 rows
// sorted by expert (pitch ldx, a multiple of 8); tile_tab [n_tiles][4] = {expert, first row, rows <= 128, 0}; out [R, N] bf16.
int ve_gemm_grouped_gguf(const void* W, int ggml_type, long row_bytes, const void* X, long ldx, void* out, long ldo, int R, int E, int N,
                         int K, const void* tile_tab, int n_tiles, void* status, cudaStream_t st) {
  if (R <= 0 || n_tiles <= 0) return 0;
  if (N <= 0 || K <= 0 || K % 32 || E <= 0) return cudaErrorInvalidValue;
  if (ggml_type >= kQ2_K && ggml_type != kIQ4_NL && K % 256) return cudaErrorInvalidValue;
  if (!iq_grids_ready(ggml_type)) return cudaErrorNotReady;
  CUtensorMap bmap;
  const int rc = make_tmap_2d(&bmap, X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, R, K, (uint64_t)ldx * 2, 32, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  const BlockGemmParams p{N, K, (const uint8_t*)W, row_bytes, (const uint8_t*)W + (size_t)E * N * row_bytes, (__nv_bfloat16*)out, ldo,
                          (const int*)tile_tab, (int*)status};
#define VE_CALL(T) launch_gguf_blocks<T>(p, bmap, n_tiles, st)
  VE_GGUF_TYPES(ggml_type, VE_CALL)
#undef VE_CALL
}

// codes: E experts of [K/16][N/16][16 * bits] uint16 back to back (16-byte aligned), N a multiple of 128; the rest as above.
int ve_gemm_grouped_exl3(const void* codes, int bits, int cb, const void* X, long ldx, void* out, long ldo, int R, int E, int N, int K,
                         const void* tile_tab, int n_tiles, void* status, cudaStream_t st) {
  if (R <= 0 || n_tiles <= 0) return 0;
  if (N <= 0 || K <= 0 || K % 16 || N % 128 || E <= 0 || cb < 0 || cb > 2) return cudaErrorInvalidValue;
  if ((uintptr_t)codes & 15) return cudaErrorMisalignedAddress;
  CUtensorMap bmap;
  const int rc = make_tmap_2d(&bmap, X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, R, K, (uint64_t)ldx * 2, 32, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  const long per = (long)(K / 16) * (N / 16) * 32 * bits;
  const BlockGemmParams p{N, K, (const uint8_t*)codes, per, (const uint8_t*)codes + (size_t)E * per, (__nv_bfloat16*)out, ldo,
                          (const int*)tile_tab, (int*)status};
#define VE_EX(B)                                                                            \
  case B:                                                                                   \
    return cb == 2 ? launch_blocks<Exl3Tile<B, 2>>(p, bmap, n_tiles, st)                    \
         : cb == 1 ? launch_blocks<Exl3Tile<B, 1>>(p, bmap, n_tiles, st)                    \
                   : launch_blocks<Exl3Tile<B, 0>>(p, bmap, n_tiles, st);
  switch (bits) {
    VE_EX(1) VE_EX(2) VE_EX(3) VE_EX(4) VE_EX(5) VE_EX(6) VE_EX(7) VE_EX(8)
    default: return cudaErrorInvalidValue;
  }
#undef VE_EX
}

}  // extern "C"
