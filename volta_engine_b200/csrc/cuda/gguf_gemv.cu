// GGUF block formats: dequantisation fused into the mat-vec (decode / verify rows, M <= 16) and a plain
// dequantise-to-bf16 kernel that feeds the tcgen05 GEMM for prefill chunks.
//   Q8_0, Q4_0, Q4_1, Q5_0, Q5_1, IQ4_NL (32-value blocks), Q2_K, Q3_K, Q4_K, Q5_K, Q6_K, IQ4_XS and the codebook
//   formats IQ1_S, IQ1_M, IQ2_XXS, IQ2_XS, IQ2_S, IQ3_XXS, IQ3_S (256-value super-blocks), bf16 activations, fp32
//   accumulation.
// Two orders of summation, each fixed by K alone, so that a row's result does not depend on M, on N or on what else is in the batch:
//   * gguf_mma_kernel: units of 256 weights (128 for Q8_0) dealt to eight warps, sums of a unit added up first, then a warp's units, then the
//     warps in order. The form for every format, unless the caller asks for the other.
//   * lane order (gguf_ordered_kernel; gguf_gemv_kernel and gguf_moe_gemv_kernel for blocks whose address the others cannot read): chunk c of 32
//     weights belongs to lane c % 32, its products are added one after the other, chunks in turn, lanes by a butterfly.
// Reference counterparts: src/kernels/cuda/gguf/gguf_linear.cu:38-160 (gemv on q8_1 activations) and the
// vendored dequantize kernels; block layouts as in quant/gguf.py.
#include "gguf_blocks.cuh"

namespace ve {

// Rows whose blocks lie at odd addresses (gguf_mma_kernel reads words): one warp per output row, a lane decodes 32 consecutive weights
// at a time byte by byte.
template <int TYPE>
__global__ void __launch_bounds__(256) gguf_gemv_kernel(const uint8_t* __restrict__ W, long row_bytes,
                                                        const __nv_bfloat16* __restrict__ x, long x_stride,
                                                        __nv_bfloat16* __restrict__ out, long out_stride,
                                                        float* __restrict__ out_f32, int M, int N, int K) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x * 8 + warp;
  if (n >= N) return;
  const uint8_t* row = W + (size_t)n * row_bytes;
  float acc[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) acc[m] = 0.f;
  const int chunks = K >> 5;
  for (int c = lane; c < chunks; c += 32) {
    float w[32];
    decode32<TYPE>(row, c, w);
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      if (m >= M) break;
      const __nv_bfloat16* xr = x + (long)m * x_stride + (long)c * 32;
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        const bf16x8 t = *reinterpret_cast<const bf16x8*>(xr + j);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 f = __bfloat1622float2(t.v[u]);
          s = fmaf(w[j + 2 * u], f.x, s);
          s = fmaf(w[j + 2 * u + 1], f.y, s);
        }
      }
      acc[m] += s;
    }
  }
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    if (m >= M) break;
    float v = warp_sum(acc[m]);
    if (lane == 0) {
      if (out_f32) out_f32[(long)m * out_stride + n] = v;
      else out[(long)m * out_stride + n] = f2bf(v);
    }
  }
}

// The same for routed experts: grid (output rows / 4 or / 8, routes), one warp per output
// row (FUSE: per gate / up pair, the gated activation applied before the store). W holds the experts of this rank back to
// back ([e_local][N][row_bytes]); route r reads activation row r / x_div and the expert ids[r] - e0; routes of experts
// that live elsewhere store zeros. The per-row sum runs in the order of the dense mat-vec (lane-strided 32-weight
// chunks, butterfly), so a route gives the same bits whatever else is in the batch.
template <int TYPE, int FUSE>
__global__ void __launch_bounds__(128) gguf_moe_gemv_kernel(const uint8_t* __restrict__ W, long row_bytes,
                                                            const int* __restrict__ ids, int e0, int e_local,
                                                            const __nv_bfloat16* __restrict__ x, long x_stride, int x_div,
                                                            __nv_bfloat16* __restrict__ out, long out_stride, int N, int K,
                                                            int act, float limit) {
  const int route = blockIdx.y;
  const int e = ids[route] - e0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half_n = N >> 1, n_out = FUSE ? half_n : N;
  const int r0 = blockIdx.x * 4 + warp;
  if (r0 >= n_out) return;
  if (e < 0 || e >= e_local) {
    if (lane == 0) out[(long)route * out_stride + r0] = f2bf(0.f);
    return;
  }
  const uint8_t* base = W + (size_t)e * N * row_bytes;
  const uint8_t* row0 = base + (size_t)r0 * row_bytes;
  const uint8_t* row1 = base + (size_t)(FUSE ? r0 + half_n : r0) * row_bytes;
  const __nv_bfloat16* xr = x + (long)(route / x_div) * x_stride;
  float acc0 = 0.f, acc1 = 0.f;
  const int chunks = K >> 5;
  for (int c = lane; c < chunks; c += 32) {
    float xv[32];
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      const bf16x8 t = *reinterpret_cast<const bf16x8*>(xr + (long)c * 32 + j);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 f = __bfloat1622float2(t.v[u]);
        xv[j + 2 * u] = f.x;
        xv[j + 2 * u + 1] = f.y;
      }
    }
    float w[32];
    decode32<TYPE>(row0, c, w);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) s = fmaf(w[j], xv[j], s);
    acc0 += s;
    if (FUSE) {
      decode32<TYPE>(row1, c, w);
      s = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j) s = fmaf(w[j], xv[j], s);
      acc1 += s;
    }
  }
  acc0 = warp_sum(acc0);
  if (FUSE) acc1 = warp_sum(acc1);
  if (lane != 0) return;
  if (FUSE) {
    // the unfused pair rounds both projections to bf16 before the activation: the same rounding points here
    float gate = bf2f(f2bf(acc0)), up = bf2f(f2bf(acc1));
    if (limit > 0.f) { gate = fminf(gate, limit); up = fminf(fmaxf(up, -limit), limit); }
    const float a = act ? 0.5f * gate * (1.f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate)))
                        : gate / (1.f + __expf(-gate));
    out[(long)route * out_stride + r0] = f2bf(a * up);
  } else {
    out[(long)route * out_stride + r0] = f2bf(acc0);
  }
}

// One product of a packed row with one row of x by a warp, in the order of the two kernels above. For sums whose tensor-core form is not
// finite: an infinite or huge activation meets the block's integers there before their scale and minimum, so it gave NaN (0 * inf, or
// inf - inf between s * q and m) or an overflow where the sum over the weights themselves is an infinity or a number.
template <int TYPE>
__device__ __noinline__ float ordered_dot(const uint8_t* __restrict__ row, const __nv_bfloat16* __restrict__ xr, int chunks) {
  const int lane = threadIdx.x & 31;
  float acc = 0.f;
  for (int c = lane; c < chunks; c += 32) {
    float w[32];
    decode32<TYPE>(row, c, w);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      const bf16x8 t = *reinterpret_cast<const bf16x8*>(xr + (long)c * 32 + j);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 f = __bfloat1622float2(t.v[u]);
        s = fmaf(w[j + 2 * u], f.x, s);
        s = fmaf(w[j + 2 * u + 1], f.y, s);
      }
    }
    acc += s;
  }
  return warp_sum(acc);
}
VE_DEVINL bool not_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u; }

struct GgufGemvArgs {
  const uint8_t* W; long row_bytes; const uint8_t* W_end;
  const __nv_bfloat16* x; long x_stride;
  __nv_bfloat16* out; float* out_f32; long out_stride;
  int M, N, K, tiles;
  // routed experts: route r reads activation row r / x_div and expert ids[r] - e0 of the bank; a route of another rank's expert gives zeros
  const int* ids; int e0, e_local, x_div, act, tiles_per_route;
  float limit;
};

// MODE 0: out[m, n] = sum_k W[n, k] x[m, k] for up to 8 * NT rows m. MODE 1: the same for routed experts, one activation row a route.
// MODE 2: routed gate / up pair, gate in rows n and up in rows N / 2 + n of the expert, the gated activation applied before the store.
//
// A tile is 16 * RT weight rows (MODE 2: eight gate and eight up rows). The eight warps of a block deal its units of 256 weights along K
// (128 for Q8_0) between them; each warp copies its units through a ring of its own with 16-byte cp.async and turns them into operand
// fragments, whose products with all activation rows are one tensor-core instruction per 16 weights. Blocks are persistent over tiles and the
// ring runs on into the next tile. What bounds it is issuing: 34816 x 5120 Q4_K at four rows
// takes 6.4 instructions a weight, 62 % of the issue slots of 16 warps an SM, at a quarter of the copy rate (decoding, the activations of every
// row tile and the scales; next come waits for dependent results and for the barrier behind a tile). A lane that decoded 32 consecutive weights of its own straight from global memory (one warp a row) read
// single bytes up to 4352 bytes apart and multiplied every row of x in fp32: 365 us for the average matrix of a 27B-class Q4_K layer at
// four rows, 538 us for Q8_0 at eight rows of the larger latent-attention shapes.
template <int TYPE, int MODE, int NT, int RT>
struct GemvCfg {
  using F = Fmt<TYPE>;
  static constexpr int kPitch = ((F::kUnit + 14 + 15) / 16 | 1) * 16;     // 16-byte pieces of a row's unit at any 2-byte offset; odd: no bank conflicts
  static constexpr int kStage = 16 * RT * kPitch;
  static constexpr int kStages = RT == 2 ? 2 : 3;
  static constexpr int kCols = MODE == 0 ? 8 * NT : 1;
  static constexpr int kRed = 8 * 16 * RT * kCols;                          // floats, one of two buffers
  static constexpr int kTab = (F::kTabBytes + 15) / 16 * 16;
  static constexpr int kSmem = kTab + 2 * kRed * 4 + 8 * kStages * kStage;
};

template <int TYPE, int MODE, int NT, int RT>
__global__ void __launch_bounds__(256, 2) gguf_mma_kernel(const GgufGemvArgs p) {
  using F = Fmt<TYPE>;
  using C = GemvCfg<TYPE, MODE, NT, RT>;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* const tab = smem_raw;
  float* const red = reinterpret_cast<float*>(smem_raw + C::kTab);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint8_t* const ring = smem_raw + C::kTab + 2 * C::kRed * 4 + warp * C::kStages * C::kStage;
  if (C::kTab) load_table<TYPE>(tab);
  if (MODE != 0) grid_dep_wait();                       // the routes come from the kernel in front (weights do not: MODE 0 starts on them)

  const int chunks = p.K >> 5;
  const int units = (chunks + F::kChunks - 1) / F::kChunks;
  const int mine = warp < units ? (units - warp + 7) / 8 : 0;            // units warp, warp + 8, ...
  const int ntile = (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int items = mine * ntile;
  const int half_n = p.N >> 1;

  // rows of this lane's quad in tile i: 2 * RT of them (fragment rows g and g + 8); false: the tile's expert is not here
  auto rows_of = [&](int i, const uint8_t** rp) -> bool {
    int tile = (int)blockIdx.x + i * (int)gridDim.x;
    const uint8_t* base = p.W;
    if (MODE != 0) {
      const int route = tile / p.tiles_per_route;
      tile -= route * p.tiles_per_route;
      const int e = p.ids[route] - p.e0;
      if (e < 0 || e >= p.e_local) return false;
      base += (size_t)e * p.N * p.row_bytes;
    }
#pragma unroll
    for (int r = 0; r < 2 * RT; ++r) {
      int n;
      if (MODE == 2) n = min(tile * 8 + g, half_n - 1) + r * half_n;
      else n = min(tile * 16 * RT + r * 8 + g, p.N - 1);                  // rows behind the matrix repeat its last one
      rp[r] = base + (size_t)n * p.row_bytes;
    }
    return true;
  };
  const uint8_t* lp[2 * RT];                            // rows of the tile being loaded
  bool l_here = false;
  int l_tile = -1, l_item = 0;
  auto load = [&]() {                                   // the next unit into its ring stage
    if (l_item < items) {
      const int ti = l_item / mine, ui = warp + 8 * (l_item - ti * mine);
      if (ti != l_tile) { l_here = rows_of(ti, lp); l_tile = ti; }
      if (l_here) {
        const int bytes = F::kBig ? F::kBytes : min(F::kChunks, chunks - ui * F::kChunks) * F::kBytes;
        uint8_t* dst = ring + (l_item % C::kStages) * C::kStage;
#pragma unroll
        for (int r = 0; r < 2 * RT; ++r) {
          const uint8_t* src = lp[r] + (size_t)ui * F::kUnit;
          const int off = (int)((uintptr_t)src & 15);   // whole 16-byte pieces: they lie inside the allocation, but for a piece that
          src -= off;                                     // the matrix ends in, which is cut there
          const int n16 = (off + bytes + 15) >> 4;
          for (int j = t; j < n16; j += 4) {
            const long left = p.W_end - (src + j * 16);
            cp_async16(dst + (r * 8 + g) * C::kPitch + j * 16, src + j * 16, left < 16 ? (int)left : 16);
          }
        }
      }
    }
    ++l_item;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < C::kStages - 1; ++s) load();
  if (C::kTab) __syncthreads();
  if (MODE == 0) grid_dep_wait();

  int item = 0;
  for (int ti = 0; ti < ntile; ++ti) {
    const int tile = (int)blockIdx.x + ti * (int)gridDim.x;
    if (ti == ntile - 1) grid_dep_launch();              // (blocks of the kernel behind would wait beside this one's and slow it)
    const uint8_t* rp[2 * RT];
    const bool here = rows_of(ti, rp);
    const __nv_bfloat16* xr = p.x + (MODE != 0 ? (long)(tile / p.tiles_per_route / p.x_div) * p.x_stride : 0) + (F::kVec8 ? 8 : 4) * t;
    float acc[RT][NT][4];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    for (int w = 0; w < mine; ++w, ++item) {
      asm volatile("cp.async.wait_group %0;" ::"n"(C::kStages - 2) : "memory");
      __syncwarp();                                       // every lane's pieces are here, and every lane is done with the stage in front
      load();
      if (!here) continue;
      const uint8_t* st = ring + (item % C::kStages) * C::kStage;
      const int ui = warp + 8 * w, c0 = ui * F::kChunks;
      const uint8_t* up[2 * RT];
#pragma unroll
      for (int r = 0; r < 2 * RT; ++r)
        up[r] = st + (r * 8 + g) * C::kPitch + (int)((uintptr_t)(rp[r] + (size_t)ui * F::kUnit) & 15);
      float blk[RT][NT][4];                               // sums of the unit
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) blk[i][j][e] = 0.f;
#pragma unroll
      for (int h = 0; h < F::kChunks; h += 4) {
        uint2 xv[4][NT][2];                               // this lane's activations of four chunks
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const bool live = (MODE != 0 ? g == 0 : j * 8 + g < p.M) && (F::kBig || c0 + h + c < chunks);
            const __nv_bfloat16* q = xr + (MODE == 0 ? (long)(j * 8 + g) * p.x_stride : 0) + (long)(c0 + h + c) * 32;
            if (F::kVec8) {
              const uint4 v = live ? *reinterpret_cast<const uint4*>(q) : make_uint4(0u, 0u, 0u, 0u);
              xv[c][j][0] = make_uint2(v.x, v.y);
              xv[c][j][1] = make_uint2(v.z, v.w);
            } else {
              xv[c][j][0] = live ? *reinterpret_cast<const uint2*>(q) : make_uint2(0u, 0u);
              xv[c][j][1] = live ? *reinterpret_cast<const uint2*>(q + 16) : make_uint2(0u, 0u);
            }
          }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (!F::kBig && c0 + h + c >= chunks) break;
          if constexpr (F::kVec8) {                       // the block's products are summed before its one scale
#pragma unroll
            for (int i = 0; i < RT; ++i) {
              uint32_t f[2][4];
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                uint32_t lut;
                const uint32_t codes = vec8_codes<TYPE>(up[2 * i + r], h + c, t, tab, lut);
                const uint2 v = reinterpret_cast<const uint2*>(tab + 8192)[lut];
                vec8_expand(codes, v.x, v.y, f[r]);
              }
#pragma unroll
              for (int j = 0; j < NT; ++j) {
                mma_bf16_16816(blk[i][j], f[0][0], f[1][0], f[0][1], f[1][1], xv[c][j][0].x, xv[c][j][0].y);
                mma_bf16_16816(blk[i][j], f[0][2], f[1][2], f[0][3], f[1][3], xv[c][j][1].x, xv[c][j][1].y);
              }
            }
          } else {
          float sx[NT][2][2];                             // sums of x over the group (formats with minima), columns 2 t and 2 t + 1
          if (F::kMin) {
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              constexpr uint32_t one = 0x3F803F80u;
              float d[4] = {0.f, 0.f, 0.f, 0.f};
              mma_bf16_16816(d, one, one, one, one, xv[c][j][0].x, xv[c][j][0].y);
              if (F::kMin == 2) { sx[j][0][0] = d[0]; sx[j][0][1] = d[1]; d[0] = d[1] = d[2] = d[3] = 0.f; }
              mma_bf16_16816(d, one, one, one, one, xv[c][j][1].x, xv[c][j][1].y);
              sx[j][F::kMin - 1][0] = d[0]; sx[j][F::kMin - 1][1] = d[1];
            }
          }
#pragma unroll
          for (int i = 0; i < RT; ++i) {
            uint32_t fa[4], fb[4];
            float sa[2], sb[2], ma[2], mb[2];
            frag<TYPE>(up[2 * i], h + c, t, tab, fa, sa, ma);
            frag<TYPE>(up[2 * i + 1], h + c, t, tab, fb, sb, mb);
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              float* ac = blk[i][j];
              float d[4] = {0.f, 0.f, 0.f, 0.f};
              mma_bf16_16816(d, fa[0], fb[0], fa[1], fb[1], xv[c][j][0].x, xv[c][j][0].y);
              if (F::kScale16) {
                ac[0] = fmaf(sa[0], d[0], ac[0]); ac[1] = fmaf(sa[0], d[1], ac[1]);
                ac[2] = fmaf(sb[0], d[2], ac[2]); ac[3] = fmaf(sb[0], d[3], ac[3]);
                d[0] = d[1] = d[2] = d[3] = 0.f;
              }
              mma_bf16_16816(d, fa[2], fb[2], fa[3], fb[3], xv[c][j][1].x, xv[c][j][1].y);
              constexpr int q = F::kScale16 ? 1 : 0;
              ac[0] = fmaf(sa[q], d[0], ac[0]); ac[1] = fmaf(sa[q], d[1], ac[1]);
              ac[2] = fmaf(sb[q], d[2], ac[2]); ac[3] = fmaf(sb[q], d[3], ac[3]);
#pragma unroll
              for (int k = 0; k < F::kMin; ++k) {
                ac[0] = fmaf(-ma[k], sx[j][k][0], ac[0]); ac[1] = fmaf(-ma[k], sx[j][k][1], ac[1]);
                ac[2] = fmaf(-mb[k], sx[j][k][0], ac[2]); ac[3] = fmaf(-mb[k], sx[j][k][1], ac[3]);
              }
            }
          }
          }
        }
      }
      if constexpr (F::kVec8) {
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          const float da = vec8_scale<TYPE>(up[2 * i]), db = vec8_scale<TYPE>(up[2 * i + 1]);
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            float* ac = acc[i][j];
            ac[0] = fmaf(da, blk[i][j][0], ac[0]); ac[1] = fmaf(da, blk[i][j][1], ac[1]);
            ac[2] = fmaf(db, blk[i][j][2], ac[2]); ac[3] = fmaf(db, blk[i][j][3], ac[3]);
          }
        }
      } else {                                            // (in two levels: one chain over all of K rounds off twice as much at K = 17408)
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] += blk[i][j][e];
      }
    }
    // warp sums -> shared memory [warp][column][row], added in warp order
    float* rb = red + (ti & 1) * C::kRed;
    if (MODE == 0) {
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            rb[(warp * C::kCols + j * 8 + 2 * t + (e & 1)) * 16 * RT + i * 16 + (e >> 1) * 8 + g] = acc[i][j][e];
    } else if (t == 0) {
      rb[warp * 16 + g] = acc[0][0][0];
      rb[warp * 16 + 8 + g] = acc[0][0][2];
    }
    __syncthreads();                                      // (the other buffer's sums were read in front of this barrier)
    const int nw = min(8, units);
    // sums that are not finite are formed again by their warp (all lanes take part), weight by weight
    auto again = [&](float v, bool bad, auto row_of, auto x_of) {
      for (uint32_t left = __ballot_sync(0xffffffffu, bad); left; left &= left - 1) {
        const int src = __ffs(left) - 1;
        const float d = ordered_dot<TYPE>(row_of(src), x_of(src), chunks);
        if (lane == src) v = d;
      }
      return v;
    };
    if (MODE == 0) {
      for (int i = threadIdx.x; i < 16 * RT * C::kCols; i += 256) {          // (whole warps: a multiple of 32)
        const int row = i % (16 * RT), m = i / (16 * RT), n = tile * 16 * RT + row;
        const bool in = m < p.M && n < p.N;
        float v = 0.f;
        for (int w = 0; w < nw; ++w) v += rb[w * C::kRed / 8 + i];
        v = again(v, in && not_finite(v), [&](int src) { return p.W + (size_t)(tile * 16 * RT + (i - lane + src) % (16 * RT)) * p.row_bytes; },
                  [&](int src) { return p.x + (long)((i - lane + src) / (16 * RT)) * p.x_stride; });
        if (in) {
          if (p.out_f32) p.out_f32[(long)m * p.out_stride + n] = v;
          else p.out[(long)m * p.out_stride + n] = f2bf(v);
        }
      }
    } else if (warp == 0) {
      constexpr int per = MODE == 2 ? 8 : 16;
      const int route = tile / p.tiles_per_route, n0 = (tile - route * p.tiles_per_route) * per, n = n0 + lane, n_out = MODE == 2 ? half_n : p.N;
      const bool in = lane < per && n < n_out;
      float v = 0.f, u = 0.f;
      if (here) {
        if (in)
          for (int w = 0; w < nw; ++w) {
            v += rb[w * 16 + lane];
            if (MODE == 2) u += rb[w * 16 + 8 + lane];
          }
        const uint8_t* base = p.W + (size_t)(p.ids[route] - p.e0) * p.N * p.row_bytes;
        auto x_of = [&](int) { return p.x + (long)(route / p.x_div) * p.x_stride; };
        v = again(v, in && not_finite(v), [&](int src) { return base + (size_t)(n0 + src) * p.row_bytes; }, x_of);
        if (MODE == 2) {
          u = again(u, in && not_finite(u), [&](int src) { return base + (size_t)(n0 + src + half_n) * p.row_bytes; }, x_of);
          // the unfused pair rounds both projections to bf16 before the activation: the same rounding points here
          float gate = bf2f(f2bf(v)), upv = bf2f(f2bf(u));
          if (p.limit > 0.f) { gate = fminf(gate, p.limit); upv = fminf(fmaxf(upv, -p.limit), p.limit); }
          v = (p.act ? 0.5f * gate * (1.f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate)))
                     : gate / (1.f + __expf(-gate))) * upv;
        }
      }
      if (in) p.out[(long)route * p.out_stride + n] = f2bf(v);
    }
  }
}

// The mat-vecs in scalar fp32 and in lane order, bit for bit the sums of gguf_gemv_kernel and gguf_moe_gemv_kernel, for callers that ask for it:
// models whose router picks groups of experts first. At such a router's edge any change of rounding in front of it picks other experts, for about
// one token in a hundred with the sums of gguf_mma_kernel, although their error against 64 bits is no larger.
// Times (gguf_mma_kernel in brackets): 7168 x 16384 Q8_0 one row 58 us (65), eight 127 us (62); Q4_K 72 (44) and 137 us (42); gate / up and down of 64
// routes of 2048 x 7168 IQ1_M 944 us (750), Q4_K 1217 us (870), Q8_0 965 us (1270). The byte-by-byte kernels: 174 and 999 us, 165 and 987 us; 2121,
// 2578 and 2638 us. Bound by issuing: IQ1_M takes 10.1 instructions a weight, 84 % of the issue slots.
// A warp takes two rows (MODE 2: a gate and an up row); steps of 1024 weights of its rows and of x come through double buffers by 16-byte
// cp.async, x chunks 80 bytes apart (no bank conflicts). Q8_0 and IQ1_M have decoders of whole words, the other formats go byte by byte.
template <int TYPE, int MT>
struct OrderedCfg {
  static constexpr int kStepBytes = Fmt<TYPE>::kBig ? 4 * Fmt<TYPE>::kBytes : 32 * Fmt<TYPE>::kBytes;
  static constexpr int kPitch = (kStepBytes + 15 + 15) / 16 * 16;
  static constexpr int kTab = TYPE == kIQ1_M ? (Fmt<TYPE>::kTabBytes + 15) / 16 * 16 : 0;
  static constexpr int kX = 32 * 80;                                          // a step of one row of x
  static constexpr int kSmem = kTab + 2 * MT * kX + 8 * 2 * 2 * kPitch;
};

template <int TYPE, int MODE, int MT>
__global__ void __launch_bounds__(256) gguf_ordered_kernel(const GgufGemvArgs p) {
  using C = OrderedCfg<TYPE, MT>;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* const tab = smem_raw;
  uint8_t* const xs = smem_raw + C::kTab;                                     // [2][MT][kX]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* const ws = xs + 2 * MT * C::kX + warp * 2 * 2 * C::kPitch;         // [2][2 rows][kPitch]
  if (C::kTab) load_table<TYPE>(tab);
  if (MODE != 0) grid_dep_wait();
  const int route = blockIdx.y;
  int e = 0;
  if (MODE != 0) e = p.ids[route] - p.e0;
  const bool here = MODE == 0 || (e >= 0 && e < p.e_local);
  const int half_n = p.N >> 1, n_out = MODE == 2 ? half_n : p.N;
  const int tiles = (n_out + (MODE == 2 ? 7 : 15)) / (MODE == 2 ? 8 : 16);
  const __nv_bfloat16* x = p.x + (MODE != 0 ? (long)(route / p.x_div) * p.x_stride : 0);
  const int chunks = p.K >> 5, steps = (chunks + 31) / 32, M = MODE != 0 ? 1 : p.M;
  bool waited = MODE != 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int first = tile * (MODE == 2 ? 8 : 16) + warp * (MODE == 2 ? 1 : 2);
    const uint8_t* rp[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int n = MODE == 2 ? min(first, half_n - 1) + r * half_n : min(first + r, p.N - 1);
      rp[r] = p.W + ((size_t)(here ? e : 0) * p.N + n) * p.row_bytes;
    }
    auto load_w = [&](int i) {
      const int bytes = (Fmt<TYPE>::kBig ? min(4, (chunks - i * 32) / 8) : min(32, chunks - i * 32)) * Fmt<TYPE>::kBytes;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint8_t* src = rp[r] + (size_t)i * C::kStepBytes;
        const int off = (int)((uintptr_t)src & 15);       // whole 16-byte pieces: inside the allocation, but for the one the matrix ends in
        src -= off;
        uint8_t* dst = ws + ((i & 1) * 2 + r) * C::kPitch;
        for (int j = lane; j < (off + bytes + 15) >> 4; j += 32) {
          const long left = p.W_end - (src + j * 16);
          cp_async16(dst + j * 16, src + j * 16, left < 16 ? (int)left : 16);
        }
      }
    };
    auto load_x = [&](int i) {
      const int n = min(32, chunks - i * 32) * 4;         // 16-byte pieces of a row
      for (int j = threadIdx.x; j < M * 128; j += 256) {
        const int m = j >> 7, c = j & 127;
        if (c < n)
          cp_async16(xs + ((i & 1) * MT + m) * C::kX + (c >> 2) * 80 + (c & 3) * 16, x + (long)m * p.x_stride + (long)i * 1024 + c * 8);
      }
    };
    float acc[2][MT];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int m = 0; m < MT; ++m) acc[r][m] = 0.f;
    if (here) {
      load_w(0);
      if (!waited) { grid_dep_wait(); waited = true; }
      load_x(0);
      asm volatile("cp.async.commit_group;" ::: "memory");
      for (int i = 0; i < steps; ++i) {
        if (i + 1 < steps) { load_w(i + 1); load_x(i + 1); }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                  // this step is here for every thread
        if (i * 32 + lane < chunks) {
          float w[2][32];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const uint8_t* b = ws + ((i & 1) * 2 + r) * C::kPitch + (int)((uintptr_t)(rp[r] + (size_t)i * C::kStepBytes) & 15);
            if constexpr (TYPE == kQ8_0) {
              b += lane * 34;
              const uint32_t* q = reinterpret_cast<const uint32_t*>((uintptr_t)b & ~(uintptr_t)3);
              const int sh = (int)((uintptr_t)b & 2) * 8;
              uint32_t v[9];
#pragma unroll
              for (int j = 0; j < 9; ++j) v[j] = q[j];
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] = __funnelshift_r(v[j], v[j + 1], sh);
              v[8] >>= sh;
              const float d = __half2float(__ushort_as_half((unsigned short)v[0]));
#pragma unroll
              for (int j = 0; j < 32; ++j) {               // byte j + 2: 2^23 + 128 + value, less 2^23 + 128
                const uint32_t u = v[(j + 2) >> 2] ^ 0x80808080u;
                w[r][j] = d * (__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7440u | ((j + 2) & 3))) - 8388736.f);
              }
            } else if constexpr (TYPE == kIQ1_M) {
              b += (lane >> 3) * 56;
              const int c = lane & 7;
              const uint32_t qs = ld32<true>(b + c * 4), qh = ld16(b + 32 + 2 * c);
              const float d = vec8_scale<TYPE>(b);
              const uint32_t sw = ld16(b + 48 + 2 * (c >> 1)) >> (6 * (c & 1));
              const float dl[2] = {d * u2f(2 * (sw & 7) + 1), d * u2f(2 * ((sw >> 3) & 7) + 1)};
#pragma unroll
              for (int l = 0; l < 4; ++l) {
                const uint32_t h = qh >> (4 * l);
                const uint32_t codes = reinterpret_cast<const uint32_t*>(tab)[((qs >> (8 * l)) & 255) | ((h & 7) << 8)];
                const uint2 val = reinterpret_cast<const uint2*>(tab + 8192)[h & 8];
                uint32_t f[4];
                vec8_expand(codes, val.x, val.y, f);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  w[r][8 * l + 2 * j] = dl[l >> 1] * __uint_as_float(f[j] << 16);
                  w[r][8 * l + 2 * j + 1] = dl[l >> 1] * __uint_as_float(f[j] & 0xffff0000u);
                }
              }
            } else {
              decode32<TYPE>(b, lane, w[r]);
            }
          }
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            if (m >= M) break;
            const uint4* xv = reinterpret_cast<const uint4*>(xs + ((i & 1) * MT + m) * C::kX + lane * 80);
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 t = xv[j];
              const uint32_t u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float lo = __uint_as_float(u[k] << 16), hi = __uint_as_float(u[k] & 0xffff0000u);
                s0 = fmaf(w[0][8 * j + 2 * k], lo, s0);
                s1 = fmaf(w[1][8 * j + 2 * k], lo, s1);
                s0 = fmaf(w[0][8 * j + 2 * k + 1], hi, s0);
                s1 = fmaf(w[1][8 * j + 2 * k + 1], hi, s1);
              }
            }
            acc[0][m] += s0;
            acc[1][m] += s1;
          }
        }
        __syncthreads();                                  // every thread is done with the buffers that the next round fills
      }
    }
    if (tile + (int)gridDim.x >= tiles) grid_dep_launch();
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      if (m >= M) break;
      const float v0 = warp_sum(acc[0][m]), v1 = warp_sum(acc[1][m]);
      if (lane != 0) continue;
      if (MODE == 2) {
        // the unfused pair rounds both projections to bf16 before the activation: the same rounding points here
        float gate = bf2f(f2bf(v0)), up = bf2f(f2bf(v1));
        if (p.limit > 0.f) { gate = fminf(gate, p.limit); up = fminf(fmaxf(up, -p.limit), p.limit); }
        const float a = p.act ? 0.5f * gate * (1.f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate)))
                              : gate / (1.f + __expf(-gate));
        if (first < n_out) p.out[(long)route * p.out_stride + first] = f2bf(here ? a * up : 0.f);
      } else {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          if (first + r >= n_out) continue;
          const long at = (long)(MODE == 1 ? route : m) * p.out_stride + first + r;
          const float v = r ? v1 : v0;
          if (MODE == 0 && p.out_f32) p.out_f32[at] = v;
          else p.out[at] = f2bf(v);
        }
      }
    }
  }
}

template <int TYPE>
__global__ void gguf_dequant_kernel(const uint8_t* __restrict__ W, long row_bytes, __nv_bfloat16* __restrict__ out,
                                    long N, int K) {
  const int chunks = K >> 5;
  const long total = N * chunks;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long n = i / chunks;
    const int c = (int)(i % chunks);
    float w[32];
    decode32<TYPE>(W + (size_t)n * row_bytes, c, w);
    __nv_bfloat16* o = out + n * (long)K + (long)c * 32;
#pragma unroll
    for (int j = 0; j < 32; j += 2) *reinterpret_cast<__nv_bfloat162*>(o + j) = __floats2bfloat162_rn(w[j], w[j + 1]);
  }
}

}  // namespace ve

using namespace ve;

template <int TYPE, int MODE, int NT, int RT>
static int launch_gguf_mma(GgufGemvArgs a, cudaStream_t st) {
  using C = GemvCfg<TYPE, MODE, NT, RT>;
  static_assert(C::kSmem <= 200 * 1024, "shared memory of an SM");
  static int per_sm = 0;                                 // resident blocks an SM, found once (the same on every B200)
  int n = per_sm;
  const cudaError_t a_rc = allow_smem<gguf_mma_kernel<TYPE, MODE, NT, RT>>(C::kSmem);
  if (a_rc != cudaSuccess) return (int)a_rc;
  if (n == 0) {
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gguf_mma_kernel<TYPE, MODE, NT, RT>, 256, C::kSmem);
    if (e != cudaSuccess) return (int)e;
    if (n < 1) n = 1;
    per_sm = n;
  }
  const int grid = a.tiles < 148 * n ? a.tiles : 148 * n;
  launch_pdl(gguf_mma_kernel<TYPE, MODE, NT, RT>, dim3(grid), dim3(256), C::kSmem, st, a);
  VE_CHECK_LAUNCH();
}

template <int TYPE, int MODE, int MT>
static int launch_gguf_ordered(const GgufGemvArgs& a, int routes, cudaStream_t st) {
  constexpr int smem = OrderedCfg<TYPE, MT>::kSmem;
  const cudaError_t e = allow_smem<gguf_ordered_kernel<TYPE, MODE, MT>>(smem);
  if (e != cudaSuccess) return (int)e;
  const int per = MODE == 2 ? 8 : 16, n = MODE == 2 ? a.N / 2 : a.N;
  // routed: up to eight tiles a block, so that the codebook is laid out once for them, as long as every SM keeps eight blocks
  const int tiles = (n + per - 1) / per;
  long share = MODE == 0 ? 1 : (long)tiles * routes / (148 * 8);
  share = share < 1 ? 1 : share > 8 ? 8 : share;
  launch_pdl(gguf_ordered_kernel<TYPE, MODE, MT>, dim3((unsigned)((tiles + share - 1) / share), routes), dim3(256), smem, st, a);
  VE_CHECK_LAUNCH();
}

// fields of a block are read from shared memory in words of their natural alignment, which the row addresses must keep
template <int TYPE>
static bool block_aligned(const void* W, long row_bytes) {
  return (((uintptr_t)W | (uintptr_t)row_bytes) & (Fmt<TYPE>::kWords ? 3 : 1)) == 0;
}

template <int TYPE>
static int run_gguf_gemv(GgufGemvArgs a, int ordered, cudaStream_t st) {
  if (!block_aligned<TYPE>(a.W, a.row_bytes)) {          // blocks at odd addresses: byte by byte
    gguf_gemv_kernel<TYPE><<<(a.N + 7) / 8, 256, 0, st>>>(a.W, a.row_bytes, a.x, a.x_stride, a.out, a.out_stride, a.out_f32, a.M, a.N, a.K);
    VE_CHECK_LAUNCH();
  }
  if (ordered)
    return a.M == 1 ? launch_gguf_ordered<TYPE, 0, 1>(a, 1, st) : a.M <= 4 ? launch_gguf_ordered<TYPE, 0, 4>(a, 1, st)
         : a.M <= 8 ? launch_gguf_ordered<TYPE, 0, 8>(a, 1, st) : launch_gguf_ordered<TYPE, 0, 16>(a, 1, st);
  // 32 weight rows a tile where several rows of x would otherwise be read again for every 16 of a large matrix; the sums are the same
  a.tiles = (a.N + 15) / 16;
  if (a.M <= 4 || (a.M <= 8 && a.N < 32 * 148)) return launch_gguf_mma<TYPE, 0, 1, 1>(a, st);
  a.tiles = (a.N + 31) / 32;
  if (a.M <= 8) return launch_gguf_mma<TYPE, 0, 1, 2>(a, st);
  return launch_gguf_mma<TYPE, 0, 2, 2>(a, st);
}

template <int TYPE>
static int run_gguf_moe(GgufGemvArgs a, int routes, int fuse_act, int ordered, cudaStream_t st) {
  if (!block_aligned<TYPE>(a.W, a.row_bytes)) {
    const dim3 grid(((fuse_act ? a.N / 2 : a.N) + 3) / 4, routes);
    if (fuse_act)
      gguf_moe_gemv_kernel<TYPE, 1><<<grid, 128, 0, st>>>(a.W, a.row_bytes, a.ids, a.e0, a.e_local, a.x, a.x_stride, a.x_div, a.out,
                                                          a.out_stride, a.N, a.K, a.act, a.limit);
    else
      gguf_moe_gemv_kernel<TYPE, 0><<<grid, 128, 0, st>>>(a.W, a.row_bytes, a.ids, a.e0, a.e_local, a.x, a.x_stride, a.x_div, a.out,
                                                          a.out_stride, a.N, a.K, a.act, a.limit);
    VE_CHECK_LAUNCH();
  }
  if (ordered) return fuse_act ? launch_gguf_ordered<TYPE, 2, 1>(a, routes, st) : launch_gguf_ordered<TYPE, 1, 1>(a, routes, st);
  a.tiles_per_route = fuse_act ? (a.N / 2 + 7) / 8 : (a.N + 15) / 16;
  a.tiles = a.tiles_per_route * routes;
  return fuse_act ? launch_gguf_mma<TYPE, 2, 1, 1>(a, st) : launch_gguf_mma<TYPE, 1, 1, 1>(a, st);
}

template <int TYPE>
static int run_gguf_dequant(const uint8_t* W, long row_bytes, __nv_bfloat16* out, long N, int K, cudaStream_t st) {
  const long total = N * (K / 32);
  const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
  gguf_dequant_kernel<TYPE><<<blocks, 256, 0, st>>>(W, row_bytes, out, N, K);
  VE_CHECK_LAUNCH();
}

// which devices have had their grid table set (a codebook format launched without it would read through a null pointer)
static bool g_iq_ready[64];

static bool iq_type(int t) {
  return t == kIQ2_XXS || t == kIQ2_XS || t == kIQ2_S || t == kIQ3_XXS || t == kIQ3_S || t == kIQ1_S || t == kIQ1_M;
}
namespace ve {
bool iq_grids_ready(int ggml_type) {
  int dev = 0;
  return !iq_type(ggml_type) || (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && g_iq_ready[dev]);
}
}  // namespace ve

extern "C" {

// `table`: device copy (on the current device, 16-byte aligned, 33920 bytes) of the grid file; it must outlive every launch.
int ve_gguf_set_iq_grids(const void* table) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= 64 || !table || ((uintptr_t)table & 15)) return cudaErrorInvalidValue;
  e = cudaMemcpyToSymbol(kIqGrids, &table, sizeof(table));
  if (e != cudaSuccess) return (int)e;
  const int rc = set_iq_grids_gemm(table);
  if (rc) return rc;
  g_iq_ready[dev] = true;
  return 0;
}

// ordered: sums in lane order (see gguf_ordered_kernel).
int ve_gguf_gemv(const void* W, int ggml_type, long row_bytes, const void* x, long x_stride, void* out, long out_stride,
                 int out_is_f32, int M, int N, int K, int ordered, cudaStream_t st) {
  if (M <= 0 || M > 16 || N <= 0 || K % 32) return cudaErrorInvalidValue;
  if (ggml_type >= kQ2_K && ggml_type != kIQ4_NL && K % 256) return cudaErrorInvalidValue;
  if (!iq_grids_ready(ggml_type)) return cudaErrorNotReady;
  GgufGemvArgs a{(const uint8_t*)W, row_bytes, (const uint8_t*)W + (size_t)N * row_bytes, (const __nv_bfloat16*)x, x_stride,
                 out_is_f32 ? nullptr : (__nv_bfloat16*)out, out_is_f32 ? (float*)out : nullptr, out_stride, M, N, K};
#define VE_CALL(T) run_gguf_gemv<T>(a, ordered, st)
  VE_GGUF_TYPES(ggml_type, VE_CALL)
#undef VE_CALL
}

// Routed-expert mat-vec over GGUF blocks; see gguf_moe_gemv_kernel. fuse_act: W rows are [gate (N/2) | up (N/2)] and the
// output has N/2 columns act(gate) * up (act 0 SiLU, 1 tanh-GELU; limit > 0 clamps gate from above and up to +-limit).
int ve_gguf_moe_gemv(const void* W, int ggml_type, long row_bytes, const void* ids, int e0, int e_local, const void* x,
                     long x_stride, int x_div, void* out, long out_stride, int routes, int N, int K, int fuse_act, int act,
                     float limit, int ordered, cudaStream_t st) {
  if (routes <= 0) return 0;
  if (N <= 0 || K % 32 || x_div <= 0 || (fuse_act && N % 2)) return cudaErrorInvalidValue;
  if (ggml_type >= kQ2_K && ggml_type != kIQ4_NL && K % 256) return cudaErrorInvalidValue;
  if (!iq_grids_ready(ggml_type)) return cudaErrorNotReady;
  GgufGemvArgs a{(const uint8_t*)W, row_bytes, (const uint8_t*)W + (size_t)e_local * N * row_bytes, (const __nv_bfloat16*)x, x_stride,
                 (__nv_bfloat16*)out, nullptr, out_stride, 1, N, K, 0, (const int*)ids, e0, e_local, x_div, act, 0, limit};
#define VE_CALL(T) run_gguf_moe<T>(a, routes, fuse_act, ordered, st)
  VE_GGUF_TYPES(ggml_type, VE_CALL)
#undef VE_CALL
}

int ve_gguf_dequant(const void* W, int ggml_type, long row_bytes, void* out, long N, int K, cudaStream_t st) {
  if (N <= 0 || K % 32) return cudaErrorInvalidValue;
  if (ggml_type >= kQ2_K && ggml_type != kIQ4_NL && K % 256) return cudaErrorInvalidValue;
  if (!iq_grids_ready(ggml_type)) return cudaErrorNotReady;
#define VE_CALL(T) run_gguf_dequant<T>((const uint8_t*)W, row_bytes, (__nv_bfloat16*)out, N, K, st)
  VE_GGUF_TYPES(ggml_type, VE_CALL)
#undef VE_CALL
}

}  // extern "C"
