// NVFP4 weight x bf16 activation mat-vec for decode / verify rows (M <= 16).
//
//   out[m, n] = gscale * sum_k e2m1(Wp[n, k]) * e4m3(Ws[n, k/16]) * x[m, k]          (+ bias / residual)
//
// Checkpoint layout is consumed as is (compressed-tensors / modelopt): Wp [N, K/2] bytes with the even
// k in the low nibble, Ws [N, K/16] E4M3 bytes, one fp32 global scale
// (reference: src/loader/nvfp4.cpp:36-57, decode rule inc/engine/quant/fp4_fp8.h:14-40).
//
// Design: HBM-bound streaming kernel. One CTA (4 warps) owns R=4 output rows; its 128 threads stride over
// K, each streaming 16 B (32 weights) per row per iteration with evict-first loads (activations come
// through L1), and the four warp partials are summed through shared memory in warp order.
// FP4 decode is the hardware cvt.e2m1x2; partial sums per 16-element block are accumulated in fp32 with
// packed f32x2 FMAs and scaled once per block, so a row's result depends only on its own activations and
// a fixed summation order: the same bits for M = 1 and for a row inside a verify block.
#include "common.cuh"

namespace ve {

VE_DEVINL uint32_t cvt_e2m1x2_f16x2(uint32_t byte) {
  uint32_t r;
  asm("{ .reg .b8 t; cvt.u8.u32 t, %1; cvt.rn.f16x2.e2m1x2 %0, t; }" : "=r"(r) : "r"(byte));
  return r;
}
VE_DEVINL float e4m3_to_float(uint32_t b) {
  uint32_t r;
  asm("{ .reg .b16 t; cvt.u16.u32 t, %1; cvt.rn.f16x2.e4m3x2 %0, t; }" : "=r"(r) : "r"(b & 0xffu));
  return __half2float(__ushort_as_half((unsigned short)(r & 0xffffu)));
}
VE_DEVINL float2 ffma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return *reinterpret_cast<float2*>(&d);
}

constexpr int kGemvRows = 4;    // output rows per warp
constexpr int kGemvWarps = 4;   // warps per CTA

template <int MR>
__global__ void __launch_bounds__(kGemvWarps * 32)
nvfp4_gemv_kernel(const uint8_t* __restrict__ Wp, const uint8_t* __restrict__ Ws, float gscale,
                  const __nv_bfloat16* __restrict__ x, long x_stride, __nv_bfloat16* __restrict__ out,
                  long out_stride, const __nv_bfloat16* __restrict__ residual, long res_stride, int M, int N, int K,
                  int m0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = blockIdx.x * kGemvRows;
  __shared__ float part[kGemvWarps][kGemvRows][MR];
  grid_dep_launch();
  grid_dep_wait();
  const int kchunks = K >> 5;  // 32-element (16 B) chunks per row
  float acc[kGemvRows][MR];
#pragma unroll
  for (int r = 0; r < kGemvRows; ++r)
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[r][m] = 0.f;

  const __nv_bfloat16* xr[MR];
#pragma unroll
  for (int m = 0; m < MR; ++m) xr[m] = x + (long)min(m0 + m, M - 1) * x_stride;

  for (int c = threadIdx.x; c < kchunks; c += kGemvWarps * 32) {
    uint4 w[kGemvRows];
    uint32_t sc[kGemvRows];
#pragma unroll
    for (int r = 0; r < kGemvRows; ++r) {
      const int n = min(n0 + r, N - 1);
      w[r] = __ldcs(reinterpret_cast<const uint4*>(Wp + (long)n * (K >> 1)) + c);
      sc[r] = __ldcs(reinterpret_cast<const unsigned short*>(Ws + (long)n * (K >> 4)) + c);
    }
#pragma unroll
    for (int blk = 0; blk < 2; ++blk) {
      float2 pb[kGemvRows][MR];
#pragma unroll
      for (int r = 0; r < kGemvRows; ++r)
#pragma unroll
        for (int m = 0; m < MR; ++m) pb[r][m] = make_float2(0.f, 0.f);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        // 8 activations per row m: k = c*32 + blk*16 + half*8 .. +7
        float2 xv[MR][4];
#pragma unroll
        for (int m = 0; m < MR; ++m) {
          const uint4 t = *reinterpret_cast<const uint4*>(xr[m] + (long)c * 32 + blk * 16 + half * 8);
          const uint32_t u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
          for (int j = 0; j < 4; ++j)
            xv[m][j] = make_float2(__uint_as_float(u[j] << 16), __uint_as_float(u[j] & 0xffff0000u));
        }
#pragma unroll
        for (int r = 0; r < kGemvRows; ++r) {
          const uint32_t word = blk == 0 ? (half == 0 ? w[r].x : w[r].y) : (half == 0 ? w[r].z : w[r].w);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t h2 = cvt_e2m1x2_f16x2((word >> (8 * j)) & 0xffu);
            const float2 wf = __half22float2(*reinterpret_cast<const __half2*>(&h2));
#pragma unroll
            for (int m = 0; m < MR; ++m) pb[r][m] = ffma2(wf, xv[m][j], pb[r][m]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < kGemvRows; ++r) {
        const float s = e4m3_to_float(sc[r] >> (8 * blk));
#pragma unroll
        for (int m = 0; m < MR; ++m) acc[r][m] = fmaf(s, pb[r][m].x + pb[r][m].y, acc[r][m]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kGemvRows; ++r)
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      float v = acc[r][m];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) part[warp][r][m] = v;
    }
  __syncthreads();
  if (threadIdx.x < kGemvRows * MR) {
    const int r = threadIdx.x / MR, m = threadIdx.x % MR;
    const int n = n0 + r;
    if (n < N && m0 + m < M) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kGemvWarps; ++w) v += part[w][r][m];
      v *= gscale;
      if (residual) v += bf2f(residual[(long)(m0 + m) * res_stride + n]);
      out[(long)(m0 + m) * out_stride + n] = f2bf(v);
    }
  }
}

// bf16 weights of few rows (routers, 256 to 512 rows), fp32 output, fp32 FMAs in one fixed order: up to four activation rows a pass. The
// matrix stays in L2 between the passes, so what the tensor cores would save (14 to 5 us at 16 rows of 512 x 2048) is small, and a router's
// scores keep their bits.
template <int MR>
__global__ void __launch_bounds__(kGemvWarps * 32)
bf16_gemv_few_kernel(const __nv_bfloat16* __restrict__ W, const __nv_bfloat16* __restrict__ x, long x_stride,
                     float* __restrict__ out, long out_stride, int M, int N, int K, int m0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = blockIdx.x * kGemvRows;
  __shared__ float part[kGemvWarps][kGemvRows][MR];
  grid_dep_launch();
  grid_dep_wait();                   // x is the output of the kernel in front (this launch is a programmatic dependent)
  float acc[kGemvRows][MR];
#pragma unroll
  for (int r = 0; r < kGemvRows; ++r)
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[r][m] = 0.f;
  const int kchunks = K >> 3;
  for (int c = threadIdx.x; c < kchunks; c += kGemvWarps * 32) {
    float2 xv[MR][4];
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      const uint4 t = *reinterpret_cast<const uint4*>(x + (long)min(m0 + m, M - 1) * x_stride + (long)c * 8);
      const uint32_t u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        xv[m][j] = make_float2(__uint_as_float(u[j] << 16), __uint_as_float(u[j] & 0xffff0000u));
    }
#pragma unroll
    for (int r = 0; r < kGemvRows; ++r) {
      const int n = min(n0 + r, N - 1);
      const uint4 t = __ldcs(reinterpret_cast<const uint4*>(W + (long)n * K) + c);
      const uint32_t u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 wf = make_float2(__uint_as_float(u[j] << 16), __uint_as_float(u[j] & 0xffff0000u));
#pragma unroll
        for (int m = 0; m < MR; ++m) {
          acc[r][m] = fmaf(wf.x, xv[m][j].x, acc[r][m]);
          acc[r][m] = fmaf(wf.y, xv[m][j].y, acc[r][m]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kGemvRows; ++r)
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      float v = acc[r][m];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) part[warp][r][m] = v;
    }
  __syncthreads();
  if (threadIdx.x < kGemvRows * MR) {
    const int r = threadIdx.x / MR, m = threadIdx.x % MR;
    if (n0 + r < N && m0 + m < M) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kGemvWarps; ++w) v += part[w][r][m];
      out[(long)(m0 + m) * out_stride + n0 + r] = v;
    }
  }
}

// bf16 weights, fp32 output (LM head, routers: logits stay fp32 for argmax / top-k / LSE), up to 8 * NT activation rows in one pass.
//
// Bound by the weights' DRAM traffic (1.55 GB and 235 us for a 151936 x 5120 head), so they are read once whatever M is: a block takes 16 * NT
// weight rows, its warps deal 32-wide steps of K, and each product with all activation rows is two tensor-core instructions per 16 rows
// and step. (In passes of four activation rows with fp32 FMAs 16 rows took four reads: 1072 us for the head and four routers of the
// 512-expert model, against 94 us for one row of the head.) Lane (g, t) holds k = 8 t .. 8 t + 7 of a step for weight rows g and g + 8 and
// activation row g, whole 16-byte loads; both operands use the same order of k. The sum of a step leaves the tensor core and is added in
// fp32: steps in pairs, a warp's pairs, warps in a tree (in one chain a sum was 1.2 to 1.6 times as far from 64 bits as sums product by
// product). Steps, warps and their order follow from N and K alone: a row's result does not depend on the rows beside it.
template <int NT, int WARPS>
__global__ void __launch_bounds__(32 * WARPS)
bf16_gemv_f32_kernel(const __nv_bfloat16* __restrict__ W, const __nv_bfloat16* __restrict__ x, long x_stride,
                     float* __restrict__ out, long out_stride, int M, int N, int K) {
  constexpr int ROWS = 16 * NT, COLS = 8 * NT, U = 4 / NT;      // U: steps in flight a warp (eight 16-byte weight loads a lane)
  __shared__ float part[WARPS][COLS][ROWS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * ROWS;
  grid_dep_wait();                   // x and, where they were just decoded, the weights come from kernels in front
  const __nv_bfloat16 *wr[2 * NT], *xr[NT];
#pragma unroll
  for (int r = 0; r < 2 * NT; ++r) wr[r] = W + (long)min(n0 + r * 8 + g, N - 1) * K + 8 * t;
#pragma unroll
  for (int j = 0; j < NT; ++j) xr[j] = x + (long)min(j * 8 + g, M - 1) * x_stride + 8 * t;
  float acc[NT][NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  const int steps = (K + 31) / 32;
  // four steps in a row a warp: 256 contiguous bytes of each weight row (64 a warp, dealt in turn: 5.8 TB/s instead of 6.6)
  for (int b0 = warp * 4; b0 < steps; b0 += WARPS * 4)
#pragma unroll
  for (int c0 = b0; c0 < b0 + 4; c0 += U) {
    uint4 w[U][2 * NT], v[U][NT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (c0 + u) * 32;
      const bool live = k + 8 * t < K;
#pragma unroll
      for (int r = 0; r < 2 * NT; ++r) w[u][r] = live ? __ldcs(reinterpret_cast<const uint4*>(wr[r] + k)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int j = 0; j < NT; ++j)
        v[u][j] = live && j * 8 + g < M ? *reinterpret_cast<const uint4*>(xr[j] + k) : make_uint4(0u, 0u, 0u, 0u);
    }
    static_assert(U % 2 == 0, "steps are added in pairs");
#pragma unroll
    for (int u = 0; u < U; u += 2)
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          float d[2][4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4 a = w[u + h][2 * i], b = w[u + h][2 * i + 1], y = v[u + h][j];
            d[h][0] = d[h][1] = d[h][2] = d[h][3] = 0.f;
            mma_bf16_16816(d[h], a.x, b.x, a.y, b.y, y.x, y.y);
            mma_bf16_16816(d[h], a.z, b.z, a.w, b.w, y.z, y.w);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][j][e] += d[0][e] + d[1][e];
        }
  }
  grid_dep_launch();                 // (not before: blocks that wait beside this one's take their issue slots)
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) part[warp][j * 8 + 2 * t + (e & 1)][i * 16 + (e >> 1) * 8 + g] = acc[i][j][e];
  __syncthreads();
  for (int i = threadIdx.x; i < COLS * ROWS; i += 32 * WARPS) {
    const int m = i / ROWS, n = n0 + i % ROWS;
    if (m < M && n < N) {
      float sum[WARPS];
#pragma unroll
      for (int q = 0; q < WARPS; ++q) sum[q] = part[q][m][i % ROWS];
#pragma unroll
      for (int h = 1; h < WARPS; h *= 2)
#pragma unroll
        for (int q = 0; q < WARPS; q += 2 * h) sum[q] += sum[q + h];
      out[(long)m * out_stride + n] = sum[0];
    }
  }
}

}  // namespace ve

using namespace ve;

extern "C" {

// x [M, K] bf16 (row stride x_stride), out [M, N] bf16. residual (optional) is added in fp32 before rounding.
int ve_nvfp4_gemv(const void* Wp, const void* Ws, float gscale, const void* x, long x_stride, void* out,
                  long out_stride, const void* residual, long res_stride, int M, int N, int K, cudaStream_t st) {
  if (K % 32 || M <= 0 || N <= 0) return cudaErrorInvalidValue;
  const int blocks = (N + kGemvRows - 1) / kGemvRows;
  int m0 = 0;
  while (m0 < M) {
    const int left = M - m0;
#define VE_LAUNCH(MR)                                                                                            \
  nvfp4_gemv_kernel<MR><<<blocks, kGemvWarps * 32, 0, st>>>(                                                     \
      (const uint8_t*)Wp, (const uint8_t*)Ws, gscale, (const __nv_bfloat16*)x, x_stride, (__nv_bfloat16*)out,    \
      out_stride, (const __nv_bfloat16*)residual, res_stride, M, N, K, m0)
    if (left >= 4) {
      VE_LAUNCH(4);
      m0 += 4;
    } else if (left >= 2) {
      VE_LAUNCH(2);
      m0 += 2;
    } else {
      VE_LAUNCH(1);
      m0 += 1;
    }
#undef VE_LAUNCH
  }
  VE_CHECK_LAUNCH();
}

int ve_bf16_gemv_f32(const void* W, const void* x, long x_stride, void* out, long out_stride, int M, int N, int K,
                     cudaStream_t st) {
  if (K % 8 || M <= 0 || N <= 0) return cudaErrorInvalidValue;
  if (N <= 16 * 148) {
    const int blocks = (N + kGemvRows - 1) / kGemvRows;
    for (int m0 = 0; m0 < M;) {
      const int left = M - m0;
#define VE_FEW(MR)                                                                                           \
  launch_pdl(bf16_gemv_few_kernel<MR>, dim3(blocks), dim3(kGemvWarps * 32), 0, st, (const __nv_bfloat16*)W, \
             (const __nv_bfloat16*)x, x_stride, (float*)out, out_stride, M, N, K, m0)
      if (left >= 4) { VE_FEW(4); m0 += 4; }
      else if (left >= 2) { VE_FEW(2); m0 += 2; }
      else { VE_FEW(1); m0 += 1; }
#undef VE_FEW
    }
    VE_CHECK_LAUNCH();
  }
  for (int m0 = 0; m0 < M; m0 += 16) {
    const int m = M - m0 < 16 ? M - m0 : 16, nt = m > 8 ? 2 : 1;
    const __nv_bfloat16* xm = (const __nv_bfloat16*)x + (long)m0 * x_stride;
    float* om = (float*)out + (long)m0 * out_stride;
    const dim3 grid((N + 16 * nt - 1) / (16 * nt));
#define VE_LAUNCH(NT, WARPS)                                                                                               \
  launch_pdl(bf16_gemv_f32_kernel<NT, WARPS>, grid, dim3(32 * WARPS), 0, st, (const __nv_bfloat16*)W, xm, x_stride, om, out_stride, m, N, K)
    if (nt == 1) VE_LAUNCH(1, 8); else VE_LAUNCH(2, 8);
#undef VE_LAUNCH
  }
  VE_CHECK_LAUNCH();
}

}  // extern "C"
