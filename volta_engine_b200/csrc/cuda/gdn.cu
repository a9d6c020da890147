// Gated DeltaNet mixer (linear attention with a gated delta rule):
//   gdn_prepare    parallel over rows: causal short convolution + SiLU over the q|k|v channels (taps from earlier rows
//                  of the same slot in the batch, else from the slot's convolution state), L2 norm of q and k per head,
//                  q scale, decay exp(g) and beta per value head
//   gdn_recurrent  one CTA per (16 columns of a value head's state, slot): walks the slot's rows in order with the state
//                  in registers:  S *= decay;  delta = (v - S^T k) * beta;  S += k (x) delta;  o = S^T q;
//                  stores the state and rolls the slot's convolution state forward
//   gdn_gated_norm y = rmsnorm(o) * w * silu(z)
// KDA (Kimi delta attention) is the same recurrence with one decay per key channel, S = diag(exp(g)) S, where
//   g = -5 sigmoid(exp(A_log[h]) (f + dt_bias)) and f is a low-rank projection of the input; its output gate is sigmoid(z)
//   (reference: src/backend/cpu/gdn_ref.cpp:32-57 kda_head_step, :94-127 project_kda_gates, :59-68 gate_norm_out).
// A row at position 0 starts its slot from zero state. fp32 state and arithmetic; the fused projection row is
// [q | k | v | z | b | a] in bf16. Reference: inc/engine/modules/gdn.h (project_gates, causal_conv1d_silu*,
// l2_norm_heads, recurrent_step[_rows], gated_rmsnorm).
#include "common.cuh"

namespace ve {

struct GdnArgs {
  const __nv_bfloat16* proj; long ld;
  const int* pos; const int* slot;
  float* conv_state;            // [slots][kc-1][C]
  float* rec_state;             // [slots][nv][dk][dv]
  const float* conv_w;          // [C][kc]
  const float* A_log; const float* dt_bias;
  float* u;                     // [rows][C]   conv + norm outputs
  float* gb;                    // [rows][2*nv] decay, beta
  float* o;                     // [rows][nv*dv]
  int rows, nk, nv, dk, dv, kc, slots;
  const float* kdec;            // KDA: [rows][nv * dk] per-key-channel decay exp(g); null = one decay per head (gb)
};

VE_DEVINL float siluf(float x) { return x / (1.f + __expf(-x)); }

// rows of the same slot directly in front of row i (at most lim)
VE_DEVINL int rows_before(const int* slot, const int* pos, int i, int lim) {
  int r = 0;
  while (r < lim && i - r - 1 >= 0 && slot[i - r - 1] == slot[i] && pos[i - r - 1] == pos[i] - r - 1) ++r;
  return r;
}

// A few rows: grid (2*nk + nv + 1, rows), block = max(dk, dv, nv) threads, one channel each. Unit < nk: q head; < 2nk: k head; < 2nk+nv: v head; last: gates.
__global__ void gdn_prepare_rows_kernel(const GdnArgs a) {
  __shared__ float red[33];
  grid_dep_launch();
  grid_dep_wait();
  const int unit = blockIdx.x, i = blockIdx.y, tid = threadIdx.x;
  const int s = a.slot[i];
  if (s < 0) return;
  const int C = 2 * a.nk * a.dk + a.nv * a.dv;
  if (unit == 2 * a.nk + a.nv) {
    if (tid < a.nv) {
      const __nv_bfloat16* row = a.proj + (long)i * a.ld + C + a.nv * a.dv;
      const float b = bf2f(row[tid]), av = bf2f(row[a.nv + tid]);
      const float x = av + a.dt_bias[tid];
      const float sp = x > 20.f ? x : log1pf(__expf(x));
      a.gb[(long)i * 2 * a.nv + tid] = __expf(-__expf(a.A_log[tid]) * sp);
      a.gb[(long)i * 2 * a.nv + a.nv + tid] = 1.f / (1.f + __expf(-b));
    }
    return;
  }
  const bool is_v = unit >= 2 * a.nk;
  const int width = is_v ? a.dv : a.dk;
  const int c0 = is_v ? 2 * a.nk * a.dk + (unit - 2 * a.nk) * a.dv : unit * a.dk;
  const int p = a.pos[i];
  const int r = rows_before(a.slot, a.pos, i, a.kc - 1);
  float val = 0.f;
  if (tid < width) {
    const int c = c0 + tid;
    float acc = 0.f;
    for (int d = 0; d < a.kc; ++d) {               // d = distance into the past of the tap
      if (p - d < 0) break;
      float x;
      if (d <= r) x = bf2f(a.proj[(long)(i - d) * a.ld + c]);
      else x = a.conv_state[((long)s * (a.kc - 1) + (a.kc - 1 - (d - r))) * C + c];
      acc += x * a.conv_w[(long)c * a.kc + (a.kc - 1 - d)];
    }
    val = siluf(acc);
  }
  if (!is_v) {
    const float ss = block_sum(val * val, red);
    const float inv = rsqrtf(ss + 1e-6f) * (unit < a.nk ? rsqrtf((float)a.dk) : 1.f);
    val *= inv;
  }
  if (tid < width) a.u[(long)i * C + c0 + tid] = val;
}

// One warp per unit, eight warps a block; each warp walks `per` rows of its unit. Unit < nk: q head; < 2nk: k head; < 2nk+nv: v head;
// last: gates. The filter of a lane's channels stays in registers, and so do the last KC - 1 inputs where a row continues the one in
// front of it. Bound by the bf16 rows read and the fp32 rows written (126 MB at 2048 rows of 10240 channels, 20 us at the copy rate): a
// block per (unit, row) with three barriers took 237 us there, a warp per row that fetched filter and taps again for each 155 us, this form 120 us.
template <int NE, int KC>         // 32-channel pieces of the widest head; taps (0: any number)
__global__ void __launch_bounds__(256) gdn_prepare_kernel(const GdnArgs a, int per) {
  grid_dep_launch();
  grid_dep_wait();
  const int lane = threadIdx.x & 31;
  const int unit = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (unit > 2 * a.nk + a.nv) return;
  const int C = 2 * a.nk * a.dk + a.nv * a.dv;
  const int i0 = blockIdx.y * per, i1 = min(a.rows, i0 + per);
  if (unit == 2 * a.nk + a.nv) {
    for (int i = i0; i < i1; ++i) {
      if (a.slot[i] < 0) continue;
      const __nv_bfloat16* row = a.proj + (long)i * a.ld + C + a.nv * a.dv;
      for (int j = lane; j < a.nv; j += 32) {
        const float b = bf2f(row[j]), av = bf2f(row[a.nv + j]);
        const float x = av + a.dt_bias[j];
        const float sp = x > 20.f ? x : log1pf(__expf(x));
        a.gb[(long)i * 2 * a.nv + j] = __expf(-__expf(a.A_log[j]) * sp);
        a.gb[(long)i * 2 * a.nv + a.nv + j] = 1.f / (1.f + __expf(-b));
      }
    }
    return;
  }
  const bool is_v = unit >= 2 * a.nk;
  const int width = is_v ? a.dv : a.dk;
  const int c0 = is_v ? 2 * a.nk * a.dk + (unit - 2 * a.nk) * a.dv : unit * a.dk;
  const int kc = KC ? KC : a.kc;
  constexpr int KR = KC ? KC : 1;
  float w[NE][KR], x[NE][KR];                          // filter, newest input last; inputs by distance into the past
  if (KC)
#pragma unroll
    for (int e = 0; e < NE; ++e)
#pragma unroll
      for (int d = 0; d < KR; ++d) {
        w[e][d] = e * 32 + lane < width ? a.conv_w[(long)(c0 + e * 32 + lane) * KC + (KC - 1 - d)] : 0.f;
        x[e][d] = 0.f;
      }
  int s0 = -1, p0 = 0;                                 // slot and position of the row whose inputs x holds
  for (int i = i0; i < i1; ++i) {
    const int s = a.slot[i];
    if (s < 0) { s0 = -1; continue; }
    const int p = a.pos[i];
    const bool next = KC && s == s0 && p == p0 + 1;
    const int r = next ? 0 : rows_before(a.slot, a.pos, i, kc - 1);
    auto tap = [&](int d, int c) -> float {            // input at distance d (zero in front of the sequence)
      if (p - d < 0) return 0.f;
      return d <= r ? bf2f(a.proj[(long)(i - d) * a.ld + c]) : a.conv_state[((long)s * (kc - 1) + (kc - 1 - (d - r))) * C + c];
    };
    float acc[NE], ss = 0.f;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      acc[e] = 0.f;
      const int t = e * 32 + lane, c = c0 + t;
      if (t < width) {
        if (KC) {
#pragma unroll
          for (int d = KR - 1; d > 0; --d) x[e][d] = next ? x[e][d - 1] : tap(d, c);
          x[e][0] = bf2f(a.proj[(long)i * a.ld + c]);
#pragma unroll
          for (int d = 0; d < KR; ++d) acc[e] += x[e][d] * w[e][d];
        } else {
          for (int d = 0; d < kc; ++d) acc[e] += tap(d, c) * a.conv_w[(long)c * kc + (kc - 1 - d)];
        }
        acc[e] = siluf(acc[e]);
      }
      ss = fmaf(acc[e], acc[e], ss);
    }
    s0 = s;
    p0 = p;
    float inv = 1.f;
    if (!is_v) inv = rsqrtf(warp_sum(ss) + 1e-6f) * (unit < a.nk ? rsqrtf((float)a.dk) : 1.f);
#pragma unroll
    for (int e = 0; e < NE; ++e)
      if (e * 32 + lane < width) a.u[(long)i * C + c0 + e * 32 + lane] = acc[e] * inv;
  }
}

// Two fp32 values in one register pair, for the packed FMA of sm_100.
VE_DEVINL uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
VE_DEVINL float2 unpack2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
VE_DEVINL uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
VE_DEVINL uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// grid (dv / COLS, nv, slots), 4 COLS threads: COLS columns of one head's state; eight lanes share two columns, DK / 8 keys of each in the
// registers of a lane.
//
// The recurrence is a serial chain over the rows, so what counts is the chain's length per row and how many chains run beside one another.
// With a column per thread (DK registers, 48 blocks for 48 heads) every row waited for its own q, k and gates from L2 between two barriers:
// 2.03 us a row, 4163 us for 2048 rows of 48 heads. Here the rows come in blocks of eight through a cp.async ring that runs two blocks
// ahead, the chain of a row is 3 * DK / 8 packed FMAs and three shuffles (the output sums of a block are reduced together behind it, 14
// shuffles instead of 48), and 384 blocks share the chip. Shared-memory reads of k and q (512 bytes a warp and 16-byte load, also where
// lanes read the same) bind next: with one column a lane they took 384 cycles a row on an SM with three blocks, 0.65 us a row in all
// against 0.29 us now (2048 rows of 48 heads: 596 us; with the kernels in front and behind 743 us), of which a row's chain of
// dependent instructions is most (138 instructions a row and warp, 41 % of the issue slots at five warps an SM).
//
// Launches of few rows, mostly one a slot, have a form of their own, bound by the state's bytes and by how fast blocks come and go, those of idle
// slots among them: 64 columns a block, blocks of four rows, a ring of two, registers for half as many warps again. us for 48 heads with the
// kernels in front and behind (a thread a column / 16 columns a block / now): one row, one slot 12.6 13.2 10.8; one row, 31 idle slots 11.4 18.8
// 10.0; four rows of one slot 16.6 16.3 10.8; 8 streams 22.5 27.4 24.7; 16 streams 32.2 44.3 40.6, where a thread a column, with whole
// rows of the state in a warp's load, is still ahead.
// COLS: columns of a block, a warp eight of them; 16 in the long form, 64 or 32 in the brief one (as dv allows).
constexpr int kGdnBrief = 32;
template <int DK, bool KDA, int COLS>
struct GdnStage {
  static constexpr bool kBrief = COLS > 16;
  static constexpr int kRows = kBrief ? 4 : 8, kStages = kBrief ? 2 : 3;
  float k[kRows][DK], q[kRows][DK], d[KDA ? kRows : 1][KDA ? DK : 4];
  float v[kRows][COLS];
  float gb[kRows][2];
};

template <int DK, bool KDA, int COLS>
__global__ void __launch_bounds__(4 * COLS, (COLS > 16 ? 192 : 96) / COLS) gdn_recurrent_kernel(const GdnArgs a) {
  using Stage = GdnStage<DK, KDA, COLS>;
  constexpr bool BRIEF = Stage::kBrief;
  constexpr int kGdnRows = Stage::kRows, kGdnStages = Stage::kStages, NT = 4 * COLS;
  extern __shared__ __align__(16) uint8_t gdn_smem[];
  Stage* const ring = reinterpret_cast<Stage*>(gdn_smem);
  __shared__ int s_first[NT / 32], s_count[NT / 32];
  constexpr int NP = DK / 16;                          // register pairs of a lane's part of a column
  // A long walk is launched plainly and lets its dependents in when it ends: chains that share an SM slow each other, and both blocks of the
  // kernel behind that wait there and an uneven first placement (this kernel's blocks let in while the one in front still holds parts of the
  // chip pile up on the SMs that are free) took 2048 rows of 48 heads from 0.31 us a row to 0.57.
  if (BRIEF) grid_dep_launch();
  grid_dep_wait();
  const int c0 = blockIdx.x * COLS, h = blockIdx.y, s = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = lane & 7;
  const int col = warp * 8 + (lane >> 3) * 2;           // first of this lane's two columns within the block
  // rows of this slot (consecutive)
  int first = a.rows, count = 0;
  for (int i = tid; i < a.rows; i += NT)
    if (a.slot[i] == s) { first = min(first, i); ++count; }
  first = __reduce_min_sync(0xffffffffu, first);
  count = __reduce_add_sync(0xffffffffu, count);
  if (lane == 0) { s_first[warp] = first; s_count[warp] = count; }
  __syncthreads();
  first = s_first[0];
  count = s_count[0];
#pragma unroll
  for (int w = 1; w < NT / 32; ++w) { first = min(first, s_first[w]); count += s_count[w]; }
  if (count == 0) return;
  const int C = 2 * a.nk * DK + a.nv * a.dv;
  const int kh = h / (a.nv / a.nk);
  const bool fresh = a.pos[first] == 0;

  auto load = [&](int blk) {                            // one block of rows into its ring stage
    if (blk * kGdnRows < count) {
      Stage& st = ring[blk % kGdnStages];
      const int n = min(kGdnRows, count - blk * kGdnRows);
      const long i0 = first + blk * kGdnRows;
      constexpr int Q = DK / 4;                          // 16-byte pieces of a key
      for (int j = tid; j < n * Q; j += NT) {
        const int r = j / Q, c = (j % Q) * 4;
        const float* ui = a.u + (i0 + r) * C + kh * DK + c;
        cp_async16(&st.q[r][c], ui);
        cp_async16(&st.k[r][c], ui + a.nk * DK);
        if (KDA) cp_async16(&st.d[r][c], a.kdec + ((i0 + r) * a.nv + h) * DK + c);
      }
      constexpr int V = COLS / 4;
      for (int j = tid; j < n * V; j += NT) {
        const int r = j / V, c = j % V * 4;
        cp_async16(&st.v[r][c], a.u + (i0 + r) * C + 2 * a.nk * DK + h * a.dv + c0 + c);
      }
      if (tid >= 32 && tid < 32 + n * 2) {
        const int r = (tid - 32) >> 1, w = tid & 1;
        cp_async4(&st.gb[r][w], a.gb + (i0 + r) * 2 * a.nv + w * a.nv + h);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int b = 0; b < kGdnStages - 1; ++b) load(b);

  // pair j of this lane: keys (j / 2 * 8 + part) * 4 + (j % 2) * 2 and the next one, columns col and col + 1
  float* const stp = a.rec_state + (((long)s * a.nv + h) * DK) * a.dv + c0 + col;
  uint64_t S[2][NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const long k = ((j >> 1) * 8 + part) * 4 + (j & 1) * 2;
    float2 lo = make_float2(0.f, 0.f), hi = lo;
    if (!fresh) { lo = *reinterpret_cast<const float2*>(stp + k * a.dv); hi = *reinterpret_cast<const float2*>(stp + (k + 1) * a.dv); }
    S[0][j] = pack2(lo.x, hi.x);
    S[1][j] = pack2(lo.y, hi.y);
  }
  float o[2][kGdnRows];
  auto row = [&](const Stage& st, int r) {
    uint64_t k2[NP], m[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
    const float2 g = *reinterpret_cast<const float2*>(st.gb[r]);
    const float2 v = *reinterpret_cast<const float2*>(&st.v[r][col]);
    const uint64_t dec = pack2(g.x, g.x);
#pragma unroll
    for (int j = 0; j < NP; j += 2) {
      const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(&st.k[r][((j >> 1) * 8 + part) * 4]);
      k2[j] = kv.x; k2[j + 1] = kv.y;
      ulonglong2 d = make_ulonglong2(dec, dec);
      if (KDA) d = *reinterpret_cast<const ulonglong2*>(&st.d[r][((j >> 1) * 8 + part) * 4]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        S[c][j] = mul2(S[c][j], d.x);
        S[c][j + 1] = mul2(S[c][j + 1], d.y);
        m[c][0] = fma2(S[c][j], k2[j], m[c][0]);
        m[c][1] = fma2(S[c][j + 1], k2[j + 1], m[c][1]);
      }
    }
    float mem[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 x = unpack2(m[c][0]), y = unpack2(m[c][1]);
      mem[c] = (x.x + x.y) + (y.x + y.y);
    }
#pragma unroll
    for (int w = 1; w < 8; w <<= 1) {
      mem[0] += __shfl_xor_sync(0xffffffffu, mem[0], w);
      mem[1] += __shfl_xor_sync(0xffffffffu, mem[1], w);
    }
    const float d0 = (v.x - mem[0]) * g.y, d1 = (v.y - mem[1]) * g.y;
    const uint64_t dl[2] = {pack2(d0, d0), pack2(d1, d1)};
    uint64_t q[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
#pragma unroll
    for (int j = 0; j < NP; j += 2) {
      const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(&st.q[r][((j >> 1) * 8 + part) * 4]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        S[c][j] = fma2(k2[j], dl[c], S[c][j]);
        S[c][j + 1] = fma2(k2[j + 1], dl[c], S[c][j + 1]);
        q[c][0] = fma2(S[c][j], qv.x, q[c][0]);
        q[c][1] = fma2(S[c][j + 1], qv.y, q[c][1]);
      }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 x = unpack2(q[c][0]), y = unpack2(q[c][1]);
      o[c][r] = (x.x + x.y) + (y.x + y.y);
    }
  };
  const int blocks = (count + kGdnRows - 1) / kGdnRows;
  for (int blk = 0; blk < blocks; ++blk) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kGdnStages - 2) : "memory");
    __syncthreads();                                     // this block's rows have landed; the stage in front of it is free
    load(blk + kGdnStages - 1);
    const Stage& st = ring[blk % kGdnStages];
    const int n = min(kGdnRows, count - blk * kGdnRows);
    if (n == kGdnRows) {
#pragma unroll
      for (int r = 0; r < kGdnRows; ++r) row(st, r);
    } else {
#pragma unroll
      for (int r = 0; r < kGdnRows; ++r) {
        o[0][r] = o[1][r] = 0.f;
        if (r < n) row(st, r);
      }
    }
    // sums over the eight lanes of a column: lane `part` ends with row `part` (of four rows, `part` and `part` - 4 with the same one)
    if (kGdnRows == 4)
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[c][j] += __shfl_xor_sync(0xffffffffu, o[c][j], 4);
#pragma unroll
    for (int w = kGdnRows / 2; w >= 1; w >>= 1) {
      const bool up = part & w;
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < w; ++j) {
          const float send = up ? o[c][j] : o[c][j + w], keep = up ? o[c][j + w] : o[c][j];
          o[c][j] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
    }
    if (part < n)
      *reinterpret_cast<float2*>(a.o + ((long)(first + blk * kGdnRows + part) * a.nv + h) * a.dv + c0 + col) = make_float2(o[0][0], o[1][0]);
  }
  if (!BRIEF) grid_dep_launch();
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const long k = ((j >> 1) * 8 + part) * 4 + (j & 1) * 2;
    const float2 x = unpack2(S[0][j]), y = unpack2(S[1][j]);
    *reinterpret_cast<float2*>(stp + k * a.dv) = make_float2(x.x, y.x);
    *reinterpret_cast<float2*>(stp + (k + 1) * a.dv) = make_float2(x.y, y.y);
  }
  {
    // roll the convolution state: the newest kc-1 inputs of the slot, oldest first. The channels are dealt to the
    // blocks of the slot (every channel is independent), so no block walks all of them alone.
    const int n1 = a.kc - 1;
    float* cs = a.conv_state + (long)s * n1 * C;
    for (int c = (h * gridDim.x + blockIdx.x) * NT + tid; c < C; c += gridDim.x * gridDim.y * NT) {
      float old[8], nw[8];
      for (int t = 0; t < n1; ++t) old[t] = fresh ? 0.f : cs[(long)t * C + c];
      for (int t = 0; t < n1; ++t) {
        const int e = n1 - 1 - t;                    // distance from the last row
        if (e < count) nw[t] = bf2f(a.proj[(long)(first + count - 1 - e) * a.ld + c]);
        else nw[t] = old[n1 - 1 - (e - count)];
      }
      for (int t = 0; t < n1; ++t) cs[(long)t * C + c] = nw[t];
    }
  }
}

// One warp per (row, head), eight a block: bound by 6 bytes read and 2 written per value. V: values of a lane's step (4 where the gate's
// rows are 8-byte aligned, else 1).
template <bool SIGMOID, int V>
__global__ void __launch_bounds__(256) gdn_gated_norm_kernel(const float* __restrict__ o, const __nv_bfloat16* __restrict__ proj, long ld,
                                      const float* __restrict__ w, __nv_bfloat16* __restrict__ out, long units, int nv, int dv,
                                      int z_off, float eps) {
  grid_dep_launch();
  grid_dep_wait();
  const long unit = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (unit >= units) return;
  const int lane = threadIdx.x & 31;
  const long i = unit / nv;
  const int h = (int)(unit % nv);
  const float* ob = o + unit * dv;
  float ss = 0.f;
  for (int c = lane * V; c < dv; c += 32 * V)
#pragma unroll
    for (int e = 0; e < V; ++e) ss = fmaf(ob[c + e], ob[c + e], ss);
  const float rs = rsqrtf(warp_sum(ss) / dv + eps);
  const __nv_bfloat16* zb = proj + i * ld + z_off + h * dv;
  for (int c = lane * V; c < dv; c += 32 * V) {
    __align__(8) __nv_bfloat16 z[V], y[V];
    if (V == 4) *reinterpret_cast<uint2*>(z) = *reinterpret_cast<const uint2*>(zb + c);
    else z[0] = zb[c];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const float zf = bf2f(z[e]);
      const float gate = SIGMOID ? 1.f / (1.f + __expf(-zf)) : siluf(zf);
      y[e] = f2bf(ob[c + e] * rs * w[c + e] * gate);
    }
    if (V == 4) *reinterpret_cast<uint2*>(out + unit * dv + c) = *reinterpret_cast<const uint2*>(y);
    else out[unit * dv + c] = y[0];
  }
}

// KDA decay per key channel: kdec[row][j] = exp(-5 sigmoid(exp(A_log[j / dk]) (f[row][j] + dt_bias[j]))). grid (rows, channel chunks).
__global__ void kda_decay_kernel(const __nv_bfloat16* __restrict__ f, long ld, const float* __restrict__ A_log,
                                 const float* __restrict__ dt_bias, float* __restrict__ kdec, int channels, int dk) {
  grid_dep_launch();
  grid_dep_wait();
  const int i = blockIdx.x;
  for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < channels; j += gridDim.y * blockDim.x) {
    const float x = __expf(A_log[j / dk]) * (bf2f(f[(long)i * ld + j]) + dt_bias[j]);
    kdec[(long)i * channels + j] = __expf(-5.f / (1.f + __expf(-x)));
  }
}

}  // namespace ve

using namespace ve;

template <int DK, bool KDA, int COLS>
static int launch_recurrent_cols(const GdnArgs& a, cudaStream_t st) {
  using Stage = GdnStage<DK, KDA, COLS>;
  constexpr int smem = Stage::kStages * (int)sizeof(Stage);
  static_assert(smem <= 48 * 1024, "no opt-in to large shared memory is made");
  const dim3 grid(a.dv / COLS, a.nv, a.slots);
  if (Stage::kBrief) launch_pdl(gdn_recurrent_kernel<DK, KDA, COLS>, grid, dim3(4 * COLS), smem, st, a);
  else gdn_recurrent_kernel<DK, KDA, COLS><<<grid, 4 * COLS, smem, st>>>(a);
  VE_CHECK_LAUNCH();
}
template <int DK, bool KDA>
static int launch_recurrent_dk(const GdnArgs& a, cudaStream_t st) {
  if (a.rows > kGdnBrief) return launch_recurrent_cols<DK, KDA, 16>(a, st);
  return a.dv % 64 == 0 ? launch_recurrent_cols<DK, KDA, 64>(a, st) : launch_recurrent_cols<DK, KDA, 32>(a, st);
}
template <bool KDA>
static int launch_recurrent(const GdnArgs& a, cudaStream_t st) {
  // rows of u and kdec are read in 16-byte pieces, the state and o in pairs: dk, dv and with them every offset are multiples of 32 floats
  if (((uintptr_t)a.u & 15) || ((uintptr_t)a.kdec & 15) || ((uintptr_t)a.rec_state & 7) || ((uintptr_t)a.o & 7)) return cudaErrorMisalignedAddress;
  if (a.dk == 128) return launch_recurrent_dk<128, KDA>(a, st);
  if (a.dk == 64) return launch_recurrent_dk<64, KDA>(a, st);
  return cudaErrorInvalidValue;
}
template <bool SIGMOID>
static int launch_gated_norm(const void* o, const void* z, long ld, const void* w, void* out, int rows, int nv, int dv, int z_off,
                             float eps, cudaStream_t st) {
  const long units = (long)rows * nv;
  const dim3 grid((unsigned)((units + 7) / 8));
  const bool vec = !((uintptr_t)z & 7) && ld % 4 == 0 && z_off % 4 == 0 && !((uintptr_t)out & 7);
  if (vec) launch_pdl(gdn_gated_norm_kernel<SIGMOID, 4>, grid, dim3(256), 0, st, (const float*)o, (const __nv_bfloat16*)z, ld,
                      (const float*)w, (__nv_bfloat16*)out, units, nv, dv, z_off, eps);
  else launch_pdl(gdn_gated_norm_kernel<SIGMOID, 1>, grid, dim3(256), 0, st, (const float*)o, (const __nv_bfloat16*)z, ld,
                  (const float*)w, (__nv_bfloat16*)out, units, nv, dv, z_off, eps);
  VE_CHECK_LAUNCH();
}

extern "C" {

int ve_gdn_prepare(const void* proj, long ld, const void* pos, const void* slot, void* conv_state, const void* conv_w,
                   const void* A_log, const void* dt_bias, void* u, void* gb, int rows, int nk, int nv, int dk, int dv,
                   int kc, int slots, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (kc < 2 || kc > 9 || dk > 256 || dv > 256 || nv % nk || nv > 256) return cudaErrorInvalidValue;
  GdnArgs a{(const __nv_bfloat16*)proj, ld, (const int*)pos, (const int*)slot, (float*)conv_state, nullptr,
            (const float*)conv_w, (const float*)A_log, (const float*)dt_bias, (float*)u, (float*)gb, nullptr,
            rows, nk, nv, dk, dv, kc, slots, nullptr};
  const int units = 2 * nk + nv + 1, width = dk > dv ? dk : dv;
  // A block per (unit, row) has the shortest path through a row; warps waste less on many, first one a row, then 16 rows after one another.
  // us at 81 units (16 key and 48 value heads), block / warp a row / 16 rows a warp: 4 rows 2.6 5.5 -, 64 rows 9.4 10.7 -, 128 rows 16.8 16.1 -,
  // 255 rows 31.5 26.8 31.6, 512 rows 61 - 34, 2048 rows 240 - 118; at 21 units 255 rows 9.5 11.4 28, 700 rows 22 - 30, 1024 rows 32 - 30.
  // (Narrow models' warps of a row fill their waves badly: they go from blocks straight to 16 rows.)
  const long work = (long)units * rows;
  const int per = work < 7000 || (work < 20500 && units < 40) ? 0 : work < 20500 ? 1 : 16;
  if (per == 0) {
    const int threads = ((width > nv ? width : nv) + 31) / 32 * 32;
    launch_pdl(gdn_prepare_rows_kernel, dim3(units, rows), dim3(threads), 0, st, a);
    VE_CHECK_LAUNCH();
  }
  const dim3 grid((units + 7) / 8, (rows + per - 1) / per);
  if (width <= 128 && kc == 4) launch_pdl(gdn_prepare_kernel<4, 4>, grid, dim3(256), 0, st, a, per);
  else if (width <= 128) launch_pdl(gdn_prepare_kernel<4, 0>, grid, dim3(256), 0, st, a, per);
  else launch_pdl(gdn_prepare_kernel<8, 0>, grid, dim3(256), 0, st, a, per);
  VE_CHECK_LAUNCH();
}

int ve_gdn_recurrent(const void* proj, long ld, const void* pos, const void* slot, void* conv_state, void* rec_state,
                     const void* u, const void* gb, void* o, int rows, int nk, int nv, int dk, int dv, int kc, int slots,
                     cudaStream_t st) {
  if (rows <= 0) return 0;
  if (kc < 2 || kc > 9 || dv > 256 || dv % 32 || nv % nk) return cudaErrorInvalidValue;
  GdnArgs a{(const __nv_bfloat16*)proj, ld, (const int*)pos, (const int*)slot, (float*)conv_state, (float*)rec_state,
            nullptr, nullptr, nullptr, (float*)u, (float*)gb, (float*)o, rows, nk, nv, dk, dv, kc, slots, nullptr};
  return launch_recurrent<false>(a, st);
}

// The recurrence with one decay per key channel (kdec [rows][nv * dk], already exponentiated).
int ve_kda_recurrent(const void* proj, long ld, const void* pos, const void* slot, void* conv_state, void* rec_state,
                     const void* u, const void* gb, void* o, const void* kdec, int rows, int nk, int nv, int dk, int dv, int kc,
                     int slots, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (kc < 2 || kc > 9 || dv > 256 || dv % 32 || nv % nk || !kdec) return cudaErrorInvalidValue;
  GdnArgs a{(const __nv_bfloat16*)proj, ld, (const int*)pos, (const int*)slot, (float*)conv_state, (float*)rec_state,
            nullptr, nullptr, nullptr, (float*)u, (float*)gb, (float*)o, rows, nk, nv, dk, dv, kc, slots, (const float*)kdec};
  return launch_recurrent<true>(a, st);
}

int ve_kda_decay(const void* f, long ld, const void* A_log, const void* dt_bias, void* kdec, int rows, int nv, int dk,
                 cudaStream_t st) {
  if (rows <= 0) return 0;
  const int chunks = (nv * dk + 1023) / 1024;          // 256 threads take four channels each
  launch_pdl(kda_decay_kernel, dim3(rows, chunks), dim3(256), 0, st, (const __nv_bfloat16*)f, ld, (const float*)A_log,
             (const float*)dt_bias, (float*)kdec, nv * dk, dk);
  VE_CHECK_LAUNCH();
}

int ve_gdn_gated_norm(const void* o, const void* proj, long ld, const void* w, void* out, int rows, int nv, int dv,
                      int conv_dim, int kc, float eps, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (dv > 1024 || dv % 32) return cudaErrorInvalidValue;
  return launch_gated_norm<false>(o, proj, ld, w, out, rows, nv, dv, conv_dim, eps, st);
}

// y = rmsnorm(o) * w * sigmoid(z); z [rows, nv * dv] bf16 with row stride ld.
int ve_kda_gated_norm(const void* o, const void* z, long ld, const void* w, void* out, int rows, int nv, int dv, float eps,
                      cudaStream_t st) {
  if (rows <= 0) return 0;
  if (dv > 1024 || dv % 32) return cudaErrorInvalidValue;
  return launch_gated_norm<true>(o, z, ld, w, out, rows, nv, dv, 0, eps, st);
}

}  // extern "C"
