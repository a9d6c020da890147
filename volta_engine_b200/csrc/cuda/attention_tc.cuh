// Prefill attention on the fifth-generation tensor cores (tcgen05, accumulators in TMEM). Included by attention.cu.
//
// One CTA = one query tile of up to 128 packed rows ((token, head-in-group) pairs of one kv head, one TMEM lane per
// row) against the pages of its sequence, bf16 cache, head_dim HD, no key split. Per 64-key page:
//     S  = Q K^T      tcgen05.mma 128 x 64 x HD    (Q and the K page K-major in 128B-swizzled shared memory)
//     P  = exp2(S * scale - m)                      (softmax warps: tcgen05.ld of one row per thread; bf16 P goes back into the
//                                                    first 32 columns of the S buffer it came from)
//     O += P V        tcgen05.mma 128 x HD x 64    (P from TMEM, the V page as it lands from TMA: the MN-major operand form)
// Warp roles: warp 0 streams pages by TMA (K and V through rings of their own: a K page is free as soon as its S is done), warp 1 issues
// the MMAs, then four softmax warps per stream (one row per thread). Heads of 128 columns leave TMEM room for two streams: the pages are
// dealt to them alternately, each with its own S buffers (2 x 64 TMEM columns; one stream: 3), its own running (reference maximum, row
// sum) and its own O accumulator, so the exponentials of one stream run under the MMAs of the other and two warps per scheduler hide the
// TMEM-load and barrier latencies; the two partial results are merged like split-KV partials in the epilogue (both accumulators live in
// the same TMEM lanes, so a thread reads both). Heads of 256 columns take one stream: a page is then 1024 cycles of tensor work against
// about 700 of softmax, which runs under the S of the next page and the PV of the one in front.
// Measured against the mma.sync kernel (attn_kernel): 2048 rows of 24 heads of 256 behind 2048 others 1072 to 245 us, without them 418 to
// 108 us; 16 heads 715 to 155 and 280 to 65 us. Prompts of a single page are slower, 10 to 13 us (fixed costs of the larger tile).
// Reference maximum of a row. Heads of 128 columns: it is only moved when a page raises it by more than 2^8 (then the O row is rescaled in
// TMEM by the thread that owns it); otherwise the old reference stays, probabilities are at most 2^8 and the final division by the row sum
// makes the result the same. The exponent is one FMA (score * scale - reference) and one ex2.approx. Heads of 256 columns: it is the running
// maximum itself, and the scaled score is rounded before the maximum is taken off, as in attn_kernel, whose rows of these heads this kernel
// took over: P is then rounded to bf16 from the same numbers (the largest probability of a page that holds the maximum is one, exactly).
// With a reference that lags, P lay up to 24 % further from 64 bits (2048 rows, scores of a few units: 0.00209 against 0.00173).
// Every wait is bounded; on expiry the CTA records a status code, skips its stores and frees its TMEM.
// Semantics are those of attn_kernel (causal limit / key_end, sliding window, optional sigmoid gate); reference:
// src/kernels/slang/ref_attention.slang:1-10,47-50,65-70.
#pragma once

namespace ve {

constexpr int kTcRows = 128;        // query rows of a tile
constexpr float kTcLazyLog2 = 8.f;  // the reference maximum moves only when a page raises it by more than this

template <int HD, int STREAMS, int NK, int NV>
__global__ void __launch_bounds__(64 + 128 * STREAMS, 1) attn_prefill_tc_kernel(const AttnParams p, const __grid_constant__ CUtensorMap kmap,
                                                                               const __grid_constant__ CUtensorMap vmap) {
  constexpr int NB = STREAMS == 1 ? 3 : 2;       // S / P buffers of a stream
  static_assert(HD % 64 == 0 && STREAMS * (NB * 64 + HD) <= 512, "S and O of every stream share the tensor memory");
  constexpr bool LAZY = STREAMS == 2;            // see kTcLazyLog2
  constexpr int TILE = kPageTok * HD * 2;        // a K or V page: 64-column chunks of 8 KB
  constexpr int Q_BYTES = kTcRows * HD * 2;                                   // 64-column chunks of 16 KB
  // TMEM columns: S of stream t, buffer b at (t * NB + b) * 64; O of stream t behind them
  constexpr uint32_t TMEM_COLS = 512, O_COL = STREAMS * NB * 64;
  const float NEG_INF = __int_as_float(0xff800000);
  grid_dep_launch();
  grid_dep_wait();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* q_s = smem;
  uint8_t* k_s = smem + Q_BYTES;                // [NK] pages
  uint8_t* v_s = k_s + NK * TILE;             // [NV] pages
  __shared__ uint64_t k_full[NK], k_empty[NK], v_full[NV], v_empty[NV], s_full[STREAMS][NB], p_full[STREAMS][NB], pv_done[STREAMS][NB];
  __shared__ float s_ml[STREAMS][2][kTcRows];   // (reference maximum, row sum) of the streams' rows
  __shared__ uint32_t tmem_holder;
  __shared__ int s_fail;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // later tiles of a sequence see more keys: they are started first so that the last wave holds the short ones
  const int tile = gridDim.x - 1 - blockIdx.x, kvh = blockIdx.y;
  const int G = p.nq / p.nkv;
  const int first = p.tile_first ? p.tile_first[tile] : tile;
  const int count = p.tile_count ? p.tile_count[tile] : 1;
  const int s = p.slot ? p.slot[first] : 0;
  if (count <= 0 || s < 0) return;              // uniform: before any barrier or TMEM use

  int lim_max = -1, pos_min = 0x7fffffff;
  for (int i = 0; i < count; ++i) {
    const int ps = p.pos[first + i];
    const int lm = p.key_end ? p.key_end[first + i] : ps;
    lim_max = max(lim_max, lm);
    pos_min = min(pos_min, ps);
  }
  const int kt_end = lim_max / kPageTok + 1;
  const int kt_begin = p.window > 0 ? max(0, pos_min - p.window + 1) / kPageTok : 0;
  const int n = kt_end - kt_begin;

  if (tid == 0) {
    for (int i = 0; i < NK; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < NV; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < STREAMS; ++i) {
      for (int b = 0; b < NB; ++b) { mbar_init(&s_full[i][b], 1); mbar_init(&p_full[i][b], 128); mbar_init(&pv_done[i][b], 1); }
    }
    s_fail = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_holder, TMEM_COLS);
    tmem_relinquish();
  }
  // a softmax thread owns one row of one stream: TMEM lane = 32 * (warp % 4) + lane, stream = (warp - 2) / 4
  const int r = (warp & 3) * 32 + lane;
  const int strm = warp >= 6 ? 1 : 0;
  const bool r_ok = warp >= 2 && r < count * G;
  const int rr = r_ok ? r : 0;
  const int r_tok = first + rr / G, r_head = kvh * G + rr % G;
  const int r_pos = p.pos[r_tok];
  const int r_lim = p.key_end ? p.key_end[r_tok] : r_pos;
  if (warp >= 2) {
    // the streams' threads share the 64-column chunks of their row of Q
#pragma unroll
    for (int c = 0; c < HD / 64; ++c) {
      if (STREAMS == 2 && (c & 1) != strm) continue;
      const uint4* src = reinterpret_cast<const uint4*>(p.q + (long)r_tok * p.q_stride + (long)r_head * HD) + c * 8;
#pragma unroll
      for (int ch = 0; ch < 8; ++ch) {
        const uint4 v = r_ok ? src[ch] : make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(q_s + c * (kTcRows * 128) + r * 128 + ((ch ^ (r & 7)) << 4)) = v;
      }
    }
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ page loads
    if (elect_one()) {
      prefetch_tmap(&kmap);
      prefetch_tmap(&vmap);
      auto row_of = [&](int j) { return (p.page_table[(long)s * p.max_pages + kt_begin + j] * p.nkv + kvh) * kPageTok; };
      auto load_k = [&](int j) {
        const int st = j % NK;
        if (j >= NK && !mbar_wait(&k_empty[st], ((j / NK) - 1) & 1)) return false;
        const int row = row_of(j);
        mbar_expect_tx(&k_full[st], TILE);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) tma_load_2d(k_s + st * TILE + c * 8192, &kmap, &k_full[st], c * 64, row);
        return true;
      };
      auto load_v = [&](int j) {
        const int st = j % NV;
        if (j >= NV && !mbar_wait(&v_empty[st], ((j / NV) - 1) & 1)) return false;
        const int row = row_of(j);
        mbar_expect_tx(&v_full[st], TILE);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) tma_load_2d(v_s + st * TILE + c * 8192, &vmap, &v_full[st], c * 64, row);
        return true;
      };
      // the scores of a page are asked for in front of the product of the page before
      // (a tile whose key limits all lie in front of its window has no page: a load that nobody waits for must not be in flight when it ends)
      bool ok = n <= 0 || load_k(0);
      for (int j = 0; j < n && ok; ++j) {
        if (j + 1 < n) ok = load_k(j + 1);
        if (ok) ok = load_v(j);
      }
      if (!ok) atomicExch(&s_fail, 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issue
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_f16(1, 1, kTcRows, kPageTok);
      constexpr uint32_t idesc_pv = make_idesc_f16(1, 1, kTcRows, HD) | (1u << 16);      // B (the V page) is MN-major
      const uint32_t q_a = smem_u32(q_s), k_a = smem_u32(k_s), v_a = smem_u32(v_s);
      bool ok = true;
      // page j belongs to stream j % STREAMS and is that stream's page j / STREAMS
      auto issue_s = [&](int j) {
        const int st = j % NK, t = j % STREAMS, i = j / STREAMS, b = i % NB;
        // the buffer held P of the stream's page i - NB: MMAs of different shapes are not ordered, so its PV has to be complete
        if (i >= NB && !mbar_wait(&pv_done[t][b], (i / NB - 1) & 1)) return false;
        if (!mbar_wait(&k_full[st], (j / NK) & 1)) return false;
        tc_fence_after();
        const uint32_t kb = k_a + st * TILE;
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const int c = kk >> 2, off = (kk & 3) * 2;
          tc_mma_f16(tmem_base + (t * NB + b) * kPageTok, make_desc_sw128(q_a + c * (kTcRows * 128)) + off,
                     make_desc_sw128(kb + c * 8192) + off, idesc_s, kk ? 1u : 0u);
        }
        tc_commit(&k_empty[st]);
        tc_commit(&s_full[t][b]);
        return true;
      };
      for (int j = 0; j < STREAMS && j < n && ok; ++j) ok = issue_s(j);
      for (int j = 0; j < n && ok; ++j) {
        if (j + STREAMS < n) ok = issue_s(j + STREAMS);
        if (!ok) break;
        const int t = j % STREAMS, i = j / STREAMS;
        ok = mbar_wait(&p_full[t][i % NB], (i / NB) & 1) && mbar_wait(&v_full[j % NV], (j / NV) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t vb = v_a + (j % NV) * TILE;
#pragma unroll
        for (int ks = 0; ks < kPageTok / 16; ++ks)
          tc_mma_f16_ta(tmem_base + O_COL + t * HD, tmem_base + (t * NB + i % NB) * kPageTok + ks * 8,
                        make_desc_sw128_mn(vb + ks * 2048, 8192u, 1024u), idesc_pv, (i | ks) ? 1u : 0u);
        tc_commit(&pv_done[t][i % NB]);
        tc_commit(&v_empty[j % NV]);
      }
      if (!ok) atomicExch(&s_fail, 1);
    }
  } else {
    // ------------------------------------------------------------------ softmax and correction of one stream
    const uint32_t t_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t o_col = O_COL + strm * HD;
    const int n_mine = (n - strm + STREAMS - 1) / STREAMS;
    float m_ref = NEG_INF, l0 = 0.f, l1 = 0.f;
    bool ok = true;
    for (int i = 0; i < n_mine; ++i) {
      const int b = i % NB, key0 = (kt_begin + STREAMS * i + strm) * kPageTok;
      ok = __all_sync(0xffffffffu, mbar_wait(&s_full[strm][b], (i / NB) & 1));
      if (!ok) break;
      tc_fence_after();
      float sv[kPageTok];
      tmem_ld32(t_lane + (strm * NB + b) * kPageTok, reinterpret_cast<uint32_t*>(sv));
      tmem_ld32(t_lane + (strm * NB + b) * kPageTok + 32, reinterpret_cast<uint32_t*>(sv) + 32);
      tmem_ld_wait();
      if (!r_ok || key0 + kPageTok - 1 > r_lim || (p.window > 0 && key0 <= r_pos - p.window)) {
#pragma unroll
        for (int e = 0; e < kPageTok; ++e) {
          const int key = key0 + e;
          const bool allow = r_ok && key <= r_lim && (p.window <= 0 || key > r_pos - p.window);
          sv[e] = allow ? sv[e] : NEG_INF;
        }
      }
      float mx0 = sv[0], mx1 = sv[1], mx2 = sv[2], mx3 = sv[3];
#pragma unroll
      for (int e = 4; e < kPageTok; e += 4) {
        mx0 = fmaxf(mx0, sv[e]);
        mx1 = fmaxf(mx1, sv[e + 1]);
        mx2 = fmaxf(mx2, sv[e + 2]);
        mx3 = fmaxf(mx3, sv[e + 3]);
      }
      const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * p.scale_log2;     // the scale is positive
      const bool grow = mx > (LAZY ? m_ref + kTcLazyLog2 : m_ref);
      float alpha = 1.f;
      if (grow) {
        alpha = ex2_approx(m_ref - mx);          // 0 for the first keys a row sees
        m_ref = mx;
      }
      const bool fix = i > 0 && __any_sync(0xffffffffu, grow);
      // The stream's previous PV is the last writer of O: a row correction waits for it. (P goes to the buffer of its own S, which no MMA
      // in flight reads.)
      if (fix) {
        ok = __all_sync(0xffffffffu, mbar_wait(&pv_done[strm][(i - 1) % NB], ((i - 1) / NB) & 1));
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c0 = 0; c0 < HD; c0 += 32) {
          uint32_t ov[32];
          tmem_ld32(t_lane + o_col + c0, ov);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * alpha);
          tmem_st32(t_lane + o_col + c0, ov);
        }
        tmem_st_wait();
      }
      l0 *= alpha;
      l1 *= alpha;
      const float neg_m = m_ref == NEG_INF ? 0.f : -m_ref;
      uint32_t w[kPageTok / 2];
#pragma unroll
      for (int e = 0; e < kPageTok / 2; ++e) {
        const float p0 = ex2_approx(LAZY ? fmaf(sv[2 * e], p.scale_log2, neg_m) : __fadd_rn(__fmul_rn(sv[2 * e], p.scale_log2), neg_m));
        const float p1 = ex2_approx(LAZY ? fmaf(sv[2 * e + 1], p.scale_log2, neg_m) : __fadd_rn(__fmul_rn(sv[2 * e + 1], p.scale_log2), neg_m));
        l0 += p0;
        l1 += p1;
        w[e] = pack_bf16(p0, p1);
      }
      __syncwarp();                                // (masks and maxima let lanes part; the store wants the whole warp)
      tmem_st32(t_lane + (strm * NB + b) * kPageTok, w);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[strm][b]);              // (a barrier a buffer: a fast warp may be a page ahead of a slow one)
    }
    if (n_mine > 0) ok = __all_sync(0xffffffffu, ok && mbar_wait(&pv_done[strm][(n_mine - 1) % NB], ((n_mine - 1) / NB) & 1));
    if (!ok) atomicExch(&s_fail, 1);
    s_ml[strm][0][r] = m_ref;
    s_ml[strm][1][r] = l0 + l1;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp >= 2 && !s_fail) {
    // ------------------------------------------------------------------ merge of the two streams and output
    // each stream's threads write their share of the columns of their row
    const uint32_t t_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    const bool two = STREAMS == 2 && n > 1;                  // (a one-page tile never wrote the second accumulator)
    const float m0 = s_ml[0][0][r], m1 = two ? s_ml[STREAMS - 1][0][r] : NEG_INF;
    const float m = fmaxf(m0, m1);
    const float a0 = m == NEG_INF ? 0.f : ex2_approx(m0 - m), a1 = (m == NEG_INF || !two) ? 0.f : ex2_approx(m1 - m);
    const float l = s_ml[0][1][r] * a0 + (two ? s_ml[STREAMS - 1][1][r] * a1 : 0.f);
    const float inv = l > 0.f ? 1.f / l : 0.f;
    const float f0 = a0 * inv, f1 = a1 * inv;
    __nv_bfloat16* orow = p.out + (long)r_tok * p.out_stride + (long)r_head * HD;
    const __nv_bfloat16* grow_ = p.gate ? p.gate + (long)r_tok * p.gate_stride + (long)r_head * HD : nullptr;
#pragma unroll 1
    for (int c0 = strm * (HD / STREAMS); c0 < (strm + 1) * (HD / STREAMS); c0 += 32) {
      uint32_t ov[32], ow[32];
      tmem_ld32(t_lane + O_COL + c0, ov);
      if (two) tmem_ld32(t_lane + O_COL + HD + c0, ow);
      tmem_ld_wait();
      if (n <= 0) {                                          // (nothing was accumulated: the row is zero)
#pragma unroll
        for (int e = 0; e < 32; ++e) ov[e] = 0u;
      }
      if (r_ok) {
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint32_t w[4];
          uint32_t gw[4] = {0u, 0u, 0u, 0u};
          if (grow_) {
            const uint4 g4 = *reinterpret_cast<const uint4*>(grow_ + c0 + q4 * 8);
            gw[0] = g4.x; gw[1] = g4.y; gw[2] = g4.z; gw[3] = g4.w;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float a = __uint_as_float(ov[q4 * 8 + 2 * e]) * f0, c = __uint_as_float(ov[q4 * 8 + 2 * e + 1]) * f0;
            if (two) {
              a = fmaf(__uint_as_float(ow[q4 * 8 + 2 * e]), f1, a);
              c = fmaf(__uint_as_float(ow[q4 * 8 + 2 * e + 1]), f1, c);
            }
            if (grow_) {
              const __nv_bfloat162 g2 = *reinterpret_cast<const __nv_bfloat162*>(&gw[e]);
              a *= 1.f / (1.f + __expf(-__low2float(g2)));
              c *= 1.f / (1.f + __expf(-__high2float(g2)));
            }
            w[e] = pack_bf16(a, c);
          }
          *reinterpret_cast<uint4*>(orow + c0 + q4 * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (tid == 0 && s_fail && p.status) atomicExch(p.status, (int)kErrMbarTimeout);
}

template <int HD, int STREAMS, int NK, int NV>
static int launch_attn_tc(const AttnParams& p, const CUtensorMap& kmap, const CUtensorMap& vmap, int ntiles, cudaStream_t st) {
  constexpr int smem = kTcRows * HD * 2 + NK * kPageTok * HD * 2 + NV * kPageTok * HD * 2 + 1024;
  static_assert(smem <= 225 * 1024, "shared memory budget (beside 2 KB of barriers and row sums)");
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc_kernel<HD, STREAMS, NK, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  launch_pdl(attn_prefill_tc_kernel<HD, STREAMS, NK, NV>, dim3(ntiles, p.nkv, 1), dim3(64 + 128 * STREAMS), smem, st, p, kmap, vmap);
  return (int)cudaGetLastError();
}

}  // namespace ve
