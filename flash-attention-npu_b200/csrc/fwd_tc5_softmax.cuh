// Softmax role and correction / epilogue role of the tcgen05 prefill kernel.
//
// The softmax warps are the kernel's slowest chain: two of them share a scheduler, and next to 2050 cycles of exponentials for a
// block of both sub-tiles a block took them 3700.  So whatever they do once a block counts: the mask's range as two compares, no
// wait for the correction warps (corr_ready), arrivals without a branch, one instruction per address of P, the maximum as a tree.
// 4 K causal, b 4, 32 heads, head dim 64 510 -> 468 us, head dim 128 674 -> 647 under the power cap.
//
// Softmax: 128 threads per query sub-tile, one thread per query row (TMEM lane); 256-column tiles have one sub-tile and two
// threads per row, 64 keys of a block each.  It restates the
// arithmetic of the reference's OnlineSoftmax epilogue
// (csrc/arch22/flash_attn_npu_v2/online_softmax.hpp:479-803) in the log2 domain:
//   P = exp2(S * scale*log2e - m * scale*log2e), rounded to the input dtype before P.V.
// The 128 scores of a row are held in registers (the softmax warps raise their register budget
// with setmaxnreg, the other roles lower theirs).
//
// P leaves the thread as 16-byte chunks of 8 keys written to shared memory in the layout the MMA
// reads an A operand in (128-byte rows, 128-byte swizzle, two 64-key halves).  At the end of a tile
// the thread writes LSE = m*scale + ln(l) and hands 1 / l to the correction warps.
//
// Correction: 128 threads serving both sub-tiles.  When a row maximum moved it multiplies O (in
// TMEM) by exp2((m_old - m_new) * scale*log2e) between two P.V accumulations, off the softmax
// threads' critical path, and at the end of a tile writes O / l
// (RescaleO, csrc/arch22/flash_attn_npu_v2/rescale_o.hpp:299-534).
#pragma once

#include "fwd_tc5_kernel.cuh"

namespace fa {
namespace tc5 {

// Maximum of m and 32 scores, as a tree (a few chains of three-operand maxima take twice as long as their 16 instructions issue).
__device__ __forceinline__ float chunk_max(const uint32_t (&a)[32], float m) {
  float r[11];
#pragma unroll
  for (int e = 0; e < 10; ++e) r[e] = max3(__uint_as_float(a[3 * e]), __uint_as_float(a[3 * e + 1]), __uint_as_float(a[3 * e + 2]));
  r[10] = max3(__uint_as_float(a[30]), __uint_as_float(a[31]), m);
  const float x = max3(r[0], r[1], r[2]), y = max3(r[3], r[4], r[5]), z = max3(r[6], r[7], r[8]);
  return max3(max3(x, y, z), r[9], r[10]);
}

// Columns outside [lo, hi] become -inf.  The valid columns of the chunk form one bit mask, so an
// element costs a bit test and a select (per-element range compares were several times slower).
__device__ __forceinline__ void chunk_mask(uint32_t (&a)[32], int col_first, int lo, int hi) {
  const int n_lo = min(max(lo - col_first, 0), 32);       // first valid element of the chunk
  const int n_hi = min(max(hi - col_first + 1, 0), 32);   // one past the last valid element
  const uint32_t below_hi = n_hi >= 32 ? 0xffffffffu : ((1u << n_hi) - 1u);
  const uint32_t below_lo = n_lo >= 32 ? 0xffffffffu : ((1u << n_lo) - 1u);
  const uint32_t valid = below_hi & ~below_lo;
#pragma unroll
  for (int e = 0; e < 32; ++e)
    if (!((valid >> e) & 1u)) a[e] = 0xff800000u;  // -inf
}

// softcap: s -> softcap * tanh(s * scale / softcap), here straight into the log2 domain (tests/test_flash_attn_npu_v2.py:
// the golden applies it to the scaled scores before the mask).  tanh.approx has a relative error of 2^-11: one unit of the
// last place of a capped score of 30 .. 50 is 0.02.
__device__ __forceinline__ void chunk_softcap(uint32_t (&a)[32], float mul, float cap_l2) {
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    float th;
    asm("tanh.approx.f32 %0, %1;\n" : "=f"(th) : "f"(__uint_as_float(a[e]) * mul));
    a[e] = __float_as_uint(th * cap_l2);
  }
}

// Build-time tuning constants of the softmax role.
#ifndef FA_TC5_POLY
#define FA_TC5_POLY 0
#endif
#ifndef FA_TC5_RESCALE_THRESHOLD
#define FA_TC5_RESCALE_THRESHOLD 0.f
#endif
constexpr int kPolyPairs = FA_TC5_POLY;  // of every 4 pairs of exponentials, how many use the polynomial
constexpr float kRescaleThreshold = FA_TC5_RESCALE_THRESHOLD;

// 32 scores -> 16 packed 16-bit pairs of P, accumulating the fp32 row sum (two partial sums).
// POLY of every 4 pairs use the polynomial, the others the special-function unit.
template <typename T, int POLY>
__device__ __forceinline__ void chunk_exp(const uint32_t (&a)[32], uint64_t scale2, uint64_t negms2, uint64_t (&sum2)[4],
                                          uint32_t (&pk)[16]) {
#pragma unroll
  for (int e = 0; e < 32; e += 2) {
    const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(a[e]), __uint_as_float(a[e + 1])), scale2, negms2);
    float p0, p1;
    if (((e >> 1) & 3) < POLY) {
      poly_exp2_x2(x2, p0, p1);
    } else {
      float x0, x1;
      unpack_f32x2(x2, x0, x1);
      p0 = fast_exp2(x0);
      p1 = fast_exp2(x1);
    }
    sum2[(e >> 1) & 3] = add_f32x2(sum2[(e >> 1) & 3], pack_f32x2(p0, p1));  // four independent chains
    pk[e >> 1] = pack2<T>(p0, p1);
  }
}

// 32 keys of P (16 packed pairs = four 16-byte chunks) of one row into the swizzled A-operand tile: 16-byte chunk kc of a row lies
// at  half(kc) + row * 128 + ((kc ^ row) & 7) * 16.  p_row holds chunk 0, so a chunk's address is one exclusive-or away.
__device__ __forceinline__ void store_p_chunk(uint32_t p_row, int c, const uint32_t (&pk)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t kc = (uint32_t)(c * 4 + q);
    const uint32_t addr = (p_row ^ ((kc & 7) << 4)) + (kc >> 3) * kHalfBytes;
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(pk[4 * q]), "r"(pk[4 * q + 1]),
                 "r"(pk[4 * q + 2]), "r"(pk[4 * q + 3])
                 : "memory");
  }
}

// The same through an exponential and a division, 1 - 2 / (e^2y + 1), as the mma.sync and decode kernels compute it: the
// form of the calls that those kernels served before (packed queries against a cache).  Two special-function results per
// score instead of one.
__device__ __forceinline__ void chunk_softcap_fine(uint32_t (&a)[32], float mul, float cap_l2) {
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    const float ex = __expf(2.f * (__uint_as_float(a[e]) * mul));
    a[e] = __float_as_uint(cap_l2 * (1.f - __fdividef(2.f, ex + 1.f)));
  }
}

template <typename T, int IN, int CAP, int HD>
__device__ __forceinline__ void softmax_loop(const Tc5Params& p, Barriers* bar, uint32_t tmem, uint32_t p_smem, int wg,
                                             int warp_in_wg, int lane) {
  // With 256 columns there is one sub-tile, and one warpgroup by itself leaves the special-function unit idle for most of a
  // block: both warpgroups share its rows.  b 2, s 2047, 16 / 8 heads, head dim 256, softcap 50: 100 -> 91 us; b 2, s 1777,
  // 8 heads, forward and backward 190 -> 188.
  constexpr bool kWide = Geo<HD>::kWide;
  constexpr int kChunks = kWide ? 2 : 4;       // of 32 keys
  const int t = kWide ? 0 : wg;                // sub-tile
  const int chunk0 = kWide ? 2 * wg : 0;       // first chunk of this thread in a block
  const bool lead = !kWide || wg == 0;         // writes the row's factors and statistics
  volatile int* abort_flag = &bar->abort_flag;
  const int row = warp_in_wg * 32 + lane;
  const uint32_t lane_addr = (uint32_t)(warp_in_wg * 32) << 16;
  const uint32_t s_tmem = tmem + lane_addr + t * 128 + chunk0 * 32;
  uint32_t s_cnt = 0, ev_cnt = 0;  // blocks, events (corr_ready) so far
  constexpr int kPBufs = Geo<HD>::kPBufs;
  const uint32_t p_row0 = p_smem + t * kPBufs * kTileBytes + row * 128 + ((row & 7) << 4);
  const uint32_t bar_sfree = smem_addr(&bar->s_free[t]), bar_odone = smem_addr(&bar->o_done[t][0]);
  // with softcap the scores are in the log2 domain once they have been capped: the scale is part of the cap
  const float scale_log2 = CAP ? 1.f : p.scale_log2;
  const float lse_scale = CAP ? 0.6931471805599453f : p.a.softmax_scale;  // running maximum -> natural log
  const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2);

  // What the row's other thread has, through a TMEM column each.  Two pairs of columns in turn: a pair is written again only
  // when the other side has been through the exchange in between, which it enters after it has read this one.
  uint32_t x_cnt = 0;
  auto exchange = [&](float v, float& other) -> bool {
    const uint32_t col = tmem + lane_addr + kXchgCol + 2 * (x_cnt & 1);
    tmem_st1(col + wg, __float_as_uint(v));
    tmem_wait_st();
    tc_fence_before();
    __syncwarp();
    mbar_arrive_lane0(smem_addr(&bar->exchanged), lane);
    if (!mbar_wait(smem_addr(&bar->exchanged), x_cnt & 1, abort_flag, 49)) return false;
    tc_fence_after();
    ++x_cnt;
    uint32_t r;
    tmem_ld1(col + 1 - wg, r);
    tmem_wait_ld();
    other = __uint_as_float(r);
    return true;
  };

  TileWalk<IN> walk(bar);
  for (int n = walk.first(p); n < p.total_tiles; n = walk.next(p)) {
    const SubTile ti = sub_tile<Geo<HD>::kRows>(p, tile_id<IN>(p, n), t);
    if (ti.row0 >= ti.q_len) continue;
    const int i = ti.row0 + row;
    if (ti.jhi <= ti.jlo) {  // no visible key for the whole sub-tile: O = 0, LSE = +inf
      if (lead && i < ti.q_len) {
        T* o_ptr = reinterpret_cast<T*>(p.a.o) + (int64_t)ti.bi * p.a.o_batch_stride +
                   (int64_t)(ti.q_row0 + i) * p.a.o_row_stride + (int64_t)ti.hh * p.a.o_head_stride;
        for (int c = 0; c < p.a.d; c += 8) *reinterpret_cast<uint4*>(o_ptr + c) = make_uint4(0, 0, 0, 0);
        p.a.lse[(int64_t)ti.bi * p.a.lse_batch_stride + (int64_t)ti.hh * p.a.lse_head_stride + ti.q_row0 + i] = INFINITY;
      }
      continue;
    }
    int lo = 0, hi = ti.k_len - 1;
    if (p.is_causal) hi = min(hi, i + ti.koff);
    if (p.is_local) {
      hi = min(hi, i + ti.koff + p.wr);
      lo = max(0, i + ti.koff - p.wl);
    }
    const int i_min = ti.row0, i_max = min(ti.q_len, ti.row0 + kBlockM) - 1;
    float m_run = -INFINITY, l_run = 0.f;
    // blocks [full_lo, full_hi) need no mask
    int full_lo = 0, full_hi = ti.k_len / kBlockN;
    if (p.is_causal || p.is_local) full_hi = min(full_hi, max(0, i_min + ti.koff + (p.is_local ? p.wr : 0) + 1) / kBlockN);
    if (p.is_local) full_lo = ceil_div(max(0, i_max + ti.koff - p.wl), kBlockN);

    for (int j = ti.jlo; j < ti.jhi; ++j) {
      const int col0 = j * kBlockN;
      const bool need_mask = j < full_lo || j >= full_hi;

      if (!mbar_wait(smem_addr(&bar->s_full[t]), s_cnt & 1, abort_flag, 41)) return;
      const uint32_t blk = s_cnt;  // running number of this block (all tiles of this CTA)
      ++s_cnt;
      tc_fence_after();
      // ---- the scores into registers (one TMEM round trip) ----
      uint32_t sc[kChunks][32];
#pragma unroll
      for (int c = 0; c < kChunks; ++c) tmem_ld32(s_tmem + c * 32, sc[c]);
      tmem_wait_ld();
      // the S columns are free: Q.K^T of the next block may overwrite them
      tc_fence_before();
      __syncwarp();
      mbar_arrive_lane0(bar_sfree, lane);
      if (CAP) {
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          if (CAP == kCapFine) chunk_softcap_fine(sc[c], p.softcap_mul, p.softcap_l2);
          else chunk_softcap(sc[c], p.softcap_mul, p.softcap_l2);
        }
      }
      if (need_mask) {
#pragma unroll
        for (int c = 0; c < kChunks; ++c) chunk_mask(sc[c], col0 + (chunk0 + c) * 32, lo, hi);
      }
      float blk_max = chunk_max(sc[0], -INFINITY);
#pragma unroll
      for (int c = 1; c < kChunks; ++c) blk_max = chunk_max(sc[c], blk_max);
      if (kWide) {
        float other;
        if (!exchange(blk_max, other)) return;
        blk_max = fmaxf(blk_max, other);
      }

      float m_new = fmaxf(m_run, blk_max);
      // The running maximum follows every increase (P <= 1, and the row maximum has P = 1 exactly, like the
      // reference's golden).  kRescaleThreshold > 0 (log2 units) would keep the old maximum while the new one is
      // within the threshold: fewer O rescales for a few ulps of P rounding on sharply peaked rows.
      if (kRescaleThreshold > 0.f && m_run != -INFINITY && (m_new - m_run) * scale_log2 <= kRescaleThreshold) m_new = m_run;
      const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
      const float corr = fast_exp2((m_run - m_use) * scale_log2);  // 0 when m_run = -inf
      if (lead && j > ti.jlo) {
        bar->corr[t][ev_cnt & 1][row] = (m_new != m_run) ? corr : 1.f;
        __syncwarp();
        mbar_arrive_lane0(smem_addr(&bar->corr_ready[t][ev_cnt & 1]), lane);
        ++ev_cnt;
      }
      m_run = m_new;
      const float neg_ms = -m_use * scale_log2;
      const uint64_t negms2 = pack_f32x2(neg_ms, neg_ms);

      // ---- exponentials, P -> shared memory ----
      uint64_t sum2[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) sum2[q] = pack_f32x2(0.f, 0.f);
      // P.V of the previous block must have read P_t before it is overwritten.  For 128 columns the wait stands behind half of
      // the row's exponentials: b4 s4096 h32 causal 669 -> 661 us, full 1204 -> 1160 (three quarters: 673, 1200, P.V starts too
      // late); elsewhere behind a quarter.  Half is slower for 64 and 256 columns (1.5 %), with softcap, whose scores are ready
      // late by themselves (b2 s4096 h16 full 431 -> 444 us, b1 s1061 h16 causal 31.8 -> 32.4), and where no tile follows another
      // (ragged input, fixed deal: 6 chunks of 705 rows against 1307 keys 32.4 -> 33.4, 5 of 135 rows 19.5 -> 19.8).
      constexpr bool kHalfAhead = HD == 128 && CAP == kCapNone && IN != kRaggedFixed;
      const uint32_t buf = blk % kPBufs, p_row = p_row0 + buf * kTileBytes;
      uint32_t pk[16], pk1[16];
      chunk_exp<T, kPolyPairs>(sc[0], scale2, negms2, sum2, pk);
      if (kHalfAhead) chunk_exp<T, kPolyPairs>(sc[1], scale2, negms2, sum2, pk1);
      if (kPBufs == 1 && blk > 0 && !mbar_wait(bar_odone, (blk - 1) & 1, abort_flag, 42)) return;
      store_p_chunk(p_row, chunk0, pk);
      if (!kHalfAhead) chunk_exp<T, kPolyPairs>(sc[1], scale2, negms2, sum2, pk1);
      store_p_chunk(p_row, chunk0 + 1, pk1);
      fence_proxy_async();  // generic-proxy stores -> visible to the MMA (async proxy)
      __syncwarp();
      mbar_arrive_lane0(smem_addr(&bar->p_full[t][buf][kWide ? wg : 0]), lane);  // the first (this warpgroup's) 64 keys of P are ready
      if constexpr (!kWide) {
        chunk_exp<T, kPolyPairs>(sc[2], scale2, negms2, sum2, pk);
        store_p_chunk(p_row, 2, pk);
        chunk_exp<T, kPolyPairs>(sc[3], scale2, negms2, sum2, pk);
        store_p_chunk(p_row, 3, pk);
        fence_proxy_async();
        __syncwarp();
        mbar_arrive_lane0(smem_addr(&bar->p_full[t][buf][1]), lane);  // last 64 keys
      }
      float s0, s1;
      unpack_f32x2(add_f32x2(add_f32x2(sum2[0], sum2[1]), add_f32x2(sum2[2], sum2[3])), s0, s1);
      l_run = l_run * corr + (s0 + s1);
    }
    if (kWide) {
      float other;
      if (!exchange(l_run, other)) return;
      l_run += other;
      if (!lead) continue;
    }
    // 1 / l for the epilogue, LSE from here.  The event behind the tile's last block n waits for P.V of block n - 1 (corr_ready).
    if (kPBufs > 1 && s_cnt > 1 && !mbar_wait(bar_odone + 8 * (s_cnt % kPBufs), ((s_cnt - 2) / kPBufs) & 1, abort_flag, 42)) return;
    bar->corr[t][ev_cnt & 1][row] = l_run > 0.f ? 1.f / l_run : 0.f;
    __syncwarp();
    mbar_arrive_lane0(smem_addr(&bar->corr_ready[t][ev_cnt & 1]), lane);
    ++ev_cnt;
    // m_run * lse_scale + ln l.  Which product is fused into the sum is written out: both factors are constants with softcap, the
    // compiler's choice changed with the code around it, and a backward that reads the LSE gets other bits then.
    const float lse = CAP ? fmaf(__log2f(l_run), 0.6931471805599453f, __fmul_rn(m_run, lse_scale)) : fmaf(m_run, lse_scale, __logf(l_run));
    if (i < ti.q_len)
      p.a.lse[(int64_t)ti.bi * p.a.lse_batch_stride + (int64_t)ti.hh * p.a.lse_head_stride + ti.q_row0 + i] = l_run > 0.f ? lse : INFINITY;
  }
}

// Multiplies the HD fp32 columns of one TMEM lane by f (two chunks in flight).
template <int HD>
__device__ __forceinline__ void rescale_o(uint32_t o_tmem, float f) {
  const uint64_t f2 = pack_f32x2(f, f);
  // 256 columns: one chunk at a time.  Spilled bytes (stored / loaded) with the form below and with this one: dense 8 / 60 and
  // 4 / 44, run-time draw 420 - 432 / 424 - 492 and 12 / 68 without softcap, none with it, fixed deal none either way.
  if constexpr (HD > 128) {
#pragma unroll 1
    for (int c = 0; c < HD; c += 32) {
      uint32_t a[32];
      tmem_ld32(o_tmem + c, a);
      tmem_wait_ld();
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        float x0, x1;
        unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(a[e]), __uint_as_float(a[e + 1])), f2), x0, x1);
        a[e] = __float_as_uint(x0);
        a[e + 1] = __float_as_uint(x1);
      }
      tmem_st32(o_tmem + c, a);
    }
    tmem_wait_st();
    return;
  }
  uint32_t a[32], b[32];
  tmem_ld32(o_tmem, a);
  tmem_ld32(o_tmem + 32, b);
  tmem_wait_ld();
#pragma unroll
  for (int half = 0; half < HD / 64; ++half) {
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
      float x0, x1;
      unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(a[e]), __uint_as_float(a[e + 1])), f2), x0, x1);
      a[e] = __float_as_uint(x0);
      a[e + 1] = __float_as_uint(x1);
      unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(b[e]), __uint_as_float(b[e + 1])), f2), x0, x1);
      b[e] = __float_as_uint(x0);
      b[e + 1] = __float_as_uint(x1);
    }
    tmem_st32(o_tmem + half * 64, a);
    tmem_st32(o_tmem + half * 64 + 32, b);
    if (half + 1 < HD / 64) {
      tmem_ld32(o_tmem + (half + 1) * 64, a);
      tmem_ld32(o_tmem + (half + 1) * 64 + 32, b);
      tmem_wait_ld();
    }
  }
  tmem_wait_st();
}

// 64 columns of a row of O, of which the first n_cols exist (head dims between the tile widths: the tiles' other columns are the
// zeros that the TMA unit fills in).  A warp's store touches 32 rows, a line each, and the load / store unit takes them one by
// one, whether 16 or 32 bytes go there: with 16 a CTA tile's epilogue held the correction warps, and through them the next tile's
// first P.V, for some 4000 cycles.  SECTORS stores whole 32-byte sectors, where the rows allow it (o_sectors); 16 / 32 bytes:
// 12 x 148 heads of 256 rows, head dim 64 102.4 / 95.4 us, head dim 128 127 / 107, of 128 rows, head dim 256 100 / 86;
// b 4, s 2048, 16 heads, head dim 256, causal 151 / 147; 4 K causal, head dim 128, no difference.
template <bool SECTORS, typename T>
__device__ __forceinline__ void store_cols(T* dst, const uint32_t (&w)[32], int n_cols) {
#pragma unroll
  for (int c = 0; c < 32; c += SECTORS ? 8 : 4) {
    if (2 * c >= n_cols) continue;
    if (SECTORS) {
      store_sector(dst + 2 * c, w, c);
    } else {  // written once, read by nobody here: streaming
      __stcs(reinterpret_cast<uint4*>(dst + 2 * c), make_uint4(w[c], w[c + 1], w[c + 2], w[c + 3]));
    }
  }
}

template <typename T, int IN, int HD>
__device__ __forceinline__ void correction_loop(const Tc5Params& p, Barriers* bar, uint32_t tmem, int warp_in_wg,
                                                int lane) {
  volatile int* abort_flag = &bar->abort_flag;
  const int row = warp_in_wg * 32 + lane;
  const uint32_t lane_addr = (uint32_t)(warp_in_wg * 32) << 16;
  uint32_t ev_cnt[2] = {0, 0}, od_cnt[2] = {0, 0};
  constexpr uint32_t kPBufs = Geo<HD>::kPBufs;
  const int d_cols = p.a.d;

  TileWalk<IN> walk(bar);
  for (int n = walk.first(p); n < p.total_tiles; n = walk.next(p)) {
    TileInfo ti;
    tile_info<Geo<HD>::kRows>(p, tile_id<IN>(p, n), ti);
    if (ti.uhi <= ti.ulo) continue;
    for (int j = ti.ulo; j < ti.uhi; ++j) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (!(ti.has[t] && j > ti.jlo[t] && j < ti.jhi[t])) continue;
        if (!mbar_wait(smem_addr(&bar->corr_ready[t][ev_cnt[t] & 1]), (ev_cnt[t] >> 1) & 1, abort_flag, 43)) return;
        const float f = bar->corr[t][ev_cnt[t] & 1][row];
        ++ev_cnt[t];
        if (!mbar_wait(smem_addr(&bar->o_done[t][od_cnt[t] % kPBufs]), (od_cnt[t] / kPBufs) & 1, abort_flag, 44)) return;  // P.V of block j-1 done
        ++od_cnt[t];
        if (__any_sync(0xffffffffu, f != 1.f)) {
          tc_fence_after();
          rescale_o<HD>(tmem + lane_addr + 256 + t * 128, f);
          tc_fence_before();
        }
        __syncwarp();
        mbar_arrive_lane0(smem_addr(&bar->o_ready[t]), lane);
      }
    }
    // ---- epilogue of both sub-tiles ----
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (!ti.has[t]) continue;
      if (!mbar_wait(smem_addr(&bar->corr_ready[t][ev_cnt[t] & 1]), (ev_cnt[t] >> 1) & 1, abort_flag, 45)) return;
      const float inv = bar->corr[t][ev_cnt[t] & 1][row];
      ++ev_cnt[t];
      if (!mbar_wait(smem_addr(&bar->o_done[t][od_cnt[t] % kPBufs]), (od_cnt[t] / kPBufs) & 1, abort_flag, 46)) return;  // last P.V done
      ++od_cnt[t];
      tc_fence_after();
      const int i = ti.row0[t] + row;
      const bool row_valid = i < ti.q_len;
      T* o_ptr = reinterpret_cast<T*>(p.a.o) + (int64_t)ti.bi * p.a.o_batch_stride +
                 (int64_t)(ti.q_row0 + i) * p.a.o_row_stride + (int64_t)ti.hh * p.a.o_head_stride;
      const uint32_t o_tmem = tmem + lane_addr + 256 + t * 128;
#pragma unroll
      for (int half = 0; half < HD / 64; ++half) {
        uint32_t a[32], b[32];
        tmem_ld32(o_tmem + half * 64, a);
        tmem_ld32(o_tmem + half * 64 + 32, b);
        tmem_wait_ld();
        if (half + 1 == HD / 64) {  // all of O has been read: P.V of the next tile may overwrite it under the last stores
          tc_fence_before();
          __syncwarp();
          mbar_arrive_lane0(smem_addr(&bar->o_free[t]), lane);
        }
        uint32_t w[32];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          w[e >> 1] = pack2<T>(__uint_as_float(a[e]) * inv, __uint_as_float(a[e + 1]) * inv);
          w[16 + (e >> 1)] = pack2<T>(__uint_as_float(b[e]) * inv, __uint_as_float(b[e + 1]) * inv);
        }
        if (row_valid) {
          if (p.o_sectors) store_cols<true>(o_ptr + half * 64, w, d_cols - half * 64);
          else store_cols<false>(o_ptr + half * 64, w, d_cols - half * 64);
        }
      }
    }
  }
}

}  // namespace tc5
}  // namespace fa
