// Attention backward on the Blackwell tensor cores for head dims 129 .. 256 (tiles of 192 or 256 columns), dense and
// packed-varlen input, optional softcap.  Arithmetic and rounding as in bwd_tc5_kernel.cuh; no atomics.
//
// A [128 x 256] fp32 accumulator takes 256 of the 512 TMEM columns, so dK and dV do not fit beside S and dP.  The work is
// cut into three kinds of items, one accumulator each, all in one persistent launch:
//   dK  128 keys     A0 = K, A1 = V    streams X = Q, Y = dO    S^T = A0 X^T, dP^T = A1 Y^T, dS^T;  acc += dS^T X
//   dV  128 keys     A0 = K            streams X = Q, Y = dO    S^T = A0 X^T, P^T;                  acc += P^T Y
//   dQ  128 rows     A0 = Q, A1 = dO   streams X = K, Y = V     S = A0 X^T, dP = A1 Y^T, dS;        acc += dS X
// That is 8 matrix products instead of 5 (S three times, dP twice), which still beats the mma.sync kernel with its fp32
// atomics 4.5 to 7 times: 2 x 1777 rows, 8 heads, head dim 256, causal: 781 -> 172 us; 6 x 1475 rows, 16/8 heads, head
// dim 192: 5.07 -> 0.72 ms; 31 packed sequences of 432 - 1731 rows, 32/8 heads, head dim 192, causal: 15.6 -> 2.5 ms.
// dQ and dK are the same program with the operands' roles exchanged: A0 / A1 stay in shared memory, X / Y stream past them
// in units of 64 rows, the 16-bit dS goes back into the TMEM columns of the S it came from and is the A operand of the
// accumulation.  TMEM: two buffers of [S 64 | dP 64] (the next unit's products run under this unit's elementwise work),
// accumulator [256, 512).
// Shared memory is what bounds the pipeline at 256 columns: A0 and A1 take 128 KiB, which leaves two X slots and one Y slot
// of 32 KiB (X is held until acc has used it, Y until dP has); with 192 columns it is three and two.  dV has no A1: its
// space is two more Y slots.
// Warps 0-15 elementwise and epilogue (0-7 the even, 8-15 the odd units), 16 issues S and acc (in this order in one warp:
// S of unit u + 2 overwrites the operand of acc of unit u, and the tensor pipe keeps the order), 17 issues dP, 19 loads.
// A parity wait only tells the current phase of a barrier from the one before, so no role may be two phases away from a
// barrier it waits on, in either direction.  The resident operands and the Y slots are therefore released by both issuers
// in every item, also in a dV item, where warp 17 has nothing to issue: it waits for a_full and every y_full there and
// releases them itself.  (Without that it reached the next dQ item's waits while a dV item of one or two units was still
// loading, passed them on the parity of the item before, and computed dP from stale tiles.)
// What a wait relies on, phase by phase:
//   a_full, y_full   the next phase needs both issuers' releases; warp 16 looks at y_full in dV items only, but in the
//                    other items its acc of a unit follows that unit's dP, and dP follows y_full
//   x_full, st_full  the next phase needs acc of this unit, which needs pds_full of this unit
//   pds_full         warp 17 waits for unit g - 2 after y_full of unit g, whose slot (and, behind a dV item, the space of
//                    A1) was released by acc of unit g - 2 or a later one, hence after pds_full of every unit before that
//   acc_done, acc_free  each needs the other's phase before it, by all warps
#pragma once

#include "bwd_tc5_kernel.cuh"

namespace fa {
namespace btc5 {

enum WideKind { kWideDK = 0, kWideDV = 1, kWideDQ = 2 };

template <int HD>
struct WideGeo {
  static_assert(HD == 192 || HD == 256, "tile widths");
  static constexpr int kChunks = HD / 64;
  static constexpr int kATile = kChunks * kHalfBytes;   // [128 x HD] resident operand
  static constexpr int kSTile = kChunks * kUnitHalf;    // [64 x HD] streamed tile
  static constexpr int XS = HD == 256 ? 2 : 3;          // X slots
  static constexpr int YS = HD == 256 ? 1 : 2;          // Y slots behind them
  static constexpr int YSV = YS + 2;                    // Y slots of a dV item: A1's space is two more
  static constexpr int kRingOff = 2 * kATile;
  static constexpr int kBarOff = kRingOff + (XS + YS) * kSTile;
  static constexpr int kStats = XS + 2;                 // per-unit LSE / D arrays: the loader is at most XS + 1 units ahead of their last reader
  // byte offset of Y slot i
  __device__ static __forceinline__ uint32_t y_off(int i) {
    return i < YS ? kRingOff + (XS + i) * kSTile : kATile + (i - YS) * kSTile;
  }
  static_assert(kATile == 2 * kSTile, "A1's space is two Y slots");
};

template <int HD>
struct BarW {
  uint64_t a_full, a_empty;  // A0 / A1 of the item have landed; its last S and dP have read them (dV: its last S has, and the dP issuer has seen a_full)
  uint64_t x_full[WideGeo<HD>::XS], x_empty[WideGeo<HD>::XS];
  uint64_t y_full[WideGeo<HD>::YSV], y_empty[WideGeo<HD>::YSV];
  uint64_t stat_full[WideGeo<HD>::kStats];  // LSE / D of a unit are in shared memory (X's own barrier may run on: dV frees X before the elementwise warps look)
  uint64_t st_full[2];   // MMA -> elementwise: S and dP of the buffer are in TMEM
  uint64_t pds_full[2];  // elementwise -> MMA: P or dS of the buffer is in TMEM (and dP has been read)
  uint64_t acc_done;     // MMA -> epilogue
  uint64_t acc_free;     // epilogue -> MMA: the accumulator is in registers
  ItemQueue queue;
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) float nlse2[WideGeo<HD>::kStats][kUnit];  // dK, dV: -LSE * log2(e) and -D * scale of the unit's query rows
  alignas(16) float ndls[WideGeo<HD>::kStats][kUnit];
};

template <int HD>
constexpr int wide_smem_bytes() { return WideGeo<HD>::kBarOff + ((int)sizeof(BarW<HD>) + 1023) / 1024 * 1024; }
static_assert(wide_smem_bytes<256>() <= 232448 && wide_smem_bytes<192>() <= 232448, "more than the 227 KiB a CTA can have");

struct ItemW {
  SeqInfo sq;
  int kind, head, hk, bi, row0, u_lo, nu, iters;  // head: dQ only; row0: first resident row (key or query row); iters = 0: nothing visible
  bool live;                                      // false: the sequence has no such rows
};
// Items: all dK, then all dV, then all dQ (with grouped heads the smallest ones come last).  Inside a kind in the order of
// ItemOrder, the heaviest block under a causal mask first.
__device__ __forceinline__ ItemW item_w(const BwdParams& p, int t) {
  ItemW w;
  const int n_kv = p.kv_items.blocks * p.kv_items.pairs;
  w.u_lo = w.nu = w.iters = 0;
  if (t < 2 * n_kv) {
    w.kind = t < n_kv ? kWideDK : kWideDV;
    if (t >= n_kv) t -= n_kv;
    const ItemPlace at = p.kv_items.place(t);
    w.bi = p.by_h_k.div(at.pair);
    w.hk = at.pair - w.bi * p.h_k;
    w.head = 0;
    w.sq = seq_info(p, w.bi);
    w.row0 = at.block * kBlk;
    w.live = w.row0 < w.sq.k_len;
    if (w.live) {  // query rows that see at least one key of the block
      const int k1 = min(w.sq.k_len, w.row0 + kBlk) - 1;
      const int i_lo = w.sq.wr >= 0 ? max(0, w.row0 - w.sq.koff - w.sq.wr) : 0;
      const int i_hi = w.sq.wl >= 0 ? min(w.sq.q_len - 1, k1 - w.sq.koff + w.sq.wl) : w.sq.q_len - 1;
      w.u_lo = i_lo / kUnit;
      w.nu = i_hi >= i_lo ? i_hi / kUnit + 1 - w.u_lo : 0;
      w.iters = w.nu * p.group;
    }
  } else {
    w.kind = kWideDQ;
    t -= 2 * n_kv;
    const ItemPlace at = p.q_items.place(t);
    w.bi = p.by_h.div(at.pair);
    w.head = at.pair - w.bi * p.h;
    w.hk = p.by_group.div(w.head);
    w.sq = seq_info(p, w.bi);
    w.row0 = (p.q_items.blocks - 1 - at.block) * kBlk;
    w.live = w.row0 < w.sq.q_len;
    if (w.live) {  // keys that at least one row of the block sees
      const int r1 = min(w.sq.q_len, w.row0 + kBlk) - 1;
      const int k_hi = w.sq.wr >= 0 ? min(w.sq.k_len - 1, r1 + w.sq.koff + w.sq.wr) : w.sq.k_len - 1;
      const int k_lo = w.sq.wl >= 0 ? max(0, w.row0 + w.sq.koff - w.sq.wl) : 0;
      w.u_lo = k_lo / kUnit;
      w.iters = w.nu = k_hi >= k_lo ? k_hi / kUnit + 1 - w.u_lo : 0;
    }
  }
  return w;
}

// Rows of the streamed sequence counted from a unit's first row: below kUnit in the unit that runs past the sequence.
struct TailRows {
  int first, last;  // of an item's first unit, and of the last unit that it streams of a head
  __device__ __forceinline__ TailRows(const BwdParams& p, const ItemW& w) {
    const int len = w.kind == kWideDQ ? w.sq.k_len : w.sq.q_len;
    // dense input: the rows behind the sequence lie outside the tensor, the TMA unit has filled them with zeros
    first = p.cu_seqlens_q ? len - w.u_lo * kUnit : 0x40000000;
    last = first - (w.nu - 1) * kUnit;
  }
  __device__ __forceinline__ int next(int left) const { return left == last ? first : left - kUnit; }  // (the next head starts over)
};

// Where the item's result goes: first element of resident row 0 (of the item) and the row stride.
template <typename T>
__device__ __forceinline__ T* item_out(const BwdParams& p, const ItemW& w, int64_t& row_stride) {
  if (w.kind == kWideDQ) {
    row_stride = p.dq_row_stride;
    return reinterpret_cast<T*>(p.dq) + (int64_t)w.sq.bq * p.dq_batch_stride + (int64_t)(w.sq.q_row0 + w.row0) * p.dq_row_stride +
           (int64_t)w.head * p.dq_head_stride;
  }
  if (w.kind == kWideDK) {
    row_stride = p.dk_row_stride;
    return reinterpret_cast<T*>(p.dk) + (int64_t)w.sq.bq * p.dk_batch_stride + (int64_t)(w.sq.k_row0 + w.row0) * p.dk_row_stride +
           (int64_t)w.hk * p.dk_head_stride;
  }
  row_stride = p.dv_row_stride;
  return reinterpret_cast<T*>(p.dv) + (int64_t)w.sq.bq * p.dv_batch_stride + (int64_t)(w.sq.k_row0 + w.row0) * p.dv_row_stride +
         (int64_t)w.hk * p.dv_head_stride;
}

struct WideMaps {  // resident operands in boxes of 128 rows, streamed ones in boxes of 64
  CUtensorMap q, dout, k, v, q_u, do_u, k_u, v_u;
};

// Two probabilities (dV items): exp2(s * a - lse2), 0 where masked; with softcap as in ew_pair.
template <typename T, bool MASK, bool SOFTCAP>
__device__ __forceinline__ uint32_t ew_prob_pair(uint32_t s0, uint32_t s1, uint64_t a2, uint64_t cap2, uint64_t nlse2, uint32_t bits, int e) {
  uint64_t x2;
  if (SOFTCAP) {
    float y0, y1, t0, t1;
    unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(s0), __uint_as_float(s1)), a2), y0, y1);
    asm("tanh.approx.f32 %0, %1;\n" : "=f"(t0) : "f"(y0));
    asm("tanh.approx.f32 %0, %1;\n" : "=f"(t1) : "f"(y1));
    x2 = fma_f32x2(pack_f32x2(t0, t1), cap2, nlse2);
  } else {
    x2 = fma_f32x2(pack_f32x2(__uint_as_float(s0), __uint_as_float(s1)), a2, nlse2);
  }
  float x0, x1;
  unpack_f32x2(x2, x0, x1);
  float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
  if (MASK) {
    p0 = ((bits >> e) & 1u) ? p0 : 0.f;
    p1 = ((bits >> (e + 1)) & 1u) ? p1 : 0.f;
  }
  return pack2<T>(p0, p1);
}

template <typename T, uint32_t AB_FMT, bool SOFTCAP, int HD>
__global__ void __launch_bounds__(kThreads, 1)
bwd_wide_kernel(const __grid_constant__ BwdParams p, const __grid_constant__ WideMaps tm, int32_t* status, int32_t* counter) {
  using G = WideGeo<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_addr(smem);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if ((base & 1023u) != 0) {
    if (tid == 0) atomicExch(status, 0x20000000);
    return;
  }
  const int group = p.group;
  const int n_items = 2 * p.kv_items.blocks * p.kv_items.pairs + p.q_items.blocks * p.q_items.pairs;
  BarW<HD>* bar = reinterpret_cast<BarW<HD>*>(smem + G::kBarOff);
  if (tid == 0) {
    mbar_init(smem_addr(&bar->a_full), 1);
    mbar_init(smem_addr(&bar->a_empty), 2);  // the S and the dP issuer
    for (int s = 0; s < G::XS; ++s) {
      mbar_init(smem_addr(&bar->x_full[s]), 1);
      mbar_init(smem_addr(&bar->x_empty[s]), 1);
    }
    for (int s = 0; s < G::YSV; ++s) {
      mbar_init(smem_addr(&bar->y_full[s]), 1);
      mbar_init(smem_addr(&bar->y_empty[s]), 2);  // dK, dQ: the dP issuer, twice; dV: the acc issuer and the dP issuer
    }
    for (int s = 0; s < G::kStats; ++s) mbar_init(smem_addr(&bar->stat_full[s]), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_addr(&bar->st_full[b]), 2);  // S and dP (dV: S, twice)
      mbar_init(smem_addr(&bar->pds_full[b]), kEwWarps / 2);
    }
    mbar_init(smem_addr(&bar->acc_done), 1);
    mbar_init(smem_addr(&bar->acc_free), kEwWarps);
    for (int k = 0; k < kQueue; ++k) mbar_init(smem_addr(&bar->queue.full[k]), 1);
    bar->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_addr(&bar->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, bar->tmem_base, 0);
  volatile int* abort_flag = &bar->abort_flag;
  // Counters that every role keeps alike: wi = items with work so far, gu = units so far (X slot, TMEM buffer and their
  // phases).  The Y slots are used unevenly by the kinds of items: bit i of yph is the phase of Y slot i's next use.
  uint32_t wi = 0, gu = 0, yph = 0;

  if (warp == kTmaWarp) {
    // ------------------------------------------------------------------ producer
    bool ok = true;
    while (ok) {
      const int t = queue_draw(counter, n_items, lane);
      if (t < 0) break;
      const ItemW w = item_w(p, t);
      if (!w.live) continue;
      const SeqInfo& sq = w.sq;
      const bool is_q = w.kind == kWideDQ, is_v = w.kind == kWideDV;
      const int rows_left = (is_q ? sq.q_len : sq.k_len) - w.row0;
      if (w.iters == 0) {  // no visible pair: zeros
        int64_t rs;
        T* o = item_out<T>(p, w, rs);
        const int chunks = p.d >> 3;
        for (int c = lane; c < min(rows_left, kBlk) * chunks; c += 32)
          *reinterpret_cast<uint4*>(o + (int64_t)(c / chunks) * rs + (c % chunks) * 8) = make_uint4(0, 0, 0, 0);
        continue;
      }
      queue_publish(&bar->queue, wi, t, lane);
      if (!mbar_wait(smem_addr(&bar->a_empty), (wi & 1) ^ 1, abort_flag, 60)) break;
      if (!is_v) {  // A1's space may still be Y slots of a dV item
#pragma unroll
        for (int i = G::YS; i < G::YSV; ++i)
          if (!mbar_wait(smem_addr(&bar->y_empty[i]), ((yph >> i) & 1) ^ 1, abort_flag, 61)) ok = false;
        if (!ok) break;
      }
      const int n_y = is_v ? G::YSV : G::YS;
      const int head0 = is_q ? w.head : w.hk, res_row = (is_q ? sq.q_row0 : sq.k_row0) + w.row0;
      const CUtensorMap* m0 = is_q ? &tm.q : &tm.k;
      const CUtensorMap* m1 = is_q ? &tm.dout : &tm.v;
      const CUtensorMap* mx = is_q ? &tm.k_u : &tm.q_u;
      const CUtensorMap* my = is_q ? &tm.v_u : &tm.do_u;
      if (elect_one()) {
        const uint32_t full = smem_addr(&bar->a_full);
        mbar_arrive_expect_tx(full, (is_v ? 1 : 2) * G::kATile);
#pragma unroll
        for (int c = 0; c < G::kChunks; ++c) tma_load_4d(base + c * kHalfBytes, m0, full, 64 * c, head0, res_row, sq.bq);
        if (!is_v) {
#pragma unroll
          for (int c = 0; c < G::kChunks; ++c) tma_load_4d(base + G::kATile + c * kHalfBytes, m1, full, 64 * c, head0, res_row, sq.bq);
        }
      }
      __syncwarp();
      const int s_row0 = is_q ? sq.k_row0 : sq.q_row0;
      int s_head = is_q ? w.hk : w.hk * group, u = 0, ys = 0;
      UnitStats stats;
      if (!is_q) stats.ask(p, sq, s_head, w.u_lo * kUnit, !is_v, lane);
      for (int it = 0; it < w.iters; ++it) {
        const uint32_t g = gu + it;
        const int xs = g % G::XS, row = (w.u_lo + u) * kUnit;
        if (!mbar_wait(smem_addr(&bar->x_empty[xs]), ((g / G::XS) & 1) ^ 1, abort_flag, 62)) { ok = false; break; }
        if (!is_q) {
          stats.put(bar->nlse2[g % G::kStats], bar->ndls[g % G::kStats], p.softmax_scale, lane);
          __syncwarp();
        }
        if (lane == 0) mbar_arrive(smem_addr(&bar->stat_full[g % G::kStats]));
        if (elect_one()) {
          const uint32_t full = smem_addr(&bar->x_full[xs]), dst = base + G::kRingOff + xs * G::kSTile;
          mbar_arrive_expect_tx(full, G::kSTile);
#pragma unroll
          for (int c = 0; c < G::kChunks; ++c) tma_load_4d(dst + c * kUnitHalf, mx, full, 64 * c, s_head, s_row0 + row, sq.bq);
        }
        __syncwarp();
        if (!mbar_wait(smem_addr(&bar->y_empty[ys]), ((yph >> ys) & 1) ^ 1, abort_flag, 63)) { ok = false; break; }
        yph ^= 1u << ys;
        if (elect_one()) {
          const uint32_t full = smem_addr(&bar->y_full[ys]), dst = base + G::y_off(ys);
          mbar_arrive_expect_tx(full, G::kSTile);
#pragma unroll
          for (int c = 0; c < G::kChunks; ++c) tma_load_4d(dst + c * kUnitHalf, my, full, 64 * c, s_head, s_row0 + row, sq.bq);
        }
        __syncwarp();
        if (++ys == n_y) ys = 0;
        if (++u == w.nu) { u = 0; ++s_head; }
        if (!is_q && it + 1 < w.iters) stats.ask(p, sq, s_head, (w.u_lo + u) * kUnit, !is_v, lane);
      }
      ++wi;
      gu += w.iters;
    }
    queue_publish(&bar->queue, wi, -1, lane);  // (after an abort too: the others are leaving through the abort flag anyway)
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------------ MMA issuer 0: S(0) | S(1) acc(0) | S(2) acc(1) | ...
    constexpr uint32_t idesc_s = make_idesc(AB_FMT, kBlk, kUnit, 0), idesc_acc = make_idesc(AB_FMT, kBlk, HD, 1);
    const uint64_t a_desc = make_smem_desc(base, 16, 1024);
    auto unit_off = [](int ks) { return (uint64_t)(((ks >> 2) * kUnitHalf + (ks & 3) * 32) >> 4); };
    bool ok = true;
    while (ok) {
      const int t = queue_get(&bar->queue, wi, abort_flag);
      if (t < 0) break;
      const ItemW w = item_w(p, t);
      const bool is_v = w.kind == kWideDV;
      const int iters = w.iters, n_y = is_v ? G::YSV : G::YS;
      const TailRows tail(p, w);
      int x_left = tail.first, y_left = tail.first;  // rows of the sequence from the next unit of X (dV: of Y) on
      auto issue_s = [&](int u) -> bool {
        const uint32_t g = gu + u;
        const int xs = g % G::XS, b = g & 1;
        if (!mbar_wait(smem_addr(&bar->x_full[xs]), (g / G::XS) & 1, abort_flag, 64)) return false;
        if (x_left < kUnit) clear_tail_rows<G::kChunks, kUnit>(base + G::kRingOff + xs * G::kSTile, x_left, lane);
        x_left = tail.next(x_left);
        tc_fence_after();
        if (elect_one()) {
          const uint64_t b_desc = make_smem_desc(base + G::kRingOff + xs * G::kSTile, 16, 1024);
          const uint32_t d_tmem = tmem + 128 * b;
          mma_ss_c<false>(d_tmem, a_desc, b_desc, idesc_s);
#pragma unroll
          for (int ks = 1; ks < HD / 16; ++ks) mma_ss_c<true>(d_tmem, a_desc + kmaj_off(ks), b_desc + unit_off(ks), idesc_s);
          mma_commit(smem_addr(&bar->st_full[b]));
          if (is_v) {
            mma_commit(smem_addr(&bar->st_full[b]));
            mma_commit(smem_addr(&bar->x_empty[xs]));
          }
          if (u == iters - 1) mma_commit(smem_addr(&bar->a_empty));
        }
        __syncwarp();
        return true;
      };
      if (!mbar_wait(smem_addr(&bar->a_full), wi & 1, abort_flag, 65)) break;
      if (!issue_s(0)) break;
      int ys = 0;
      for (int u = 0; u < iters; ++u) {
        if (u + 1 < iters && !issue_s(u + 1)) { ok = false; break; }
        const uint32_t g = gu + u;
        const int xs = g % G::XS, b = g & 1;
        if (is_v) {
          if (!mbar_wait(smem_addr(&bar->y_full[ys]), (yph >> ys) & 1, abort_flag, 66)) { ok = false; break; }
          if (y_left < kUnit) clear_tail_rows<G::kChunks, kUnit>(base + G::y_off(ys), y_left, lane);
          y_left = tail.next(y_left);
        }
        yph ^= 1u << ys;
        if (!mbar_wait(smem_addr(&bar->pds_full[b]), (g >> 1) & 1, abort_flag, 67)) { ok = false; break; }
        // the epilogue of the previous item must have the accumulator in registers
        if (u == 0 && !mbar_wait(smem_addr(&bar->acc_free), (wi & 1) ^ 1, abort_flag, 68)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint64_t z_desc = make_smem_desc(base + (is_v ? G::y_off(ys) : G::kRingOff + xs * G::kSTile), kUnitHalf, 1024);
          const uint32_t src = tmem + 128 * b;
          // k-step ks = streamed rows 16 ks .. 16 ks + 15: the 8 packed columns their thread wrote inside its own 32
          if (u == 0) mma_ts_c<false>(tmem + 256, src, z_desc, idesc_acc);
          else mma_ts_c<true>(tmem + 256, src, z_desc, idesc_acc);
#pragma unroll
          for (int ks = 1; ks < 4; ++ks) mma_ts_c<true>(tmem + 256, src + 32 * (ks >> 1) + 8 * (ks & 1), z_desc + nmaj_off(ks), idesc_acc);
          mma_commit(is_v ? smem_addr(&bar->y_empty[ys]) : smem_addr(&bar->x_empty[xs]));
          if (u == iters - 1) mma_commit(smem_addr(&bar->acc_done));
        }
        __syncwarp();
        if (++ys == n_y) ys = 0;
      }
      ++wi;
      gu += iters;
    }
  } else if (warp == kMmaWarp + 1) {
    // ------------------------------------------------------------------ MMA issuer 1: dP (dK and dQ items)
    constexpr uint32_t idesc_s = make_idesc(AB_FMT, kBlk, kUnit, 0);
    const uint64_t a_desc = make_smem_desc(base + G::kATile, 16, 1024);
    auto unit_off = [](int ks) { return (uint64_t)(((ks >> 2) * kUnitHalf + (ks & 3) * 32) >> 4); };
    bool ok = true;
    while (ok) {
      const int t = queue_get(&bar->queue, wi, abort_flag);
      if (t < 0) break;
      const ItemW w = item_w(p, t);
      int ys = 0;
      if (!mbar_wait(smem_addr(&bar->a_full), wi & 1, abort_flag, 69)) break;
      if (w.kind == kWideDV) {  // nothing to issue: only keeps in step with the barriers
        if (lane == 0) mbar_arrive(smem_addr(&bar->a_empty));
        for (int u = 0; u < w.iters; ++u) {
          if (!mbar_wait(smem_addr(&bar->y_full[ys]), (yph >> ys) & 1, abort_flag, 58)) { ok = false; break; }
          yph ^= 1u << ys;
          if (lane == 0) mbar_arrive(smem_addr(&bar->y_empty[ys]));
          if (++ys == G::YSV) ys = 0;
        }
      } else {
        const TailRows tail(p, w);
        int y_left = tail.first;
        for (int u = 0; u < w.iters; ++u) {
          const uint32_t g = gu + u;
          const int b = g & 1;
          if (!mbar_wait(smem_addr(&bar->y_full[ys]), (yph >> ys) & 1, abort_flag, 70)) { ok = false; break; }
          yph ^= 1u << ys;
          if (y_left < kUnit) clear_tail_rows<G::kChunks, kUnit>(base + G::y_off(ys), y_left, lane);
          y_left = tail.next(y_left);
          // dP of the unit before in this buffer must have been read
          if (g >= 2 && !mbar_wait(smem_addr(&bar->pds_full[b]), ((g - 2) >> 1) & 1, abort_flag, 71)) { ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
            const uint64_t b_desc = make_smem_desc(base + G::y_off(ys), 16, 1024);
            const uint32_t d_tmem = tmem + 128 * b + 64;
            mma_ss_c<false>(d_tmem, a_desc, b_desc, idesc_s);
#pragma unroll
            for (int ks = 1; ks < HD / 16; ++ks) mma_ss_c<true>(d_tmem, a_desc + kmaj_off(ks), b_desc + unit_off(ks), idesc_s);
            mma_commit(smem_addr(&bar->st_full[b]));
            mma_commit(smem_addr(&bar->y_empty[ys]));
            mma_commit(smem_addr(&bar->y_empty[ys]));
            if (u == w.iters - 1) mma_commit(smem_addr(&bar->a_empty));
          }
          __syncwarp();
          if (++ys == G::YS) ys = 0;
        }
      }
      ++wi;
      gu += w.iters;
    }
  } else if (warp < kEwWarps) {
    // ------------------------------------------------------------------ elementwise: lane = resident row, 32 of the unit's 64 columns
    const int r = (warp & 3) * 32 + lane, q2 = (warp >> 2) & 1, grp = warp >> 3, q4 = warp >> 2;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const float a1 = SOFTCAP ? p.softmax_scale / p.softcap : p.scale_log2, cap1 = p.softcap * kLog2e;
    const uint64_t sl2 = pack_f32x2(a1, a1), cap2 = pack_f32x2(cap1, cap1), sc2 = pack_f32x2(p.softmax_scale, p.softmax_scale);
    const uint32_t st_tmem = tmem + lane_addr + 128 * grp + 32 * q2;  // this thread's 32 columns of S; dP 64 columns on
    // one unit: kind and mask are compile-time here, the branches are outside
    auto unit = [&](auto kind_tag, auto mask_tag, int st, uint64_t nl_row, uint64_t nd_row, uint32_t bits) {
      constexpr int KIND = decltype(kind_tag)::value;
      constexpr bool MASK = decltype(mask_tag)::value;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t sv[16], dv[16], pk[8], unused;
        tmem_ld16(st_tmem + 16 * hf, sv);
        if (KIND != kWideDV) tmem_ld16(st_tmem + 64 + 16 * hf, dv);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
          uint64_t nl = nl_row, nd = nd_row;
          if (KIND != kWideDQ) {  // per column
            const float2 l2 = *reinterpret_cast<const float2*>(&bar->nlse2[st][32 * q2 + 16 * hf + e]);
            nl = pack_f32x2(l2.x, l2.y);
          }
          if (KIND == kWideDK) {
            const float2 d2 = *reinterpret_cast<const float2*>(&bar->ndls[st][32 * q2 + 16 * hf + e]);
            nd = pack_f32x2(d2.x, d2.y);
          }
          if (KIND == kWideDV)
            pk[e >> 1] = ew_prob_pair<T, MASK, SOFTCAP>(sv[e], sv[e + 1], sl2, cap2, nl, bits, 16 * hf + e);
          else
            ew_pair<T, MASK, SOFTCAP>(false, sv[e], sv[e + 1], dv[e], dv[e + 1], sl2, cap2, nl, sc2, nd, bits, 16 * hf + e, unused, pk[e >> 1]);
        }
        // into the columns this thread has already read (the first 16 of its 32): nobody else's data
        tmem_st8(st_tmem + 8 * hf, pk);
      }
    };
    bool ok = true;
    while (ok) {
      const int t = queue_get(&bar->queue, wi, abort_flag);
      if (t < 0) break;
      const ItemW w = item_w(p, t);
      const SeqInfo& sq = w.sq;
      const bool is_q = w.kind == kWideDQ;
      const int j = w.row0 + r;  // this thread's row: a query row or a key
      int64_t rs;
      T* out = item_out<T>(p, w, rs) + (int64_t)r * rs + 64 * q4;
      const bool row_ok = j < (is_q ? sq.q_len : sq.k_len);
      // streamed rows that pair with this row: keys a query row sees, or query rows that see a key
      int lo, hi;
      float nl1 = -INFINITY, nd1 = 0.f;
      if (is_q) {
        hi = sq.wr >= 0 ? min(sq.k_len - 1, j + sq.koff + sq.wr) : sq.k_len - 1;
        lo = sq.wl >= 0 ? j + sq.koff - sq.wl : 0;
        if (row_ok) {
          const int64_t li = (int64_t)sq.bq * p.lse_batch_stride + (int64_t)w.head * p.lse_head_stride + sq.q_row0 + j;
          nl1 = -p.lse[li] * kLog2e;
          nd1 = -p.delta[li] * p.softmax_scale;
        }
      } else {
        lo = sq.wr >= 0 ? j - sq.koff - sq.wr : -0x40000000;
        hi = row_ok ? (sq.wl >= 0 ? j - sq.koff + sq.wl : 0x40000000) : -0x40000001;
      }
      const uint64_t nl_row = pack_f32x2(nl1, nl1), nd_row = pack_f32x2(nd1, nd1);
      int um = (int)((grp - gu) & 1u);  // u modulo w.nu: the unit of its head
      for (int u = um; u < w.iters; u += 2, um += 2) {  // the units whose running number has this group's parity
        while (um >= w.nu) um -= w.nu;
        const uint32_t g = gu + u;
        const int st = g % G::kStats, c0 = (w.u_lo + um) * kUnit;
        if (!is_q && !mbar_wait(smem_addr(&bar->stat_full[st]), (g / G::kStats) & 1, abort_flag, 72)) { ok = false; break; }
        if (!mbar_wait(smem_addr(&bar->st_full[grp]), (g >> 1) & 1, abort_flag, 73)) { ok = false; break; }
        tc_fence_after();
        // does any (row of the block, column of the unit) pair fall outside the mask?  (the same answer in every thread)
        bool need_mask;
        if (is_q) {
          need_mask = c0 + kUnit > sq.k_len;
          if (sq.wr >= 0) need_mask = need_mask || (c0 + kUnit - 1 > w.row0 + sq.koff + sq.wr);
          if (sq.wl >= 0) need_mask = need_mask || (c0 < min(sq.q_len, w.row0 + kBlk) - 1 + sq.koff - sq.wl);
        } else {  // rows beyond the sequence need no mask: their -LSE is -inf
          need_mask = w.row0 + kBlk > sq.k_len;
          if (sq.wr >= 0) need_mask = need_mask || (w.row0 + kBlk - 1 > c0 + sq.koff + sq.wr);
          if (sq.wl >= 0) need_mask = need_mask || (w.row0 < min(sq.q_len, c0 + kUnit) - 1 + sq.koff - sq.wl);
        }
        const uint32_t bits = need_mask ? range_bits(c0 + 32 * q2, lo, hi) : 0xffffffffu;
        auto by_mask = [&](auto kind_tag) {
          if (need_mask) unit(kind_tag, std::true_type{}, st, nl_row, nd_row, bits);
          else unit(kind_tag, std::false_type{}, st, nl_row, nd_row, bits);
        };
        if (w.kind == kWideDK) by_mask(std::integral_constant<int, kWideDK>{});
        else if (w.kind == kWideDV) by_mask(std::integral_constant<int, kWideDV>{});
        else by_mask(std::integral_constant<int, kWideDQ>{});
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_lane0(smem_addr(&bar->pds_full[grp]), lane);
      }
      if (!ok) break;
      // ---- epilogue: 64 columns of this row; the accumulator is handed back once it is in registers
      if (!mbar_wait(smem_addr(&bar->acc_done), wi & 1, abort_flag, 74)) break;
      tc_fence_after();
      if (64 * q4 < HD) {
        uint32_t a0[32], a1r[32];
        tmem_ld32(tmem + lane_addr + 256 + 64 * q4, a0);
        tmem_ld32(tmem + lane_addr + 256 + 64 * q4 + 32, a1r);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_lane0(smem_addr(&bar->acc_free), lane);
        if (row_ok) {
          const bool sectors = w.kind == kWideDQ ? p.dq_sectors : w.kind == kWideDK ? p.dk_sectors : p.dv_sectors;
          store_slice<T>(out, a0, p.d - 64 * q4, sectors);
          store_slice<T>(out + 32, a1r, p.d - 64 * q4 - 32, sectors);
        }
      } else if (lane == 0) {
        mbar_arrive(smem_addr(&bar->acc_free));
      }
      ++wi;
      gu += w.iters;
    }
  }

  tc_fence_before();
  __syncthreads();
  finish(status, bar->abort_flag, tid);
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace btc5
}  // namespace fa
