// Prefill attention-forward kernel for sm_100a: tcgen05 MMA with accumulators in TMEM, K/V tiles
// streamed by TMA through a shared-memory ring, online softmax in registers (one thread per
// query row), persistent CTAs.
//
// It replaces, for prefill (dense, packed varlen, or many query tokens against a KV cache, paged or
// not), the cube+vector pipeline of the reference kernel
// (csrc/arch22/flash_attn_npu_v2/mha_fwd_kvcache.cpp:632-965: QK -> online softmax -> PV ->
// rescale O, with S / P / O_tmp round-tripping through a global workspace).  Here S, P and O never
// leave the SM: S and O live in TMEM, P goes through shared memory (16-bit, the layout of an MMA
// A operand) into the second MMA.
//
// CTA = 16 warps:  warps 0-3    softmax of query sub-tile 0 (128 rows, one thread per row)
//                  warps 4-7    softmax of query sub-tile 1 (256-column tiles: the same rows as warps 0-3, keys 64-127)
//                  warps 8-11   correction (rescale of O in TMEM when a row maximum moved) and
//                               epilogue (O / l -> global) for both sub-tiles
//                  warps 12-13  MMA issuers, one per sub-tile (one elected lane each)
//                  warp  14     TMA producer (one elected lane)
//                  warp  15     clears the V rows past the end of a sequence (KV caches, packed input)
// TMEM (512 columns): S0 [0,128)  S1 [128,256)  O0 [256,384)  O1 [384,512).
// Shared memory: Q0 Q1 | P0 P1 | ring of K / V tiles (32 KiB each).
// Dependency chain per sub-tile: a softmax thread copies its row of S into registers and frees the
// S columns at once, so Q.K^T of the next KV block runs while this block's exponentials are
// computed; P.V follows when P is in shared memory.  The softmax warps therefore never wait for the
// tensor pipe in steady state, and the tensor pipe has two sub-tiles' worth of independent work.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "tc5_ptx.cuh"
#include "tile_order.cuh"

namespace fa {
namespace tc5 {

constexpr int kBlockM = 128;          // rows of one query sub-tile
constexpr int kTileM = 2 * kBlockM;   // rows of one CTA tile
constexpr int kBlockN = 128;          // keys per KV block
constexpr int kSlots = 3, kMaxSlots = 4;  // ring of 32 KiB K / V buffers (64 columns: four of 16 KiB)
constexpr int kXchgCol = 128;  // TMEM columns of the exchange between warpgroups that share rows (S1's)
constexpr int kThreads = 512;
constexpr int kMmaWarp = 12 /* and 13: one per sub-tile */, kTmaWarp = 14;
// Registers per thread after the roles have re-balanced them (setmaxnreg, one value per warpgroup).
// A CTA can only re-distribute the registers it was launched with (512 threads x 128), never more:
// a setmaxnreg.inc that the other warpgroups' releases cannot cover would block for ever.
#ifndef FA_TC5_REGS_SOFTMAX
#define FA_TC5_REGS_SOFTMAX 192
#define FA_TC5_REGS_CORR 88
#define FA_TC5_REGS_MMA 40
#endif
constexpr int kRegsSoftmax = FA_TC5_REGS_SOFTMAX, kRegsCorr = FA_TC5_REGS_CORR, kRegsMma = FA_TC5_REGS_MMA;
static_assert(256 * kRegsSoftmax + 128 * (kRegsCorr + kRegsMma) <= kThreads * 128, "more registers than the CTA was launched with");
constexpr int kHalfBytes = kBlockN * 128;   // one 64-column half of a [128 x 128] 16-bit tile (128-byte rows)
constexpr int kTileBytes = 2 * kHalfBytes;  // 32 KiB
constexpr int kBarBytes = 3072;  // barriers, per-row rescale factors and 1 / l
// Q0 Q1 | P0 P1 | ring | barriers.  The dynamic shared memory base must be 1024-byte aligned (the
// kernel checks it): there is no room left for a round-up.
constexpr int kSmemBytes = 4 * kTileBytes + kSlots * kTileBytes + kBarBytes;
static_assert(kSmemBytes <= 232448, "more than the 227 KiB a CTA can have");

// Geometry by tile width HD (64, 128 or 256 columns; the head dim is at most HD).  Up to 128 a CTA tile is two
// 128-row sub-tiles and a K / V tile fills one ring slot, 32 KiB or, for 64 columns, 16.  What that leaves with 64 columns holds a
// second P buffer for each sub-tile: S of a block is complete only when P.V of two blocks before is (one warp issues both, in this
// order), so the softmax warps need not wait for a P buffer at all.  4 K, b 4, 32 heads, head dim 64: causal 444 -> 435 us, full
// 799 -> 750; b 2, s 2999, 16 / 4 heads, causal 80.3 -> 73.6.  For 256 the 256 fp32
// columns of O leave TMEM room for one sub-tile only: the CTA tile is 128 rows (shared by the two softmax warpgroups), Q takes both Q slots (64 KiB), the
// second P slot joins the ring, and the ring is two slots of 64 KiB.
template <int HD>
struct Geo {
  static_assert(HD == 64 || HD == 128 || HD == 256, "tile widths");
  static constexpr int kHalves = HD / 64;                                      // 64-column halves of a Q / K / V tile
  static constexpr bool kWide = HD > 128;
  static constexpr int kRows = kWide ? kBlockM : kTileM;                       // query rows of a CTA tile
  static constexpr int kQStep = HD == 64 ? kHalfBytes : kTileBytes;             // bytes from Q0 to Q1
  static constexpr int kPBufs = HD == 64 ? 2 : 1;                              // P buffers of a sub-tile
  static constexpr int kPOff = 2 * kQStep;
  static constexpr int kSlotBytes = kWide ? 2 * kTileBytes : HD == 64 ? kHalfBytes : kTileBytes;
  static constexpr int kRing = kWide ? 2 : HD == 64 ? 4 : kSlots;
  static constexpr int kRingOff = kPOff + (kWide ? 1 : 2 * kPBufs) * kTileBytes;  // Q0 Q1 | P0 [P0'] [P1 [P1']] | ring
  static_assert(kRingOff + kRing * kSlotBytes + kBarBytes <= kSmemBytes, "shared memory layout");
};

// Input of a kernel instance: dense, or ragged (a KV cache or packed sequences: tiles and tails differ by batch entry),
// whose tiles are dealt out in a fixed order or drawn at run time.
enum InputKind { kDense = 0, kRaggedFixed = 1, kRaggedDraw = 2 };
// Softcap of a kernel instance: none, by tanh.approx, or by the finer form (packed queries against a cache; softmax role).
enum CapKind { kCapNone = 0, kCapApprox = 1, kCapFine = 2 };

struct Tc5Params {
  fa_fwd_params a;
  int32_t is_causal, is_local, wl, wr;
  int32_t group;    // h / h_k
  int32_t m_tiles;  // ceil(max seqlen_q / 256)
  int32_t total_tiles;
  FastDiv by_h, by_group, by_m_tiles;             // h, group, m_tiles
  FastDiv by_chunk, by_pairs, by_last_pairs;      // tiles of an L2 chunk, its pairs, the pairs of the last chunk (static_tile)
  float scale_log2;
  float softcap_mul, softcap_l2;  // softcap: scores become softcap_l2 * tanh(s * softcap_mul) in the log2 domain (scale / softcap, softcap * log2 e)
  int32_t o_sectors;         // rows of O start on 32-byte boundaries and are whole 32-byte sectors long
  int32_t chunk_bh;          // (batch, head) pairs per L2 chunk of the tile order (static_tile)
  int32_t chunk_heads;       // ragged input: query heads per L2 chunk (TileDraw)
  // 1: the rows behind the last key of a sequence hold foreign data (the unused tail of a KV cache or of a page,
  // the next sequence of a packed tensor) and must be cleared in V before P.V: P is 0 there, but 0 x NaN is NaN.
  // 0: dense input, those rows lie outside the tensor and the TMA unit already returns zeros for them.
  int32_t fix_tail;
  int32_t* status;  // device word: 0 ok, otherwise the wait that gave up
};


struct TileInfo {
  int bi, hh, hk, q_row0, q_len, k_row0, k_len, koff;
  int bk;  // batch row of K / V (cache_batch_idx for a contiguous cache)
  int row0[2];  // first row (within the sequence) of each sub-tile
  int jlo[2], jhi[2];
  bool has[2];
  int ulo, uhi;  // union of the block ranges
};

// Tile order of dense input (and of ragged input whose tiles are dealt out): the (batch, head) pairs are cut into chunks whose K / V fit in L2 together; inside a
// chunk all pairs run their last (heaviest, causal) query tile first, then the one before, and so
// on, so the K / V prefixes a chunk re-reads tile after tile come from L2 and not from HBM.  The
// chunk length makes a chunk a whole even number of rounds of the grid (StaticWalk), which keeps the
// per-CTA sums as even as one chunk over everything would.
struct TileId {
  int bi, hh, mt;  // batch entry, query head, query tile
};
__device__ __forceinline__ TileId static_tile(const Tc5Params& p, int n) {
  const int per_m = p.a.b * p.a.h;
  const int per_chunk = p.chunk_bh * p.m_tiles;
  const int ck = p.by_chunk.div(n), r = n - ck * per_chunk;
  const int cnt = min(p.chunk_bh, per_m - ck * p.chunk_bh);  // pairs in this chunk (the last one may be short)
  const int level = cnt == p.chunk_bh ? p.by_pairs.div(r) : p.by_last_pairs.div(r);
  const int rem = ck * p.chunk_bh + r - level * cnt, bi = p.by_h.div(rem);
  return {bi, rem - bi * p.a.h, p.m_tiles - 1 - level};  // heavy (late, causal) tiles first
}

__device__ __forceinline__ int q_length(const Tc5Params& p, int bi) {
  return p.a.cu_seqlens_q ? p.a.cu_seqlens_q[bi + 1] - p.a.cu_seqlens_q[bi] : p.a.seqlen_q;
}
__device__ __forceinline__ int k_length(const Tc5Params& p, int bi) {
  // KV cache (contiguous or paged): keys in use per batch entry, plus the tokens the prologue appended; clamped here,
  // the producer reports it
  if (p.a.seqused_k) return cache_len(p.a, bi, nullptr) + p.a.seqlen_new;
  return p.a.cu_seqlens_k ? p.a.cu_seqlens_k[bi + 1] - p.a.cu_seqlens_k[bi] : p.a.seqlen_k;
}

// The key blocks [jlo, jhi) that the rows of a sub-tile see, which starts at row row0 (of the sequence); none: jlo = jhi.
__device__ __forceinline__ void block_range(const Tc5Params& p, int row0, int q_len, int k_len, int& jlo, int& jhi) {
  jlo = jhi = 0;
  if (row0 >= q_len) return;
  const int koff = k_len - q_len, i_max = min(q_len, row0 + kBlockM) - 1;
  int j_lo = 0, j_hi = k_len;
  if (p.is_causal) j_hi = min(k_len, i_max + koff + 1);
  if (p.is_local) {
    j_hi = min(k_len, i_max + koff + p.wr + 1);
    j_lo = max(0, row0 + koff - p.wl);
  }
  if (j_hi > j_lo) {
    jlo = j_lo / kBlockN;
    jhi = ceil_div(j_hi, kBlockN);
  }
}

// What a softmax warp needs of a tile: its own sub-tile.
struct SubTile {
  int bi, hh, q_row0, q_len, k_len, koff;
  int row0, jlo, jhi;
};
template <int ROWS>
__device__ __forceinline__ SubTile sub_tile(const Tc5Params& p, const TileId id, int t) {
  SubTile s;
  s.bi = id.bi;
  s.hh = id.hh;
  s.q_row0 = p.a.cu_seqlens_q ? p.a.cu_seqlens_q[id.bi] : 0;
  s.q_len = q_length(p, id.bi);
  s.k_len = k_length(p, id.bi);
  s.koff = s.k_len - s.q_len;
  s.row0 = id.mt * ROWS + t * kBlockM;
  block_range(p, s.row0, s.q_len, s.k_len, s.jlo, s.jhi);
  return s;
}

template <int ROWS>  // query rows of a CTA tile: 256 (two sub-tiles) or 128 (sub-tile 0 only)
__device__ __forceinline__ void tile_info(const Tc5Params& p, const TileId id, TileInfo& ti) {
  const int mt = id.mt;
  ti.bi = id.bi;
  ti.hh = id.hh;
  ti.hk = p.by_group.div(ti.hh);
  ti.q_row0 = p.a.cu_seqlens_q ? p.a.cu_seqlens_q[ti.bi] : 0;
  ti.q_len = q_length(p, ti.bi);
  ti.k_row0 = p.a.cu_seqlens_k ? p.a.cu_seqlens_k[ti.bi] : 0;
  ti.k_len = k_length(p, ti.bi);
  ti.bk = (p.a.cache_batch_idx && !p.a.block_table) ? p.a.cache_batch_idx[ti.bi] : ti.bi;
  ti.koff = ti.k_len - ti.q_len;
  ti.ulo = 0x7fffffff;
  ti.uhi = 0;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int r0 = (ROWS == kBlockM && t == 1) ? 0x3fffffff : mt * ROWS + t * kBlockM;  // no second sub-tile in 128-row tiles
    ti.row0[t] = r0;
    block_range(p, r0, ti.q_len, ti.k_len, ti.jlo[t], ti.jhi[t]);
    ti.has[t] = ti.jhi[t] > ti.jlo[t];
    if (ti.has[t]) {
      ti.ulo = min(ti.ulo, ti.jlo[t]);
      ti.uhi = max(ti.uhi, ti.jhi[t]);
    }
  }
  if (ti.uhi == 0) ti.ulo = 0;
}

// Ragged input whose tiles are drawn (TileDraw): the tiles a CTA has drawn, handed by the producer warp to the other roles.
constexpr int kQueue = 4;
constexpr int kQueueReaders = 15;  // warps that read every tile
struct TileQueue {
  alignas(16) uint32_t response[4];  // of the request for another CTA's tile
  uint64_t answered;                 // the response has arrived
  uint64_t full[kQueue], empty[kQueue];
  int32_t tile[kQueue];              // (batch entry * heads + head) * m_tiles + query tile; total_tiles: no more
};

struct Barriers {
  uint64_t q_full[2], q_empty[2], kv_full[kMaxSlots], kv_empty[kMaxSlots];
  uint64_t s_full[2];      // MMA -> softmax: S_t = Q_t K_j^T is in TMEM
  uint64_t s_free[2];      // softmax -> MMA: every row of S_t has been copied into registers
  // softmax -> MMA: half h (64 keys) of P_t is in shared memory.  One barrier per half: a waiter must
  // never fall two phases behind a barrier, which two arrivals per block on one barrier would allow.
  uint64_t p_full[2][2][2];  // [sub-tile][P buffer][half]
  // softmax -> correction: what the sub-tile's next event hands over is in corr (rescale factors of a block, or 1 / l at the end
  // of a tile).  Events alternate between two barriers and two rows of corr, so that the softmax warps never wait for a row:
  // event c - 2 has been read by then.  Before event c of block n (or behind the last block n) a softmax warp has seen P.V of block
  // n - 2 (n - 1) complete, which was issued after every correction warp had read its factors, or, for the first block of a
  // tile, the 1 / l of the tile before.  With two P buffers it sees the former in S of block n (Geo) and waits for the latter just
  // for this.  It does not look at every phase of o_done then, so each P buffer has its own: when it waits for block n - 1 there,
  // the phase before, block n - 3's, is over (the correction warps waited for it before they let P.V of block n - 2 be issued),
  // and the phase behind, block n + 1's, cannot end before the warp has delivered its P.  (The wait lies behind that warp's last
  // arrival for block n; with one barrier for both buffers it had to lie in front of it: b 4, s 4096, 32 heads, head dim 64, full
  // 763 -> 728 us, causal 445 -> 423.)
  uint64_t corr_ready[2][2];
  uint64_t o_ready[2];     // correction -> MMA: O_t has been rescaled, P.V of block j may accumulate
  uint64_t o_done[2][2];   // MMA -> correction, softmax: P.V of a block has completed (O_t updated, P_t read); [sub-tile][P buffer]
  uint64_t o_free[2];      // correction -> MMA: the epilogue has read O_t
  uint64_t fix_req;        // MMA (both warps) -> warp 15: the last V tile of the CTA tile has landed and needs its tail cleared
  uint64_t v_fixed;        // warp 15 -> MMA (both warps): done
  uint64_t exchanged;      // 256-column tiles: both softmax warpgroups have left their value in TMEM
  uint32_t tmem_base;
  int abort_flag;
  uint32_t fix_seen[2];    // tail repairs each issuing warp has been through (phase of fix_req / v_fixed)
  uint32_t fix_slot;       // ring slot of the V tile to repair
  float corr[2][2][kBlockM];  // [sub-tile][event & 1]
  TileQueue queue;
};
static_assert(sizeof(Barriers) <= kBarBytes, "barrier block does not fit");

// Static tile schedule of dense input and of ragged input with few tiles: CTA c of G takes positions c, 2G-1-c, 2G+c, 4G-1-c, ... (serpentine) of an order
// that starts with the heaviest tiles, which evens out the per-CTA sums of a decreasing sequence (causal, 4K: 1 % spread
// instead of 6 % with a plain stride).
struct StaticWalk {
  int round = 0;
  __device__ explicit StaticWalk(Barriers*) {}
  __device__ __forceinline__ int first(const Tc5Params& p) const {
    const int g = (int)gridDim.x, c = (int)blockIdx.x;
    if (round * g >= p.total_tiles) return p.total_tiles;
    const int n = round * g + ((round & 1) ? g - 1 - c : c);
    return n < p.total_tiles ? n : p.total_tiles;
  }
  __device__ __forceinline__ int next(const Tc5Params& p) {
    ++round;
    return first(p);
  }
};

// Ragged input: tile counts and lengths are on the device, and a fixed deal leaves the CTAs uneven (12 packed sequences
// of 37 - 2999 rows, 16 heads: the longest CTA has 1.7 x the mean).  The grid has a CTA per tile instead, and a running
// CTA takes over the tile of one that has not started (clusterlaunchcontrol) until none is left: no counter in memory,
// nothing to reset.  The producer warp draws and publishes the tile; the other roles read it here.  Kernel time, those
// sequences (head dim 64) 332 -> 236 us; 4 chunks of 301 - 2048 rows against 1777 - 8192 cached keys 570 -> 508 us a call.
// With no more tiles than SMs there is nothing to even out and the draw costs 2 - 5 us a call (its loads of the lengths,
// the hand-over, the last request): such launches keep the fixed deal.  300 + 200 packed rows, 32 heads: 18.5 us dealt,
// 22.5 us drawn; two chunks of 256 rows against 4096 keys 79 and 84 us.
struct QueueWalk {
  Barriers* bar;
  uint32_t k = 0;
  __device__ explicit QueueWalk(Barriers* b) : bar(b) {}
  __device__ __forceinline__ int next(const Tc5Params& p) {
    TileQueue& q = bar->queue;
    const uint32_t s = k % kQueue;
    if (!mbar_wait(smem_addr(&q.full[s]), (k / kQueue) & 1, &bar->abort_flag, 61)) return p.total_tiles;
    const int n = q.tile[s];
    ++k;
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(smem_addr(&q.empty[s]));
    return n;
  }
  __device__ __forceinline__ int first(const Tc5Params& p) { return next(p); }
};
template <int IN>
using TileWalk = typename std::conditional<IN == kRaggedDraw, QueueWalk, StaticWalk>::type;
// The tile number that a walk gives -> tile (p.total_tiles: no more).
template <int IN>
__device__ __forceinline__ TileId tile_id(const Tc5Params& p, int n) {
  if (IN != kRaggedDraw) return static_tile(p, n);
  const int pair = p.by_m_tiles.div(n), bi = p.by_h.div(pair);
  return {bi, pair - bi * p.a.h, n - pair * p.m_tiles};
}

// The producer's side.  Position n (a CTA index) -> tile: the heads are cut into chunks whose K / V stay in L2 together;
// a chunk runs its tiles by level (tile_order.cuh), level = query tile + (causal) the tiles' worth of keys in front of the
// queries, i.e. about the work of the tile.  The grid's surplus positions have no tile.
template <int ROWS>
struct TileLevels {
  const Tc5Params& p;
  int lane;
  int live = 0, top = 0;  // tiles of one head; highest level

  __device__ __forceinline__ void entry(int bi, int& lo, int& n) const {  // levels [lo, lo + n) of batch entry bi
    const int q_len = q_length(p, bi);
    n = min(max(0, ceil_div(q_len, ROWS)), p.m_tiles);
    lo = (p.is_causal || p.is_local) ? max(0, k_length(p, bi) - q_len) / ROWS : 0;
  }
  __device__ TileLevels(const Tc5Params& p_, int lane_) : p(p_), lane(lane_) {
    for (int bi = lane; bi < p.a.b; bi += 32) {
      int lo, n;
      entry(bi, lo, n);
      live += n;
      if (n > 0) top = max(top, lo + n - 1);
    }
    live = __reduce_add_sync(0xffffffffu, live);
    top = __reduce_max_sync(0xffffffffu, top);
  }
  __device__ __forceinline__ uint32_t members(int level, int b0) const {  // batch entries b0 .. b0 + 31 with a tile in the level
    int lo = 0, n = 0;
    if (b0 + lane < p.a.b) entry(b0 + lane, lo, n);
    return __ballot_sync(0xffffffffu, level >= lo && level < lo + n);
  }
  __device__ __forceinline__ int count(int level) const {
    int c = 0;
    for (int b0 = 0; b0 < p.a.b; b0 += 32) c += __popc(members(level, b0));
    return c;
  }
};

template <int ROWS>
struct TileDraw {
  const Tc5Params& p;
  Barriers* bar;
  int lane, pos;
  uint32_t k = 0, asked = 0;
  bool pending = false, more = true;
  TileLevels<ROWS> levels;
  TileCursor cursor;

  __device__ TileDraw(const Tc5Params& p_, Barriers* b, int lane_) : p(p_), bar(b), lane(lane_), pos(blockIdx.x), levels(p_, lane_) {}
  // position -> tile.  False: the position has no tile.
  __device__ __forceinline__ bool locate(int n, int& tile) {
    int hh, r;
    if (!tile_locate(cursor, levels, p.a.h, p.chunk_heads, n, hh, r)) return false;
    int bi = 0;
    for (int b0 = 0; b0 < p.a.b; b0 += 32) {
      uint32_t m = levels.members(cursor.level, b0);
      const int c = __popc(m);
      if (r < c) {
        for (; r > 0; --r) m &= m - 1;  // drop the r lowest members
        bi = b0 + __ffs(m) - 1;
        break;
      }
      r -= c;
    }
    int lo, nt;
    levels.entry(bi, lo, nt);
    tile = (bi * p.a.h + hh) * p.m_tiles + cursor.level - lo;
    return true;
  }
  __device__ __forceinline__ void ask() {
    if (lane == 0) {
      const uint32_t full = smem_addr(&bar->queue.answered);
      fence_proxy_async();  // the last response has been read
      mbar_arrive_expect_tx(full, 16);
      try_cancel(smem_addr(bar->queue.response), full);
    }
    __syncwarp();
    pending = true;
  }
  __device__ __forceinline__ bool answer() {  // -> pos, more
    pending = false;
    if (!mbar_wait(smem_addr(&bar->queue.answered), asked & 1, &bar->abort_flag, 62)) return false;
    ++asked;
    more = canceled_cta(smem_addr(bar->queue.response), pos);
    __syncwarp();
    return true;
  }
  __device__ __forceinline__ bool publish(int tile) {
    TileQueue& q = bar->queue;
    const uint32_t s = k % kQueue;
    if (!mbar_wait(smem_addr(&q.empty[s]), ((k / kQueue) & 1) ^ 1, &bar->abort_flag, 63)) return false;
    ++k;
    if (lane == 0) {
      q.tile[s] = tile;
      mbar_arrive(smem_addr(&q.full[s]));
    }
    __syncwarp();
    return true;
  }
  // The CTA's next tile, published to the other roles.  A request is always answered and read before the next one, and
  // none is made after one that found nothing.
  __device__ __forceinline__ int next(const Tc5Params&) {
    prefetch();
    if (!answer()) return p.total_tiles;
    return first(p);
  }
  __device__ __forceinline__ int first(const Tc5Params&) {
    int tile = p.total_tiles;
    while (more && !locate(pos, tile)) {
      ask();
      if (!answer()) return p.total_tiles;
    }
    if (!more) tile = p.total_tiles;
    return publish(tile) ? tile : p.total_tiles;
  }
  // Called when the tile's loads are nearly through: a CTA must not commit itself to a tile a whole tile ahead.
  __device__ __forceinline__ void prefetch() {
    if (!pending) ask();
  }
};
struct StaticDraw : StaticWalk {
  __device__ StaticDraw(const Tc5Params&, Barriers* b, int) : StaticWalk(b) {}
  __device__ __forceinline__ void prefetch() {}
};

}  // namespace tc5
}  // namespace fa
