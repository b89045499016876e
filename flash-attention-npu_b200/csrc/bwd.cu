// Attention backward: C-ABI entry point and launch (kernels in bwd_kernel.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "bwd_kernel.cuh"
#include "tc5_api.cuh"

namespace fa {

int fail_bwd(int code, const std::string& msg);  // api.cu: records the thread's last error
bool bwd_tc5_eligible(const fa_bwd_params& a);   // bwd_tc5.cu
int bwd_tc5_launch(const BwdParams& p, const fa_bwd_params& a, cudaStream_t st, std::string* err);
bool bwd_wide_eligible(const fa_bwd_params& a);  // bwd_wide.cu
int bwd_wide_launch(const BwdParams& p, const fa_bwd_params& a, cudaStream_t st, std::string* err);
void count_launches(int n);                      // api.cu: fa_b200_launch_count

static size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

// Pairs per chunk of the work-item order (ItemOrder in tile_order.cuh): all of them when what they stream (two 16-bit
// tensors of `rows` rows and `heads` heads) stays in L2 together, otherwise one.  Forward and backward, all pairs against one
// at a time: 14 - 60 MB 0.89 - 0.98 x, 64 - 88 MB 0.98 - 1.00 x, 92 - 96 MB 0.99 - 1.035 x (b 24, s 512, 16 heads, d 128: 298
// -> 309 us), 104 - 114 MB 1.01 - 1.06 x; the 4 K causal case, 268 MB, in chunks of ten pairs: dK / dV kernel 917 -> 1017 us.
// With grouped heads the dK / dV items are fewer and longer, and balance is worth more: 96 MB 1306 -> 1252 us (b 3, s 4096, 32 / 8
// heads, d 64).  Only a causal mask makes the blocks of a pair unequal; without one a pair at a time.
static int bwd_chunk(bool causal, int pairs, int64_t rows, int heads, int d, bool grouped) {
  const int64_t budget = (grouped ? 96ll : 88ll) << 20;
  return causal && 4 * rows * heads * d <= budget ? pairs : 1;
}

template <int HD, typename T>
static cudaError_t launch_bwd(const BwdParams& p, int n_kblocks, cudaStream_t st) {
  constexpr int smem = BwdSmem<HD>::BYTES;
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(bwd_kernel<HD, T>), smem);
  if (e != cudaSuccess) return e;
  bwd_kernel<HD, T><<<dim3(n_kblocks, p.h_k, p.b), kBwdThreads, smem, st>>>(p);
  return cudaGetLastError();
}

}  // namespace fa

extern "C" {

// Which kernels a call runs on: the two of head dims up to 128, or the one of wider heads; neither: the mma.sync kernel.
static bool bwd_runs_tc5(const fa_bwd_params* a) { return a->kernel != 1 && fa::bwd_tc5_eligible(*a); }
static bool bwd_runs_wide(const fa_bwd_params* a) { return a->kernel == 0 && fa::bwd_wide_eligible(*a); }

// First part of the workspace: the fp32 dQ accumulator of the mma.sync kernel, or the work-item counters of the tcgen05
// kernels (which write dQ directly).
static size_t bwd_accum_bytes(const fa_bwd_params* a, int64_t rows) {
  if (bwd_runs_tc5(a) || bwd_runs_wide(a)) return 16;
  const int d_pad = a->d <= 64 ? 64 : (a->d <= 128 ? 128 : 256);
  return fa::align16((size_t)rows * a->h * d_pad * sizeof(float));
}

size_t fa_b200_bwd_workspace_bytes(const fa_bwd_params* a) {
  if (!a) return 0;
  const int64_t rows = a->cu_seqlens_q ? a->total_q : (int64_t)a->b * a->seqlen_q;
  return bwd_accum_bytes(a, rows) + fa::align16((size_t)rows * a->h * sizeof(float));
}

int fa_b200_bwd(const fa_bwd_params* a, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace fa;
  if (!a) return fail_bwd(FA_ERR_INVALID, "null parameter block");
  if (!a->q || !a->k || !a->v || !a->o || !a->dout || !a->lse || !a->dq || !a->dk || !a->dv)
    return fail_bwd(FA_ERR_INVALID, "q, k, v, o, dout, lse, dq, dk and dv must be non-null");
  if (a->dtype != FA_FP16 && a->dtype != FA_BF16) return fail_bwd(FA_ERR_INVALID, "FlashAttention only supports FP16 and BF16 data types");
  if (a->b <= 0 || a->h <= 0 || a->h_k <= 0 || a->h % a->h_k != 0)
    return fail_bwd(FA_ERR_INVALID, "Number of heads in key/value must divide number of heads in query");
  if (a->d <= 0 || a->d % 8 != 0) return fail_bwd(FA_ERR_INVALID, "head dimension must be a multiple of 8 (pad it on the caller side)");
  if (a->d > 256) return fail_bwd(FA_ERR_INVALID, "FlashAttention only supports head dimension at most 256");
  if (a->softcap < 0.f) return fail_bwd(FA_ERR_INVALID, "softcap must be non-negative (0.0 disables softcap)");
  if ((a->cu_seqlens_q != nullptr) != (a->cu_seqlens_k != nullptr))
    return fail_bwd(FA_ERR_INVALID, "cu_seqlens_q and cu_seqlens_k must be passed together");
  const bool varlen = a->cu_seqlens_q != nullptr;
  const int64_t rows = varlen ? a->total_q : (int64_t)a->b * a->seqlen_q;
  if (rows == 0 || a->seqlen_k == 0) return FA_OK;
  const int64_t canon_head = varlen ? a->total_q : a->seqlen_q;
  if (a->lse_head_stride != canon_head || (!varlen && a->lse_batch_stride != (int64_t)a->h * a->seqlen_q))
    return fail_bwd(FA_ERR_INVALID, "softmax_lse must be contiguous (b, h, s_q) / (h, total_q)");
  const size_t need = fa_b200_bwd_workspace_bytes(a);
  if (!workspace || workspace_bytes < need) return fail_bwd(FA_ERR_WORKSPACE, "workspace missing or too small");
  if ((reinterpret_cast<uintptr_t>(workspace) & 15) != 0) return fail_bwd(FA_ERR_WORKSPACE, "workspace must be 16-byte aligned");
  const int64_t st[] = {a->q_row_stride, a->q_head_stride, a->k_row_stride, a->k_head_stride, a->v_row_stride, a->v_head_stride,
                        a->o_row_stride, a->o_head_stride, a->do_row_stride, a->do_head_stride, a->dq_row_stride,
                        a->dq_head_stride, a->dk_row_stride, a->dk_head_stride, a->dv_row_stride, a->dv_head_stride,
                        a->q_batch_stride, a->k_batch_stride, a->v_batch_stride, a->do_batch_stride, a->dq_batch_stride,
                        a->dk_batch_stride, a->dv_batch_stride, a->o_batch_stride};
  for (int64_t s : st)
    if (s % 8 != 0) return fail_bwd(FA_ERR_INVALID, "tensor strides must be multiples of 8 elements (16-byte rows)");
  const void* ptrs[] = {a->q, a->k, a->v, a->o, a->dout, a->dq, a->dk, a->dv};
  for (const void* ptr : ptrs)
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0) return fail_bwd(FA_ERR_INVALID, "tensors must be 16-byte aligned");

  cudaStream_t cs = reinterpret_cast<cudaStream_t>(stream);
  BwdParams p;
  std::memset(&p, 0, sizeof(p));
  p.q = a->q; p.k = a->k; p.v = a->v; p.o = a->o; p.dout = a->dout; p.lse = a->lse;
  p.dq = a->dq; p.dk = a->dk; p.dv = a->dv;
  p.cu_seqlens_q = a->cu_seqlens_q; p.cu_seqlens_k = a->cu_seqlens_k;
  p.q_batch_stride = a->q_batch_stride; p.q_row_stride = a->q_row_stride; p.q_head_stride = a->q_head_stride;
  p.k_batch_stride = a->k_batch_stride; p.k_row_stride = a->k_row_stride; p.k_head_stride = a->k_head_stride;
  p.v_batch_stride = a->v_batch_stride; p.v_row_stride = a->v_row_stride; p.v_head_stride = a->v_head_stride;
  p.o_batch_stride = a->o_batch_stride; p.o_row_stride = a->o_row_stride; p.o_head_stride = a->o_head_stride;
  p.do_batch_stride = a->do_batch_stride; p.do_row_stride = a->do_row_stride; p.do_head_stride = a->do_head_stride;
  p.dq_batch_stride = a->dq_batch_stride; p.dq_row_stride = a->dq_row_stride; p.dq_head_stride = a->dq_head_stride;
  p.dk_batch_stride = a->dk_batch_stride; p.dk_row_stride = a->dk_row_stride; p.dk_head_stride = a->dk_head_stride;
  p.dv_batch_stride = a->dv_batch_stride; p.dv_row_stride = a->dv_row_stride; p.dv_head_stride = a->dv_head_stride;
  p.lse_batch_stride = a->lse_batch_stride; p.lse_head_stride = a->lse_head_stride;
  p.b = a->b; p.seqlen_q = a->seqlen_q; p.seqlen_k = a->seqlen_k; p.h = a->h; p.h_k = a->h_k; p.d = a->d;
  p.d_pad = a->d <= 64 ? 64 : (a->d <= 128 ? 128 : 256);
  p.total_q = (int32_t)rows;
  p.dq_sectors = whole_sectors(p.dq, p.d, p.b, p.dq_row_stride, p.dq_head_stride, p.dq_batch_stride);
  p.dk_sectors = whole_sectors(p.dk, p.d, p.b, p.dk_row_stride, p.dk_head_stride, p.dk_batch_stride);
  p.dv_sectors = whole_sectors(p.dv, p.d, p.b, p.dv_row_stride, p.dv_head_stride, p.dv_batch_stride);
  // window normalisation of the golden (tests/fa_small_op_golden.py:21-33; the same rule as the forward's host code)
  int wl = a->window_left, wr = a->window_right;
  if (wl >= a->seqlen_k - 1) wl = -1;
  if (wr >= a->seqlen_q - 1) wr = -1;
  if (a->causal) wr = 0;
  p.is_causal = (wl < 0 && wr == 0) ? 1 : 0;
  p.is_local = ((wl >= 0 || wr >= 0) && !p.is_causal) ? 1 : 0;
  p.wl = wl; p.wr = wr;
  p.softmax_scale = a->softmax_scale;
  p.scale_log2 = a->softmax_scale * kLog2e;
  p.softcap = a->softcap;
  {
    const int64_t k_rows = varlen ? a->total_k : (int64_t)a->b * a->seqlen_k;
    const int kv_pairs = a->h_k * a->b, q_pairs = a->h * a->b;
    p.kv_items.set((a->seqlen_k + kBwdItem - 1) / kBwdItem, kv_pairs, bwd_chunk(p.is_causal, kv_pairs, rows, a->h, a->d, a->h > a->h_k));
    p.q_items.set((a->seqlen_q + kBwdItem - 1) / kBwdItem, q_pairs, bwd_chunk(p.is_causal, q_pairs, k_rows, a->h_k, a->d, a->h > a->h_k));
    p.group = a->h / a->h_k;
    p.by_group.set(p.group);
    p.by_h_k.set(a->h_k);
    p.by_h.set(a->h);
  }
  const size_t acc_bytes = bwd_accum_bytes(a, rows);
  p.dq_accum = reinterpret_cast<float*>(workspace);
  p.delta = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + acc_bytes);

  if (a->kernel < 0 || a->kernel > 2) return fail_bwd(FA_ERR_INVALID, "kernel must be 0 (automatic), 1 (mma.sync) or 2 (tcgen05)");
  const bool tc5 = bwd_runs_tc5(a), wide = bwd_runs_wide(a);
  if (a->kernel == 2 && !tc5)
    return fail_bwd(FA_ERR_UNSUPPORTED, "kernel = 2: this tcgen05 backward covers head dims up to 128 (packed input: total_k given); "
                                        "wider heads have theirs with kernel = 0");
  cudaError_t e = cudaSuccess;
  if (!tc5 && !wide) e = cudaMemsetAsync(p.dq_accum, 0, acc_bytes, cs);
  if (e != cudaSuccess) return fail_bwd(FA_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
  const bool bf = a->dtype == FA_BF16;
  auto launch_delta = [&](auto kern, int lanes) {
    const int64_t per_block = kDeltaThreads / lanes * kDeltaRows, n_rows = varlen ? rows : a->seqlen_q;
    const int64_t grid = (n_rows + per_block - 1) / per_block * a->h * (varlen ? 1 : a->b);
    kern<<<(unsigned)grid, kDeltaThreads, 0, cs>>>(p);
  };
  if (a->d <= 64) bf ? launch_delta(bwd_delta_kernel<__nv_bfloat16, 8>, 8) : launch_delta(bwd_delta_kernel<__half, 8>, 8);
  else bf ? launch_delta(bwd_delta_kernel<__nv_bfloat16, 16>, 16) : launch_delta(bwd_delta_kernel<__half, 16>, 16);
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail_bwd(FA_ERR_CUDA, std::string("backward (delta) launch: ") + cudaGetErrorString(e));
  if (tc5 || wide) {
    std::string err;
    const int rc = tc5 ? bwd_tc5_launch(p, *a, cs, &err) : bwd_wide_launch(p, *a, cs, &err);
    if (rc != FA_OK) return fail_bwd(rc, err);
    count_launches(tc5 ? 3 : 2);
    return FA_OK;
  }
  const int n_kblocks = (a->seqlen_k + kBwdBN - 1) / kBwdBN;
  if (p.d_pad == 64) e = bf ? launch_bwd<64, __nv_bfloat16>(p, n_kblocks, cs) : launch_bwd<64, __half>(p, n_kblocks, cs);
  else if (p.d_pad == 128) e = bf ? launch_bwd<128, __nv_bfloat16>(p, n_kblocks, cs) : launch_bwd<128, __half>(p, n_kblocks, cs);
  else e = bf ? launch_bwd<256, __nv_bfloat16>(p, n_kblocks, cs) : launch_bwd<256, __half>(p, n_kblocks, cs);
  if (e != cudaSuccess) return fail_bwd(FA_ERR_CUDA, std::string("backward launch: ") + cudaGetErrorString(e));
  const int conv_grid = (int)std::min<int64_t>((rows * a->h * (p.d_pad / 4) + 255) / 256, 148 * 8);
  if (bf) bwd_convert_kernel<__nv_bfloat16><<<conv_grid, 256, 0, cs>>>(p);
  else bwd_convert_kernel<__half><<<conv_grid, 256, 0, cs>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail_bwd(FA_ERR_CUDA, std::string("backward (convert) launch: ") + cudaGetErrorString(e));
  count_launches(3);
  return FA_OK;
}

}  // extern "C"
