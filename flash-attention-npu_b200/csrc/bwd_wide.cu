// tcgen05 backward for head dims 129 .. 256: TMA descriptors and launch (kernel in bwd_wide_kernel.cuh).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <type_traits>

#include "bwd_wide_kernel.cuh"
#include "tc5_api.cuh"

namespace fa {

// Packed input needs the number of k / v rows for the TMA bounds; alignment and strides are checked by fa_b200_bwd.
bool bwd_wide_eligible(const fa_bwd_params& a) { return a.d > 128 && a.d <= 256 && !(a.cu_seqlens_q && a.total_k <= 0); }

int bwd_wide_launch(const BwdParams& p, const fa_bwd_params& a, cudaStream_t st, std::string* err) {
  using namespace btc5;
  int32_t* status = device_status_word();
  if (!status) { *err = "cannot look up the device status word"; return FA_ERR_CUDA; }
  const bool varlen = a.cu_seqlens_q != nullptr;
  const int64_t q_rows = varlen ? a.total_q : a.seqlen_q, k_rows = varlen ? a.total_k : a.seqlen_k;
  const int64_t outer = varlen ? 1 : a.b;
  WideMaps m;
  auto both = [&](CUtensorMap* big, CUtensorMap* unit, const void* ptr, int heads, int64_t rows, int64_t hs, int64_t rs, int64_t bs) {
    return tma_encode_rows(big, ptr, a.dtype, a.d, heads, rows, outer, hs, rs, bs, kBlk) &&
           tma_encode_rows(unit, ptr, a.dtype, a.d, heads, rows, outer, hs, rs, bs, kUnit);
  };
  if (!both(&m.q, &m.q_u, a.q, a.h, q_rows, a.q_head_stride, a.q_row_stride, a.q_batch_stride) ||
      !both(&m.dout, &m.do_u, a.dout, a.h, q_rows, a.do_head_stride, a.do_row_stride, a.do_batch_stride) ||
      !both(&m.k, &m.k_u, a.k, a.h_k, k_rows, a.k_head_stride, a.k_row_stride, a.k_batch_stride) ||
      !both(&m.v, &m.v_u, a.v, a.h_k, k_rows, a.v_head_stride, a.v_row_stride, a.v_batch_stride)) {
    *err = "cuTensorMapEncodeTiled failed";
    return FA_ERR_CUDA;
  }
  int dev = 0, num_sm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&num_sm, cudaDevAttrMultiProcessorCount, dev);
  const long long items = 2LL * ((a.seqlen_k + kBlk - 1) / kBlk) * a.h_k * a.b + (long long)((a.seqlen_q + kBlk - 1) / kBlk) * a.h * a.b;
  if (items > 0x7fffffffLL) { *err = "too many work items"; return FA_ERR_UNSUPPORTED; }
  const unsigned grid = (unsigned)std::min<long long>(items, num_sm);
  // the work-item counter: the first bytes of the workspace, cleared by the kernel in front (bwd_delta_kernel)
  int32_t* counter = reinterpret_cast<int32_t*>(p.dq_accum);
  cudaError_t e = cudaSuccess;
  auto launch = [&](auto kern, int smem) {
    if (e == cudaSuccess) e = allow_smem(reinterpret_cast<const void*>(kern), smem);
    if (e == cudaSuccess) {
      kern<<<grid, kThreads, smem, st>>>(p, m, status, counter);
      e = cudaGetLastError();
    }
  };
  auto by_type = [&](auto cap_tag, auto hd_tag) {
    constexpr bool C = decltype(cap_tag)::value;
    constexpr int HD = decltype(hd_tag)::value;
    if (a.dtype == FA_BF16) launch(bwd_wide_kernel<__nv_bfloat16, 1, C, HD>, wide_smem_bytes<HD>());
    else launch(bwd_wide_kernel<__half, 0, C, HD>, wide_smem_bytes<HD>());
  };
  auto by_cap = [&](auto hd_tag) {
    if (a.softcap > 0.f) by_type(std::true_type{}, hd_tag);
    else by_type(std::false_type{}, hd_tag);
  };
  if (a.d <= 192) by_cap(std::integral_constant<int, 192>{});
  else by_cap(std::integral_constant<int, 256>{});
  if (e != cudaSuccess) { *err = std::string("tcgen05 backward launch: ") + cudaGetErrorString(e); return FA_ERR_CUDA; }
  return FA_OK;
}

}  // namespace fa
