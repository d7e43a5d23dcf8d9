// A step's varlen metadata to the device, by way of a kernel's parameters.
//
// The arrays are a few hundred to a few thousand words.  As a copy from pinned memory they cost
// the stream 7 us between its kernels once there are more than about a kilobyte of them (the copy
// engine and the hand-overs to and from it; a block of four prompts of 1024 tokens with its
// neighbouring ops 119 -> 126 us when the task table came along), and the staging buffer had to
// be kept until the copy was over.  Parameters travel with the launch and belong to it.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <vector>

#include "../../include/megaattn_b200.h"
#include "kparams.h"
#include "launch.cuh"

namespace ma {
namespace {

constexpr int kParts = 7;
constexpr int kUpThreads = 512;

template <int N>
struct Words {
  int part_end[kParts];     // parts lie one after another in w: where each ends,
  int part_to[kParts];      // and what is added to a word's place to get where it goes
  int32_t w[N];
};

template <int N>
__global__ void __launch_bounds__(kUpThreads) upload_kernel(int32_t* dst, const __grid_constant__ Words<N> s) {
  let_next_start();
  wait_for_previous();       // (it may be reading the arrays)
  for (int i = threadIdx.x; i < s.part_end[kParts - 1]; i += kUpThreads) {
    int k = 0;
#pragma unroll
    for (int j = 0; j + 1 < kParts; ++j) k += i >= s.part_end[j];
    dst[i + s.part_to[k]] = s.w[i];
  }
}

template <int N>
cudaError_t upload(int32_t* dst, const int32_t* src, const int (&off)[kParts], const int (&len)[kParts], int from, int to,
            cudaStream_t stream) {
  Words<N> s;
  int at = 0, seen = 0;
  for (int k = 0; k < kParts; ++k) {              // words [from, to) of the parts laid end to end
    const int lo = std::max(from - seen, 0), hi = std::min(to - seen, len[k]);
    if (hi > lo) memcpy(s.w + at, src + off[k] + lo, sizeof(int32_t) * (hi - lo));
    s.part_to[k] = off[k] + lo - at;
    if (hi > lo) at += hi - lo;
    s.part_end[k] = at;
    seen += len[k];
  }
  return launch_behind(upload_kernel<N>, 1, kUpThreads, 0, stream, dst, s);
}

}  // namespace
}  // namespace ma

extern "C" int ma_upload_meta(const ma_stage_tasks_args* a, uint64_t meta_dev, void* stream) {
  if (!a || !meta_dev || (meta_dev & 15u)) return MA_ERR_INVALID;
  const int rc = ma_stage_tasks(a);
  if (rc < 0) return rc;
  const ma_stage_meta_args& m = a->meta;
  const int R = m.num_row_tiles, B = m.num_batch;
  const int off[ma::kParts] = {m.off_cu_q, m.off_cu_k, m.off_batch_idx, m.off_m_block, m.off_order, m.off_actv,
                               a->off_tasks};
  const int len[ma::kParts] = {B + 1, B + 1, R, R, R, MA_NUM_ACTV, 4 + ma::kTaskWords * m.staging[a->off_tasks]};
  int total = 0;
  for (int n : len) total += n;
  int32_t* dst = reinterpret_cast<int32_t*>(meta_dev);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // (a launch copies all of its parameter block, so there is one for small steps)
  constexpr int kSmall = 960, kLarge = 7680;
  cudaError_t e = cudaSuccess;
  if (total <= kSmall) {
    e = ma::upload<kSmall>(dst, m.staging, off, len, 0, total, st);
  } else {
    for (int from = 0; from < total && e == cudaSuccess; from += kLarge)
      e = ma::upload<kLarge>(dst, m.staging, off, len, from, std::min(total, from + kLarge), st);
  }
  return e == cudaSuccess ? rc : MA_ERR_CUDA;
}
