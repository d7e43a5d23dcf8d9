// A step's varlen metadata to the device, by way of a kernel's parameters.
//
// The arrays are a few hundred to a few thousand words.  As a copy from pinned memory they cost
// the stream 7 us between its kernels once there are more than about a kilobyte of them (the copy
// engine and the hand-overs to and from it; a block of four prompts of 1024 tokens with its
// neighbouring ops 119 -> 126 us when the task table came along), and the staging buffer had to
// be kept until the copy was over.  Parameters travel with the launch and belong to it.
// The same launch brings a paged step's page table and key lengths to the plan's own: it is the first
// one behind the host's checks of both, so a step that is refused leaves the plan's as they were.  The
// lengths are the words that were checked (the kernel walks the page table by them).
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

constexpr int kParts = 8;           // the last: key lengths, to the plan's own
constexpr int kUpThreads = 512;
constexpr int kMaxBlocks = 32;

template <int N>
struct Words {
  int part_end[kParts];     // parts lie one after another in w: where each ends,
  int part_to[kParts];      // and what is added to a word's place to get where it goes
  int32_t w[N];
};

template <int N>
__global__ void __launch_bounds__(kUpThreads)
upload_kernel(int32_t* dst, const __grid_constant__ Words<N> s, const __grid_constant__ PagedIn paged) {
  let_next_start();
  wait_for_previous();       // (it may be reading the arrays)
  if (paged.table) {
    const int first = blockIdx.x * kUpThreads + threadIdx.x, step = gridDim.x * kUpThreads;
    const long long total = static_cast<long long>(paged.num_batch) * paged.width;
    for (long long i = first; i < total; i += step) {
      const int b = static_cast<int>(i / paged.width), j = static_cast<int>(i % paged.width);
      paged.table_out[static_cast<long long>(b) * paged.pitch_out + j] = paged.table[b * paged.pitch + j];
    }
  }
  if (blockIdx.x != 0) return;
  for (int i = threadIdx.x; i < s.part_end[kParts - 1]; i += kUpThreads) {
    int k = 0;
#pragma unroll
    for (int j = 0; j + 1 < kParts; ++j) k += i >= s.part_end[j];
    (k == kParts - 1 ? paged.lens_out : dst)[i + s.part_to[k]] = s.w[i];
  }
}

template <int N>
cudaError_t upload(int32_t* dst, const int32_t* const (&src)[kParts], const int (&off)[kParts],
                   const int (&len)[kParts], int from, int to, const PagedIn& paged, cudaStream_t stream) {
  Words<N> s;
  int at = 0, seen = 0;
  for (int k = 0; k < kParts; ++k) {              // words [from, to) of the parts laid end to end
    const int lo = std::max(from - seen, 0), hi = std::min(to - seen, len[k]);
    if (hi > lo) memcpy(s.w + at, src[k] + lo, sizeof(int32_t) * (hi - lo));
    s.part_to[k] = off[k] + lo - at;
    if (hi > lo) at += hi - lo;
    s.part_end[k] = at;
    seen += len[k];
  }
  const long long entries = paged.table ? static_cast<long long>(paged.num_batch) * paged.width : 0;
  const int blocks = static_cast<int>(std::min<long long>(1 + entries / 2048, kMaxBlocks));
  return launch_behind(upload_kernel<N>, blocks, kUpThreads, 0, stream, dst, s, paged);
}

}  // namespace

int upload_meta(const ma_stage_tasks_args* a, uint64_t meta_dev, const PagedIn& paged, cudaStream_t stream) {
  if (!a || !meta_dev || (meta_dev & 15u)) return MA_ERR_INVALID;
  const int rc = ma_stage_tasks(a);
  if (rc < 0) return rc;
  const ma_stage_meta_args& m = a->meta;
  const int R = m.num_row_tiles, B = m.num_batch;
  const int off[kParts] = {m.off_cu_q, m.off_cu_k, m.off_batch_idx, m.off_m_block, m.off_order, m.off_actv,
                           a->off_tasks, 0};
  const int len[kParts] = {B + 1, B + 1, R, R, R, MA_NUM_ACTV, 4 + kTaskWords * m.staging[a->off_tasks],
                           paged.table ? B : 0};
  const int32_t* src[kParts];
  for (int k = 0; k < kParts; ++k) src[k] = k == kParts - 1 ? paged.lens : m.staging + off[k];
  int total = 0;
  for (int n : len) total += n;
  int32_t* dst = reinterpret_cast<int32_t*>(meta_dev);
  // (a launch copies all of its parameter block, so there is one for small steps)
  constexpr int kSmall = 960, kLarge = 7680;
  cudaError_t e = cudaSuccess;
  if (total <= kSmall) {
    e = upload<kSmall>(dst, src, off, len, 0, total, paged, stream);
  } else {
    PagedIn in = paged;
    for (int from = 0; from < total && e == cudaSuccess; from += kLarge) {
      e = upload<kLarge>(dst, src, off, len, from, std::min(total, from + kLarge), in, stream);
      in.table = nullptr;         // (copied with the first words)
    }
  }
  return e == cudaSuccess ? rc : MA_ERR_CUDA;
}

}  // namespace ma

extern "C" int ma_upload_meta(const ma_stage_tasks_args* a, uint64_t meta_dev, void* stream) {
  return ma::upload_meta(a, meta_dev, ma::PagedIn{}, static_cast<cudaStream_t>(stream));
}
