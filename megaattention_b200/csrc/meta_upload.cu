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
#include "paged.cuh"

namespace ma {
namespace {

constexpr int kParts = 7, kPagedParts = 8;     // (a paged step's key lengths: to the plan's own)
constexpr int kUpThreads = 512;
constexpr int kMaxBlocks = 32;

template <int N, int P>
struct Words {
  int part_end[P];          // parts lie one after another in w: where each ends,
  int part_to[P];           // and what is added to a word's place to get where it goes
  int32_t w[N];
};

// One block's job; the page table's copy has as many as its size asks for.
template <int N, int P>
__device__ __forceinline__ void put_words(int32_t* dst, int32_t* lens_out, const Words<N, P>& s) {
  for (int i = threadIdx.x; i < s.part_end[P - 1]; i += kUpThreads) {
    int k = 0;
#pragma unroll
    for (int j = 0; j + 1 < P; ++j) k += i >= s.part_end[j];
    (P == kPagedParts && k == P - 1 ? lens_out : dst)[i + s.part_to[k]] = s.w[i];
  }
}

// (Packed steps have a kernel of their own: with the paged one's parameters in it three short prompts
// took 30.4 us for 29.9.)
template <int N>
__global__ void __launch_bounds__(kUpThreads)
upload_kernel(int32_t* dst, const __grid_constant__ Words<N, kParts> s) {
  let_next_start();
  wait_for_previous();       // (it may be reading the arrays)
  put_words(dst, dst, s);
}

template <int N>
__global__ void __launch_bounds__(kUpThreads)
upload_paged_kernel(int32_t* dst, const __grid_constant__ PagedIn in, const __grid_constant__ Words<N, kPagedParts> s) {
  let_next_start();
  wait_for_previous();
  if (in.table) {
    for_each_entry(in.num_batch, in.width, blockIdx.x * kUpThreads + threadIdx.x, gridDim.x * kUpThreads,
                   [&](int b, int j) {
                     in.table_out[static_cast<long long>(b) * in.pitch_out + j] = in.table[b * in.pitch + j];
                   });
  }
  if (blockIdx.x == 0) put_words(dst, in.lens_out, s);
}

// Words [from, to) of the parts laid end to end.
template <int N, int P>
void pack(Words<N, P>& s, const int32_t* const (&src)[kPagedParts], const int (&off)[kPagedParts],
          const int (&len)[kPagedParts], int from, int to) {
  int at = 0, seen = 0;
  for (int k = 0; k < P; ++k) {
    const int lo = std::max(from - seen, 0), hi = std::min(to - seen, len[k]);
    if (hi > lo) memcpy(s.w + at, src[k] + lo, sizeof(int32_t) * (hi - lo));
    s.part_to[k] = off[k] + lo - at;
    if (hi > lo) at += hi - lo;
    s.part_end[k] = at;
    seen += len[k];
  }
}

template <int N>
cudaError_t upload(int32_t* dst, const int32_t* const (&src)[kPagedParts], const int (&off)[kPagedParts],
                   const int (&len)[kPagedParts], int from, int to, const PagedIn& in, cudaStream_t stream) {
  if (!in.lens) {
    Words<N, kParts> s;
    pack(s, src, off, len, from, to);
    return launch_behind(upload_kernel<N>, 1, kUpThreads, 0, stream, dst, s);
  }
  Words<N, kPagedParts> s;
  pack(s, src, off, len, from, to);
  const long long entries = in.table ? static_cast<long long>(in.num_batch) * in.width : 0;
  const int blocks = static_cast<int>(std::min<long long>(1 + entries / 2048, kMaxBlocks));
  return launch_behind(upload_paged_kernel<N>, blocks, kUpThreads, 0, stream, dst, in, s);
}

}  // namespace

int upload_meta(const ma_stage_tasks_args* a, uint64_t meta_dev, const PagedIn& paged, cudaStream_t stream) {
  if (!a || !meta_dev || (meta_dev & 15u)) return MA_ERR_INVALID;
  const int rc = ma_stage_tasks(a);
  if (rc < 0) return rc;
  const ma_stage_meta_args& m = a->meta;
  const int R = m.num_row_tiles, B = m.num_batch;
  const int off[kPagedParts] = {m.off_cu_q, m.off_cu_k, m.off_batch_idx, m.off_m_block, m.off_order, m.off_actv,
                           a->off_tasks, 0};
  const int len[kPagedParts] = {B + 1, B + 1, R, R, R, MA_NUM_ACTV, 4 + kTaskWords * m.staging[a->off_tasks],
                           paged.lens ? B : 0};
  const int32_t* src[kPagedParts];
  for (int k = 0; k < kParts; ++k) src[k] = m.staging + off[k];
  src[kParts] = paged.lens;
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
