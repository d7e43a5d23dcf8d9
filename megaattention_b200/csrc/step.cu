// A serving step in one call: what is between a layer's call and its launch, natively.
//
// Small steps waited for the host: a layer of three short prompts is 31 us on the GPU and was 52 us
// of Python and torch calls, and a paged call had another 100 us between the arrival of the key lengths
// and its launch.  Here the descriptors are encoded, the batch's metadata staged and the kernels
// launched without leaving C.  A paged batch's lengths and the range of its page numbers come back by
// one kernel, which writes them to pinned memory; it runs while the descriptors are encoded, and what is
// left after it is the metadata and two launches.  Nothing of the plan changes before the checks are
// over: its copies of lengths and table are written with the metadata.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <new>
#include <vector>

#include "../../include/megaattn_b200.h"
#include "kparams.h"
#include "launch.cuh"
#include "paged.cuh"

namespace ma {
int plan_encode_inputs(const ma_plan* pl, CUtensorMap* fresh, uint64_t Q, uint64_t K, uint64_t V, uint64_t W_o,
                       int64_t tot_q, int64_t tot_k, int64_t w_width);
void plan_take_inputs(ma_plan* pl, const CUtensorMap* fresh);
void plan_inputs(const ma_plan* pl, CUtensorMap* maps);
int plan_check_launch(const ma_plan* pl, const ma_launch_args* a);
int upload_meta(const ma_stage_tasks_args* a, uint64_t meta_dev, const PagedIn& paged, cudaStream_t stream);

namespace {

constexpr int kCollectThreads = 256;

// host: num_batch lengths, then {smallest, largest} page number of every block's share of the table.
__global__ void __launch_bounds__(kCollectThreads) collect_kernel(
    const int32_t* lens, const int32_t* table, int32_t num_batch, int32_t width, int64_t pitch, int32_t* host) {
  __shared__ int32_t lo_s[kCollectThreads / 32], hi_s[kCollectThreads / 32];
  wait_for_previous();
  const int first = blockIdx.x * kCollectThreads + threadIdx.x, step = gridDim.x * kCollectThreads;
  for (int b = first; b < num_batch; b += step) host[b] = lens[b];
  int32_t lo = 0x7fffffff, hi = -0x7fffffff - 1;
  for_each_entry(num_batch, width, first, step, [&](int b, int j) {
    const int32_t page = table[b * pitch + j];
    lo = min(lo, page);
    hi = max(hi, page);
  });
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) { lo_s[threadIdx.x >> 5] = lo; hi_s[threadIdx.x >> 5] = hi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kCollectThreads / 32; ++w) { lo = min(lo, lo_s[w]); hi = max(hi, hi_s[w]); }
    host[num_batch + 2 * blockIdx.x] = lo;
    host[num_batch + 2 * blockIdx.x + 1] = hi;
  }
}

}  // namespace
}  // namespace ma

extern "C" int ma_step(ma_plan* plan, const ma_step_args* a, void* stream_) {
  if (!plan || !a || !a->cu_q || a->num_batch < 1 || !a->meta_dev) return MA_ERR_INVALID;
  const bool paged = a->page_table != 0;
  if (paged && (!a->cache_seqlens || !a->page_table_out || !a->cache_seqlens_out || !a->host_words ||
                a->table_width < 1 || a->table_width > a->table_pitch_out || a->table_pitch < 0))
    return MA_ERR_INVALID;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int B = a->num_batch;
  int blocks = 0;
  if (paged) {
    const int64_t total = static_cast<int64_t>(B) * a->table_width;
    blocks = static_cast<int>(std::min<int64_t>((total + 2047) / 2048, MA_STEP_BLOCKS));
    if (ma::launch_behind(ma::collect_kernel, blocks, ma::kCollectThreads, 0, stream,
                          reinterpret_cast<const int32_t*>(a->cache_seqlens),
                          reinterpret_cast<const int32_t*>(a->page_table), B, a->table_width, a->table_pitch,
                          a->host_words) != cudaSuccess)
      return MA_ERR_CUDA;
  }
  CUtensorMap fresh[7];
  int rc = ma::plan_encode_inputs(plan, fresh, a->Q, a->K, a->V, a->W_o, a->tot_q, a->tot_k, a->w_width);
  // (the lengths are on their way into host_words: nobody leaves before they are there)
  if (paged && cudaStreamSynchronize(stream) != cudaSuccess) return MA_ERR_CUDA;
  if (rc != MA_OK) return rc;
  try {
    static thread_local std::vector<int64_t> cu_k;
    static thread_local std::vector<int32_t> words;
    const int64_t* ck = a->cu_k ? a->cu_k : a->cu_q;
    if (paged) {
      cu_k.assign(static_cast<size_t>(B) + 1, 0);
      int32_t lo = a->host_words[B], hi = a->host_words[B + 1];
      for (int i = 1; i < blocks; ++i) {
        lo = std::min(lo, a->host_words[B + 2 * i]);
        hi = std::max(hi, a->host_words[B + 2 * i + 1]);
      }
      for (int b = 0; b < B; ++b) {
        const int64_t n = a->host_words[b];
        if ((n + 127) / 128 > a->table_width) return MA_STEP_NARROW;
        cu_k[b + 1] = cu_k[b] + n;
      }
      if (lo < 0 || hi >= a->tot_k / 128) return MA_STEP_PAGES;
      ck = cu_k.data();
    }
    const int64_t cap = std::max<int64_t>(0, std::min<int64_t>(a->max_row_tiles, a->cu_q[B] / 128 + B));
    words.resize(static_cast<size_t>(3 * (B + 1) + 2 * cap + 2));
    int32_t* cu_q32 = words.data();
    int32_t* cu_k32 = cu_q32 + B + 1;
    int32_t* cu_m = cu_k32 + B + 1;
    int32_t* batch_idx = cu_m + B + 1;
    int32_t* m_block = batch_idx + cap;
    const int R = ma_row_desc(a->cu_q, ck, B, static_cast<int32_t>(cap), cu_q32, cu_k32, cu_m, batch_idx, m_block);
    if (R == MA_ERR_INVALID) return MA_STEP_LENGTHS;
    if (R < 1) return MA_STEP_TILES;
    ma_stage_tasks_args s = a->stage;
    s.meta.cu_q = cu_q32; s.meta.cu_k = cu_k32; s.meta.batch_idx = batch_idx; s.meta.m_block = m_block;
    s.meta.num_batch = B; s.meta.num_row_tiles = R;
    s.meta.prime = std::min(s.meta.prime, R);
    rc = ma::plan_check_launch(plan, &a->launch);
    if (rc != MA_OK) return rc;
    ma::PagedIn in{};
    if (paged)
      in = {reinterpret_cast<const int*>(a->page_table), a->host_words, reinterpret_cast<int*>(a->page_table_out),
            reinterpret_cast<int*>(a->cache_seqlens_out), a->table_pitch, a->table_pitch_out, a->table_width, B};
    rc = ma::upload_meta(&s, a->meta_dev, in, stream);
    if (rc != MA_OK) return rc;
    // (a launch that fails leaves the plan with the inputs that its owner knows of)
    CUtensorMap before[7];
    ma::plan_inputs(plan, before);
    ma::plan_take_inputs(plan, fresh);
    rc = ma_launch(plan, &a->launch, stream_);
    if (rc != MA_OK) ma::plan_take_inputs(plan, before);
    return rc == MA_OK ? R : rc;
  } catch (const std::bad_alloc&) {
    return MA_ERR_CAPACITY;
  }
}
