// Packed copy of the fused launch's output: tile-padded C_sym -> [tot_q, hidden].
//
// The sequences' tiles lie one after another in C_sym, so packed row i of sequence b comes
// from row 128 * (tiles before b) + i.  Bound by memory: 4 bytes per element.  A warp per
// token row, four accesses of 16 bytes in flight per lane; the row -> sequence map travels in
// the kernel's parameters (256 sequences per launch), so the copy depends on nothing that a
// later step may overwrite.  It takes the place of one strided copy per row tile: 108 tiles
// of 4096 columns took 0.9 ms of launches.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/megaattn_b200.h"
#include "launch.cuh"

namespace ma {
namespace {

constexpr int kDtSeqs = 256;
constexpr int kDtThreads = 256;

struct DetileSeqs {
  int n;                          // sequences of this launch
  int row0[kDtSeqs + 1];          // first packed row of each
  int src0[kDtSeqs];              // first C_sym row of each
};

template <typename T>
__global__ void __launch_bounds__(kDtThreads)
detile_kernel(const char* csym_, char* out_, size_t src_pitch,
              size_t dst_pitch, int n_vec, const __grid_constant__ DetileSeqs s) {
  wait_for_previous();
  const char* __restrict__ csym = from_here(csym_);
  char* __restrict__ out = from_here(out_);
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (kDtThreads / 32);
  for (int row = s.row0[0] + blockIdx.x * (kDtThreads / 32) + (threadIdx.x >> 5);
       row < s.row0[s.n]; row += warps) {
    int lo = 0, hi = s.n - 1;     // the last sequence that starts at or before this row
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s.row0[mid] <= row) lo = mid; else hi = mid - 1;
    }
    const T* src = reinterpret_cast<const T*>(
        csym + static_cast<size_t>(s.src0[lo] + (row - s.row0[lo])) * src_pitch);
    T* dst = reinterpret_cast<T*>(out + static_cast<size_t>(row) * dst_pitch);
    for (int c = lane; c < n_vec; c += 128) {
      T v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c + u * 32 < n_vec) v[u] = src[c + u * 32];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c + u * 32 < n_vec) dst[c + u * 32] = v[u];
    }
  }
}

}  // namespace
}  // namespace ma

extern "C" int ma_detile(const ma_detile_args* a, void* stream) {
  if (!a || !a->csym || !a->out || !a->cu_q) return MA_ERR_INVALID;
  if (a->num_batch < 1 || a->hidden < 1 || a->row_pitch < a->hidden || (a->row_pitch & 7))
    return MA_ERR_INVALID;
  if ((a->csym & 15u) || (a->out & 15u)) return MA_ERR_INVALID;
  if (a->cu_q[0] != 0) return MA_ERR_INVALID;
  for (int b = 0; b < a->num_batch; ++b)
    if (a->cu_q[b + 1] < a->cu_q[b]) return MA_ERR_INVALID;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return MA_ERR_CUDA;
  const size_t src_pitch = static_cast<size_t>(a->row_pitch) * 2;
  const size_t dst_pitch = static_cast<size_t>(a->hidden) * 2;
  // widest access that every packed row is aligned to
  const int width = a->hidden % 8 == 0 ? 16 : (a->hidden % 2 == 0 ? 4 : 2);
  const int n_vec = static_cast<int>(dst_pitch / width);
  const char* src = reinterpret_cast<const char*>(a->csym);
  char* dst = reinterpret_cast<char*>(a->out);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaSuccess;
  long long tiles = 0;
  for (int b0 = 0; b0 < a->num_batch && e == cudaSuccess; b0 += ma::kDtSeqs) {
    ma::DetileSeqs s;
    s.n = a->num_batch - b0 < ma::kDtSeqs ? a->num_batch - b0 : ma::kDtSeqs;
    for (int i = 0; i < s.n; ++i) {
      s.row0[i] = a->cu_q[b0 + i];
      if (tiles * 128 > 0x7fffffffLL) return MA_ERR_CAPACITY;
      s.src0[i] = static_cast<int>(tiles * 128);
      tiles += (static_cast<long long>(a->cu_q[b0 + i + 1]) - a->cu_q[b0 + i] + 127) / 128;
    }
    s.row0[s.n] = a->cu_q[b0 + s.n];
    const int rows = s.row0[s.n] - s.row0[0];
    if (rows == 0) continue;
    const int need = (rows + 7) / 8;
    const int grid = need < sms * 8 ? need : sms * 8;
    if (width == 16)
      e = ma::launch_behind(ma::detile_kernel<uint4>, grid, ma::kDtThreads, 0, st, src, dst, src_pitch, dst_pitch,
                            n_vec, s);
    else if (width == 4)
      e = ma::launch_behind(ma::detile_kernel<uint32_t>, grid, ma::kDtThreads, 0, st, src, dst, src_pitch, dst_pitch,
                            n_vec, s);
    else
      e = ma::launch_behind(ma::detile_kernel<uint16_t>, grid, ma::kDtThreads, 0, st, src, dst, src_pitch, dst_pitch,
                            n_vec, s);
  }
  return e == cudaSuccess ? MA_OK : MA_ERR_CUDA;
}
