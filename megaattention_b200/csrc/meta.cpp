// Host side of one step's varlen metadata: the row-tile schedule of a batch (the arithmetic of
// metadata/row_desc.py), the attention claim order (runtime/workspace.py: claim_order) and the
// active counts, written where the caller wants them.  In numpy these took 95 us of a step's
// host time - more than the whole launch of a small layer; here a few.
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <vector>

#include "../../include/megaattn_b200.h"
#include "kparams.h"

extern "C" int ma_row_desc(const int64_t* cu_q, const int64_t* cu_k, int32_t num_batch,
                           int32_t max_row_tiles, int32_t* cu_q_out, int32_t* cu_k_out,
                           int32_t* cu_m_blocks, int32_t* batch_idx, int32_t* m_block) {
  if (!cu_q || !cu_k || num_batch < 1 || !cu_q_out || !cu_k_out || !cu_m_blocks || !batch_idx ||
      !m_block)
    return MA_ERR_INVALID;
  if (cu_q[0] != 0 || cu_k[0] != 0) return MA_ERR_INVALID;
  int64_t tiles = 0;
  cu_q_out[0] = cu_k_out[0] = cu_m_blocks[0] = 0;
  for (int b = 0; b < num_batch; ++b) {
    const int64_t lq = cu_q[b + 1] - cu_q[b], lk = cu_k[b + 1] - cu_k[b];
    if (lq <= 0 || lk < lq) return MA_ERR_INVALID;
    if (cu_q[b + 1] > 0x7fffffff || lk > 0x7fffffff) return MA_ERR_CAPACITY;
    const int64_t n = (lq + 127) / 128;
    if (tiles + n > max_row_tiles) return MA_ERR_CAPACITY;
    for (int64_t j = 0; j < n; ++j) {
      batch_idx[tiles + j] = b;
      m_block[tiles + j] = static_cast<int32_t>(j);
    }
    tiles += n;
    cu_q_out[b + 1] = static_cast<int32_t>(cu_q[b + 1]);
    // (paged sequences share pages: their lengths may sum past 2^31, and only differences of
    // this sum are used)
    cu_k_out[b + 1] = static_cast<int32_t>(static_cast<uint32_t>(cu_k[b + 1]));
    cu_m_blocks[b + 1] = static_cast<int32_t>(tiles);
  }
  return static_cast<int>(tiles);
}

extern "C" int ma_stage_meta(const ma_stage_meta_args* a) {
  if (!a || !a->cu_q || !a->cu_k || !a->batch_idx || !a->m_block || !a->staging)
    return MA_ERR_INVALID;
  const int R = a->num_row_tiles, B = a->num_batch;
  if (R < 1 || B < 1 || a->num_super_groups < 1 || a->tp_size < 1 || a->hidden < 1)
    return MA_ERR_INVALID;
  int32_t* order = a->staging + a->off_order;
  try {
    // key blocks every row tile's attention visits
    std::vector<int32_t> nblk(R);
    int64_t sum = 0;
    int32_t most = 0;
    for (int t = 0; t < R; ++t) {
      const int b = a->batch_idx[t];
      if (b < 0 || b >= B) return MA_ERR_INVALID;
      const int64_t lq = static_cast<int64_t>(a->cu_q[b + 1]) - a->cu_q[b];
      const int64_t lk = static_cast<int32_t>(static_cast<uint32_t>(a->cu_k[b + 1]) -
                                              static_cast<uint32_t>(a->cu_k[b]));
      const int64_t last = (static_cast<int64_t>(a->m_block[t]) + 1) * 128 + (lk - lq);
      const int64_t n = std::min((lk + 127) / 128, (last + 127) / 128);
      if (n < 0) return MA_ERR_INVALID;
      nblk[t] = static_cast<int32_t>(n);
      sum += n;
      most = std::max(most, nblk[t]);
    }
    int prime = a->prime;
    if (a->auto_prime) {          // interleaved below 2.0, fa_prime_tiles_b200's switch point
      const int64_t tiles = static_cast<int64_t>(R) * ((a->hidden + 127) / 128);
      prime = static_cast<double>(2 * sum) / static_cast<double>(tiles) < 2.0 ? -1 : 0;
    }
    // longest first, stable: counting sort on the number of blocks
    std::vector<int32_t> at(static_cast<size_t>(most) + 2, 0), sorted(R);
    for (int t = 0; t < R; ++t) ++at[most - nblk[t] + 1];
    for (int i = 1; i <= most + 1; ++i) at[i] += at[i - 1];
    for (int t = 0; t < R; ++t) sorted[at[most - nblk[t]]++] = t;
    if (prime < 0) {              // longest, shortest, second longest, second shortest, ...
      const int half = (R + 1) / 2;
      for (int i = 0; i < half; ++i) order[2 * i] = sorted[i];
      for (int i = half; i < R; ++i) order[2 * (R - 1 - i) + 1] = sorted[i];
    } else {                      // the `prime` shortest to the front
      const int p = std::min(prime, R);
      for (int i = 0; i < p; ++i) order[i] = sorted[R - 1 - i];
      for (int i = p; i < R; ++i) order[i] = sorted[i - p];
    }
  } catch (const std::bad_alloc&) {
    return MA_ERR_CAPACITY;
  }
  memcpy(a->staging + a->off_cu_q, a->cu_q, sizeof(int32_t) * (B + 1));
  memcpy(a->staging + a->off_cu_k, a->cu_k, sizeof(int32_t) * (B + 1));
  memcpy(a->staging + a->off_batch_idx, a->batch_idx, sizeof(int32_t) * R);
  memcpy(a->staging + a->off_m_block, a->m_block, sizeof(int32_t) * R);
  int32_t* actv = a->staging + a->off_actv;
  const int64_t total = static_cast<int64_t>(R) * a->num_super_groups, tp = a->tp_size;
  const int64_t slots = (total + tp - 1) / tp;
  const int64_t owned = std::max<int64_t>(total - a->rank, 0);
  actv[0] = R * a->H_local;
  actv[1] = static_cast<int32_t>(total);
  actv[2] = R;
  actv[3] = static_cast<int32_t>(slots);
  actv[4] = static_cast<int32_t>((slots + 63) / 64);
  actv[5] = static_cast<int32_t>((owned + tp - 1) / tp);
  return MA_OK;
}

extern "C" int ma_stage_tasks(const ma_stage_tasks_args* a) {
  if (!a || a->off_tasks < 0 || (a->off_tasks & 3)) return MA_ERR_INVALID;
  const ma_stage_meta_args& m = a->meta;
  const int rc = ma_stage_meta(&m);
  if (rc != MA_OK) return rc;
  if (m.num_row_tiles > a->max_tasks) return MA_ERR_CAPACITY;
  const int32_t* order = m.staging + m.off_order;
  int32_t* head = m.staging + a->off_tasks;
  head[0] = m.num_row_tiles;
  head[1] = head[2] = head[3] = 0;
  for (int i = 0; i < m.num_row_tiles; ++i) {
    int32_t* r = head + 4 + i * ma::kTaskWords;
    const int t = order[i], b = m.batch_idx[t];
    r[0] = t;
    r[1] = b;
    r[2] = m.m_block[t];
    r[3] = m.cu_q[b];
    r[4] = m.cu_q[b + 1] - m.cu_q[b];
    r[5] = m.cu_k[b];
    r[6] = static_cast<int32_t>(static_cast<uint32_t>(m.cu_k[b + 1]) - static_cast<uint32_t>(m.cu_k[b]));
    r[7] = 0;
  }
  return MA_OK;
}
