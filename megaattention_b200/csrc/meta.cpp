// Host side of one step's varlen metadata: the row-tile schedule of a batch (the arithmetic of
// metadata/row_desc.py), the attention claim order (runtime/workspace.py: claim_order) and the
// active counts, written where the caller wants them.  In numpy these took 95 us of a step's
// host time - more than the whole launch of a small layer; here a few.
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <functional>
#include <new>
#include <vector>

#include "../../include/megaattn_b200.h"
#include "kparams.h"

namespace {

// Key blocks that row tile t's attention visits, of the host's lengths (< 0: bad lengths).
int64_t key_blocks(const ma_stage_meta_args& a, int t) {
  const int b = a.batch_idx[t];
  const int64_t lq = static_cast<int64_t>(a.cu_q[b + 1]) - a.cu_q[b];
  const int64_t lk = static_cast<int32_t>(static_cast<uint32_t>(a.cu_k[b + 1]) -
                                          static_cast<uint32_t>(a.cu_k[b]));
  const int64_t last = (static_cast<int64_t>(a.m_block[t]) + 1) * 128 + (lk - lq);
  return std::min((lk + 127) / 128, (last + 127) / 128);
}

// The claim order asked for (ma_stage_meta), by default interleaved below a work ratio of 2.0,
// fa_prime_tiles_b200's switch point.
int claim_prime(const ma_stage_meta_args& a, int64_t blocks) {
  if (!a.auto_prime) return a.prime;
  const int64_t tiles = static_cast<int64_t>(a.num_row_tiles) * ((a.hidden + 127) / 128);
  return static_cast<double>(2 * blocks) / static_cast<double>(tiles) < 2.0 ? -1 : 0;
}

// Claim order of things sorted longest first.
void arrange(const int32_t* sorted, int n, int prime, int32_t* order) {
  if (prime < 0) {              // longest, shortest, second longest, second shortest, ...
    const int half = (n + 1) / 2;
    for (int i = 0; i < half; ++i) order[2 * i] = sorted[i];
    for (int i = half; i < n; ++i) order[2 * (n - 1 - i) + 1] = sorted[i];
  } else {                      // the `prime` shortest to the front
    const int p = std::min(prime, n);
    for (int i = 0; i < p; ++i) order[i] = sorted[n - 1 - i];
    for (int i = p; i < n; ++i) order[i] = sorted[i - p];
  }
}

// Splitting of row tiles' keys.  A task's key blocks are a serial chain, 2 us each, and with few or
// uneven tasks the longest one is the launch while other CTAs have nothing to do.  Lengths here are
// in key blocks: a task costs two more than it has (its first loads, the epilogue), a part another
// one for putting its sums down, reading a head's parts back half a one per part, and the O_proj of
// a row tile's 128 columns a fifth of one per head.  Launches in us as 1 / 2 / 3 / 4 / 6 / 8 parts of the
// longest: 64 tokens behind 4000 keys, 8 heads 103 / 85 / 79 / 75 / 75 / 77; one token behind 15000, 4
// heads 243 / 152 / 122 / 106 / 93 / 89; 100 and 300 behind 1500 and 2500 81 / 77 / 75 / 69 / 73 / 75;
// 2000 behind 15871 270 / 179 / 212 / 185; 12 short turns on up to 5217 keys 122 / 95 / 89 / 89 / 97 / 101.
constexpr int kMinPart = 5;
constexpr int kTaskCost = 2, kPartCost = 1;
constexpr double kJoinCost = 0.5, kOprojCost = 0.2, kWorthIt = 0.9;

struct Unit { int32_t tile, split, len; };    // split: as in the task table
struct Group { int32_t at, n; };              // n tasks of one cost, or n row tiles of one length

// What the launch's attention takes, claimed longest first (costs come in that order) by `lanes`
// groups of CTAs (one CTA of a group per task of a row tile), or something above `limit` where it takes
// longer than that.  free_at: lanes by the time they are free at.
int32_t makespan(const std::vector<Group>& costs, int lanes, double limit, std::vector<int32_t>& free_at) {
  int64_t sum = 0;
  for (const Group& c : costs) sum += static_cast<int64_t>(c.at) * c.n;
  free_at.assign(static_cast<size_t>(sum / lanes) + costs.front().at + 2, 0);
  free_at[0] = lanes;
  int32_t now = 0, most = 0;
  for (const Group& c : costs) {
    for (int32_t left = c.n; left > 0;) {
      while (free_at[now] == 0) ++now;
      const int32_t n = std::min(left, free_at[now]);
      left -= n;
      free_at[now] -= n;
      free_at[now + c.at] += n;
      most = std::max(most, now + c.at);
    }
    if (most > limit) return most;
  }
  return most;
}

// Parts of every row tile, from splits of the longest into 2, 3, ... parts and of the others into
// parts of that length; false: none is worth it.  A launch ends with its attention, or once all of
// its work is done, O_proj's too (CTAs without attention have that to do: 4500 tokens of one prompt,
// 4096 columns, attention alone would be shorter in two parts, the launch is 118 us and 119).
// The host does this in every call, a paged call's behind its wait (one head, prefixed batches: 31 us when
// every split was simulated task by task, now 4; 8 heads 8 and 3).  So the splits are taken in the
// order of what their longest part and their work come to at least, up to the one that cannot be
// better any more, and row tiles of one length are one thing.
bool choose_parts(const std::vector<int32_t>& nblk, int H, int num_out, int ctas, int slots,
                  std::vector<int32_t>& parts) {
  const int R = static_cast<int>(nblk.size()), per_tile = (H + 1) / 2;
  const int lanes = std::max(1, ctas / per_tile);
  const int32_t most = *std::max_element(nblk.begin(), nblk.end());
  // (three tasks per CTA fill each other's gaps)
  if (slots < 2 || most < 2 * kMinPart || static_cast<int64_t>(R) * per_tile > 3 * ctas) return false;
  const double oproj = kOprojCost * R * num_out * H / ctas;
  int64_t whole = 0;
  for (int32_t n : nblk) whole += n + kTaskCost;
  if (most + kTaskCost <= static_cast<double>(whole) / lanes + oproj) return false;

  std::vector<int32_t> sorted(nblk);
  std::sort(sorted.begin(), sorted.end(), std::greater<int32_t>());
  std::vector<Group> tiles, costs;              // tiles: longest first
  std::vector<int32_t> free_at;
  for (int32_t n : sorted) {
    if (n == 0) break;                          // (nothing to see: no part at all)
    if (tiles.empty() || tiles.back().at != n) tiles.push_back({n, 0});
    ++tiles.back().n;
  }
  costs = tiles;
  for (Group& c : costs) c.at += kTaskCost;
  const int empty = static_cast<int>(std::count(sorted.begin(), sorted.end(), 0));
  if (empty) costs.push_back({kTaskCost, empty});
  const double all = static_cast<double>(whole) / lanes + oproj;
  double best = kWorthIt * std::max<double>(makespan(costs, lanes, HUGE_VAL, free_at), all);

  whole -= static_cast<int64_t>(kTaskCost) * empty;
  struct Split { double least, mean; int k; int32_t len; } splits[ma::kMaxParts];
  int num = 0, best_k = 0;
  for (int k = 2; k <= ma::kMaxParts && most >= k * kMinPart; ++k) {
    const int32_t len = (most + k - 1) / k;
    int64_t used = 0, sum = whole;
    int32_t longest = 0;
    for (const Group& t : tiles) {
      if (t.at <= len) {                        // (this one and the shorter ones stay whole)
        longest = std::max(longest, t.at + kTaskCost);
        break;
      }
      const int32_t m = (t.at + len - 1) / len;
      used += static_cast<int64_t>(m) * t.n;
      sum += static_cast<int64_t>((m - 1) * kTaskCost + m * kPartCost) * t.n;
      longest = std::max(longest, (t.at + m - 1) / m + kTaskCost + kPartCost);
    }
    if (used > slots) break;
    const double mean = static_cast<double>(sum) / lanes + oproj;
    splits[num++] = {std::max<double>(longest, mean) + k * kJoinCost, mean, k, len};
  }
  std::sort(splits, splits + num, [](const Split& x, const Split& y) {
    return x.least < y.least || (x.least == y.least && x.k < y.k);
  });
  int32_t best_len = 0;
  for (int i = 0; i < num && splits[i].least <= best; ++i) {
    const Split& sp = splits[i];
    costs.clear();
    for (const Group& t : tiles) {
      const int32_t m = (t.at + sp.len - 1) / sp.len, cost = t.at / m + kTaskCost + (m > 1 ? kPartCost : 0);
      const int32_t longer = t.at % m;
      if (longer) costs.push_back({cost + 1, longer * t.n});
      costs.push_back({cost, (m - longer) * t.n});
    }
    std::sort(costs.begin(), costs.end(), [](const Group& x, const Group& y) { return x.at > y.at; });
    const double join = sp.k * kJoinCost;
    const double t = std::max<double>(makespan(costs, lanes, best - join, free_at), sp.mean) + join;
    if (t < best || (t == best && best_k && sp.k < best_k)) { best = t; best_k = sp.k; best_len = sp.len; }
  }
  if (best_len == 0) return false;
  for (int t = 0; t < R; ++t) parts[t] = std::max(1, (nblk[t] + best_len - 1) / best_len);
  return true;
}

}  // namespace

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
      const int64_t n = key_blocks(*a, t);
      if (n < 0) return MA_ERR_INVALID;
      nblk[t] = static_cast<int32_t>(n);
      sum += n;
      most = std::max(most, nblk[t]);
    }
    // longest first, stable: counting sort on the number of blocks
    std::vector<int32_t> at(static_cast<size_t>(most) + 2, 0), sorted(R);
    for (int t = 0; t < R; ++t) ++at[most - nblk[t] + 1];
    for (int i = 1; i <= most + 1; ++i) at[i] += at[i - 1];
    for (int t = 0; t < R; ++t) sorted[at[most - nblk[t]]++] = t;
    arrange(sorted.data(), R, claim_prime(*a, sum), order);
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
  const int R = m.num_row_tiles;
  const int32_t* order = m.staging + m.off_order;
  int32_t* head = m.staging + a->off_tasks;
  // positions of the table: {row tile, split}
  std::vector<Unit> units;
  try {
    std::vector<int32_t> nblk(R), parts(R, 1);
    for (int t = 0; t < R; ++t) nblk[t] = static_cast<int32_t>(key_blocks(m, t));
    const int slots = std::min({a->split_slots, a->max_tasks - R, 0xffff});
    if (m.H_local >= 1 && a->num_ctas >= 1 && choose_parts(nblk, m.H_local, (m.hidden + 127) / 128, a->num_ctas, slots, parts)) {
      int64_t sum = 0;
      std::vector<Unit> all;
      int slot = 0;
      for (int t = 0; t < R; ++t) {
        const int32_t n = nblk[t], k = parts[t];
        sum += n;
        for (int i = 0; i < k; ++i)
          all.push_back({t, k > 1 ? k | i << 8 | static_cast<int32_t>(static_cast<uint32_t>(slot) << 16) : 0,
                         static_cast<int32_t>(static_cast<int64_t>(n) * (i + 1) / k - static_cast<int64_t>(n) * i / k)});
        if (k > 1) slot += k;
      }
      std::stable_sort(all.begin(), all.end(), [](const Unit& x, const Unit& y) { return x.len > y.len; });
      const int N = static_cast<int>(all.size());
      std::vector<int32_t> sorted(N), at(N);
      for (int i = 0; i < N; ++i) sorted[i] = i;
      arrange(sorted.data(), N, claim_prime(m, sum), at.data());
      for (int i = 0; i < N; ++i) units.push_back(all[at[i]]);
    } else {
      for (int i = 0; i < R; ++i) units.push_back({order[i], 0, 0});
    }
  } catch (const std::bad_alloc&) {
    return MA_ERR_CAPACITY;
  }
  head[0] = static_cast<int32_t>(units.size());
  head[1] = head[2] = head[3] = 0;
  for (int i = 0; i < head[0]; ++i) {
    int32_t* r = head + 4 + i * ma::kTaskWords;
    const int t = units[i].tile, b = m.batch_idx[t];
    r[0] = t;
    r[1] = b;
    r[2] = m.m_block[t];
    r[3] = m.cu_q[b];
    r[4] = m.cu_q[b + 1] - m.cu_q[b];
    r[5] = m.cu_k[b];
    r[6] = static_cast<int32_t>(static_cast<uint32_t>(m.cu_k[b + 1]) - static_cast<uint32_t>(m.cu_k[b]));
    r[7] = units[i].split;
  }
  return MA_OK;
}
