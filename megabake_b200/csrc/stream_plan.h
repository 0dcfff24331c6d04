// Host side of the streaming decode kernel: how projections are cut, how their units are dealt to the CTAs, and how
// shared memory is divided.  Pure functions of the configuration and the batch.
#pragma once
#include <algorithm>
#include <numeric>
#include <vector>

#include "stream_common.cuh"

namespace mk {

constexpr int kStreamPlans = 4;           // 8, 16 and 32 tokens (one, two and four MMA tiles), 8 tokens on fewer CTAs
constexpr int kStreamFew = 3;
constexpr int kStreamMaxGrid = 512;
constexpr int kStreamSmemLimit = 232448;  // 227 KiB

inline int stream_plan_tiles(int plan) { return plan == kStreamFew ? 1 : 1 << plan; }

// The kernel for a token class (up to 1, 4, 8, 16, 32 tokens); one translation unit per head size.  Two to four tokens are laid out as up
// to eight are, and only the squares of a norm are summed as one token's (see stream_squares).  With the operand spread over all lanes
// they were slower: a warp polls half lines of four tokens without a rest (us a step, two sequences 1.7B 835 -> 786, three at 777
// positions 886 -> 839, four at 1500 977 -> 915; 0.5B 633 -> 520; 135M 640 -> 476).
constexpr int kStreamClasses = 5;
constexpr int kStreamClassTokens[kStreamClasses] = {1, 8, 8, 16, 32};  // the layout's
const void* stream_kernel_64(int token_class);
const void* stream_kernel_128(int token_class);
inline int stream_class_of(int tokens) { return tokens <= 1 ? 0 : (tokens <= 4 ? 1 : (tokens <= 8 ? 2 : (tokens <= 16 ? 3 : 4))); }
inline const void* stream_kernel(int token_class, int head_dim) {
  return head_dim == 64 ? stream_kernel_64(token_class) : stream_kernel_128(token_class);
}

// Cut a reduction of `k` into the fewest slices of at most `copies` copies each.  (A slice that does not end at the row's end
// should be a multiple of four chunks: windows are dealt to eight warps.)
inline bool stream_cut(StreamPhase& ph, int copies) {
  const int chunks = ph.k / kChunkK;
  for (int nslice = 1; nslice <= chunks; ++nslice) {
    if (chunks % nslice) continue;
    ph.nslice = nslice;
    ph.cs = chunks / nslice;
    ph.ncopy = (ph.cs + kStreamKb - 1) / kStreamKb;
    if (ph.ncopy <= copies) return true;
  }
  return false;
}

// Rows per tile: what leaves the busiest CTA the fewest rows.  2048 rows in tiles of 16 are 128 tiles for 148 CTAs, 14 % of
// which would stand idle; in tiles of 14 they are 147.  A tile costs about two rows' time besides its rows.
inline void stream_rows(StreamPhase& ph, const int* matrices, int count, int grid) {
  int best_cost = 1 << 30;
  for (int rows = kStreamRows; rows >= 8; rows -= 2) {
    int tiles = 0;
    for (int i = 0; i < count; ++i) tiles += (matrices[i] + rows - 1) / rows;
    const int units = tiles * ph.nslice;
    const int cost = (units + grid - 1) / grid * (rows + 2);
    if (cost < best_cost) {
      best_cost = cost;
      ph.rows = rows;
      ph.ntiles = tiles;
    }
  }
}

inline bool stream_phases(const mk_config& c, int plan, int grid, StreamPhase* ph) {
  const int nt = stream_plan_tiles(plan), q_size = c.q_heads * c.head_dim, kv_size = c.kv_heads * c.head_dim;
  const int ks[kStreamPhases] = {c.hidden, q_size, c.hidden, c.intermediate, c.hidden};
  const int ns[kStreamPhases] = {q_size + 2 * kv_size, c.hidden, c.intermediate, c.hidden, c.vocab};
  bool ok = true;
  for (int i = 0; i < kStreamPhases; ++i) {
    StreamPhase& p = ph[i];
    p = StreamPhase{};
    p.k = ks[i];
    p.n = ns[i];
    // Up to eight tokens a long reduction is not cut: its operand is small enough to be read in parts by every CTA, which
    // saves a hand-over of partial sums.
    const bool cross = i == SP_O || i == SP_DOWN;
    const int fit = cross ? stream_fit(nt) : 2;  // (normalised: stream_fit_normalised, or less)
    ok = stream_cut(p, cross && nt == 1 ? 8 : fit) && (cross || p.nslice == 1) && ok;
    p.parts = (p.ncopy + fit - 1) / fit;
    const int qkv[3] = {q_size, kv_size, kv_size};
    stream_rows(p, i == SP_QKV ? qkv : &ns[i], i == SP_QKV ? 3 : 1, grid);
  }
  StreamPhase& qkv = ph[SP_QKV];
  qkv.row1 = q_size;
  qkv.row2 = q_size + kv_size;
  qkv.tile1 = (q_size + qkv.rows - 1) / qkv.rows;
  qkv.tile2 = qkv.tile1 + (kv_size + qkv.rows - 1) / qkv.rows;
  return ok;
}

// Fewer CTAs for up to eight sequences.  Every CTA polls for every hand-over and is in the way of the stores, so three quarters of the
// SMs go through a short layer faster than all of them, though a CTA's tiles get taller and a phase of few rounds longer: at
// 60 GB/s each they still take in what HBM delivers.  Where they lose is a round of tiles or of cache runs more:
//  - the projections of a layer take no more rounds of tiles, summed over the four, and the output head no more than a round per layer
//    of the model more (rounds of a layer, us a step of 16 layers at 60 positions on 148 and 112 CTAs, one / eight sequences: 135M shape
//    4 -> 4, 255 / 283 -> 249 / 264; hidden 1408 with 22 heads 9 -> 9, 402 / 440 -> 397 / 434; hidden 768 5 -> 6, 280 / 302 -> 281 / 315;
//    hidden 1152 6 -> 7, 333 / 359 -> 352 / 381; 1.7B 9 -> 13, 495 / 546 -> 544 / 591; two layers of the 135M shape, head 21 -> 28,
//    53 / 58 -> 55 / 60);
//  - there are four CTAs to every KV head of every sequence of the launch, else a long context is cut into too few runs (1000 to 16000
//    positions, KV heads x sequences: 15 442 -> 431, 341 -> 332, 24 518 -> 489, 298 -> 279; 32 365 -> 376, 594 -> 645; 48 753 -> 878;
//    128 363 -> 394).
//  - the hidden size is 512 at least: below it there is less to gain than a tile of the cache more costs (hidden 256, 8 layers, one
//    sequence at 1000 134 -> 138, four at 4000 153 -> 163).
// With more than eight sequences long contexts are a round of cache tiles longer (0.5B, 32 at 1900 904 -> 955).  A handle with a limit
// on its SMs uses what it was given.  Returns the number of CTAs, 0 where the shape has all of them in any case.
inline int stream_few_ctas(const mk_config& c, int sms) {
  const int few = (3 * sms / 4 + 7) / 8 * 8;
  if (c.sm_limit > 0 || c.hidden < 512 || few >= sms) return 0;
  StreamPhase less[kStreamPhases], all[kStreamPhases];
  stream_phases(c, kStreamFew, few, less);
  stream_phases(c, 0, sms, all);
  auto rounds = [](const StreamPhase& p, int grid) { return (p.ntiles * p.nslice + grid - 1) / grid; };
  int more = 0;
  for (int i = 0; i < SP_HEAD; ++i) more += rounds(less[i], few) - rounds(all[i], sms);
  return more <= 0 && rounds(less[SP_HEAD], few) - rounds(all[SP_HEAD], sms) <= c.layers ? few : 0;
}
inline bool stream_few_fits(const mk_config& c, int batch, int few) { return batch <= 8 && 4 * batch * c.kv_heads <= few; }
// The most CTAs, up to `ctas`, of which each has a unit of a layer's projections.  One that has none, of the output head alone, would
// wait for no layer, and takes what the first layers leave in the head's operand for the last one's.  (Left-over units go to the CTAs
// that have the least so far, see stream_deal_units: as many units as CTAs are enough.  Shapes of a hidden size of 128 and about; the
// 135M shape has 392.)
inline int stream_busy_ctas(const mk_config& c, int plan, int ctas) {
  StreamPhase ph[kStreamPhases];
  for (;;) {
    stream_phases(c, plan, ctas, ph);
    int units = 0;
    for (int i = 0; i < SP_HEAD; ++i) units += ph[i].ntiles * ph[i].nslice;
    if (units >= ctas) return ctas;
    ctas = units;
  }
}
// CTAs of a plan's launches, 0: no launch uses the plan.
inline int stream_grid(const mk_config& c, int plan, int sms) {
  if (plan == 0) return stream_busy_ctas(c, plan, sms);
  if (plan < kStreamFew) return c.max_tokens > (4 << plan) ? stream_busy_ctas(c, plan, sms) : 0;
  const int few = stream_few_ctas(c, sms);
  return stream_few_fits(c, 1, few) ? few : 0;
}
// The plan of a launch.
inline int stream_plan_of(const mk_config& c, int tokens, int few) {
  if (few > 0 && stream_few_fits(c, tokens, few)) return kStreamFew;
  return tokens <= 8 ? 0 : (tokens <= 16 ? 1 : 2);
}

// Hidden sizes up to 2048: an operand of 2048 columns fits a warp's registers at 32 tokens (two copies of a slice), and only
// such shapes have been measured and tested here.  Wider ones would fit up to 16 tokens and are left on the tensor engine;
// that is not a limit of the hardware.  What to expect of a change: on the 8B shape's 32 layers this kernel, the tensor
// engine and an eager evaluation are 2.0 to 2.2 % apart, each from each, as correct bf16 evaluations of that depth are.
inline bool stream_shape_ok(const mk_config& c) {
  if (c.tp_size > 1 || c.hidden > 2048) return false;
  StreamPhase ph[kStreamPhases];
  for (int i = 0; i < kStreamFew; ++i)  // (the other plan's reductions are cut as the first one's)
    if (stream_grid(c, i, 148) > 0 && !stream_phases(c, i, 148, ph)) return false;
  return true;
}

// Every CTA's units of each phase, as ranges: table[phase][cta], table[phase][grid] = count.  Every phase is dealt evenly
// (an SM takes in at most about 60 GB/s, so a CTA with more units than the rest ends a phase late); the units that
// are left over go to the CTAs with the fewest bytes so far.
inline void stream_deal_units(const StreamPhase* ph, int grid, int* table) {
  std::vector<long long> load(grid, 0);
  std::vector<int> order(grid), extra(grid);
  for (int kind = 0; kind < kStreamPhases; ++kind) {
    const int units = ph[kind].ntiles * ph[kind].nslice;
    const long long cost = static_cast<long long>(ph[kind].rows) * ph[kind].cs * (kind == SP_GU ? 2 : 1);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return load[a] < load[b]; });
    std::fill(extra.begin(), extra.end(), 0);
    for (int i = 0; i < units % grid; ++i) extra[order[i]] = 1;
    int* row = table + kind * (grid + 1);
    row[0] = 0;
    for (int i = 0; i < grid; ++i) {
      row[i + 1] = row[i] + units / grid + extra[i];
      load[i] += cost * (units / grid + extra[i]);
    }
  }
}

// Adjacent KV heads of a cache tile: as many as leave about one (sequence, head group) per two CTAs.  Wider tiles read
// longer runs of a cache row (DRAM pages) and leave a warp to itself; fewer groups mean more parts to add up.
inline int stream_heads_per_tile(const mk_config& c, int batch) {
  const int gs = c.q_heads / c.kv_heads;
  int hpu = 1;
  while (2 * hpu * gs <= 8 && c.kv_heads % (2 * hpu) == 0 && batch * (c.kv_heads / (2 * hpu)) >= 64) hpu *= 2;
  return hpu;
}

// Attention: one row per warp and query head of its KV head, and behind them eight warps' statistics of eight query heads.
// One token: the normalised operand on its way to the fragments (16 windows of 64 bytes per warp).
inline int stream_scratch_bytes(const mk_config& c, int batch) {
  return std::max(batch == 1 ? 8192 : 4096, 8 * (c.q_heads / c.kv_heads) * (c.head_dim + 2) * 4 + 512);
}
// Two buffers of partial sums up to eight tokens.  With 16, one and a block barrier more per tile leave room for a sixth slot (1.7B shape,
// sixteen sequences at 200 positions 1088 -> 1068 us, at 1024 1441 -> 1431, fourteen of different lengths 1389 -> 1344); with 32
// there is no room for it either way.
inline int stream_psum_bytes(int batch) {
  return std::max(1024, (batch <= 8 ? 2 : 1) * kStreamWarps * 2 * kStreamClassTokens[stream_class_of(batch)] * kStreamPartPitch * 4);
}
// The ring takes as many slots as fit.
inline void stream_divide(KParams& p, int scratch, int batch) {
  p.stream_scratch_bytes = scratch;
  p.stream_slots = std::min(kStreamMaxSlots, (kStreamSmemLimit - 1024 - kStreamMiscBytes - scratch - stream_psum_bytes(batch)) / kStreamSlotBytes);
}
inline int stream_smem_bytes(const KParams& p) {
  return 1024 + p.stream_slots * kStreamSlotBytes + kStreamMiscBytes + p.stream_scratch_bytes + stream_psum_bytes(p.m);
}

}  // namespace mk
