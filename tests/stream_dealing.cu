// Host build of the streaming decode kernel's dealing of cached positions, for test_stream_dealing.py: walks one layer the
// way the kernel's producer and its helper thread do and checks what the consumers rely on.  Beside it its quotient.
#include <cmath>
#include <cstring>
#include <vector>

#include "../megabake_b200/csrc/stream_attention.cuh"
#include "../megabake_b200/csrc/stream_plan.h"

using namespace mk;

static mk_config shape(const int* s) {  // hidden, query heads, KV heads, head size, intermediate, vocabulary, layers, SM limit
  mk_config c{};
  c.hidden = s[0];
  c.q_heads = s[1];
  c.kv_heads = s[2];
  c.head_dim = s[3];
  c.intermediate = s[4];
  c.vocab = s[5];
  c.layers = s[6];
  c.sm_limit = s[7];
  c.max_tokens = 32;
  return c;
}
// CTAs of a launch of `batch` sequences.
extern "C" int grid_of(const int* s, int batch, int sms) {
  const mk_config c = shape(s);
  const int few = stream_grid(c, kStreamFew, sms);
  return stream_grid(c, stream_plan_of(c, batch, few), sms);
}
// Units of a phase's busiest CTA.
extern "C" int rounds_of(const int* s, int kind, int grid) {
  StreamPhase ph[kStreamPhases];
  stream_phases(shape(s), 0, grid, ph);
  std::vector<int> table(kStreamPhases * (grid + 1));
  stream_deal_units(ph, grid, table.data());
  int most = 0;
  for (int i = 0; i < grid; ++i) most = std::max(most, table[kind * (grid + 1) + i + 1] - table[kind * (grid + 1) + i]);
  return most;
}

// Returns 0, or the number of the first rule that is broken; `longest` and `lists`: the most parts and lists of a CTA.
extern "C" int check_dealing(int grid, int batch, int q_heads, int kv_heads, int head_dim, int ragged, const int* len, int* longest, int* lists) {
  mk_config c{};
  c.q_heads = q_heads;
  c.kv_heads = kv_heads;
  c.head_dim = head_dim;
  static KParams p;
  p = KParams{};
  p.batch = batch;
  p.kv_heads = kv_heads;
  p.ragged = ragged;
  p.stream_hpu = stream_heads_per_tile(c, batch);
  p.stream_tile_keys = kStreamSlotBytes / (head_dim * 2 * p.stream_hpu);
  const int groups = kv_heads / p.stream_hpu;
  struct Group {
    int tiles = 0, parts = 0, nseg = 0;
    std::vector<int> seen;  // by part number
  };
  std::vector<Group> all(static_cast<size_t>(batch) * groups);
  *longest = *lists = 0;
  for (int cta = 0; cta < grid; ++cta) {
    const StreamTiles s = stream_tiles(p, len, cta, grid);
    int at = s.first, streamed = s.first, parts = 0, n_lists = 0;
    do {
      StreamSegment list[kStreamSegments + 1];
      list[kStreamSegments].nt = -12345;
      const int n = stream_next_parts(s, cta, at, list);
      if (n > kStreamSegments || list[kStreamSegments].nt != -12345) return 1;
      if (n == 0 && at < s.last) return 2;
      for (int i = 0; i < n; ++i) {
        const StreamSegment& g = list[i];
        const StreamSegment copied = stream_segment(s, streamed, cta);  // the producer's own walk
        if (copied.b != g.b || copied.group != g.group || copied.t0 != g.t0 || copied.t1 != g.t1) return 3;
        streamed += copied.t1 - copied.t0;
        if (g.b < 0 || g.b >= batch || g.group < 0 || g.group >= groups) return 4;
        const int length = len[ragged ? g.b : 0];
        if (g.len != length || g.nt != length / p.stream_tile_keys + 1) return 5;
        if (g.t0 < 0 || g.t1 <= g.t0 || g.t1 > g.nt) return 6;
        if (g.seg < 0 || g.seg >= g.nseg || g.nseg > kStreamMaxSegments) return 7;
        Group& of = all[static_cast<size_t>(g.b) * groups + g.group];
        if (of.parts > 0 && of.nseg != g.nseg) return 8;
        of.nseg = g.nseg;
        of.parts += 1;
        of.tiles += g.t1 - g.t0;
        of.seen.resize(g.nseg);
        if (of.seen[g.seg]++) return 9;
      }
      parts += n;
      n_lists += 1;
    } while (at < s.last);
    if (streamed != s.last && s.first < s.last) return 10;
    if (parts > *longest) *longest = parts;
    if (n_lists > *lists) *lists = n_lists;
  }
  for (int b = 0; b < batch; ++b)
    for (int g = 0; g < groups; ++g) {
      const Group& of = all[static_cast<size_t>(b) * groups + g];
      if (of.tiles != len[ragged ? b : 0] / p.stream_tile_keys + 1) return 11;  // every position exactly once
      if (of.parts != of.nseg) return 12;                                        // every part is handed in
    }
  return 0;
}

// Numerators of `count` random mantissas with exponents low to high over denominators 1 to 2^14: quotients that are not the
// division's, and those that are not after the rounding to bf16.
extern "C" void quotients(int low, int high, int count, long long* differ, long long* differ_rounded) {
  unsigned long long state = 88172645463325252ull;
  *differ = *differ_rounded = 0;
  for (int i = 0; i < count; ++i) {
    state ^= state << 13, state ^= state >> 7, state ^= state << 17;
    const float a = std::ldexp(1.f + static_cast<float>((state >> 20) & 0x7FFFFF) / 8388608.f, low + static_cast<int>(state % (high - low + 1)));
    const float b = i % 2 ? 1.f + static_cast<float>((state >> 43) % 65536) * 0.25f
                          : std::ldexp(1.f + static_cast<float>((state >> 41) & 0x7FFFFF) / 8388608.f, static_cast<int>((state >> 8) % 14));
    const float mine = stream_quotient(a, b, 1.f / b), exact = a / b;
    *differ += mine != exact;
    *differ_rounded += __bfloat162float(__float2bfloat16_rn(mine)) != __bfloat162float(__float2bfloat16_rn(exact));
  }
}
extern "C" float quotient(float a, float b) { return stream_quotient(a, b, 1.f / b); }
