// Host build of the streaming decode kernel's units, for test_stream_order.py.
#include <algorithm>
#include <vector>

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

extern "C" int has_plan(const int* s) { return stream_shape_ok(shape(s)); }

// CTAs of a launch of `batch` sequences, and how many of them have units, but none of a layer's projections.
extern "C" int ctas_without_a_layer(const int* s, int batch, int sms, int* ctas) {
  const mk_config c = shape(s);
  const int plan = stream_plan_of(c, batch, stream_grid(c, kStreamFew, sms)), grid = stream_grid(c, plan, sms);
  StreamPhase ph[kStreamPhases];
  stream_phases(c, plan, grid, ph);
  std::vector<int> table(kStreamPhases * (grid + 1));
  stream_deal_units(ph, grid, table.data());
  int idle = 0;
  for (int cta = 0; cta < grid; ++cta) {
    auto units = [&](int kind) { return table[kind * (grid + 1) + cta + 1] - table[kind * (grid + 1) + cta]; };
    idle += units(SP_HEAD) > 0 && units(SP_QKV) + units(SP_O) + units(SP_GU) + units(SP_DOWN) == 0;
  }
  *ctas = grid;
  return idle;
}
