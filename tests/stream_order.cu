// Host build of the streaming decode kernel's units, for test_stream_order.py: who has one, and a walk through the layers that follows what
// each CTA knows of the others when it looks for a word that two layers before was reset by one of them.
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

namespace {
// What a CTA does in a layer, in order: q/k/v, attention parts, their sums, o_proj, its cut tiles' sums, gate and up, down_proj, its sums.
enum { QKV, PARTS, ATT, O, O_SUM, GU, DOWN, DOWN_SUM, kSteps };
int step_of(int kind) { return kind == SP_QKV ? QKV : (kind == SP_O ? O : (kind == SP_GU ? GU : (kind == SP_DOWN ? DOWN : kSteps))); }

using Known = std::vector<int>;  // by CTA: the last of its results that something known depends on, layer * kSteps + step
void learn(Known& to, const Known& of) {
  if (to.size() < of.size()) to.resize(of.size(), -1);
  for (size_t i = 0; i < of.size(); ++i) to[i] = std::max(to[i], of[i]);
}
}  // namespace

// `met`: the projection ahead of whose first result a layer's fence is met (SP_HEAD: behind all of them).  Returns how many looks at
// another CTA's word find one whose reset nothing known comes behind; the first of them in `where`.
extern "C" int looks_too_early(const int* s, int batch, int sms, int ragged, const int* len, int met, int* where) {
  const mk_config c = shape(s);
  const int plan = stream_plan_of(c, batch, stream_grid(c, kStreamFew, sms)), grid = stream_grid(c, plan, sms);
  StreamPhase ph[kStreamPhases];
  stream_phases(c, plan, grid, ph);
  std::vector<int> table(kStreamPhases * (grid + 1));
  stream_deal_units(ph, grid, table.data());
  auto owner = [&](int kind, int unit) {  // of a unit
    const int* row = table.data() + kind * (grid + 1);
    return static_cast<int>(std::upper_bound(row, row + grid + 1, unit) - row) - 1;
  };
  auto adds = [&](int kind, int tile) {  // who adds up a cut tile: the kernel's shares [tiles * cta / grid, tiles * (cta + 1) / grid)
    int cta = static_cast<int>(static_cast<long long>(tile) * grid / ph[kind].ntiles);
    while (static_cast<long long>(ph[kind].ntiles) * (cta + 1) / grid <= tile) ++cta;
    return cta;
  };
  auto writer = [&](int kind, int tile) { return ph[kind].nslice > 1 ? adds(kind, tile) : owner(kind, tile); };
  auto final_step = [&](int kind) { return step_of(kind) + (ph[kind].nslice > 1 ? 1 : 0); };

  KParams p{};
  p.batch = batch;
  p.kv_heads = c.kv_heads;
  p.ragged = ragged;
  p.stream_hpu = stream_heads_per_tile(c, batch);
  p.stream_tile_keys = kStreamSlotBytes / (c.head_dim * 2 * p.stream_hpu);
  const int gs = c.q_heads / c.kv_heads, groups = c.kv_heads / p.stream_hpu, heads = gs * p.stream_hpu;
  struct Part {
    int b, group, seg, nseg;
    bool last;
  };
  std::vector<std::vector<Part>> parts(grid);
  std::vector<int> first_of(batch * groups, 0);  // the CTA that adds up a (sequence, head group)
  for (int cta = 0; cta < grid; ++cta) {
    const StreamTiles t = stream_tiles(p, len, cta, grid);
    for (int at = t.first; at < t.last;) {
      const StreamSegment g = stream_segment(t, at, cta);
      parts[cta].push_back({g.b, g.group, g.seg, g.nseg, g.t1 == g.nt});
      if (g.seg == 0) first_of[g.b * groups + g.group] = cta;
      at += g.t1 - g.t0;
    }
  }

  const int layers = 8;
  std::vector<Known> now(grid, Known(grid, -1));  // of each CTA
  std::vector<Known> said[kSteps];                // with the results of this layer, and of the layer before's down_proj
  for (auto& all : said) all.assign(grid, Known());
  std::vector<Known> sums(batch * groups), before = said[0];
  std::vector<std::vector<Known>> records(batch * groups, std::vector<Known>(kStreamMaxSegments));
  int early = 0;
  // CTA `reader`, knowing `known`, looks for a word that `by` writes in step `step` of layer `layer`.
  auto look = [&](const Known& known, int reader, int by, int layer, int step) {
    if (layer < 3 || by == reader) return;
    const int reset = layer - 2;  // what has been there since layer - 3 was reset then
    const bool ahead = step < DOWN;  // of that layer's fence
    const int fence = ahead ? reset : reset + 1;
    const int covered = met == SP_DOWN ? fence * kSteps + DOWN : (fence + 1) * kSteps;  // results from here on come behind the fence
    if (known[by] < covered && early++ == 0) where[0] = reader, where[1] = by, where[2] = layer, where[3] = step;
  };
  auto speak = [&](int cta, int layer, int step) {
    now[cta][cta] = layer * kSteps + step;
    said[step][cta] = now[cta];
  };
  for (int layer = 0; layer <= layers; ++layer) {
    const bool head = layer == layers;
    auto units = [&](int kind, int cta) { return table[kind * (grid + 1) + cta + 1] - table[kind * (grid + 1) + cta]; };
    // the whole residual stream that a projection left, as `reader` reads it
    auto stream = [&](int reader, int kind, int of, const std::vector<Known>& from) {
      const Known had = now[reader];
      for (int tile = 0; tile < ph[kind].ntiles; ++tile) {
        const int by = writer(kind, tile);
        look(had, reader, by, of, final_step(kind));
        learn(now[reader], from[by]);
      }
    };
    before = said[final_step(SP_DOWN)];
    for (int cta = 0; cta < grid; ++cta)
      if (units(head ? SP_HEAD : SP_QKV, cta) > 0) {
        if (layer > 0) stream(cta, SP_DOWN, layer - 1, before);
        if (!head) speak(cta, layer, QKV);
      }
    if (head) break;
    // attention: the rows of q, k and v of a part's heads
    const StreamPhase& qkv = ph[SP_QKV];
    for (int cta = 0; cta < grid; ++cta)
      for (const Part& part : parts[cta]) {
        const Known had = now[cta];
        auto rows = [&](int tile0, int row0, int count) {
          for (int tile = tile0 + row0 / qkv.rows; tile <= tile0 + (row0 + count - 1) / qkv.rows; ++tile) {
            look(had, cta, owner(SP_QKV, tile), layer, QKV);
            learn(now[cta], said[QKV][owner(SP_QKV, tile)]);
          }
        };
        rows(0, part.group * heads * c.head_dim, heads * c.head_dim);
        if (part.last) {
          rows(qkv.tile1, part.group * p.stream_hpu * c.head_dim, p.stream_hpu * c.head_dim);
          rows(qkv.tile2, part.group * p.stream_hpu * c.head_dim, p.stream_hpu * c.head_dim);
        }
        const int of = part.b * groups + part.group;
        now[cta][cta] = layer * kSteps + PARTS;
        if (part.seg > 0) records[of][part.seg] = now[cta];
        else sums[of] = now[cta];
      }
    for (int cta = grid - 1; cta >= 0; --cta)
      for (const Part& part : parts[cta])
        if (part.seg == 0) {
          const int of = part.b * groups + part.group;
          if (part.nseg > 1) {  // the last part of the CTA's
            for (int seg = 1; seg < part.nseg; ++seg) learn(now[cta], records[of][seg]);
            sums[of] = now[cta];
          }
          now[cta][cta] = std::max(now[cta][cta], layer * kSteps + ATT);
          sums[of][cta] = layer * kSteps + ATT;
        }
    for (const int kind : {SP_O, SP_GU, SP_DOWN}) {
      const StreamPhase& own = ph[kind];
      const int step = step_of(kind);
      // the residual stream's columns of a tile of o_proj or down_proj
      auto residual = [&](Known& known, const Known& had, int cta, int tile) {
        const int from = kind == SP_O ? SP_DOWN : SP_O, of = kind == SP_O ? layer - 1 : layer;
        if (of < 0) return;
        const auto& all = kind == SP_O ? before : said[final_step(SP_O)];
        const int last = std::min(own.n, (tile + 1) * own.rows) - 1;
        for (int t = tile * own.rows / ph[from].rows; t <= last / ph[from].rows; ++t) {
          look(had, cta, writer(from, t), of, final_step(from));
          learn(known, all[writer(from, t)]);
        }
      };
      for (int cta = 0; cta < grid; ++cta) {
        const int count = units(kind, cta), first = table[kind * (grid + 1) + cta];
        bool spoken = false;
        for (int unit = first; unit < first + count; ++unit) {
          const int slice = unit / own.ntiles, tile = unit - slice * own.ntiles;
          const Known had = now[cta];
          if (kind == SP_GU) {
            stream(cta, SP_O, layer, said[final_step(SP_O)]);
          } else if (kind == SP_O) {
            const int col0 = slice * own.cs * kChunkK, col1 = std::min(own.k, col0 + own.cs * kChunkK);
            for (int group = col0 / (heads * c.head_dim); group <= (col1 - 1) / (heads * c.head_dim); ++group)
              for (int b = 0; b < batch; ++b) {
                look(had, cta, first_of[b * groups + group], layer, ATT);
                learn(now[cta], sums[b * groups + group]);
              }
          } else {
            const int col0 = slice * own.cs * kChunkK, col1 = std::min(own.k, col0 + own.cs * kChunkK);
            for (int t = col0 / ph[SP_GU].rows; t <= (col1 - 1) / ph[SP_GU].rows; ++t) {
              look(had, cta, owner(SP_GU, t), layer, GU);
              learn(now[cta], said[GU][owner(SP_GU, t)]);
            }
          }
          if (kind != SP_GU && own.nslice == 1) residual(now[cta], had, cta, tile);
          if (!spoken) speak(cta, layer, step);  // its first result knows the least
          spoken = true;
        }
      }
      if (own.nslice > 1)
        for (int cta = 0; cta < grid; ++cta) {
          bool spoken = false;
          for (int tile = 0; tile < own.ntiles; ++tile) {
            if (adds(kind, tile) != cta) continue;
            const Known had = now[cta];
            for (int slice = 0; slice < own.nslice; ++slice) {
              const int by = owner(kind, slice * own.ntiles + tile);
              look(had, cta, by, layer, step);
              learn(now[cta], said[step][by]);
            }
            residual(now[cta], had, cta, tile);
            if (!spoken) speak(cta, layer, step + 1);
            spoken = true;
          }
        }
    }
  }
  return early;
}

extern "C" int fence_met() { return kStreamFenceMet; }
