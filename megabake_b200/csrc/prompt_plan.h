// How a prompt pass cuts its projections (host side, pure functions of the configuration and the token count) and the
// parameter blocks of its kernels (prompt_kernels.cuh).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "megakernel.cuh"

namespace mk {

enum { PP_QKV = 0, PP_O = 1, PP_GU = 2, PP_DOWN = 3, PP_HEAD = 4, kPromptPhases = 5 };

// Launch classes.  Up to 128 tokens a prompt is bound by reading the weights: one CTA per tile, and tiles that give every SM
// some.  (Pairs with 64 MMA rows to a CTA for q/k/v, gate/up and the head are level up to 64 tokens and faster from 65 on, 1.7B shape, us,
// one CTA / a pair: 1 token 1226 / 1269, 64 1249 / 1241, 65 1494 / 1383, 100 1435 / 1371, 128 1447 / 1392; 0.5B, 128 1090 / 1044.  But a
// unit's walk along K begins at a place that the number of CTAs decides, so they add the same products up in another order: 2.5 % at the
// logits after 24 layers, no further from 64-bit results, and further than results may move.)  Beyond, by tensor cores and L2: CTA pairs (256 tokens each), and tiles chosen for one, two, or three and more of
// those (beyond three the cut of three: 1.7B shape, 1024 tokens 4422 us, 2048 8316).
constexpr int kPromptClasses = 4;
constexpr int kPromptRow = 128;   // token rows per CTA (64 rows are used for up to 64 tokens)
constexpr int kPromptStages = 16; // most stages of a pipeline
// Shared memory of a projection's CTA: one per SM, whose first stages travel while the kernels before it end.  (With two to an
// SM, so that they could travel while another projection is at work, CTAs that start early crowd on the SMs that are free first:
// 64 tokens of the 1.7B shape 1442 us against 1345.)
constexpr int kPromptSmem = 225 * 1024;

// Token-operand descriptors, shared with the tensor engine: (normalised rows, attention output, SiLU * up) x (boxes of 16, 32,
// 64, 128 tokens) x (1 to 4 K chunks).
constexpr int kOperandTiles = 4, kOperandChunks = 4, kOperandKinds = 3;
enum { kOperandXnorm = 0, kOperandAttn = 1, kOperandAct = 2 };

inline int prompt_class(int tokens, int grid) {
  return tokens <= kPromptRow || grid < 2 ? 0 : std::min(3, (tokens + 2 * kPromptRow - 1) / (2 * kPromptRow));
}

// One projection, the same for every layer of a class.
struct PromptPhase {
  int k, kc;             // reduction length, in elements and in 64-element chunks
  int nseg, nmat;        // matrices side by side along the output (q, k, v); matrices of a tile (gate and up: two)
  int n[3];              // rows of each
  int rows;              // weight rows of a tile (of each of its matrices)
  int tile_start[4];     // first tile of each segment, then the total
  int ksplit, kslice;    // K slices, and chunks per slice
};

inline void prompt_tiles(PromptPhase& p, int rows) {
  p.rows = rows;
  int tiles = 0;
  for (int s = 0; s < p.nseg; ++s) {
    p.tile_start[s] = tiles;
    tiles += (p.n[s] + rows - 1) / rows;
  }
  for (int s = p.nseg; s < 4; ++s) p.tile_start[s] = tiles;
}

// The five projections of a class.  `grid`: SMs to use.
inline void prompt_phases(const mk_config& c, int cls, int grid, PromptPhase* out) {
  const int q_size = c.q_heads * c.head_dim, kv_size = c.kv_heads * c.head_dim;
  const int ks[kPromptPhases] = {c.hidden, q_size, c.hidden, c.intermediate, c.hidden};
  const int ns[kPromptPhases] = {q_size, c.hidden, c.intermediate, c.hidden, c.vocab};
  for (int i = 0; i < kPromptPhases; ++i) {
    PromptPhase p{};
    p.k = ks[i];
    p.kc = ks[i] / kChunkK;
    p.nseg = i == PP_QKV ? 3 : 1;
    p.nmat = i == PP_GU ? 2 : 1;
    p.n[0] = ns[i];
    if (i == PP_QKV) p.n[1] = p.n[2] = kv_size;
    const bool wide = cls > 0, may_split = i == PP_O || i == PP_DOWN;
    // A tile of q or k rows is whole heads: its epilogue rotates pairs half a head apart.  Elsewhere the MMA's N decides for a
    // pair (multiples of 32), the logits' 32-byte stores, the swizzle's eight rows otherwise.
    const int step = i == PP_QKV ? c.head_dim : (wide ? 32 : (i == PP_HEAD ? 16 : 8));
    const int most = wide ? 256 : 128 / p.nmat;
    long long best = -1;
    PromptPhase chosen = p;
    for (int split = 1; split <= (may_split ? kMaxSplit : 1); ++split) {
      if (p.kc % split) continue;
      for (int rows = most / step * step; rows >= step; rows -= step) {
        PromptPhase t = p;
        prompt_tiles(t, rows);
        t.ksplit = split;
        t.kslice = p.kc / split;
        long long cost;
        if (wide) {
          // per chunk: the MMAs (an N = 256 one of a pair takes 128 cycles) or the operands out of L2 at 44 bytes per cycle
          // and SM; plus what a unit costs besides, its epilogue included
          const long long units = static_cast<long long>(t.tile_start[3]) * split * cls, pairs = std::max(1, grid / 2);
          const long long chunk = std::max<long long>(2 * p.nmat * rows, (kPromptRow + p.nmat * rows / 2) * 128 / 44);
          cost = (units + pairs - 1) / pairs * (t.kslice * chunk + 2000 + 8 * rows) + split * 600;
        } else {
          // per chunk of the busiest SM: its weights at 30 bytes per cycle, weights and (64) tokens at 42, or the pipeline's step
          const long long units = static_cast<long long>(t.tile_start[3]) * split;
          const long long chunk = std::max({p.nmat * rows * 128 / 30, (64 + p.nmat * rows) * 128 / 42, 256});
          cost = (units + grid - 1) / grid * (t.kslice * chunk + 2500) + split * 300;
        }
        if (best < 0 || cost < best) {
          best = cost;
          chosen = t;
        }
      }
    }
    out[i] = chosen;
  }
}

// Whether a call of the attention op (not causal; heads: of all sequences) goes to the tcgen05 kernel, with blocks of 128 queries,
// or to the one on mma.sync, with blocks of 64.  Times in us of a round of blocks as fitted to both kernels over heads 9 to 1024, 1 to
// 320 queries and 64 to 1400 keys: the first has one block to an SM and half the time per tile of 64 keys; the second has two with head size
// 64, and half the idle rows where the queries are few.  32 heads of 64 x 32 sequences with a mask, one query and 128 keys: 48 us on
// tcgen05, 27 on mma.sync; 64 x 128 50 and 33; 128 x 512 91 and 145.  The fit is of times from before masks came in tiles; over 423
// shapes timed since, the kernel taken is within a tenth of the other but for seven, which are within 17 %.
inline bool attention_on_tcgen05(int head_dim, int q_len, int k_len, long long heads, bool masked, int sms, bool limited) {
  if (k_len < 65) return false;  // one tile: 9.3 us against 10.0 for 32 heads of 64 x 64 with a mask
  const double tiles = (k_len + 63) / 64;
  const long long wide = heads * ((q_len + 127) / 128), narrow = heads * ((q_len + 63) / 64);
  auto rounds = [](long long blocks, int resident) -> double {  // the last one counts whole, but not beside many
    const double exact = static_cast<double>(blocks) / resident;
    const long long whole = (blocks + resident - 1) / resident;
    return whole > 4 ? exact : static_cast<double>(whole);
  };
  if (head_dim == 128) {  // one block to an SM either way
    if (q_len > 8) return true;
    return rounds(wide, sms) * (6.7 + (2 * wide <= sms ? 1.2 : 1.5) * tiles) <= rounds(narrow, sms) * (5.15 + 1.64 * tiles);
  }
  const double first = wide <= sms ? 5.3 + 0.91 * tiles : rounds(wide, sms) * (5.9 + 0.92 * tiles);
  const double second = narrow <= sms || limited ? rounds(narrow, sms) * ((q_len <= 16 ? 4.2 : 5.2) + (masked ? 1.25 : 1.08) * tiles)
                                                 : rounds(narrow, 2 * sms) * (6.2 + (masked ? 1.87 : 1.57) * tiles);
  return first <= second;
}

// Whether a mask's tiles, 64 positions of 128 queries, come by TMA (where its rows allow it) or each row to its thread with plain loads.
// A copy costs its whole box, also the rows past the last query; the plain loads of a full block are 32 lines a request.  So few queries
// take the loads, unless there are many tiles to hide behind; with head size 128, three stages deep, four tiles have to pay for the
// longer prologue.  us, loads / tiles: head size 64, 32 heads x 4 sequences, 1 x 512 13.6 / 20.6, 24 x 128 7.5 / 8.9, 65 x 200 9.8 / 10.8,
// 96 x 128 7.8 / 7.7, 128 x 512 14.2 / 13.2, 16 x 1024 20.6 / 19.6; head size 128, 32 heads, 64 x 1400 33.4 / 34.4, 200 x 72 9.4 / 9.9,
// 200 x 200 12.6 / 12.6, 96 x 256 12.1 / 11.6, 512 x 512 20.3 / 18.1.
inline bool attention_mask_in_tiles(int head_dim, int q_len, int k_len) {
  return head_dim == 128 ? q_len >= 96 && k_len > 192 : q_len >= 96 || (q_len >= 16 && k_len >= 1024);
}

// The same of a mask whose rows begin off 16-byte boundaries: eight copies a tile, one of each residue of the rows modulo eight, or loads,
// a word of a row at a time or two.  The copies are worth it from fewer positions on, where the last block of queries is not mostly
// empty.  us, loads / copies: head size 64, 32 heads, 96 x 130 8.7 / 8.1, 500 x 500 17.6 / 13.8, 130 x 205 11.2 / 12.1, 130 x 650 23.4 / 15.7,
// 64 x 330 12.4 / 10.7, x 4 sequences 13.0 / 11.9, 32 x 650 18.3 / 16.6, 32 x 330 12.1 / 16.4, 16 x 650 17.6 / 24.7; head size 128, 32 heads,
// 96 x 205 12.4 / 11.6, 500 x 500 21.4 / 19.4, 130 x 205 13.4 / 13.9, 200 x 330 18.4 / 15.4, 64 x 205 x 4 12.5 / 13.3.
inline bool attention_mask_in_eights(int head_dim, int q_len, int k_len) {
  const bool full = (q_len - 1) % 128 >= 63;  // the last block
  if (q_len >= 96) return k_len > (full ? (head_dim == 128 ? 192 : 128) : 256);
  return head_dim == 64 && k_len >= (q_len >= 64 ? 320 : 640) && q_len >= 32;
}

// What a CTA still waits for before it leaves: that the last use of every pipeline slot has been consumed, so that no commit
// is on its way to a barrier of shared memory that is somebody else's by then.  The uses count up over the launch, use u lies in
// slot u % stages, and a slot's barrier has the parity of its use; wait(slot, parity) returns false to give up.
template <typename Wait>
__host__ __device__ inline bool prompt_drain(int uses, int stages, Wait wait) {
  for (int u = uses < stages ? 0 : uses - stages; u < uses; ++u)
    if (!wait(u % stages, static_cast<uint32_t>(u / stages) & 1u)) return false;
  return true;
}

// Rows of the weight descriptors' boxes: a CTA of a pair brings half a tile.
inline int prompt_box_rows(const PromptPhase& p, int cls) { return cls > 0 ? p.rows / 2 : p.rows; }

// ---------------------------------------------------------------------------
// kernel parameters

// What bounds the kernels' waits and where a verdict goes.
struct PromptGuard {
  Control* ctrl;
  volatile int* status_mirror;
  long long timeout_cycles;
  uint32_t polls;  // a wait looks at its limit after every polls + 1 tries (a power of two)
};

// The event trace (mk_set_trace).  list: null, or [ctas][cap].
struct PromptTrace {
  unsigned long long* list;
  int cap, ctas;
};

struct PromptGemm {
  PromptGuard guard;
  const CUtensorMap* a;     // token operand: box of 64 x tokens x kb
  const CUtensorMap* b[3];  // weights: q, k, v, or gate, up, or the only one; box of 64 x (rows or rows / 2)
  const bf16* bias[3];
  bf16* dst;                // + token * ld + column
  float* partial;           // cut projections: [slice][token][n]
  const bf16 *cos_t, *sin_t;
  const long long* pos;
  int n[3], tile_start[4], out_col[3];
  int m, ld, rows, nmat;
  int ksplit, kslice;
  int token_tiles, units;
  int kb;                                     // K chunks per stage
  int stages, a_bytes, b_bytes, stage_bytes;  // per CTA: a chunk's tokens, a chunk's weights of one matrix, and a whole stage
  int instr_n;                                // N of an MMA
  int up_column;                              // gate and up: where the up accumulator begins
  int buffers;                                // accumulator buffers in tensor memory, 256 columns each
  int head_dim, max_positions;
  int stream_weights;                         // weights are read once
};

struct PromptNorm {
  PromptGuard guard;
  const bf16* src;       // residual stream, or null: embedding rows of the token ids
  const bf16* embed;
  const long long *ids, *pos;
  const float* partial;  // [parts][m][k]: the previous projection's K slices
  const bf16* weight;
  bf16 *h_out, *xnorm;
  int m, k, parts;
  int embed_rows, max_positions, check;  // check: the first kernel of a pass looks at every id and position
  float eps;
};

struct AttnArgs;
struct AttnTcMaps;

// One prompt pass: everything its launches are made from.
struct PromptPass {
  const mk_config* config;
  const mk_weights* weights;
  const PromptPhase* phases;    // of the class
  int cls, grid;
  const CUtensorMap* maps;      // of the class: 7 per layer, then the output head
  const CUtensorMap* operands;  // [kind][token tile][chunks - 1], as the tensor engine's
  bf16 *hidden_a, *hidden_b, *xnorm, *qkv, *attn, *act;
  float* partial;
  const long long *ids, *pos;
  const bf16* mask;
  bf16* logits;
  int m, batch, seq;
  const AttnArgs* attention;
  const AttnTcMaps* attention_maps;
  PromptGuard guard;
  PromptTrace trace;
};

cudaError_t prompt_prepare();  // shared-memory attributes of the kernels, on the current device
cudaError_t prompt_forward(const PromptPass& pass, cudaStream_t stream);
// Whether a launch takes the tcgen05 kernel, the one that reads its operands through `maps`.
bool prompt_attention_tc_wanted(const AttnArgs& args, int head_dim, int q_heads, int batch, int sms, bool limited, bool in_pass);
// sms: the SMs to use; limited: no more blocks than that; in_pass: causal, of a prompt pass.
cudaError_t prompt_attention_launch(const AttnArgs& args, const AttnTcMaps& maps, const PromptGuard& guard, int head_dim, int q_heads, int kv_heads,
                                    int batch, int sms, bool limited, bool in_pass, cudaStream_t stream);

}  // namespace mk
