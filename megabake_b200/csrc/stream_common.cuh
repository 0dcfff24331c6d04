// Decode for up to 32 sequences: data structures and synchronisation of the streaming kernel.
//
// A decode step is bound by reading the weights (and the caches) once, so everything here serves one aim: HBM
// never waits for the chain of dependent steps (projection -> attention -> projection ...).  One thread per CTA
// (the producer) walks the CTA's whole list of copies for the launch - weight tiles and cache tiles in the order
// in which they will be used - into one ring of shared-memory slots, and is held back by nothing but free
// slots.  Eight consumer warps take the slots in the same order.  While they wait for another CTA's results the
// ring fills (160-200 KB per SM, four microseconds of HBM time), and when the results are there they empty it at
// three to four times the rate at which HBM fills it.
//
// Hand-over between CTAs: "unset" words.  Every buffer that one CTA writes and another reads starts out filled
// with kUnset, a bit pattern no result has (a bf16 pair of NaNs with all bits set, which conversions never
// produce); a reader loads the data itself and reads again what is still unset.  A hand-over is one store and
// one load: no flag, no fence, no barrier.  Every buffer exists three times, used in turn by the layers; whoever writes a
// word in layer l resets the same word of layer l - 1's copy, whose readers are done: to write in layer l a CTA has
// read data that depends on every result of layer l - 1.  That copy is written again in layer l + 2.  A CTA that looks for it there has
// read something of layer l + 1 (each has a unit of every layer, see stream_busy_ctas), and what it has read depends on a result that the
// resetting CTA stored behind a fence behind the reset.  The fence of layer l lies between gate/up and the first result of down_proj
// (kStreamFenceMet): behind the resets of layer l up to gate and up and of down_proj in layer l - 1.  The launch ends with a grid
// barrier, behind which the last layer's words are reset.
#pragma once
#include "device_common.cuh"

namespace mk {

constexpr int kStreamWarps = 8;
constexpr int kStreamConsumers = kStreamWarps * 32;
constexpr int kStreamThreads = 128 + kStreamConsumers;  // a warp group for the producer, two for the consumers
constexpr int kStreamTokens = 32;        // largest batch
constexpr int kStreamMaxSlots = 16;
constexpr int kStreamRows = 16;          // weight rows of a tile: the M of mma.sync
constexpr int kStreamKb = 16;            // 64-element chunks per copy: 32 KB (chunks past the end of a row read as zero)
constexpr int kStreamWpc = kStreamKb * 2 / kStreamWarps;  // 32-element windows of a copy per warp
constexpr int kStreamSlotBytes = kStreamKb * 2048;  // one weight copy, or one cache tile
constexpr int kStreamPartPitch = 20;     // floats per token of a tile's partial sums (16 rows; the padding keeps stores conflict-free)
constexpr int kStreamMaxSegments = 24;   // parts a (sequence, head group)'s context may be cut into
constexpr int kStreamLengths = 1024;     // valid lengths kept in shared memory (layers x sequences when they differ per sequence)
constexpr uint32_t kUnset = 0xFFFFFFFFu;
constexpr int kStreamStoredBarrier = 2, kStreamFencedBarrier = 3;  // named barriers of the consumers and the fencing warp (stream_fence)
constexpr int kStreamFenceThreads = kStreamConsumers + 32;

enum { SP_QKV = 0, SP_O = 1, SP_GU = 2, SP_DOWN = 3, SP_HEAD = 4, kStreamPhases = 5 };
constexpr int kStreamFenceMet = SP_DOWN;  // no result of this projection, or of one behind it, is stored ahead of its layer's fence

// Token classes: a kernel is compiled for at most 1, 4, 8, 16 or 32 tokens (4 in the layout of 8).
__host__ __device__ constexpr int stream_token_tiles(int tm) { return tm <= 8 ? 1 : tm / 8; }
// Copies of a slice whose operand a warp's registers hold.
__host__ __device__ constexpr int stream_fit(int nt) { return nt == 4 ? 2 : 4; }
// ... of a normalised operand, which is of the hidden size, at most 2048: two.  A phase's length in instructions is its time, so
// its code holds no more (with four, us a step: 1.7B shape, 16 sequences 1638 against 1583) - but for one token, where the shorter
// code came out 1 to 2 % slower (831 against 848).
__host__ __device__ constexpr int stream_fit_normalised(int tm) { return tm == 1 ? 4 : 2; }

// Every CTA reads the whole residual stream, and while it waits it reads the same few lines again and again: with few tokens
// those lines lie in a handful of L2 slices and the readers hold up the writers' stores.  So results are written to
// several copies, and a CTA reads one of them: the one of its place on the chip, so that a copy is read from few places (SMs with
// adjacent numbers are neighbours; 135M shape, 16 steps 8094 -> 7875 us against dealing the copies round robin, 0.5B 520 -> 509,
// 1.7B no difference).
__host__ __device__ constexpr int stream_copies(int tm) { return tm == 1 ? 8 : (tm <= 8 ? 2 : 1); }

__device__ __forceinline__ int stream_copy_of_sm(int copies) {
  uint32_t id, count;
  asm volatile("mov.u32 %0, %smid;" : "=r"(id));
  asm volatile("mov.u32 %0, %nsmid;" : "=r"(count));
  return min(static_cast<int>(id * copies / count), copies - 1);
}

// One kind of projection (the same for every layer).  Rows are cut into tiles of at most 16; the K range of o and down into
// `nslice` slices, which go to different CTAs and hand fp32 partial sums to the tile's owner.  The token operand of a
// slice fits the consumers' registers, or (`parts` > 1) is fetched in parts for every tile.
struct StreamPhase {
  int k, n;          // reduction length, rows
  int cs;            // 64-element chunks per slice
  int nslice;
  int rows;          // weight rows of a tile: at most 16, even
  int ncopy;         // copies per (tile, slice, matrix)
  int parts;         // passes over a slice whose operand is larger than the registers (then fetched again for every tile)
  int ntiles;
  int tile1, tile2;  // QKV: first tile of the k and of the v matrix
  int row1, row2;    // QKV: first row of the k and of the v matrix
};

struct StreamLayer {
  const bf16 *input_norm, *post_norm;
  const bf16* bias[3];
};

// What the kernel needs beyond KParams; one per token-tile count, in device memory.  Buffers that the layers use in
// turn: [.][layer % 3].
struct StreamPlan {
  StreamPhase ph[kStreamPhases];
  const CUtensorMap* maps;     // 7 per layer (q k v o gate up down), then the output head
  const StreamLayer* layers;
  const bf16* final_norm;
  const int* units;            // [kStreamPhases][grid + 1]: first unit of every CTA
  const bf16* src[kStreamPhases][3];  // token operand, laid out by stream_place
  bf16* dst[kStreamPhases][3];        // results
  const bf16* res[kStreamPhases][3];  // O, DOWN: residual stream to add to
  float* part[kStreamPhases][3];      // cut projections: fp32 partial sums [slice][tile][token][16]
  bf16* attn[3];                      // attention output
  unsigned long long* rec;     // attention parts: [batch * q_heads][kStreamMaxSegments][head_dim + 2] stamped words
};

// The part of a (sequence, group) that starts at tile `at` of this CTA's run.
struct StreamSegment {
  int b, group, t0, t1, nt;  // tiles [t0, t1) of nt
  int seg, nseg;             // this part's number and how many parts there are
  int len;                   // cached positions of the sequence: the new one's place
};
// A CTA's parts of a layer come in lists of at most this many.  Equal lengths need one list; a long sequence beside many
// short ones makes the runs long, and a run through the short ones crosses a head group per tile.
constexpr int kStreamSegments = 16;
constexpr int kStreamMoreParts = 1 << 16;  // in a list's count: another list of the same layer follows

// Shared memory beside the ring.  What the phases need now and then lives here and not in registers, which the token
// operand fills.
struct StreamMisc {
  uint64_t full[kStreamMaxSlots];
  uint64_t empty[kStreamMaxSlots];
  const KParams* p;  // for what is off the path: the phases are handed the parameters themselves, which are operands of their instructions (and
                     // through this pointer loads that miss L1: a step 0.5 to 2 % longer)
  Control* ctrl;
  long long deadline;
  int cta, grid;
  int copy;      // which copy of the hand-over buffers this CTA reads
  int tokens, token_class;  // of this launch, and the TM of its kernel
  int wabort;    // the limit on waits has run out: nobody waits any more
  int progress;  // layer the consumers are in; layers + 1: at the grid barrier; -1: finished
  int bad;       // prologue verdict
  int complete;  // the grid barrier was reached: one thread's verdict, so that all threads end the launch the same way
  int trace_n, trace_on;
  int fence_aside;  // stream_fence
  int copies;       // hand-over buffers exist this often
  int psum_offset;  // bytes from the end of this block to the partial sums (the attention area comes first)
  int first_tile[kStreamPhases], first_slice[kStreamPhases], units[kStreamPhases];  // where this CTA's units start, how many
  StreamLayer lw[2];            // this layer's and the next one's vectors
  StreamSegment seg[2][kStreamSegments];  // two lists of this CTA's attention parts, worked out ahead by a helper thread
  int seg_count[2];             // ... how many, and whether the layer has more (kStreamMoreParts)
  int seg_ready;                // lists put in place so far
  int seg_taken;                // the list the consumers are at: all of them are done with the ones before
  StreamPlan plan;
  int id_s[kStreamTokens];
  int pos_s[kStreamTokens];
  float ss[kStreamWarps][kStreamTokens];  // per-warp sums of squares
  int len_s[kStreamLengths];
};
constexpr int kStreamMiscBytes = 8192;
static_assert(sizeof(StreamMisc) <= kStreamMiscBytes, "stream misc block too large");
__device__ __forceinline__ uint8_t* stream_scratch(StreamMisc* sm) { return reinterpret_cast<uint8_t*>(sm) + kStreamMiscBytes; }
__device__ __forceinline__ float* stream_psum(StreamMisc* sm) { return reinterpret_cast<float*>(stream_scratch(sm) + sm->psum_offset); }

// Where column `column` of token `tok` lies in the buffers that feed projections.  The B fragment of mma.sync gives lane
// t = lane % 4 the elements 2t, 2t + 1 of every eight; within a window of 32 columns the pairs are stored so that one
// 16-byte load of lane t brings its pairs of all four groups of eight, and the windows of all tokens of the token class
// (TM) lie side by side, so that a warp's load is whole lines.
__host__ __device__ __forceinline__ int stream_perm(int column) {
  return ((column & 7) >> 1) * 8 + ((column >> 3) & 3) * 2 + (column & 1);
}
__host__ __device__ __forceinline__ int stream_place(int tm, int tok, int column) {
  return ((column >> 5) * tm + tok) * 32 + stream_perm(column);
}

// The phases of a layer are inlined into one loop.  Whatever a phase derives from the thread number or the shared-memory
// address is loop-invariant, and the compiler would compute it all ahead of the loop and keep it in registers the token
// operands need: values passed through here at the start of a phase are opaque, so their derivatives stay inside it.
template <typename V>
__device__ __forceinline__ V stream_opaque(V v) {
  if constexpr (sizeof(V) == 4) asm volatile("" : "+r"(v));
  else asm volatile("" : "+l"(v));
  return v;
}

// The fence of a layer, by a warp of the producer's group: the consumers tell it that their results and resets of the layer up to gate
// and up are stored, go on, and meet it again ahead of the first result of down_proj, in the block barrier that is there anyway.  A
// fence orders what its thread knows of, and the first barrier has made the consumers' stores known to it; it has come through when those
// are performed for the whole GPU, and no consumer stores a result of down_proj before the second barrier.  (A reader needs none: it
// looks for a word when the loop that waited for an earlier one has ended.)  (1400 cycles a layer of the
// 135M shape by clock stamps, ahead of down_proj.)
// Two to eight tokens only where the ring holds the gate and up matrices of a layer: elsewhere the CTAs end that phase one by one as HBM
// brings them their weights, and those that are through and have no fence to wait for look for the others' results all the longer.  With nine
// to sixteen, who wait for more anyway, it is as well there.  With 32 tokens there is no difference.  A step, fence on the way -> aside (60
// to 1900 positions): 135M shape, one sequence -2.1 %, ten -4.5, sixteen -2.9; 0.5B, one -5.2, eight -3.4, ten -4.4, sixteen -3.6; 1.7B, whose
// gate and up the ring does not hold, one 0, two to six +1.0 to 1.3, nine -1.5 to -2.4, twelve and fourteen -1.3 to -1.7, sixteen -1.7 to -2.7.
// With one token the first look at down_proj's operand comes late, too: it is not there at once, and a look that comes too early is in
// the way of the stores.  Without the 300 ns: 135M +1.5 to 3.8 %, 0.5B +0.3 to 0.7, 1.7B +0.4 to 0.5.  (Two to eight tokens gain nothing in the
// mean, 500 ns: 135M -0.2, 0.5B +0.5.  One look first and a rest only where the operand is unset, one token: 135M +3.8 to 6.5, 0.5B +1.4
// to 2.2, 1.7B +1.2.)
constexpr int kStreamLookLate = 300;  // ns
template <int TM>
__device__ __forceinline__ bool stream_fence_aside(const KParams& p, int grid) {
  if (TM != 8) return TM < 32;
  return 4ll * p.inter * p.hidden <= static_cast<long long>(p.stream_slots) * kStreamSlotBytes * grid;
}
// Whether it is in a launch of this token class.
template <int TM>
__device__ __forceinline__ bool stream_is_aside(const StreamMisc* sm) {
  return TM == 8 ? sm->fence_aside != 0 : TM < 32;
}
__device__ __forceinline__ void stream_fence(int layers) {
  for (int layer = 0; layer < layers; ++layer) {
    named_bar_sync(kStreamStoredBarrier, kStreamFenceThreads);
    __threadfence();
    named_bar_arrive(kStreamFencedBarrier, kStreamFenceThreads);
  }
}

__device__ __forceinline__ void stream_sync() { named_bar_sync(1, kStreamConsumers); }

__device__ __forceinline__ bool stream_aborted(StreamMisc* sm) { return *reinterpret_cast<volatile int*>(&sm->wabort) != 0; }

// Waits look at one word of shared memory; the limit on them is kept by a thread with nothing else to do (stream_watch).
// The word may change between two warps' looks at it: after a wait that it ended every warp goes on through the same
// phases, parts and block barriers, with whatever it has.
__device__ __forceinline__ void stream_wait(StreamMisc* sm, uint32_t bar, uint32_t parity) {
  while (!mbar_try_wait(bar, parity))
    if (stream_aborted(sm)) return;
}

// The bound on every wait of this CTA: ends them all when another CTA has given up or the deadline has passed.
__device__ __forceinline__ void stream_watch(StreamMisc* sm) {
  Ctx cx;
  cx.p = sm->p;
  cx.ctrl = sm->ctrl;
  cx.deadline = sm->deadline;
  cx.cta = sm->cta;
  while (*reinterpret_cast<volatile int*>(&sm->progress) >= 0) {
    const int at = *reinterpret_cast<volatile int*>(&sm->progress);
    if (give_up(cx, at > sm->p->layers ? SITE_GRID_BARRIER : SITE_ATT_EXCHANGE, at)) {
      *reinterpret_cast<volatile int*>(&sm->wabort) = 1;
      return;
    }
    __nanosleep(2000);
  }
}

__device__ __forceinline__ uint4 ld_relaxed_v4(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_relaxed_v2(const void* p) {
  uint2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_v2(void* p, uint32_t a, uint32_t b) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ bool unset4(const uint4& v) { return v.x == kUnset || v.y == kUnset || v.z == kUnset || v.w == kUnset; }

static __device__ __noinline__ void stream_trace_record(StreamMisc* sm, int code) {
  const int n = sm->trace_n, cap = sm->p->trace_cap;
  if (n >= cap) return;
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  sm->p->trace[static_cast<size_t>(sm->cta) * cap + n] = (static_cast<unsigned long long>(code) << 56) | (t & 0x00FFFFFFFFFFFFFFull);
  sm->trace_n = n + 1;
}
// What a consumer thread carries through all phases.
struct StreamThread {
  StreamMisc* sm;
  int wtid;
  int turn, last_turn;  // layer % 3, and the layer before's
  int pbuf;      // which half of the partial-sum area the next tile uses
  int list;      // the list of attention parts that comes next
  bool tracing;  // this thread records events
  __device__ __forceinline__ void trace(int code) const {
    if (tracing) stream_trace_record(sm, code);
  }
};

// The ring as one role sees it: the slot that comes next and the parity of its current use.
struct StreamPipe {
  uint32_t base, full0, empty0;
  int nslots, slot;
  uint32_t parity;
  __device__ __forceinline__ uint32_t addr() const { return base + static_cast<uint32_t>(slot) * kStreamSlotBytes; }
  __device__ __forceinline__ uint32_t full() const { return full0 + static_cast<uint32_t>(slot) * 8u; }
  __device__ __forceinline__ uint32_t empty() const { return empty0 + static_cast<uint32_t>(slot) * 8u; }
  __device__ __forceinline__ void next() {
    if (++slot == nslots) {
      slot = 0;
      parity ^= 1u;
    }
  }
};
// Consumer side: every warp waits for the slot, and releases it with one arrival.
__device__ __forceinline__ void stream_release(StreamPipe& pipe, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(pipe.empty());
  pipe.next();
}

// ---------------------------------------------------------------------------
// How the cached positions of a layer are dealt to the CTAs.
//
// A tile is `tile_keys` positions of `hpu` adjacent KV heads of one sequence, once from the key and once from the
// value cache.  The tiles of a layer, ordered by sequence, head group and position, are cut into equal contiguous
// runs, one per CTA, so that all SMs read the same number of bytes whatever batch, heads and lengths are; a run
// crosses head groups where it must, and a group's context is then summed up from the parts.  Starting another head group
// costs a CTA about as much as two tiles (its q, the hand-over of the sums), so where runs that end with their group
// are at most two tiles longer, they are taken instead.
struct StreamTiles {
  int groups, tile_keys, batch, per, first, last;
  int runs;        // > 0: every group is cut into this many runs, none of which crosses groups
  int nt;          // tiles per (sequence, group) when all lengths are equal, else 0 (the new position included)
  const int* len;  // valid lengths: one, or one per sequence
  __host__ __device__ __forceinline__ int tiles_of(int b) const {
    return nt > 0 ? nt : len[b] / tile_keys + 1;
  }
  __host__ __device__ __forceinline__ int length_of(int b) const { return nt > 0 ? len[0] : len[b]; }
};

__host__ __device__ __forceinline__ StreamTiles stream_tiles(const KParams& p, const int* len, int cta, int grid) {
  StreamTiles s;
  s.groups = p.kv_heads / p.stream_hpu;
  s.tile_keys = p.stream_tile_keys;
  s.batch = p.batch;
  s.len = len;
  int total, longest;
  if (p.ragged) {
    s.nt = 0;
    total = 0;
    longest = 1;
    for (int b = 0; b < p.batch; ++b) {
      const int n = s.tiles_of(b);
      total += n;
      longest = max(longest, n);
    }
    total *= s.groups;
  } else {
    s.nt = len[0] / s.tile_keys + 1;
    total = s.nt * s.groups * p.batch;
    longest = s.nt;
  }
  // never more parts than a combining CTA has records for
  s.per = max((total + grid - 1) / grid, (longest + kStreamMaxSegments - 3) / (kStreamMaxSegments - 2));
  s.runs = 0;
  const int groups = s.groups * p.batch;
  if (s.nt > 0 && groups <= grid) {
    const int per = max((s.nt + grid / groups - 1) / (grid / groups), (s.nt + kStreamMaxSegments - 1) / kStreamMaxSegments);
    if (per <= s.per + 2) {
      s.per = per;
      s.runs = (s.nt + per - 1) / per;
      const int which = cta / s.runs, at = (cta - which * s.runs) * per;
      s.first = s.last = which < groups ? which * s.nt + at : total;
      if (which < groups) s.last = min(s.first + per, (which + 1) * s.nt);
      return s;
    }
  }
  s.first = min(total, cta * s.per);
  s.last = min(total, s.first + s.per);
  return s;
}

__device__ __forceinline__ const int* stream_lengths(const KParams& p, const StreamMisc* sm, int layer) {
  return sm->len_s + (p.ragged ? layer * p.batch : layer);
}

__host__ __device__ __forceinline__ StreamSegment stream_segment(const StreamTiles& s, int at, int cta) {
  StreamSegment g;
  int start;  // first tile of the (sequence, group)
  if (s.nt > 0) {
    const int which = at / s.nt;
    g.b = which / s.groups;
    g.group = which - g.b * s.groups;
    g.nt = s.nt;
    start = which * s.nt;
  } else {
    int b = 0, base = 0, n = s.tiles_of(0);
    while (at >= base + n * s.groups) {
      base += n * s.groups;
      n = s.tiles_of(++b);
    }
    g.b = b;
    g.group = (at - base) / n;
    g.nt = n;
    start = base + g.group * n;
  }
  g.t0 = at - start;
  g.t1 = min(g.nt, g.t0 + s.last - at);
  if (s.runs > 0) {
    g.seg = g.t0 / s.per;
    g.nseg = s.runs;
  } else {
    const int first_cta = start / s.per;
    g.seg = cta - first_cta;
    g.nseg = (start + g.nt - 1) / s.per - first_cta + 1;
  }
  g.len = s.length_of(g.b);
  return g;
}

// The parts that follow from tile `at` of this CTA's run on, as many as a list holds; `at` moves past them.
__host__ __device__ __forceinline__ int stream_next_parts(const StreamTiles& s, int cta, int& at, StreamSegment* list) {
  int n = 0;
  while (n < kStreamSegments && at < s.last) {
    const StreamSegment g = stream_segment(s, at, cta);
    list[n++] = g;
    at += g.t1 - g.t0;
  }
  return n;
}

// A helper thread works out the parts of each layer, a list ahead: the divisions would be on every consumer's path.  It and the
// consumers wait for each other without a look at `wabort`: consumers that have given up on everything else still come by
// here, and a warp that skipped its parts because it saw the abort, beside one that did not, would leave that one alone at
// a block barrier.
__device__ __forceinline__ void stream_plan_parts(const KParams& p, StreamMisc* sm) {
  int list = 0;
  for (int layer = 0; layer < p.layers; ++layer) {
    const StreamTiles tiles = stream_tiles(p, stream_lengths(p, sm, layer), sm->cta, sm->grid);
    int at = tiles.first;
    do {
      while (*reinterpret_cast<volatile int*>(&sm->seg_taken) < list - 1) __nanosleep(200);  // the list before the last is still in use
      const int n = stream_next_parts(tiles, sm->cta, at, sm->seg[list & 1]);
      sm->seg_count[list & 1] = n | (at < tiles.last ? kStreamMoreParts : 0);
      ++list;
      __threadfence_block();
      *reinterpret_cast<volatile int*>(&sm->seg_ready) = list;
    } while (at < tiles.last);
  }
}

// Consumers: the count of list `list`, once it is there.
__device__ __forceinline__ int stream_next_list(StreamMisc* sm, int list) {
  while (*reinterpret_cast<volatile int*>(&sm->seg_ready) <= list) {
  }
  __threadfence_block();
  return sm->seg_count[list & 1];
}

}  // namespace mk
