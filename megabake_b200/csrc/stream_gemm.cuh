// Projections of the streaming decode kernel: y[token, row] = x[token, :] . W[row, :] for up to 32 tokens.
//
// A unit is a tile of up to 16 weight rows over one K slice.  Its copies hold the rows x 16 64-element chunks, each chunk
// [rows][128 B] with the 128-byte swizzle of a tiled TMA copy.  The eight warps split K, not rows: of every copy
// warp w multiplies the 32-element windows w, w + 8, ... (ldmatrix.x4 for the weights as the A operand,
// mma.sync m16n8k16), so that one tile occupies all warps and the token operand of a warp, an eighth of the
// slice, stays in its registers for all tiles of the slice: per window and warp two ldmatrix and two
// MMAs per eight tokens, nothing else.  A 32 KB copy then takes the SM about 350 cycles (shared-memory reads at
// 128 B per cycle are the limit) where HBM delivers one per 1450 cycles.  The warps' partial sums meet in shared
// memory once per tile and are added in warp order, whole rows of a token to a warp: what eight lanes store lies together, and L2
// takes it as one or two sectors.  Every other CTA polls those lines, and a store waits for the requests before it (with a row pair
// to a warp, eight stores a tile and copy: 135M shape, 16 steps 9215 -> 8717 us, 0.5B 586 -> 544, 1.7B, one sequence 826 -> 805).
//
// Between two hand-overs a phase is a chain of dependent instructions on at most two warps per scheduler, so its length
// in instructions is its time: pointers are fetched before the operand is waited for, and kernels are compiled per
// token class so that a one-token launch carries nothing else.
#pragma once
#include "stream_common.cuh"

namespace mk {

enum { SG_NORM = 0, SG_PLAIN = 1, SG_MLP = 2 };  // QKV and HEAD; O and DOWN; GU

// Four words of lane t's 16-byte vector of a window of a row in plain order.
__device__ __forceinline__ uint4 stream_plain_vec(const bf16* window, int t) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(window) + t;
  return make_uint4(__ldg(w), __ldg(w + 4), __ldg(w + 8), __ldg(w + 12));
}

// Layer 0's residual stream is the embedding rows of the token ids: dealt to the CTAs and written like any result, so that
// its readers need not know.
template <int TM>
__device__ __forceinline__ void stream_embed(const KParams& p, StreamMisc* sm, int wtid) {
  const int pairs = p.hidden / 2, items = p.m * pairs;
  uint32_t* const dst = reinterpret_cast<uint32_t*>(const_cast<bf16*>(sm->plan.src[SP_QKV][0]));
  for (int i = sm->cta * kStreamConsumers + wtid; i < items; i += sm->grid * kStreamConsumers) {
    const int tok = i / pairs, col = (i - tok * pairs) * 2;
    const uint32_t word = __ldg(reinterpret_cast<const uint32_t*>(p.embed + static_cast<size_t>(sm->id_s[tok]) * p.hidden + col));
    // a table entry may hold the unset pattern (two NaNs); any other NaN says the same
    for (int c = 0; c < stream_copies(TM); ++c)
      st_relaxed_u32(dst + (static_cast<size_t>(c) * TM * p.hidden + stream_place(TM, tok, col)) / 2, word == kUnset ? 0x7FFF7FFFu : word);
  }
}

__device__ __forceinline__ float stream_square(uint32_t x, float sum) {
  const float lo = __uint_as_float(x << 16), hi = __uint_as_float(x & 0xFFFF0000u);
  return fmaf(hi, hi, fmaf(lo, lo, sum));
}
__device__ __forceinline__ float stream_square4(const uint4& x, float sum) {
  return stream_square(x.x, 0.f) + stream_square(x.y, 0.f) + stream_square(x.z, 0.f) + stream_square(x.w, sum);
}

// Largest word of a fragment set: kUnset if any word is unset.
__device__ __forceinline__ uint32_t stream_top(uint32_t top, const uint4& v) { return max(max(top, max(v.x, v.y)), max(v.z, v.w)); }

// Every CTA wants a normalised operand, and its results come from all of them: one word per warp is watched until it is there.  (All
// of it at once, again and again, would hold up the stores it is waiting for: one token, 135M shape, 16 steps 7763 -> 7346 us, 0.5B
// 503 -> 481, 1.7B 739 -> 733.)  The operands of o_proj and down_proj are read at once, a round trip less: with a watch 0.5B at one
// 490, 1.7B, eight sequences 3536 against 3494, sixteen 1464 against 1451.  A rest between two looks, one token: 1.7B 0.7 % slower.
template <int TM>
__device__ __forceinline__ void stream_watch_word(StreamMisc* sm, const bf16* at) {
  while (ld_relaxed_u32(reinterpret_cast<const uint32_t*>(at)) == kUnset && !stream_aborted(sm))
    if constexpr (TM > 1) __nanosleep(40);
}

// Token operand of one K slice in fragment order: frag[i][n] is this lane's vector of window i * 8 + warp for token
// n * 8 + lane / 4.  All addresses are one base plus constants.
template <int TM, int NC, bool NORM>
__device__ __forceinline__ void stream_operand(StreamMisc* sm, const bf16* src, int T, int ncopy, int live, int kbase, int wtid,
                                               uint32_t (&frag)[NC * kStreamWpc][stream_token_tiles(TM)][4]) {
  constexpr int NT = stream_token_tiles(TM);
  const int lane = wtid & 31, grp = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < NC * kStreamWpc; ++i)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      // unset where there is something to fetch
      const uint32_t init = (i < live && n * 8 + grp < T) ? kUnset : 0u;
      frag[i][n][0] = frag[i][n][1] = frag[i][n][2] = frag[i][n][3] = init;
    }
  const bf16* const base = src + (kbase >> 5) * TM * 32 + grp * 32 + t * 8;
  if (NORM && live > 0) stream_watch_word<TM>(sm, src + ((kbase >> 5) + (live - 1) * 8) * TM * 32);
  uint32_t top;
  do {  // every load of a pass is issued before any is looked at; what was there is mostly not read again
    top = 0u;
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (c < ncopy) {
#pragma unroll
        for (int jj = 0; jj < kStreamWpc; ++jj)
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            uint32_t(&f)[4] = frag[c * kStreamWpc + jj][n];
            // (16 tokens: what is asked again costs less than looking at 32 vectors first, and their spills: 1484 -> 1455 us, 0.5B
            // 673 -> 659; with 8 and 32 tokens there is no gain)
            if (TM == 16 ? c * kStreamWpc + jj < live && n * 8 + grp < T : stream_top(0u, make_uint4(f[0], f[1], f[2], f[3])) == kUnset) {
              const uint4 v = ld_relaxed_v4(base + ((c * kStreamWpc + jj) * 8 * TM + n * 8) * 32);
              f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
            }
          }
      }
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (c < ncopy) {
#pragma unroll
        for (int jj = 0; jj < kStreamWpc; ++jj)
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const uint32_t(&f)[4] = frag[c * kStreamWpc + jj][n];
            top = stream_top(top, make_uint4(f[0], f[1], f[2], f[3]));
          }
      }
  } while (top == kUnset && !stream_aborted(sm));
}

// RMSNorm of an operand in registers.  The sums of squares are the diagonal of X X^T on the tensor cores: the fragments of
// two token tiles are the A operand of the same instruction (rows 0-7 and 8-15).
template <int NT, int NC>
__device__ __forceinline__ void stream_gram(int ncopy, const uint32_t (&frag)[NC * kStreamWpc][NT][4], float (&gram)[NT][4]) {
#pragma unroll
  for (int c = 0; c < NC; ++c)
    if (c < ncopy) {
#pragma unroll
      for (int jj = 0; jj < kStreamWpc; ++jj)
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const int i = c * kStreamWpc + jj, lo = n & ~1, hi = NT > 1 ? (n | 1) : 0;
            const uint32_t a[4] = {frag[i][lo][2 * s], NT > 1 ? frag[i][hi][2 * s] : 0u, frag[i][lo][2 * s + 1], NT > 1 ? frag[i][hi][2 * s + 1] : 0u};
            mma_bf16_16816(gram[n], a, frag[i][n][2 * s], frag[i][n][2 * s + 1]);
          }
    }
}
// The same of two to four tokens: a fused multiply-add an element in fp32, added up as the spread operand of one token is, so that a
// sequence gets the bits it gets alone.  Products on the tensor cores are added up there by rules of their own.
template <int NC>
__device__ __forceinline__ float stream_squares(int ncopy, const uint32_t (&frag)[NC * kStreamWpc][1][4]) {
  static_assert(NC == 2 && kStreamWpc == 4, "eight windows to a warp");
  float s[kStreamWpc];
#pragma unroll
  for (int i = 0; i < kStreamWpc; ++i) s[i] = stream_square4(make_uint4(frag[i][0][0], frag[i][0][1], frag[i][0][2], frag[i][0][3]), 0.f);
  if (ncopy > 1) {
#pragma unroll
    for (int i = 0; i < kStreamWpc; ++i) {
      const uint32_t(&f)[4] = frag[kStreamWpc + i][0];
      s[i] += stream_square4(make_uint4(f[0], f[1], f[2], f[3]), 0.f);
    }
  }
  float sum = (s[0] + s[2]) + (s[1] + s[3]);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  return sum + __shfl_xor_sync(0xffffffffu, sum, 1);
}
// x * rinv and the product with the norm weight, on bf16 pairs: the two roundings of the Hugging Face RMSNorm.
__device__ __forceinline__ uint32_t stream_norm_pair(uint32_t x, uint32_t w, float r) {
  return mul_bf16x2(w, pack2(__uint_as_float(x << 16) * r, __uint_as_float(x & 0xFFFF0000u) * r));
}
// The norm weights of a warp's windows are asked for before its operand is waited for: behind it, four small loads a window
// were on the path of every normalised phase (1.7B shape, 8 sequences, 4 steps 3888 -> 3675 us; 16 sequences 1574 -> 1550).
// With 32 tokens the registers are the operand's, and there the change made no difference.
template <int NT> constexpr bool kStreamWeightsAhead = NT <= 2;
template <int NT, int NC>
__device__ __forceinline__ void stream_normalise(const bf16* normw, int ncopy, int live, int kbase, int wtid, const float (&r)[NT],
                                                 const uint4 (&ahead)[kStreamWeightsAhead<NT> ? NC * kStreamWpc : 1],
                                                 uint32_t (&frag)[NC * kStreamWpc][NT][4]) {
  const bf16* wrow = normw + kbase;
#pragma unroll
  for (int c = 0; c < NC; ++c)
    if (c < ncopy) {
#pragma unroll
      for (int jj = 0; jj < kStreamWpc; ++jj) {
        const int i = c * kStreamWpc + jj;
        if (i < live) {
          const uint4 w = kStreamWeightsAhead<NT> ? ahead[kStreamWeightsAhead<NT> ? i : 0] : stream_plain_vec(wrow + i * 256, wtid & 3);
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            uint32_t(&f)[4] = frag[i][n];
            f[0] = stream_norm_pair(f[0], w.x, r[n]); f[1] = stream_norm_pair(f[1], w.y, r[n]);
            f[2] = stream_norm_pair(f[2], w.z, r[n]); f[3] = stream_norm_pair(f[3], w.w, r[n]);
          }
        }
      }
    }
}

// The normalised operand of one token.  In fragment order only four lanes would have work, so a warp deals its vectors to all
// lanes, normalises them there and passes them to the fragment's lanes through shared memory of its own.
template <int NC>
__device__ __forceinline__ void stream_operand_spread(const KParams& p, StreamMisc* sm, const bf16* src, const bf16* normw, int k, int ncopy, int live, int wtid,
                                                      uint32_t (&frag)[NC * kStreamWpc][1][4]) {
  constexpr int IT = NC * kStreamWpc * 4 / 32;  // vectors per lane; a second one only where a warp has more than eight windows
  const int warp = wtid >> 5, lane = wtid & 31;
  const int first = (lane >> 2) * 8 + warp;  // this lane's first window; the next one is 64 on
  const int left = live - (lane >> 2);       // this lane has vector i if 8 i < left
  const bool more = live > 8;
  const float fk = static_cast<float>(k), eps = p.eps;
  uint4 w[IT], x[IT];
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    w[i] = x[i] = make_uint4(0u, 0u, 0u, 0u);
    if ((i == 0 || more) && 8 * i < left) w[i] = stream_plain_vec(normw + (first + i * 64) * 32, lane & 3);
  }
  const bf16* base = src + first * 32 + (lane & 3) * 8;
  if (live > 0) stream_watch_word<1>(sm, src + (warp + (live - 1) * 8) * 32);
  uint32_t top;
  do {
    top = 0u;
#pragma unroll
    for (int i = 0; i < IT; ++i)
      if ((i == 0 || more) && 8 * i < left) x[i] = ld_relaxed_v4(base + i * 64 * 32);
#pragma unroll
    for (int i = 0; i < IT; ++i) top = stream_top(top, x[i]);
  } while (top == kUnset && !stream_aborted(sm));
  float sum = stream_square4(x[0], 0.f);
  if (IT > 1 && more) {
#pragma unroll
    for (int i = 1; i < IT; ++i) sum = stream_square4(x[i], sum);
  }
  sum = warp_sum(sum);
  if (lane == 0) sm->ss[warp][0] = sum;
  stream_sync();
  uint4* mine = reinterpret_cast<uint4*>(stream_scratch(sm)) + warp * NC * kStreamWpc * 4;
  float v[kStreamWarps];
#pragma unroll
  for (int s = 0; s < kStreamWarps; ++s) v[s] = sm->ss[s][0];
  const float r = rsqrtf((((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]))) / fk + eps);
#pragma unroll
  for (int i = 0; i < IT; ++i)
    if (i == 0 || more)
      mine[i * 32 + lane] = make_uint4(stream_norm_pair(x[i].x, w[i].x, r), stream_norm_pair(x[i].y, w[i].y, r),
                                       stream_norm_pair(x[i].z, w[i].z, r), stream_norm_pair(x[i].w, w[i].w, r));
  __syncwarp();
  const uint4* from = mine + lane;  // window i: four vectors
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int jj = 0; jj < kStreamWpc; ++jj) {
      const int i = c * kStreamWpc + jj;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (c < ncopy && lane < 4) v = from[i * 4];
      frag[i][0][0] = v.x; frag[i][0][1] = v.y; frag[i][0][2] = v.z; frag[i][0][3] = v.w;
    }
}

// One projection phase for this CTA's units.  TM: token class; NACC: weight matrices per tile (gate and up: two); NC:
// copies of a slice whose operand fits the registers; GROUP: what happens to operand and result; FEW: at most four tokens.
template <int TM, int NACC, int NC, int GROUP, bool FEW>
__device__ __forceinline__ void stream_project(const KParams& p, StreamThread& th, StreamPipe& pipe, int kind, int layer) {
  constexpr int NT = stream_token_tiles(TM), WPC = kStreamWpc;
  constexpr int SETS = NT <= 2 ? 2 : 1;  // accumulator sets: consecutive MMAs of a tile do not wait for one another
  constexpr int LPT = 4 / NT;            // lanes per token in the epilogue
  constexpr bool NORM = GROUP != SG_PLAIN;
  constexpr bool PARTS = GROUP == SG_PLAIN && NT == 1;
  constexpr bool CUT = GROUP == SG_PLAIN;  // slices of a tile may go to different CTAs
  StreamMisc* const sm = stream_opaque(th.sm);
  const int wtid = stream_opaque(th.wtid);
  const int half = layer & 1, turn = th.turn, last_turn = th.last_turn;
  const StreamPhase& ph = sm->plan.ph[kind];
  const int warp = wtid >> 5, lane = wtid & 31, T = TM == 1 ? 1 : sm->tokens;
  const int ncopy = ph.ncopy, k = ph.k, n_cols = ph.n, ntiles = ph.ntiles;
  const int nslice = CUT ? ph.nslice : 1, cs = ph.cs, parts = PARTS ? ph.parts : 1;
  const int live = (2 * cs - warp + 7) >> 3;  // 32-element windows of a slice that are this warp's
  const int count = sm->units[kind];
  int slice = CUT ? sm->first_slice[kind] : 0;
  constexpr int COPIES = stream_copies(TM);
  const size_t copy_elems = static_cast<size_t>(TM) * n_cols;
  const bf16* const src = sm->plan.src[kind][turn] + static_cast<size_t>(sm->copy) * TM * k;
  bf16* const dst = sm->plan.dst[kind][turn];
  bf16* const clear = sm->plan.dst[kind][last_turn];
  const bf16* const normw = !NORM ? nullptr : (GROUP == SG_MLP ? sm->lw[half].post_norm : (kind == SP_HEAD ? sm->plan.final_norm : sm->lw[half].input_norm));
  const bool cut = CUT && nslice > 1;
  // Epilogue: a warp finishes whole rows of NT tokens, lanes = row pair (8) x share of the warps' sums x token.
  const int pair = lane & 7, q = (lane >> 3) % LPT, tok = warp * NT + (lane >> 3) / LPT;
  const bool finisher = tok < T && 2 * pair < ph.rows;
  // A fragment address of this lane inside a copy, for the two 16-element steps of its first window
  const int row = (lane & 7) + ((lane >> 3) & 1) * 8;
  // (rows past the tile's last one read the next chunk: results nobody takes).  Four chunks on, the swizzle is the same.
  const int rows = ph.rows, at_row = (warp >> 1) * rows + row;
  const uint32_t copy_step = static_cast<uint32_t>(rows) * 512u;
  uint32_t off[2];
#pragma unroll
  for (int s = 0; s < 2; ++s)
    off[s] = static_cast<uint32_t>(at_row * 128 + ((((warp & 1) * 4 + 2 * s + (lane >> 4)) ^ (at_row & 7)) << 4));

  // The two results of one item, columns col and col + 1 of token `tok`.
  auto residual_at = [&](int col) -> const uint32_t* {
    return reinterpret_cast<const uint32_t*>(sm->plan.res[kind][turn] + sm->copy * copy_elems + stream_place(TM, tok, col));
  };
  auto settled = [&](const uint32_t* at, uint32_t word) -> uint32_t {  // a residual word that was asked for earlier
    while (word == kUnset && !stream_aborted(sm)) word = ld_relaxed_u32(at);
    return word;
  };
  auto store = [&](int col, uint32_t word) {  // the copies are dealt to the lanes that share a token
    constexpr int kept = GROUP == SG_NORM ? 1 : COPIES;
    const size_t at = (GROUP == SG_NORM ? tok * n_cols + col : stream_place(TM, tok, col)) + q * copy_elems;
    if (q < kept) {
#pragma unroll
      for (int c = 0; c < kept; c += LPT) st_relaxed_u32(reinterpret_cast<uint32_t*>(dst + at + c * copy_elems), word);
#pragma unroll
      for (int c = 0; c < kept; c += LPT) st_relaxed_u32(reinterpret_cast<uint32_t*>(clear + at + c * copy_elems), kUnset);
    }
  };
  auto finish_residual = [&](int col, uint32_t old, float a0, float a1) {
    old = settled(residual_at(col), old);
    store(col, pack2(__uint_as_float(old << 16) + bf16_round(a0), __uint_as_float(old & 0xFFFF0000u) + bf16_round(a1)));
  };

  if constexpr (NORM) {
    const int at = lane * 256 + warp * 32;
    if (count > 0 && at < k) asm volatile("prefetch.global.L1 [%0];" ::"l"(normw + at));
  }
  bool fence = GROUP == SG_PLAIN && kind == kStreamFenceMet && stream_is_aside<TM>(sm);  // the layer's fence has not been met yet
  int tile = sm->first_tile[kind];
#pragma unroll 1
  for (int left = count; left > 0;) {  // runs of units of one slice
    uint32_t frag[NC * WPC][NT][4];
    // part `part` of the slice; a slice of several parts (never a normalised one) is fetched again for every tile
    auto fetch = [&](int part) {
      const int at = part * NC * kStreamKb;  // first chunk
      const int chunks = min(cs - at, NC * kStreamKb);
      stream_operand<TM, NC, NORM>(sm, src, T, (chunks + kStreamKb - 1) / kStreamKb, (2 * chunks - warp + 7) >> 3, (slice * cs + at) * kChunkK + warp * 32,
                             wtid, frag);
    };
    if constexpr (!NORM) {
      if (TM == 1 && kind == SP_DOWN && left == count) __nanosleep(kStreamLookLate);
      fetch(0);
    } else if constexpr (TM == 1) {
      stream_operand_spread<NC>(p, sm, src, normw, k, ncopy, live, wtid, frag);
    } else {
      const int kbase = slice * cs * kChunkK + warp * 32;
      uint4 ahead[kStreamWeightsAhead<NT> ? NC * WPC : 1];
      if constexpr (kStreamWeightsAhead<NT>) {
#pragma unroll
        for (int i = 0; i < NC * WPC; ++i) {
          ahead[i] = make_uint4(0u, 0u, 0u, 0u);
          if (i < live) ahead[i] = stream_plain_vec(normw + kbase + i * 256, lane & 3);
        }
      }
      fetch(0);
      if constexpr (FEW) {
        const float sum = stream_squares<NC>(ncopy, frag);
        if ((lane & 3) == 0) sm->ss[warp][lane >> 2] = sum;
      } else {
        float gram[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) gram[n][0] = gram[n][1] = gram[n][2] = gram[n][3] = 0.f;
        stream_gram<NT, NC>(ncopy, frag, gram);
        if (((lane >> 2) >> 1) == (lane & 3)) {  // this lane has the diagonal element of token lane / 4
#pragma unroll
          for (int n = 0; n < NT; ++n)
            sm->ss[warp][n * 8 + (lane >> 2)] = (n & 1) ? (((lane >> 2) & 1) ? gram[n][3] : gram[n][2]) : (((lane >> 2) & 1) ? gram[n][1] : gram[n][0]);
        }
      }
      stream_sync();
      const float fk = static_cast<float>(k), eps = p.eps;
      float r[NT];
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        float v[kStreamWarps];
#pragma unroll
        for (int w = 0; w < kStreamWarps; ++w) v[w] = sm->ss[w][n * 8 + (lane >> 2)];
        r[n] = rsqrtf((((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]))) / fk + eps);
      }
      stream_normalise<NT, NC>(normw, ncopy, live, kbase, wtid, r, ahead, frag);
    }
    const int run = CUT ? min(left, ntiles - tile) : left, last = tile + run;
    left -= run;
    th.trace(EV_B_STAGED);
    const int first = tile;
#pragma unroll 1
    for (; tile < last; ++tile) {
      int col = tile * rows + 2 * pair, col_end = n_cols;  // this lane's pair of output columns
      if constexpr (GROUP == SG_NORM) {  // the tiles of q, k and v start at each matrix's first row
        if (kind == SP_QKV) {
          if (tile >= ph.tile2) col += ph.row2 - ph.tile2 * rows;
          else if (tile >= ph.tile1) col += ph.row1 - ph.tile1 * rows, col_end = ph.row2;
          else col_end = ph.row1;
        }
      }
      const bool mine = finisher && col < col_end;
      uint32_t old = 0u;
      float b0 = 0.f, b1 = 0.f;
      if (mine) {  // requested now, looked at behind the products
        if constexpr (GROUP == SG_PLAIN) {
          if (!cut) old = ld_relaxed_u32(residual_at(col));
        }
        if constexpr (GROUP == SG_NORM) {
          if (kind == SP_QKV && sm->lw[half].bias[0] != nullptr) {
            const int seg = tile >= ph.tile2 ? 2 : (tile >= ph.tile1 ? 1 : 0);
            const bf16* bias = sm->lw[half].bias[seg] + col - (seg == 0 ? 0 : (seg == 1 ? ph.row1 : ph.row2));
            b0 = ldg_bf16(bias);
            b1 = ldg_bf16(bias + 1);
          }
        }
      }
      float acc[NACC][NT][SETS][4];
#pragma unroll
      for (int a = 0; a < NACC; ++a)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int s = 0; s < SETS; ++s) acc[a][n][s][0] = acc[a][n][s][1] = acc[a][n][s][2] = acc[a][n][s][3] = 0.f;
#pragma unroll 1
      for (int part = 0; part < parts; ++part) {
        const int here = PARTS ? min(ncopy - part * NC, NC) : ncopy;
        if (PARTS && parts > 1 && (part > 0 || tile > first)) fetch(part);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (c < here) {
#pragma unroll
          for (int a = 0; a < NACC; ++a) {
            stream_wait(sm, pipe.full(), pipe.parity);
            const uint32_t base = pipe.addr();
#pragma unroll
            for (int jj = 0; jj < WPC; ++jj) {  // windows past the slice meet a zero operand
#pragma unroll
              for (int s = 0; s < 2; ++s) {
                uint32_t af[4];
                ldmatrix_x4(af, base + off[s] + jj * copy_step);
#pragma unroll
                for (int n = 0; n < NT; ++n)
                  mma_bf16_16816(acc[a][n][jj % SETS], af, frag[c * WPC + jj][n][2 * s], frag[c * WPC + jj][n][2 * s + 1]);
              }
            }
            stream_release(pipe, lane);
          }
        }
      }
      }
      // partial sums of the warps: [warp][matrix][token][row]
      float* psum = stream_psum(sm) + (th.pbuf ? kStreamWarps * 2 * TM * kStreamPartPitch : 0);
#pragma unroll
      for (int a = 0; a < NACC; ++a)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int ptok = n * 8 + (lane & 3) * 2 + (e & 1), prow = (lane >> 2) + (e >> 1) * 8;
            float v = acc[a][n][0][e];
            if constexpr (SETS == 2) v += acc[a][n][1][e];
            if (TM > 1 || ptok < TM) psum[((warp * NACC + a) * TM + ptok) * kStreamPartPitch + prow] = v;
          }
      if (GROUP == SG_PLAIN && fence) named_bar_sync(kStreamFencedBarrier, kStreamFenceThreads);
      else stream_sync();
      fence = false;
      float2 sum[NACC];
#pragma unroll
      for (int a = 0; a < NACC; ++a) {
        sum[a] = make_float2(0.f, 0.f);
        if (TM > 1 || tok < TM) {
#pragma unroll
          for (int w = 0; w < kStreamWarps / LPT; ++w) {
            const float2 v = *reinterpret_cast<const float2*>(
                psum + (((q * (kStreamWarps / LPT) + w) * NACC + a) * TM + tok) * kStreamPartPitch + 2 * pair);
            sum[a].x += v.x;
            sum[a].y += v.y;
          }
        }
#pragma unroll
        for (int o = 1; o < LPT; o <<= 1) {
          sum[a].x += __shfl_xor_sync(0xffffffffu, sum[a].x, 8 * o);
          sum[a].y += __shfl_xor_sync(0xffffffffu, sum[a].y, 8 * o);
        }
      }
      if (mine) {
        if (cut) {  // fp32 pair for the tile's owner
          const size_t at = ((static_cast<size_t>(slice) * ntiles + tile) * T + tok) * kStreamRows + 2 * pair;
          if (q == 0) {
            st_relaxed_v2(sm->plan.part[kind][turn] + at, __float_as_uint(sum[0].x), __float_as_uint(sum[0].y));
            st_relaxed_v2(sm->plan.part[kind][last_turn] + at, kUnset, kUnset);
          }
        } else if constexpr (GROUP == SG_PLAIN) {
          finish_residual(col, old, sum[0].x, sum[0].y);
        } else if constexpr (GROUP == SG_MLP) {
          // (the same bits either way; the shorter one with two to eight tokens, 0.5B shape 1 to 1.8 % of a step, others 0 to 0.5: with one
          // and with sixteen the 1.7B shape is 0.3 and 0.5 % slower)
          auto gate = [](float x) { return bf16_round(TM == 8 ? silu_to_bf16(x) : silu(x)); };
          const float s0 = gate(bf16_round(sum[0].x)), s1 = gate(bf16_round(sum[0].y));
          store(col, pack2(s0 * bf16_round(sum[NACC - 1].x), s1 * bf16_round(sum[NACC - 1].y)));
        } else if (kind == SP_QKV) {
          store(col, pack2(sum[0].x + b0, sum[0].y + b1));
        } else if (q == 0) {
          bf16* out = p.logits + static_cast<size_t>(tok) * n_cols + col;
          if ((n_cols & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 3) == 0) {  // logits may begin at any element
            *reinterpret_cast<uint32_t*>(out) = pack2(sum[0].x, sum[0].y);
          } else {
            if (col < n_cols) out[0] = __float2bfloat16_rn(sum[0].x);
            if (col + 1 < n_cols) out[1] = __float2bfloat16_rn(sum[0].y);
          }
        }
      }
      if (TM <= 8) th.pbuf ^= 1;  // two buffers: the next tile's sums go to the other one
      else stream_sync();          // one buffer: everybody has read it
    }
    ++slice;
    tile = 0;
  }

  if (GROUP == SG_PLAIN && fence) named_bar_sync(kStreamFencedBarrier, kStreamFenceThreads);  // a CTA without a unit of down_proj
  if constexpr (CUT) {
    if (cut) {  // this CTA's share of the tiles is summed over the slices
      const int j0 = static_cast<int>(static_cast<long long>(ntiles) * sm->cta / sm->grid);
      const int j1 = static_cast<int>(static_cast<long long>(ntiles) * (sm->cta + 1) / sm->grid);
      const float* const part = sm->plan.part[kind][turn];
#pragma unroll 1
      for (int own = j0; own < j1; ++own) {
        const int col = own * rows + 2 * pair;
        const size_t stride = static_cast<size_t>(ntiles) * T * kStreamRows;
        const float* at = part + (static_cast<size_t>(own) * T + tok) * kStreamRows + 2 * pair;
        float a0 = 0.f, a1 = 0.f;
        uint32_t old = 0u;
        if (finisher && col < n_cols) {
          old = ld_relaxed_u32(residual_at(col));
#pragma unroll 1
          for (int s = q; s < nslice; s += 2 * LPT) {  // two slices per lane in flight, added in slice order
            const bool two = s + LPT < nslice;
            uint2 v0, v1 = make_uint2(0u, 0u);
            do {
              v0 = ld_relaxed_v2(at + s * stride);
              if (two) v1 = ld_relaxed_v2(at + (s + LPT) * stride);
            } while (max(max(v0.x, v0.y), max(v1.x, v1.y)) == kUnset && !stream_aborted(sm));
            a0 = (a0 + __uint_as_float(v0.x)) + __uint_as_float(v1.x);
            a1 = (a1 + __uint_as_float(v0.y)) + __uint_as_float(v1.y);
          }
        }
#pragma unroll
        for (int o = 1; o < LPT; o <<= 1) {
          a0 += __shfl_xor_sync(0xffffffffu, a0, 8 * o);
          a1 += __shfl_xor_sync(0xffffffffu, a1, 8 * o);
        }
        if (finisher && col < n_cols) finish_residual(col, old, a0, a1);
      }
    }
  }
  th.trace(EV_PHASE_DONE);
}

}  // namespace mk
