// Decode attention of the streaming kernel: RoPE, KV append and softmax(q K^T) V over the cache tiles that the
// producer streams through the ring, started before the step's q exists.
//
// A tile's slot holds [64-dimension chunk][position][128 B], 128-byte swizzled, for `hpu` adjacent KV heads.  Warp w
// works for KV head w % hpu and takes every (8 / hpu)-th block of 16 positions; it keeps the running maximum, sum and
// value sums of its head's query heads in registers (one pass over the cache: scores and values of a tile are used as
// soon as they are there), so that neither the block nor another CTA is involved until a part is finished.  Both
// products run on mma.sync m16n8k16:
//   scores: D[16 positions][query heads] = K tile (ldmatrix)         x q[dims][heads]
//   values: D[16 dims][heads]           += V tile^T (ldmatrix.trans) x p[positions][heads]
// where p's B fragment is the transpose of the score fragment (movmatrix).  The new position is not in the cache
// yet: the warp whose block holds it writes its rows into the tile (and into the caches) before it reads them.
//
// What comes behind the last tile is a chain of dependent instructions that every CTA's o_proj waits for, as is all of a context of
// one tile, so its length counts: no value sums for blocks that hold no position, one exchange of statistics instead of two, the
// warps' sums weighed in every lane instead of passed along, as many stores as there are copies and no loop.  Of the 2.9 us from
// the first score to the last result of a context of 49 positions (135M shape, by clock) 1.4 are left; a step, us: 135M, one
// sequence at 48 447 -> 407, 18 at 55 790 -> 702; 0.5B, one at 99 467 -> 447; 1.7B, one at 1024 745 -> 731, three at 777 827 -> 812, six of up
// to 1500 975 -> 927, sixteen at 1024 1425 -> 1404, 32 at 500 1728 -> 1705.  The same bits.
#pragma once
#include "stream_common.cuh"

namespace mk {

__device__ __forceinline__ float word_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float word_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// Rotate the pairs of adjacent elements lo (dimensions i, i + 1) and hi (their partners, head_dim / 2 further on).  Every
// operation of rope_pair rounds to bf16, so it is one packed instruction for two elements.
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ void stream_rope(uint32_t& lo, uint32_t& hi, uint32_t c, uint32_t s, int style) {
  const uint32_t a = mul_bf16x2(lo, c), b = mul_bf16x2(hi, s);
  if (style == MK_ROPE_HALF_SWAP) {
    hi = add_bf16x2(b, a);
  } else {
    hi = add_bf16x2(mul_bf16x2(hi, c), mul_bf16x2(lo, s));
  }
  lo = sub_bf16x2(a, b);
}

// HD / 8 words (dimensions 8i + 2t, + 1) of one head, once they are set.
template <int HD>
__device__ __forceinline__ void stream_head_words(StreamMisc* sm, const bf16* head, int t, bool live, uint32_t (&x)[HD / 8]) {
  const uint32_t* at = reinterpret_cast<const uint32_t*>(head) + t;
#pragma unroll
  for (int i = 0; i < HD / 8; ++i) x[i] = live ? kUnset : 0u;
  bool again;
  do {
    again = false;
#pragma unroll
    for (int i = 0; i < HD / 8; ++i)
      if (x[i] == kUnset) x[i] = ld_relaxed_u32(at + i * 4);
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) again = again || x[i] == kUnset;
  } while (again && !stream_aborted(sm));
}

// a / b from 1 / b and one correction by the remainder (Markstein, 1990): the quotient rounded to nearest wherever that and the
// remainder are normal numbers.  A division takes a branch of its own for a = 0, and a short context has many: positions
// behind it weigh nothing (a context of one tile: 135M shape, 16 steps 8644 -> 8094 us, 0.5B 546 -> 520).
__host__ __device__ __forceinline__ float stream_quotient(float a, float b, float inverse) {
  const float q = a * inverse;
  return fmaf(fmaf(-q, b, a), inverse, q);
}

template <int TM, int HD>
__device__ __forceinline__ void stream_attention(const KParams& p, StreamThread& th, StreamPipe& pipe, int layer) {
  StreamMisc* const sm = stream_opaque(th.sm);
  const int wtid = stream_opaque(th.wtid);
  const bf16* const qkv = sm->plan.dst[SP_QKV][th.turn];  // [sequence][q | k | v], plain order
  const uint32_t stamp = p.att_epoch + static_cast<uint32_t>(layer) + 1u;
  float* const scratch = reinterpret_cast<float*>(stream_scratch(sm));  // [slot of a (warp, head)][HD + 2]
  constexpr int KS = HD / 16;    // 16-dimension steps of the score product = dimension tiles of the value product
  constexpr int DPL = HD / 32;   // output dimensions per lane when a warp handles one head
  constexpr int BPW = 128 / HD;  // blocks of 16 positions per warp and tile
  const int warp = wtid >> 5, lane = wtid & 31, lg = lane >> 2, lt = lane & 3;
  const int gs = p.q_heads / p.kv_heads, hpu = p.stream_hpu, tk = p.stream_tile_keys;
  const int nsplit = kStreamWarps / hpu, hh = warp & (hpu - 1), split = warp / hpu;
  const int heads = gs * hpu;  // query heads of a group: at most eight
  const int q_size = p.q_heads * HD, kv_size = p.kv_heads * HD, qkv_ld = p.qkv_ld;
  const uint32_t chunk_bytes = static_cast<uint32_t>(tk) * 128u;
  const float scale = p.att_scale * 1.4426950408889634f;  // scores in units of log2
  const int style = p.rope_style;
  constexpr int kRow = HD + 2;
  float4* const stats = reinterpret_cast<float4*>(scratch + kStreamWarps * gs * kRow);  // behind the sums: [KV head][split][pair of query heads]

  // Lists of parts, mostly one (every layer has at least one, if empty).
  int count = stream_next_list(sm, th.list);
#pragma unroll 1
  for (int part = 0;; ++part) {
    if (part == (count & (kStreamMoreParts - 1))) {
      ++th.list;
      if (!(count & kStreamMoreParts)) break;
      stream_sync();  // everybody is done with the list: the helper may write the next but one
      if (wtid == 0) *reinterpret_cast<volatile int*>(&sm->seg_taken) = th.list;
      count = stream_next_list(sm, th.list);
      part = -1;
      continue;
    }
    if (TM > 8 && part > 0) {  // the scratch has been read
      if (nsplit == 1) __syncwarp();
      else stream_sync();
    }
    const StreamSegment sg = sm->seg[th.list & 1][part];
    const int len = sg.len;  // the new position
    const int kvh = sg.group * hpu + hh, pos = sm->pos_s[sg.b];
    const bf16* row = qkv + static_cast<size_t>(sg.b) * qkv_ld;

    // q of this warp's KV head, rotated: B fragments, lane lg = query head of the KV head
    uint32_t cs[HD / 16], sn[HD / 16], q[HD / 8];
    {
      const uint32_t* ct = reinterpret_cast<const uint32_t*>(p.cos_t + static_cast<size_t>(pos) * HD) + lt;
      const uint32_t* st = reinterpret_cast<const uint32_t*>(p.sin_t + static_cast<size_t>(pos) * HD) + lt;
#pragma unroll
      for (int i = 0; i < HD / 16; ++i) {
        cs[i] = __ldg(ct + i * 4);
        sn[i] = __ldg(st + i * 4);
      }
    }
    // The part that ends the context has the new position in its last tile: the warp of its block fetches the new key
    // and value, a word and its rotation partner per lane.
    const int new_block = (len % tk) >> 4;  // block of the tile
    const bool own_warp = sg.t1 == sg.nt && new_block % nsplit == split, owner = own_warp && lane < HD / 4;
    uint32_t kn[2] = {0u, 0u}, vn[2] = {0u, 0u}, kc = 0u, ks = 0u;
    const uint32_t* const kw = reinterpret_cast<const uint32_t*>(row + q_size + kvh * HD) + lane;
    if (owner) {
      kc = __ldg(reinterpret_cast<const uint32_t*>(p.cos_t + static_cast<size_t>(pos) * HD) + lane);
      ks = __ldg(reinterpret_cast<const uint32_t*>(p.sin_t + static_cast<size_t>(pos) * HD) + lane);
      kn[0] = ld_relaxed_u32(kw);
      kn[1] = ld_relaxed_u32(kw + HD / 4);
      vn[0] = ld_relaxed_u32(kw + kv_size / 2);
      vn[1] = ld_relaxed_u32(kw + kv_size / 2 + HD / 4);
    }
    stream_head_words<HD>(sm, row + (kvh * gs + min(lg, gs - 1)) * HD, lt, lg < gs, q);
#pragma unroll
    for (int i = 0; i < HD / 16; ++i) stream_rope(q[i], q[i + HD / 16], cs[i], sn[i], style);
    if (owner) {
      while (max(max(kn[0], kn[1]), max(vn[0], vn[1])) == kUnset && !stream_aborted(sm)) {
        kn[0] = ld_relaxed_u32(kw);
        kn[1] = ld_relaxed_u32(kw + HD / 4);
        vn[0] = ld_relaxed_u32(kw + kv_size / 2);
        vn[1] = ld_relaxed_u32(kw + kv_size / 2 + HD / 4);
      }
      stream_rope(kn[0], kn[1], kc, ks, style);
      const size_t cell = (static_cast<size_t>(sg.b) * p.capacity + len) * kv_size + kvh * HD;  // in-kernel KV append
      uint32_t* const kd = reinterpret_cast<uint32_t*>(static_cast<bf16*>(p.kc[layer]) + cell) + lane;
      uint32_t* const vd = reinterpret_cast<uint32_t*>(static_cast<bf16*>(p.vc[layer]) + cell) + lane;
      kd[0] = kn[0];
      kd[HD / 4] = kn[1];
      vd[0] = vn[0];
      vd[HD / 4] = vn[1];
    }
    // Write a row of the new position (two words per lane) into this head's part of the tile at `base`.
    auto patch = [&](uint32_t base, const uint32_t (&w)[2]) {
      if (owner) {
        const int key = len % tk;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int d = 2 * lane + i * (HD / 2);
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(base + (d >> 6) * chunk_bytes + key * 128 + ((((d & 63) >> 3) ^ (key & 7)) << 4) + (d & 7) * 2), "r"(w[i]) : "memory");
        }
      }
      __syncwarp();
    };

    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};  // of query heads 2 lt, 2 lt + 1; l: this lane's positions only
    float o[KS][4];
#pragma unroll
    for (int d = 0; d < KS; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
    th.trace(EV_ATT_INPUTS);

#pragma unroll 1
    for (int tl = sg.t0; tl < sg.t1; ++tl) {
      const int key0 = tl * tk;
      const bool patched = own_warp && tl == sg.nt - 1;
      // Blocks behind the new position's meet no values: of a short context's only tile that is most of them.
      const int blocks = ((len - key0) >> 4) - split;  // of this warp's: block bi is live if bi * nsplit <= blocks
      // --- scores of this warp's blocks of the tile (two at most)
      float s[BPW][4];
      stream_wait(sm, pipe.full(), pipe.parity);
      {
        const uint32_t base = pipe.addr() + static_cast<uint32_t>(hh) * (HD / 64) * chunk_bytes;
        if (patched) patch(base, kn);
#pragma unroll
        for (int bi = 0; bi < BPW; ++bi) {
          s[bi][0] = s[bi][1] = s[bi][2] = s[bi][3] = 0.f;
          const int key = (split + bi * nsplit) * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
          const uint32_t krow = base + static_cast<uint32_t>(key) * 128u;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
            uint32_t af[4];
            ldmatrix_x4(af, krow + (ks >> 2) * chunk_bytes + ((((ks & 3) * 2 + (lane >> 4)) ^ (key & 7)) << 4));
            mma_bf16_16816(s[bi], af, q[2 * ks], q[2 * ks + 1]);
          }
        }
      }
      if (patched) fence_proxy_async_smem();  // the next copy into this slot comes after the stores above
      stream_release(pipe, lane);
      float mt[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int bi = 0; bi < BPW; ++bi) {
        const int key = key0 + (split + bi * nsplit) * 16 + lg;
        const bool v0 = key <= len, v1 = key + 8 <= len;
        s[bi][0] = v0 ? bf16_round(s[bi][0]) * scale : -INFINITY;
        s[bi][1] = v0 ? bf16_round(s[bi][1]) * scale : -INFINITY;
        s[bi][2] = v1 ? bf16_round(s[bi][2]) * scale : -INFINITY;
        s[bi][3] = v1 ? bf16_round(s[bi][3]) * scale : -INFINITY;
        mt[0] = fmaxf(mt[0], fmaxf(s[bi][0], s[bi][2]));
        mt[1] = fmaxf(mt[1], fmaxf(s[bi][1], s[bi][3]));
      }
#pragma unroll
      for (int x = 4; x < 32; x <<= 1) {
        mt[0] = fmaxf(mt[0], __shfl_xor_sync(0xffffffffu, mt[0], x));
        mt[1] = fmaxf(mt[1], __shfl_xor_sync(0xffffffffu, mt[1], x));
      }
      if (sg.nt == 1) {
        // The whole context is this tile: the warps exchange maximum and sum first, and the probabilities are
        // normalised before they are rounded, as the reference's are.
        float own[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float safe = mt[h] == -INFINITY ? 0.f : mt[h];
          own[h] = 0.f;
#pragma unroll
          for (int bi = 0; bi < BPW; ++bi) own[h] += ex2(s[bi][h] - safe) + ex2(s[bi][h + 2] - safe);
        }
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) {
          own[0] += __shfl_xor_sync(0xffffffffu, own[0], x);
          own[1] += __shfl_xor_sync(0xffffffffu, own[1], x);
        }
        // A warp that holds its heads' whole context alone has nothing to exchange.
        float4* const stat = stats + hh * nsplit * 4 + lt;
        if (nsplit > 1) {
          if (lg == 0) stat[split * 4] = make_float4(mt[0], own[0], mt[1], own[1]);
          stream_sync();
        }
        if (blocks >= 0) {
          float4 all[8];
#pragma unroll
          for (int s8 = 0; s8 < 8; ++s8) {
            all[s8] = make_float4(-INFINITY, 0.f, -INFINITY, 0.f);
            if (nsplit == 1) {
              if (s8 == 0) all[s8] = make_float4(mt[0], own[0], mt[1], own[1]);
            } else if (s8 < nsplit) {
              all[s8] = stat[s8 * 4];
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h == 1 && gs == 1) continue;  // nobody's head
            float top = -INFINITY, total = 0.f;
#pragma unroll
            for (int s8 = 0; s8 < 8; ++s8) top = fmaxf(top, h == 0 ? all[s8].x : all[s8].z);
#pragma unroll
            for (int s8 = 0; s8 < 8; ++s8) total = fmaf(h == 0 ? all[s8].y : all[s8].w, ex2((h == 0 ? all[s8].x : all[s8].z) - top), total);
            m[h] = top;
            l[h] = (split == 0 && lg == 0) ? 1.f : 0.f;  // the parts are only to be added
            const float inverse = 1.f / total;
#pragma unroll
            for (int bi = 0; bi < BPW; ++bi) {
              if (bi * nsplit > blocks) continue;
              s[bi][h] = bf16_round(stream_quotient(ex2(s[bi][h] - top), total, inverse));
              s[bi][h + 2] = bf16_round(stream_quotient(ex2(s[bi][h + 2] - top), total, inverse));
            }
          }
        }
      } else if (blocks >= 0) {
        float alpha[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float mn = fmaxf(m[h], mt[h]);
          const float safe = mn == -INFINITY ? 0.f : mn;  // nothing seen yet: every exponential is zero
          alpha[h] = ex2(m[h] - safe);
          m[h] = mn;
          l[h] *= alpha[h];
#pragma unroll
          for (int bi = 0; bi < BPW; ++bi) {
            s[bi][h] = ex2(s[bi][h] - safe);
            s[bi][h + 2] = ex2(s[bi][h + 2] - safe);
            l[h] += s[bi][h] + s[bi][h + 2];
          }
        }
#pragma unroll
        for (int d = 0; d < KS; ++d) {
          o[d][0] *= alpha[0];
          o[d][1] *= alpha[1];
          o[d][2] *= alpha[0];
          o[d][3] *= alpha[1];
        }
      }
      // --- value sums
      stream_wait(sm, pipe.full(), pipe.parity);
      if (blocks >= 0) {
        const uint32_t base = pipe.addr() + static_cast<uint32_t>(hh) * (HD / 64) * chunk_bytes;
        if (patched) {
          // positions past the context meet zero probabilities, but what the cache holds there must be finite for
          // the product to be zero: clear those rows of the new position's block
          const int piece = lane % (HD / 8), block0 = (len - key0) & ~15;
#pragma unroll 1
          for (int r = (len & 15) + 1 + lane / (HD / 8); r < 16; r += 32 / (HD / 8)) {
            const int key = block0 + r;
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(base + (piece >> 3) * chunk_bytes + key * 128 + ((piece & 7) << 4)), "r"(0u) : "memory");
          }
          patch(base, vn);
        }
#pragma unroll
        for (int bi = 0; bi < BPW; ++bi) {
          if (bi * nsplit > blocks) continue;
          // probabilities as a bf16 and the bf16 of what it leaves out: they are not normalised yet, so one rounding here
          // would not be the reference's, and the tensor cores have time for both
          const uint32_t w0 = pack2(s[bi][0], s[bi][1]), w1 = pack2(s[bi][2], s[bi][3]);
          const uint32_t b0 = movmatrix_trans(w0), b1 = movmatrix_trans(w1);
          const uint32_t c0 = movmatrix_trans(pack2(s[bi][0] - word_lo(w0), s[bi][1] - word_hi(w0)));
          const uint32_t c1 = movmatrix_trans(pack2(s[bi][2] - word_lo(w1), s[bi][3] - word_hi(w1)));
          const int key = (split + bi * nsplit) * 16 + (lane & 7) + (lane >> 4) * 8;
          const uint32_t vrow = base + static_cast<uint32_t>(key) * 128u;
#pragma unroll
          for (int d = 0; d < KS; ++d) {
            uint32_t af[4];
            ldmatrix_x4_trans(af, vrow + (d >> 2) * chunk_bytes + ((((d & 3) * 2 + ((lane >> 3) & 1)) ^ (key & 7)) << 4));
            mma_bf16_16816(o[d], af, b0, b1);
            mma_bf16_16816(o[d], af, c0, c1);
          }
        }
        if (patched) fence_proxy_async_smem();
      }
      stream_release(pipe, lane);
    }
    th.trace(EV_ATT_VALUES);

#pragma unroll
    for (int x = 4; x < 32; x <<= 1) {
      l[0] += __shfl_xor_sync(0xffffffffu, l[0], x);
      l[1] += __shfl_xor_sync(0xffffffffu, l[1], x);
    }
    // --- the warps' sums, head by head: one warp per query head, HD / 32 adjacent dimensions per lane
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = 2 * lt + h;
      if (n < gs) {
        float* mine = scratch + (split * heads + hh * gs + n) * kRow;
#pragma unroll
        for (int d = 0; d < KS; ++d) {
          mine[d * 16 + lg] = o[d][h];
          mine[d * 16 + lg + 8] = o[d][h + 2];
        }
        if (lg == 0) {
          mine[HD] = m[h];
          mine[HD + 1] = l[h];
        }
      }
    }
    if (nsplit == 1) __syncwarp();
    else stream_sync();
    bf16* const attn = sm->plan.attn[th.turn];
    bf16* const clear = sm->plan.attn[th.last_turn];
    const int h0 = nsplit == 1 ? hh * gs : warp, h1 = nsplit == 1 ? h0 + gs : min(warp + 1, heads);
#pragma unroll 1
    for (int hl = h0; hl < h1; ++hl) {
      // Every lane weighs all warps' sums itself (a warp that saw no position has -inf: weight zero): the block waits for this
      // warp, and a maximum and a sum passed from lane to lane are a chain of eight exchanges.
      const float* const mine = scratch + hl * kRow;
      const int split_row = heads * kRow;
      float2 st[8];
#pragma unroll
      for (int s8 = 0; s8 < 8; ++s8) {
        st[s8] = make_float2(-INFINITY, 0.f);
        if (s8 < nsplit) st[s8] = *reinterpret_cast<const float2*>(mine + s8 * split_row + HD);
      }
      float mm = fmaxf(fmaxf(fmaxf(st[0].x, st[1].x), fmaxf(st[2].x, st[3].x)), fmaxf(fmaxf(st[4].x, st[5].x), fmaxf(st[6].x, st[7].x)));
      const float safe = mm > -INFINITY ? mm : 0.f;  // (a part may hold nothing but scores of -inf: its weights are zero)
      float acc[DPL];
#pragma unroll
      for (int i = 0; i < DPL; ++i) acc[i] = 0.f;
#pragma unroll
      for (int s8 = 0; s8 < 8; ++s8) {
        const float w = ex2(st[s8].x - safe);
        st[s8].y = __fmul_rn(st[s8].y, w);  // (rounded before it is added)
        if (s8 < nsplit) {
#pragma unroll
          for (int i = 0; i < DPL / 2; ++i) {
            const float2 v = *reinterpret_cast<const float2*>(mine + s8 * split_row + lane * DPL + 2 * i);
            acc[2 * i] = fmaf(w, v.x, acc[2 * i]);
            acc[2 * i + 1] = fmaf(w, v.y, acc[2 * i + 1]);
          }
        }
      }
      float ll = ((st[0].y + st[1].y) + (st[2].y + st[3].y)) + ((st[4].y + st[5].y) + (st[6].y + st[7].y));
      const int head = sg.group * heads + hl;
      unsigned long long* rec = sm->plan.rec + (static_cast<size_t>(sg.b) * p.q_heads + head) * kStreamMaxSegments * kRow;
      const unsigned long long tag = static_cast<unsigned long long>(stamp) << 32;
      if (sg.seg > 0) {  // a later part of the context: hand it to the CTA of the first one
        unsigned long long* to = rec + sg.seg * kRow;
#pragma unroll
        for (int i = 0; i < DPL; ++i) st_relaxed_u64(to + lane * DPL + i, tag | __float_as_uint(acc[i]));
        if (lane == 0) {
          st_relaxed_u64(to + HD, tag | __float_as_uint(mm));
          st_relaxed_u64(to + HD + 1, tag | __float_as_uint(ll));
        }
        continue;
      }
#pragma unroll 1
      for (int s0 = 1; s0 < sg.nseg; s0 += 4) {
        unsigned long long w[4][DPL + 2];
#pragma unroll
        for (int s4 = 0; s4 < 4; ++s4)
#pragma unroll
          for (int i = 0; i < DPL + 2; ++i) w[s4][i] = tag;
        bool again;
        do {  // four parts at a time: all loads of a pass are issued before any is looked at
          again = false;
#pragma unroll
          for (int s4 = 0; s4 < 4; ++s4)
            if (s0 + s4 < sg.nseg) {
              const unsigned long long* part = rec + (s0 + s4) * kRow;
#pragma unroll
              for (int i = 0; i < DPL; i += 2) ld_relaxed_v2_u64(part + lane * DPL + i, w[s4][i], w[s4][i + 1]);
              ld_relaxed_v2_u64(part + HD, w[s4][DPL], w[s4][DPL + 1]);
            }
#pragma unroll
          for (int s4 = 0; s4 < 4; ++s4)
            if (s0 + s4 < sg.nseg) {
#pragma unroll
              for (int i = 0; i < DPL + 2; ++i) again = again || static_cast<uint32_t>(w[s4][i] >> 32) != stamp;
            }
        } while (again && !stream_aborted(sm));
#pragma unroll
        for (int s4 = 0; s4 < 4; ++s4)
          if (s0 + s4 < sg.nseg) {
            const float om = __uint_as_float(static_cast<uint32_t>(w[s4][DPL])), pl = __uint_as_float(static_cast<uint32_t>(w[s4][DPL + 1]));
            const float mn = fmaxf(mm, om);
            const float safe = mn > -INFINITY ? mn : 0.f;
            const float wa = ex2(mm - safe), wb = ex2(om - safe);
            mm = mn;
            ll = ll * wa + pl * wb;
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[i] = acc[i] * wa + __uint_as_float(static_cast<uint32_t>(w[s4][i])) * wb;
          }
      }
      constexpr int copies = stream_copies(TM);
      bf16* const out = attn + stream_place(TM, sg.b, head * HD + lane * DPL);
      bf16* const reset = clear + stream_place(TM, sg.b, head * HD + lane * DPL);
      // A word is two adjacent columns; the next two of a lane, of the same group of eight, lie 8 elements on.
#pragma unroll
      for (int i = 0; i < DPL / 2; ++i) {
        const uint32_t word = pack2(acc[2 * i] / ll, acc[2 * i + 1] / ll);
#pragma unroll
        for (int c = 0; c < copies; ++c) st_relaxed_u32(reinterpret_cast<uint32_t*>(out + static_cast<size_t>(c) * TM * q_size + 8 * i), word);
      }
#pragma unroll
      for (int i = 0; i < DPL / 2; ++i)
#pragma unroll
        for (int c = 0; c < copies; ++c) st_relaxed_u32(reinterpret_cast<uint32_t*>(reset + static_cast<size_t>(c) * TM * q_size + 8 * i), kUnset);
    }
    // The next part's sums come when these have been read.  Behind the last part that is so without a barrier, and the warps that add
    // nothing up could go on; but up to eight tokens they would look for o_proj's operand the whole time, in the way of those who
    // write it (us with the barrier and without: 1.7B shape, one sequence 738 and 742, three 819 and 823, eight 875 and 878, twelve 1056 and
    // 1048, sixteen 1403 and 1399; 135M 411 and 414).
    if (TM <= 8) {
      if (nsplit == 1) __syncwarp();
      else stream_sync();
    }
  }
}

}  // namespace mk
