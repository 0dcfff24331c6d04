// Prompt attention on the fifth-generation tensor cores: what megabake::attention and the prompt pass launch.
//
// A unit is (sequence, query head, block of 128 query tokens).  Tiles of 64 positions go in turn to two groups of four warps;
// a thread has one query row and all 64 scores of its group's tile, so maximum and sum of a row need no other thread, and the
// two groups' statistics and sums meet once, at the end of the unit.  Per tile and group:
//   scores  D[128 queries, 64 positions] = Q . K^T   (tensor memory, read once into registers)
//   values  D[128 queries, head_dim]     = P . V     (P from shared memory, V as it lies in the cache: MN-major), added to
//           sums in registers, which are rescaled where the row's maximum grew
// One warp issues the MMAs: the next tile's scores while a group is at this one's, which keeps both groups busy.  One thread
// brings Q and the tiles with tiled TMA copies (with cp.async two warps took 1200 to 2500 cycles a tile, twice the softmax's).
// Rounding points are those of prompt_unit (prompt_attention.cuh): score = bf16(bf16(q.k) * scale) (+ mask, rounded again),
// fp32 softmax against the running maximum, exp rounded to bf16 for the value product, division by the fp32 sum at the end.
// What bounds it: the chain of a group's tile, one block of eight such warps to an SM (32 heads of 64 x 512 with a mask 12.9 us on
// the device).  From the first look at memory: scores after 1.9 us, then 1.75 a tile of a group (0.45 scores and mask, 0.65
// exponentials, of which 0.27 are the unit's rate, 0.3 sums, 0.35 P and waits), 1.2 exchange, 1.3 quotients and stores.
// A mask with rows on 16-byte boundaries and queries enough (attention_mask_in_tiles) comes by TMA beside the keys and values: a
// thread reading its own row touched 32 lines a request, 2000 cycles of the load unit for a pair of tiles (512: 13.7 -> 12.9 us, 1024
// 41.5 -> 38.2, head size 128 20.5 -> 17.7, a third of it the columns that both groups now finish).  With rows off those boundaries eight
// copies of a residue of the rows each (AM_EIGHTS, attention_mask_in_eights): 500 positions 17.6 -> 13.8, 501 17.6 -> 13.6, 4 x 250 21.9
// -> 19.3, head size 128, 500 21.4 -> 19.4.  (Fetched a row at a time through shared memory 500 came to 15.8 and 501 to 20.4; by two
// warps of their own 27.8.)  What is left keeps the loads.
#pragma once
#include <type_traits>

#include "prompt_attention.cuh"
#include "prompt_plan.h"

namespace mk {

constexpr int kAttnQueries = 128, kAttnKeys = 64;
constexpr int kAttnThreads = 384;  // two groups of four warps; of the third the loader and the MMA warp

// How a mask comes.  In tiles: by TMA beside the keys and values, where its rows begin on 16-byte boundaries.  In eights: rows that lie
// eight apart begin at the same place within 16 bytes, however long they are, so each of the eight residues is a matrix of its own
// whose rows are 16 klen bytes apart, and a copy that begins on the boundary before a row's first element is wide enough to hold 64 of
// them from any element on.  Otherwise with loads of each thread's row.
enum { AM_LOADS = 0, AM_TILES = 1, AM_EIGHTS = 2 };
constexpr int kMaskBox = kAttnKeys + 8, kMaskRows = kAttnQueries / 8 + 1;  // elements and rows of a copy of one residue
constexpr int kMaskRegion = (kMaskRows * kMaskBox * 2 + 127) / 128 * 128;

template <int HD, int MASK = AM_LOADS>
struct AttnTc {
  static constexpr int kChunks = HD / 64;                         // 64-dimension chunks of a row
  static constexpr int kStages = HD == 64 ? (MASK == AM_EIGHTS ? 4 : (MASK == AM_TILES ? 5 : 6)) : 3;
  static constexpr int kKeys = 2 * kChunks * kAttnKeys * 128;     // a K and a V tile
  static constexpr int kTile = kKeys + (MASK == AM_EIGHTS ? 8 * kMaskRegion : (MASK == AM_TILES ? kAttnQueries * 128 : 0));
  static constexpr int kArrives = kKeys + (MASK == AM_EIGHTS ? 8 * kMaskRows * kMaskBox * 2 : (MASK == AM_TILES ? kAttnQueries * 128 : 0));  // bytes
  static constexpr int kQ = kChunks * kAttnQueries * 128, kP = kAttnQueries * 128;
  static constexpr int kSmem = 1024 + kQ + 2 * kP + kStages * kTile;
  static constexpr int kColumns = HD == 64 ? 256 : 512;           // 2 x 64 of scores, 2 x head_dim of values
  // The groups' exchange at the end of a unit, 2 x [head_dim / 2 + 2][128] fp32, takes the place of Q, P and (head size 128) a stage.
  static_assert((HD + 4) * 128 * 4 <= kQ + 2 * kP + kTile, "exchange");
  static_assert(kSmem <= 232448, "shared memory");
};

struct AttnTcMisc {
  uint64_t qfull, kvfull[8], kvempty[8], sfull[2], sfree[2], pfull[2], pvfull[2];
  uint32_t tmem_base;
  int abort;
};

// Descriptors of a launch's operands, rows of 64-element chunks: (64, rows, chunks of all heads, sequences).  Rows past the last
// one read as zeros.
struct AttnTcMaps {
  CUtensorMap q, k, v, mask[8];  // mask: (positions, queries, sequences), or of each residue (positions, every eighth row)
  int q_ok;     // the queries begin on a 16-byte boundary; otherwise their rows are fetched with plain loads
  int mask_by;  // AM_*
};

// B operand stored with its N dimension contiguous: 64-element chunks [8 rows of K][128 B], 128-byte swizzle.  Rows of K in
// groups of eight are 1024 bytes apart (stride offset), chunks of N `chunk_bytes` (leading offset).
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t chunk_bytes) {
  return umma_desc_sw128(smem_addr) - (static_cast<uint64_t>(1) << 16) + (static_cast<uint64_t>(chunk_bytes >> 4) << 16);
}
constexpr uint32_t kIdescBMajorN = 1u << 16;

__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_loaded() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

struct AttnTcWait {
  const PromptGuard* guard;
  AttnTcMisc* misc;
  long long deadline;
};
static __device__ __noinline__ bool attn_give_up(const AttnTcWait& w) {
  if (*reinterpret_cast<volatile int*>(&w.misc->abort)) return true;
  Control* const ctrl = w.guard->ctrl;
  if (ld_relaxed_u32(&ctrl->abort) == 0) {
    if (clock64() < w.deadline) return false;
    if (atomicCAS(&ctrl->status, 0, static_cast<int>(MK_STATUS_TIMEOUT)) == 0) {
      ctrl->where = SITE_ATT_EXCHANGE;
      ctrl->cta = blockIdx.x;
      ctrl->detail = 0;
    }
    atomicExch(&ctrl->abort, 1u);
    __threadfence();
  }
  // whatever was reported first, this is what the op looks for before its next call
  if (w.guard->status_mirror) *w.guard->status_mirror = static_cast<int>(MK_STATUS_TIMEOUT);
  *reinterpret_cast<volatile int*>(&w.misc->abort) = 1;
  return true;
}
__device__ __forceinline__ bool attn_wait(const AttnTcWait& w, uint64_t* bar, uint32_t parity) {
  const uint32_t at = smem_u32(bar);
  uint32_t spins = 0;
  while (!mbar_try_wait(at, parity))
    if ((++spins & w.guard->polls) == 0 && attn_give_up(w)) return false;
  return true;
}

// What every role knows of a unit.
struct AttnTcUnit {
  int b, h, kvh, q0, ntiles;
};
__device__ __forceinline__ AttnTcUnit attn_unit(const AttnArgs& A, int q_heads, int kv_heads, int batch, int i) {
  AttnTcUnit u;
  const int heads = batch * q_heads, qblocks = (A.sq + kAttnQueries - 1) / kAttnQueries;
  const int qb = qblocks - 1 - i / heads, bh = i % heads;  // causal blocks cost in proportion to their index: heaviest first
  u.b = bh / q_heads;
  u.h = bh - u.b * q_heads;
  u.kvh = u.h / (q_heads / kv_heads);
  u.q0 = qb * kAttnQueries;
  const int kend = A.causal ? min(A.klen, u.q0 + kAttnQueries) : A.klen;
  u.ntiles = (kend + kAttnKeys - 1) / kAttnKeys;
  return u;
}

// One thread of warp 8: the queries, then tile t into stage t % kStages (t counts over the launch).
template <int HD, int MASK>
__device__ __forceinline__ void attn_load(const AttnTcMaps& maps, int sq, const AttnTcWait& w, AttnTcMisc* misc, const AttnTcUnit& u, uint32_t q, uint32_t stages,
                                          int base) {
  using T = AttnTc<HD, MASK>;
  const uint64_t policy = l2_policy_evict_normal();
  if (maps.q_ok) {
    mbar_expect_tx(smem_u32(&misc->qfull), T::kQ);
    tma_load_4d(q, &maps.q, 0, u.q0, u.h * T::kChunks, u.b, smem_u32(&misc->qfull), policy);
  }
  for (int t = 0; t < u.ntiles; ++t) {
    const int at = base + t, s = at % T::kStages, use = at / T::kStages;
    if (use > 0 && !attn_wait(w, &misc->kvempty[s], (use - 1) & 1)) return;
    const uint32_t bar = smem_u32(&misc->kvfull[s]), dst = stages + s * T::kTile;
    mbar_expect_tx(bar, T::kArrives);
    tma_load_4d(dst, &maps.k, 0, t * kAttnKeys, u.kvh * T::kChunks, u.b, bar, policy);
    tma_load_4d(dst + T::kKeys / 2, &maps.v, 0, t * kAttnKeys, u.kvh * T::kChunks, u.b, bar, policy);
    if constexpr (MASK == AM_TILES) tma_load_3d(dst + T::kKeys, &maps.mask[0], t * kAttnKeys, u.q0, u.b, bar, policy);
    if constexpr (MASK == AM_EIGHTS)
      for (int j = 0; j < 8; ++j) tma_load_2d(dst + T::kKeys + j * kMaskRegion, &maps.mask[j], t * kAttnKeys, (u.b * sq + u.q0) >> 3, bar, policy);
  }
}

// Warp 10.  `base` and `uses`: tiles of earlier units, all and of each group (uses of the barriers).
template <int HD, int MASK>
__device__ __forceinline__ void attn_mma(const AttnTcWait& w, AttnTcMisc* misc, const AttnTcUnit& u, uint32_t q, uint32_t p, uint32_t stages, uint32_t tmem,
                                         int base, const int* uses) {
  using T = AttnTc<HD, MASK>;
  constexpr uint32_t kScores = umma_idesc_bf16(kAttnQueries, kAttnKeys), kValues = umma_idesc_bf16(kAttnQueries, HD) | kIdescBMajorN;
  auto scores = [&](int t) -> bool {
    const int at = base + t, s = at % T::kStages;
    if (!__all_sync(0xffffffffu, attn_wait(w, &misc->kvfull[s], (at / T::kStages) & 1))) return false;
    tc_fence_after();
    const uint64_t a = umma_desc_sw128(q), b = umma_desc_sw128(stages + s * T::kTile);
    if (elect_one()) {
#pragma unroll
      for (int c = 0; c < T::kChunks; ++c)
#pragma unroll
        for (int x = 0; x < 4; ++x)
          umma_bf16(tmem + (t & 1) * kAttnKeys, a + (c * kAttnQueries * 128 + x * 32) / 16, b + (c * kAttnKeys * 128 + x * 32) / 16, kScores,
                    c + x > 0 ? 1u : 0u);
      umma_commit(smem_u32(&misc->sfull[t & 1]));
    }
    __syncwarp();
    return true;
  };
  for (int t = 0; t < min(2, u.ntiles); ++t)
    if (!scores(t)) return;
  for (int t = 0; t < u.ntiles; ++t) {
    const int g = t & 1, use = uses[g] + (t >> 1);
    if (t + 2 < u.ntiles) {  // the group has this tile's scores in registers
      if (!__all_sync(0xffffffffu, attn_wait(w, &misc->sfree[g], use & 1))) return;
      if (!scores(t + 2)) return;
    }
    if (!__all_sync(0xffffffffu, attn_wait(w, &misc->pfull[g], use & 1))) return;
    tc_fence_after();
    const int s = (base + t) % T::kStages;
    const uint64_t a = umma_desc_sw128(p + g * T::kP), b = umma_desc_mn_sw128(stages + s * T::kTile + T::kKeys / 2, kAttnKeys * 128);
    if (elect_one()) {
#pragma unroll
      for (int x = 0; x < 4; ++x)  // 16 positions: 32 bytes of a row of P, two groups of eight rows of V
        umma_bf16(tmem + 2 * kAttnKeys + g * HD, a + x * 2, b + x * (2048 / 16), kValues, x > 0 ? 1u : 0u);
      umma_commit(smem_u32(&misc->kvempty[s]));
      umma_commit(smem_u32(&misc->pvfull[g]));
    }
    __syncwarp();
  }
}

// The mask of a thread's row for 64 positions from j on, as bf16 pairs.  `wide`: rows begin on 16-byte boundaries.  Otherwise the
// aligned words that hold the elements, shifted into place; past the row's last word it is repeated (those positions are
// masked below).  Plain loads: the kernel that writes the mask may be at work while this one begins, which the read-only path
// does not allow, and no compiler moves them ahead of griddepcontrol.wait.
__device__ __forceinline__ void attn_mask(const bf16* row, int j, int klen, bool wide, uint32_t (&m)[32]) {
  if (wide && j + 64 <= klen) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint4 v = reinterpret_cast<const uint4*>(row + j)[i];
      m[4 * i] = v.x; m[4 * i + 1] = v.y; m[4 * i + 2] = v.z; m[4 * i + 3] = v.w;
    }
  } else {
    const uintptr_t first = reinterpret_cast<uintptr_t>(row + j) & ~static_cast<uintptr_t>(3);
    const uint32_t shift = (reinterpret_cast<uintptr_t>(row + j) & 2) ? 16u : 0u;
    const int last = static_cast<int>((reinterpret_cast<uintptr_t>(row + klen - 1) - first) >> 2);  // the word of the last position
    const unsigned int* const words = reinterpret_cast<const unsigned int*>(first);
    uint32_t word = words[0];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const uint32_t next = words[min(i + 1, last)];
      m[i] = __funnelshift_r(word, next, shift);
      word = next;
    }
  }
}

// The row of a unit that was given up: not a number, so that it cannot pass for a result.
template <int HD>
__device__ __forceinline__ void attn_store_nan(const AttnArgs& A, const AttnTcUnit& u, int row) {
  const int r = u.q0 + row;
  if (r >= A.sq) return;
  uint32_t* const out = reinterpret_cast<uint32_t*>(A.out + u.b * A.out_bstride + static_cast<long long>(r) * A.out_tstride + u.h * A.out_hstride);
#pragma unroll 1
  for (int d = 0; d < HD / 2; ++d) out[d] = 0x7FC07FC0u;
}

// Warps 0 to 7.  A wait that was given up ends the loop; the block barriers behind it are passed all the same.
template <int HD, int MASK>
__device__ __forceinline__ void attn_softmax(const AttnArgs& A, const AttnTcWait& w, AttnTcMisc* misc, const AttnTcUnit& u, uint8_t* smem, uint32_t p,
                                             uint32_t stages, uint32_t tmem, int base, const int* uses, int warp, int lane) {
  using T = AttnTc<HD, MASK>;
  const int g = warp >> 2, quad = warp & 3, row = quad * 32 + lane, r = u.q0 + row;
  const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
  const uint32_t s_at = tmem + lanes + g * kAttnKeys, v_at = tmem + lanes + 2 * kAttnKeys + g * HD;
  const uint32_t p_at = p + g * T::kP + row * 128;
  const bool exact_scale = bf16_round(A.scale) == A.scale;  // head size 64: 1/8; the product is rounded once either way
  const uint32_t scale2 = pack2(A.scale, A.scale);
  const bf16* const mrow = A.mask + (static_cast<long long>(u.b) * A.sq + min(r, A.sq - 1)) * A.klen;
  const bool wide = (A.klen & 7) == 0 && (reinterpret_cast<uintptr_t>(A.mask) & 15) == 0;
  constexpr bool MT = MASK != AM_LOADS;
  const bool fetched = !MT && A.mask;  // the mask comes with plain loads
  bool ok = true, unseen = false;  // unseen: this warp saw nothing of the tile whose sums come next
  float m = -INFINITY, l = 0.f, alpha = 1.f, o[HD];
#pragma unroll
  for (int d = 0; d < HD; ++d) o[d] = 0.f;
  auto add_values = [&](int use) {  // the value sums of this group's last tile
    ok = __all_sync(0xffffffffu, attn_wait(w, &misc->pvfull[g], use & 1));
    if (!ok || unseen) return;
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < HD; c += 32) {
      uint32_t v[32];
      tmem_ld32_async(v_at + c, v);
      tmem_loaded();
#pragma unroll
      for (int d = 0; d < 32; ++d) o[c + d] = fmaf(o[c + d], alpha, __uint_as_float(v[d]));
    }
  };
  // This row's place in its residue's copy, from the word of the tile's first element on, and whether that is the word's second element.
  const int at_row = u.b * A.sq + u.q0 + row, residue = at_row & 7, first_element = (residue * A.klen) & 7;
  const uint32_t eighth = static_cast<uint32_t>(residue * kMaskRegion + ((at_row >> 3) - ((at_row - row) >> 3)) * kMaskBox * 2 + (first_element >> 1) * 4);
  const uint32_t halfword = (first_element & 1) * 16;
  uint32_t x[32];  // the mask of a tile's row, its scores, its probabilities
  if (fetched && g < u.ntiles) attn_mask(mrow, g * kAttnKeys, A.klen, wide, x);
#pragma unroll 1
  for (int t = g; t < u.ntiles && ok; t += 2) {
    const int use = uses[g] + (t >> 1), j0 = t * kAttnKeys;
    // (causal: a warp whose rows all come before the tile has nothing to see in it)
    const bool blind = A.causal && j0 > u.q0 + quad * 32 + 31;
    ok = __all_sync(0xffffffffu, attn_wait(w, &misc->sfull[g], use & 1));
    if (!ok) break;
    tc_fence_after();
    float grown = 1.f;
    // With head size 64 there are registers for the next tile's mask: asked for before this tile's exponentials.
    uint32_t ahead[HD == 64 && !MT ? 32 : 1];
    if (!blind) {
      uint32_t mask_at = 0u;
      if constexpr (MT) {  // (the scores came behind the same copies; this thread's own look makes them visible to it)
        const int at = base + t, s = at % T::kStages;
        ok = __all_sync(0xffffffffu, attn_wait(w, &misc->kvfull[s], (at / T::kStages) & 1));
        mask_at = stages + s * T::kTile + T::kKeys + (MASK == AM_EIGHTS ? eighth : row * 128);
      }
      // What a pair of scores goes through depends on the launch and the tile: straight lines, not three tests a pair.
      auto take = [&](auto exact, auto masked) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t s[32];
          tmem_ld32_async(s_at + c * 32, s);
          if constexpr (MASK == AM_EIGHTS) {
            uint32_t words[17];
#pragma unroll
            for (int i = 0; i < 17; ++i) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(words[i]) : "r"(mask_at + (c * 16 + i) * 4) : "memory");
#pragma unroll
            for (int i = 0; i < 16; ++i) x[c * 16 + i] = __funnelshift_r(words[i], words[i + 1], halfword);
          }
          if constexpr (MASK == AM_TILES) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x[c * 16 + 4 * i]), "=r"(x[c * 16 + 4 * i + 1]), "=r"(x[c * 16 + 4 * i + 2]),
                           "=r"(x[c * 16 + 4 * i + 3]) : "r"(mask_at + (((c * 4 + i) ^ (row & 7)) << 4)) : "memory");
          }
          tmem_loaded();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            uint32_t v = pack2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]));
            if constexpr (decltype(exact)::value) v = mul_bf16x2(v, scale2);
            else v = pack2(__uint_as_float(v << 16) * A.scale, __uint_as_float(v & 0xffff0000u) * A.scale);
            if constexpr (decltype(masked)::value) v = add_bf16x2(v, x[c * 16 + i]);
            x[c * 16 + i] = v;
          }
        }
      };
      if (MT || A.mask) {
        if (exact_scale) take(std::true_type(), std::true_type());
        else take(std::false_type(), std::true_type());
      } else {
        if (exact_scale) take(std::true_type(), std::false_type());
        else take(std::false_type(), std::false_type());
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&misc->sfree[g]));
      if constexpr (HD == 64 && !MT) {
        if (fetched && t + 2 < u.ntiles) attn_mask(mrow, j0 + 2 * kAttnKeys, A.klen, wide, ahead);
      }
      const int last = (A.causal ? min(A.klen - 1, r) : A.klen - 1) - j0;  // the last position of the tile that the row sees
      if (__any_sync(0xffffffffu, last < kAttnKeys - 1)) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (2 * i > last) x[i] = (x[i] & 0xffff0000u) | 0xFF80u;
          if (2 * i + 1 > last) x[i] = (x[i] & 0xffffu) | 0xFF800000u;
        }
      }
      uint32_t top = x[0];
#pragma unroll
      for (int i = 1; i < 32; ++i) top = max_bf16x2(top, x[i]);
      const float n = fmaxf(m, fmaxf(__uint_as_float(top << 16), __uint_as_float(top & 0xffff0000u)));
      // exp(x - n) = 2^((x - n) log2(e)), the difference first: a mask of the lowest finite value must not overflow; a row
      // without a visible key so far: 2^(-inf) = 0
      const float safe = n > -INFINITY ? n : 0.f;
      grown = ex2((m - safe) * kLog2e);
      m = n;
      float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float e0 = ex2((__uint_as_float(x[i] << 16) - safe) * kLog2e), e1 = ex2((__uint_as_float(x[i] & 0xffff0000u) - safe) * kLog2e);
        sum0 += e0;
        sum1 += e1;
        x[i] = pack2(e0, e1);
      }
      l = fmaf(l, grown, sum0 + sum1);
    } else {
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&misc->sfree[g]));
#pragma unroll
      for (int i = 0; i < 32; ++i) x[i] = 0u;
    }
    if (t >= 2) add_values(use - 1);  // and with that the last tile's P has been read
    alpha = grown;
    unseen = blind;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(p_at + ((i ^ (row & 7)) << 4)), "r"(x[4 * i]), "r"(x[4 * i + 1]), "r"(x[4 * i + 2]),
                   "r"(x[4 * i + 3]) : "memory");
    fence_proxy_async_smem();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&misc->pfull[g]));
    if (fetched && t + 2 < u.ntiles) {
      if constexpr (HD == 64 && !MT) {
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = ahead[i];
      } else {
        attn_mask(mrow, j0 + 2 * kAttnKeys, A.klen, wide, x);
      }
    }
  }
  const int mine = (u.ntiles - g + 1) / 2;  // tiles of this group
  if (mine > 0 && ok) add_values(uses[g] + mine - 1);
  // The groups' statistics and sums meet: each finishes half of the columns (divides, rounds once, stores) and leaves the other
  // half to the other.  Every MMA of the unit has finished once both are here: Q, P and the tiles' stages may be written over.
  constexpr int kHalf = HD / 2, kShare = (kHalf + 2) * 128;
  float* const exchange = reinterpret_cast<float*>(smem) + row;
  named_bar_sync(1, 256);
  {
    float* const to = exchange + g * kShare;
    to[0] = m;
    to[128] = l;
    if (g == 0) {
#pragma unroll
      for (int d = 0; d < kHalf; ++d) to[(2 + d) * 128] = o[kHalf + d];
    } else {
#pragma unroll
      for (int d = 0; d < kHalf; ++d) {
        to[(2 + d) * 128] = o[d];
        o[d] = o[kHalf + d];
      }
    }
  }
  named_bar_sync(1, 256);
  if (*reinterpret_cast<volatile int*>(&misc->abort) != 0) {
    if (g == 0) attn_store_nan<HD>(A, u, row);
  } else if (r < A.sq) {
    const float* const from = exchange + (1 - g) * kShare;
    const float m0 = g == 0 ? m : from[0], m1 = g == 0 ? from[0] : m, l0 = g == 0 ? l : from[128], l1 = g == 0 ? from[128] : l, n = fmaxf(m0, m1);
    const float a = m0 > -INFINITY ? expf(m0 - n) : 0.f, b = m1 > -INFINITY ? expf(m1 - n) : 0.f;
    const float total = l0 * a + l1 * b, d = total > 0.f ? total : 1.f;  // a row that sees no key: zeros
    const float inverse = 1.f / d;
    // The first group's share is the one that the fused step adds, whichever group is at it, so that a column's result does not hang on
    // the half it lies in; a quotient by the reciprocal, corrected by its remainder (Markstein, 1990); what is no finite number stays
    // what it is.  (Selects: a copy of the code for each group was no faster.)
    auto quotient = [&](float mine, float theirs) -> float {
      const float v = fmaf(g == 0 ? mine : theirs, a, (g == 0 ? theirs : mine) * b), by = v * inverse;
      return fabsf(by) < INFINITY ? fmaf(fmaf(-by, d, v), inverse, by) : by;
    };
    bf16* const out = A.out + u.b * A.out_bstride + static_cast<long long>(r) * A.out_tstride + u.h * A.out_hstride + g * kHalf;
    const bool vectors = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#pragma unroll
    for (int d0 = 0; d0 < kHalf; d0 += 8) {
      uint32_t x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        x[e] = pack2(quotient(o[d0 + 2 * e], from[(2 + d0 + 2 * e) * 128]), quotient(o[d0 + 2 * e + 1], from[(3 + d0 + 2 * e) * 128]));
      if (vectors) {
        *reinterpret_cast<uint4*>(out + d0) = make_uint4(x[0], x[1], x[2], x[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) reinterpret_cast<uint32_t*>(out + d0)[e] = x[e];
      }
    }
  }
}

template <int HD, int MASK>
__global__ void __launch_bounds__(kAttnThreads, 1)
prompt_attention_tc(const __grid_constant__ AttnArgs A, const __grid_constant__ AttnTcMaps maps, const __grid_constant__ PromptGuard guard, int q_heads,
                    int kv_heads, int batch, int units) {
  using T = AttnTc<HD, MASK>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ AttnTcMisc misc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  grid_dependents_go();
  if (tid == 0) {
    mbar_init(smem_u32(&misc.qfull), 1);
    for (int s = 0; s < T::kStages; ++s) {
      mbar_init(smem_u32(&misc.kvfull[s]), 1);
      mbar_init(smem_u32(&misc.kvempty[s]), 1);
    }
    for (int g = 0; g < 2; ++g) {
      mbar_init(smem_u32(&misc.sfull[g]), 1);
      mbar_init(smem_u32(&misc.sfree[g]), 4);
      mbar_init(smem_u32(&misc.pfull[g]), 4);
      mbar_init(smem_u32(&misc.pvfull[g]), 1);
    }
    misc.abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&maps.q);
    tma_prefetch_desc(&maps.k);
    tma_prefetch_desc(&maps.v);
    if constexpr (MASK != AM_LOADS)
      for (int j = 0; j < (MASK == AM_EIGHTS ? 8 : 1); ++j) tma_prefetch_desc(&maps.mask[j]);
  }
  if (warp == 10) {
    tmem_alloc(smem_u32(&misc.tmem_base), T::kColumns);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&misc.tmem_base);
  const uint32_t q = smem_u32(smem), p = q + T::kQ, stages = p + 2 * T::kP;
  grid_dependency_wait();
  const AttnTcWait w{&guard, &misc, clock64() + guard.timeout_cycles};
  int base = 0, uses[2] = {0, 0}, done = 0;  // tiles of earlier units, and their number
  // The units of this block (one, unless the handle limits its SMs), as one role sees them.
  auto walk = [&](auto role) {
#pragma unroll 1
    for (int i = blockIdx.x; i < units; i += gridDim.x) {
      const AttnTcUnit u = attn_unit(A, q_heads, kv_heads, batch, i);
      role(u);
      // Given up or not is one answer for the block: a thread that saw the word set a unit early would not come to this barrier
      // again, and the others would wait there for good.  (Whoever sets the word sees it set.)
      if (named_bar_any(3, kAttnThreads, *reinterpret_cast<volatile int*>(&misc.abort) != 0)) break;
      base += u.ntiles;
      uses[0] += (u.ntiles + 1) / 2;
      uses[1] += u.ntiles / 2;
      ++done;
    }
  };
  // 384 threads x 168 registers at launch = 128 x 72 + 256 x 216: with head size 128 a row of value sums is 128 of them
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 10) {
      walk([&](const AttnTcUnit& u) {
        if (!maps.q_ok) named_bar_sync(2, 288);  // the queries are there
        else if (!__all_sync(0xffffffffu, attn_wait(w, &misc.qfull, done & 1))) return;
        attn_mma<HD, MASK>(w, &misc, u, q, p, stages, tmem, base, uses);
      });
    } else {
      walk([&](const AttnTcUnit& u) {
        if (warp == 8 && lane == 0) {
          // The exchange's plain accesses come before a later unit's copies.  (The operands are complete and visible behind
          // griddepcontrol.wait, to copies too: without a fence for them 128 positions 6.97 -> 6.59 us, 512 12.8 -> 12.6.)
          if (done > 0) fence_proxy_async_smem();
          attn_load<HD, MASK>(maps, A.sq, w, &misc, u, q, stages, base);
        }
        __syncwarp();
      });
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    walk([&](const AttnTcUnit& u) {
      if (!maps.q_ok) {  // [chunk][row][128 B], swizzled; rows past the last one repeat it
        constexpr int kPieces = HD / 8;
        const bf16* const from = A.q + u.b * A.q_bstride + u.h * HD;
#pragma unroll 1
        for (int x = tid; x < kAttnQueries * kPieces; x += 256) {
          const int row = x / kPieces, piece = x % kPieces;
          const bf16* at = from + static_cast<long long>(min(u.q0 + row, A.sq - 1)) * A.q_ld + piece * 8;
          *reinterpret_cast<uint4*>(smem + (piece >> 3) * kAttnQueries * 128 + row * 128 + (((piece & 7) ^ (row & 7)) << 4)) =
              make_uint4(ldcg_u32(at), ldcg_u32(at + 2), ldcg_u32(at + 4), ldcg_u32(at + 6));
        }
        fence_proxy_async_smem();
        named_bar_sync(2, 288);
      }
      attn_softmax<HD, MASK>(A, w, &misc, u, smem, p, stages, tmem, base, uses, warp, lane);
      fence_proxy_async_smem();
    });
    if (tid < kAttnQueries && *reinterpret_cast<volatile int*>(&misc.abort))  // the units behind the one that was given up
      for (int i = blockIdx.x + (done + 1) * gridDim.x; i < units; i += gridDim.x) attn_store_nan<HD>(A, attn_unit(A, q_heads, kv_heads, batch, i), tid);
  }
  if (*reinterpret_cast<volatile int*>(&misc.abort)) prompt_stay();
  tc_fence_before();
  __syncthreads();
  if (warp == 10) {
    tc_fence_after();
    tmem_dealloc(tmem, T::kColumns);
  }
}

}  // namespace mk
