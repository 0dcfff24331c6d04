// The kernels of a prompt pass (prefill without tensor parallelism): per layer RMSNorm, q/k/v projection with RoPE, attention
// (prompt_attention.cuh), o_proj, RMSNorm, gate/up projection with SiLU * up, down_proj; then RMSNorm and the output head.
//
// They are launched one behind the other with programmatic dependent launch: a kernel's CTAs become resident while the one
// before it is at work, set up barriers and tensor memory and fetch their first weights, and wait there
// (griddepcontrol.wait) until everything the kernel before has written is visible.  One persistent kernel with grid barriers
// spent 3 to 4 us per barrier and phase ramp, eight of them a layer.
//
// Projections: D[tokens, rows] = X[tokens, K] . W[rows, K]^T on tcgen05 with the tokens on the MMA's M side, so that a thread
// of the epilogue has one token's row: contiguous outputs (32-byte stores), the two halves of a RoPE pair, gate and up.
// Beyond 128 tokens a CTA pair works on 256 tokens x up to 256 rows (cta_group::2): each CTA brings its own 128 tokens and
// half of the weight rows, which is half of the bytes per product of two CTAs on their own, and L2 is what bounds them.
#pragma once
#include "device_common.cuh"
#include "prompt_attention.cuh"
#include "prompt_plan.h"

namespace mk {

constexpr int kPromptProducers = 2;
constexpr int kPromptEpilogueWarps = 8;
constexpr int kPromptMmaWarp = kPromptProducers, kPromptFirstEpilogue = kPromptProducers + 1;
constexpr int kPromptThreads = (kPromptFirstEpilogue + kPromptEpilogueWarps) * 32;  // copies, MMAs, epilogue
enum { PE_QKV = 0, PE_PARTIAL = 1, PE_SILU = 2, PE_LOGITS = 3 };

// ---------------------------------------------------------------- CTA pairs
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same without ordering memory: what the CTAs wrote to global memory is not waited for.
__device__ __forceinline__ void cluster_sync_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// The address of this CTA's `addr` in the shared memory of the pair's first CTA.
__device__ __forceinline__ uint32_t leader_address(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// A copy into this CTA's shared memory that counts on a barrier of the pair's first CTA (no multicast).
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const void* tmap, int x, int y, int z, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%2, %3, %4}], [%5], %6;"
      ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(policy)
      : "memory");
}

template <int CTAS>
__device__ __forceinline__ void prompt_tmem_alloc(uint32_t smem_dst, uint32_t columns) {
  if constexpr (CTAS == 1) {
    tmem_alloc(smem_dst, columns);
    tmem_relinquish();
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
}
template <int CTAS>
__device__ __forceinline__ void prompt_tmem_dealloc(uint32_t taddr, uint32_t columns) {
  if constexpr (CTAS == 1) tmem_dealloc(taddr, columns);
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}
// The four K = 16 steps of one 64-element chunk.  Descriptors come as their low words (the address, in 16-byte units) and one high
// word: the steps are 32 bytes apart, and no carry leaves the low word.
template <int CTAS>
__device__ __forceinline__ void prompt_mma_chunk(uint32_t d, uint32_t a, uint32_t b, uint32_t high, uint32_t idesc, uint32_t accumulate) {
#define MK_PROMPT_MMA(group)                                                                                            \
  asm volatile(                                                                                                         \
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t.reg .b32 la, lb;\n\t"                                                  \
      "setp.ne.b32 p, %5, 0;\n\t"                                                                                       \
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"                                                              \
      "tcgen05.mma.cta_group::" group ".kind::f16 [%0], da, db, %4, p;\n\t"                                             \
      "add.u32 la, %1, 2;\n\tadd.u32 lb, %2, 2;\n\tmov.b64 da, {la, %3};\n\tmov.b64 db, {lb, %3};\n\t"                  \
      "tcgen05.mma.cta_group::" group ".kind::f16 [%0], da, db, %4, 1;\n\t"                                             \
      "add.u32 la, %1, 4;\n\tadd.u32 lb, %2, 4;\n\tmov.b64 da, {la, %3};\n\tmov.b64 db, {lb, %3};\n\t"                  \
      "tcgen05.mma.cta_group::" group ".kind::f16 [%0], da, db, %4, 1;\n\t"                                             \
      "add.u32 la, %1, 6;\n\tadd.u32 lb, %2, 6;\n\tmov.b64 da, {la, %3};\n\tmov.b64 db, {lb, %3};\n\t"                  \
      "tcgen05.mma.cta_group::" group ".kind::f16 [%0], da, db, %4, 1;\n\t}"                                            \
      ::"r"(d), "r"(a), "r"(b), "r"(high), "r"(idesc), "r"(accumulate) : "memory")
  if constexpr (CTAS == 1) MK_PROMPT_MMA("1");
  else MK_PROMPT_MMA("2");
#undef MK_PROMPT_MMA
}
// Arrive on the barrier, in both CTAs of a pair, once every MMA this thread issued so far has finished.
template <int CTAS>
__device__ __forceinline__ void prompt_commit(uint32_t bar) {
  if constexpr (CTAS == 1) {
    umma_commit(bar);
  } else {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(static_cast<unsigned short>(3)) : "memory");
  }
}

// 32-byte store of eight words: a whole sector per lane.
__device__ __forceinline__ void st_global_v8(void* p, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
               "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}
// 32 lanes x 16 columns of tensor memory, without the wait: several loads fly together.
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- bounded waits
struct PromptWait {
  const PromptGuard* guard;
  long long deadline;
};
__device__ __noinline__ bool prompt_give_up(const PromptWait& w, int site) {
  Control* const ctrl = w.guard->ctrl;
  if (ld_relaxed_u32(&ctrl->abort) != 0) return true;
  if (clock64() < w.deadline) return false;
  if (atomicCAS(&ctrl->status, 0, static_cast<int>(MK_STATUS_TIMEOUT)) == 0) {
    ctrl->where = site;
    ctrl->cta = blockIdx.x;
    ctrl->detail = 0;
    if (w.guard->status_mirror) *w.guard->status_mirror = static_cast<int>(MK_STATUS_TIMEOUT);
  }
  atomicExch(&ctrl->abort, 1u);
  __threadfence();
  return true;
}
__device__ __forceinline__ bool prompt_wait(const PromptWait& w, uint32_t bar, uint32_t parity, int site) {
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity))
    if ((++spins & w.guard->polls) == 0 && prompt_give_up(w, site)) return false;
  return true;
}

// ---------------------------------------------------------------- projections
// A unit is (weight tile, K slice, token tile), the token tile counting fastest: the CTAs that share weights run together.
struct PromptUnit {
  int tile, slice, tt;
};
__device__ __forceinline__ PromptUnit prompt_unit_at(const PromptGemm& g, int unit) {
  PromptUnit u;
  const int piece = unit / g.token_tiles;
  u.tt = unit - piece * g.token_tiles;
  u.tile = piece / g.ksplit;
  u.slice = piece - u.tile * g.ksplit;
  return u;
}

// The copies.  One thread needs 630 cycles for a stage (a wait, an arrival, two or three copies, each a chain of its own), more
// than the MMAs and the copies themselves take: kPromptProducers warps take the stages in turn.  (A producer waits for every
// other use of a slot only; with no fewer stages than producers the use between has been consumed by then, stages being
// consumed in order, and the barrier's parity says which of the two is meant.)
template <int CTAS, int TM>
__device__ __forceinline__ void prompt_producer(const PromptGemm& g, uint8_t* smem, uint32_t full0, uint32_t empty0, int rank, int first, int step,
                                                int producer) {
  const uint64_t weight_policy = g.stream_weights ? l2_policy_evict_first() : l2_policy_evict_normal();
  const uint64_t token_policy = l2_policy_evict_normal();
  const int kb = CTAS == 1 ? g.kb : 1, groups = g.kslice / kb, nmat = g.nmat, stages = g.stages, units = g.units;
  const uint32_t base = smem_u32(smem), stage_bytes = g.stage_bytes, a_bytes = kb * g.a_bytes, b_bytes = g.b_bytes;
  const uint32_t tx = CTAS * stage_bytes;
  const uint32_t count0 = CTAS == 2 ? leader_address(full0) : full0;  // where copies are counted
  const CUtensorMap* const a_map = g.a;
  // Every CTA walks its K slice from a starting point of its own: together the grid's loads spread over the 128-byte columns of
  // the weight rows, which lie a power of two apart.
  const int rotation = static_cast<int>(static_cast<long long>(first) * groups / step);
  struct Place {
    const CUtensorMap *b0, *b1;
    int b_row, a_row, chunk0;
  };
  auto place_of = [&](int unit) -> Place {
    const PromptUnit u = prompt_unit_at(g, unit);
    const int seg = nmat == 2 ? 0 : (u.tile >= g.tile_start[2] ? 2 : (u.tile >= g.tile_start[1] ? 1 : 0));
    Place p;
    p.b0 = seg == 0 ? g.b[0] : (seg == 1 ? g.b[1] : g.b[2]);
    p.b1 = g.b[1];
    p.b_row = (u.tile - (seg == 0 ? 0 : (seg == 1 ? g.tile_start[1] : g.tile_start[2]))) * g.rows + (CTAS == 2 ? rank * (g.rows / 2) : 0);
    p.a_row = u.tt * CTAS * TM + rank * TM;
    p.chunk0 = u.slice * g.kslice;
    return p;
  };
  auto chunk_of = [&](const Place& p, int i) -> int {
    const int at = i + rotation;
    return p.chunk0 + (at >= groups ? at - groups : at) * kb;
  };
  auto copy = [&](uint32_t dst, const CUtensorMap* map, int row, int chunk, uint32_t bar, uint64_t policy) {
    if constexpr (CTAS == 2) tma_load_3d_pair(dst, map, 0, row, chunk, bar, policy);
    else tma_load_3d(dst, map, 0, row, chunk, bar, policy);
  };
  auto load_b = [&](const Place& p, int chunk, int s) {
    if (rank == 0) mbar_expect_tx(full0 + s * 8u, tx);
    uint32_t dst = base + s * stage_bytes + a_bytes;
    const uint32_t bar = count0 + s * 8u;
    for (int c = 0; c < kb; ++c) {
      copy(dst, p.b0, p.b_row, chunk + c, bar, weight_policy);
      dst += b_bytes;
      if (nmat == 2) {
        copy(dst, p.b1, p.b_row, chunk + c, bar, weight_policy);
        dst += b_bytes;
      }
    }
  };
  // the first stages' weights do not depend on the kernel before this one
  const int total = first < units ? ((units - first + step - 1) / step) * groups : 0;
  for (int n = producer; n < min(total, stages); n += kPromptProducers) {
    const int unit = n / groups;
    const Place p = place_of(first + unit * step);
    load_b(p, chunk_of(p, n - unit * groups), n);
  }
  // What the kernels before have written is complete and visible when this wait ends, to copies as to loads, as at any end of a kernel: a
  // proxy fence here is for nothing and takes 0.3 us of every projection (64 tokens of the 1.7B shape 1267 -> 1252 us, 128 1452 -> 1426;
  // 135M, 128 tokens 1077 -> 1034).
  grid_dependency_wait();
  grid_dependents_go();
  const PromptWait w{&g.guard, clock64() + g.guard.timeout_cycles};
  bool ok = true;
  int n = 0, s = 0;  // stage uses so far, of all producers
  uint32_t parity = 0;
  auto next = [&]() {
    ++n;
    if (++s == stages) {
      s = 0;
      parity ^= 1u;
    }
  };
  for (int unit = first; unit < units && ok; unit += step) {
    const Place p = place_of(unit);
    for (int i = 0; i < groups; ++i, next()) {
      if (n % kPromptProducers != producer) continue;
      const int chunk = chunk_of(p, i);
      if (n >= stages) {
        ok = prompt_wait(w, empty0 + s * 8u, parity ^ 1u, SITE_PRODUCER_EMPTY);
        if (!ok) break;
        load_b(p, chunk, s);
      }
      copy(base + s * stage_bytes, a_map, p.a_row, chunk, count0 + s * 8u, token_policy);
    }
  }
  // the MMA warp's last arrivals here, those of the pair's first CTA among them, come before this one leaves
  ok = ok && prompt_drain(n, stages, [&](int slot, uint32_t phase) { return prompt_wait(w, empty0 + slot * 8u, phase, SITE_DRAIN); });
  if (!ok) prompt_stay();
}

// KB: chunks per stage; BLOCKS: MMAs per K step (gate and up with accumulators of their own).
template <int CTAS, int TM, int KB, int BLOCKS>
__device__ __noinline__ void prompt_mma_loop(const PromptGemm& g, uint32_t base, uint32_t full0, uint32_t empty0, uint32_t accfull0,
                                             uint32_t accempty0, uint32_t tmem, int first, int step) {
  const PromptWait w{&g.guard, clock64() + g.guard.timeout_cycles};
  // The whole warp walks the schedule and one elected lane issues: descriptors stay in uniform registers.
  auto uniform = [](uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); };
  const int groups = uniform(g.kslice / KB), stages = uniform(g.stages), units = uniform(g.units);
  constexpr int kBuffers = BLOCKS == 2 ? 1 : 2;
  const uint32_t idesc = uniform(umma_idesc_bf16(CTAS * TM, g.instr_n));
  const uint64_t desc = umma_desc_sw128(0);
  const uint32_t high = static_cast<uint32_t>(desc >> 32), low = uniform(static_cast<uint32_t>(desc) + (base >> 4));
  const uint32_t block_step = uniform(g.b_bytes) >> 4;
  const uint32_t stage_step = uniform(g.stage_bytes) >> 4, a_step = uniform(g.a_bytes) >> 4, b_step = uniform(g.b_bytes * g.nmat) >> 4;
  const uint32_t d_tmem = uniform(tmem);
  int s = 0, q = 0;
  uint32_t parity = 0, at = low;
  for (int unit = first; unit < units; unit += step, ++q) {
    const int buf = kBuffers == 2 ? (q & 1) : 0;
    const uint32_t use = kBuffers == 2 ? (q >> 1) : q;
    if (!__all_sync(0xffffffffu, prompt_wait(w, accempty0 + buf * 8u, (use & 1u) ^ 1u, SITE_MMA_ACC))) return;
    tc_fence_after();
    const uint32_t d0 = d_tmem + buf * 256;
    uint32_t accumulate = 0u;
#pragma unroll 1
    for (int i = 0; i < groups; ++i) {
      if (!__all_sync(0xffffffffu, mbar_try_wait(full0 + s * 8u, parity)) &&
          !__all_sync(0xffffffffu, prompt_wait(w, full0 + s * 8u, parity, SITE_MMA_FULL)))
        return;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int c = 0; c < KB; ++c)
#pragma unroll
          for (int x = 0; x < BLOCKS; ++x)
            prompt_mma_chunk<CTAS>(d0 + x * 256u, at + c * a_step, at + KB * a_step + c * b_step + x * block_step, high, idesc, c == 0 ? accumulate : 1u);
        prompt_commit<CTAS>(empty0 + s * 8u);
        if (i + 1 == groups) prompt_commit<CTAS>(accfull0 + buf * 8u);
      }
      __syncwarp();
      accumulate = 1u;
      at += stage_step;
      if (++s == stages) {
        s = 0;
        parity ^= 1u;
        at = low;
      }
    }
  }
}

__device__ __forceinline__ void prompt_pack16(const float* v, uint32_t* w) {
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = pack2(v[2 * i], v[2 * i + 1]);
}
// v += sixteen biases, which may lie on any element.
__device__ __forceinline__ void prompt_add_bias(const bf16* bias, float* v) {
  if ((reinterpret_cast<uintptr_t>(bias) & 15) == 0) {
    float x[16];
    unpack8(__ldg(reinterpret_cast<const uint4*>(bias)), x);
    unpack8(__ldg(reinterpret_cast<const uint4*>(bias) + 1), x + 8);
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] += x[e];
  } else {
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] += ldg_bf16(bias + e);
  }
}

template <int CTAS, int TM, int EPI>
__device__ __forceinline__ void prompt_epilogue(const PromptGemm& g, uint32_t accfull0, uint32_t accempty0, uint32_t tmem, int rank, int first,
                                                int step, int ewarp, int lane) {
  constexpr int kParts = kPromptEpilogueWarps / 4;
  const int quad = (ewarp + kPromptFirstEpilogue) & 3;  // tensor-memory lanes a warp may read: 32 * (warp index % 4)
  const int part = ewarp >> 2;                          // the warps of a quadrant take items in turn
  // M = 128 (or 256 of a pair): token row r is lane r.  M = 64: row r is lane 32 * (r / 16) + r % 16.
  const int row = TM == 64 ? (lane < 16 ? quad * 16 + lane : TM) : quad * 32 + lane;
  const int warp_row = TM == 64 ? quad * 16 : quad * 32;
  grid_dependency_wait();
  const PromptWait w{&g.guard, clock64() + g.guard.timeout_cycles};
  const int refused = EPI == PE_LOGITS ? *reinterpret_cast<volatile int*>(&g.guard.ctrl->prompt_refused) : 0;
  int q = 0;
  for (int unit = first; unit < g.units; unit += step, ++q) {
    const PromptUnit u = prompt_unit_at(g, unit);
    const int buf = g.buffers == 2 ? (q & 1) : 0;
    const uint32_t use = g.buffers == 2 ? (q >> 1) : q;
    int seg = 0;
    if (EPI == PE_QKV) seg = u.tile >= g.tile_start[2] ? 2 : (u.tile >= g.tile_start[1] ? 1 : 0);
    const int n0 = (u.tile - g.tile_start[seg]) * g.rows;        // first row of the tile in its matrix
    const int live = min(g.rows, g.n[seg] - n0);                 // rows of the tile
    const int token0 = u.tt * CTAS * TM + rank * TM;
    const int token = token0 + row;
    const bool mine = row < TM && token < g.m;
    const bool any = token0 + warp_row < g.m;                    // the warp has a token
    const uint32_t acc = tmem + (static_cast<uint32_t>(quad * 32) << 16) + buf * 256;
    const bool ok = __all_sync(0xffffffffu, prompt_wait(w, accfull0 + buf * 8u, use & 1u, SITE_EPI_ACC));
    if (!ok) return;
    tc_fence_after();
    if (any) {
      if constexpr (EPI == PE_QKV) {
        const int hd = g.head_dim, hw = hd / 2, per_head = hw / 16, items = live / hd * per_head;
        bf16* const out = g.dst + static_cast<size_t>(mine ? token : 0) * g.ld + g.out_col[seg] + n0;
        const bf16* const bias = g.bias[seg] ? g.bias[seg] + n0 : nullptr;
        long long pos = mine ? g.pos[token] : 0;
        if (pos < 0 || pos >= g.max_positions) pos = 0;  // reported by the first kernel
#pragma unroll 1
        for (int it = part; it < items; it += kParts) {
          const int head = it / per_head, i = (it - head * per_head) * 16, c = head * hd + i;
          uint32_t lo[16], hi[16];
          tmem_ld16_async(acc + c, lo);
          tmem_ld16_async(acc + c + hw, hi);
          uint4 cs[2], sn[2];
          if (seg < 2) {
            const uint4* ct = reinterpret_cast<const uint4*>(g.cos_t + pos * hd + i);
            const uint4* st = reinterpret_cast<const uint4*>(g.sin_t + pos * hd + i);
            cs[0] = __ldg(ct); cs[1] = __ldg(ct + 1);
            sn[0] = __ldg(st); sn[1] = __ldg(st + 1);
          }
          tmem_ld_wait();
          float a[16], b[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            a[e] = __uint_as_float(lo[e]);
            b[e] = __uint_as_float(hi[e]);
          }
          if (bias != nullptr) {
            prompt_add_bias(bias + c, a);
            prompt_add_bias(bias + c + hw, b);
          }
          prompt_pack16(a, lo);
          prompt_pack16(b, hi);
          if (seg < 2) {
            // x1 cos - x2 sin, x2 cos + x1 sin; every operation rounds to bf16, so a packed one does two elements
            const uint32_t cw[8] = {cs[0].x, cs[0].y, cs[0].z, cs[0].w, cs[1].x, cs[1].y, cs[1].z, cs[1].w};
            const uint32_t sw[8] = {sn[0].x, sn[0].y, sn[0].z, sn[0].w, sn[1].x, sn[1].y, sn[1].z, sn[1].w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const uint32_t x1 = lo[e], x2 = hi[e];
              lo[e] = sub_bf16x2(mul_bf16x2(x1, cw[e]), mul_bf16x2(x2, sw[e]));
              hi[e] = add_bf16x2(mul_bf16x2(x2, cw[e]), mul_bf16x2(x1, sw[e]));
            }
          }
          if (mine) {
            st_global_v8(out + c, lo);
            st_global_v8(out + c + hw, hi);
          }
        }
      } else {
        const int items = (live + 15) / 16;
#pragma unroll 1
        for (int it = part; it < items; it += kParts) {
          const int c = it * 16;
          uint32_t r[16], r2[16];
          tmem_ld16_async(acc + c, r);
          if (EPI == PE_SILU) tmem_ld16_async(acc + g.up_column + c, r2);
          tmem_ld_wait();
          float v[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[e]);
          if constexpr (EPI == PE_PARTIAL) {
            float* out = g.partial + (static_cast<size_t>(u.slice) * g.m + (mine ? token : 0)) * g.n[0] + n0 + c;
            if (mine) {  // rows come in eights
              st_global_v8(out, r);
              if (c + 16 <= live) st_global_v8(out + 8, r + 8);
            }
          } else if constexpr (EPI == PE_SILU) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = silu_to_bf16(bf16_round(v[e]));
            uint32_t o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)  // the product of two bf16 values is exact in fp32: one rounding, packed
              o[e] = mul_bf16x2(pack2(v[2 * e], v[2 * e + 1]), pack2(__uint_as_float(r2[2 * e]), __uint_as_float(r2[2 * e + 1])));
            bf16* out = g.dst + static_cast<size_t>(mine ? token : 0) * g.ld + n0 + c;
            if (mine) {
              if (c + 16 <= live && (n0 & 15) == 0) {
                st_global_v8(out, o);
              } else {  // rows come in eights
                *reinterpret_cast<uint4*>(out) = make_uint4(o[0], o[1], o[2], o[3]);
                if (c + 16 <= live) *reinterpret_cast<uint4*>(out + 8) = make_uint4(o[4], o[5], o[6], o[7]);
              }
            }
          } else {
            bf16* out = g.dst + static_cast<size_t>(mine ? token : 0) * g.ld + n0 + c;
            uint32_t o[8];
            prompt_pack16(v, o);
            if (refused) {
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = 0x7FC07FC0u;
            }
            if (mine) {
              if (c + 16 <= live && (reinterpret_cast<uintptr_t>(out) & 31) == 0) {
                st_global_v8(out, o);
              } else if (c + 16 <= live && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
                reinterpret_cast<uint4*>(out)[0] = make_uint4(o[0], o[1], o[2], o[3]);
                reinterpret_cast<uint4*>(out)[1] = make_uint4(o[4], o[5], o[6], o[7]);
              } else {  // logits may begin at any element and a vocabulary may end anywhere
#pragma unroll
                for (int e = 0; e < 16; ++e)
                  if (c + e < live) reinterpret_cast<unsigned short*>(out)[e] = static_cast<unsigned short>(o[e >> 1] >> ((e & 1) * 16));
              }
            }
          }
        }
      }
    }
    tc_fence_before();
    __syncwarp();
    // The accumulator is handed back if another unit of this CTA's will use it: an arrival that nobody waits for could reach the
    // pair's first CTA after it has left (the barrier at the end orders no memory).
    if (lane == 0 && unit + g.buffers * step < g.units) {
      if constexpr (CTAS == 2) mbar_arrive_cluster(leader_address(accempty0 + buf * 8u));
      else mbar_arrive(accempty0 + buf * 8u);
    }
  }
}

template <int CTAS, int TM, int EPI>
__global__ void __launch_bounds__(kPromptThreads, 1) prompt_gemm(const __grid_constant__ PromptGemm g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kPromptStages], empty[kPromptStages], accfull[2], accempty[2];
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = CTAS == 2 ? static_cast<int>(cluster_rank()) : 0;
  const int first = blockIdx.x / CTAS, step = gridDim.x / CTAS;
  constexpr uint32_t kColumns = 512;
  if (tid == 0) {
    for (int s = 0; s < g.stages; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&accfull[b]), 1);
      mbar_init(smem_u32(&accempty[b]), CTAS * kPromptEpilogueWarps);
    }
    mbar_fence_init();
    for (int a = 0; a < 3; ++a)
      if (g.b[a]) tma_prefetch_desc(g.b[a]);
    tma_prefetch_desc(g.a);
  }
  if (warp == kPromptMmaWarp) prompt_tmem_alloc<CTAS>(smem_u32(&tmem_base), kColumns);
  tc_fence_before();
  if constexpr (CTAS == 2) cluster_sync_all();
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_base);
  const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty), accfull0 = smem_u32(accfull), accempty0 = smem_u32(accempty);
  if (warp < kPromptProducers) {
    if (lane == 0) prompt_producer<CTAS, TM>(g, smem, full0, empty0, rank, first, step, warp);
  } else if (warp == kPromptMmaWarp) {
    grid_dependency_wait();
    constexpr int kBlocks = CTAS == 2 && EPI == PE_SILU ? 2 : 1;
    if (CTAS == 1 && g.kb == 2) prompt_mma_loop<1, TM, 2, 1>(g, smem_u32(smem), full0, empty0, accfull0, accempty0, tmem, first, step);
    else if (rank == 0) prompt_mma_loop<CTAS, TM, 1, kBlocks>(g, smem_u32(smem), full0, empty0, accfull0, accempty0, tmem, first, step);
  } else {
    prompt_epilogue<CTAS, TM, EPI>(g, accfull0, accempty0, tmem, rank, first, step, warp - kPromptFirstEpilogue, lane);
  }
  __syncwarp();
  tc_fence_before();
  if constexpr (CTAS == 2) cluster_sync_relaxed();  // neither CTA leaves while the other may still use its barriers
  else __syncthreads();
  if (warp == kPromptMmaWarp) {
    tc_fence_after();
    prompt_tmem_dealloc<CTAS>(tmem, kColumns);
  }
}

// ---------------------------------------------------------------- RMSNorm
// A block per token row: residual stream (or the token's embedding row) plus the previous projection's K slices, added in
// slice order and rounded as x + bf16(sum); the sum is the new residual stream, its RMSNorm with the two roundings of the
// Hugging Face one the next projection's operand.
template <int V>
__global__ void __launch_bounds__(256) prompt_norm(const __grid_constant__ PromptNorm a) {
  __shared__ float red[8];
  __shared__ int bad_s;
  const int tid = threadIdx.x, threads = blockDim.x, nvec = a.k / 8, warps = threads >> 5;
  grid_dependents_go();  // at once: the projection behind it takes longer to get under way than this kernel takes
  uint4 w[V], x[V];
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int v = j * threads + tid;
    w[j] = v < nvec ? __ldg(reinterpret_cast<const uint4*>(a.weight) + v) : make_uint4(0, 0, 0, 0);
  }
  grid_dependency_wait();
  if (a.check) {  // the first kernel of a pass; the verdict is for the caller and for the output head, which then writes NaN
    if (tid == 0) bad_s = 0;
    __syncthreads();
    if (blockIdx.x == 0) {
      for (int i = tid; i < a.m; i += threads)
        if (a.ids[i] < 0 || a.ids[i] >= a.embed_rows || a.pos[i] < 0 || a.pos[i] >= a.max_positions) bad_s = 1;
      __syncthreads();
      if (tid == 0) {
        Control* const ctrl = a.guard.ctrl;
        ctrl->prompt_refused = bad_s;
        if (bad_s && atomicCAS(&ctrl->status, 0, static_cast<int>(MK_STATUS_BAD_INDEX)) == 0) {
          ctrl->where = SITE_PROLOGUE;
          ctrl->cta = 0;
          ctrl->detail = 0;
          if (a.guard.status_mirror) *a.guard.status_mirror = static_cast<int>(MK_STATUS_BAD_INDEX);
        }
      }
    }
  }
  for (int t = blockIdx.x; t < a.m; t += gridDim.x) {  // one, unless the handle limits its SMs
    const bf16* row;
    if (a.src == nullptr) {
      long long id = a.ids[t];
      if (id < 0 || id >= a.embed_rows) id = 0;  // never dereference out of range
      row = a.embed + id * a.k;
    } else {
      row = a.src + static_cast<size_t>(t) * a.k;
    }
    float4 lo[V][kMaxSplit], hi[V][kMaxSplit];
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int v = j * threads + tid;
      x[j] = make_uint4(0, 0, 0, 0);
      if (v < nvec) {
        x[j] = __ldcg(reinterpret_cast<const uint4*>(row) + v);
#pragma unroll
        for (int p = 0; p < kMaxSplit; ++p)
          if (p < a.parts) {
            const float4* part = reinterpret_cast<const float4*>(a.partial + (static_cast<size_t>(p) * a.m + t) * a.k) + v * 2;
            lo[j][p] = __ldcg(part);
            hi[j][p] = __ldcg(part + 1);
          }
      }
    }
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int v = j * threads + tid;
      if (v >= nvec) continue;
      float f[8];
      unpack8(x[j], f);
      if (a.parts > 0) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int p = 0; p < kMaxSplit; ++p)
          if (p < a.parts) {
            acc[0] += lo[j][p].x; acc[1] += lo[j][p].y; acc[2] += lo[j][p].z; acc[3] += lo[j][p].w;
            acc[4] += hi[j][p].x; acc[5] += hi[j][p].y; acc[6] += hi[j][p].z; acc[7] += hi[j][p].w;
          }
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = bf16_round(f[e] + bf16_round(acc[e]));
        x[j] = pack8(f);
      }
      if (a.h_out) reinterpret_cast<uint4*>(a.h_out + static_cast<size_t>(t) * a.k)[v] = x[j];
#pragma unroll
      for (int e = 0; e < 8; ++e) sum = fmaf(f[e], f[e], sum);
    }
    sum = warp_sum(sum);
    if ((tid & 31) == 0) red[tid >> 5] = sum;
    __syncthreads();
    float total = 0.f;
    for (int i = 0; i < warps; ++i) total += red[i];
    const float rinv = 1.0f / sqrtf(total / static_cast<float>(a.k) + a.eps);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int v = j * threads + tid;
      if (v < nvec) reinterpret_cast<uint4*>(a.xnorm + static_cast<size_t>(t) * a.k)[v] = normalise_vec(x[j], w[j], rinv);
    }
    __syncthreads();  // `red` has been read
  }
}

}  // namespace mk
