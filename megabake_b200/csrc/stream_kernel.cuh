// The streaming decode kernel: one cooperative launch per step, up to 32 sequences.
// See stream_common.cuh for the scheme.  One instantiation per token class (at most TM tokens; FEW: at
// most four of TM = 8) and head size.
#pragma once
#include "stream_attention.cuh"
#include "stream_gemm.cuh"

namespace mk {

// warp 0, one thread: every copy of this CTA in the order of use.
__device__ __forceinline__ void stream_producer(const KParams& p, StreamMisc* sm, StreamPipe pipe) {
  const CUtensorMap* const maps = sm->plan.maps;
  const CUtensorMap* const kv_maps = p.kv_maps;
  const uint64_t policy = l2_policy_evict_first();
  const int layers = p.layers, my_cta = sm->cta, grid = sm->grid;
  const int hpu = p.stream_hpu, tk = p.stream_tile_keys, cpg = hpu * (p.head_dim / kChunkK);
  const uint32_t kv_bytes = static_cast<uint32_t>(cpg * tk) * 128u;
  int issued = 0;
  // A free slot: the ring's first round needs no wait.
  auto claim = [&](uint32_t bytes) -> bool {
    if (issued >= pipe.nslots) stream_wait(sm, pipe.empty(), pipe.parity ^ 1u);
    if (stream_aborted(sm)) return false;
    mbar_expect_tx(pipe.full(), bytes);
    ++issued;
    return true;
  };
  auto weights = [&](int kind, const CUtensorMap* m) -> bool {
    const StreamPhase& ph = sm->plan.ph[kind];
    const int ncopy = ph.ncopy, cs = ph.cs, tile1 = ph.tile1, tile2 = ph.tile2, ntiles = ph.ntiles;
    const int count = sm->units[kind];
    const int nacc = kind == SP_GU ? 2 : 1;
    const int rows = ph.rows;
    const uint32_t bytes = static_cast<uint32_t>(rows) * kStreamKb * 128u;
    int tile = sm->first_tile[kind], slice = sm->first_slice[kind];
#pragma unroll 1
    for (int left = count; left > 0;) {  // the walk of stream_project
      const int run = min(left, ntiles - tile);
      left -= run;
#pragma unroll 1
      for (const int last = tile + run; tile < last; ++tile) {
        const CUtensorMap* map = m;
        int row0 = tile * rows;
        if (kind == SP_QKV && tile >= tile1) {
          map = tile >= tile2 ? m + 2 : m + 1;
          row0 -= (tile >= tile2 ? tile2 : tile1) * rows;
        }
#pragma unroll 1
        for (int c = 0; c < ncopy; ++c)
#pragma unroll 1
          for (int a = 0; a < nacc; ++a) {
            if (!claim(bytes)) return false;
            tma_load_3d(pipe.addr(), map + a, 0, row0, slice * cs + c * kStreamKb, pipe.full(), policy);
            pipe.next();
          }
      }
      ++slice;
      tile = 0;
    }
    return true;
  };
  auto run = [&]() {
#pragma unroll 1
    for (int step = 0; step <= 4 * layers; ++step) {  // q k v, o, gate up, down of every layer, then the output head: one copy of the code
      const int layer = step >> 2, kind = step == 4 * layers ? SP_HEAD : step & 3;
      const CUtensorMap* m = maps + 7 * layer;
      // descriptors are fetched like data: ask for the next ones before they are needed
      if (kind == SP_QKV) {
        for (int i = 3; i < 7; ++i) tma_prefetch_desc(m + i);
        tma_prefetch_desc(kv_maps + layer);
        tma_prefetch_desc(kv_maps + layers + layer);
      } else if (kind == SP_GU) {
        for (int i = 7; i < 10; ++i)
          if (layer + 1 < layers || i == 7) tma_prefetch_desc(m + i);  // the next layer's q, k, v, or the output head's
      }
      if (!weights(kind, m + (kind == SP_O ? 3 : kind == SP_GU ? 4 : kind == SP_DOWN ? 6 : 0))) return;
      if (kind != SP_QKV) continue;
      const StreamTiles tiles = stream_tiles(p, stream_lengths(p, sm, layer), my_cta, grid);
#pragma unroll 1
      for (int at = tiles.first; at < tiles.last;) {
        const StreamSegment sg = stream_segment(tiles, at, my_cta);
#pragma unroll 1
        for (int tl = sg.t0; tl < sg.t1; ++tl)
#pragma unroll 1
          for (int v = 0; v < 2; ++v) {
            if (!claim(kv_bytes)) return;
            tma_load_4d(pipe.addr(), kv_maps + v * layers + layer, 0, tl * tk, sg.group * cpg, sg.b, pipe.full(), policy);
            pipe.next();
          }
        at += sg.t1 - sg.t0;
      }
    }
  };
  run();
  {  // every copy already issued must land before the CTA exits; consumers that have given up do not wait for it
    const int back = min(issued, pipe.nslots);
    for (int i = 0; i < back; ++i) {
      const int s = (issued - back + i) % pipe.nslots;
      const uint32_t bar = pipe.full0 + static_cast<uint32_t>(s) * 8u;
      const uint32_t parity = ((issued - back + i) / pipe.nslots) & 1;
      for (uint32_t spins = 0; spins < (1u << 16) && !mbar_try_wait(bar, parity); ++spins) {
      }
    }
  }
}

// Ask L2 for the small vectors that no copy brings (norm weights, biases): all layers, once, by a warp that has nothing
// else to do.
__device__ __forceinline__ void stream_prefetch_vectors(const KParams& p, StreamMisc* sm, int at, int step) {
  for (int layer = 0; layer < p.layers; ++layer) {
    const StreamLayer* lw = sm->plan.layers + layer;
    for (int i = at; i < p.hidden / 64; i += step) {
      prefetch_l2(lw->input_norm + i * 64);
      prefetch_l2(lw->post_norm + i * 64);
    }
    for (int seg = 0; seg < 3; ++seg)
      if (lw->bias[seg] != nullptr)
        for (int i = at; i < (seg == 0 ? p.q_heads : p.kv_heads) * p.head_dim / 64; i += step) prefetch_l2(lw->bias[seg] + i * 64);
  }
  for (int i = at; i < p.hidden / 64; i += step) prefetch_l2(sm->plan.final_norm + i * 64);
}

__device__ __forceinline__ void stream_reset(bf16* buffer, long long elems, int at, int step) {
  uint4* v = reinterpret_cast<uint4*>(buffer);
  for (long long i = at; i < elems / 8; i += step) __stcg(v + i, make_uint4(kUnset, kUnset, kUnset, kUnset));
}

template <int TM, int HD, bool FEW>
__device__ __forceinline__ void stream_consumers(const KParams& p, StreamMisc* sm, StreamPipe pipe, int wtid) {
  constexpr int NT = stream_token_tiles(TM);
  constexpr int CNORM = stream_fit_normalised(TM), CPLAIN = stream_fit(NT);
  constexpr int kLayerWords = sizeof(StreamLayer) / 4;
  const int layers = p.layers;
  StreamThread th;
  th.sm = sm;
  th.wtid = wtid;
  th.pbuf = 0;
  th.turn = 0;
  th.last_turn = 2;
  th.list = 0;
  th.tracing = wtid == 0 && sm->trace_on != 0;
  stream_embed<TM>(p, sm, wtid);
#pragma unroll 1
  for (int layer = 0;; ++layer) {  // the last round is the output head
    const bool head = layer == layers;
    if (wtid == 0) {
      *reinterpret_cast<volatile int*>(&sm->progress) = layer;
      *reinterpret_cast<volatile int*>(&sm->seg_taken) = th.list;
    }
    // the next layer's vectors: requested here, passed on through shared memory at the end of the layer
    uint32_t word = 0u;
    if (wtid < kLayerWords && layer + 1 < layers) word = __ldg(reinterpret_cast<const uint32_t*>(sm->plan.layers + layer + 1) + wtid);
    stream_project<TM, 1, CNORM, SG_NORM, FEW>(p, th, pipe, head ? SP_HEAD : SP_QKV, layer);  // RMSNorm; q, k, v (+ bias) or the output head
    if (head) break;
    stream_attention<TM, HD>(p, th, pipe, layer);                       // RoPE, append, attention
    th.trace(EV_ATTENTION_DONE);
#pragma unroll 1
    for (int kind = SP_O;; kind = SP_DOWN) {  // one copy of the code for both (1.7B shape, 16 sequences 1551 -> 1465 us, 32 2334 -> 2268)
      stream_project<TM, 1, CPLAIN, SG_PLAIN, FEW>(p, th, pipe, kind, layer);  // o_proj, down_proj + residual
      if (kind == SP_DOWN) break;
      stream_project<TM, 2, CNORM, SG_MLP, FEW>(p, th, pipe, SP_GU, layer);    // RMSNorm, SiLU(gate) * up
      if (wtid < kLayerWords) reinterpret_cast<uint32_t*>(&sm->lw[(layer + 1) & 1])[wtid] = word;
      // this layer's resets come before the next layer's results (see stream_common.cuh)
      if (stream_is_aside<TM>(sm)) named_bar_arrive(kStreamStoredBarrier, kStreamFenceThreads);
      else __threadfence();
    }
    stream_sync();  // the next layer's vectors are in place
    th.last_turn = th.turn;
    th.turn = th.turn == 2 ? 0 : th.turn + 1;
  }

  // The only grid barrier: every result of the launch has been read, the logits are out.
  stream_sync();
  if (wtid == 0) {
    *reinterpret_cast<volatile int*>(&sm->progress) = layers + 1;
    red_release_add_u32(&sm->ctrl->barrier, 1u);
    const uint32_t target = p.epoch + static_cast<uint32_t>(sm->grid);
    while (static_cast<int32_t>(ld_acquire_u32(&sm->ctrl->barrier) - target) < 0 && !stream_aborted(sm)) {
    }
    sm->complete = !stream_aborted(sm);
    *reinterpret_cast<volatile int*>(&sm->progress) = -1;
  }
  stream_sync();
  th.trace(EV_BARRIER_DONE);
  if (!sm->complete) return;
  if (sm->cta == 0)
    for (int i = wtid; i < layers * (p.ragged ? p.batch : 1); i += kStreamConsumers) {
      const int per = p.ragged ? p.batch : 1;
      p.len[i / per][i % per] = sm->len_s[i] + 1;
    }
  {  // the words the last layer left set
    const int at = sm->cta * kStreamConsumers + wtid, step = sm->grid * kStreamConsumers, h = (layers - 1) % 3;
    const long long t = static_cast<long long>(sm->token_class) * sm->copies;
    const StreamPlan& plan = sm->plan;
    stream_reset(plan.attn[h], t * p.q_heads * p.head_dim, at, step);
    for (int kind = 0; kind < SP_HEAD; ++kind) {
      const StreamPhase& ph = plan.ph[kind];
      stream_reset(plan.dst[kind][h], t * ph.n, at, step);  // (q, k, v: one copy is used)
      if (ph.nslice > 1)
        stream_reset(reinterpret_cast<bf16*>(plan.part[kind][h]), static_cast<long long>(ph.nslice) * ph.ntiles * sm->tokens * kStreamRows * 2, at, step);
    }
  }
  if (p.sample) {
    Ctx cx;
    cx.p = &p;
    cx.cta = sm->cta;
    cx.grid = sm->grid;
    greedy_sample<1, kStreamConsumers>(cx, wtid, stream_psum(sm));
  }
}

template <int TM, int HD, bool FEW = false>
__global__ void __launch_bounds__(kStreamThreads, 1) decode_stream(const __grid_constant__ KParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5;
  StreamMisc* sm = reinterpret_cast<StreamMisc*>(smem + p.stream_slots * kStreamSlotBytes);
  if (tid == 0) {
    for (int s = 0; s < p.stream_slots; ++s) {
      mbar_init(smem_u32(&sm->full[s]), 1);
      mbar_init(smem_u32(&sm->empty[s]), kStreamWarps);
    }
    sm->p = &p;
    sm->ctrl = p.ctrl;
    sm->deadline = clock64() + p.timeout_cycles;
    sm->cta = blockIdx.x;
    sm->copy = stream_copy_of_sm(stream_copies(TM));
    sm->grid = gridDim.x;
    sm->tokens = p.m;
    sm->token_class = TM;
    sm->wabort = 0;
    sm->progress = 0;
    sm->seg_ready = 0;
    sm->seg_taken = 0;
    sm->copies = stream_copies(TM);
    sm->bad = 0;
    sm->trace_n = 0;
    sm->fence_aside = stream_fence_aside<TM>(p, gridDim.x);
    sm->trace_on = p.trace_cap != 0;
    sm->psum_offset = p.stream_scratch_bytes;
    mbar_fence_init();
  }
  for (int i = tid; i < static_cast<int>(sizeof(StreamPlan)) / 4; i += kStreamThreads)
    reinterpret_cast<int*>(&sm->plan)[i] = reinterpret_cast<const int*>(p.splan)[i];
  if (tid < kStreamPhases) {
    const int* range = p.splan->units + tid * (gridDim.x + 1) + blockIdx.x;
    const StreamPhase& ph = p.splan->ph[tid];
    sm->units[tid] = range[1] - range[0];
    sm->first_slice[tid] = range[0] / ph.ntiles;
    sm->first_tile[tid] = range[0] - sm->first_slice[tid] * ph.ntiles;
  }
  if (tid < static_cast<int>(sizeof(StreamLayer)) / 4)
    reinterpret_cast<uint32_t*>(&sm->lw[0])[tid] = reinterpret_cast<const uint32_t*>(p.splan->layers)[tid];
  __syncthreads();
  // Prologue validation: the same inputs in every CTA, so the verdict is grid-uniform.
  {
    int bad = 0;
    for (int t = tid; t < p.m; t += kStreamThreads) {
      long long id = p.ids[t], pos = p.pos[t];
      if (id < 0 || id >= p.embed_rows || pos < 0 || pos >= p.max_positions) {
        bad = MK_STATUS_BAD_INDEX;
        id = pos = 0;
      }
      sm->id_s[t] = static_cast<int>(id);
      sm->pos_s[t] = static_cast<int>(pos);
    }
    const int per = p.ragged ? p.batch : 1;
    for (int i = tid; i < p.layers * per; i += kStreamThreads) {
      const int len = p.len[i / per][i % per];
      if (len < 0 || len + 1 > p.capacity) bad = MK_STATUS_KV_OVERFLOW;
      sm->len_s[i] = len;
    }
    if (bad) atomicMax(&sm->bad, bad);
  }
  __syncthreads();
  const int bad = *reinterpret_cast<volatile int*>(&sm->bad);
  if (bad) {
    Ctx cx;
    cx.p = &p;
    cx.ctrl = p.ctrl;
    cx.cta = blockIdx.x;
    cx.grid = gridDim.x;
    refuse_outputs(cx, bad, tid, kStreamThreads);
    return;
  }
  StreamPipe pipe;
  pipe.base = smem_u32(smem);
  pipe.full0 = smem_u32(&sm->full[0]);
  pipe.empty0 = smem_u32(&sm->empty[0]);
  pipe.nslots = p.stream_slots;
  pipe.slot = 0;
  pipe.parity = 0;
  // 384 threads x 168 registers at launch = 128 x 56 + 256 x 224: the token operand of a slice is up to 128 registers
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (tid == 0) stream_producer(p, sm, pipe);
    else if (warp == 1) stream_fence(sm->fence_aside ? p.layers : 0);
    else if (tid == 64) stream_watch(sm);
    else if (warp == 2 && blockIdx.x == 0) stream_prefetch_vectors(p, sm, tid - 65, 31);
    else if (tid == 96) stream_plan_parts(p, sm);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    stream_consumers<TM, HD, FEW>(p, sm, pipe, tid - 128);
  }
}

}  // namespace mk
