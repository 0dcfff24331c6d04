// Launches of the prompt kernels (prompt_kernels.cuh).
#include "prompt_attention_tc.cuh"
#include "prompt_kernels.cuh"

namespace mk {
namespace {

// A launch that may begin while the kernel before it in the stream is still at work (`dependent`), its blocks in clusters of
// `cluster`.  The first kernel of a prompt pass is not: it, and through it the ones behind it, read weights ahead of their
// griddepcontrol.wait, which whatever came before may have written.
template <typename... Params, typename... Args>
cudaError_t launch(void (*kernel)(Params...), int blocks, int threads, int smem, int cluster, bool dependent, cudaStream_t stream, const Args&... args) {
  cudaLaunchAttribute attributes[2];
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(blocks);
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = attributes;
  if (dependent) {
    attributes[config.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[config.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attributes[config.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attributes[config.numAttrs].val.clusterDim.x = cluster;
    attributes[config.numAttrs].val.clusterDim.y = attributes[config.numAttrs].val.clusterDim.z = 1;
    ++config.numAttrs;
  }
  return cudaLaunchKernelEx(&config, kernel, args...);
}

// An event of a traced pass, in the list of every CTA: the launches before it have ended.  A launch of its own, so that the kernels
// are the same with and without the trace (stamps inside them, never taken: 64 tokens of the 1.7B shape 1279 -> 1311 us).
__global__ void __launch_bounds__(256) prompt_stamp(const __grid_constant__ PromptTrace t, int at, int code) {
  grid_dependents_go();
  grid_dependency_wait();
  unsigned long long now;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
  for (int cta = threadIdx.x; cta < t.ctas; cta += blockDim.x)
    t.list[static_cast<size_t>(cta) * t.cap + at] = (static_cast<unsigned long long>(code) << 56) | (now & 0x00FFFFFFFFFFFFFFull);
}

template <int EPI>
cudaError_t launch_gemm(const PromptGemm& g, int cls, int grid, cudaStream_t stream) {
  if (cls > 0)
    return launch(prompt_gemm<2, kPromptRow, EPI>, 2 * std::min(g.units, grid / 2), kPromptThreads, kPromptSmem, 2, true, stream, g);
  const int blocks = std::min(g.units, grid);
  if (g.m <= 64) return launch(prompt_gemm<1, 64, EPI>, blocks, kPromptThreads, kPromptSmem, 1, true, stream, g);
  return launch(prompt_gemm<1, kPromptRow, EPI>, blocks, kPromptThreads, kPromptSmem, 1, true, stream, g);
}

template <int EPI>
cudaError_t prepare_gemm() {
  cudaError_t e = cudaFuncSetAttribute(prompt_gemm<2, kPromptRow, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPromptSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(prompt_gemm<1, kPromptRow, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPromptSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(prompt_gemm<1, 64, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPromptSmem);
  return e;
}

cudaError_t launch_norm(const PromptNorm& n, int blocks, bool dependent, cudaStream_t stream) {
  const int nvec = n.k / 8, threads = std::min(256, (nvec + 31) / 32 * 32);
  if (nvec <= threads) return launch(prompt_norm<1>, blocks, threads, 0, 1, dependent, stream, n);
  if (nvec <= 2 * threads) return launch(prompt_norm<2>, blocks, threads, 0, 1, dependent, stream, n);
  return launch(prompt_norm<4>, blocks, threads, 0, 1, dependent, stream, n);  // (hidden up to 8192: check_config)
}

}  // namespace

cudaError_t prompt_prepare() {
  cudaError_t e = prepare_gemm<PE_QKV>();
  if (e == cudaSuccess) e = prepare_gemm<PE_PARTIAL>();
  if (e == cudaSuccess) e = prepare_gemm<PE_SILU>();
  if (e == cudaSuccess) e = prepare_gemm<PE_LOGITS>();
  const auto attention = [&](auto kernel, int smem) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  };
  const auto attention_tc = [&](auto by) {
    constexpr int kBy = decltype(by)::value;
    attention(prompt_attention_tc<64, kBy>, AttnTc<64, kBy>::kSmem);
    attention(prompt_attention_tc<128, kBy>, AttnTc<128, kBy>::kSmem);
  };
  attention_tc(std::integral_constant<int, AM_LOADS>());
  attention_tc(std::integral_constant<int, AM_TILES>());
  attention_tc(std::integral_constant<int, AM_EIGHTS>());
  if (e == cudaSuccess) e = cudaFuncSetAttribute(prompt_attention<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, PromptLaunch<64>::kSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(prompt_attention<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, PromptLaunch<128>::kSmem);
  return e;
}

// In a prompt pass, where the projections' shared memory keeps the tcgen05 kernel's tensor memory and barriers from being set up
// ahead and tiles past the diagonal are not visited, it is the faster one from here on (1.7B shape, us for the whole pass: 64 tokens
// 1266 on mma.sync and 1307, 200 1774 and 1771, 500 2588 and 2496; 135M shape, 250 tokens 1257 and 1281).  On its own:
// attention_on_tcgen05.
constexpr int kAttnTcInPass = 257;

bool prompt_attention_tc_wanted(const AttnArgs& args, int head_dim, int q_heads, int batch, int sms, bool limited, bool in_pass) {
  if (in_pass) return args.klen >= kAttnTcInPass;
  return attention_on_tcgen05(head_dim, args.sq, args.klen, static_cast<long long>(batch) * q_heads, args.mask != nullptr, sms, limited);
}

cudaError_t prompt_attention_launch(const AttnArgs& args, const AttnTcMaps& maps, const PromptGuard& guard, int head_dim, int q_heads, int kv_heads,
                                    int batch, int sms, bool limited, bool in_pass, cudaStream_t stream) {
  const bool tc = prompt_attention_tc_wanted(args, head_dim, q_heads, batch, sms, limited, in_pass);
  const int per = tc ? kAttnQueries : kPromptQueries, units = batch * q_heads * ((args.sq + per - 1) / per);
  const int blocks = limited ? std::min(units, sms) : units;
  // Everything a kernel reads or writes comes behind its griddepcontrol.wait, so that it may be launched as a dependent one behind
  // any kernel: two to three microseconds less between the two.
  if (tc) {
    const auto go = [&](auto kernel, int smem) {
      return launch(kernel, blocks, kAttnThreads, smem, 1, true, stream, args, maps, guard, q_heads, kv_heads, batch, units);
    };
    const auto by_mask = [&](auto by) {
      constexpr int kBy = decltype(by)::value;
      if (head_dim == 64) return go(prompt_attention_tc<64, kBy>, AttnTc<64, kBy>::kSmem);
      return go(prompt_attention_tc<128, kBy>, AttnTc<128, kBy>::kSmem);
    };
    if (maps.mask_by == AM_EIGHTS) return by_mask(std::integral_constant<int, AM_EIGHTS>());
    if (maps.mask_by == AM_TILES) return by_mask(std::integral_constant<int, AM_TILES>());
    return by_mask(std::integral_constant<int, AM_LOADS>());
  }
  if (head_dim == 64)
    return launch(prompt_attention<64>, blocks, kWorkers, PromptLaunch<64>::kSmem, 1, true, stream, args, q_heads, kv_heads, batch, units);
  return launch(prompt_attention<128>, blocks, kWorkers, PromptLaunch<128>::kSmem, 1, true, stream, args, q_heads, kv_heads, batch, units);
}

cudaError_t prompt_forward(const PromptPass& pass, cudaStream_t stream) {
  const mk_config& c = *pass.config;
  const int cls = pass.cls, m = pass.m, q_size = c.q_heads * c.head_dim, kv_size = c.kv_heads * c.head_dim;
  const int per_tile = cls > 0 ? 2 * kPromptRow : (m <= 64 ? 64 : kPromptRow), rows_per_cta = cls > 0 ? kPromptRow : per_tile;
  // the token operand's box: the smallest that holds the launch, a CTA's rows otherwise
  const int box = m <= 16 ? 0 : (m <= 32 ? 1 : (m <= 64 ? 2 : 3)), box_rows = 16 << box;
  auto gemm = [&](int kind, int operand) {
    const PromptPhase& p = pass.phases[kind];
    PromptGemm g{};
    g.guard = pass.guard;
    // Without pairs a chunk's MMAs take less than a step of the pipeline: two chunks to a stage (1.7B shape, 70 tokens 1536 ->
    // 1443 us, 128 1535 -> 1482).
    g.kb = cls == 0 && p.kslice % 2 == 0 ? 2 : 1;
    g.a = pass.operands + (operand * kOperandTiles + box) * kOperandChunks + g.kb - 1;
    for (int s = 0; s < 3; ++s) g.n[s] = p.n[s];
    for (int s = 0; s < 4; ++s) g.tile_start[s] = p.tile_start[s];
    g.m = m;
    g.rows = p.rows;
    g.nmat = p.nmat;
    g.ksplit = p.ksplit;
    g.kslice = p.kslice;
    g.token_tiles = (m + per_tile - 1) / per_tile;
    g.units = p.tile_start[3] * p.ksplit * g.token_tiles;
    g.a_bytes = box_rows * 128;
    g.b_bytes = prompt_box_rows(p, cls) * 128;
    g.stage_bytes = g.kb * (g.a_bytes + p.nmat * g.b_bytes);
    // an MMA reads a CTA's full rows of tokens, past a smaller box whatever lies there: room for that behind the last stage
    const int room = kPromptSmem - 1024 - rows_per_cta * 128;
    g.stages = std::min(kPromptStages, room / g.stage_bytes);  // (at least two: a stage is 64 KB at most)
    const bool joined = p.nmat == 2 && cls == 0;  // gate and up as one MMA of twice the rows
    g.instr_n = ((joined ? 2 * p.rows : p.rows) + 15) / 16 * 16;  // (a tile may end within an MMA's N: columns nobody reads)
    g.up_column = joined ? p.rows : 256;
    g.buffers = p.nmat == 2 && !joined ? 1 : 2;
    g.head_dim = c.head_dim;
    g.max_positions = c.max_positions;
    g.stream_weights = g.token_tiles == 1;
    return g;
  };
  const mk_weights& w = *pass.weights;
  PromptNorm norm{};
  norm.guard = pass.guard;
  norm.embed = static_cast<const bf16*>(w.embed);
  norm.ids = pass.ids;
  norm.pos = pass.pos;
  norm.partial = pass.partial;
  norm.xnorm = pass.xnorm;
  norm.m = m;
  norm.k = c.hidden;
  norm.embed_rows = c.embed_rows > 0 ? c.embed_rows : c.vocab;
  norm.max_positions = c.max_positions;
  norm.eps = c.rms_eps;
  const int rows = c.sm_limit > 0 ? std::min(m, pass.grid) : m;
  int events = 0;
  auto stamp = [&](cudaError_t before, int code) -> cudaError_t {
    if (before != cudaSuccess || pass.trace.list == nullptr || events >= pass.trace.cap) return before;
    return launch(prompt_stamp, 1, 256, 0, 1, events > 0, stream, pass.trace, events++, code);
  };
  cudaError_t e = stamp(cudaSuccess, EV_PHASE_ENTER);
  for (int l = 0; l <= c.layers && e == cudaSuccess; ++l) {
    const bool head = l == c.layers;
    const CUtensorMap* maps = pass.maps + 7 * static_cast<size_t>(l);
    // the residual stream: embedding rows, then down_proj's sums on hidden_a; it goes to hidden_b
    norm.src = l == 0 ? nullptr : pass.hidden_a;
    norm.parts = l == 0 ? 0 : pass.phases[PP_DOWN].ksplit;
    norm.weight = static_cast<const bf16*>(head ? w.final_norm : w.layers[l].input_norm);
    norm.h_out = head ? nullptr : pass.hidden_b;
    norm.check = l == 0;
    e = stamp(launch_norm(norm, rows, l > 0, stream), EV_PHASE_DONE);
    norm.check = 0;
    if (e != cudaSuccess) return e;
    if (head) {
      PromptGemm g = gemm(PP_HEAD, kOperandXnorm);
      g.b[0] = maps;
      g.dst = pass.logits;
      g.ld = c.vocab;
      return stamp(launch_gemm<PE_LOGITS>(g, cls, pass.grid, stream), EV_PHASE_DONE);
    }
    const mk_layer_weights& lw = w.layers[l];
    PromptGemm g = gemm(PP_QKV, kOperandXnorm);
    const void* biases[3] = {lw.q_bias, lw.k_bias, lw.v_bias};
    for (int s = 0; s < 3; ++s) {
      g.b[s] = maps + s;
      g.bias[s] = c.qkv_bias ? static_cast<const bf16*>(biases[s]) : nullptr;
    }
    g.out_col[1] = q_size;
    g.out_col[2] = q_size + kv_size;
    g.dst = pass.qkv;
    g.ld = q_size + 2 * kv_size;
    g.cos_t = static_cast<const bf16*>(w.rope_cos);
    g.sin_t = static_cast<const bf16*>(w.rope_sin);
    g.pos = pass.pos;
    e = stamp(launch_gemm<PE_QKV>(g, cls, pass.grid, stream), EV_PHASE_DONE);
    if (e == cudaSuccess)
      e = stamp(prompt_attention_launch(*pass.attention, *pass.attention_maps, pass.guard, c.head_dim, c.q_heads, c.kv_heads, pass.batch, pass.grid,
                                        c.sm_limit > 0, true, stream), EV_ATTENTION_DONE);
    if (e != cudaSuccess) return e;
    g = gemm(PP_O, kOperandAttn);
    g.b[0] = maps + 3;
    g.partial = pass.partial;
    e = stamp(launch_gemm<PE_PARTIAL>(g, cls, pass.grid, stream), EV_PHASE_DONE);
    if (e != cudaSuccess) return e;
    norm.src = pass.hidden_b;
    norm.parts = pass.phases[PP_O].ksplit;
    norm.weight = static_cast<const bf16*>(lw.post_norm);
    norm.h_out = pass.hidden_a;
    e = stamp(launch_norm(norm, rows, true, stream), EV_PHASE_DONE);
    if (e != cudaSuccess) return e;
    g = gemm(PP_GU, kOperandXnorm);
    g.b[0] = maps + 4;
    g.b[1] = maps + 5;
    g.dst = pass.act;
    g.ld = c.intermediate;
    e = stamp(launch_gemm<PE_SILU>(g, cls, pass.grid, stream), EV_PHASE_DONE);
    if (e != cudaSuccess) return e;
    g = gemm(PP_DOWN, kOperandAct);
    g.b[0] = maps + 6;
    g.partial = pass.partial;
    e = stamp(launch_gemm<PE_PARTIAL>(g, cls, pass.grid, stream), EV_PHASE_DONE);
  }
  return e;
}

}  // namespace mk
