// Host side of the C ABI declared in include/megabake_b200.h: workspace carving,
// TMA descriptor encoding, the per-launch parameter block and the cooperative
// launch of the megakernel.  No device memory is allocated here.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <algorithm>
#include <vector>

#include "decoder_kernel.cuh"
#include "kv_attention.cuh"
#include "prompt_attention_tc.cuh"
#include "prompt_plan.h"
#include "stream_plan.h"

using namespace mk;

namespace {

thread_local char g_error[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
  return code;
}

#define MK_CUDA(call)                                                                       \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess) return fail(MK_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct Carve {
  size_t ctrl, tmaps, kvmaps, phases, hidden, hidden2, xnorm, qkv, attn, act, partial, att_xch, att_part, host_io;
  size_t pmaps;                                        // prompt kernels: weight descriptors per class
  size_t splan, smaps, slayers, sunits, srec;          // streaming decode kernel
  size_t handover, handover_bytes, shalf[5][3], spart[2][3];       // its hand-over buffers, filled with the unset word
  size_t total;
};

int qkv_width(const mk_config& c) { return (c.q_heads + 2 * c.kv_heads) * c.head_dim; }
constexpr int kCacheMapSets = 8;  // cache-descriptor sets a handle remembers (one per KV state it is called with in turn)
constexpr int kOperandMaps = kOperandKinds * kOperandTiles * kOperandChunks;  // token operands (prompt_plan.h), behind the weight descriptors
constexpr int kPhaseTables = 2;   // split-K, plain
int token_tile_of(int m) { return m <= 16 ? 16 : (m <= 32 ? 32 : (m <= 64 ? 64 : 128)); }
size_t maps_per_table(const mk_config& c) { return 7 * static_cast<size_t>(c.layers) + 1; }
size_t phases_per_table(const mk_config& c) { return 4 * static_cast<size_t>(c.layers) + 1; }

// Handles that ask for the tensor engine (the attention ops' among them) have no streaming plans and buffers.
bool stream_wanted(const mk_config& c) { return c.engine != MK_ENGINE_TCGEN05 && stream_shape_ok(c); }

// Prompt passes of a single-GPU handle run on kernels of their own, in classes by token count.
int prompt_classes(const mk_config& c, int grid) { return c.tp_size > 1 ? 0 : 1 + prompt_class(c.max_tokens, grid); }

Carve carve(const mk_config& c, int grid) {
  Carve v{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  const size_t m = static_cast<size_t>(c.max_tokens);
  v.ctrl = take(sizeof(Control));
  v.tmaps = take(sizeof(CUtensorMap) * (kPhaseTables * maps_per_table(c) + kOperandMaps));
  v.pmaps = take(sizeof(CUtensorMap) * prompt_classes(c, grid) * maps_per_table(c));
  v.kvmaps = take(sizeof(CUtensorMap) * 2 * static_cast<size_t>(c.layers) * kCacheMapSets);  // decode attention: per set, key caches then value caches
  v.phases = take(sizeof(GemmPhase) * kPhaseTables * phases_per_table(c));
  v.hidden = take(m * c.hidden * 2);
  v.hidden2 = take(m * c.hidden * 2);
  v.xnorm = take(m * c.hidden * 2);
  v.qkv = take(m * qkv_width(c) * 2);
  v.attn = take(m * c.q_heads * c.head_dim * 2);
  v.act = take(m * c.intermediate * 2);
  v.partial = take(static_cast<size_t>(kMaxSplit) * m * c.hidden * 4);
  v.att_xch = take(m * c.kv_heads * kMaxChunks * kExchangeFloats * 4);
  v.att_part = take(m * c.q_heads * kMaxChunks * c.head_dim * 4);
  v.host_io = take(3 * m * sizeof(int64_t));  // mk_decode_step_host: ids, positions, sampled tokens
  if (stream_wanted(c)) {
    const size_t tokens = std::min<size_t>(m, kStreamTokens);
    v.splan = take(sizeof(StreamPlan) * kStreamPlans);
    v.smaps = take(sizeof(CUtensorMap) * kStreamPlans * maps_per_table(c));
    v.slayers = take(sizeof(StreamLayer) * c.layers);
    v.sunits = take(sizeof(int) * kStreamPlans * kStreamPhases * (kStreamMaxGrid + 1));
    v.srec = take(tokens * c.q_heads * kStreamMaxSegments * (c.head_dim + 2) * 8);
    size_t part[2] = {0, 0};
    for (int i = 0; i < kStreamPlans; ++i) {
      StreamPhase ph[kStreamPhases];
      const int ctas = stream_grid(c, i, grid);
      if (ctas == 0) continue;
      stream_phases(c, i, ctas, ph);
      const size_t t = std::min<size_t>(tokens, 8u * stream_plan_tiles(i));
      for (int k = 0; k < kStreamPhases; ++k) {
        const size_t sums = static_cast<size_t>(ph[k].ntiles) * t * kStreamRows * sizeof(float);
        if (ph[k].nslice > 1) part[k == SP_O ? 0 : 1] = std::max(part[k == SP_O ? 0 : 1], sums * ph[k].nslice);
      }
    }
    v.handover = off;
    size_t copied = 0;
    for (int i = 0; i <= stream_class_of(static_cast<int>(tokens)); ++i) copied = std::max<size_t>(copied, kStreamClassTokens[i] * stream_copies(kStreamClassTokens[i]));
    const size_t widths[5] = {static_cast<size_t>(qkv_width(c)), static_cast<size_t>(c.q_heads) * c.head_dim, static_cast<size_t>(c.hidden),
                              static_cast<size_t>(c.hidden), static_cast<size_t>(c.intermediate)};
    for (int b = 0; b < 5; ++b)
      for (int h = 0; h < 3; ++h) v.shalf[b][h] = take(copied * widths[b] * 2);
    for (int b = 0; b < 2; ++b)
      for (int h = 0; h < 3; ++h) v.spart[b][h] = take(part[b]);
    v.handover_bytes = off - v.handover;
  }
  v.total = off;
  return v;
}

int check_config(const mk_config& c) {
  if (c.hidden <= 0 || c.layers <= 0 || c.q_heads <= 0 || c.kv_heads <= 0 || c.intermediate <= 0 || c.vocab <= 0 ||
      c.max_tokens <= 0 || c.max_positions <= 0)
    return fail(MK_ERR_INVALID, "config: every size must be positive");
  if (c.layers > MK_MAX_LAYERS) return fail(MK_ERR_UNSUPPORTED, "config: at most %d layers", MK_MAX_LAYERS);
  if (c.head_dim != 64 && c.head_dim != 128) return fail(MK_ERR_UNSUPPORTED, "config: head_dim must be 64 or 128");
  if (c.q_heads % c.kv_heads) return fail(MK_ERR_INVALID, "config: q_heads must be a multiple of kv_heads");
  if (c.q_heads / c.kv_heads > 8) return fail(MK_ERR_UNSUPPORTED, "config: at most 8 query heads per kv head");
  if (c.hidden % 64 || c.intermediate % 64)
    return fail(MK_ERR_UNSUPPORTED, "config: hidden and intermediate must be multiples of 64");
  if (c.hidden > kNormVecs * kWorkers * 8)
    return fail(MK_ERR_UNSUPPORTED, "config: hidden above %d (a norm phase keeps a row in the registers of one CTA)", kNormVecs * kWorkers * 8);
  if (c.engine != MK_ENGINE_TCGEN05 && c.engine != MK_ENGINE_FMA && c.engine != MK_ENGINE_AUTO)
    return fail(MK_ERR_INVALID, "config: engine");
  if (c.rope_style != MK_ROPE_HF && c.rope_style != MK_ROPE_HALF_SWAP) return fail(MK_ERR_INVALID, "config: rope_style");
  if (c.tp_size < 0 || c.tp_size > kMaxTp) return fail(MK_ERR_UNSUPPORTED, "config: tensor-parallel groups have 1..%d ranks", kMaxTp);
  if (c.tp_size > 1 && (c.tp_rank < 0 || c.tp_rank >= c.tp_size)) return fail(MK_ERR_INVALID, "config: tp_rank outside the group");
  if (c.embed_rows < 0) return fail(MK_ERR_INVALID, "config: embed_rows");
  return MK_OK;
}

// What this library needs to know of a device, asked for once: the clock-rate query goes to the driver's control path and
// took 2 to 170 ms per handle on a busy host.
struct DeviceFacts {
  int known = 0, sms = 0, major = 0, coop = 0, khz = 0;
};
int device_facts(int device, DeviceFacts* out) {
  constexpr int kDevices = 64;
  static std::mutex lock;
  static DeviceFacts all[kDevices];
  std::lock_guard<std::mutex> guard(lock);
  if (device < 0 || device >= kDevices) return fail(MK_ERR_INVALID, "device %d outside [0, %d)", device, kDevices);
  DeviceFacts& f = all[device];
  if (!f.known) {
    MK_CUDA(cudaDeviceGetAttribute(&f.sms, cudaDevAttrMultiProcessorCount, device));
    MK_CUDA(cudaDeviceGetAttribute(&f.major, cudaDevAttrComputeCapabilityMajor, device));
    MK_CUDA(cudaDeviceGetAttribute(&f.coop, cudaDevAttrCooperativeLaunch, device));
    MK_CUDA(cudaDeviceGetAttribute(&f.khz, cudaDevAttrClockRate, device));
    f.known = 1;
  }
  *out = f;
  if (f.major != 10) return fail(MK_ERR_UNSUPPORTED, "device %d is sm_%d0; this library is built for sm_100a only", device, f.major);
  if (!f.coop) return fail(MK_ERR_UNSUPPORTED, "device %d does not support cooperative launch", device);
  return MK_OK;
}

int device_grid(const mk_config& c, int device, int* grid) {
  DeviceFacts facts;
  if (int e = device_facts(device, &facts)) return e;
  const int sms = facts.sms;
  *grid = (c.sm_limit > 0 && c.sm_limit < sms) ? c.sm_limit : sms;
  return MK_OK;
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &result) == cudaSuccess &&
        result == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(sym);
  });
  return fn;
}

// bf16 [rows, k] row-major -> boxes of box_rows rows x 64 columns, 128-byte swizzle.
int encode_weight_map(CUtensorMap* out, const void* base, int rows, int k, int box_rows, int box_chunks = 1,
                      bool swizzle = true) {
  if (reinterpret_cast<uintptr_t>(base) % 16) return fail(MK_ERR_ALIGNMENT, "weight base %p is not 16-byte aligned", base);
  auto fn = encode_fn();
  if (!fn) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * 2};
  // swizzle: the tensor core's operand layout (64 elements = 128 bytes per row, 128-byte swizzle).
  // !swizzle: plain rows of box_chunks * 128 bytes for the CUDA-core consumer (up to 256 elements).
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kChunkK * box_chunks), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d (rows %d, k %d)", (int)r, rows, k);
  return MK_OK;
}

// Tensor engine, weights: bf16 [rows, k] row-major seen as (64 elements, rows, k / 64 chunks); a box is
// box_rows rows x box_chunks chunks, each chunk 128-byte swizzled: one copy brings several K chunks of a tile.
int encode_weight_map3(CUtensorMap* out, const void* base, int rows, int k, int box_rows, int box_chunks) {
  if (reinterpret_cast<uintptr_t>(base) % 16) return fail(MK_ERR_ALIGNMENT, "weight base %p is not 16-byte aligned", base);
  auto fn = encode_fn();
  if (!fn) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(kChunkK), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(k / kChunkK)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(k) * 2, static_cast<cuuint64_t>(kChunkK) * 2};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(kChunkK), static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(box_chunks)};
  const cuuint32_t elem[3] = {1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled (3-D) failed with %d (rows %d, k %d, box %d x %d)", (int)r, rows, k, box_rows, box_chunks);
  return MK_OK;
}

// The weight descriptor of a tensor-engine phase: three-dimensional when the driver accepts the chunk-major
// view (its chunk stride, 128 bytes, is smaller than its row stride), else one 64-column box per copy.
int encode_phase_weight_map(CUtensorMap* out, const void* base, int rows, int k, GemmPhase& ph, bool& use3d) {
  if (use3d) {
    if (encode_weight_map3(out, base, rows, k, ph.rows, ph.kb) == MK_OK) {
      ph.map3d = 1;
      return MK_OK;
    }
    use3d = false;  // fall back for this and every later matrix of the handle
  }
  ph.map3d = 0;
  return encode_weight_map(out, base, rows, k, ph.rows);
}

// Tensor engine, token operand: bf16 [tokens, k] row-major seen as (64 elements, tokens, k / 64 chunks), box = 64 elements x
// `tile` tokens x `chunks` chunks, each 128-byte swizzled; token rows past `tokens` read as zeros.
int encode_operand_map(CUtensorMap* out, const void* base, int tokens, int k, int tile, int chunks, bool use3d) {
  if (reinterpret_cast<uintptr_t>(base) % 16) return fail(MK_ERR_ALIGNMENT, "operand base %p is not 16-byte aligned", base);
  auto fn = encode_fn();
  if (!fn) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims3[3] = {static_cast<cuuint64_t>(kChunkK), static_cast<cuuint64_t>(tokens), static_cast<cuuint64_t>(k / kChunkK)};
  const cuuint64_t dims2[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(tokens)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(k) * 2, static_cast<cuuint64_t>(kChunkK) * 2};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(kChunkK), static_cast<cuuint32_t>(tile), static_cast<cuuint32_t>(chunks)};
  const cuuint32_t elem[3] = {1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, use3d ? 3 : 2, const_cast<void*>(base), use3d ? dims3 : dims2, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled (operand) failed with %d (tokens %d, k %d)", (int)r, tokens, k);
  return MK_OK;
}

// Decode attention on the tensor engine: a cache [batch, capacity, kv_heads * head_dim] seen as
// (64 dimensions, positions, 64-dimension chunks of a row, sequences); a box is one stage of a unit:
// 64 x tile_keys positions x the unit's chunks, each chunk 128-byte swizzled.
int encode_cache_map(CUtensorMap* out, const void* base, int batch, int capacity, int row_elems, int tile_keys, int unit_chunks) {
  if (reinterpret_cast<uintptr_t>(base) % 16) return fail(MK_ERR_ALIGNMENT, "cache base %p is not 16-byte aligned", base);
  auto fn = encode_fn();
  if (!fn) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[4] = {static_cast<cuuint64_t>(kChunkK), static_cast<cuuint64_t>(capacity),
                              static_cast<cuuint64_t>(row_elems / kChunkK), static_cast<cuuint64_t>(batch)};
  const cuuint64_t strides[3] = {static_cast<cuuint64_t>(row_elems) * 2, static_cast<cuuint64_t>(kChunkK) * 2,
                                 static_cast<cuuint64_t>(capacity) * row_elems * 2};
  const cuuint32_t box[4] = {static_cast<cuuint32_t>(kChunkK), static_cast<cuuint32_t>(tile_keys), static_cast<cuuint32_t>(unit_chunks), 1};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled (cache) failed with %d", (int)r);
  return MK_OK;
}

// Prompt attention: rows of `heads` x head_dim elements, `rows` to a sequence, seen as (64 elements, rows, chunks of all heads,
// sequences); a box is `box_rows` rows of one head.
int encode_attention_map(CUtensorMap* out, const void* base, int batch, int rows, int heads, int head_dim, long long ld, long long batch_stride, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint32_t chunks = static_cast<cuuint32_t>(head_dim / kChunkK);
  const cuuint64_t dims[4] = {static_cast<cuuint64_t>(kChunkK), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(heads) * chunks,
                              static_cast<cuuint64_t>(batch)};
  const cuuint64_t strides[3] = {static_cast<cuuint64_t>(ld) * 2, static_cast<cuuint64_t>(kChunkK) * 2, static_cast<cuuint64_t>(batch_stride) * 2};
  const cuuint32_t box[4] = {static_cast<cuuint32_t>(kChunkK), static_cast<cuuint32_t>(box_rows), chunks, 1};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MK_ERR_CUDA, "cuTensorMapEncodeTiled (attention) failed with %d", (int)r);
  return MK_OK;
}
int encode_attention_maps(AttnTcMaps* maps, const AttnArgs& A, const mk_config& c, int grid, int batch, bool in_pass) {
  const int q_heads = c.q_heads, kv_heads = c.kv_heads, head_dim = c.head_dim;
  if (!prompt_attention_tc_wanted(A, head_dim, q_heads, batch, grid, c.sm_limit > 0, in_pass)) return MK_OK;  // nobody reads them
  maps->q_ok = (reinterpret_cast<uintptr_t>(A.q) & 15) == 0;
  if (int e = encode_attention_map(&maps->k, A.k, batch, A.klen, kv_heads, head_dim, A.kv_ld, A.kv_bstride, kAttnKeys)) return e;
  if (int e = encode_attention_map(&maps->v, A.v, batch, A.klen, kv_heads, head_dim, A.kv_ld, A.kv_bstride, kAttnKeys)) return e;
  // The mask comes by TMA: in tiles where its rows begin on 16-byte boundaries (a tiled copy's strides are multiples of that), else the
  // rows of each residue modulo eight as a matrix of their own.
  maps->mask_by = AM_LOADS;
  if (A.mask != nullptr && (reinterpret_cast<uintptr_t>(A.mask) & 15) == 0) {
    if ((A.klen & 7) != 0) maps->mask_by = attention_mask_in_eights(head_dim, A.sq, A.klen) ? AM_EIGHTS : AM_LOADS;
    else maps->mask_by = attention_mask_in_tiles(head_dim, A.sq, A.klen) ? AM_TILES : AM_LOADS;
  }
  if (maps->mask_by == AM_TILES) {
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(A.klen), static_cast<cuuint64_t>(A.sq), static_cast<cuuint64_t>(batch)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(A.klen) * 2, static_cast<cuuint64_t>(A.sq) * A.klen * 2};
    const cuuint32_t box[3] = {kAttnKeys, kAttnQueries, 1}, elem[3] = {1, 1, 1};
    const CUresult r = encode_fn()(&maps->mask[0], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(A.mask), dims, strides, box, elem,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) maps->mask_by = AM_LOADS;
  }
  const long long rows = static_cast<long long>(batch) * A.sq;
  for (int j = 0; j < 8 && maps->mask_by == AM_EIGHTS; ++j) {
    const int lead = static_cast<int>((static_cast<long long>(j) * A.klen) & 7);  // elements between the boundary and row j's first
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(A.klen) + lead, static_cast<cuuint64_t>((rows - j + 7) / 8)};  // ends with the last row
    const cuuint64_t stride[1] = {static_cast<cuuint64_t>(A.klen) * 16};
    const cuuint32_t box[2] = {kMaskBox, kMaskRows}, elem[2] = {1, 1};
    const CUresult r = encode_fn()(&maps->mask[j], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(A.mask + static_cast<long long>(j) * A.klen - lead), dims,
                                   stride, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) maps->mask_by = AM_LOADS;
  }
  return maps->q_ok ? encode_attention_map(&maps->q, A.q, batch, A.sq, q_heads, head_dim, A.q_ld, A.q_bstride, kAttnQueries) : MK_OK;
}

}  // namespace

struct mk_handle_s {
  bool quick_limit;     // tests: limits shorter than a launch
  mk_config cfg;
  int device, grid;
  uint8_t* ws;
  Carve cv;
  bool bound;
  mk_weights weights;
  std::vector<mk_layer_weights> layers;
  uint32_t epoch, att_epoch;
  int64_t launches;
  long long timeout_cycles;
  float att_scale;
  unsigned long long* trace;
  int trace_cap;
  struct CacheMapSet {
    std::vector<const void*> seen;  // cache pointers the set's descriptors were encoded for (keys, then values)
    int capacity = 0, batch = 0, heads = 0, keys = 0;  // geometry the boxes were encoded for
    uint64_t used = 0;              // launch counter at the last use (least recently used is replaced)
  };
  CacheMapSet kv_sets[kCacheMapSets];
  cudaEvent_t kv_done;  // behind the last mk_kv_attention, once there was one
  bool kv_maps_refused; // tests: the first encoding counts as refused by the driver
  bool kv_maps_ok;      // the driver takes the four-dimensional view of a cache
  bool stream_ok[kStreamPlans];  // the streaming decode kernel's plan for this many token tiles is bound
  int stream_grid[kStreamPlans];  // CTAs of each plan's launches, 0: the plan is not used
  PromptPhase prompt[kPromptClasses][kPromptPhases];
  bool use3d;           // weight descriptors of the tensor engine are three-dimensional (several K chunks per copy)
  uint32_t tp_epoch;    // all-reduces launched so far (tensor parallel)
  uint8_t* tp_peer[kMaxTp];
  bool tp_bound;
  volatile int* mirror;  // host-mapped status word, or null
  std::mutex lock;
};

namespace {

template <typename T>
T* at(mk_handle h, size_t off) { return reinterpret_cast<T*>(h->ws + off); }

// Rows per tile: the smallest height for which the phase's row tiles fit in the
// fewest possible rounds over `slots` CTAs (each round gives every CTA one unit).
int choose_rows(const GemmPhase& ph, int slots, int max_rows = kTileRows) {
  const int nseg = ph.nacc == 2 ? 1 : ph.nseg;
  long long total = 0;
  for (int s = 0; s < nseg; ++s) total += ph.n[s];
  if (slots < 1) slots = 1;
  for (long long rounds = (total + static_cast<long long>(max_rows) * slots - 1) / (static_cast<long long>(max_rows) * slots);;
       ++rounds) {
    for (int rows = static_cast<int>((total + rounds * slots - 1) / (rounds * slots)); rows <= max_rows; ++rows) {
      long long tiles = 0;
      for (int s = 0; s < nseg; ++s) tiles += (ph.n[s] + rows - 1) / rows;
      if (tiles <= rounds * slots) return rows;
    }
  }
}

// A TMA box of fewer than ~40 rows (5 KB) cannot keep an SM's share of HBM
// bandwidth busy (the copy engine retires roughly one box per 0.1 us), so a
// projection with few output rows per CTA is cut along K as well.
constexpr int kGoodBoxRows = 40;

void finish_phase(GemmPhase& ph, int grid, bool allow_split, int max_rows = kTileRows) {
  ph.kc = ph.k / kChunkK;
  int best_split = 1, best_rows = choose_rows(ph, grid, max_rows);
  if (allow_split && best_rows < kGoodBoxRows) {
    static const int candidates[] = {2, 3, 4};
    for (int split : candidates) {
      if (ph.kc % split || ph.kc / split < 2 || grid / split < 1) continue;
      const int rows = choose_rows(ph, grid / split, max_rows);
      if (rows > best_rows) {
        best_rows = rows;
        best_split = split;
      }
      if (rows >= kGoodBoxRows) break;
    }
  }
  ph.ksplit = best_split;
  ph.kslice = ph.kc / best_split;
  ph.rows = best_rows;
  ph.kb = 1;
  ph.gran = (ph.rows * 128 + kGranule - 1) / kGranule;
  const int nseg = ph.nacc == 2 ? 1 : ph.nseg;
  int tile = 0;
  for (int s = 0; s < nseg; ++s) {
    ph.tile_start[s] = tile;
    tile += (ph.n[s] + ph.rows - 1) / ph.rows;
  }
  ph.tile_start[nseg] = tile;
  ph.ntiles = tile;
  ph.nunits = tile * best_split;
}

// Tensor engine: tile heights are multiples of 8 (a swizzled chunk of a tile must start on a 1 KiB boundary
// inside a ring entry), and an entry carries `kb` K chunks per matrix: as many as divide the K range and keep
// the entry under ~36 KB (three entries of the 120 KB ring in flight); two at most when launches can have
// token tiles of 128 (the activation ring holds 64 KB, two entries of 32).
void finish_phase_tc(GemmPhase& ph, int grid, bool allow_split, int max_tokens) {
  finish_phase(ph, grid, allow_split);
  ph.rows = std::min(kTileRows, (ph.rows + 7) / 8 * 8);
  const int nseg = ph.nacc == 2 ? 1 : ph.nseg;
  int tile = 0;
  for (int s = 0; s < nseg; ++s) {
    ph.tile_start[s] = tile;
    tile += (ph.n[s] + ph.rows - 1) / ph.rows;
  }
  ph.tile_start[nseg] = tile;
  ph.ntiles = tile;
  ph.nunits = tile * ph.ksplit;
  int kb = 1;
  for (int cand = 2; cand <= (max_tokens > 64 ? 2 : kOperandChunks); ++cand)
    if (ph.kslice % cand == 0 && ph.nacc * cand * ph.rows * 128 <= 36 * 1024) kb = cand;
  ph.kb = kb;
  ph.gran = ph.nacc * kb * ph.rows / 8;
}

// The split-K table (o_proj and down_proj cut along K so that every SM streams, fp32 partial sums added by
// the next norm phase) serves every launch of a single-GPU handle.
bool split_table_ok(const mk_config& c) { return c.tp_size <= 1; }

void base_params(mk_handle h, KParams& p) {
  memset(&p, 0, sizeof(p));
  const mk_config& c = h->cfg;
  p.hidden = c.hidden; p.layers = c.layers; p.q_heads = c.q_heads; p.kv_heads = c.kv_heads;
  p.head_dim = c.head_dim; p.inter = c.intermediate; p.vocab = c.vocab; p.eps = c.rms_eps;
  p.embed_rows = c.embed_rows > 0 ? c.embed_rows : c.vocab;
  p.tp_size = c.tp_size > 1 ? c.tp_size : 1;
  p.tp_rank = c.tp_size > 1 ? c.tp_rank : 0;
  p.tp_epoch = h->tp_epoch;
  for (int r = 0; r < kMaxTp; ++r) p.tp_peer[r] = h->tp_peer[r];
  p.rope_style = c.rope_style; p.prefill_rope_style = MK_ROPE_HF;
  p.att_scale = h->att_scale;
  p.engine = MK_ENGINE_TCGEN05;
  p.epoch = h->epoch;
  p.att_epoch = h->att_epoch;
  p.qkv_ld = qkv_width(c);
  p.max_positions = c.max_positions;
  p.timeout_cycles = h->timeout_cycles;
  p.trace = h->trace;
  p.trace_cap = h->trace ? h->trace_cap : 0;
  p.status_mirror = h->mirror;
  p.ctrl = at<Control>(h, h->cv.ctrl);
  p.att_xch = at<float>(h, h->cv.att_xch);
  p.att_part = at<float>(h, h->cv.att_part);
  if (h->cv.phases == 0) return;  // a view without decoder buffers (the static-scratch attention): the rest stays null
  p.phases = at<GemmPhase>(h, h->cv.phases);
  p.hidden_buf = at<bf16>(h, h->cv.hidden);
  p.xnorm = at<bf16>(h, h->cv.xnorm);
  p.qkv = at<bf16>(h, h->cv.qkv);
  p.attn = at<bf16>(h, h->cv.attn);
  p.act = at<bf16>(h, h->cv.act);
  p.embed = static_cast<const bf16*>(h->weights.embed);
  p.cos_t = static_cast<const bf16*>(h->weights.rope_cos);
  p.sin_t = static_cast<const bf16*>(h->weights.rope_sin);
}

// Shared-memory attributes belong to the function: set once per device and process (each call costs milliseconds once
// kernels have run).  head_dim 0: the tensor engine only.
int prepare_kernels(int device, int head_dim) {
  constexpr int kDevices = 64;
  static std::mutex lock;
  static bool tensor_done[kDevices], stream_done[kDevices][2];
  std::lock_guard<std::mutex> guard(lock);
  if (device < 0 || device >= kDevices) return fail(MK_ERR_INVALID, "device %d outside [0, %d)", device, kDevices);
  if (!tensor_done[device]) {
    MK_CUDA(cudaFuncSetAttribute(megakernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
    MK_CUDA(cudaFuncSetAttribute(megakernel, cudaFuncAttributePreferredSharedMemoryCarveout, (kSmemBytes * 100 + 233471) / 233472));
    MK_CUDA(prompt_prepare());
    MK_CUDA(cudaFuncSetAttribute(kv_attention_parts<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, KvLaunch<64>::kSmem));
    MK_CUDA(cudaFuncSetAttribute(kv_attention_parts<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, KvLaunch<128>::kSmem));
    int per_sm = 0;
    MK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, megakernel, kThreads, kSmemBytes));
    if (per_sm < 1) return fail(MK_ERR_UNSUPPORTED, "the megakernel does not fit on an SM of device %d", device);
    tensor_done[device] = true;
  }
  if (head_dim && !stream_done[device][head_dim == 128]) {
    for (int i = 0; i < kStreamClasses; ++i)
      MK_CUDA(cudaFuncSetAttribute(stream_kernel(i, head_dim), cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmemLimit));
    stream_done[device][head_dim == 128] = true;
  }
  return MK_OK;
}

int launch(mk_handle h, KParams& p, void* stream, int attention_phases = 0) {
  void* args[] = {&p};
  const int grid = p.splan ? h->stream_grid[stream_plan_of(h->cfg, p.m, h->stream_grid[kStreamFew])] : h->grid;
  // The launch before may have had more CTAs or longer lists: nothing of it stays.
  if (p.trace) MK_CUDA(cudaMemsetAsync(p.trace, 0, sizeof(*p.trace) * p.trace_cap * h->grid, static_cast<cudaStream_t>(stream)));
  if (p.splan)
    MK_CUDA(cudaLaunchCooperativeKernel(stream_kernel(stream_class_of(p.m), p.head_dim), dim3(grid), dim3(kStreamThreads), args,
                                        stream_smem_bytes(p), static_cast<cudaStream_t>(stream)));
  else
    MK_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&megakernel), dim3(grid), dim3(kThreads), args,
                                        kSmemBytes, static_cast<cudaStream_t>(stream)));
  h->epoch += static_cast<uint32_t>(p.nbar) * static_cast<uint32_t>(grid);
  h->att_epoch += static_cast<uint32_t>(attention_phases);
  h->launches += 1;
  return MK_OK;
}

// Whether the RoPE tables begin on boundaries of `bytes`.
bool tables_aligned(mk_handle h, uintptr_t bytes) {
  return ((reinterpret_cast<uintptr_t>(h->weights.rope_cos) | reinterpret_cast<uintptr_t>(h->weights.rope_sin)) & (bytes - 1)) == 0;
}

// The streaming kernel takes decode launches of up to 32 sequences, unless the tensor engine is asked for.  (It reads the RoPE tables in
// words; the tensor engine takes them from any element on.)
bool stream_usable(mk_handle h, int batch, bool ragged) {
  return tables_aligned(h, 4) && batch <= kStreamTokens && h->stream_ok[stream_plan_of(h->cfg, batch, h->stream_grid[kStreamFew])] &&
         h->kv_maps_ok && (ragged ? h->cfg.layers * batch : h->cfg.layers) <= kStreamLengths;
}

int token_tiles(int m) { return (m + token_tile_of(m) - 1) / token_tile_of(m); }

// No wait of the prompt kernels takes 64 tries while work goes on; a limit of less than a millisecond is looked at after each.
PromptGuard prompt_guard(mk_handle h) {
  return {at<Control>(h, h->cv.ctrl), h->mirror, h->timeout_cycles, h->quick_limit ? 0u : 63u};
}

// What the two launches of a decode attention share.  The workspace has one such area: its users order their calls.
struct KvScratch {
  uint32_t* verdict;
  float *stats, *parts;
};
KvScratch workspace_kv_scratch(mk_handle h) {
  return {&at<Control>(h, h->cv.ctrl)->pad, at<float>(h, h->cv.att_xch), at<float>(h, h->cv.att_part)};
}

int launch_kv_attention(mk_handle h, const void* query, const void* key, const void* value, void* key_cache, void* value_cache,
                        int32_t* valid_length, int batch, int capacity, void* output, const KvScratch& scratch, cudaStream_t stream) {
  const mk_config& c = h->cfg;
  const bool small = c.head_dim == 64;
  KvAttentionArgs a{};
  a.q = static_cast<const bf16*>(query); a.knew = static_cast<const bf16*>(key); a.vnew = static_cast<const bf16*>(value);
  a.k = static_cast<bf16*>(key_cache); a.v = static_cast<bf16*>(value_cache); a.out = static_cast<bf16*>(output);
  a.length = valid_length;
  a.verdict = scratch.verdict; a.stats = scratch.stats; a.parts = scratch.parts; a.ctrl = at<Control>(h, h->cv.ctrl);
  a.status_mirror = h->mirror;
  a.batch = batch; a.q_heads = c.q_heads; a.kv_heads = c.kv_heads; a.capacity = capacity;
  a.width = std::min(c.kv_heads, 8);
  while (c.kv_heads % a.width) --a.width;
  a.shares = 8 / a.width;
  // as many runs of positions as make one wave of blocks, but no fewer than four tiles of 16 positions to a warp
  const int blocks_per_run = batch * (c.kv_heads / a.width), wave = h->grid * (small ? KvLaunch<64>::kBlocks : KvLaunch<128>::kBlocks);
  const int by_length = (capacity + 64 * a.shares - 1) / (64 * a.shares);
  a.chunks = std::max(1, std::min({wave / blocks_per_run, kMaxChunks / a.shares, by_length}));
  a.slots = a.chunks * a.shares;
  a.scale_log2 = h->att_scale * kLog2e;
  const int units = blocks_per_run * a.chunks, blocks = c.sm_limit > 0 ? std::min(units, wave) : units;
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.stream = stream;
  config.attrs = &early;
  config.numAttrs = 1;
  config.gridDim = dim3(blocks);
  config.blockDim = dim3(256);
  config.dynamicSmemBytes = small ? KvLaunch<64>::kSmem : KvLaunch<128>::kSmem;
  MK_CUDA(small ? cudaLaunchKernelEx(&config, kv_attention_parts<64>, a, units) : cudaLaunchKernelEx(&config, kv_attention_parts<128>, a, units));
  config.gridDim = dim3((batch * c.q_heads * (c.head_dim / 4) + 127) / 128);
  config.blockDim = dim3(128);
  config.dynamicSmemBytes = 0;
  MK_CUDA(cudaLaunchKernelEx(&config, kv_attention_combine, a, c.head_dim));
  h->launches += 2;
  return MK_OK;
}

// Keys of a prompt: the limit of the interface, 10240 per query head of a KV head.  The kernel, one pass over the keys, has none.
int prompt_keys(mk_handle h) { return (kScoreBytes / 4 / (h->cfg.q_heads / h->cfg.kv_heads)) & ~7; }

int attention_fits(mk_handle h, int keys, const char* what) {
  const int gs = h->cfg.q_heads / h->cfg.kv_heads;
  const int heads = gs * decode_heads_per_unit(h->cfg.kv_heads, gs, h->cfg.head_dim);  // query heads of one attention unit
  const int max_len = (kScoreBytes / 4 / heads) & ~7;
  const int need = (keys + max_len - 1) / max_len;
  if (need > kMaxChunks || need > h->grid)
    return fail(MK_ERR_UNSUPPORTED, "%s: %d keys exceed %d chunks of %d", what, keys, kMaxChunks, max_len);
  return MK_OK;
}

}  // namespace

namespace {
// The streaming decode kernel's plans: descriptors (boxes of 16 rows x the phase's chunks), the per-layer vectors,
// and every CTA's units of each phase.
int bind_stream(mk_handle h, const mk_weights& w, std::vector<CUtensorMap>& maps, std::vector<StreamLayer>& layers,
                std::vector<int>& units, StreamPlan* plans) {
  const mk_config& c = h->cfg;
  const int L = c.layers, q_size = c.q_heads * c.head_dim, kv_size = c.kv_heads * c.head_dim;
  const size_t nmaps = maps_per_table(c);
  maps.resize(kStreamPlans * nmaps);
  units.assign(static_cast<size_t>(kStreamPlans) * kStreamPhases * (kStreamMaxGrid + 1), 0);
  for (int l = 0; l < L; ++l) {
    const mk_layer_weights& lw = w.layers[l];
    StreamLayer& sl = layers[l];
    sl.input_norm = static_cast<const bf16*>(lw.input_norm);
    sl.post_norm = static_cast<const bf16*>(lw.post_norm);
    const void* biases[3] = {lw.q_bias, lw.k_bias, lw.v_bias};
    for (int i = 0; i < 3; ++i) sl.bias[i] = c.qkv_bias ? static_cast<const bf16*>(biases[i]) : nullptr;
  }
  for (int i = 0; i < kStreamPlans; ++i) {
    h->stream_ok[i] = false;
    h->stream_grid[i] = stream_grid(c, i, h->grid);
    if (h->stream_grid[i] == 0) continue;
    StreamPlan& plan = plans[i];
    stream_phases(c, i, h->stream_grid[i], plan.ph);
    for (int l = 0; l < L; ++l) {
      const mk_layer_weights& lw = w.layers[l];
      const void* mats[7] = {lw.q, lw.k, lw.v, lw.o, lw.gate, lw.up, lw.down};
      const int rows[7] = {q_size, kv_size, kv_size, c.hidden, c.intermediate, c.intermediate, c.hidden};
      const int which[7] = {SP_QKV, SP_QKV, SP_QKV, SP_O, SP_GU, SP_GU, SP_DOWN};
      for (int m = 0; m < 7; ++m)
        if (int e = encode_weight_map3(&maps[i * nmaps + 7 * l + m], mats[m], rows[m], plan.ph[which[m]].k, plan.ph[which[m]].rows, kStreamKb)) return e;
    }
    if (int e = encode_weight_map3(&maps[i * nmaps + 7 * L], w.lm_head, c.vocab, c.hidden, plan.ph[SP_HEAD].rows, kStreamKb)) return e;
    int* table = units.data() + static_cast<size_t>(i) * kStreamPhases * (kStreamMaxGrid + 1);
    stream_deal_units(plan.ph, h->stream_grid[i], table);
    plan.maps = at<CUtensorMap>(h, h->cv.smaps) + i * nmaps;
    plan.layers = at<StreamLayer>(h, h->cv.slayers);
    plan.final_norm = static_cast<const bf16*>(w.final_norm);
    plan.units = at<int>(h, h->cv.sunits) + static_cast<size_t>(i) * kStreamPhases * (kStreamMaxGrid + 1);
    for (int half = 0; half < 3; ++half) {
      const int next = (half + 1) % 3;
      bf16 *qkv = at<bf16>(h, h->cv.shalf[0][half]), *attn = at<bf16>(h, h->cv.shalf[1][half]), *res_in = at<bf16>(h, h->cv.shalf[2][half]);
      bf16 *res_next = at<bf16>(h, h->cv.shalf[2][next]), *res_mid = at<bf16>(h, h->cv.shalf[3][half]), *act = at<bf16>(h, h->cv.shalf[4][half]);
      const bf16* src[kStreamPhases] = {res_in, attn, res_mid, act, res_in};
      bf16* dst[kStreamPhases] = {qkv, res_mid, act, res_next, nullptr};
      const bf16* res[kStreamPhases] = {nullptr, res_in, nullptr, res_mid, nullptr};
      for (int k = 0; k < kStreamPhases; ++k) {
        plan.src[k][half] = src[k];
        plan.dst[k][half] = dst[k];
        plan.res[k][half] = res[k];
        plan.part[k][half] = at<float>(h, h->cv.spart[k == SP_O ? 0 : 1][half]);
      }
      plan.attn[half] = attn;
    }
    plan.rec = at<unsigned long long>(h, h->cv.srec);
    h->stream_ok[i] = h->grid <= kStreamMaxGrid;
  }
  return MK_OK;
}
}  // namespace

extern "C" {

const char* mk_last_error(void) { return g_error; }

size_t mk_workspace_bytes(const mk_config* config, int device) {
  if (!config || check_config(*config) != MK_OK) return 0;
  int grid = 0;
  if (device_grid(*config, device, &grid) != MK_OK) return 0;
  return carve(*config, grid).total;
}

int mk_create(const mk_config* config, void* workspace, size_t workspace_bytes, int device, void* stream,
              mk_handle* out) {
  if (!config || !workspace || !out) return fail(MK_ERR_INVALID, "mk_create: null argument");
  if (int e = check_config(*config)) return e;
  if (reinterpret_cast<uintptr_t>(workspace) % 256) return fail(MK_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  MK_CUDA(cudaSetDevice(device));
  int grid = 0;
  if (int e = device_grid(*config, device, &grid)) return e;
  const Carve cv = carve(*config, grid);
  if (workspace_bytes < cv.total)
    return fail(MK_ERR_WORKSPACE, "workspace has %zu bytes, %zu needed", workspace_bytes, cv.total);
  DeviceFacts facts;
  if (int e = device_facts(device, &facts)) return e;
  if (int e = prepare_kernels(device, config->head_dim)) return e;
  mk_handle h = new (std::nothrow) mk_handle_s();
  if (!h) return fail(MK_ERR_INVALID, "out of host memory");
  h->cfg = *config;
  h->device = device;
  h->grid = grid;
  h->ws = static_cast<uint8_t*>(workspace);
  h->cv = cv;
  h->bound = false;
  h->epoch = 0;
  h->att_epoch = 0;
  h->launches = 0;
  h->trace = nullptr;
  h->trace_cap = 0;
  h->mirror = nullptr;
  {  // does this driver take the chunk-major three-dimensional view of a weight matrix?
    CUtensorMap probe;
    h->use3d = getenv("MEGABAKE_NO_3D_MAPS") == nullptr &&
               encode_weight_map3(&probe, workspace, 128, 256, 64, 2) == MK_OK;
  }
  for (int i = 0; i < kStreamPlans; ++i) h->stream_ok[i] = false, h->stream_grid[i] = 0;
  h->kv_maps_ok = getenv("MEGABAKE_NO_CACHE_MAPS") == nullptr;
  h->kv_maps_refused = getenv("MEGABAKE_REFUSE_CACHE_MAPS") != nullptr;
  h->tp_epoch = 0;
  h->tp_bound = false;
  h->kv_done = nullptr;
  for (int r = 0; r < kMaxTp; ++r) h->tp_peer[r] = nullptr;
  double ms = 2000.0;
  if (const char* env = getenv("MEGABAKE_WAIT_LIMIT_MS")) ms = atof(env) > 0 ? atof(env) : ms;
  h->timeout_cycles = static_cast<long long>(ms * static_cast<double>(facts.khz));
  h->quick_limit = ms < 1.0;
  h->att_scale = static_cast<float>(std::pow(static_cast<double>(config->head_dim), -0.5));
  memset(&h->weights, 0, sizeof(h->weights));
  cudaError_t e = cudaMemsetAsync(workspace, 0, cv.total, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) {
    delete h;
    return fail(MK_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
  }
  if (cv.handover_bytes > 0) {
    e = cudaMemsetAsync(h->ws + cv.handover, 0xFF, cv.handover_bytes, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) {
      delete h;
      return fail(MK_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
    }
  }
  *out = h;
  return MK_OK;
}

int mk_destroy(mk_handle h) {
  if (h && h->kv_done) cudaEventDestroy(h->kv_done);
  delete h;
  return MK_OK;
}

int mk_bind_weights(mk_handle h, const mk_weights* w, void* stream) {
  if (!h || !w || !w->layers) return fail(MK_ERR_INVALID, "mk_bind_weights: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  const mk_config& c = h->cfg;
  if (!w->embed || !w->final_norm || !w->lm_head || !w->rope_cos || !w->rope_sin)
    return fail(MK_ERR_INVALID, "mk_bind_weights: embed, final_norm, lm_head and the rope tables are required");
  const int L = c.layers;
  const int q_size = c.q_heads * c.head_dim, kv_size = c.kv_heads * c.head_dim;
  const size_t nmaps = maps_per_table(c), nphases = phases_per_table(c);
  std::vector<CUtensorMap> maps(kPhaseTables * nmaps);
  std::vector<GemmPhase> phases(kPhaseTables * nphases);
  CUtensorMap* dmaps = at<CUtensorMap>(h, h->cv.tmaps);
  CUtensorMap* operand_maps = dmaps + kPhaseTables * nmaps;
  auto operand_map = [&](int kind, int tile, int chunks) { return operand_maps + (kind * kOperandTiles + tile) * kOperandChunks + chunks - 1; };
  bf16* hidden_a = at<bf16>(h, h->cv.hidden);
  bf16* hidden_b = at<bf16>(h, h->cv.hidden2);
  bf16* qkv = at<bf16>(h, h->cv.qkv);
  bf16* attn = at<bf16>(h, h->cv.attn);
  bf16* act = at<bf16>(h, h->cv.act);
  float* partial = at<float>(h, h->cv.partial);
  for (int l = 0; l < L; ++l) {
    const mk_layer_weights& lw = w->layers[l];
    if (!lw.input_norm || !lw.q || !lw.k || !lw.v || !lw.o || !lw.post_norm || !lw.gate || !lw.up || !lw.down)
      return fail(MK_ERR_INVALID, "mk_bind_weights: layer %d has a null weight", l);
    if (c.qkv_bias && (!lw.q_bias || !lw.k_bias || !lw.v_bias))
      return fail(MK_ERR_INVALID, "mk_bind_weights: layer %d lacks a q/k/v bias", l);
  }
  // Table 0: split-K: o and down store K-slice partials; the next
  // normalising phase adds them to the residual stream, which ping-pongs between
  // hidden_b (after attention) and hidden_a (after the MLP).  Table 1: plain.
  bool use3d = h->use3d;
  for (int table = 0; table < kPhaseTables; ++table) {
    const bool split = table != 1;
    if (split && !split_table_ok(c)) continue;
    GemmPhase* tp = phases.data() + table * nphases;
    CUtensorMap* tmaps_host = maps.data() + table * nmaps;
    CUtensorMap* tmaps_dev = dmaps + table * nmaps;
    int prev_parts = 0;  // K slices of the projection whose partials the next normalising phase adds
    for (int l = 0; l < L; ++l) {
      const mk_layer_weights& lw = w->layers[l];
      GemmPhase* ph = tp + 4 * l;
      memset(ph, 0, sizeof(GemmPhase) * 4);
      // q, k, v
      ph[0].nseg = 3; ph[0].nacc = 1; ph[0].k = c.hidden;
      const void* qkv_mats[3] = {lw.q, lw.k, lw.v};
      const int seg_rows[3] = {q_size, kv_size, kv_size};
      const void* biases[3] = {lw.q_bias, lw.k_bias, lw.v_bias};
      int col = 0;
      for (int s = 0; s < 3; ++s) {
        ph[0].tmap[s] = tmaps_dev + 7 * l + s;
        ph[0].w[s] = static_cast<const bf16*>(qkv_mats[s]);
        ph[0].bias[s] = c.qkv_bias ? static_cast<const bf16*>(biases[s]) : nullptr;
        ph[0].n[s] = seg_rows[s];
        ph[0].out_col[s] = col;
        col += seg_rows[s];
      }
      ph[0].epi = EPI_STORE; ph[0].gather = (l == 0);
      ph[0].normw = static_cast<const bf16*>(lw.input_norm);
      ph[0].src = hidden_a; ph[0].src_ld = c.hidden; ph[0].dst = qkv; ph[0].dst_ld = qkv_width(c);
      if (split) {
        ph[0].add_parts = prev_parts; ph[0].partial = partial; ph[0].h_out = hidden_b;
      }
      // o_proj; its activation operand is the attention output (bf16 or chunk partials)
      ph[1].nseg = 1; ph[1].nacc = 1; ph[1].k = q_size;
      ph[1].tmap[0] = tmaps_dev + 7 * l + 3; ph[1].w[0] = static_cast<const bf16*>(lw.o);
      ph[1].n[0] = c.hidden;
      ph[1].epi = split ? EPI_PARTIAL : EPI_RESIDUAL;
      ph[1].src = attn; ph[1].src_ld = q_size; ph[1].dst = hidden_a; ph[1].dst_ld = c.hidden;
      ph[1].partial = partial;
      // gate, up -> silu(gate) * up
      ph[2].nseg = 1; ph[2].nacc = 2; ph[2].k = c.hidden;
      ph[2].tmap[0] = tmaps_dev + 7 * l + 4; ph[2].tmap[1] = tmaps_dev + 7 * l + 5;
      ph[2].w[0] = static_cast<const bf16*>(lw.gate); ph[2].w[1] = static_cast<const bf16*>(lw.up);
      ph[2].n[0] = c.intermediate; ph[2].n[1] = c.intermediate;
      ph[2].epi = EPI_SILU; ph[2].normw = static_cast<const bf16*>(lw.post_norm);
      ph[2].src = split ? hidden_b : hidden_a; ph[2].src_ld = c.hidden; ph[2].dst = act; ph[2].dst_ld = c.intermediate;
      // down
      ph[3].nseg = 1; ph[3].nacc = 1; ph[3].k = c.intermediate;
      ph[3].tmap[0] = tmaps_dev + 7 * l + 6; ph[3].w[0] = static_cast<const bf16*>(lw.down);
      ph[3].n[0] = c.hidden;
      ph[3].epi = split ? EPI_PARTIAL : EPI_RESIDUAL;
      ph[3].src = act; ph[3].src_ld = c.intermediate; ph[3].dst = hidden_a; ph[3].dst_ld = c.hidden;
      ph[3].partial = partial;
      if (c.tp_size > 1) {  // tensor parallel: the residual add moves behind the all-reduce (tp_allreduce)
        ph[1].epi = EPI_TP; ph[1].tp_buf = 0;
        ph[3].epi = EPI_TP; ph[3].tp_buf = 1;
      }
      ph[1].gate = 1;  // decode attention streams cache tiles through the weight ring just before this phase
      for (int i = 0; i < 4; ++i) {
        const bool may_split = split && ph[i].epi == EPI_PARTIAL;
        finish_phase_tc(ph[i], h->grid, may_split, c.max_tokens);
      }
      if (split) {
        ph[2].add_parts = ph[1].ksplit; ph[2].partial = partial; ph[2].h_out = hidden_a;
        prev_parts = ph[3].ksplit;
      }
      for (int t = 0; t < kOperandTiles; ++t) {  // token operands: normalised rows, attention output, SiLU*up
        ph[0].bmap[t] = operand_map(kOperandXnorm, t, ph[0].kb);
        ph[1].bmap[t] = operand_map(kOperandAttn, t, ph[1].kb);
        ph[2].bmap[t] = operand_map(kOperandXnorm, t, ph[2].kb);
        ph[3].bmap[t] = operand_map(kOperandAct, t, ph[3].kb);
      }
      // One TMA descriptor per matrix, boxed to the tile height and the K chunks per copy its phase chose.
      const void* mats[7] = {lw.q, lw.k, lw.v, lw.o, lw.gate, lw.up, lw.down};
      const int rows[7] = {q_size, kv_size, kv_size, c.hidden, c.intermediate, c.intermediate, c.hidden};
      const int ks[7] = {c.hidden, c.hidden, c.hidden, q_size, c.hidden, c.hidden, c.intermediate};
      const int which[7] = {0, 0, 0, 1, 2, 2, 3};
      for (int i = 0; i < 7; ++i)
        if (int e = encode_phase_weight_map(&tmaps_host[7 * l + i], mats[i], rows[i], ks[i], ph[which[i]], use3d)) return e;
    }
    GemmPhase& head = tp[4 * L];
    memset(&head, 0, sizeof(head));
    head.nseg = 1; head.nacc = 1; head.k = c.hidden;
    head.tmap[0] = tmaps_dev + 7 * L; head.w[0] = static_cast<const bf16*>(w->lm_head);
    head.n[0] = c.vocab;
    head.epi = EPI_STORE; head.normw = static_cast<const bf16*>(w->final_norm);
    head.src = hidden_a; head.src_ld = c.hidden; head.to_logits = 1; head.dst_ld = c.vocab;
    if (split) {
      head.add_parts = prev_parts; head.partial = partial;
    }
    finish_phase_tc(head, h->grid, false, c.max_tokens);
    for (int t = 0; t < kOperandTiles; ++t) head.bmap[t] = operand_map(kOperandXnorm, t, head.kb);
    if (int e = encode_phase_weight_map(&tmaps_host[7 * L], w->lm_head, c.vocab, c.hidden, head, use3d)) return e;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  {
    CUtensorMap operand_host[kOperandMaps];
    memset(operand_host, 0, sizeof(operand_host));
    const void* bases[3] = {at<bf16>(h, h->cv.xnorm), attn, act};
    const int widths[3] = {c.hidden, q_size, c.intermediate};
    static const int tiles[kOperandTiles] = {16, 32, 64, 128};
    for (int kind = 0; kind < 3; ++kind)
      for (int t = 0; t < kOperandTiles; ++t)
        for (int chunks = 1; chunks <= kOperandChunks && tiles[t] * chunks * 128 <= kBBytes / 2; ++chunks)
          if (int e = encode_operand_map(&operand_host[(kind * kOperandTiles + t) * kOperandChunks + chunks - 1], bases[kind], c.max_tokens,
                                         widths[kind], tiles[t], chunks, use3d)) return e;
    MK_CUDA(cudaMemcpyAsync(operand_maps, operand_host, sizeof(operand_host), cudaMemcpyHostToDevice, s));
    MK_CUDA(cudaStreamSynchronize(s));
  }
  MK_CUDA(cudaMemcpyAsync(dmaps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, s));
  MK_CUDA(cudaMemcpyAsync(at<GemmPhase>(h, h->cv.phases), phases.data(), phases.size() * sizeof(GemmPhase),
                          cudaMemcpyHostToDevice, s));
  std::vector<CUtensorMap> stream_maps;
  std::vector<StreamLayer> stream_layers(L);
  std::vector<int> stream_units;
  StreamPlan stream_plans[kStreamPlans];
  memset(stream_plans, 0, sizeof(stream_plans));
  if (stream_wanted(c) && h->use3d) {
    if (int e = bind_stream(h, *w, stream_maps, stream_layers, stream_units, stream_plans)) return e;
    MK_CUDA(cudaMemcpyAsync(at<CUtensorMap>(h, h->cv.smaps), stream_maps.data(), stream_maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, s));
    MK_CUDA(cudaMemcpyAsync(at<StreamLayer>(h, h->cv.slayers), stream_layers.data(), stream_layers.size() * sizeof(StreamLayer), cudaMemcpyHostToDevice, s));
    MK_CUDA(cudaMemcpyAsync(at<int>(h, h->cv.sunits), stream_units.data(), stream_units.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    MK_CUDA(cudaMemcpyAsync(at<StreamPlan>(h, h->cv.splan), stream_plans, sizeof(stream_plans), cudaMemcpyHostToDevice, s));
  }
  std::vector<CUtensorMap> prompt_maps(prompt_classes(c, h->grid) * nmaps);
  if (h->use3d && !prompt_maps.empty()) {
    for (int cls = 0; cls < prompt_classes(c, h->grid); ++cls) {
      PromptPhase* const pp = h->prompt[cls];
      prompt_phases(c, cls, h->grid, pp);
      CUtensorMap* const to = prompt_maps.data() + cls * nmaps;
      for (int l = 0; l < L; ++l) {
        const mk_layer_weights& lw = w->layers[l];
        const void* mats[7] = {lw.q, lw.k, lw.v, lw.o, lw.gate, lw.up, lw.down};
        const int rows[7] = {q_size, kv_size, kv_size, c.hidden, c.intermediate, c.intermediate, c.hidden};
        const int which[7] = {PP_QKV, PP_QKV, PP_QKV, PP_O, PP_GU, PP_GU, PP_DOWN};
        for (int i = 0; i < 7; ++i)
          if (int e = encode_weight_map3(&to[7 * l + i], mats[i], rows[i], pp[which[i]].k, prompt_box_rows(pp[which[i]], cls), 1)) return e;
      }
      if (int e = encode_weight_map3(&to[7 * L], w->lm_head, c.vocab, c.hidden, prompt_box_rows(pp[PP_HEAD], cls), 1)) return e;
    }
    MK_CUDA(cudaMemcpyAsync(at<CUtensorMap>(h, h->cv.pmaps), prompt_maps.data(), prompt_maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, s));
  }
  // The source vectors die at return: make sure the copies have read them.
  MK_CUDA(cudaStreamSynchronize(s));
  h->layers.assign(w->layers, w->layers + L);
  h->weights = *w;
  h->weights.layers = h->layers.data();
  h->bound = true;
  return MK_OK;
}

namespace {
int decode_once(mk_handle h, const int64_t* ids, const int64_t* positions, int batch, void* const* key_caches,
                void* const* value_caches, int32_t* const* valid_lengths, int capacity, void* logits, void* stream,
                int64_t* tokens_out = nullptr, bool sample = false, bool ragged = false);

}  // namespace

namespace {
// One decode step (mk_decode), or one step of mk_decode_steps (`sample`: the kernel picks the greedy
// tokens, stores them in tokens_out and as the next ids, and advances the positions).  Lock held.
int decode_step(mk_handle h, const int64_t* ids, const int64_t* positions, int batch, void* const* key_caches,
                void* const* value_caches, int32_t* const* valid_lengths, int capacity, void* logits, void* stream,
                int64_t* tokens_out, bool sample);
}  // namespace

int mk_decode(mk_handle h, const int64_t* ids, const int64_t* positions, int batch, void* const* key_caches,
              void* const* value_caches, int32_t* const* valid_lengths, int capacity, void* logits, void* stream) {
  if (!h || !ids || !positions || !key_caches || !value_caches || !valid_lengths || !logits)
    return fail(MK_ERR_INVALID, "mk_decode: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  return decode_step(h, ids, positions, batch, key_caches, value_caches, valid_lengths, capacity, logits, stream, nullptr, false);
}

int mk_decode_ragged(mk_handle h, const int64_t* ids, const int64_t* positions, int batch, void* const* key_caches,
                     void* const* value_caches, int32_t* const* valid_lengths, int capacity, void* logits, void* stream) {
  if (!h || !ids || !positions || !key_caches || !value_caches || !valid_lengths || !logits)
    return fail(MK_ERR_INVALID, "mk_decode_ragged: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  if (!h->bound) return fail(MK_ERR_UNBOUND, "mk_decode_ragged before mk_bind_weights");
  if (batch < 1 || batch > h->cfg.max_tokens) return fail(MK_ERR_INVALID, "mk_decode_ragged: batch %d outside [1, %d]", batch, h->cfg.max_tokens);
  if (capacity < 1) return fail(MK_ERR_INVALID, "mk_decode_ragged: capacity %d", capacity);
  if (int e = attention_fits(h, capacity, "mk_decode_ragged")) return e;
  for (int l = 0; l < h->cfg.layers; ++l) {
    if (!key_caches[l] || !value_caches[l] || !valid_lengths[l]) return fail(MK_ERR_INVALID, "mk_decode_ragged: layer %d state is null", l);
    if (reinterpret_cast<uintptr_t>(key_caches[l]) % 16 || reinterpret_cast<uintptr_t>(value_caches[l]) % 16)
      return fail(MK_ERR_ALIGNMENT, "mk_decode_ragged: layer %d cache is not 16-byte aligned", l);
  }
  return decode_once(h, ids, positions, batch, key_caches, value_caches, valid_lengths, capacity, logits, stream, nullptr, false, true);
}

int mk_decode_steps(mk_handle h, int64_t* ids, int64_t* positions, int batch, void* const* key_caches,
                    void* const* value_caches, int32_t* const* valid_lengths, int capacity, int steps, int64_t* tokens_out,
                    void* logits, void* stream) {
  if (!h || !ids || !positions || !key_caches || !value_caches || !valid_lengths || !logits || !tokens_out)
    return fail(MK_ERR_INVALID, "mk_decode_steps: null argument");
  if (steps < 1) return fail(MK_ERR_INVALID, "mk_decode_steps: steps %d", steps);
  std::lock_guard<std::mutex> guard(h->lock);
  for (int step = 0; step < steps; ++step)
    if (int e = decode_step(h, ids, positions, batch, key_caches, value_caches, valid_lengths, capacity, logits, stream,
                            tokens_out + static_cast<size_t>(step) * batch, true))
      return e;
  return MK_OK;
}

int mk_decode_step_host(mk_handle h, const int64_t* host_ids, const int64_t* host_positions, int batch,
                        void* const* key_caches, void* const* value_caches, int32_t* const* valid_lengths, int capacity,
                        void* logits, int64_t* host_tokens_out, void* stream) {
  if (!h || !host_ids || !host_positions || !key_caches || !value_caches || !valid_lengths || !logits || !host_tokens_out)
    return fail(MK_ERR_INVALID, "mk_decode_step_host: null argument");
  if (batch < 1 || batch > h->cfg.max_tokens)
    return fail(MK_ERR_INVALID, "mk_decode_step_host: batch %d outside [1, %d]", batch, h->cfg.max_tokens);
  std::lock_guard<std::mutex> guard(h->lock);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t* io = at<int64_t>(h, h->cv.host_io);
  int64_t *ids = io, *positions = io + h->cfg.max_tokens, *tokens = io + 2 * static_cast<size_t>(h->cfg.max_tokens);
  const size_t bytes = static_cast<size_t>(batch) * sizeof(int64_t);
  MK_CUDA(cudaMemcpyAsync(ids, host_ids, bytes, cudaMemcpyHostToDevice, s));
  MK_CUDA(cudaMemcpyAsync(positions, host_positions, bytes, cudaMemcpyHostToDevice, s));
  if (int e = decode_step(h, ids, positions, batch, key_caches, value_caches, valid_lengths, capacity, logits, stream, tokens, true))
    return e;
  MK_CUDA(cudaMemcpyAsync(host_tokens_out, tokens, bytes, cudaMemcpyDeviceToHost, s));
  MK_CUDA(cudaStreamSynchronize(s));
  return MK_OK;
}

namespace {
int decode_step(mk_handle h, const int64_t* ids, const int64_t* positions, int batch, void* const* key_caches,
                void* const* value_caches, int32_t* const* valid_lengths, int capacity, void* logits, void* stream,
                int64_t* tokens_out, bool sample) {
  if (!h->bound) return fail(MK_ERR_UNBOUND, "mk_decode before mk_bind_weights");
  if (batch < 1 || batch > h->cfg.max_tokens) return fail(MK_ERR_INVALID, "mk_decode: batch %d outside [1, %d]", batch, h->cfg.max_tokens);
  if (capacity < 1) return fail(MK_ERR_INVALID, "mk_decode: capacity %d", capacity);
  if (int e = attention_fits(h, capacity, "mk_decode")) return e;
  const int L = h->cfg.layers;
  for (int l = 0; l < L; ++l) {
    if (!key_caches[l] || !value_caches[l] || !valid_lengths[l]) return fail(MK_ERR_INVALID, "mk_decode: layer %d state is null", l);
    if (reinterpret_cast<uintptr_t>(key_caches[l]) % 16 || reinterpret_cast<uintptr_t>(value_caches[l]) % 16)
      return fail(MK_ERR_ALIGNMENT, "mk_decode: layer %d cache is not 16-byte aligned", l);
  }
  return decode_once(h, ids, positions, batch, key_caches, value_caches, valid_lengths, capacity, logits, stream, tokens_out, sample);
}
}  // namespace

namespace {
int decode_once(mk_handle h, const int64_t* ids, const int64_t* positions, int batch, void* const* key_caches,
                void* const* value_caches, int32_t* const* valid_lengths, int capacity, void* logits, void* stream,
                int64_t* tokens_out, bool sample, bool ragged) {
  KParams p;
  base_params(h, p);
  const int L = h->cfg.layers;
  for (int l = 0; l < L; ++l) {
    p.kc[l] = key_caches[l];
    p.vc[l] = value_caches[l];
    p.len[l] = valid_lengths[l];
  }
  const int ntt = token_tiles(batch);
  p.mode = MODE_DECODE; p.m = batch; p.batch = batch; p.seq = 1; p.capacity = capacity;
  p.split = split_table_ok(h->cfg) ? 1 : 0;
  p.phases = at<GemmPhase>(h, h->cv.phases) + (p.split ? 0 : phases_per_table(h->cfg));
  bool streamed = stream_usable(h, batch, ragged);
  p.ragged = ragged ? 1 : 0;
  if (h->kv_maps_ok) {
    // Tiled descriptors of the caches for the tensor engine's decode attention, encoded again only when a
    // cache pointer or the geometry differs from the last call's (the copy is ordered on `stream`
    // before the launch; its pageable source is staged before cudaMemcpyAsync returns).
    const mk_config& c = h->cfg;
    const int gs = c.q_heads / c.kv_heads, row_elems = c.kv_heads * c.head_dim;
    const int hpu = streamed ? stream_heads_per_tile(c, batch) : decode_heads_per_unit(c.kv_heads, gs, c.head_dim);
    const int tile_keys = (streamed ? kStreamSlotBytes : kDecTileBytes) / (c.head_dim * 2 * hpu);
    const bool shape_ok = (hpu & (hpu - 1)) == 0 && tile_keys % 16 == 0 && tile_keys <= 256 && c.head_dim % kChunkK == 0;
    int slot = -1, oldest = 0;
    for (int i = 0; i < kCacheMapSets && shape_ok && slot < 0; ++i) {
      const auto& set = h->kv_sets[i];
      if (set.used < h->kv_sets[oldest].used) oldest = i;
      bool same = static_cast<int>(set.seen.size()) == 2 * L && set.capacity == capacity && set.batch == batch &&
                  set.heads == hpu && set.keys == tile_keys;
      for (int l = 0; l < L && same; ++l) same = set.seen[l] == key_caches[l] && set.seen[L + l] == value_caches[l];
      if (same) slot = i;
    }
    CUtensorMap* const device_sets = at<CUtensorMap>(h, h->cv.kvmaps);
    if (shape_ok && slot < 0) {
      std::vector<CUtensorMap> fresh(2 * static_cast<size_t>(L));
      bool encoded = !h->kv_maps_refused;
      for (int l = 0; l < L && encoded; ++l) {
        encoded = encode_cache_map(&fresh[l], key_caches[l], batch, capacity, row_elems, tile_keys, hpu * (c.head_dim / kChunkK)) == MK_OK &&
                  encode_cache_map(&fresh[L + l], value_caches[l], batch, capacity, row_elems, tile_keys, hpu * (c.head_dim / kChunkK)) == MK_OK;
      }
      if (encoded) {
        slot = oldest;
        MK_CUDA(cudaMemcpyAsync(device_sets + static_cast<size_t>(slot) * 2 * L, fresh.data(), fresh.size() * sizeof(CUtensorMap),
                                cudaMemcpyHostToDevice, static_cast<cudaStream_t>(stream)));
        auto& set = h->kv_sets[slot];
        set.seen.assign(2 * static_cast<size_t>(L), nullptr);
        for (int l = 0; l < L; ++l) {
          set.seen[l] = key_caches[l];
          set.seen[L + l] = value_caches[l];
        }
        set.capacity = capacity;
        set.batch = batch;
        set.heads = hpu;
        set.keys = tile_keys;
      } else {
        h->kv_maps_ok = false;  // this driver refuses the view: the tensor engine with plain copies from here on
      }
    }
    if (slot < 0) streamed = false;
    if (slot >= 0) {
      h->kv_sets[slot].used = static_cast<uint64_t>(h->launches) + 1;
      p.kv_maps = device_sets + static_cast<size_t>(slot) * 2 * L;
    }
  }
  p.n_gemm = 4 * L + 1;
  p.nbar = 7 * L + 1;  // tensor engine: five per layer and one behind each norm phase (two per layer, one for the lm_head)
  if (streamed) {
    const mk_config& c = h->cfg;
    const int plan = stream_plan_of(c, batch, h->stream_grid[kStreamFew]);
    p.splan = at<StreamPlan>(h, h->cv.splan) + plan;
    p.nbar = 1;
    p.stream_hpu = stream_heads_per_tile(c, batch);
    p.stream_tile_keys = kStreamSlotBytes / (c.head_dim * 2 * p.stream_hpu);
    stream_divide(p, stream_scratch_bytes(c, batch), batch);
  }
  p.stream_once = (ntt == 1);
  p.ids = reinterpret_cast<long long*>(const_cast<int64_t*>(ids));
  p.pos = reinterpret_cast<long long*>(const_cast<int64_t*>(positions));
  p.logits = static_cast<bf16*>(logits);
  if (p.tp_size > 1) {
    if (!h->tp_bound) return fail(MK_ERR_UNBOUND, "mk_decode: tensor-parallel handle without mk_tp_bind");
    if (sample) return fail(MK_ERR_UNSUPPORTED, "mk_decode_steps: the device-side sampler needs the whole vocabulary on one rank");
    p.nbar += 2 * L;  // one more grid barrier behind each of the two all-reduces of a layer
  }
  if (sample) {
    p.sample = 1;
    p.tokens_out = reinterpret_cast<long long*>(tokens_out);
    if (!streamed) p.nbar += 1;  // the sampler runs behind one more grid barrier (the streaming kernel already ends with one)
  }
  if (int e = launch(h, p, stream, L)) return e;
  if (p.tp_size > 1) h->tp_epoch += 2u * static_cast<uint32_t>(L);
  return MK_OK;
}
}  // namespace

int mk_prefill(mk_handle h, const int64_t* ids, const int64_t* positions, const void* mask, int batch, int sequence,
               void* logits, void* stream) {
  if (!h || !ids || !positions || !logits) return fail(MK_ERR_INVALID, "mk_prefill: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  if (!h->bound) return fail(MK_ERR_UNBOUND, "mk_prefill before mk_bind_weights");
  const long long m = static_cast<long long>(batch) * sequence;
  if (batch < 1 || sequence < 1 || m > h->cfg.max_tokens)
    return fail(MK_ERR_INVALID, "mk_prefill: %d x %d tokens outside [1, %d]", batch, sequence, h->cfg.max_tokens);
  if (int e = attention_fits(h, sequence, "mk_prefill")) return e;
  if (!tables_aligned(h, 16)) return fail(MK_ERR_ALIGNMENT, "mk_prefill: the rope tables must be 16-byte aligned");
  if (sequence > prompt_keys(h)) return fail(MK_ERR_UNSUPPORTED, "mk_prefill: sequence %d exceeds %d keys", sequence, prompt_keys(h));
  const int L = h->cfg.layers;
  if (h->cfg.tp_size <= 1 && h->use3d) {
    const size_t nmaps = maps_per_table(h->cfg);
    PromptPass pass{};
    pass.config = &h->cfg;
    pass.weights = &h->weights;
    pass.cls = prompt_class(static_cast<int>(m), h->grid);
    pass.grid = h->grid;
    pass.phases = h->prompt[pass.cls];
    pass.maps = at<CUtensorMap>(h, h->cv.pmaps) + pass.cls * nmaps;
    pass.operands = at<CUtensorMap>(h, h->cv.tmaps) + kPhaseTables * nmaps;
    pass.hidden_a = at<bf16>(h, h->cv.hidden); pass.hidden_b = at<bf16>(h, h->cv.hidden2);
    pass.xnorm = at<bf16>(h, h->cv.xnorm); pass.qkv = at<bf16>(h, h->cv.qkv);
    pass.attn = at<bf16>(h, h->cv.attn); pass.act = at<bf16>(h, h->cv.act);
    pass.partial = at<float>(h, h->cv.partial);
    pass.ids = reinterpret_cast<const long long*>(ids);
    pass.pos = reinterpret_cast<const long long*>(positions);
    pass.mask = static_cast<const bf16*>(mask);
    pass.logits = static_cast<bf16*>(logits);
    pass.m = static_cast<int>(m); pass.batch = batch; pass.seq = sequence;
    pass.guard = prompt_guard(h);
    pass.trace = {h->trace, h->trace_cap, h->grid};
    if (h->trace) MK_CUDA(cudaMemsetAsync(h->trace, 0, sizeof(*h->trace) * h->trace_cap * h->grid, static_cast<cudaStream_t>(stream)));
    const mk_config& c = h->cfg;
    const int q_size = c.q_heads * c.head_dim, kv_size = c.kv_heads * c.head_dim;
    AttnArgs A{};
    A.q = pass.qkv; A.q_ld = A.kv_ld = q_size + 2 * kv_size;
    A.q_bstride = A.kv_bstride = static_cast<long long>(sequence) * A.q_ld;
    A.k = pass.qkv + q_size; A.v = A.k + kv_size;
    A.out = pass.attn; A.out_bstride = static_cast<long long>(sequence) * q_size; A.out_tstride = q_size; A.out_hstride = c.head_dim;
    A.mask = pass.mask; A.sq = A.klen = sequence; A.causal = pass.mask == nullptr; A.scale = h->att_scale;
    AttnTcMaps maps{};
    if (int e = encode_attention_maps(&maps, A, c, h->grid, batch, true)) return e;
    pass.attention = &A;
    pass.attention_maps = &maps;
    MK_CUDA(prompt_forward(pass, static_cast<cudaStream_t>(stream)));
    h->launches += 7 * L + 2;
    return MK_OK;
  }
  KParams p;
  base_params(h, p);
  const int ntt = token_tiles(static_cast<int>(m));
  p.mode = MODE_PREFILL; p.m = static_cast<int>(m); p.batch = batch; p.seq = sequence; p.capacity = 0;
  p.split = split_table_ok(h->cfg) ? 1 : 0;
  p.phases = at<GemmPhase>(h, h->cv.phases) + (p.split ? 0 : phases_per_table(h->cfg));
  p.n_gemm = 4 * L + 1;
  p.nbar = 8 * L + 1;  // as decode, plus one behind the rotation of q and k
  p.stream_once = (ntt == 1);
  p.ids = reinterpret_cast<long long*>(const_cast<int64_t*>(ids));
  p.pos = reinterpret_cast<long long*>(const_cast<int64_t*>(positions));
  p.mask = static_cast<const bf16*>(mask);
  p.logits = static_cast<bf16*>(logits);
  if (p.tp_size > 1) {
    if (!h->tp_bound) return fail(MK_ERR_UNBOUND, "mk_prefill: tensor-parallel handle without mk_tp_bind");
    p.nbar += 2 * L;
  }
  if (int e = launch(h, p, stream)) return e;
  if (p.tp_size > 1) h->tp_epoch += 2u * static_cast<uint32_t>(L);
  return MK_OK;
}

int mk_linear(mk_handle h, const void* x, const void* weight, const void* bias, void* y, int m, int n, int k,
              void* stream) {
  if (!h || !x || !weight || !y) return fail(MK_ERR_INVALID, "mk_linear: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  if (m < 1 || m > h->cfg.max_tokens) return fail(MK_ERR_INVALID, "mk_linear: m %d outside [1, %d]", m, h->cfg.max_tokens);
  if (n < 1 || k < 64 || k % 64) return fail(MK_ERR_UNSUPPORTED, "mk_linear: k must be a positive multiple of 64");
  if (reinterpret_cast<uintptr_t>(x) % 16 || reinterpret_cast<uintptr_t>(y) % 2)
    return fail(MK_ERR_ALIGNMENT, "mk_linear: x must be 16-byte aligned");
  KParams p;
  base_params(h, p);
  GemmPhase& ph = p.linear_phase;
  memset(&ph, 0, sizeof(ph));
  ph.nseg = 1; ph.nacc = 1; ph.k = k;
  ph.w[0] = static_cast<const bf16*>(weight); ph.bias[0] = static_cast<const bf16*>(bias);
  ph.n[0] = n;
  ph.epi = EPI_STORE;
  ph.src = static_cast<const bf16*>(x); ph.src_ld = k;
  ph.dst = static_cast<bf16*>(y); ph.dst_ld = n;
  finish_phase_tc(ph, h->grid, false, h->cfg.max_tokens);
  // Phase and descriptors go into the kernel's parameter block: nothing is uploaded, nothing synchronised.
  bool use3d = h->use3d;
  if (int e = encode_phase_weight_map(&p.linear_wmap, weight, n, k, ph, use3d)) return e;
  if (int e = encode_operand_map(&p.linear_xmap, x, m, k, token_tile_of(m), ph.kb, ph.map3d != 0)) return e;
  p.phases = nullptr;
  p.mode = MODE_LINEAR; p.m = m; p.batch = m; p.seq = 1;
  p.n_gemm = 1;
  p.nbar = 0;
  p.stream_once = (token_tiles(m) == 1);
  return launch(h, p, stream);
}

namespace {
int check_kv_attention(mk_handle h, const void* key_cache, const void* value_cache, int batch, int capacity, const char* what) {
  if (batch < 1 || batch > h->cfg.max_tokens) return fail(MK_ERR_INVALID, "%s: batch %d outside [1, %d]", what, batch, h->cfg.max_tokens);
  if (int e = attention_fits(h, capacity, what)) return e;
  if (reinterpret_cast<uintptr_t>(key_cache) % 16 || reinterpret_cast<uintptr_t>(value_cache) % 16)
    return fail(MK_ERR_ALIGNMENT, "%s: caches must be 16-byte aligned", what);
  return MK_OK;
}
}  // namespace

int mk_kv_attention(mk_handle h, const void* query, const void* key, const void* value, void* key_cache,
                    void* value_cache, int32_t* valid_length, int batch, int capacity, void* output, void* stream) {
  if (!h || !query || !key || !value || !key_cache || !value_cache || !valid_length || !output)
    return fail(MK_ERR_INVALID, "mk_kv_attention: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  if (int e = check_kv_attention(h, key_cache, value_cache, batch, capacity, "mk_kv_attention")) return e;
  // The scratch is the handle's: a call waits for the one before it, on whatever stream that was.  (A captured call is
  // ordered by whoever launches the graph: an event from outside would end the capture.)
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  MK_CUDA(cudaStreamIsCapturing(s, &capturing));
  const bool ordered = capturing == cudaStreamCaptureStatusNone;
  if (ordered) {
    if (!h->kv_done) MK_CUDA(cudaEventCreateWithFlags(&h->kv_done, cudaEventDisableTiming));
    else MK_CUDA(cudaStreamWaitEvent(s, h->kv_done, 0));
  }
  if (int e = launch_kv_attention(h, query, key, value, key_cache, value_cache, valid_length, batch, capacity, output, workspace_kv_scratch(h), s))
    return e;
  if (ordered) MK_CUDA(cudaEventRecord(h->kv_done, s));
  return MK_OK;
}

int mk_kv_attention_scratch(mk_handle h, const void* query, const void* key, const void* value, void* key_cache,
                            void* value_cache, int32_t* valid_length, int batch, int capacity, void* output, void* scratch,
                            size_t scratch_bytes, void* stream) {
  if (!h || !query || !key || !value || !key_cache || !value_cache || !valid_length || !output || !scratch)
    return fail(MK_ERR_INVALID, "mk_kv_attention_scratch: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  if (int e = check_kv_attention(h, key_cache, value_cache, batch, capacity, "mk_kv_attention_scratch")) return e;
  if (reinterpret_cast<uintptr_t>(scratch) % 16) return fail(MK_ERR_ALIGNMENT, "mk_kv_attention_scratch: scratch must be 16-byte aligned");
  const size_t need = kv_scratch_bytes(batch, h->cfg.q_heads, h->cfg.head_dim);
  if (scratch_bytes < need) return fail(MK_ERR_WORKSPACE, "mk_kv_attention_scratch: scratch has %zu bytes, %zu needed", scratch_bytes, need);
  uint8_t* const base = static_cast<uint8_t*>(scratch);
  const KvScratch own{reinterpret_cast<uint32_t*>(base), reinterpret_cast<float*>(base + 256),
                      reinterpret_cast<float*>(base + 256 + kv_scratch_stats(batch, h->cfg.q_heads))};
  return launch_kv_attention(h, query, key, value, key_cache, value_cache, valid_length, batch, capacity, output, own,
                             static_cast<cudaStream_t>(stream));
}

size_t mk_kv_attention_scratch_bytes(int batch, int q_heads, int head_dim) {
  return batch < 1 || q_heads < 1 || head_dim < 1 ? 0 : kv_scratch_bytes(batch, q_heads, head_dim);
}

int mk_attention(mk_handle h, const void* query, const void* key, const void* value, const void* mask, float scale,
                 int batch, int q_len, int k_len, void* output, void* stream) {
  if (!h || !query || !key || !value || !output) return fail(MK_ERR_INVALID, "mk_attention: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  if (batch < 1 || q_len < 1 || k_len < 1) return fail(MK_ERR_INVALID, "mk_attention: sizes must be positive");
  if (k_len > prompt_keys(h)) return fail(MK_ERR_UNSUPPORTED, "mk_attention: %d keys exceed %d", k_len, prompt_keys(h));
  if (reinterpret_cast<uintptr_t>(key) % 16 || reinterpret_cast<uintptr_t>(value) % 16)
    return fail(MK_ERR_ALIGNMENT, "mk_attention: key/value must be 16-byte aligned");
  if (reinterpret_cast<uintptr_t>(query) % 4 || reinterpret_cast<uintptr_t>(output) % 4)  // read and written in pairs of elements
    return fail(MK_ERR_ALIGNMENT, "mk_attention: query/output must be 4-byte aligned");
  const int q_size = h->cfg.q_heads * h->cfg.head_dim, kv_size = h->cfg.kv_heads * h->cfg.head_dim;
  AttnArgs A{};
  A.q = static_cast<const bf16*>(query); A.q_bstride = static_cast<long long>(q_len) * q_size; A.q_ld = q_size;
  A.k = static_cast<bf16*>(const_cast<void*>(key)); A.v = static_cast<bf16*>(const_cast<void*>(value));
  A.kv_bstride = static_cast<long long>(k_len) * kv_size; A.kv_ld = kv_size;
  A.out = static_cast<bf16*>(output);  // [batch * heads, q_len, head_dim]
  A.out_bstride = static_cast<long long>(h->cfg.q_heads) * q_len * h->cfg.head_dim;
  A.out_tstride = h->cfg.head_dim; A.out_hstride = q_len * h->cfg.head_dim;
  A.mask = static_cast<const bf16*>(mask); A.sq = q_len; A.klen = k_len; A.scale = scale;
  const long long units = static_cast<long long>(batch) * h->cfg.q_heads * ((q_len + kPromptQueries - 1) / kPromptQueries);
  if (units > INT32_MAX) return fail(MK_ERR_UNSUPPORTED, "mk_attention: %lld blocks of queries", units);
  AttnTcMaps maps{};
  if (int e = encode_attention_maps(&maps, A, h->cfg, h->grid, batch, false)) return e;
  MK_CUDA(prompt_attention_launch(A, maps, prompt_guard(h), h->cfg.head_dim, h->cfg.q_heads, h->cfg.kv_heads,
                                  batch, h->grid, h->cfg.sm_limit > 0, false, static_cast<cudaStream_t>(stream)));
  h->launches += 1;
  return MK_OK;
}

int mk_status(mk_handle h, void* stream, mk_status_info* out) {
  if (!h) return fail(MK_ERR_INVALID, "mk_status: null handle");
  std::lock_guard<std::mutex> guard(h->lock);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  MK_CUDA(cudaStreamSynchronize(s));
  Control c;
  MK_CUDA(cudaMemcpy(&c, at<Control>(h, h->cv.ctrl), sizeof(c), cudaMemcpyDeviceToHost));
  if (out) {
    out->status = c.status; out->where = c.where; out->cta = c.cta; out->detail = c.detail;
  }
  if (c.status != MK_STATUS_OK || c.abort) {
    // Counters are in an unknown state after an aborted launch: start over.
    MK_CUDA(cudaMemset(at<Control>(h, h->cv.ctrl), 0, sizeof(Control)));
    if (h->cv.handover_bytes > 0)  // hand-over words of the aborted launch
      MK_CUDA(cudaMemset(h->ws + h->cv.handover, 0xFF, h->cv.handover_bytes));
    h->epoch = 0;
    if (h->mirror) *h->mirror = 0;
    return fail(MK_ERR_DEVICE_STATUS, "device status %d at site %d (cta %d, detail %d)", c.status, c.where, c.cta, c.detail);
  }
  return MK_OK;
}

int mk_set_status_mirror(mk_handle h, int32_t* host_word) {
  if (!h) return fail(MK_ERR_INVALID, "mk_set_status_mirror: null handle");
  std::lock_guard<std::mutex> guard(h->lock);
  if (host_word) {
    void* device_view = nullptr;
    MK_CUDA(cudaHostGetDevicePointer(&device_view, host_word, 0));  // fails unless the word is pinned, mapped host memory
    *host_word = 0;
    h->mirror = static_cast<volatile int*>(device_view);
  } else {
    h->mirror = nullptr;
  }
  return MK_OK;
}

size_t mk_tp_exchange_bytes(const mk_config* config) {
  if (!config || check_config(*config) != MK_OK || config->tp_size < 2) return 0;
  return kTpFlagBytes + 2 * static_cast<size_t>(config->tp_size) * config->max_tokens * config->hidden * sizeof(float);
}

int mk_tp_bind(mk_handle h, void* const* exchange, size_t exchange_bytes, void* stream) {
  if (!h || !exchange) return fail(MK_ERR_INVALID, "mk_tp_bind: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  const mk_config& c = h->cfg;
  if (c.tp_size < 2) return fail(MK_ERR_INVALID, "mk_tp_bind: the handle was not created for a tensor-parallel group");
  if (exchange_bytes < mk_tp_exchange_bytes(&c))
    return fail(MK_ERR_WORKSPACE, "mk_tp_bind: exchange buffers have %zu bytes, %zu needed", exchange_bytes, mk_tp_exchange_bytes(&c));
  for (int r = 0; r < c.tp_size; ++r) {
    if (!exchange[r]) return fail(MK_ERR_INVALID, "mk_tp_bind: rank %d has no exchange buffer", r);
    if (reinterpret_cast<uintptr_t>(exchange[r]) % 256) return fail(MK_ERR_ALIGNMENT, "mk_tp_bind: exchange buffers must be 256-byte aligned");
    h->tp_peer[r] = static_cast<uint8_t*>(exchange[r]);
  }
  // This rank's own flags start at zero; stamps count up from one.  (Every rank clears its own before any launch:
  // the caller synchronises the group between mk_tp_bind and the first decode.)
  MK_CUDA(cudaMemsetAsync(h->tp_peer[c.tp_rank], 0, kTpFlagBytes, static_cast<cudaStream_t>(stream)));
  h->tp_epoch = 0;
  h->tp_bound = true;
  return MK_OK;
}

int mk_ipc_export(void* pointer, mk_ipc_handle* out) {
  if (!pointer || !out) return fail(MK_ERR_INVALID, "mk_ipc_export: null argument");
  static_assert(sizeof(cudaIpcMemHandle_t) <= sizeof(out->bytes), "handle does not fit");
  cudaIpcMemHandle_t handle;
  MK_CUDA(cudaIpcGetMemHandle(&handle, pointer));
  CUdeviceptr base = 0;
  size_t size = 0;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult found;
  if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &found) != cudaSuccess ||
      found != cudaDriverEntryPointSuccess)
    return fail(MK_ERR_CUDA, "cuMemGetAddressRange is not available from this driver");
  const CUresult r = reinterpret_cast<CUresult (*)(CUdeviceptr*, size_t*, CUdeviceptr)>(fn)(
      &base, &size, reinterpret_cast<CUdeviceptr>(pointer));
  if (r != CUDA_SUCCESS) return fail(MK_ERR_CUDA, "cuMemGetAddressRange failed with %d", static_cast<int>(r));
  memset(out, 0, sizeof(*out));
  memcpy(out->bytes, &handle, sizeof(handle));
  out->offset = static_cast<uint64_t>(reinterpret_cast<CUdeviceptr>(pointer) - base);
  return MK_OK;
}

int mk_ipc_open(const mk_ipc_handle* in, void** pointer, void** base_out) {
  if (!in || !pointer || !base_out) return fail(MK_ERR_INVALID, "mk_ipc_open: null argument");
  cudaIpcMemHandle_t handle;
  memcpy(&handle, in->bytes, sizeof(handle));
  void* base = nullptr;
  MK_CUDA(cudaIpcOpenMemHandle(&base, handle, cudaIpcMemLazyEnablePeerAccess));
  *base_out = base;
  *pointer = static_cast<uint8_t*>(base) + in->offset;
  return MK_OK;
}

int mk_ipc_close(void* base) {
  if (!base) return MK_OK;
  MK_CUDA(cudaIpcCloseMemHandle(base));
  return MK_OK;
}

int mk_describe(mk_handle h, char* buffer, size_t bytes) {
  if (!h || !buffer || bytes == 0) return fail(MK_ERR_INVALID, "mk_describe: null argument");
  std::lock_guard<std::mutex> guard(h->lock);
  size_t used = 0;
  auto add = [&](const char* fmt, ...) {
    if (used >= bytes) return;
    va_list ap;
    va_start(ap, fmt);
    const int n = vsnprintf(buffer + used, bytes - used, fmt, ap);
    va_end(ap);
    if (n > 0) used += static_cast<size_t>(n);
  };
  char streamed[64] = "no";
  if (h->stream_ok[0]) snprintf(streamed, sizeof streamed, "yes");
  int most = 0;  // sequences of the largest launch on fewer CTAs
  while (h->stream_ok[kStreamFew] && most < h->cfg.max_tokens && stream_few_fits(h->cfg, most + 1, h->stream_grid[kStreamFew])) ++most;
  if (most > 0) snprintf(streamed, sizeof streamed, "yes (%d ctas up to batch %d)", h->stream_grid[kStreamFew], most);
  add("ctas %d, weight copies %s, streaming decode %s, tp %d/%d\n", h->grid,
      h->use3d ? "3-D (several K chunks per copy)" : "2-D (one K chunk per copy)", streamed,
      h->cfg.tp_size > 1 ? h->cfg.tp_rank : 0,
      h->cfg.tp_size > 1 ? h->cfg.tp_size : 1);
  if (h->bound) {
    std::vector<GemmPhase> phases(phases_per_table(h->cfg) * kPhaseTables);
    MK_CUDA(cudaMemcpy(phases.data(), at<GemmPhase>(h, h->cv.phases), phases.size() * sizeof(GemmPhase), cudaMemcpyDeviceToHost));
    static const char* names[5] = {"qkv", "o", "gate/up", "down", "lm_head"};
    for (int table = 0; table < kPhaseTables; ++table) {
      if (table == 0 && !split_table_ok(h->cfg)) continue;
      add("table %d:", table);
      for (int i = 0; i < 5; ++i) {
        const GemmPhase& ph = phases[table * phases_per_table(h->cfg) + (i < 4 ? i : 4 * h->cfg.layers)];
        add(" %s rows %d ksplit %d kb %d units %d;", names[i], ph.rows, ph.ksplit, ph.kb, ph.nunits);
      }
      add("\n");
    }
    for (int cls = 0; h->use3d && cls < prompt_classes(h->cfg, h->grid); ++cls) {
      add("prompt class %d:", cls);
      for (int i = 0; i < kPromptPhases; ++i) {
        const PromptPhase& ph = h->prompt[cls][i];
        add(" %s rows %d ksplit %d tiles %d;", names[i], ph.rows, ph.ksplit, ph.tile_start[3]);
      }
      add("\n");
    }
  }
  return MK_OK;
}

int mk_debug_skew_barrier(mk_handle h, uint32_t delta) {
  if (!h) return fail(MK_ERR_INVALID, "mk_debug_skew_barrier: null handle");
  std::lock_guard<std::mutex> guard(h->lock);
  h->epoch += delta;
  return MK_OK;
}

int mk_set_trace(mk_handle h, void* buffer, int events_per_cta) {
  if (!h) return fail(MK_ERR_INVALID, "mk_set_trace: null handle");
  if (buffer && events_per_cta < 1) return fail(MK_ERR_INVALID, "mk_set_trace: events_per_cta must be positive");
  std::lock_guard<std::mutex> guard(h->lock);
  h->trace = static_cast<unsigned long long*>(buffer);
  h->trace_cap = buffer ? events_per_cta : 0;
  return MK_OK;
}

int mk_launch_info(mk_handle h, int32_t* ctas, int32_t* smem_bytes, int64_t* launches) {
  if (!h) return fail(MK_ERR_INVALID, "mk_launch_info: null handle");
  if (ctas) *ctas = h->grid;
  if (smem_bytes) *smem_bytes = kSmemBytes;
  if (launches) *launches = h->launches;
  return MK_OK;
}


}  // extern "C"

// ---------------------------------------------------------------------------
// mk_kv_attention_static: the stand-alone decode attention on scratch that lives
// in the library image instead of in a caller workspace.
//
// Who needs it: a caller that may not obtain device memory at the point of the
// call -- a serving process that handed all of its HBM to its own pool at start
// and forbids later allocations so a request can never fail or stall on one, or
// a call site inside a latency-critical loop where an allocation would
// serialise the device.  Such a caller has no workspace to give mk_create, so
// the exchange buffers of the split-context attention live in a fixed array of
// the module, sized for small decode batches.
constexpr size_t kStaticScratchBytes = 4u << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

namespace {

constexpr int kStaticDevices = 16;

struct StaticSlot {
  bool ready = false;
  uint8_t* base = nullptr;   // device address of g_static_scratch on this device
  int grid = 0;
  long long timeout_cycles = 0;
  uint32_t epoch = 0, att_epoch = 0;
  int64_t launches = 0;
  std::mutex lock;
};
StaticSlot g_static_slots[kStaticDevices];

// Scratch layout: control block, (max, sum, stamp) exchange, fp32 chunk partials.
struct StaticLayout { size_t ctrl, att_xch, att_part, total; };

StaticLayout static_layout(int batch, int q_heads, int kv_heads, int head_dim) {
  StaticLayout v{};
  v.ctrl = 0;
  v.att_xch = align_up(sizeof(Control), 256);
  v.att_part = align_up(v.att_xch + static_cast<size_t>(batch) * kv_heads * kMaxChunks * kExchangeFloats * 4, 256);
  v.total = align_up(v.att_part + static_cast<size_t>(batch) * q_heads * kMaxChunks * head_dim * 4, 256);
  return v;
}

// One-time set-up per device: symbol address, launch attributes, zeroed scratch.
int static_setup(StaticSlot& slot, int device, cudaStream_t stream) {
  DeviceFacts facts;
  if (int e = device_facts(device, &facts)) return e;
  void* address = nullptr;
  const cudaError_t found = cudaGetSymbolAddress(&address, g_static_scratch);
  if (found != cudaSuccess || !address)
    return fail(MK_ERR_CUDA, "cudaGetSymbolAddress(static scratch) on device %d: %s", device, cudaGetErrorString(found));
  if (int e = prepare_kernels(device, 0)) return e;
  // Barrier counter, abort flag, status word and every exchange stamp must start at zero.
  MK_CUDA(cudaMemsetAsync(address, 0, kStaticScratchBytes, stream));
  double ms = 2000.0;
  if (const char* env = getenv("MEGABAKE_WAIT_LIMIT_MS")) ms = atof(env) > 0 ? atof(env) : ms;
  slot.base = static_cast<uint8_t*>(address);
  slot.grid = facts.sms;
  slot.timeout_cycles = static_cast<long long>(ms * static_cast<double>(facts.khz));
  slot.epoch = slot.att_epoch = 0;
  slot.launches = 0;
  slot.ready = true;
  return MK_OK;
}

}  // namespace

extern "C" {

// The status word and the abort flag of the static array, which no handle owns: synchronises
// `stream`, copies them out and, if a launch was refused or gave up a wait, clears them and
// restarts the barrier count, so that the next mk_kv_attention_static call on the device works
// again (without this a timed-out wait would leave the abort flag set for the life of the process
// and every later call would return at its first wait).  Allocates nothing.
int mk_kv_attention_static_status(int device, void* stream, mk_status_info* out) {
  if (device < 0 || device >= kStaticDevices)
    return fail(MK_ERR_INVALID, "mk_kv_attention_static_status: device %d outside [0, %d)", device, kStaticDevices);
  int current = -1;
  MK_CUDA(cudaGetDevice(&current));
  if (current != device)
    return fail(MK_ERR_INVALID, "mk_kv_attention_static_status: device %d is not the current device (%d)", device, current);
  StaticSlot& slot = g_static_slots[device];
  std::lock_guard<std::mutex> guard(slot.lock);
  if (out) out->status = out->where = out->cta = out->detail = 0;
  if (!slot.ready) return MK_OK;  // nothing has run on this device yet
  MK_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  Control c;
  MK_CUDA(cudaMemcpy(&c, slot.base, sizeof(c), cudaMemcpyDeviceToHost));
  if (out) {
    out->status = c.status; out->where = c.where; out->cta = c.cta; out->detail = c.detail;
  }
  if (c.status != MK_STATUS_OK || c.abort) {
    MK_CUDA(cudaMemset(slot.base, 0, sizeof(Control)));
    slot.epoch = 0;
    return fail(MK_ERR_DEVICE_STATUS, "static scratch: device status %d at site %d (cta %d, detail %d)", c.status, c.where,
                c.cta, c.detail);
  }
  return MK_OK;
}

// Overlapping calls on one device (two streams, two threads) share the scratch and race:
// callers serialise them.  The first call on a device does the set-up (symbol lookup,
// function attributes, clearing the scratch on `stream`); make it before any stream capture.
int mk_kv_attention_static(int q_heads, int kv_heads, int head_dim, const void* query, const void* key,
                           const void* value, void* key_cache, void* value_cache, int32_t* valid_length, int batch,
                           int capacity, void* output, int device, void* stream) {
  if (!query || !key || !value || !key_cache || !value_cache || !valid_length || !output)
    return fail(MK_ERR_INVALID, "mk_kv_attention_static: null argument");
  if (device < 0 || device >= kStaticDevices)
    return fail(MK_ERR_INVALID, "mk_kv_attention_static: device %d outside [0, %d)", device, kStaticDevices);
  if (batch < 1 || capacity < 1 || q_heads < 1 || kv_heads < 1)
    return fail(MK_ERR_INVALID, "mk_kv_attention_static: sizes must be positive");
  if (head_dim != 64 && head_dim != 128) return fail(MK_ERR_UNSUPPORTED, "mk_kv_attention_static: head_dim must be 64 or 128");
  if (q_heads % kv_heads || q_heads / kv_heads > 8)
    return fail(MK_ERR_UNSUPPORTED, "mk_kv_attention_static: q_heads must be 1..8 times kv_heads");
  const StaticLayout lay = static_layout(batch, q_heads, kv_heads, head_dim);
  if (lay.total > kStaticScratchBytes)
    return fail(MK_ERR_WORKSPACE,
                "mk_kv_attention_static: batch %d x %d query heads x head_dim %d needs %zu bytes of scratch, the static "
                "array holds %zu; use mk_kv_attention with a caller workspace", batch, q_heads, head_dim, lay.total,
                kStaticScratchBytes);
  if (reinterpret_cast<uintptr_t>(key_cache) % 16 || reinterpret_cast<uintptr_t>(value_cache) % 16)
    return fail(MK_ERR_ALIGNMENT, "mk_kv_attention_static: caches must be 16-byte aligned");
  int current = -1;
  MK_CUDA(cudaGetDevice(&current));
  if (current != device)
    return fail(MK_ERR_INVALID, "mk_kv_attention_static: device %d is not the current device (%d)", device, current);
  StaticSlot& slot = g_static_slots[device];
  std::lock_guard<std::mutex> guard(slot.lock);
  if (!slot.ready) {
    if (int e = static_setup(slot, device, static_cast<cudaStream_t>(stream))) return e;
  }
  // A handle on the stack (no device memory of its own) lets the shared parameter and
  // launch helpers serve this entry point unchanged.
  mk_handle_s view;
  memset(&view.cfg, 0, sizeof(view.cfg));
  view.cfg.hidden = q_heads * head_dim; view.cfg.layers = 1; view.cfg.q_heads = q_heads; view.cfg.kv_heads = kv_heads;
  view.cfg.head_dim = head_dim; view.cfg.intermediate = 64; view.cfg.vocab = 64; view.cfg.rms_eps = 1e-5f;
  view.cfg.rope_style = MK_ROPE_HF; view.cfg.max_tokens = batch; view.cfg.max_positions = capacity;
  view.cfg.engine = MK_ENGINE_TCGEN05;
  view.device = device; view.grid = slot.grid; view.ws = slot.base;
  view.cv = Carve{};
  view.cv.ctrl = lay.ctrl; view.cv.att_xch = lay.att_xch; view.cv.att_part = lay.att_part; view.cv.total = lay.total;
  view.bound = false;
  memset(&view.weights, 0, sizeof(view.weights));
  view.epoch = slot.epoch; view.att_epoch = slot.att_epoch; view.launches = slot.launches;
  view.timeout_cycles = slot.timeout_cycles;
  view.att_scale = static_cast<float>(std::pow(static_cast<double>(head_dim), -0.5));
  for (int i = 0; i < kStreamPlans; ++i) view.stream_ok[i] = false, view.stream_grid[i] = 0;
  view.trace = nullptr; view.trace_cap = 0;
  view.mirror = nullptr; view.use3d = false; view.kv_done = nullptr;
  view.tp_epoch = 0; view.tp_bound = false;
  for (int r = 0; r < kMaxTp; ++r) view.tp_peer[r] = nullptr;
  if (int e = attention_fits(&view, capacity, "mk_kv_attention_static")) return e;
  if (int e = launch_kv_attention(&view, query, key, value, key_cache, value_cache, valid_length, batch, capacity, output,
                                  workspace_kv_scratch(&view), static_cast<cudaStream_t>(stream)))
    return e;
  slot.epoch = view.epoch; slot.att_epoch = view.att_epoch; slot.launches = view.launches;
  return MK_OK;
}

}  // extern "C"
