// Device code shared by the kernels: the launch context and its bounded waits, arithmetic on bf16 vectors, RoPE, refused
// launches and the device-side sampler.
#pragma once
#include "megakernel.cuh"
#include "ptx.cuh"

namespace mk {

struct SmemMisc;
struct SmemMiscTc;

struct Ctx {
  const KParams* p;
  Control* ctrl;
  SmemMisc* misc;
  SmemMiscTc* tc;
  uint8_t* smem_a;
  uint8_t* smem_b;
  long long deadline;
  int cta, grid;
};

// ---------------------------------------------------------------------------
// bounded waits

// Waits between CTAs or GPUs (grid barrier, attention exchange, tensor-parallel flag) give up at the
// deadline; waits inside a CTA's own pipeline (ring slots, accumulators) an eighth of the limit later,
// so that when a peer is late the status names the wait on the peer, not a thread starved behind it.
__device__ __forceinline__ bool give_up(const Ctx& cx, int site, int detail) {
  if (ld_relaxed_u32(&cx.ctrl->abort) != 0) return true;
  const bool internal = site == SITE_PRODUCER_EMPTY || site == SITE_MMA_FULL || site == SITE_MMA_B || site == SITE_MMA_ACC ||
                        site == SITE_EPI_ACC || site == SITE_B_EMPTY || site == SITE_KV_TILE;
  if (clock64() > cx.deadline + (internal ? (cx.p->timeout_cycles >> 3) : 0)) {
    if (atomicCAS(&cx.ctrl->status, 0, static_cast<int>(MK_STATUS_TIMEOUT)) == 0) {
      cx.ctrl->where = site;
      cx.ctrl->cta = cx.cta;
      cx.ctrl->detail = detail;
      if (cx.p->status_mirror) *cx.p->status_mirror = static_cast<int>(MK_STATUS_TIMEOUT);
    }
    atomicExch(&cx.ctrl->abort, 1u);
    __threadfence();
    return true;
  }
  return false;
}

// ---------------------------------------------------------------------------
// arithmetic on rows of activations

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// bf16 -> fp32 is a 16-bit shift; keeping it in integer registers avoids taking addresses.
__device__ __forceinline__ void unpack8(const uint4 u, float* f) {
  f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xFFFF0000u);
  f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xFFFF0000u);
  f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xFFFF0000u);
  f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xFFFF0000u);
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return static_cast<uint32_t>(__bfloat16_as_ushort(h.x)) | (static_cast<uint32_t>(__bfloat16_as_ushort(h.y)) << 16);
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}

// Normalise one 8-element vector: w * bf16(x * rinv), the two roundings of the
// Hugging Face RMSNorm.
// The second product is taken on bf16 pairs: the product of two bf16 values is exact in fp32, so
// the packed multiply's single rounding equals rounding the fp32 product (4 instructions for 8 values;
// the staging loops are bound by the instruction rate of the four worker warps).
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint4 normalise_vec(const uint4 xu, const uint4 wu, float r) {
  float x[8];
  unpack8(xu, x);
  return make_uint4(mul_bf16x2(wu.x, pack2(x[0] * r, x[1] * r)), mul_bf16x2(wu.y, pack2(x[2] * r, x[3] * r)),
                    mul_bf16x2(wu.z, pack2(x[4] * r, x[5] * r)), mul_bf16x2(wu.w, pack2(x[6] * r, x[7] * r)));
}

// 2^x; softmax weights are 2^(s log2(e) - m log2(e)).
constexpr float kLog2e = 1.4426950408889634f;
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float silu(float x) { return x / (1.0f + expf(-x)); }
// The same for |x| < 80 without a branch, so that several overlap: a quotient from an approximate reciprocal, corrected by
// its remainder (Markstein, 1990).  For every bf16 x in that range the result has the bits of the division above (the sign
// of zero aside).
__device__ __forceinline__ float silu_inner(float x) {
  const float d = 1.0f + expf(-x), y = __fdividef(1.0f, d), q = x * y;
  return fmaf(fmaf(-q, d, x), y, q);
}

// A value that rounds to the bf16 of the division's result, from two approximations and no branch: for each of the 65536 bf16 x,
// infinities and not-numbers included.  (The reciprocal must not flush: 2^-127 times x = -88 is a normal bf16.)  In the prompts' gate/up, whose
// epilogue follows its unit, 1.7B shape, 64 tokens 1264 -> 1252 us, 128 1437 -> 1426, 300 2261 -> 2226, 512 2432 -> 2409.
__device__ __forceinline__ float silu_to_bf16(float x) {
  float y;
  asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(1.0f + ex2(x * -kLog2e)));
  return x * y;
}

// exp(score - max) over the sum of a softmax, for weights that are zero or at least kQuotientLeast: without a branch, so that
// several overlap.  `reciprocal` is 1 / sum, rounded; a quotient that two remainders have corrected has the bits of the division
// (Markstein, 1990), and within these limits no remainder is lost to underflow.
constexpr float kQuotientLeast = 0x1p-60f;
__device__ __forceinline__ bool quotient_fits(float weight) { return !(weight > 0.f && weight < kQuotientLeast); }
__device__ __forceinline__ float quotient(float weight, float sum, float reciprocal) {
  float q = weight * reciprocal;
  q = fmaf(fmaf(-q, sum, weight), reciprocal, q);
  return fmaf(fmaf(-q, sum, weight), reciprocal, q);
}

__device__ __forceinline__ float ldcg_bf16(const bf16* ptr) {
  return __bfloat162float(__ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(ptr))));
}

__device__ __forceinline__ void rope_pair(float x1, float x2, float c, float s, int style, float& first, float& second) {
  if (style == MK_ROPE_HALF_SWAP) {
    const float a = bf16_round(x1 * c), b = bf16_round(x2 * s);
    first = bf16_round(a - b);
    second = bf16_round(b + a);
  } else {
    first = bf16_round(bf16_round(x1 * c) + bf16_round(-x2 * s));
    second = bf16_round(bf16_round(x2 * c) + bf16_round(x1 * s));
  }
}

// ---------------------------------------------------------------------------
// outputs of a launch that the prologue refused, and the device-side greedy sampler

// A launch whose prologue found a bad id, position or a full cache does no work.  Its outputs are
// filled with NaN so that a caller who reads them before looking at the status cannot mistake
// uninitialised memory for logits (the reference raises at this point: src/megabake/lowering.py:229).
static __device__ __noinline__ void refuse_outputs(const Ctx& cx, int bad, int tid, int nthreads) {
  const KParams& p = *cx.p;
  bf16* out = nullptr;
  long long count = 0;
  if (p.mode == MODE_DECODE || p.mode == MODE_PREFILL) {
    out = p.logits;
    count = static_cast<long long>(p.m) * p.vocab;
  }
  const bf16 nan = __ushort_as_bfloat16(0x7FC0);
  for (long long i = static_cast<long long>(cx.cta) * nthreads + tid; out != nullptr && i < count;
       i += static_cast<long long>(cx.grid) * nthreads)
    out[i] = nan;
  if (cx.cta == 0 && tid == 0) {
    if (atomicCAS(&cx.ctrl->status, 0, bad) == 0) {
      cx.ctrl->where = SITE_PROLOGUE;
      cx.ctrl->cta = 0;
      cx.ctrl->detail = 0;
      if (p.status_mirror) *p.status_mirror = bad;
    }
    if (p.sample && p.tokens_out)
      for (int t = 0; t < p.m; ++t) p.tokens_out[t] = -1;
  }
  // Keep the monotonic barrier counter consistent with what the host expects.
  if (tid == 0 && p.nbar > 0) atomicAdd(&cx.ctrl->barrier, static_cast<uint32_t>(p.nbar));
}

// Greedy token of every sequence of the launch, taken from the bf16 logits the lm_head phase has
// written (the caller has passed a grid barrier since): the largest value, the lowest index among
// equal ones, as torch.argmax on the host would return.  CTA t serves token t.  The token goes to
// tokens_out[t] and becomes the next launch's id; the position moves on by one.  The kCount calling
// threads synchronise on named barrier kBarrier; `scratch` holds 64 words of shared memory.
template <int kBarrier, int kCount>
__device__ __noinline__ void greedy_sample(const Ctx& cx, int wtid, float* scratch) {
  const KParams& p = *cx.p;
  constexpr int nthreads = kCount;
  auto sync = [] { named_bar_sync(kBarrier, kCount); };
  const int lane = wtid & 31, warp = wtid >> 5, nwarps = nthreads >> 5;
  int* scratch_idx = reinterpret_cast<int*>(scratch + 32);
  for (int t = cx.cta; t < p.m; t += cx.grid) {
    const bf16* row = p.logits + static_cast<size_t>(t) * p.vocab;
    float best = -INFINITY;
    int idx = 0x7fffffff;
    if ((p.vocab & 7) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {  // (logits may begin at any element)
      // Eight vectors in flight: with one, a vocabulary of 49152 was 24 round trips to L2.
      constexpr int kAhead = 8;
      const uint4* vrow = reinterpret_cast<const uint4*>(row);
      const int count = p.vocab / 8;
#pragma unroll 1
      for (int v0 = wtid; v0 < count; v0 += kAhead * nthreads) {
        uint4 u[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i) u[i] = __ldcg(vrow + min(v0 + i * nthreads, count - 1));
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const int v = v0 + i * nthreads;
          float f[8];
          unpack8(u[i], f);
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (v < count && f[e] > best) { best = f[e]; idx = v * 8 + e; }
        }
      }
    } else {
      for (int i = wtid; i < p.vocab; i += nthreads) {
        const float f = ldcg_bf16(row + i);
        if (f > best) { best = f; idx = i; }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
      if (ob > best || (ob == best && oi < idx)) { best = ob; idx = oi; }
    }
    sync();  // the scratch of the previous token has been read
    if (lane == 0) { scratch[warp] = best; scratch_idx[warp] = idx; }
    sync();
    if (wtid == 0) {
      for (int w = 1; w < nwarps; ++w)
        if (scratch[w] > best || (scratch[w] == best && scratch_idx[w] < idx)) { best = scratch[w]; idx = scratch_idx[w]; }
      if (idx == 0x7fffffff) idx = 0;  // every logit NaN
      if (p.tokens_out) p.tokens_out[t] = idx;
      p.ids[t] = idx;
      p.pos[t] += 1;
    }
  }
}

}  // namespace mk
