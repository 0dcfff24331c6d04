#pragma once
// Prompt attention on warp-level tensor cores: short prompts and few queries (attention_on_tcgen05 and
// prompt.cu have the lines to the tcgen05 kernel), and the prompt
// phase of the persistent kernel, which tensor parallel runs.
#include "device_common.cuh"

namespace mk {

struct AttnArgs {
  // query of (sequence b, query token qi, head h): q + b*q_bstride + qi*q_ld + h*head_dim
  const bf16* q; long long q_bstride; int q_ld;
  // key/value of (b, position j, kv head g): k + b*kv_bstride + j*kv_ld + g*head_dim
  bf16* k; bf16* v; long long kv_bstride; int kv_ld;
  // output of (b, qi, h): out + b*out_bstride + qi*out_tstride + h*out_hstride
  bf16* out; long long out_bstride; int out_tstride; int out_hstride;
  const bf16* mask;   // additive bf16 [batch, 1, sq, klen] or null
  int sq;             // query tokens per sequence
  int klen;           // keys per sequence
  int causal;         // without a mask tensor: key j <= query qi
  float scale;
};

// A unit is (sequence, query head, block of 64 query tokens).  The eight worker warps are four row
// groups of 16 query rows times two key halves: warps w and w + 4 keep the same q fragments in registers
// and split every 64-position K / V tile between them (positions 0-31 and 32-63), which halves the
// instruction chain of a tile; their statistics and value sums meet in shared memory at the end of the unit.
// Tiles of the unit's KV head stream through shared memory several stages deep, one block barrier per
// tile; the mask values of the next tile are in registers before it is needed.
// One pass: score = bf16(bf16(q.k) * scale) (+ additive mask, rounded again), the rounding points of the
// reference (src/megabake/lowering.py:274-300, the Hugging Face eager form); softmax in fp32 against the running
// row maximum, the value sums rescaled when it grows; exp(s - maximum) rounded to bf16 for the value product, as
// the probability is there; the division by the fp32 row sum comes last and the result is rounded once.
// What bounds it is the latency of a tile's chain (copy, scores, maximum, exp, values), 16 rows at a time; with a
// second pass over the keys for the exact maximum and sum, waits for every copy and mask loads in the chain
// 32 heads x 512 x 512 masked took 100 us.
// Without a mask tensor attention is causal: key j <= query token index, tiles past the block's last
// query are skipped, and so are the halves a warp's rows cannot see.  Causal blocks cost in proportion to
// their index, so the units are sorted heaviest first.
// One instantiation per head size: the fragment arrays then have their exact extents.
constexpr int kPromptQueries = 64;  // query rows per unit
constexpr int kPromptKeys = 64;     // positions per K / V tile

__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// Programmatic dependent launch: what the kernels before this one have written is there; the kernels behind it may come.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependents_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A launch that is given up: copies and MMAs under way end within microseconds.  A CTA stays for fifty, by the clock (a sleep may
// be shorter than it was asked to be), before its shared and tensor memory are somebody else's.
__device__ __forceinline__ void prompt_stay() {
  unsigned long long begin, now;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(begin));
  int looks = 0;
  do {
    __nanosleep(1000);
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
  } while (now - begin < 50000ull && ++looks < 10000);
}

__device__ __forceinline__ uint32_t ldcg_u32(const void* ptr) { return __ldcg(reinterpret_cast<const unsigned int*>(ptr)); }

template <int HD> constexpr int kPromptPitch = HD * 2 + 16;  // bytes per tile row: 16 bytes of padding keep fragment loads conflict-free
template <int HD> constexpr int kPromptStage = 2 * kPromptKeys * kPromptPitch<HD>;     // a K tile and a V tile
template <int HD> constexpr int kPromptSums = 4 * (HD / 2 + 4) * 32 * 4;  // bytes: [row group][output element or m0, l0, m1, l1][lane]

__device__ __forceinline__ int prompt_units(int batch, int q_heads, int sq) {
  return batch * q_heads * ((sq + kPromptQueries - 1) / kPromptQueries);
}

// Unit i of prompt_units(): 256 threads on named barrier 1.
template <int HD, int kStages>
__device__ __forceinline__ void prompt_unit(const AttnArgs& A, int q_heads, int kv_heads, int batch, int i, uint32_t ring,
                                            float* exchange, int wtid) {
  constexpr int ksteps = HD / 16;  // k steps of the score product
  constexpr int dtiles = HD / 8;   // 8-column tiles of the output row
  constexpr int pitch = kPromptPitch<HD>, kStage = kPromptStage<HD>;
  constexpr int pieces = HD / 8;   // 16-byte pieces per row
  const int gs = q_heads / kv_heads, heads = batch * q_heads;
  const int warp = wtid >> 5, lane = wtid & 31, g = lane >> 2, t = lane & 3;
  const int rw = warp & 3, kh = warp >> 2;  // row group, key half
  const int qblocks = (A.sq + kPromptQueries - 1) / kPromptQueries;
  float* const sums = exchange + rw * (dtiles * 4 + 4) * 32 + lane;
  // mask values come in pairs (keys j, j + 1; j is even) where every row starts on a 4-byte boundary
  const bool pairs = A.mask && (A.klen & 1) == 0 && (reinterpret_cast<uintptr_t>(A.mask) & 3) == 0;
  const bool exact_scale = bf16_round(A.scale) == A.scale;  // head size 64: 1/8; the product is rounded once either way
  const uint32_t scale2 = pack2(A.scale, A.scale);
  const int qb = qblocks - 1 - i / heads, bh = i % heads;  // heaviest first
  const int h = bh % q_heads, b = bh / q_heads, kvh = h / gs;
  const int q0 = qb * kPromptQueries + rw * 16;
  const int r0 = q0 + g, r1 = r0 + 8;  // this thread's two query rows
  const int r0c = min(r0, A.sq - 1), r1c = min(r1, A.sq - 1);
  const bf16* kbase = A.k + b * A.kv_bstride + kvh * HD;
  const bf16* vbase = A.v + b * A.kv_bstride + kvh * HD;
  const int kend = A.causal ? min(A.klen, qb * kPromptQueries + kPromptQueries) : A.klen;
  const int ntiles = (kend + kPromptKeys - 1) / kPromptKeys;

  auto issue = [&](int s) {  // tile s into stage s % kStages; a group of its own, empty past the last tile
    if (s < ntiles) {
      const uint32_t ks_addr = ring + (s % kStages) * kStage, vs_addr = ks_addr + kPromptKeys * pitch;
#pragma unroll
      for (int it0 = 0; it0 < kPromptKeys * pieces; it0 += kWorkers) {
        const int it = it0 + wtid;
        const int r = it / pieces, piece = it % pieces;
        const long long j = static_cast<long long>(min(s * kPromptKeys + r, A.klen - 1)) * A.kv_ld;  // rows past the last key repeat it; they are masked below
        cp_async16(ks_addr + r * pitch + piece * 16, reinterpret_cast<const uint4*>(kbase + j) + piece);
        cp_async16(vs_addr + r * pitch + piece * 16, reinterpret_cast<const uint4*>(vbase + j) + piece);
      }
    }
    cp_async_commit();
  };
  named_bar_sync(1, kWorkers);  // every warp is done with the previous unit's tiles and its exchange area
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) issue(s);
  const bf16* qrow0 = A.q + b * A.q_bstride + static_cast<long long>(r0c) * A.q_ld + h * HD;
  const bf16* qrow1 = A.q + b * A.q_bstride + static_cast<long long>(r1c) * A.q_ld + h * HD;
  uint32_t qf[ksteps][4];
#pragma unroll
  for (int ks = 0; ks < ksteps; ++ks) {
    qf[ks][0] = ldcg_u32(qrow0 + ks * 16 + t * 2);
    qf[ks][1] = ldcg_u32(qrow1 + ks * 16 + t * 2);
    qf[ks][2] = ldcg_u32(qrow0 + ks * 16 + 8 + t * 2);
    qf[ks][3] = ldcg_u32(qrow1 + ks * 16 + 8 + t * 2);
  }
  const bf16* mrow0 = A.mask + (static_cast<long long>(b) * A.sq + r0c) * A.klen;
  const bf16* mrow1 = A.mask + (static_cast<long long>(b) * A.sq + r1c) * A.klen;
  uint32_t mk[4][2];  // mask of this warp's half of the coming tile: [8-key block][row]
  auto load_mask = [&](int s) {  // (plain loads: the kernel that writes the mask may be at work while this one begins)
    if (!A.mask) return;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int j = s * kPromptKeys + kh * 32 + nt * 8 + t * 2;
      if (pairs) {
        const int at = min(j, A.klen - 2);
        mk[nt][0] = *reinterpret_cast<const unsigned int*>(mrow0 + at);
        mk[nt][1] = *reinterpret_cast<const unsigned int*>(mrow1 + at);
      } else {
        const int at = min(j, A.klen - 1), at1 = min(j + 1, A.klen - 1);
        const unsigned short* const row0 = reinterpret_cast<const unsigned short*>(mrow0);
        const unsigned short* const row1 = reinterpret_cast<const unsigned short*>(mrow1);
        mk[nt][0] = row0[at] | static_cast<uint32_t>(row0[at1]) << 16;
        mk[nt][1] = row1[at] | static_cast<uint32_t>(row1[at1]) << 16;
      }
    }
  };
  load_mask(0);

  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;  // maximum of the row, this thread's share of the sum of exp
  float o[dtiles][4];
#pragma unroll
  for (int d = 0; d < dtiles; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
#pragma unroll 1
  for (int s = 0; s < ntiles; ++s) {
    const int j0 = s * kPromptKeys + kh * 32;  // the first key of this warp's half
    const uint32_t ks_addr = ring + (s % kStages) * kStage, vs_addr = ks_addr + kPromptKeys * pitch;
    cp_async_wait_group<kStages - 2>();
    named_bar_sync(1, kWorkers);  // the tile is complete, and every warp has left the stage of the copies that start now
    issue(s + kStages - 1);
    if (j0 >= kend || (A.causal && j0 > q0 + 15)) continue;  // no query of this warp sees its half (barriers stay uniform)
    float sv[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) sv[nt][0] = sv[nt][1] = sv[nt][2] = sv[nt][3] = 0.f;
    const uint32_t krow = ks_addr + (kh * 32 + (lane >> 4) * 8 + (lane & 7)) * pitch + ((lane >> 3) & 1) * 16;
#pragma unroll
    for (int ks = 0; ks < ksteps; ++ks) {
#pragma unroll
      for (int nt = 0; nt < 4; nt += 2) {
        uint32_t kf[4];  // matrices: (keys nt*8..+7, dims ks*16..+7), (same keys, dims + 8), then the same two for keys + 8
        ldmatrix_x4(kf, krow + nt * 8 * pitch + ks * 32);
        mma_bf16_16816(sv[nt], qf[ks], kf[0], kf[1]);
        mma_bf16_16816(sv[nt + 1], qf[ks], kf[2], kf[3]);
      }
    }
    const bool edge = j0 + 32 > A.klen || (A.causal && j0 + 31 > q0);
    float t0 = -INFINITY, t1 = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {  // two scores at a time: one conversion rounds both
        uint32_t v = pack2(sv[nt][r * 2], sv[nt][r * 2 + 1]);
        if (exact_scale) v = mul_bf16x2(v, scale2);
        else v = pack2(__uint_as_float(v << 16) * A.scale, __uint_as_float(v & 0xffff0000u) * A.scale);
        if (A.mask) v = add_bf16x2(v, mk[nt][r]);
        sv[nt][r * 2] = __uint_as_float(v << 16);
        sv[nt][r * 2 + 1] = __uint_as_float(v & 0xffff0000u);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (edge) {
          const int j = j0 + nt * 8 + t * 2 + (e & 1);
          if (j >= A.klen || (A.causal && j > ((e < 2) ? r0 : r1))) sv[nt][e] = -INFINITY;
        }
      }
      t0 = fmaxf(t0, fmaxf(sv[nt][0], sv[nt][1]));
      t1 = fmaxf(t1, fmaxf(sv[nt][2], sv[nt][3]));
    }
    if (s + 1 < ntiles) load_mask(s + 1);
    t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, 1)); t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, 2));
    t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, 1)); t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, 2));
    const float n0 = fmaxf(m0, t0), n1 = fmaxf(m1, t1);
    // exp(x - n) = 2^((x - n) log2(e)), the difference first: a mask of the lowest finite value must not overflow; a row
    // without a visible key so far: 2^(-inf) = 0
    const float s0 = n0 > -INFINITY ? n0 : 0.f, s1 = n1 > -INFINITY ? n1 : 0.f;
    if (__any_sync(0xffffffffu, n0 > m0 || n1 > m1)) {
      const float a0 = ex2((m0 - s0) * kLog2e), a1 = ex2((m1 - s1) * kLog2e);
      l0 *= a0;
      l1 *= a1;
#pragma unroll
      for (int d = 0; d < dtiles; ++d) {
        o[d][0] *= a0; o[d][1] *= a0;
        o[d][2] *= a1; o[d][3] *= a1;
      }
      m0 = n0;
      m1 = n1;
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      sv[nt][0] = ex2((sv[nt][0] - s0) * kLog2e);
      sv[nt][1] = ex2((sv[nt][1] - s0) * kLog2e);
      sv[nt][2] = ex2((sv[nt][2] - s1) * kLog2e);
      sv[nt][3] = ex2((sv[nt][3] - s1) * kLog2e);
      l0 += sv[nt][0] + sv[nt][1];
      l1 += sv[nt][2] + sv[nt][3];
    }
#pragma unroll
    for (int k2 = 0; k2 < 2; ++k2) {  // 16 keys: two score tiles are one A fragment
      const uint32_t pa[4] = {pack2(sv[k2 * 2][0], sv[k2 * 2][1]), pack2(sv[k2 * 2][2], sv[k2 * 2][3]),
                              pack2(sv[k2 * 2 + 1][0], sv[k2 * 2 + 1][1]), pack2(sv[k2 * 2 + 1][2], sv[k2 * 2 + 1][3])};
      const uint32_t vrow = vs_addr + ((kh * 2 + k2) * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * pitch + (lane >> 4) * 16;
#pragma unroll
      for (int d = 0; d < dtiles; d += 2) {
        uint32_t vb[4];
        // matrices: (keys 0..7, dims d*8..), (keys + 8, same dims), then the same two for dims (d+1)*8..
        ldmatrix_x4_trans(vb, vrow + d * 16);
        mma_bf16_16816(o[d], pa, vb[0], vb[1]);
        mma_bf16_16816(o[d + 1], pa, vb[2], vb[3]);
      }
    }
  }
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  // the second half's statistics and fp32 sums join the first half's, which divides, rounds once and stores
  if (kh == 1) {
    sums[0] = m0; sums[32] = l0; sums[64] = m1; sums[96] = l1;
#pragma unroll
    for (int d = 0; d < dtiles; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) sums[(4 + d * 4 + e) * 32] = o[d][e];
  }
  named_bar_sync(1, kWorkers);
  if (kh == 0) {
    // this thread's output elements: rows r0, r1; columns d * 8 + t * 2, + 1
    const float om0 = sums[0], om1 = sums[64];
    const float n0 = fmaxf(m0, om0), n1 = fmaxf(m1, om1);
    const float a0 = m0 > -INFINITY ? expf(m0 - n0) : 0.f, b0 = om0 > -INFINITY ? expf(om0 - n0) : 0.f;
    const float a1 = m1 > -INFINITY ? expf(m1 - n1) : 0.f, b1 = om1 > -INFINITY ? expf(om1 - n1) : 0.f;
    const float w0 = l0 * a0 + sums[32] * b0, w1 = l1 * a1 + sums[96] * b1;
    const float d0 = w0 > 0.f ? w0 : 1.f, d1 = w1 > 0.f ? w1 : 1.f;  // a row that sees no key: zeros
#pragma unroll
    for (int d = 0; d < dtiles; ++d) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        o[d][e] = (o[d][e] * (e < 2 ? a0 : a1) + sums[(4 + d * 4 + e) * 32] * (e < 2 ? b0 : b1)) / (e < 2 ? d0 : d1);
      if (r0 < A.sq)
        *reinterpret_cast<uint32_t*>(A.out + b * A.out_bstride + static_cast<long long>(r0) * A.out_tstride + h * A.out_hstride +
                                     d * 8 + t * 2) = pack2(o[d][0], o[d][1]);
      if (r1 < A.sq)
        *reinterpret_cast<uint32_t*>(A.out + b * A.out_bstride + static_cast<long long>(r1) * A.out_tstride + h * A.out_hstride +
                                     d * 8 + t * 2) = pack2(o[d][2], o[d][3]);
    }
  }
}

// As a kernel: a block per unit.  A unit is a chain of latencies on 8 warps, so what counts is how many are resident: two
// blocks per SM with head size 64 (at most 128 registers), where the persistent kernel holds one.  32 heads of 64, masked:
// 64 positions 9.3 us, 512 21.6 (on tcgen05, with blocks of 128 queries: 10.0 and 14.3).
template <int HD>
struct PromptLaunch {
  static constexpr int kBlocks = HD == 64 ? 2 : 1, kStages = HD == 64 ? 4 : 3;
  static constexpr int kSmem = kStages * kPromptStage<HD> + kPromptSums<HD>;
};
template <int HD>
__global__ void __launch_bounds__(kWorkers, PromptLaunch<HD>::kBlocks)
prompt_attention(const __grid_constant__ AttnArgs A, int q_heads, int kv_heads, int batch, int units) {
  extern __shared__ __align__(128) uint8_t prompt_smem[];
  constexpr int kStages = PromptLaunch<HD>::kStages;
  float* const sums = reinterpret_cast<float*>(prompt_smem + kStages * kPromptStage<HD>);
  grid_dependents_go();
  grid_dependency_wait();
#pragma unroll 1
  for (int i = blockIdx.x; i < units; i += gridDim.x)  // one, unless the handle limits its SMs
    prompt_unit<HD, kStages>(A, q_heads, kv_heads, batch, i, smem_u32(prompt_smem), sums, threadIdx.x);
}

}  // namespace mk
