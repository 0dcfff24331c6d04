#pragma once
// Decode attention on its own (megabake::kv_attention): one query token per sequence against a cache of
// [batch, capacity, kv_heads, head_dim], the new position appended, the valid length moved on by one.
//
// It is bound by reading the cache.  A block takes `width` adjacent KV heads (up to eight) of one sequence and a run of
// positions, a warp one head, or one of the 8 / width shares of its 16-position tiles: the warps of a block read
// together what lies together, 1 KB a position at eight heads of 64, and every warp runs its own copy pipeline
// (cp.async, three stages) without a block barrier.  Blocks of 8 warps, two per SM with head size 64, keep 128 KB of
// copies in flight per SM.  Scores are bf16(q.k) times the scale, the softmax a running one in fp32, the weights rounded
// to bf16 for the value product; every warp leaves its maximum, sum and value sums, and a second launch, which the
// stream orders behind the first, adds them up, divides and rounds once.  What the first launch leaves for the second is the
// call's own: two streams' launches may run side by side.  16 sequences of 1024 positions, 32 heads of 64:
// as a phase of the persistent kernel, whose blocks waited for one another's partial sums, 74 us.  Both launches may begin while
// the kernel before them ends (programmatic dependent launch; they wait before they touch memory): 31.0 -> 28.7 us a call, floor 20.6.
#include "device_common.cuh"
#include "prompt_attention.cuh"

namespace mk {

struct KvAttentionArgs {
  const bf16 *q, *knew, *vnew;
  bf16 *k, *v, *out;
  int* length;
  uint32_t* verdict;  // 1: the first launch refused the length
  float* stats;   // [batch * q_heads][slots][maximum, sum]
  float* parts;   // [batch * q_heads][slots][head_dim]
  Control* ctrl;
  volatile int* status_mirror;
  int batch, q_heads, kv_heads, capacity;
  int width, shares;   // KV heads per block, warps per head
  int chunks, slots;   // runs of positions; slots = chunks * shares
  float scale_log2;
};

// Scratch of a call: [verdict, 256 bytes][stats][parts], sized for the most slots.
inline size_t kv_scratch_stats(int batch, int q_heads) { return (static_cast<size_t>(batch) * q_heads * kMaxChunks * 8 + 255) / 256 * 256; }
inline size_t kv_scratch_bytes(int batch, int q_heads, int head_dim) {
  return 256 + kv_scratch_stats(batch, q_heads) + static_cast<size_t>(batch) * q_heads * kMaxChunks * head_dim * 4;
}

template <int HD>
struct KvLaunch {
  static constexpr int kPitch = HD * 2 + 16, kStage = 2 * 16 * kPitch, kStages = 3, kBlocks = HD == 64 ? 2 : 1;
  static constexpr int kSmem = 8 * kStages * kStage;
};

template <int HD>
__global__ void __launch_bounds__(256, KvLaunch<HD>::kBlocks) kv_attention_parts(const __grid_constant__ KvAttentionArgs a, int units) {
  constexpr int pitch = KvLaunch<HD>::kPitch, kStage = KvLaunch<HD>::kStage, kStages = KvLaunch<HD>::kStages;
  constexpr int ksteps = HD / 16, dtiles = HD / 16, pieces = HD / 8;
  extern __shared__ __align__(128) uint8_t kv_smem[];
  grid_dependents_go();
  grid_dependency_wait();
  const int len = *a.length, n = len + 1;
  const bool bad = len < 0 || n > a.capacity;
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.verdict = bad ? 1u : 0u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int hw = warp % a.width, share = warp / a.width;
  if (bad || share >= a.shares) return;
  const int groups = a.kv_heads / a.width, gs = a.q_heads / a.kv_heads;
  const int kv_size = a.kv_heads * HD, q_size = a.q_heads * HD;
  const int per = ((n + a.chunks - 1) / a.chunks + 15) & ~15;
  uint8_t* const mine = kv_smem + warp * kStages * kStage;
  const uint32_t ring = smem_u32(mine);
#pragma unroll 1
  for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
    const int ch = unit % a.chunks, rest = unit / a.chunks;
    const int kvh = (rest % groups) * a.width + hw, b = rest / groups;
    const int begin = ch * per, end = min(n, begin + per);
    const int tiles = end > begin ? (end - begin + 15) / 16 : 0;
    const int count = tiles > share ? (tiles - share + a.shares - 1) / a.shares : 0;  // this warp's: share, share + shares, ..
    bf16* const kbase = a.k + static_cast<size_t>(b) * a.capacity * kv_size + kvh * HD;
    bf16* const vbase = a.v + static_cast<size_t>(b) * a.capacity * kv_size + kvh * HD;
    const bf16* const knew = a.knew + static_cast<size_t>(b) * kv_size + kvh * HD;
    const bf16* const vnew = a.vnew + static_cast<size_t>(b) * kv_size + kvh * HD;
    auto issue = [&](int i) {  // a group of its own, empty past the last tile
      if (i < count) {
        const int j0 = begin + (share + i * a.shares) * 16;
        const uint32_t ks = ring + (i % kStages) * kStage, vs = ks + 16 * pitch;
#pragma unroll
        for (int it = lane; it < 16 * pieces; it += 32) {
          const int r = it / pieces, piece = it % pieces;
          const size_t at = static_cast<size_t>(min(j0 + r, len)) * kv_size;  // row `len` is put right below
          cp_async16(ks + r * pitch + piece * 16, reinterpret_cast<const uint4*>(kbase + at) + piece);
          cp_async16(vs + r * pitch + piece * 16, reinterpret_cast<const uint4*>(vbase + at) + piece);
        }
      }
      cp_async_commit();
    };
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) issue(i);
    uint32_t qf[ksteps][2];  // B fragments: query head g, dims 2t, + 1 and + 8 of every 16
    {
      const unsigned short* q = reinterpret_cast<const unsigned short*>(a.q) + static_cast<size_t>(b) * q_size + (kvh * gs + g) * HD;
#pragma unroll
      for (int ks = 0; ks < ksteps; ++ks)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int d = ks * 16 + half * 8 + t * 2;
          qf[ks][half] = g < gs ? q[d] | static_cast<uint32_t>(q[d + 1]) << 16 : 0u;
        }
    }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;  // query heads 2t and 2t + 1
    float o[dtiles][4];
#pragma unroll
    for (int d = 0; d < dtiles; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
#pragma unroll 1
    for (int i = 0; i < count; ++i) {
      const int j0 = begin + (share + i * a.shares) * 16;
      const uint32_t ks_addr = ring + (i % kStages) * kStage, vs_addr = ks_addr + 16 * pitch;
      cp_async_wait_group<kStages - 2>();
      __syncwarp();  // every lane's copies are in, and every lane has left the stage that is filled next
      issue(i + kStages - 1);
      if (j0 + 16 > len) {  // the new position: into the cache and into its row of the tile; value rows past it, zero
        unsigned short* const ktile = reinterpret_cast<unsigned short*>(mine + (i % kStages) * kStage);
        unsigned short* const vtile = ktile + 16 * pitch / 2;
        for (int d = lane; d < HD; d += 32) {
          const unsigned short kv = reinterpret_cast<const unsigned short*>(knew)[d], vv = reinterpret_cast<const unsigned short*>(vnew)[d];
          reinterpret_cast<unsigned short*>(kbase + static_cast<size_t>(len) * kv_size)[d] = kv;
          reinterpret_cast<unsigned short*>(vbase + static_cast<size_t>(len) * kv_size)[d] = vv;
          ktile[(len - j0) * (pitch / 2) + d] = kv;
          for (int r = len - j0; r < 16; ++r) vtile[r * (pitch / 2) + d] = r == len - j0 ? vv : 0;
        }
        __syncwarp();
      }
      float s[4] = {0.f, 0.f, 0.f, 0.f};  // (key g, heads 2t, 2t + 1), (key g + 8, same heads)
#pragma unroll
      for (int ks = 0; ks < ksteps; ++ks) {
        uint32_t kf[4];
        ldmatrix_x4(kf, ks_addr + (lane & 15) * pitch + ks * 32 + (lane >> 4) * 16);
        mma_bf16_16816(s, kf, qf[ks][0], qf[ks][1]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] = j0 + g + (e >> 1) * 8 < n ? bf16_round(s[e]) * a.scale_log2 : -INFINITY;
      float n0 = fmaxf(s[0], s[2]), n1 = fmaxf(s[1], s[3]);
#pragma unroll
      for (int x = 4; x < 32; x *= 2) {
        n0 = fmaxf(n0, __shfl_xor_sync(0xffffffffu, n0, x));
        n1 = fmaxf(n1, __shfl_xor_sync(0xffffffffu, n1, x));
      }
      n0 = fmaxf(n0, m0);
      n1 = fmaxf(n1, m1);
      const float s0 = n0 > -INFINITY ? n0 : 0.f, s1 = n1 > -INFINITY ? n1 : 0.f;  // every score so far -inf: weights of zero
      if (__any_sync(0xffffffffu, n0 > m0 || n1 > m1)) {
        const float a0 = ex2(m0 - s0), a1 = ex2(m1 - s1);
        l0 *= a0;
        l1 *= a1;
#pragma unroll
        for (int d = 0; d < dtiles; ++d) {
          o[d][0] *= a0; o[d][1] *= a1;
          o[d][2] *= a0; o[d][3] *= a1;
        }
        m0 = n0;
        m1 = n1;
      }
      s[0] = ex2(s[0] - s0); s[1] = ex2(s[1] - s1);
      s[2] = ex2(s[2] - s0); s[3] = ex2(s[3] - s1);
      l0 += s[0] + s[2];
      l1 += s[1] + s[3];
      const uint32_t p0 = movmatrix_trans(pack2(s[0], s[1])), p1 = movmatrix_trans(pack2(s[2], s[3]));
#pragma unroll
      for (int d = 0; d < dtiles; ++d) {
        uint32_t vf[4];  // V^T: (dims 0-7 | 8-15) x (keys 0-7 | 8-15) from rows (keys) of the tile
        ldmatrix_x4_trans(vf, vs_addr + ((lane & 7) + (lane >> 4) * 8) * pitch + (d * 2 + ((lane >> 3) & 1)) * 16);
        mma_bf16_16816(o[d], vf, p0, p1);
      }
    }
#pragma unroll
    for (int x = 4; x < 32; x *= 2) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, x);
      l1 += __shfl_xor_sync(0xffffffffu, l1, x);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int head = t * 2 + c;
      if (head >= gs) continue;
      const size_t at = (static_cast<size_t>(b) * a.q_heads + kvh * gs + head) * a.slots + ch * a.shares + share;
      if (g == 0) {
        a.stats[at * 2] = c ? m1 : m0;
        a.stats[at * 2 + 1] = c ? l1 : l0;
      }
      if (count == 0) continue;  // its sum is 0 and nobody reads its value sums
#pragma unroll
      for (int d = 0; d < dtiles; ++d) {
        a.parts[at * HD + d * 16 + g] = o[d][c];
        a.parts[at * HD + d * 16 + g + 8] = o[d][2 + c];
      }
    }
  }
}

// Four columns of an output row per thread.
__global__ void __launch_bounds__(128) kv_attention_combine(const __grid_constant__ KvAttentionArgs a, int head_dim) {
  grid_dependents_go();
  grid_dependency_wait();
  const int quads = head_dim / 4, at = blockIdx.x * 128 + threadIdx.x;
  const int row = at / quads, d = (at - row * quads) * 4;
  const bool bad = *a.verdict != 0;
  if (at == 0) {
    if (!bad) {
      *a.length += 1;
    } else if (atomicCAS(&a.ctrl->status, 0, static_cast<int>(MK_STATUS_KV_OVERFLOW)) == 0) {
      a.ctrl->where = SITE_PROLOGUE;
      a.ctrl->cta = 0;
      a.ctrl->detail = 0;
      if (a.status_mirror) *a.status_mirror = static_cast<int>(MK_STATUS_KV_OVERFLOW);
    }
  }
  if (row >= a.batch * a.q_heads) return;
  unsigned short* const out = reinterpret_cast<unsigned short*>(a.out) + static_cast<size_t>(row) * head_dim + d;
  if (bad) {
    for (int e = 0; e < 4; ++e) out[e] = 0x7FC0;  // NaN
    return;
  }
  const float2* const stats = reinterpret_cast<const float2*>(a.stats) + static_cast<size_t>(row) * a.slots;
  const float4* const parts = reinterpret_cast<const float4*>(a.parts + static_cast<size_t>(row) * a.slots * head_dim + d);
  float2 st[kMaxChunks];
  float4 pt[kMaxChunks];
  float top = -INFINITY, total = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int s = 0; s < kMaxChunks; ++s) {
    st[s] = s < a.slots ? __ldcg(stats + s) : make_float2(-INFINITY, 0.f);
    pt[s] = s < a.slots ? __ldcg(parts + static_cast<size_t>(s) * quads) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int s = 0; s < kMaxChunks; ++s) top = fmaxf(top, st[s].x);
#pragma unroll
  for (int s = 0; s < kMaxChunks; ++s) {
    if (st[s].y != 0.f) {  // 0: no position, and no value sums; not a number where a score was not: so is the result
      const float w = ex2(st[s].x - top);
      total += w * st[s].y;
      acc[0] += w * pt[s].x; acc[1] += w * pt[s].y;
      acc[2] += w * pt[s].z; acc[3] += w * pt[s].w;
    }
  }
  for (int e = 0; e < 4; ++e) out[e] = __bfloat16_as_ushort(__float2bfloat16_rn(acc[e] / total));
}

}  // namespace mk
