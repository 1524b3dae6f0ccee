// Attention of a few queries over a long key range (cached decoding), and the lowering of boolean masks.
//
// Decoding reads every cached key and value once and does next to no arithmetic, so bytes in flight decide.  The tile kernels give a
// (row, query head) one CTA with 128 query rows of which one is real, and read a key head once per query head.  Here a key head's query
// heads (times the queries of the call) are the up to 16 rows of one m16n8k16 tile, so keys and values are read once; a 64-key block is
// split over the four warps of a CTA, each with its own cp.async ring (3 stages of 16 keys, two CTAs per SM: 128 KB in flight) and its own
// running maximum, sum and output in registers.  Blocks are dealt round-robin to the up to 8 CTAs of a cluster, which meet once at the end in
// distributed shared memory: no workspace, no second launch.  Blocks without a visible key are not read, so the unused end of a cache costs
// its mask bytes only.
// One layer of a decode step with its mask (32 / 8 heads, cold L2, launch included), before on the one-tile kernel and here:
//   1 x 61 slots of 64: 116 -> 9 us;  16 x 732 of 128: 374 -> 31 us;  2 x 8012 of 128: 855 -> 31 us;  64 x 4096 of 128: 5287 -> 199 us (5.4 TB/s).
//
// Matrix operands are bf16 with fp32 accumulation, probabilities bf16 in the second product and fp32 in the sum, as in the tile kernels.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/ptx.cuh"
#include "common/tmap.h"

TTB_DEFINE_VIOLATION_COUNTER(decode)

namespace ttb {
namespace dec {

namespace cg = cooperative_groups;

static constexpr int kWarps = 4;
static constexpr int kKeys = 16 * kWarps;  // keys of a block; 16 per warp
static constexpr int kStages = 3;
static constexpr int kMaxRows = 16;
static constexpr int kMaxSplit = 8;          // portable cluster size
static constexpr int kMaxBitBytes = 16384;   // visibility words of one CTA
static constexpr float kLog2e = 1.4426950408889634f;

struct Params {
  const __nv_bfloat16* q;  // [b, s, hq, D]
  const __nv_bfloat16* k;  // [b, sk, hkv, D]
  const __nv_bfloat16* v;
  __nv_bfloat16* o;        // [b, s, hq, D]
  const uint8_t* mask;     // row (b, i) at mask + b * mask_b + i * mask_r, sk bytes, nonzero = visible; or nullptr
  long long mask_b, mask_r;
  const int* lo;           // [b, s] first / last visible key, or nullptr (0 / sk - 1)
  const int* hi;
  int s, sk, hq, hkv;
  float scale;
  // APPEND: one query per row; q is still to be rotated, and the new key (to be rotated as well) and value go to slot slots[0] of the caches k and v first
  const __nv_bfloat16 *k_new, *v_new;  // [b, hkv, D]
  const float* rope;                   // [rope_len, D / 2, 2] cosine and sine
  const int* pos;                      // [b]
  const long long* slots;
  int rope_len, interleaved;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool keep) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(keep ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int D>
struct Layout {
  static constexpr int kTile = 16 * D * 2;                    // 16 keys of one operand
  static constexpr int kWarpBytes = kStages * 2 * kTile;      // ring of one warp
  static constexpr int kRing = kWarps * kWarpBytes;
  static constexpr int kPart = kMaxRows * D * 4;              // fp32 output of one warp; reuses the warp's ring
  static_assert(kPart <= kWarpBytes, "a warp's partial output fits its ring");
  static constexpr int kStats = (kWarps + 1) * kMaxRows * 2 * 4;  // maximum and sum per warp, and of the CTA
  static constexpr int kQueryPitch = D * 2 + 16;
  static constexpr int kQueries = kMaxRows * kQueryPitch;         // APPEND: the rotated queries
};

// grid (splits = cluster, key heads, batch)
// With APPEND the step between the projections and the cache, a launch of 2 - 5 us that moved a few KB, happens here: the queries are rotated into shared memory, and the CTA whose
// blocks hold the new slot writes the cache before it reads.
template <int D, bool APPEND>
__global__ void __launch_bounds__(kWarps * 32)
decode_kernel(Params p) {
  using L = Layout<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  float* stats = reinterpret_cast<float*>(smem + L::kRing);
  uint64_t* bits = reinterpret_cast<uint64_t*>(smem + L::kRing + L::kStats + (APPEND ? L::kQueries : 0));  // [own blocks][s + 1]: one word per query, then their union
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x, splits = gridDim.x, hk = blockIdx.y, bi = blockIdx.z;
  const int group = p.hq / p.hkv, rows = p.s * group;
  const int blocks = (p.sk + kKeys - 1) / kKeys;
  const int own = blocks > split ? (blocks - split + splits - 1) / splits : 0;
  const int words = p.s + 1;

  // Which keys of the own blocks each query sees, one bit per key.
  for (int w = warp; w < own * p.s; w += kWarps) {
    const int i = w / p.s, qi = w % p.s;
    const int j0 = (split + i * splits) * kKeys;
    const long long row = static_cast<long long>(bi) * p.s + qi;
    const int lo = p.lo != nullptr ? p.lo[row] : 0, hi = p.hi != nullptr ? p.hi[row] : p.sk - 1;
    uint32_t half[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int j = j0 + x * 32 + lane;
      bool seen = j < p.sk && j >= lo && j <= hi;
      if (seen && p.mask != nullptr) seen = p.mask[bi * p.mask_b + qi * p.mask_r + j] != 0;
      half[x] = __ballot_sync(0xffffffffu, seen);
    }
    if (lane == 0) bits[i * words + qi] = static_cast<uint64_t>(half[1]) << 32 | half[0];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < own; i += kWarps * 32) {
    uint64_t any = 0;
    for (int qi = 0; qi < p.s; ++qi) any |= bits[i * words + qi];
    bits[i * words + p.s] = any;
  }

  // Query rows as the A operand: row r is query r / group, head r % group of this key head.
  uint32_t qf[D / 16][4];
  const int r0 = lane >> 2, r1 = r0 + 8;
  const int q0 = r0 / group, q1 = r1 / group;  // query of the two rows of this lane
  if constexpr (APPEND) {
    uint8_t* queries = smem + L::kRing + L::kStats;
    const long long slot = p.slots[0];
    const bool mine = slot >= 0 && slot < p.sk && static_cast<int>(slot / kKeys) % splits == split;  // the host has checked the cache's own counter; nothing is written outside it
    int at = p.pos[bi];
    if (at < 0 || at >= p.rope_len) {
      if (threadIdx.x == 0 && hk == 0 && split == 0) TTB_NOTE_VIOLATION(decode);
      at = 0;
    }
    const float2* table = reinterpret_cast<const float2*>(p.rope + static_cast<long long>(at) * D);
    const __nv_bfloat16* q = p.q + (static_cast<long long>(bi) * p.hq + hk * group) * D;
    const long long new_at = (static_cast<long long>(bi) * p.hkv + hk) * D;
    const long long cache_at = ((static_cast<long long>(bi) * p.sk + slot) * p.hkv + hk) * D;
    for (int idx = threadIdx.x; idx < (kMaxRows + 1) * (D / 2); idx += kWarps * 32) {
      const int r = idx / (D / 2), e = idx % (D / 2);
      const int c0 = p.interleaved ? 2 * e : e, c1 = p.interleaved ? 2 * e + 1 : e + D / 2;
      __nv_bfloat16 o0 = __float2bfloat16_rn(0.f), o1 = o0;  // unused rows of the tile are zeros
      if (r < group || (r == kMaxRows && mine)) {
        const __nv_bfloat16* src = r < kMaxRows ? q + r * D : p.k_new + new_at;
        const float x = __bfloat162float(src[c0]), y = __bfloat162float(src[c1]);
        const float2 cs = table[e];
        o0 = __float2bfloat16_rn(x * cs.x - y * cs.y), o1 = __float2bfloat16_rn(y * cs.x + x * cs.y);
      }
      if (r < kMaxRows) {
        __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(queries + r * L::kQueryPitch);
        to[c0] = o0, to[c1] = o1;
      } else if (mine) {
        const_cast<__nv_bfloat16*>(p.k)[cache_at + c0] = o0, const_cast<__nv_bfloat16*>(p.k)[cache_at + c1] = o1;
      }
    }
    if (mine && threadIdx.x < D / 8)
      *reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(p.v) + cache_at + threadIdx.x * 8) = *reinterpret_cast<const uint4*>(p.v_new + new_at + threadIdx.x * 8);
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) ldsm4(smem_u32(queries) + (((lane >> 3) & 1) * 8 + (lane & 7)) * L::kQueryPitch + kk * 32 + (lane >> 4) * 16, qf[kk]);
  } else {
    auto qrow = [&](int r) { return p.q + ((static_cast<long long>(bi) * p.s + r / group) * p.hq + hk * group + r % group) * D; };
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      const int c = kk * 16 + (lane & 3) * 2;
      qf[kk][0] = r0 < rows ? *reinterpret_cast<const uint32_t*>(qrow(r0) + c) : 0u;
      qf[kk][1] = r1 < rows ? *reinterpret_cast<const uint32_t*>(qrow(r1) + c) : 0u;
      qf[kk][2] = r0 < rows ? *reinterpret_cast<const uint32_t*>(qrow(r0) + c + 8) : 0u;
      qf[kk][3] = r1 < rows ? *reinterpret_cast<const uint32_t*>(qrow(r1) + c + 8) : 0u;
    }
    __syncthreads();
  }

  const uint32_t ring = smem_u32(smem) + warp * L::kWarpBytes;
  const int shift = warp * 16;
  const long long pitch = static_cast<long long>(p.hkv) * D;
  const __nv_bfloat16* kb = p.k + (static_cast<long long>(bi) * p.sk * p.hkv + hk) * D;
  const __nv_bfloat16* vb = p.v + (static_cast<long long>(bi) * p.sk * p.hkv + hk) * D;
  auto next = [&](int i) {  // next own block in which this warp's 16 keys hold a visible one
    while (i < own && ((bits[i * words + p.s] >> shift) & 0xffffu) == 0) ++i;
    return i;
  };
  constexpr int kChunks = D / 8;  // 16-byte chunks of a key
  auto load = [&](int i, int stage) {
    if (i < own) {
      const int j0 = (split + i * splits) * kKeys + shift;
      const uint32_t any = static_cast<uint32_t>(bits[i * words + p.s] >> shift) & 0xffffu;
#pragma unroll
      for (int c = lane; c < 16 * kChunks; c += 32) {
        const int key = c / kChunks, ch = c % kChunks;
        const bool keep = (any >> key) & 1u;  // masked keys (and slots past the end) are zeros, whatever the cache holds there
        const long long off = keep ? (j0 + key) * pitch + ch * 8 : 0;
        const uint32_t dst = ring + stage * 2 * L::kTile + key * (D * 2) + ((ch ^ (key & 7)) << 4);
        cp16(dst, kb + off, keep);
        cp16(dst + L::kTile, vb + off, keep);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  const float c = p.scale * kLog2e;

  int cur = next(0), ahead = cur;
#pragma unroll
  for (int st = 0; st < kStages - 1; ++st) {
    load(ahead, st);
    if (ahead < own) ahead = next(ahead + 1);
  }
  for (int it = 0; cur < own; ++it) {
    load(ahead, (it + kStages - 1) % kStages);
    if (ahead < own) ahead = next(ahead + 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
    __syncwarp();
    const uint32_t tk = ring + (it % kStages) * 2 * L::kTile, tv = tk + L::kTile;
    float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    const int mrow = lane & 7, msel = lane >> 3;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      // matrices: keys 0-7 / dims 0-7, keys 0-7 / dims 8-15, keys 8-15 / dims 0-7, keys 8-15 / dims 8-15
      const int key = (msel >> 1) * 8 + mrow, ch = kk * 2 + (msel & 1);
      uint32_t b[4];
      ldsm4(tk + key * (D * 2) + ((ch ^ (key & 7)) << 4), b);
      mma16816(sc[0], qf[kk], b[0], b[1]);
      mma16816(sc[1], qf[kk], b[2], b[3]);
    }
    const uint32_t w0 = r0 < rows ? static_cast<uint32_t>(bits[cur * words + q0] >> shift) : 0u;
    const uint32_t w1 = r1 < rows ? static_cast<uint32_t>(bits[cur * words + q1] >> shift) : 0u;
    float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = n * 8 + (lane & 3) * 2 + e;
        sc[n][e] = (w0 >> j) & 1u ? sc[n][e] * c : -INFINITY;
        sc[n][2 + e] = (w1 >> j) & 1u ? sc[n][2 + e] * c : -INFINITY;
        x0 = fmaxf(x0, sc[n][e]);
        x1 = fmaxf(x1, sc[n][2 + e]);
      }
    }
    x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 1));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 1));
    x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 2));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 2));
    const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
    const float base0 = n0 == -INFINITY ? 0.f : n0, base1 = n1 == -INFINITY ? 0.f : n1;
    const float f0 = fast_exp2(m0 - base0), f1 = fast_exp2(m1 - base1);
    m0 = n0, m1 = n1;
    uint32_t pf[4];
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const float e0 = fast_exp2(sc[n][0] - base0), e1 = fast_exp2(sc[n][1] - base0);
      const float e2 = fast_exp2(sc[n][2] - base1), e3 = fast_exp2(sc[n][3] - base1);
      s0 += e0 + e1, s1 += e2 + e3;
      pf[n * 2] = pack_bf16x2(e0, e1);
      pf[n * 2 + 1] = pack_bf16x2(e2, e3);
    }
    l0 = l0 * f0 + s0, l1 = l1 * f1 + s1;  // per lane; the four lanes of a row meet at the end
#pragma unroll
    for (int n = 0; n < D / 8; ++n) acc[n][0] *= f0, acc[n][1] *= f0, acc[n][2] *= f1, acc[n][3] *= f1;
#pragma unroll
    for (int n = 0; n < D / 16; ++n) {
      // transposed matrices: keys 0-7 / dims 0-7, keys 8-15 / dims 0-7, keys 0-7 / dims 8-15, keys 8-15 / dims 8-15
      const int key = (msel & 1) * 8 + mrow, ch = n * 2 + (msel >> 1);
      uint32_t b[4];
      ldsm4t(tv + key * (D * 2) + ((ch ^ (key & 7)) << 4), b);
      mma16816(acc[2 * n], pf, b[0], b[1]);
      mma16816(acc[2 * n + 1], pf, b[2], b[3]);
    }
    __syncwarp();  // the stage is refilled two iterations on
    cur = next(cur + 1);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
  l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 2);

  // The warps meet in shared memory (each in its own ring), then the CTAs of the cluster.
  float* part = reinterpret_cast<float*>(smem + warp * L::kWarpBytes);
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
    const int col = n * 8 + (lane & 3) * 2;
    *reinterpret_cast<float2*>(part + r0 * D + col) = make_float2(acc[n][0], acc[n][1]);
    *reinterpret_cast<float2*>(part + r1 * D + col) = make_float2(acc[n][2], acc[n][3]);
  }
  if ((lane & 3) == 0) {
    stats[(warp * kMaxRows + r0) * 2] = m0, stats[(warp * kMaxRows + r0) * 2 + 1] = l0;
    stats[(warp * kMaxRows + r1) * 2] = m1, stats[(warp * kMaxRows + r1) * 2 + 1] = l1;
  }
  __syncthreads();
  float* total = stats + kWarps * kMaxRows * 2;  // maximum and sum of the CTA
  for (int idx = threadIdx.x; idx < rows * D; idx += kWarps * 32) {
    const int r = idx / D, d = idx % D;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m = fmaxf(m, stats[(w * kMaxRows + r) * 2]);
    const float base = m == -INFINITY ? 0.f : m;
    float l = 0.f, x = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = fast_exp2(stats[(w * kMaxRows + r) * 2] - base);
      l += f * stats[(w * kMaxRows + r) * 2 + 1];
      x += f * reinterpret_cast<const float*>(smem + w * L::kWarpBytes)[r * D + d];
    }
    if (splits == 1) {
      p.o[((static_cast<long long>(bi) * p.s + r / group) * p.hq + hk * group + r % group) * D + d] = __float2bfloat16_rn(l > 0.f ? x / l : 0.f);
    } else {
      reinterpret_cast<float*>(smem)[r * D + d] = x;  // the slot of warp 0, read by this thread alone
      if (d == 0) total[r * 2] = m, total[r * 2 + 1] = l;
    }
  }
  if (splits == 1) return;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int idx = split * kWarps * 32 + threadIdx.x; idx < rows * D; idx += splits * kWarps * 32) {
    const int r = idx / D, d = idx % D;
    float m = -INFINITY;
    for (int x = 0; x < splits; ++x) m = fmaxf(m, cluster.map_shared_rank(total, x)[r * 2]);
    const float base = m == -INFINITY ? 0.f : m;
    float l = 0.f, o = 0.f;
    for (int x = 0; x < splits; ++x) {
      const float* t = cluster.map_shared_rank(total, x);
      const float f = fast_exp2(t[r * 2] - base);
      l += f * t[r * 2 + 1];
      o += f * cluster.map_shared_rank(reinterpret_cast<float*>(smem), x)[r * D + d];
    }
    p.o[((static_cast<long long>(bi) * p.s + r / group) * p.hq + hk * group + r % group) * D + d] = __float2bfloat16_rn(l > 0.f ? o / l : 0.f);
  }
  cluster.sync();  // no CTA leaves while another reads its shared memory
}

template <int D, bool APPEND>
static int launch(const Params& p, int b, cudaStream_t st) {
  const int blocks = (p.sk + kKeys - 1) / kKeys;
  int splits = 1;  // fill the SMs twice over as long as every CTA has a block of its own
  while (splits < kMaxSplit && static_cast<long long>(b) * p.hkv * splits < 2ll * sm_count() && blocks >= 2 * splits) splits *= 2;
  const int own = (blocks + splits - 1) / splits;
  const long long bit_bytes = static_cast<long long>(own) * (p.s + 1) * 8;
  if (bit_bytes > kMaxBitBytes) return kErrTooLarge;
  constexpr int fixed = Layout<D>::kRing + Layout<D>::kStats + (APPEND ? Layout<D>::kQueries : 0);
  const int smem = fixed + static_cast<int>(bit_bytes);
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(decode_kernel<D, APPEND>, cudaFuncAttributeMaxDynamicSharedMemorySize, fixed + kMaxBitBytes) != cudaSuccess) return kErrDriver;
    attr = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(splits, p.hkv, b);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = splits, at[0].val.clusterDim.y = 1, at[0].val.clusterDim.z = 1;
  cfg.attrs = at, cfg.numAttrs = 1;
  TTB_COUNT_LAUNCH(1);
  return cudaLaunchKernelEx(&cfg, decode_kernel<D, APPEND>, p) == cudaSuccess ? kOk : kErrDriver;
}

// First and last visible key of every mask row and whether all keys between them are visible; one warp per row, 16 bytes per lane and
// load.  One pass over the mask where the tensor operations that it replaces made nine.  Causal prefill of 2 x 8000 tokens over a cache of 8012 with
// this and the MASKED two-tile kernel: 16.0 -> 1.38 ms a layer (66 -> 760 TFLOP/s).
__global__ void __launch_bounds__(256)
mask_bounds_kernel(const uint8_t* __restrict__ mask, long long stride_b, long long stride_r, int b, int s, int sk, int* __restrict__ lo, int* __restrict__ hi,
                   uint8_t* __restrict__ solid) {
  const long long w = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= static_cast<long long>(b) * s) return;
  const uint8_t* row = mask + (w / s) * stride_b + (w % s) * stride_r;
  int first = sk, last = -1, count = 0;
  auto one = [&](int j) {
    if (row[j] != 0) first = min(first, j), last = max(last, j), ++count;
  };
  const int head = min(sk, static_cast<int>((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15));
  const int vecs = (sk - head) / 16;
  if (lane < head) one(lane);
  for (int x = lane; x < vecs; x += 32) {
    const uint4 u = *reinterpret_cast<const uint4*>(row + head + x * 16);
    const uint32_t part[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t z = __vcmpne4(part[i], 0u) & 0x01010101u;  // 1 in every nonzero byte
      if (z != 0) {
        const int at = head + x * 16 + i * 4;
        count += __popc(z);
        first = min(first, at + ((__ffs(z) - 1) >> 3));
        last = max(last, at + ((31 - __clz(z)) >> 3));
      }
    }
  }
  const int tail = head + vecs * 16 + lane;
  if (tail < sk) one(tail);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
    last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
    count += __shfl_xor_sync(0xffffffffu, count, o);
  }
  if (lane == 0) {
    lo[w] = first, hi[w] = last;
    solid[w] = count == 0 || count == last - first + 1;
  }
}

}  // namespace dec
}  // namespace ttb

// Attention of s queries with s * (hq / hkv) <= 16 over sk keys: q / o [b, s, hq, d], k / v [b, sk, hkv, d], d 64 or 128, all 16-byte aligned.
// mask (nullable): nonzero byte = visible, row (b, i) at mask + b * mask_b + i * mask_r; lo / hi (nullable) int32 [b, s] as in ttb_attn_fwd.
// A query without a visible key gives 0.
extern "C" int ttb_attn_decode(const void* q, const void* k, const void* v, void* o, const void* mask, long long mask_b, long long mask_r, const int* lo, const int* hi,
                               int b, int s, int sk, int hq, int hkv, int d, float scale, void* stream) {
  using namespace ttb;
  if ((d != 64 && d != 128) || b <= 0 || s <= 0 || sk <= 0 || hkv <= 0 || hq % hkv || s * (hq / hkv) > dec::kMaxRows || b > 65535 || hkv > 65535) return kErrBadShape;
  for (const void* t : {q, k, v, static_cast<const void*>(o)})
    if (reinterpret_cast<uintptr_t>(t) & 15) return kErrBadShape;
  dec::Params p{};
  p.q = static_cast<const __nv_bfloat16*>(q), p.k = static_cast<const __nv_bfloat16*>(k), p.v = static_cast<const __nv_bfloat16*>(v), p.o = static_cast<__nv_bfloat16*>(o);
  p.mask = static_cast<const uint8_t*>(mask), p.mask_b = mask_b, p.mask_r = mask_r, p.lo = lo, p.hi = hi;
  p.s = s, p.sk = sk, p.hq = hq, p.hkv = hkv, p.scale = scale;
  auto st = static_cast<cudaStream_t>(stream);
  return d == 128 ? dec::launch<128, false>(p, b, st) : dec::launch<64, false>(p, b, st);
}

// ttb_rope_append for one token per row followed by ttb_attn_decode on the caches, in one launch and with the same values: q, o [b, hq, d], k, v [b, hkv, d] before the rotation, caches [b, max_seq,
// hkv, d], rope [rope_len, d / 2, 2] fp32, pos int32 [b], slots[0] the slot of the new tokens; mask as above, max_seq bytes a row (mask_b 0: the same for all rows).
extern "C" int ttb_attn_decode_append(const void* q, const void* k, const void* v, void* o, void* k_cache, void* v_cache, const float* rope, const int* pos, const long long* slots, const void* mask,
                                      long long mask_b, int b, int max_seq, int hq, int hkv, int d, int interleaved, int rope_len, float scale, void* stream) {
  using namespace ttb;
  if ((d != 64 && d != 128) || b <= 0 || max_seq <= 0 || hkv <= 0 || hq % hkv || hq / hkv > dec::kMaxRows || b > 65535 || hkv > 65535 || rope_len <= 0) return kErrBadShape;
  for (const void* t : {q, k, v, static_cast<const void*>(o), static_cast<const void*>(k_cache), static_cast<const void*>(v_cache), static_cast<const void*>(rope)})
    if (reinterpret_cast<uintptr_t>(t) & 15) return kErrBadShape;
  dec::Params p{};
  p.q = static_cast<const __nv_bfloat16*>(q), p.k = static_cast<const __nv_bfloat16*>(k_cache), p.v = static_cast<const __nv_bfloat16*>(v_cache), p.o = static_cast<__nv_bfloat16*>(o);
  p.mask = static_cast<const uint8_t*>(mask), p.mask_b = mask_b;
  p.s = 1, p.sk = max_seq, p.hq = hq, p.hkv = hkv, p.scale = scale;
  p.k_new = static_cast<const __nv_bfloat16*>(k), p.v_new = static_cast<const __nv_bfloat16*>(v), p.rope = rope, p.pos = pos, p.slots = slots;
  p.rope_len = rope_len, p.interleaved = interleaved;
  auto st = static_cast<cudaStream_t>(stream);
  return d == 128 ? dec::launch<128, true>(p, b, st) : dec::launch<64, true>(p, b, st);
}

// lo / hi int32 [b, s]: first / last nonzero byte of every mask row (sk / -1 for rows without one); solid uint8 [b, s]: 1 if all bytes between are nonzero.
extern "C" int ttb_mask_bounds(const void* mask, long long stride_b, long long stride_r, int b, int s, int sk, int* lo, int* hi, void* solid, void* stream) {
  using namespace ttb;
  if (b <= 0 || s <= 0 || sk <= 0) return kErrBadShape;
  const long long warps = static_cast<long long>(b) * s;
  TTB_COUNT_LAUNCH(1);
  dec::mask_bounds_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(mask), stride_b, stride_r, b, s, sk, lo, hi, static_cast<uint8_t*>(solid));
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}
