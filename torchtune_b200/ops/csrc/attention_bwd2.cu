// Attention backward, second form: transposed score tiles, two query stages, probabilities kept in tensor memory, dQ drained by warps of its own.
//
// One CTA owns 128 keys of one key head and walks the query blocks of the head's group that see them.  Per block: Sᵀ = K·Qᵀ and dPᵀ = V·dOᵀ with keys
// as rows, P = exp2(S·c − lse), dS = P·(dP − delta)·scale, then dV += Pᵀ·dO, dK += dSᵀ·Q and a partial dQ = dS·K that is added to an fp32 buffer.
// With keys as rows Pᵀ is the A operand of its product just as the softmax warps write it over their own part of the scores in tensor memory, and dSᵀ
// serves both of its products from one copy in shared memory.  That leaves room for a second stage of Q and for staging dQ (224 KB with K, V, dO and dS), where the
// first form (attention.cu) keeps P and dS, one stage of Q and dO, and runs loads, products, exponentials and dQ one after the other.
//
// Tensor memory: S (P over it), dP (the partial dQ over it), dV, dK.  The MMA warp issues, for block i: dV(i) when P(i) is there, S(i + 1) at once behind
// it (in issue order, so it may overwrite P(i)), dK(i) and dQ(i) when dS(i) is there, and dP(i + 1) when dQ(i) has been read.  Exponentials of block i + 1 thus run
// under dK(i), dQ(i) and dP(i + 1), and dO(i + 1), whose place is free once dV(i) is done, arrives under them as well.  dQ leaves as TMA reductions of 32 x 32 tiles: whole
// 128-byte lines to the L2, where 16-byte atomics of a row per lane had made four requests of each.
// Warps 4-11: softmax, two warps per 32 keys, 64 queries each; warps 12-15: dQ; 0 TMA, 1 MMA, 2 tensor memory, 3 lse and delta.
//
// Whole backward pass with delta and the conversion of dQ, first form -> here: 1 x 16384 causal, head dim 128 9822 -> 5514 us (997 TFLOP/s), head dim 64 6917 -> 4324 us;
// 4 x 2048 of 128 937 -> 588 us, in documents of 512 394 -> 296 us.  With dQ added by 16-byte atomics instead of TMA reductions the first took 13 300 us.  What bounds it:
// at head dim 128 the chain dS -> dQ -> dP -> dS beside 2560 cycles of products per block, at head dim 64 the exponentials.
//
// Structured masks as in attention.cu (bounds lo / hi per query); soft-capped scores and boolean masks stay on the first form.  Every wait is bounded.
#include <type_traits>

#include "common/attn_math.cuh"
#include "common/ptx.cuh"
#include "common/tmap.h"

namespace ttb {
namespace fb2 {

using namespace attn;
static constexpr int kThreads = 512;
static constexpr int kMaxSmem = 232448;

struct Params {
  int s, sk, hq, hkv;
  float scale;
  int causal;        // hi[q] = q when no `hi` array is given (requires sk == s)
  const int* lo;     // [b, s] or nullptr
  const int* hi;     // [b, s] or nullptr
  int monotone;      // lo and hi do not decrease along the sequence
  const float* lse;    // [b, hq, s], log2 domain
  const float* delta;  // [b, hq, s]
  __nv_bfloat16* dk;   // [b, sk, hkv, D]
  __nv_bfloat16* dv;
  int* err;
};

template <int D>
struct Layout {
  static constexpr int kTile = kBlk * D * 2;
  static constexpr int kDs = 5 * kTile;                 // after K, V, Q[2], dO
  static constexpr int kOut = kDs + 2 * kPanelBytes;    // dQ: two 32 x 32 fp32 tiles per warp
  static constexpr int kStats = kOut + 4 * 2 * 4096;    // [stage][-lse, delta][128]
  static constexpr int kBars = kStats + 2 * 2 * kBlk * 4;
  static constexpr int kTotal = kBars + 256;
  static constexpr int kDynamic = kTotal + 1024 < kMaxSmem ? kTotal + 1024 : kMaxSmem;
};

__device__ __forceinline__ uint32_t swizzled(int row, int col) {  // byte offset of (row, col) in 128-row panels of 64 columns
  return (col >> 6) * kPanelBytes + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4);
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
attn_bwd2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                 const __grid_constant__ CUtensorMap tmdQ, Params p) {
  using L = Layout<D>;
  constexpr int kPanels = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (smem + L::kTotal > smem_raw + L::kDynamic) {  // head dim 128 leaves 768 bytes to align with; the dynamic part starts at a multiple of 1024 as it is
    if (threadIdx.x == 0) atomicExch(p.err, 310);
    return;
  }
  uint8_t* sK = smem;
  uint8_t* sV = smem + L::kTile;
  uint8_t* sQ = smem + 2 * L::kTile;   // two stages
  uint8_t* sdO = smem + 4 * L::kTile;
  uint8_t* sdS = smem + L::kDs;        // [128 keys, 128 queries] bf16
  float* stats = reinterpret_cast<float*>(smem + L::kStats);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;      // [2]
  uint64_t* q_empty = bars + 3;     // [2]
  uint64_t* stat_full = bars + 5;   // [2]
  uint64_t* stat_empty = bars + 7;  // [2]
  uint64_t* s_full = bars + 9;
  uint64_t* p_ready = bars + 10;
  uint64_t* dp_full = bars + 11;
  uint64_t* ds_ready = bars + 12;
  uint64_t* dq_full = bars + 13;
  uint64_t* dq_free = bars + 14;
  uint64_t* do_full = bars + 15;
  uint64_t* do_empty = bars + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hk = blockIdx.y, bi = blockIdx.z;
  const int group = p.hq / p.hkv;
  const int kv0 = blockIdx.x * kBlk;
  const int row_base = bi * p.s, krow_base = bi * p.sk;
  const int nq_blocks = (p.s + kBlk - 1) / kBlk;
  int qb_begin = (p.hi == nullptr && p.causal) ? static_cast<int>(blockIdx.x) : 0;
  int qb_end = nq_blocks;
  if (p.monotone) {
    if (p.hi != nullptr)
      while (qb_begin < nq_blocks && p.hi[row_base + min((qb_begin + 1) * kBlk, p.s) - 1] < kv0) ++qb_begin;
    if (p.lo != nullptr)
      for (int qb = qb_begin; qb < nq_blocks; ++qb)
        if (p.lo[row_base + qb * kBlk] > kv0 + kBlk - 1) {
          qb_end = qb;
          break;
        }
  }
  const int per_head = max(qb_end - qb_begin, 0);
  const int n = per_head * group;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&stat_full[i], 1);
      mbar_init(&stat_empty[i], 8);
    }
    mbar_init(s_full, 1);
    mbar_init(p_ready, 8);
    mbar_init(dp_full, 1);
    mbar_init(ds_ready, 8);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, 4);
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 384;

  // the lanes of a warp agree, so that a wait that gives up leaves none of them behind in a warp-wide instruction
  auto wait = [](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0; };
  auto stopped = [&] { return __any_sync(0xffffffffu, *abort_flag != 0) != 0; };
  if (warp < 4) {
    if (warp == 0) {
      // -------------------------------------------------------------- TMA producer
      if (n > 0 && lane == 0) {
        mbar_arrive_expect_tx(kv_full, 2 * L::kTile);
        for (int j = 0; j < kPanels; ++j) {
          tma_load_2d(sK + j * kPanelBytes, &tmK, kv_full, hk * D + j * 64, krow_base + kv0);
          tma_load_2d(sV + j * kPanelBytes, &tmV, kv_full, hk * D + j * 64, krow_base + kv0);
        }
      }
      for (int i = 0; i < n && !stopped(); ++i) {
        const int st = i & 1;
        const int h = hk * group + i / per_head, q0 = (qb_begin + i % per_head) * kBlk;
        if (!wait(&q_empty[st], ((i >> 1) & 1) ^ 1)) {
          fail(abort_flag, p.err, 311);
          break;
        }
        if (lane == 0) {
          mbar_arrive_expect_tx(&q_full[st], L::kTile);
          for (int j = 0; j < kPanels; ++j) tma_load_2d(sQ + st * L::kTile + j * kPanelBytes, &tmQ, &q_full[st], h * D + j * 64, row_base + q0);
        }
        if (!wait(do_empty, (i & 1) ^ 1)) {
          fail(abort_flag, p.err, 316);
          break;
        }
        if (lane == 0) {
          mbar_arrive_expect_tx(do_full, L::kTile);
          for (int j = 0; j < kPanels; ++j) tma_load_2d(sdO + j * kPanelBytes, &tmdO, do_full, h * D + j * 64, row_base + q0);
        }
        __syncwarp();
      }
    } else if (warp == 1) {
      // -------------------------------------------------------------- MMA issuer
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);  // K·Qᵀ, V·dOᵀ
      constexpr uint32_t idesc_t = make_idesc_bf16(128, D, false, true);     // Pᵀ·dO (A from tensor memory), dSᵀ·Q
      constexpr uint32_t idesc_q = make_idesc_bf16(128, D, true, true);      // dS·K: dSᵀ read with keys as the contraction
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), adO = smem_u32(sdO), adS = smem_u32(sdS);
      auto scores = [&](int i) {
        const uint32_t aQ = smem_u32(sQ + (i & 1) * L::kTile);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_f16(tS, desc_kmajor(aK, k), desc_kmajor(aQ, k), idesc_s, k != 0);
        umma_commit(s_full);
      };
      auto dprobs = [&] {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_f16(tdP, desc_kmajor(aV, k), desc_kmajor(adO, k), idesc_s, k != 0);
        umma_commit(dp_full);
      };
      bool ok = n == 0 || (wait(kv_full, 0) && wait(&q_full[0], 0) && wait(do_full, 0));
      tc_fence_after();
      if (ok && n > 0 && lane == 0) {
        scores(0);
        dprobs();
      }
      __syncwarp();
      for (int i = 0; i < n && ok && !stopped(); ++i) {
        const int st = i & 1;
        const uint32_t aQ = smem_u32(sQ + st * L::kTile);
        const bool more = i + 1 < n;
        if (!wait(p_ready, i & 1) || (more && !wait(&q_full[st ^ 1], ((i + 1) >> 1) & 1))) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (lane == 0) {
          // queries 64 x ... of P are 32 columns of the softmax warps' own score columns
#pragma unroll
          for (int k = 0; k < kBlk / 16; ++k) umma_f16_ts(tdV, tS + (k >> 2) * 64 + (k & 3) * 8, desc_mnmajor(adO, k), idesc_t, (i | k) != 0);
          umma_commit(do_empty);
          if (more) scores(i + 1);
        }
        __syncwarp();
        if (!wait(ds_ready, i & 1)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (lane == 0) {
#pragma unroll
          for (int k = 0; k < kBlk / 16; ++k) umma_f16(tdP, desc_mnmajor(adS, k), desc_mnmajor(aK, k), idesc_q, k != 0);
          umma_commit(dq_full);
#pragma unroll
          for (int k = 0; k < kBlk / 16; ++k) umma_f16(tdK, desc_kmajor(adS, k), desc_mnmajor(aQ, k), idesc_t, (i | k) != 0);
          umma_commit(&q_empty[st]);
        }
        __syncwarp();
        if (more) {
          if (!wait(dq_free, i & 1) || !wait(do_full, (i + 1) & 1)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (lane == 0) dprobs();
          __syncwarp();
        }
      }
      if (!ok) fail(abort_flag, p.err, 312);
    } else if (warp == 3) {
      // -------------------------------------------------------------- lse and delta of the query blocks
      for (int i = 0; i < n && !stopped(); ++i) {
        const int st = i & 1;
        const int h = hk * group + i / per_head, q0 = (qb_begin + i % per_head) * kBlk;
        const long long at = (static_cast<long long>(bi) * p.hq + h) * p.s;
        float nl[4], de[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int q = q0 + x * 32 + lane;
          const float l = q < p.s ? p.lse[at + q] : -INFINITY;
          nl[x] = l == -INFINITY ? -INFINITY : -l;  // exp2 gives 0 for queries past the end and for those that see nothing
          de[x] = q < p.s ? p.delta[at + q] : 0.f;
        }
        if (!wait(&stat_empty[st], ((i >> 1) & 1) ^ 1)) {
          fail(abort_flag, p.err, 313);
          break;
        }
        float* to = stats + st * 2 * kBlk;
#pragma unroll
        for (int x = 0; x < 4; ++x) to[x * 32 + lane] = nl[x], to[kBlk + x * 32 + lane] = de[x];
        __threadfence_block();
        __syncwarp();
        if (lane == 0) mbar_arrive(&stat_full[st]);
      }
    }
  } else if (warp < 12) {
    // ---------------------------------------------------------------- softmax backward, then dK and dV
    const int quarter = warp & 3, half = (warp - 4) >> 2;
    const int r = quarter * 32 + lane;  // key row
    const int key = kv0 + r;
    const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
    const float c = p.scale * kLog2e;
    const uint64_t c2 = pack_f32x2(c, c), sc2 = pack_f32x2(p.scale, p.scale);
    bool ok = true;
    for (int i = 0; i < n && !stopped(); ++i) {
      const int st = i & 1;
      const int q0 = (qb_begin + i % per_head) * kBlk;
      bool interior = (p.monotone || (p.lo == nullptr && p.hi == nullptr)) && q0 + kBlk <= p.s && kv0 + kBlk <= p.sk;
      if (interior) {
        const int lo_max = p.lo != nullptr ? p.lo[row_base + q0 + kBlk - 1] : 0;
        const int hi_min = p.hi != nullptr ? p.hi[row_base + q0] : (p.causal ? q0 : p.sk - 1);
        interior = lo_max <= kv0 && hi_min >= kv0 + kBlk - 1;
      }
      if (!wait(&stat_full[st], (i >> 1) & 1) || !wait(s_full, i & 1)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const float* nlse = stats + st * 2 * kBlk + half * 64;
      const float* delta = nlse + kBlk;
      uint64_t pr[2][16];  // this thread's probabilities, two queries each
      auto probabilities = [&](auto masked) {
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          uint32_t seen = 0xffffffffu;  // queries of the chunk that see this thread's key
          if constexpr (masked.value) {
            const int first = q0 + half * 64 + ch * 32, q = min(first + lane, p.s - 1);
            const int lo = p.lo != nullptr ? __ldg(p.lo + row_base + q) : 0;
            const int hi = p.hi != nullptr ? __ldg(p.hi + row_base + q) : (p.causal ? q : p.sk - 1);
            seen = 0;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int lo_j = __shfl_sync(0xffffffffu, lo, j), hi_j = __shfl_sync(0xffffffffu, hi, j);  // by all lanes, whatever the first comparison says
              seen |= (key >= lo_j && key <= hi_j ? 1u : 0u) << j;
            }
            const int left = p.s - first;  // queries of this batch row; behind them lie the next row's, whose scores may be infinite
            if (left < 32) seen = left > 0 ? seen & ((1u << left) - 1) : 0;
            if (key >= p.sk) seen = 0;
          }
          uint32_t sv[32], pk[16];
          tmem_ld_32x32(tS + lane_sel + half * 64 + ch * 32, sv);
          tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const float4 nl = *reinterpret_cast<const float4*>(nlse + ch * 32 + g * 4);
            const float f[4] = {nl.x, nl.y, nl.z, nl.w};
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int e = g * 4 + x * 2;
              float t0, t1;
              unpack_f32x2(fma_f32x2(pack_u32x2(sv[e], sv[e + 1]), c2, pack_f32x2(f[x * 2], f[x * 2 + 1])), t0, t1);
              t0 = fast_exp2(t0), t1 = fast_exp2(t1);
              if constexpr (masked.value) {
                t0 = (seen >> e) & 1u ? t0 : 0.f;
                t1 = (seen >> (e + 1)) & 1u ? t1 : 0.f;
              }
              pr[ch][e / 2] = pack_f32x2(t0, t1);
              pk[e / 2] = pack_bf16x2(t0, t1);
            }
          }
          tmem_st_32x16(tS + lane_sel + half * 64 + ch * 16, pk);  // over scores this warp has read
        }
      };
      if (interior)
        probabilities(std::false_type{});
      else
        probabilities(std::true_type{});
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      if (!wait(dp_full, i & 1)) {
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        uint32_t dv[32];
        tmem_ld_32x32(tdP + lane_sel + half * 64 + ch * 32, dv);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float4 d0 = *reinterpret_cast<const float4*>(delta + ch * 32 + g * 8), d1 = *reinterpret_cast<const float4*>(delta + ch * 32 + g * 8 + 4);
          const float f[8] = {-d0.x, -d0.y, -d0.z, -d0.w, -d1.x, -d1.y, -d1.z, -d1.w};
          uint32_t du[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int e = g * 8 + x * 2;
            float t0, t1;
            unpack_f32x2(mul_f32x2(mul_f32x2(pr[ch][e / 2], sc2), add_f32x2(pack_u32x2(dv[e], dv[e + 1]), pack_f32x2(f[x * 2], f[x * 2 + 1]))), t0, t1);
            du[x] = pack_bf16x2(t0, t1);
          }
          *reinterpret_cast<uint4*>(sdS + swizzled(r, half * 64 + ch * 32 + g * 8)) = make_uint4(du[0], du[1], du[2], du[3]);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&stat_empty[st]);
        mbar_arrive(ds_ready);
      }
    }
    // the last block's dK is behind the commit that gives its stage back
    if (ok && n > 0 && !stopped()) ok = wait(&q_empty[(n - 1) & 1], ((n - 1) >> 1) & 1);
    if (!ok) {
      fail(abort_flag, p.err, 314);
    } else if (!stopped()) {
      tc_fence_after();
      // the first half's warps write dK, the second half's dV
      const uint32_t from = half == 0 ? tdK : tdV;
      __nv_bfloat16* to = (half == 0 ? p.dk : p.dv) + (static_cast<long long>(krow_base + key) * p.hkv + hk) * D;
#pragma unroll 1
      for (int ch = 0; ch < D / 32; ++ch) {
        uint32_t a[32];
        if (n > 0) {
          tmem_ld_32x32(from + lane_sel + ch * 32, a);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) a[j] = 0;
        }
        if (key < p.sk) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 u;
            u.x = pack_bf16x2(__uint_as_float(a[g * 8 + 0]), __uint_as_float(a[g * 8 + 1]));
            u.y = pack_bf16x2(__uint_as_float(a[g * 8 + 2]), __uint_as_float(a[g * 8 + 3]));
            u.z = pack_bf16x2(__uint_as_float(a[g * 8 + 4]), __uint_as_float(a[g * 8 + 5]));
            u.w = pack_bf16x2(__uint_as_float(a[g * 8 + 6]), __uint_as_float(a[g * 8 + 7]));
            *reinterpret_cast<uint4*>(to + ch * 32 + g * 8) = u;
          }
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- dQ: partial tiles into the fp32 buffer
    const int quarter = warp & 3;
    const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
    uint8_t* out = smem + L::kOut + quarter * 8192;
    auto put = [&](const uint32_t (&v)[32], int ch, int h, int row0) {
      uint8_t* tile = out + (ch & 1) * 4096;
      if (lane == 0) tma_store_wait_read<1>();  // the reduction that used this tile two chunks ago has read it
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4*>(tile + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(v[j * 4], v[j * 4 + 1], v[j * 4 + 2], v[j * 4 + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (row0 < p.s) tma_add_3d(&tmdQ, tile, h * D + ch * 32, row0, bi);  // rows past the end of the batch row are cut off by the map
        tma_store_commit();
      }
    };
    for (int i = 0; i < n && !stopped(); ++i) {
      const int h = hk * group + i / per_head, row0 = (qb_begin + i % per_head) * kBlk + quarter * 32;
      if (!wait(dq_full, i & 1)) {
        fail(abort_flag, p.err, 315);
        break;
      }
      tc_fence_after();
      uint32_t v[2][32];
#pragma unroll
      for (int c0 = 0; c0 < D / 32; c0 += 2) {
        tmem_ld_32x32(tdP + lane_sel + c0 * 32, v[0]);
        tmem_ld_32x32(tdP + lane_sel + (c0 + 1) * 32, v[1]);
        tmem_ld_wait();
        if (c0 + 2 == D / 32) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_free);
        }
        put(v[0], c0, h, row0);
        put(v[1], c0 + 1, h, row0);
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 2) tmem_dealloc(tmem_base, 512);
}

template <int D>
static int launch(const void* q, const void* k, const void* v, const void* d_o, float* dq, int b, const Params& p, cudaStream_t st) {
  CUtensorMap tq, tk, tv, tdo, tdq;
  auto map = [&](CUtensorMap* m, const void* base, int s, int heads) {
    return make_tmap_2d(m, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, static_cast<uint64_t>(b) * s, static_cast<uint64_t>(heads) * D, static_cast<uint64_t>(heads) * D, kBlk, 64,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  };
  int rc;
  if ((rc = map(&tq, q, p.s, p.hq)) != kOk || (rc = map(&tk, k, p.sk, p.hkv)) != kOk || (rc = map(&tv, v, p.sk, p.hkv)) != kOk || (rc = map(&tdo, d_o, p.s, p.hq)) != kOk) return rc;
  const uint64_t width = static_cast<uint64_t>(p.hq) * D;
  if ((rc = make_tmap_3d(&tdq, dq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, width, p.s, b, width * 4, width * 4 * p.s, 32, 32, 1, CU_TENSOR_MAP_SWIZZLE_128B)) != kOk) return rc;
  auto kern = attn_bwd2_kernel<D>;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<D>::kDynamic) != cudaSuccess) return kErrDriver;
    attr = true;
  }
  TTB_COUNT_LAUNCH(1);
  kern<<<dim3((p.sk + kBlk - 1) / kBlk, p.hkv, b), kThreads, Layout<D>::kDynamic, st>>>(tq, tk, tv, tdo, tdq, p);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}

}  // namespace fb2
}  // namespace ttb

// The backward of attn_fwd / attn_fwd2 without soft cap and boolean mask; delta as attn_delta_kernel leaves it.  Called by ttb_attn_bwd.
int ttb_attn_bwd2(const void* q, const void* k, const void* v, const void* d_o, const float* lse, const float* delta, float* dq, void* dk, void* dv, const int* lo, const int* hi,
                  int monotone, int b, int s, int sk, int hq, int hkv, int d, float scale, int causal, int* err, cudaStream_t stream) {
  using namespace ttb;
  fb2::Params p{};
  p.s = s, p.sk = sk, p.hq = hq, p.hkv = hkv, p.scale = scale, p.causal = causal, p.lo = lo, p.hi = hi, p.monotone = monotone;
  p.lse = lse, p.delta = delta, p.dk = static_cast<__nv_bfloat16*>(dk), p.dv = static_cast<__nv_bfloat16*>(dv), p.err = err;
  return d == 128 ? fb2::launch<128>(q, k, v, d_o, dq, b, p, stream) : fb2::launch<64>(q, k, v, d_o, dq, b, p, stream);
}
