// Grouped products (mixture of experts) on pairs of SMs: C[rows of e, N] = X[rows of e, K] · op(W[e]) for every expert e.
//
// An expert has a few hundred rows, seldom a multiple of anything.  With the rows on the 128 rows of an MMA tile a fifth of the products were padding, and one CTA per tile reads
// both operands at the rate that bounds the single-CTA kernel.  Here the weights take the 256 rows of a CTA pair's tile and the tokens its columns, of which there may be any
// multiple of 32 up to 256: an expert's rows are cut into equal pieces, so at most 31 of a piece are padding, and every weight is loaded for up to 256 tokens.
// The accumulator comes out with weight rows as lanes: a warp's 32 x 32 values are turned in shared memory (2-byte stores, 64 bytes per token) and leave as 16-byte stores,
// which also leave out the rows of the next expert that a last piece has computed.
// Pipeline, barriers and failure handling are those of gemm2sm.cu; the piece's size travels with the tile through the table that a small kernel builds from the row counts on the
// device, so no host read is needed.
// 16 experts of 5120 x 8192, us forward / input gradient with one CTA per 128 x 256 tile -> here, out of a graph over more weights than the L2 holds: 300 rows 217 / 245 -> 207 / 230 (6.5 TB/s of
// weights), 4096 rows 372 / 404 -> 338 / 360, 12000 rows 846 / 894 -> 751 / 808 (1340 TFLOP/s).  Where products of this kernel are slower, see ops._cuda._groups_on_pairs.  At 4096 rows the pieces of
// few tokens wait for weights and those of many for products; mixing them (all experts at a block of weight rows) read the tokens again for each block and took 14 % longer.
#include <cstring>

#include "common/pair.cuh"
#include "common/tmap.h"

namespace ttb {
namespace gg {

using namespace g2;

static constexpr int BM = 128;  // weight rows per CTA
static constexpr int PM = 256;  // and per pair
static constexpr int kMaxTokens = 256;
static constexpr int kStep = 32;  // tokens come in multiples of this, half of them for each CTA: boxes of 64, 32 and 16
static constexpr int BK = 64;
static constexpr int kThreads = 256;
static constexpr int kABytes = BM * BK * 2;
static constexpr int kBBytes = kMaxTokens / 2 * BK * 2;
static constexpr int kStageBytes = kABytes + kBBytes;
static constexpr int kStages = 6;
static constexpr int kTurnBytes = 2 * 32 * 64;  // two 32 x 32 sub-tiles of a warp
static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 4 * kTurnBytes + 1024;
static_assert(kSmemBytes <= 232448, "shared memory budget of one CTA");

struct Params {
  int N, K;  // weight rows (columns of C), contraction
  __nv_bfloat16* C;
  long long ldc;
  // per piece: expert, first piece of the expert and their number, first row and rows of the expert; then the number of pieces
  const int *expert, *first, *pieces, *row0, *rows, *total;
  int* err;
};

struct Tile {
  int expert, block, row, rows, n;  // rows of the piece, and the columns it takes
};
__device__ __forceinline__ int piece_size(int rows, int pieces) { return (rows + pieces * kStep - 1) / (pieces * kStep) * kStep; }
// Expert by expert, and for each block of weight rows all pieces of the expert: the weights are read from HBM once, and the expert's tokens stay in the L2.
__device__ __forceinline__ Tile tile_of(const Params& p, int t, int blocks) {
  const int any = t / blocks, first = p.first[any], pieces = p.pieces[any], rows = p.rows[any];  // any piece of the expert
  const int local = t - first * blocks, size = piece_size(rows, pieces), from = local % pieces * size;
  const int mine = max(min(size, rows - from), 0);
  return {p.expert[any], local / pieces, p.row0[any] + from, mine, (mine + kStep - 1) / kStep * kStep};
}

// W_MN: W[e] is [K, N] row-major (forward of experts stored contraction first), else [N, K].
template <bool W_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
grouped_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX64, const __grid_constant__ CUtensorMap tmX32, const __grid_constant__ CUtensorMap tmX16,
               const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);  // used in the even CTA
  uint64_t* empty = full + kStages;                                            // both CTAs
  uint64_t* tfull = empty + kStages;                                           // [2] both CTAs
  uint64_t* tempty = tfull + 2;                                                // [2] used in the even CTA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* turn = smem + kStages * kStageBytes + 1024;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int blocks = (p.N + PM - 1) / PM, num_tiles = *p.total * blocks;
  const int num_kb = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 8);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX64);
    prefetch_tmap(&tmX32);
    prefetch_tmap(&tmX16);
  }
  __syncthreads();
  if (warp == 2) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync();  // both CTAs' barriers are initialised and both hold their tensor memory before anything crosses over
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      const uint32_t full0 = map_to_cta(&full[0], 0);
      int stage = 0;
      uint32_t phase = 1;
      for (int t = pair; t < num_tiles && !*abort_flag; t += num_pairs) {
        const Tile tile = tile_of(p, t, blocks);
        if (tile.n == 0) continue;  // an expert without rows, or a piece that rounding left empty
        const int w_row = tile.block * PM + static_cast<int>(cta) * BM;
        const int mine = tile.n / 2, x_row = tile.row + static_cast<int>(cta) * mine;
        const uint32_t bytes = 2 * (kABytes + mine * BK * 2);  // of both CTAs' loads
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_idle(&empty[stage], phase, 64)) {
            *abort_flag = 1;
            atomicExch(p.err, 121);
            break;
          }
          uint8_t* sw = smem + stage * kStageBytes;
          uint8_t* sx = sw + kABytes;
          if (cta == 0) mbar_arrive_expect_tx(&full[stage], bytes);
          const uint32_t bar = full0 + stage * 8;
          if (W_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_3d_pair(sw + j * 8192, &tmW, bar, w_row + j * 64, kb * BK, tile.expert);
          } else {
            tma_load_3d_pair(sw, &tmW, bar, kb * BK, w_row, tile.expert);
          }
          int j = 0;
          for (; j + 64 <= mine; j += 64) tma_load_2d_pair(sx + j * 128, &tmX64, bar, kb * BK, x_row + j);
          if (mine & 32) tma_load_2d_pair(sx + j * 128, &tmX32, bar, kb * BK, x_row + j), j += 32;
          if (mine & 16) tma_load_2d_pair(sx + j * 128, &tmX16, bar, kb * BK, x_row + j);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1 && cta == 0) {
    // ------------------------------------------------------------------ MMA issuer (one thread of the even CTA)
    if (elect_one()) {
      const uint64_t desc_w = W_MN ? make_smem_desc_sw128(smem_u32(smem), 8192, 1024) : make_smem_desc_sw128(smem_u32(smem), 16, 1024);
      const uint64_t desc_x = make_smem_desc_sw128(smem_u32(smem) + kABytes, 16, 1024);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 1;
      for (int t = pair; t < num_tiles && !*abort_flag; t += num_pairs) {
        const Tile tile = tile_of(p, t, blocks);
        if (tile.n == 0) continue;
        const uint32_t idesc = make_idesc_bf16(PM, tile.n, W_MN, false);
        if (!mbar_wait(&tempty[acc], acc_phase)) {
          *abort_flag = 1;
          atomicExch(p.err, 122);
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * kMaxTokens;
        bool ok = true;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&full[stage], phase)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t at = static_cast<uint64_t>(stage * (kStageBytes >> 4));
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) umma_f16_pair(d_tmem, desc_w + at + k * ((W_MN ? 2048 : 32) >> 4), desc_x + at + k * (32 >> 4), idesc, (kb | k) != 0);
          umma_commit_pair(&empty[stage]);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) {
          *abort_flag = 1;
          atomicExch(p.err, 123);
          break;
        }
        umma_commit_pair(&tfull[acc]);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ epilogue (both CTAs, own 128 weight rows)
    const int quarter = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    int toggle = 0;
    for (int t = pair; t < num_tiles && !*abort_flag; t += num_pairs) {
      const Tile tile = tile_of(p, t, blocks);
      if (tile.n == 0) continue;
      if (!mbar_wait_idle(&tfull[acc], acc_phase, 128)) {
        *abort_flag = 1;
        if (lane == 0) atomicExch(p.err, 124);
        break;
      }
      tc_fence_after();
      const int col = tile.block * PM + static_cast<int>(cta) * BM + quarter * 32;  // of C: this warp's 32 weight rows
      const uint32_t taddr = tmem_base + acc * kMaxTokens + (static_cast<uint32_t>(quarter * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < tile.n; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + c, r);
        tmem_ld_wait();
        uint8_t* buf = turn + quarter * kTurnBytes + (toggle & 1) * (kTurnBytes / 2);
        ++toggle;
#pragma unroll
        for (int i = 0; i < 32; ++i) *reinterpret_cast<__nv_bfloat16*>(buf + i * 64 + lane * 2) = __float2bfloat16_rn(__uint_as_float(r[i]));
        __syncwarp();
        const int at = lane >> 2, piece = lane & 3;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int token = c + i * 8 + at;
          if (token < tile.rows && col + piece * 8 + 8 <= p.N)
            *reinterpret_cast<uint4*>(p.C + (tile.row + token) * p.ldc + col + piece * 8) = *reinterpret_cast<const uint4*>(buf + (i * 8 + at) * 64 + piece * 16);
        }
        // the other buffer is next; the one after it is written only once the whole warp has passed the barrier above again
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(&tempty[acc], 0));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }

  // Neither CTA may leave (or give its tensor memory back) while the other one's MMAs, commits or loads can still touch it.
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  if (warp == 2) tmem_dealloc_pair(tmem_base, 512);
}

// Sum of the values of all threads with a lower index in a block of 1024; `total` that of all.
__device__ __forceinline__ long long sum_before(long long v, long long* warp_sums, long long& total) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  long long sum = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long other = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += other;
  }
  __syncthreads();  // warp_sums of an earlier call are read
  if (lane == 31) warp_sums[warp] = sum;
  __syncthreads();
  long long ahead = 0;
  total = 0;
#pragma unroll 8
  for (int w = 0; w < 32; ++w) {
    if (w == warp) ahead = total;
    total += warp_sums[w];
  }
  return ahead + sum - v;
}

// One block, a thread per expert: first row and pieces of every expert; `table` is Params' five arrays of max_pieces entries each and the total.  Few experts are listed by the size of
// their pieces, so that the tiles that the pairs take in turn are of one size and all pairs get the same work; with many it averages out.  No row lies outside the result, whatever
// the counts say.  One thread that goes through the experts, size by size, took 4 us of 8 experts, 12 of 16 and 50 of 64 (64 products of 2048 x 768: 118 us with it, 66 here).
__global__ void __launch_bounds__(1024) piece_table_kernel(const long long* __restrict__ counts, int num_experts, int max_pieces, long long rows, int* __restrict__ table) {
  __shared__ long long warp_sums[32];
  __shared__ int row0[1024], count[1024], piece0[1024];
  const int e = threadIdx.x;
  long long total;
  const long long c = e < num_experts ? min(max(counts[e], 0ll), rows) : 0;
  const long long first_row = sum_before(c, warp_sums, total), end_row = min(first_row + c, rows);
  const int mine = end_row > first_row ? static_cast<int>(end_row - first_row) : 0, pieces = (mine + kMaxTokens - 1) / kMaxTokens;
  row0[e] = static_cast<int>(min(first_row, rows)), count[e] = mine;
  int at = static_cast<int>(sum_before(pieces, warp_sums, total));  // its barriers also publish the counts
  if (num_experts <= 64 && mine > 0) {
    const int size = piece_size(mine, pieces);
    at = 0;
    for (int o = 0; o < num_experts; ++o) {
      const int n = count[o], of = (n + kMaxTokens - 1) / kMaxTokens;
      if (n == 0 || o == e) continue;
      const int theirs = piece_size(n, of);
      if (theirs > size || (theirs == size && o < e)) at += of;
    }
  }
  piece0[e] = at;
  if (e == 0) table[5 * max_pieces] = total < max_pieces ? static_cast<int>(total) : max_pieces;
  __syncthreads();
  for (int o = threadIdx.x >> 5; o < num_experts; o += 32) {
    const int n = count[o], of = (n + kMaxTokens - 1) / kMaxTokens;
    for (int i = threadIdx.x & 31; i < of && piece0[o] + i < max_pieces; i += 32) {
      int* to = table + piece0[o] + i;
      to[0] = o;
      to[max_pieces] = piece0[o];
      to[2 * max_pieces] = of;
      to[3 * max_pieces] = row0[o];
      to[4 * max_pieces] = n;
    }
  }
}

template <bool W_MN>
static int launch(const void* X, const void* W, const Params& p, long long rows, int num_experts, int max_pieces, long long ldx, long long ldw, long long expert_stride, cudaStream_t st) {
  CUtensorMap tmW, tmX[3];
  int rc = kOk;
  for (int i = 0; i < 3 && rc == kOk; ++i) rc = make_tmap_2d(&tmX[i], X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows, p.K, ldx, 64 >> i, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != kOk) return rc;
  rc = W_MN ? make_tmap_3d(&tmW, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, p.N, p.K, num_experts, ldw * 2, expert_stride * 2, 64, BK, 1, CU_TENSOR_MAP_SWIZZLE_128B)
            : make_tmap_3d(&tmW, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, p.K, p.N, num_experts, ldw * 2, expert_stride * 2, BK, BM, 1, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != kOk) return rc;
  auto kernel = grouped_kernel<W_MN>;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess) return kErrDriver;
    attr = true;
  }
  const long long tiles = static_cast<long long>(max_pieces) * ((p.N + PM - 1) / PM);
  const int pairs = tiles < sm_count() / 2 ? static_cast<int>(tiles) : sm_count() / 2;
  TTB_COUNT_LAUNCH(1);
  kernel<<<2 * pairs, kThreads, kSmemBytes, st>>>(tmW, tmX[0], tmX[1], tmX[2], p);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}

}  // namespace gg
}  // namespace ttb

// C[rows, N] = X[rows, K] · op(W[e]) for the rows of each expert e, as ttb_gemm_grouped_bf16.  `counts` is a device array of E <= 1024 int64 row counts (rows of an expert are contiguous,
// in expert order); `table` a device int array of 5 * max_pieces + 1 entries with max_pieces = ceil(rows / 256) + E.  w_mn = 0: W[e] is [N, K] row-major; 1: W[e] is [K, N].
extern "C" int ttb_gemm_grouped_bf16_2sm(const void* X, const void* W, void* C, const void* counts, void* table, long long rows, int num_experts, int N, int K, int w_mn, long long ldx,
                                         long long ldw, long long expert_stride, long long ldc, int* err, void* stream) {
  using namespace ttb;
  if (rows <= 0 || rows >= (1ll << 31) || num_experts <= 0 || num_experts > 1024 || N <= 0 || K <= 0) return kErrBadShape;
  if ((ldx & 7) || (ldw & 7) || (ldc & 7) || (N & 7) || (K & 7) || (expert_stride & 7) || (reinterpret_cast<uintptr_t>(C) & 15)) return kErrBadShape;
  const int max_pieces = static_cast<int>((rows + gg::kMaxTokens - 1) / gg::kMaxTokens) + num_experts;
  int* t = static_cast<int*>(table);
  auto st = static_cast<cudaStream_t>(stream);
  TTB_COUNT_LAUNCH(1);
  gg::piece_table_kernel<<<1, 1024, 0, st>>>(static_cast<const long long*>(counts), num_experts, max_pieces, rows, t);
  if (cudaGetLastError() != cudaSuccess) return kErrDriver;
  gg::Params p{};
  p.N = N, p.K = K, p.C = static_cast<__nv_bfloat16*>(C), p.ldc = ldc, p.err = err;
  p.expert = t, p.first = t + max_pieces, p.pieces = t + 2 * max_pieces, p.row0 = t + 3 * max_pieces, p.rows = t + 4 * max_pieces, p.total = t + 5 * max_pieces;
  return w_mn ? gg::launch<true>(X, W, p, rows, num_experts, max_pieces, ldx, ldw, expert_stride, st) : gg::launch<false>(X, W, p, rows, num_experts, max_pieces, ldx, ldw, expert_stride, st);
}
