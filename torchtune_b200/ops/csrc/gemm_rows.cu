// Linear layers of a few tokens (decoding, short prompts): Y[M, N] = X[M, K] · W[N, K]ᵀ with M <= 64.
//
// Every weight is read once and used M times, so the time is that of the weights from HBM and bytes in flight decide.  The tile kernels put the
// tokens on the 128 rows of an MMA tile and give a 64- or 256-column block of weights to one CTA over the whole contraction: 2048 x 2048
// ran on 32 CTAs.  Here weight rows are the 16 rows of an m16n8k16 tile and tokens its columns, and both operands take the same
// permutation of the contraction: a lane loads 16 contiguous bytes of a weight row straight into the registers of two MMAs, nothing staged,
// 4 KB per warp and chunk with the next chunk in flight during the products.  Tokens go through a three-stage cp.async ring that
// the warps of a CTA share.  The contraction is split over the warps of a CTA and the up to 8 CTAs of a cluster until two CTAs per SM exist;
// partial sums meet in (distributed) shared memory in fp32 and in a fixed order: no workspace, no atomics.
// Up to three weights of one input (query, key and value projections) share a launch; the gated form takes a pair of weights and
// writes gate(x · W1ᵀ, x · W3ᵀ).
// M is limited to 64 because one shared-memory read of a token fragment serves one 16-row tile: beyond about 32 tokens these reads and the
// products, not the weights, set the pace.
// us per launch in a graph, weights from HBM, before on the tile kernels (whole contractions; cut into ranges since, 1 x 4096 x 14336 takes them 27) -> here: 1 x 2048 x 2048 10.7 -> 4.5, 1 x 4096 x 4096 24.3 -> 9.7,
// 1 x 4096 x 14336 72 -> 23.8 (4.9 TB/s), 16 x 4096 x 14336 53 -> 25.6, 1 x 128256 x 4096 285 -> 181 (5.8 TB/s), 16 x (14336 + 14336) x 4096 gated 88 -> 48.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/ptx.cuh"
#include "common/tmap.h"

namespace ttb {
namespace rows {

namespace cg = cooperative_groups;

static constexpr int kThreads = 256;
static constexpr int kWarps = 8;
static constexpr int kChunk = 128;     // contraction steps of a warp and chunk
static constexpr int kStages = 3;
static constexpr int kMaxSplit = 8;    // portable cluster size
static constexpr int kMaxSegments = 3;
static constexpr int kPartPitch = 20;  // floats per token of a warp's 16 partial rows: lanes of a fragment store hit distinct banks

struct Segment {
  const __nv_bfloat16* w;
  void* y;                    // [M, n] bf16, or fp32 with out_f32 (2: rounded to bf16 first)
  const __nv_bfloat16* bias;  // [n] or nullptr
  long long ldw, ldy;
  int n, first_tile;
};

struct Params {
  Segment seg[kMaxSegments];
  int segments;
  const __nv_bfloat16* up;  // gated form: second weight, same shape and pitch as seg[0].w
  const __nv_bfloat16* x;
  const __nv_bfloat16* residual;  // [M, n] of segment 0, or nullptr
  long long ldx, ldr;
  int M, K, out_f32;
  float alpha;
  float glu_limit, glu_alpha;  // glu_limit > 0: the clamped gate
  const __nv_bfloat16* norm;   // gain of an RMS norm of x, or nullptr
  float eps;
};

__device__ __forceinline__ uint4 load_weight(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(b[i]);
    f[2 * i] = t.x, f[2 * i + 1] = t.y;
  }
}

// MT: token tiles of 8.  WK: warps of a CTA that share 16 rows and split a chunk of WK * kChunk contraction steps.
template <int MT, int WK>
struct Layout {
  static constexpr int kTokens = MT * 8;
  static constexpr int kRowWarps = kWarps / WK;
  static constexpr int kStep = WK * kChunk;
  static constexpr int kPitch = kStep * 2 + 64;  // bytes of a token: the two tokens of a quarter warp read different halves of the 32 banks
  static constexpr int kStageBytes = kTokens * kPitch;
  static constexpr int kPartBytes = kWarps * kTokens * kPartPitch * 4;
  static constexpr int kSmem = kStages * kStageBytes > kPartBytes ? kStages * kStageBytes : kPartBytes;
};

// Partial sums of the warps and of the cluster's CTAs meet in (distributed) shared memory, in the order of warps and CTAs, and become results.  part: [warp][token][kPartPitch], 16 rows
// of each token.
template <int MT, int WK, bool GATED>
__device__ __forceinline__ void finish(const Params& p, const Segment& sg, float* part, const float (&acc)[MT][4], int row0, int split, int splits) {
  using L = Layout<MT, WK>;
  constexpr int kOutWarps = GATED ? L::kRowWarps / 2 : L::kRowWarps;
  constexpr int kOutRows = kOutWarps * 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  {
    float* mine = part + warp * L::kTokens * kPartPitch;
#pragma unroll
    for (int n = 0; n < MT; ++n) {
      float* at = mine + (n * 8 + t * 2) * kPartPitch + g;
      at[0] = acc[n][0];
      at[kPartPitch] = acc[n][1];
      at[8] = acc[n][2];
      at[kPartPitch + 8] = acc[n][3];
    }
  }
  cg::cluster_group cluster = cg::this_cluster();
  if (splits > 1)
    cluster.sync();
  else
    __syncthreads();
  for (int idx = split * kThreads + threadIdx.x; idx < kOutRows * p.M; idx += splits * kThreads) {
    const int r = idx % kOutRows, token = idx / kOutRows, row = row0 + r;
    const int at = ((r / 16) * WK * L::kTokens + token) * kPartPitch + r % 16;
    constexpr int kNextWarp = L::kTokens * kPartPitch, kSecond = kOutWarps * WK * kNextWarp;
    float v = 0.f, u = 0.f;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) {
      const float* from = splits > 1 ? cluster.map_shared_rank(part, s) : part;
#pragma unroll
      for (int k = 0; k < WK; ++k) {
        v += from[at + k * kNextWarp];
        if (GATED) u += from[at + kSecond + k * kNextWarp];
      }
    }
    if (row >= sg.n) continue;
    if (GATED) {
      // pre-activations rounded to bf16, as the other gated kernels have them
      const float a = __bfloat162float(__float2bfloat16_rn(v)), b = __bfloat162float(__float2bfloat16_rn(u));
      if (p.glu_limit > 0.f) {
        const float ac = fminf(a, p.glu_limit), bc = fminf(fmaxf(b, -p.glu_limit), p.glu_limit);
        v = __fdividef(ac, 1.f + __expf(-p.glu_alpha * ac)) * (bc + 1.f);
      } else {
        v = a / (1.f + __expf(-a)) * b;
      }
    } else {
      v *= p.alpha;
      if (sg.bias != nullptr) v += __bfloat162float(sg.bias[row]);
      if (p.residual != nullptr) v += __bfloat162float(p.residual[token * p.ldr + row]);
    }
    if (p.out_f32)
      static_cast<float*>(sg.y)[token * sg.ldy + row] = p.out_f32 == 2 ? __bfloat162float(__float2bfloat16_rn(v)) : v;
    else
      static_cast<__nv_bfloat16*>(sg.y)[token * sg.ldy + row] = __float2bfloat16_rn(v);
  }
  if (splits > 1) cluster.sync();  // no CTA leaves while another reads its shared memory
}

// grid (tiles * splits), cluster (splits): consecutive CTAs split the contraction of one tile of kRowWarps * 16 weight rows.
template <int MT, int WK, bool GATED>
__global__ void __launch_bounds__(kThreads, 2)
gemm_rows_kernel(const __grid_constant__ Params p, int splits) {
  using L = Layout<MT, WK>;
  constexpr int kOutWarps = GATED ? L::kRowWarps / 2 : L::kRowWarps;  // the other half of a gated CTA's warps holds the rows of the second weight
  constexpr int kOutRows = kOutWarps * 16;
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / splits, split = blockIdx.x % splits;
  int si = 0;
  if (p.segments > 1 && tile >= p.seg[1].first_tile) si = 1;
  if (p.segments > 2 && tile >= p.seg[2].first_tile) si = 2;
  const Segment& sg = p.seg[si];
  const int row0 = (tile - sg.first_tile) * kOutRows;
  const int wr = warp / WK, wk = warp % WK;
  const bool second = GATED && wr >= kOutWarps;
  const int wrow = row0 + (second ? wr - kOutWarps : wr) * 16;
  const int g = lane >> 2, t = lane & 3;
  const __nv_bfloat16* w = second ? p.up : sg.w;
  const long long ldw = sg.ldw;
  // rows past the end read the last row; their results are not stored
  const __nv_bfloat16* w0 = w + static_cast<long long>(min(wrow + g, sg.n - 1)) * ldw;
  const __nv_bfloat16* w1 = w + static_cast<long long>(min(wrow + g + 8, sg.n - 1)) * ldw;
  const int chunks = (p.K + L::kStep - 1) / L::kStep;
  const int own = chunks > split ? (chunks - split + splits - 1) / splits : 0;

  auto load_w = [&](int i, uint4 (&a)[4], uint4 (&b)[4]) {
    const int k0 = (split + i * splits) * L::kStep + wk * kChunk + t * 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + j * 32;  // K is a multiple of 8, so 16 bytes are inside or outside as a whole
      if (i < own && k < p.K) {
        a[j] = load_weight(w0 + k);
        b[j] = load_weight(w1 + k);
      } else {
        a[j] = make_uint4(0, 0, 0, 0);
        b[j] = make_uint4(0, 0, 0, 0);
      }
    }
  };
  const uint32_t ring = smem_u32(smem);
  auto load_x = [&](int i) {
    if (i < own) {
      const int k0 = (split + i * splits) * L::kStep;
      const uint32_t dst = ring + (i % kStages) * L::kStageBytes;
      constexpr int kPieces = L::kStep / 8;
      for (int c = threadIdx.x; c < L::kTokens * kPieces; c += kThreads) {
        const int token = c / kPieces, piece = c % kPieces;
        const int k = k0 + piece * 8;
        const bool keep = token < p.M && k < p.K;
        const __nv_bfloat16* src = p.x + (keep ? token * p.ldx + k : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + token * L::kPitch + piece * 16), "l"(src), "r"(keep ? 16 : 0) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[MT][4];
#pragma unroll
  for (int n = 0; n < MT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  auto products = [&](int i, const uint4 (&a)[4], const uint4 (&b)[4]) {
    const uint8_t* xs = smem + (i % kStages) * L::kStageBytes + g * L::kPitch + wk * (kChunk * 2) + t * 16;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int n = 0; n < MT; ++n) {
        const uint4 v = *reinterpret_cast<const uint4*>(xs + n * 8 * L::kPitch + j * 64);
        mma16816(acc[n], a[j].x, b[j].x, a[j].y, b[j].y, v.x, v.y);
        mma16816(acc[n], a[j].z, b[j].z, a[j].w, b[j].w, v.z, v.w);
      }
    }
  };

  uint4 a0[4], b0[4], a1[4], b1[4];
  load_w(0, a0, b0);
  load_x(0);
  load_x(1);
  for (int i = 0; i < own; i += 2) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // stage i is complete for all, and all have finished with stage i - 1, which is filled next
    load_w(i + 1, a1, b1);
    load_x(i + 2);
    products(i, a0, b0);
    if (i + 1 >= own) break;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    load_w(i + 2, a0, b0);
    load_x(i + 3);
    products(i + 1, a1, b1);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  finish<MT, WK, GATED>(p, sg, reinterpret_cast<float*>(smem), acc, row0, split, splits);
}

// Up to 16 tokens whose share of a CTA's contraction fits shared memory as a whole: they are staged once, and the warps stream their weights without meeting until the end.  With NORM, x is normalised on
// the way in (the sums of squares in the order of the norm's own kernel, so the values are the same ones): a norm by itself is a launch of 2 us in a decode step, and here its reads
// hide behind the first weights.
// us in a graph, weights from HBM, with the ring above -> here, 1 / 16 tokens: 6144 x 4096 14.6 / 16.9 -> 13.2 / 15.8, 4096 x 14336 25.1 / 27.6 -> 23.0 / 25.2 (5.1 TB/s), 128256 x 2048
// 94.8 / 104 -> 82.4 / 97.2 (6.4 TB/s), 128256 x 4096 186 -> 163 (6.4 TB/s).  A chat turn of the 16-layer 1B model, with the norms, 25.1 -> 23.0 ms.
template <int MT, int WK, bool GATED, bool NORM>
__global__ void __launch_bounds__(kThreads, 2)
gemm_rows_resident_kernel(const __grid_constant__ Params p, int splits) {
  using L = Layout<MT, WK>;
  constexpr int kOutWarps = GATED ? L::kRowWarps / 2 : L::kRowWarps;
  constexpr int kOutRows = kOutWarps * 16;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float sums[kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / splits, split = blockIdx.x % splits;
  int si = 0;
  if (p.segments > 1 && tile >= p.seg[1].first_tile) si = 1;
  if (p.segments > 2 && tile >= p.seg[2].first_tile) si = 2;
  const Segment& sg = p.seg[si];
  const int row0 = (tile - sg.first_tile) * kOutRows;
  const int wr = warp / WK, wk = warp % WK;
  const bool second = GATED && wr >= kOutWarps;
  const int wrow = row0 + (second ? wr - kOutWarps : wr) * 16;
  const int g = lane >> 2, t = lane & 3;
  const __nv_bfloat16* w = second ? p.up : sg.w;
  const __nv_bfloat16* w0 = w + static_cast<long long>(min(wrow + g, sg.n - 1)) * sg.ldw;
  const __nv_bfloat16* w1 = w + static_cast<long long>(min(wrow + g + 8, sg.n - 1)) * sg.ldw;
  const int chunks = (p.K + L::kStep - 1) / L::kStep;
  const int own = chunks > split ? (chunks - split + splits - 1) / splits : 0;
  auto load_w = [&](int i, uint4 (&a)[4], uint4 (&b)[4]) {
    const int k0 = (split + i * splits) * L::kStep + wk * kChunk + t * 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + j * 32;
      if (i < own && k < p.K) {
        a[j] = load_weight(w0 + k);
        b[j] = load_weight(w1 + k);
      } else {
        a[j] = make_uint4(0, 0, 0, 0);
        b[j] = make_uint4(0, 0, 0, 0);
      }
    }
  };
  uint4 a0[4], b0[4], a1[4], b1[4];
  load_w(0, a0, b0);
  load_w(1, a1, b1);

  // the own chunks of a token, one after the other; the two tokens of a quarter warp read different halves of the 32 banks
  const int pitch = (chunks + splits - 1) / splits * L::kStep * 2 + 64;
  if (NORM) {
    // half of the CTA takes a token, as the norm's kernel of 128 threads does
    for (int m0 = 0; m0 < p.M; m0 += 2) {
      const int m = m0 + (threadIdx.x >> 7), at = threadIdx.x & 127;
      float ss = 0.f;
      uint4 u[4];
      if (m < p.M) {
        const uint4* xr = reinterpret_cast<const uint4*>(p.x + m * p.ldx);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          u[k] = at + k * 128 < p.K / 8 ? xr[at + k * 128] : make_uint4(0, 0, 0, 0);
          float f[8];
          unpack8(u[k], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (m0 > 0) __syncthreads();  // the last pair's sums are read
      if (lane == 0) sums[warp] = ss;
      __syncthreads();
      if (m < p.M) {
        const float* four = sums + (warp & 4);
        const float rstd = rsqrtf(((four[0] + four[2]) + (four[1] + four[3])) / p.K + p.eps);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = at + k * 128, chunk = i / (L::kStep / 8);
          if (i < p.K / 8 && chunk % splits == split) {
            float f[8], s[8];
            unpack8(u[k], f);
            unpack8(__ldg(reinterpret_cast<const uint4*>(p.norm) + i), s);
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(__float2bfloat16_rn(f[j] * rstd)) * s[j];
            *reinterpret_cast<uint4*>(smem + m * pitch + (chunk / splits * (L::kStep / 8) + i % (L::kStep / 8)) * 16) =
                make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
          }
        }
      }
    }
  } else {
    constexpr int kPieces = L::kStep / 8;
    for (int c = threadIdx.x; c < own * kPieces; c += kThreads) {
      const int k = (split + c / kPieces * splits) * L::kStep + c % kPieces * 8;
      if (k < p.K) {
        for (int m = 0; m < p.M; ++m)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem) + m * pitch + c * 16), "l"(p.x + m * p.ldx + k) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();

  float acc[MT][4];
#pragma unroll
  for (int n = 0; n < MT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  auto products = [&](int i, const uint4 (&a)[4], const uint4 (&b)[4]) {
    const int at = wk * kChunk + t * 8, k0 = (split + i * splits) * L::kStep + at;
    const uint8_t* xs = smem + g * pitch + (i * L::kStep + at) * 2;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int n = 0; n < MT; ++n) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (g + n * 8 < p.M && k0 + j * 32 < p.K) v = *reinterpret_cast<const uint4*>(xs + n * 8 * pitch + j * 64);
        mma16816(acc[n], a[j].x, b[j].x, a[j].y, b[j].y, v.x, v.y);
        mma16816(acc[n], a[j].z, b[j].z, a[j].w, b[j].w, v.z, v.w);
      }
    }
  };
  for (int i = 0; i < own; i += 2) {
    products(i, a0, b0);
    load_w(i + 2, a0, b0);
    if (i + 1 >= own) break;
    products(i + 1, a1, b1);
    load_w(i + 3, a1, b1);
  }
  __syncthreads();
  finish<MT, WK, GATED>(p, sg, reinterpret_cast<float*>(smem), acc, row0, split, splits);
}

static constexpr int kMaxResident = 96 * 1024;  // two CTAs per SM

template <typename Kernel>
static int start(Kernel kernel, bool& attr, int most, int smem, const Params& p, int tiles, int splits, cudaStream_t st) {
  if (!attr) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return kErrDriver;
    attr = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * splits);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = splits, at[0].val.clusterDim.y = 1, at[0].val.clusterDim.z = 1;
  cfg.attrs = at, cfg.numAttrs = 1;
  TTB_COUNT_LAUNCH(1);
  return cudaLaunchKernelEx(&cfg, kernel, p, splits) == cudaSuccess ? kOk : kErrDriver;
}

template <int MT, int WK, bool GATED>
static int launch(Params& p, int tiles, int splits, cudaStream_t st) {
  static bool attr[3] = {false, false, false};
  if constexpr (MT <= 2) {
    using L = Layout<MT, WK>;
    const int chunks = (p.K + L::kStep - 1) / L::kStep;
    long long bytes = p.M * ((chunks + splits - 1) / splits * L::kStep * 2ll + 64);
    bytes = bytes > L::kPartBytes ? bytes : L::kPartBytes;
    // with fewer than four chunks to a CTA the staging in front is what counts (16 x 3072 x 2048: 7.0 us with the ring, 7.5 with all of it first)
    if (bytes <= kMaxResident && (p.norm != nullptr || chunks >= 4 * splits)) {
      if (p.norm == nullptr) return start(gemm_rows_resident_kernel<MT, WK, GATED, false>, attr[0], kMaxResident, static_cast<int>(bytes), p, tiles, splits, st);
      if constexpr (MT == 1) return start(gemm_rows_resident_kernel<MT, WK, GATED, true>, attr[1], kMaxResident, static_cast<int>(bytes), p, tiles, splits, st);
    }
  }
  if (p.norm != nullptr) return kErrBadShape;
  constexpr int smem = Layout<MT, WK>::kSmem;
  return start(gemm_rows_kernel<MT, WK, GATED>, attr[2], smem, smem, p, tiles, splits, st);
}

// Rows per CTA: the most (fewest re-reads of the tokens, longest loads per row) that can still fill more than half of the two CTA places per SM; the
// split is the largest power of two that stays within them, since a second, nearly empty wave costs more than it brings.
template <int MT, bool GATED>
static int dispatch(Params& p, cudaStream_t st) {
  constexpr int kMaxWk = MT == 1 ? (GATED ? 4 : 8) : MT == 2 ? 4 : MT == 4 ? 2 : 1;  // MT * WK <= 8 keeps a stage within 20 KB
  const int want = 2 * sm_count();
  int wk = 1, tiles = 0;
  for (;; wk *= 2) {
    const int out_rows = kWarps / wk * 16 / (GATED ? 2 : 1);
    tiles = 0;
    for (int i = 0; i < p.segments; ++i) p.seg[i].first_tile = tiles, tiles += (p.seg[i].n + out_rows - 1) / out_rows;
    if (wk == kMaxWk || 2ll * tiles * kMaxSplit > want) break;
  }
  const int chunks = (p.K + wk * kChunk - 1) / (wk * kChunk);
  int splits = 1;
  while (splits < kMaxSplit && 2ll * tiles * splits <= want && 2 * splits <= chunks) splits *= 2;
  if (wk == 1) return launch<MT, 1, GATED>(p, tiles, splits, st);
  if constexpr (kMaxWk >= 2) {
    if (wk == 2) return launch<MT, 2, GATED>(p, tiles, splits, st);
  }
  if constexpr (kMaxWk >= 4) {
    if (wk == 4) return launch<MT, 4, GATED>(p, tiles, splits, st);
  }
  if constexpr (kMaxWk >= 8) {
    if (wk == 8) return launch<MT, 8, GATED>(p, tiles, splits, st);
  }
  return kErrBadShape;
}

template <bool GATED>
static int by_tokens(Params& p, cudaStream_t st) {
  if (p.M <= 8) return dispatch<1, GATED>(p, st);
  if (p.M <= 16) return dispatch<2, GATED>(p, st);
  if (p.M <= 32) return dispatch<4, GATED>(p, st);
  return dispatch<8, GATED>(p, st);
}

static bool unaligned(const void* t, long long ld) { return (reinterpret_cast<uintptr_t>(t) & 15) || (ld & 7); }

}  // namespace rows
}  // namespace ttb

// Y_i[M, n_i] = alpha * X[M, K] · W_i[n_i, K]ᵀ (+ bias_i) (+ residual, first weight only) for up to three weights of one input, M <= 64, K a
// multiple of 8, X and W rows 16-byte aligned.  bf16 results; fp32 with out_f32 = 1, the bf16 ones widened with 2.
static int rows_product(const void* x, long long ldx, const void* norm, float eps, int M, int K, int count, const void* const* w, const long long* ldw, const int* n, void* const* y,
                        const long long* ldy, const void* const* bias, const void* residual, long long ldr, int out_f32, float alpha, void* stream) {
  using namespace ttb;
  if (M <= 0 || M > 64 || K <= 0 || (K & 7) || count < 1 || count > rows::kMaxSegments || rows::unaligned(x, ldx)) return kErrBadShape;
  rows::Params p{};
  p.segments = count, p.M = M, p.K = K, p.out_f32 = out_f32, p.alpha = alpha;
  p.x = static_cast<const __nv_bfloat16*>(x), p.ldx = ldx, p.norm = static_cast<const __nv_bfloat16*>(norm), p.eps = eps;
  p.residual = static_cast<const __nv_bfloat16*>(residual), p.ldr = ldr;
  for (int i = 0; i < count; ++i) {
    if (n[i] <= 0 || rows::unaligned(w[i], ldw[i])) return kErrBadShape;
    p.seg[i].w = static_cast<const __nv_bfloat16*>(w[i]), p.seg[i].y = y[i], p.seg[i].bias = bias == nullptr ? nullptr : static_cast<const __nv_bfloat16*>(bias[i]);
    p.seg[i].ldw = ldw[i], p.seg[i].ldy = ldy[i], p.seg[i].n = n[i];
  }
  return rows::by_tokens<false>(p, static_cast<cudaStream_t>(stream));
}
static int rows_gated(const void* x, long long ldx, const void* norm, float eps, const void* w1, const void* w3, long long ldw, void* h, long long ldh, int M, int N, int K, float glu_limit,
                      float glu_alpha, void* stream) {
  using namespace ttb;
  if (M <= 0 || M > 64 || N <= 0 || K <= 0 || (K & 7) || rows::unaligned(x, ldx) || rows::unaligned(w1, ldw) || rows::unaligned(w3, ldw)) return kErrBadShape;
  rows::Params p{};
  p.segments = 1, p.M = M, p.K = K, p.alpha = 1.f, p.glu_limit = glu_limit, p.glu_alpha = glu_alpha;
  p.x = static_cast<const __nv_bfloat16*>(x), p.ldx = ldx, p.norm = static_cast<const __nv_bfloat16*>(norm), p.eps = eps;
  p.up = static_cast<const __nv_bfloat16*>(w3);
  p.seg[0].w = static_cast<const __nv_bfloat16*>(w1), p.seg[0].y = h, p.seg[0].ldw = ldw, p.seg[0].ldy = ldh, p.seg[0].n = N;
  return rows::by_tokens<true>(p, static_cast<cudaStream_t>(stream));
}

extern "C" int ttb_gemm_rows(const void* x, long long ldx, int M, int K, int count, const void* const* w, const long long* ldw, const int* n, void* const* y, const long long* ldy,
                             const void* const* bias, const void* residual, long long ldr, int out_f32, float alpha, void* stream) {
  return rows_product(x, ldx, nullptr, 0.f, M, K, count, w, ldw, n, y, ldy, bias, residual, ldr, out_f32, alpha, stream);
}

// H[M, N] = silu(X · W1ᵀ) ⊙ (X · W3ᵀ), or the clamped gate with glu_limit > 0 (as ttb_gemm_swiglu_bf16_2sm), M <= 64; both weights [N, K] with pitch ldw.
extern "C" int ttb_gemm_rows_gated(const void* x, long long ldx, const void* w1, const void* w3, long long ldw, void* h, long long ldh, int M, int N, int K, float glu_limit,
                                   float glu_alpha, void* stream) {
  return rows_gated(x, ldx, nullptr, 0.f, w1, w3, ldw, h, ldh, M, N, K, glu_limit, glu_alpha, stream);
}

// Whether the two below take rows of these sizes: tokens that fit shared memory, widths whose norm has a kernel of 128 threads per row.
extern "C" int ttb_gemm_rows_norms(int M, int K) { return M > 0 && M <= 8 && K >= 1024 && K <= 4096 && K % 8 == 0 && M * (K * 2ll + 64) <= ttb::rows::kMaxResident; }

// ttb_gemm_rows and ttb_gemm_rows_gated on rmsnorm(X) = bf16(X · rsqrt(mean(X²) + eps)) · norm, value for value what ttb_rmsnorm_fwd gives.
extern "C" int ttb_gemm_rows_normed(const void* x, long long ldx, const void* norm, float eps, int M, int K, int count, const void* const* w, const long long* ldw, const int* n, void* const* y,
                                    const long long* ldy, const void* const* bias, void* stream) {
  if (!ttb_gemm_rows_norms(M, K) || norm == nullptr || (reinterpret_cast<uintptr_t>(norm) & 15)) return ttb::kErrBadShape;
  return rows_product(x, ldx, norm, eps, M, K, count, w, ldw, n, y, ldy, bias, nullptr, 0, 0, 1.f, stream);
}
extern "C" int ttb_gemm_rows_gated_normed(const void* x, long long ldx, const void* norm, float eps, const void* w1, const void* w3, long long ldw, void* h, long long ldh, int M, int N, int K,
                                          void* stream) {
  if (!ttb_gemm_rows_norms(M, K) || norm == nullptr || (reinterpret_cast<uintptr_t>(norm) & 15)) return ttb::kErrBadShape;
  return rows_gated(x, ldx, norm, eps, w1, w3, ldw, h, ldh, M, N, K, 0.f, 0.f, stream);
}
