// Token sampling for generation: temperature, optional top-k, one draw per row, in one kernel launch.
//
// The reference divides the logits by the temperature, keeps the top_k largest, takes a softmax and draws with the exponential
// race argmax(p / q), q ~ Exp(1) (torchtune/generation/_generation.py:14-66).  Since p_v = exp(t_v − lse) the winner is
// argmax(t_v − log q_v) over the kept columns, so neither the softmax nor the [rows, vocab] probability tensor is needed.
// A radix select over the order-preserving integer image of t finds the top_k-th largest value, one more pass takes the arg-max.
// Ties go to the lowest index, as torch.argmax does.
//
// A cluster of eight CTAs works on a row: each reads its part of the row once and keeps it in shared memory (128 256 fp32 logits: 64 KB
// per CTA), so the passes after the first don't touch memory, and the CTAs meet in distributed shared memory.  Digits of 11, 11 and 10
// bits: the first one splits an octave in four, which spreads the logits of a warp over enough counters that its atomics rarely
// meet (with 8 bits, sign and exponent alone, almost all lanes hit the same few), and the later ones only see the columns of one bucket.
// 128 256 fp32 columns, top 300, one CTA per row and four passes over it before -> here: 1 row 156 -> 31 us, 16 rows 170 -> 39 us.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/tmap.h"

namespace ttb {

namespace cg = cooperative_groups;

static constexpr int kSampleThreads = 512;
static constexpr int kSampleSplit = 8;        // CTAs of a row: one cluster
static constexpr int kSampleBins = 2048;
static constexpr int kSampleCache = 48 * 1024;  // columns a CTA keeps in shared memory (192 KB); a longer part is read again in every pass

__device__ __forceinline__ uint32_t ordered_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

template <typename T>
__device__ __forceinline__ float scaled_logit(const T* row, int v, float temp);
// bf16 logits: the eager statement divides in bf16, so the quotient is rounded to bf16 before it is compared
template <>
__device__ __forceinline__ float scaled_logit<__nv_bfloat16>(const __nv_bfloat16* row, int v, float temp) {
  return __bfloat162float(__float2bfloat16_rn(__fdiv_rn(__bfloat162float(row[v]), temp)));
}
template <>
__device__ __forceinline__ float scaled_logit<float>(const float* row, int v, float temp) {
  return __fdiv_rn(row[v], temp);
}

struct SampleShared {
  unsigned int hist[kSampleBins];
  unsigned int warp_sum[kSampleThreads / 32];
  uint32_t prefix;  // written by CTA 0 of the cluster
  int k;
  float best[kSampleSplit];  // CTA 0: the candidates of all CTAs
  int best_i[kSampleSplit];
  float red_v[kSampleThreads / 32];
  int red_i[kSampleThreads / 32];
};

// grid (kSampleSplit, rows), cluster (kSampleSplit, 1)
template <typename T>
__global__ void __launch_bounds__(kSampleThreads)
sample_kernel(const T* __restrict__ logits, long long ld, const float* __restrict__ q, long long ldq, int* __restrict__ out, int V, float temp, int top_k) {
  extern __shared__ float cache[];
  __shared__ SampleShared sh;
  cg::cluster_group cluster = cg::this_cluster();
  const int part = blockIdx.x, row = blockIdx.y, tid = threadIdx.x;
  const T* lr = logits + static_cast<long long>(row) * ld;
  const float* qr = q + static_cast<long long>(row) * ldq;
  const int width = (V + kSampleSplit - 1) / kSampleSplit;
  const int v0 = min(V, part * width), n = min(V, v0 + width) - v0;
  const bool cached = width <= kSampleCache;
  if (cached)
#pragma unroll 8
    for (int i = tid; i < n; i += kSampleThreads) cache[i] = scaled_logit<T>(lr, v0 + i, temp);  // read back by the same thread only
  auto value = [&](int i) { return cached ? cache[i] : scaled_logit<T>(lr, v0 + i, temp); };
  uint32_t threshold = 0;  // keep every column
  if (top_k > 0 && top_k < V) {
    uint32_t prefix = 0, mask = 0;
    int k = top_k;
#pragma unroll 1
    for (int pass = 0; pass < 3; ++pass) {
      const int bits = pass < 2 ? 11 : 10, shift = pass == 0 ? 21 : pass == 1 ? 10 : 0, bins = 1 << bits;
      for (int b = tid; b < bins; b += kSampleThreads) sh.hist[b] = 0;
      __syncthreads();
#pragma unroll 4
      for (int i = tid; i < n; i += kSampleThreads) {
        const uint32_t key = ordered_key(value(i));
        if ((key & mask) == prefix) atomicAdd(&sh.hist[(key >> shift) & (bins - 1)], 1u);
      }
      cluster.sync();
      if (part == 0) {
        // every thread owns consecutive bins, the highest ones first, and finds out how many columns lie above them
        const int per = bins / kSampleThreads;  // 4, 4, 2
        unsigned int c[4] = {0, 0, 0, 0}, total = 0;
        const int high = bins - 1 - tid * per;
        for (int r = 0; r < kSampleSplit; ++r) {
          const unsigned int* h = cluster.map_shared_rank(sh.hist, r);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < per) c[j] += h[high - j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) total += c[j];
        unsigned int scan = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned int up = __shfl_up_sync(0xffffffffu, scan, o);
          if ((tid & 31) >= o) scan += up;
        }
        if ((tid & 31) == 31) sh.warp_sum[tid >> 5] = scan;
        __syncthreads();
        unsigned int above = scan - total;
        for (int w = 0; w < (tid >> 5); ++w) above += sh.warp_sum[w];
        const unsigned int want = static_cast<unsigned int>(k);
        if (above < want && above + total >= want) {  // exactly one thread: the k-th largest column is in its bins
          int j = 0;
          while (above + c[j] < want) above += c[j], ++j;
          sh.prefix = prefix | (static_cast<uint32_t>(high - j) << shift);
          sh.k = static_cast<int>(want - above);
        }
      }
      cluster.sync();
      const SampleShared* first = cluster.map_shared_rank(&sh, 0);
      prefix = first->prefix, k = first->k;
      mask |= static_cast<uint32_t>(bins - 1) << shift;
    }
    threshold = prefix;  // key of the top_k-th largest value
  } else {
    cluster.sync();  // all CTAs have started: their shared memory may be written
  }
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  for (int i = tid; i < n; i += kSampleThreads) {
    const float t = value(i);
    if (ordered_key(t) < threshold) continue;
    const float s = t - __logf(qr[v0 + i]);
    if (s > best || (s == best && v0 + i < best_i)) best = s, best_i = v0 + i;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
    if (ov > best || (ov == best && oi < best_i)) best = ov, best_i = oi;
  }
  if ((tid & 31) == 0) sh.red_v[tid >> 5] = best, sh.red_i[tid >> 5] = best_i;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kSampleThreads / 32; ++w)
      if (sh.red_v[w] > best || (sh.red_v[w] == best && sh.red_i[w] < best_i)) best = sh.red_v[w], best_i = sh.red_i[w];
    SampleShared* first = cluster.map_shared_rank(&sh, 0);
    first->best[part] = best, first->best_i[part] = best_i;
  }
  cluster.sync();
  if (part == 0 && tid == 0) {
    for (int r = 0; r < kSampleSplit; ++r)
      if (sh.best[r] > best || (sh.best[r] == best && sh.best_i[r] < best_i)) best = sh.best[r], best_i = sh.best_i[r];
    out[row] = best_i == 0x7fffffff ? 0 : best_i;
  }
}

template <typename T>
static int launch_sample(const void* logits, long long ld, const float* q, long long ldq, int* out, int rows, int V, float temp, int top_k, cudaStream_t s) {
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(sample_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleCache * 4) != cudaSuccess) return kErrDriver;
    attr = true;
  }
  const int width = (V + kSampleSplit - 1) / kSampleSplit;
  for (int r0 = 0; r0 < rows; r0 += 65535) {  // grid.y
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSampleSplit, rows - r0 < 65535 ? rows - r0 : 65535);
    cfg.blockDim = dim3(kSampleThreads);
    cfg.dynamicSmemBytes = width <= kSampleCache ? width * 4 : 0;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kSampleSplit, at[0].val.clusterDim.y = 1, at[0].val.clusterDim.z = 1;
    cfg.attrs = at, cfg.numAttrs = 1;
    TTB_COUNT_LAUNCH(1);
    if (cudaLaunchKernelEx(&cfg, sample_kernel<T>, static_cast<const T*>(logits) + r0 * ld, ld, q + r0 * ldq, ldq, out + r0, V, temp, top_k) != cudaSuccess) return kErrDriver;
  }
  return kOk;
}

}  // namespace ttb

// logits: [rows, V] bf16 (is_bf16 != 0) or fp32, row pitch ld elements; q: [rows, V] fp32 draws from Exp(1), pitch ldq; out: [rows] int32.
// top_k <= 0 or >= V keeps every column.
extern "C" int ttb_sample(const void* logits, long long ld, int is_bf16, const float* q, long long ldq, int* out, int rows, int V, float temperature, int top_k,
                          void* stream) {
  using namespace ttb;
  if (rows <= 0 || V <= 0 || q == nullptr || out == nullptr) return kErrBadShape;
  const float temp = fmaxf(temperature, 1e-5f);
  auto s = static_cast<cudaStream_t>(stream);
  return is_bf16 ? launch_sample<__nv_bfloat16>(logits, ld, q, ldq, out, rows, V, temp, top_k, s) : launch_sample<float>(logits, ld, q, ldq, out, rows, V, temp, top_k, s);
}
