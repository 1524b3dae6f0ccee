// Row-wise softmax cross-entropy over a chunk of logits, fused with its gradient.
//
// For each row: lse = logsumexp(logits), loss = lse - logits[label]; with `write_grad` the
// logits are overwritten in place by d(loss)/d(logits) = softmax - onehot (bf16), which the
// caller feeds straight into the dgrad/wgrad GEMMs of the output projection, so the fp32
// [tokens, vocab] tensor of the unfused path never exists.  Rows whose label equals
// ignore_index produce loss 0 and a zero gradient row.
// Reference math: torchtune/modules/loss/cross_entropy_loss.py:87-115 (logits upcast to fp32,
// summed CE) and torchtune/rlhf/sequence_processing.py:138-178 (per-token log-probs).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/tmap.h"

TTB_DEFINE_VIOLATION_COUNTER(loss)

namespace ttb {

static constexpr int kCEThreads = 512;

// Merge two (max, sum-of-exp) partials; a partial that saw no element has s == 0 and is skipped
// (its max is -inf and must not enter an inf - inf subtraction).
__device__ __forceinline__ void online_merge(float& m, float& s, float m2, float s2) {
  if (s2 == 0.f) return;
  if (s == 0.f) {
    m = m2, s = s2;
    return;
  }
  const float nm = fmaxf(m, m2);
  s = s * __expf(m - nm) + s2 * __expf(m2 - nm);
  m = nm;
}

// mode 0: loss + in-place gradient;  mode 1: loss only;  mode 2: in-place gradient scaled by
// row_scale[row] of the *negative* loss (i.e. gradient of log p(label)), for DPO backward.
// CAP: the softmax runs over z = cap · tanh(x / cap) (Gemma-2 logit soft cap) and the gradient written back is the one with
// respect to the raw logit x: (softmax(z) − onehot) · (1 − (z / cap)²).
template <bool CAP>
__global__ void __launch_bounds__(kCEThreads)
softmax_ce_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
                  float* __restrict__ loss_out, const float* __restrict__ row_scale, int rows, int V, long long ld,
                  long long ignore_index, int mode, float cap, float inv_cap) {
  __shared__ float sm_m[kCEThreads / 32], sm_s[kCEThreads / 32];
  __shared__ float sh_m, sh_s;
  const int row = blockIdx.x;
  if (row >= rows) return;
  __nv_bfloat16* lr = logits + static_cast<long long>(row) * ld;
  const long long label = labels[row];
  const bool out_of_range = label != ignore_index && (label < 0 || label >= V);  // treated like an ignored row, and counted
  if (out_of_range && threadIdx.x == 0) TTB_NOTE_VIOLATION(loss);
  const bool ignored = label == ignore_index || out_of_range;
  const int nvec = V >> 3;

  if (ignored) {
    if (mode != 1) {
      const uint4 z = make_uint4(0, 0, 0, 0);
      for (int i = threadIdx.x; i < nvec; i += kCEThreads) reinterpret_cast<uint4*>(lr)[i] = z;
    }
    if (threadIdx.x == 0 && loss_out != nullptr) loss_out[row] = 0.f;
    return;
  }

  float m = -INFINITY, s = 0.f;
  for (int i = threadIdx.x; i < nvec; i += kCEThreads) {
    const uint4 u = reinterpret_cast<const uint4*>(lr)[i];
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(b[j]);
      f[2 * j] = t.x, f[2 * j + 1] = t.y;
    }
    if (CAP) {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = cap * tanhf(f[j] * inv_cap);
    }
    float lm = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
    float ls = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ls += __expf(f[j] - lm);
    online_merge(m, s, lm, ls);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
    online_merge(m, s, m2, s2);
  }
  if ((threadIdx.x & 31) == 0) sm_m[threadIdx.x >> 5] = m, sm_s[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tm = sm_m[0], ts = sm_s[0];
    for (int w = 1; w < kCEThreads / 32; ++w) online_merge(tm, ts, sm_m[w], sm_s[w]);
    sh_m = tm, sh_s = ts;
  }
  __syncthreads();
  const float row_max = sh_m;
  const float lse = row_max + __logf(sh_s);
  if (threadIdx.x == 0 && loss_out != nullptr) {
    float at_label = __bfloat162float(lr[label]);
    if (CAP) at_label = cap * tanhf(at_label * inv_cap);
    loss_out[row] = lse - at_label;
  }
  if (mode == 1) return;
  __syncthreads();  // the label logit was read above, before anything is overwritten

  const float sign_scale = mode == 2 ? -row_scale[row] : 1.f;
  for (int i = threadIdx.x; i < nvec; i += kCEThreads) {
    uint4 u = reinterpret_cast<const uint4*>(lr)[i];
    __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
    const long long c0 = static_cast<long long>(i) * 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = __bfloat1622float2(b[j]);
      float d0 = 1.f, d1 = 1.f;  // dz/dx
      if (CAP) {
        const float u0 = tanhf(t.x * inv_cap), u1 = tanhf(t.y * inv_cap);
        t.x = cap * u0, t.y = cap * u1;
        d0 = 1.f - u0 * u0, d1 = 1.f - u1 * u1;
      }
      float g0 = __expf(t.x - lse), g1 = __expf(t.y - lse);
      if (c0 + 2 * j == label) g0 -= 1.f;
      if (c0 + 2 * j + 1 == label) g1 -= 1.f;
      b[j] = __floats2bfloat162_rn(g0 * d0 * sign_scale, g1 * d1 * sign_scale);
    }
    reinterpret_cast<uint4*>(lr)[i] = u;
  }
}

// ----------------------------------------------------------------------------- the same from the statistics of the logits' GEMM
// Where the product that made the logits left each row's maximum and sum of exponentials per tile of 256 columns (gemm2sm.cu), the softmax needs no pass over the logits: one kernel
// merges a row's partials in their order (rows next to each other in a warp, the tiles dealt to eight warps), and the gradient is one element-wise pass, 64 bytes in flight per
// thread and no reduction, bound by its reads and writes.  8192 x 128256: 1.0 - 1.55 ms with the kernel above, 0.65 ms here (6.5 TB/s); the
// GEMM's epilogue hides behind the products of its next tile where their contraction is long (ops._cuda._stats_pay).
static constexpr int kStatTile = 256;

__global__ void __launch_bounds__(256)
ce_merge_kernel(const float2* __restrict__ stats, const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels, float* __restrict__ loss_out, float* __restrict__ lse_out,
                int rows, int V, long long ld, long long ignore_index) {
  __shared__ float2 part[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * 32 + lane, tiles = (V + kStatTile - 1) / kStatTile;
  float m = -INFINITY, s = 0.f;
  auto join = [&](float2 p) {
    const float nm = fmaxf(m, p.x), base = nm == -INFINITY ? 0.f : nm;
    s = s * __expf(m - base) + p.y * __expf(p.x - base);
    m = nm;
  };
  if (row < rows) {
    int t = warp;
    for (; t + 24 < tiles; t += 32) {
      const float2 p[4] = {stats[static_cast<long long>(t) * rows + row], stats[static_cast<long long>(t + 8) * rows + row], stats[static_cast<long long>(t + 16) * rows + row],
                           stats[static_cast<long long>(t + 24) * rows + row]};
#pragma unroll
      for (int j = 0; j < 4; ++j) join(p[j]);
    }
    for (; t < tiles; t += 8) join(stats[static_cast<long long>(t) * rows + row]);
  }
  part[warp][lane] = make_float2(m, s);
  __syncthreads();
  if (warp != 0 || row >= rows) return;
  m = -INFINITY, s = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) join(part[w][lane]);
  const long long label = labels[row];
  const bool out_of_range = label != ignore_index && (label < 0 || label >= V);  // treated like an ignored row, and counted
  if (out_of_range) TTB_NOTE_VIOLATION(loss);
  const bool ignored = label == ignore_index || out_of_range;
  const float lse = m + __logf(s);
  lse_out[row] = ignored ? INFINITY : lse;  // no probability is left of an ignored row
  loss_out[row] = ignored ? 0.f : lse - __bfloat162float(logits[row * ld + label]);
}

// logits <- softmax - onehot, rows with lse = inf <- 0.  blockIdx.y: row.
__global__ void __launch_bounds__(256)
ce_grad_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels, const float* __restrict__ lse, int V, long long ld) {
  const long long row = blockIdx.y;
  uint4* lr = reinterpret_cast<uint4*>(logits + row * ld);
  const int nvec = V >> 3, first = blockIdx.x * 1024 + threadIdx.x;
  const float z = lse[row];
  if (z == INFINITY) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (first + j * 256 < nvec) lr[first + j * 256] = make_uint4(0, 0, 0, 0);
    return;
  }
  const int label = static_cast<int>(labels[row]);
  uint4 u[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (first + j * 256 < nvec) u[j] = lr[first + j * 256];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = first + j * 256;
    if (i >= nvec) break;
    __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u[j]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 t = __bfloat1622float2(b[k]);
      float g0 = __expf(t.x - z), g1 = __expf(t.y - z);
      if (i * 8 + 2 * k == label) g0 -= 1.f;
      if (i * 8 + 2 * k + 1 == label) g1 -= 1.f;
      b[k] = __floats2bfloat162_rn(g0, g1);
    }
    lr[i] = u[j];
  }
}

// ----------------------------------------------------------------------------- log-probabilities of given tokens from fp32 logits
// out[r] = log softmax(x_r / T)[token_r], one pass over fp32 logits in which row r lies at (r / inner) * stride_outer + (r % inner) * stride_inner, so a slice of a
// batch is read where it is.  The plain statement divides, normalises into a second and gathers from a third [rows, V] tensor.  One
// CTA per row, 16 bytes per lane and load; bound by the read: 4096 x 128 256 in 326 us (6.4 TB/s), where division, softmax and gather took 3.9 ms.
static constexpr int kLPThreads = 512;

__device__ __forceinline__ void exact_merge(float& m, float& s, float m2, float s2) {
  if (m2 == -INFINITY && s2 == 0.f) return;
  if (m == -INFINITY && s == 0.f) {
    m = m2, s = s2;
    return;
  }
  const float nm = fmaxf(m, m2);
  s = s * expf(m - nm) + s2 * expf(m2 - nm);
  m = nm;
}

template <bool DIVIDE>
__global__ void __launch_bounds__(kLPThreads)
token_logprob_kernel(const float* __restrict__ x, long long stride_outer, long long stride_inner, int inner, const long long* __restrict__ tokens, float* __restrict__ out, int V, float temp) {
  __shared__ float sm_m[kLPThreads / 32], sm_s[kLPThreads / 32];
  const int row = blockIdx.x, tid = threadIdx.x;
  const float* xr = x + (row / inner) * stride_outer + (row % inner) * stride_inner;
  const float4* xv = reinterpret_cast<const float4*>(xr);
  const int nvec = V >> 2;
  float m = -INFINITY, s = 0.f;
  auto take = [&](const float4 (&a)[4], int count) {
    float f[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) f[4 * j] = a[j].x, f[4 * j + 1] = a[j].y, f[4 * j + 2] = a[j].z, f[4 * j + 3] = a[j].w;
    float lm = -INFINITY;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (DIVIDE) f[j] = __fdiv_rn(f[j], temp);
      if (j < count) lm = fmaxf(lm, f[j]);
    }
    const float nm = fmaxf(m, lm);
    const float base = nm == -INFINITY ? 0.f : nm;
    float ls = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (j < count) ls += expf(f[j] - base);
    s = (m == -INFINITY ? s : s * expf(m - base)) + ls;  // s is 0 or NaN while no column was above -inf
    m = nm;
  };
  int i = tid;
  for (; i + 3 * kLPThreads < nvec; i += 4 * kLPThreads) {
    const float4 a[4] = {__ldg(xv + i), __ldg(xv + i + kLPThreads), __ldg(xv + i + 2 * kLPThreads), __ldg(xv + i + 3 * kLPThreads)};
    take(a, 16);
  }
  for (; i < nvec; i += kLPThreads) {
    const float4 a[4] = {__ldg(xv + i)};
    take(a, 4);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
    exact_merge(m, s, m2, s2);
  }
  if ((tid & 31) == 0) sm_m[tid >> 5] = m, sm_s[tid >> 5] = s;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kLPThreads / 32; ++w) exact_merge(m, s, sm_m[w], sm_s[w]);
    const long long token = tokens[row];
    if (token < 0 || token >= V) {
      TTB_NOTE_VIOLATION(loss);
      out[row] = NAN;
    } else {
      const float t = DIVIDE ? __fdiv_rn(xr[token], temp) : xr[token];
      out[row] = (t - m) - logf(s);  // a row of -inf alone, +inf and NaN give NaN, as the plain statement does
    }
  }
}

// ----------------------------------------------------------------------------- gradient times a scalar on the device
// y = bf16(x · *factor); 16 bytes per lane and load, bound by memory: 128 256 x 2048 in 174 us (6.0 TB/s), where
// the broadcast multiplication of tensors, two bytes at a time, took 859 us.
// In place a factor of one, that of a loss that is differentiated by itself, needs no pass at all.
__global__ void __launch_bounds__(256)
scale_bf16_kernel(const uint4* x, uint4* y, long long nvec, const float* __restrict__ factor) {
  const float f = *factor;
  if (f == 1.f && x == y) return;
  const long long step = static_cast<long long>(gridDim.x) * 256;
  auto scaled = [&](uint4 u) {
    __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(b[j]);
      b[j] = __floats2bfloat162_rn(t.x * f, t.y * f);
    }
    return u;
  };
  long long i = blockIdx.x * 256ll + threadIdx.x;
  for (; i + 3 * step < nvec; i += 4 * step) {
    uint4 u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = x[i + j * step];
#pragma unroll
    for (int j = 0; j < 4; ++j) y[i + j * step] = scaled(u[j]);
  }
  for (; i < nvec; i += step) y[i] = scaled(x[i]);
}

// ----------------------------------------------------------------------------- distillation divergences
// Per row, with p_s = softmax(student), p_t = softmax(teacher) over V columns (fp32 math on bf16 logits):
//   forward KL term   F = −Σ p_t · log p_s          d F / d s_j = p_s(j) − p_t(j)
//   reverse KL        R =  Σ p_s · (log p_s − log p_t)   d R / d s_j = p_s(j) · ((log p_s(j) − log p_t(j)) − R)
// loss_out[row] = w_fwd · F + w_rev · R, grad[row, :] = the same combination of the two gradients (bf16; may alias nothing).
// Columns whose student logit is ±inf contribute nothing (the reference masks them, torchtune/modules/loss/kd_losses.py:54-60,
// 129-140); rows whose label equals ignore_index give loss 0 and a zero gradient row.
static constexpr int kKDThreads = 512;

__device__ __forceinline__ float kd_block_sum(float v, float* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < kKDThreads / 32; ++w) t += scratch[w];
  return t;
}
__device__ __forceinline__ float kd_block_max(float v, float* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = -INFINITY;
  for (int w = 0; w < kKDThreads / 32; ++w) t = fmaxf(t, scratch[w]);
  return t;
}

__global__ void __launch_bounds__(kKDThreads)
kd_divergence_kernel(const __nv_bfloat16* __restrict__ student, const __nv_bfloat16* __restrict__ teacher, const long long* __restrict__ labels,
                     float* __restrict__ loss_out, __nv_bfloat16* __restrict__ grad, int rows, int V, long long ld_s, long long ld_t, long long ld_g,
                     long long ignore_index, float w_fwd, float w_rev) {
  __shared__ float scratch[kKDThreads / 32];
  const int row = blockIdx.x;
  if (row >= rows) return;
  const int nvec = V >> 3;
  const uint4* sr = reinterpret_cast<const uint4*>(student + static_cast<long long>(row) * ld_s);
  const uint4* tr = reinterpret_cast<const uint4*>(teacher + static_cast<long long>(row) * ld_t);
  uint4* gr = grad != nullptr ? reinterpret_cast<uint4*>(grad + static_cast<long long>(row) * ld_g) : nullptr;
  if (labels[row] == ignore_index) {
    if (gr != nullptr) {
      const uint4 z = make_uint4(0, 0, 0, 0);
      for (int i = threadIdx.x; i < nvec; i += kKDThreads) gr[i] = z;
    }
    if (threadIdx.x == 0) loss_out[row] = 0.f;
    return;
  }
  auto unpack = [](const uint4& u, float (&f)[8]) {
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(b[j]);
      f[2 * j] = t.x, f[2 * j + 1] = t.y;
    }
  };
  // pass 1: row maxima (finite values only for the student, whose ±inf columns are masked out)
  float ms = -INFINITY, mt = -INFINITY;
  for (int i = threadIdx.x; i < nvec; i += kKDThreads) {
    float a[8], b[8];
    unpack(sr[i], a);
    unpack(tr[i], b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (!isinf(a[j])) ms = fmaxf(ms, a[j]);
      mt = fmaxf(mt, b[j]);
    }
  }
  ms = kd_block_max(ms, scratch);
  mt = kd_block_max(mt, scratch);
  // pass 2: partition sums and the two cross terms
  float zs = 0.f, zt = 0.f, c_fwd = 0.f, c_rev = 0.f;
  for (int i = threadIdx.x; i < nvec; i += kKDThreads) {
    float a[8], b[8];
    unpack(sr[i], a);
    unpack(tr[i], b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float et = __expf(b[j] - mt);
      zt += et;
      if (isinf(a[j])) {
        if (a[j] > 0.f) zs = INFINITY;  // +inf student logit: the softmax is degenerate, as in the eager statement
        continue;
      }
      const float ds = a[j] - ms;
      const float es = __expf(ds);
      zs += es;
      c_fwd += et * ds;
      if (!isinf(b[j])) c_rev += es * ((b[j] - mt) - ds);
    }
  }
  zs = kd_block_sum(zs, scratch);
  zt = kd_block_sum(zt, scratch);
  c_fwd = kd_block_sum(c_fwd, scratch);
  c_rev = kd_block_sum(c_rev, scratch);
  const float log_zs = __logf(zs), log_zt = __logf(zt);
  // Σ p_t log p_s over unmasked columns needs the teacher mass on those columns; with no masked column it is exactly 1
  float pt_mass = 0.f;
  if (w_fwd != 0.f) {
    for (int i = threadIdx.x; i < nvec; i += kKDThreads) {
      float a[8], b[8];
      unpack(sr[i], a);
      unpack(tr[i], b);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (!isinf(a[j])) pt_mass += __expf(b[j] - mt);
    }
    pt_mass = kd_block_sum(pt_mass, scratch) / zt;
  }
  const float fwd = -(c_fwd / zt - log_zs * pt_mass);          // −Σ p_t log p_s
  const float rev = -(c_rev / zs - (log_zt - log_zs));          // Σ p_s (log p_s − log p_t)
  if (threadIdx.x == 0) loss_out[row] = w_fwd * fwd + w_rev * rev;
  if (gr == nullptr) return;
  for (int i = threadIdx.x; i < nvec; i += kKDThreads) {
    float a[8], b[8], g[8];
    unpack(sr[i], a);
    unpack(tr[i], b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (isinf(a[j])) {
        g[j] = 0.f;
        continue;
      }
      const float lps = a[j] - ms - log_zs, lpt = b[j] - mt - log_zt;
      const float ps = __expf(lps), pt = __expf(lpt);
      float v = w_fwd * (ps * pt_mass - pt);
      if (w_rev != 0.f) v += w_rev * ps * ((isinf(b[j]) ? 0.f : (lps - lpt)) - rev);
      g[j] = v;
    }
    uint4 u;
    __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int j = 0; j < 4; ++j) ob[j] = __floats2bfloat162_rn(g[2 * j], g[2 * j + 1]);
    gr[i] = u;
  }
}

}  // namespace ttb

using namespace ttb;

extern "C" int ttb_softmax_ce(void* logits, const long long* labels, float* loss_out, const float* row_scale, int rows,
                              int V, long long ld, long long ignore_index, int mode, void* stream) {
  if ((V & 7) || (ld & 7)) return kErrBadShape;
  if (rows <= 0) return kOk;
  TTB_COUNT_LAUNCH(1);
  softmax_ce_kernel<false><<<rows, kCEThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(logits), labels, loss_out, row_scale, rows, V, ld, ignore_index, mode, 0.f, 0.f);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}

// Loss of every row (0 where the label is ignore_index) from the statistics that ttb_gemm_bf16_2sm_stats left; lse [rows] is scratch.  With grad the logits become the gradient
// softmax - onehot, in place.
extern "C" int ttb_softmax_ce_stats(void* logits, const float* stats, const long long* labels, float* loss_out, float* lse, int rows, int V, long long ld, long long ignore_index, int grad,
                                    void* stream) {
  if ((V & 7) || (ld & 7) || (reinterpret_cast<uintptr_t>(logits) & 15) || V <= 0) return kErrBadShape;
  if (rows <= 0) return kOk;
  auto st = static_cast<cudaStream_t>(stream);
  TTB_COUNT_LAUNCH(1);
  ce_merge_kernel<<<(rows + 31) / 32, 256, 0, st>>>(reinterpret_cast<const float2*>(stats), static_cast<const __nv_bfloat16*>(logits), labels, loss_out, lse, rows, V, ld, ignore_index);
  if (grad != 0) {
    auto* lg = static_cast<__nv_bfloat16*>(logits);
    for (int r = 0; r < rows; r += 65535) {  // rows of one launch: the grid's second dimension
      const int n = rows - r < 65535 ? rows - r : 65535;
      TTB_COUNT_LAUNCH(1);
      ce_grad_kernel<<<dim3((V / 8 + 1023) / 1024, n), 256, 0, st>>>(lg + r * ld, labels + r, lse + r, V, ld);
    }
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}

// The same with the logits soft-capped at `softcap` (> 0) before the softmax; see the kernel.
extern "C" int ttb_softmax_ce_capped(void* logits, const long long* labels, float* loss_out, const float* row_scale, int rows,
                                     int V, long long ld, long long ignore_index, int mode, float softcap, void* stream) {
  if ((V & 7) || (ld & 7) || !(softcap > 0.f)) return kErrBadShape;
  if (rows <= 0) return kOk;
  TTB_COUNT_LAUNCH(1);
  softmax_ce_kernel<true><<<rows, kCEThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(logits), labels, loss_out, row_scale, rows, V, ld, ignore_index, mode, softcap, 1.f / softcap);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}

// out[r] = log softmax(x_r / temp)[tokens[r]] for fp32 rows of V columns (a multiple of 4, all rows 16-byte aligned) at (r / inner) * stride_outer + (r % inner) * stride_inner.
extern "C" int ttb_token_logprobs_f32(const float* x, long long stride_outer, long long stride_inner, int inner, const long long* tokens, float* out, int rows, int V, float temp,
                                      void* stream) {
  if (rows <= 0) return kOk;
  if (V <= 0 || (V & 3) || (stride_outer & 3) || (stride_inner & 3) || inner <= 0 || (reinterpret_cast<uintptr_t>(x) & 15)) return kErrBadShape;
  TTB_COUNT_LAUNCH(1);
  auto st = static_cast<cudaStream_t>(stream);
  if (temp == 1.f)
    token_logprob_kernel<false><<<rows, kLPThreads, 0, st>>>(x, stride_outer, stride_inner, inner, tokens, out, V, temp);
  else
    token_logprob_kernel<true><<<rows, kLPThreads, 0, st>>>(x, stride_outer, stride_inner, inner, tokens, out, V, temp);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}

// y = bf16(x * factor[0]) for n bf16 values (a multiple of 8, 16-byte aligned); y may be x.
extern "C" int ttb_scale_bf16(const void* x, void* y, long long n, const float* factor, void* stream) {
  if (n <= 0) return kOk;
  if ((n & 7) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(y) & 15)) return kErrBadShape;
  const long long blocks = (n / 8 + 1023) / 1024;
  TTB_COUNT_LAUNCH(1);
  scale_bf16_kernel<<<static_cast<int>(blocks < 8ll * sm_count() ? blocks : 8ll * sm_count()), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint4*>(x),
                                                                                                                        static_cast<uint4*>(y), n / 8, factor);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}


// student, teacher: [rows, V] bf16 (row pitches ld_s / ld_t, multiples of 8); labels: [rows] int64; loss_out: [rows] fp32;
// grad: [rows, V] bf16 (pitch ld_g) or null.  loss = w_fwd · forward-KL term + w_rev · reverse KL per row (see the kernel).
extern "C" int ttb_kd_divergence(const void* student, const void* teacher, const long long* labels, float* loss_out, void* grad, int rows, int V, long long ld_s,
                                 long long ld_t, long long ld_g, long long ignore_index, float w_fwd, float w_rev, void* stream) {
  if ((V & 7) || (ld_s & 7) || (ld_t & 7) || (grad != nullptr && (ld_g & 7))) return kErrBadShape;
  if (rows <= 0) return kOk;
  TTB_COUNT_LAUNCH(1);
  kd_divergence_kernel<<<rows, kKDThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(student), static_cast<const __nv_bfloat16*>(teacher), labels, loss_out, static_cast<__nv_bfloat16*>(grad), rows, V, ld_s, ld_t,
      ld_g, ignore_index, w_fwd, w_rev);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrDriver;
}
