// The layers of a plain decoder on its KV caches, issued by one call: the launches that the modules' own forward passes make outside autograd, in the same order, by the
// same rules and with the same results.
//
// A forward pass of 37 tokens through 16 layers of 2048 / 8192 is 160 launches that the GPU works off in about 2 ms; the modules took 9.2 ms to issue them (58 us a
// launch, of which the launch itself is 3) and 7.1 ms to record a step, which takes 0.8 ms from here.  A prompt of 37 tokens and 24 generated ones: 39.9 -> 25.1 ms.
// What the mask means to the attention kernel (first and last visible key of a row) is worked out once for all layers.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common/tmap.h"

extern "C" {
int ttb_rmsnorm_fwd(const void* x, const void* scale, void* y, float* rstd, int rows, int D, float eps, void* stream);
int ttb_swiglu_fwd(const void* g, const void* u, void* y, long long rows, int H, long long ldg, long long ldu, long long ldy, void* stream);
int ttb_rope_append(const void* q, const void* k, const void* v, void* q_out, void* k_cache, void* v_cache, const float* cache, const int* pos, const long long* slots, long long tokens, int hq,
                    int hkv, int d, int seq_len, int max_seq, int interleaved, int cache_len, void* stream);
int ttb_attn_decode(const void* q, const void* k, const void* v, void* o, const void* mask, long long mask_b, long long mask_r, const int* lo, const int* hi, int b, int s, int sk, int hq, int hkv,
                    int d, float scale, void* stream);
int ttb_attn_decode_append(const void* q, const void* k, const void* v, void* o, void* k_cache, void* v_cache, const float* rope, const int* pos, const long long* slots, const void* mask,
                           long long mask_b, int b, int max_seq, int hq, int hkv, int d, int interleaved, int rope_len, float scale, void* stream);
int ttb_mask_bounds(const void* mask, long long stride_b, long long stride_r, int b, int s, int sk, int* lo, int* hi, void* solid, void* stream);
int ttb_attn_fwd2_masked(const void* q, const void* k, const void* v, void* o, float* lse, const int* lo, const int* hi, const void* solid, long long bound_b, const void* mask, long long mask_b,
                         long long mask_r, int b, int s, int sk, int hq, int hkv, int d, float scale, int* err, void* stream);
int ttb_gemm_rows(const void* x, long long ldx, int M, int K, int count, const void* const* w, const long long* ldw, const int* n, void* const* y, const long long* ldy, const void* const* bias,
                  const void* residual, long long ldr, int out_f32, float alpha, void* stream);
int ttb_gemm_rows_gated(const void* x, long long ldx, const void* w1, const void* w3, long long ldw, void* h, long long ldh, int M, int N, int K, float glu_limit, float glu_alpha, void* stream);
int ttb_gemm_rows_norms(int M, int K);
int ttb_gemm_rows_normed(const void* x, long long ldx, const void* norm, float eps, int M, int K, int count, const void* const* w, const long long* ldw, const int* n, void* const* y,
                         const long long* ldy, const void* const* bias, void* stream);
int ttb_gemm_rows_gated_normed(const void* x, long long ldx, const void* norm, float eps, const void* w1, const void* w3, long long ldw, void* h, long long ldh, int M, int N, int K, void* stream);
int ttb_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int b_mn, long long lda, long long ldb, long long ldc, int out_fp32, int accumulate, const void* bias,
                  float alpha, int* err, void* stream);
int ttb_gemm_bf16_2sm(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int b_mn, long long lda, long long ldb, long long ldc, int accumulate, const void* bias, float alpha,
                      int* err, void* stream);
int ttb_gemm_bf16_2sm_residual(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int b_mn, long long lda, long long ldb, long long ldc, long long ldr, const void* bias, int* err,
                               void* stream);
int ttb_gemm_bf16_splitk(const void* A, const void* B, float* work, void* C, int M, int N, int K, int a_mn, int b_mn, long long lda, long long ldb, long long ldc, int out_fp32, int accumulate,
                         const void* bias, const void* residual, long long ldr, int splits, float alpha, int* err, void* stream);
int ttb_gemm_swiglu_bf16_2sm(const void* X, const void* W1, const void* W3, void* H, void* gate_out, void* up_out, int M, int N, int K, long long lda, long long ldb, long long ldc, float glu_limit,
                             float glu_alpha, int* err, void* stream);
}

namespace ttb {
namespace layers {

// y += r; y and r bf16, 16 bytes per lane
__global__ void __launch_bounds__(256) add_kernel(uint4* __restrict__ y, const uint4* __restrict__ r, long long n) {
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
    uint4 a = y[i];
    const uint4 b = r[i];
    __nv_bfloat162* x = reinterpret_cast<__nv_bfloat162*>(&a);
    const __nv_bfloat162* z = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 u = __bfloat1622float2(x[j]), v = __bfloat1622float2(z[j]);
      x[j] = __floats2bfloat162_rn(u.x + v.x, u.y + v.y);
    }
    y[i] = a;
  }
}

struct Layer {
  const void *sa_scale, *wq, *wk, *wv, *wo, *mlp_scale, *w1, *w3, *w2, *bq, *bk, *bv;
  void *k_cache, *v_cache;
  const long long* slots;  // [0 ... s): slots of the new tokens
  const float* rope;       // [rope_len, D / 2, 2]
  long long rope_len;
};

struct Sizes {
  int count, b, s, dim, hq, hkv, D, hidden, max_seq;
  int M() const { return b * s; }
};

static int ceil_div(int a, int b) { return (a + b - 1) / b; }

// ---- which kernel takes a product: the rules of ops._cuda (_runs_rows, _splits, _fills_pairs, _gates_in_pairs), where their reasons stand; ttb_product_rules lets a test compare the two
static bool runs_rows(int M, int N, int K) {
  const int most = N <= 4096 ? 64 : N <= 32768 ? 32 : K < 4096 ? 16 : 8;
  return M > 0 && M <= most && K > 0 && K % 8 == 0;
}
static int splits_of(int M, int N, int K) {
  if (K < 4096) return 1;
  const int tiles = ceil_div(M, 128) * ceil_div(N, N > 128 ? 256 : N > 64 ? 128 : 64);
  int s = 148 / tiles;
  s = s < 16 ? s : 16;
  s = s < K / 512 ? s : K / 512;
  return s > 1 ? s : 1;
}
static int sm_pairs() { return sm_count() / 2 > 1 ? sm_count() / 2 : 1; }
static bool fills_pairs(int M, int N, int K, int pairs) {
  const long long tiles = static_cast<long long>(ceil_div(M, 256)) * ceil_div(N, 256);
  return K >= 128 && (tiles >= pairs || (K >= 8192 && 2 * tiles > pairs && M > 128 && N > 128));
}
static bool gates_in_pairs(int M, int N, int K, int pairs) { return K >= 128 && static_cast<long long>(ceil_div(M, 256)) * ceil_div(N, 128) >= pairs; }
static bool decodes(const Sizes& z) { return z.s * (z.hq / z.hkv) <= 16 && static_cast<long long>(ceil_div(z.max_seq, 64)) * (z.s + 1) * 8 <= 16384; }

static long long split_bytes(int M, int N, int K) {
  if (runs_rows(M, N, K)) return 0;
  const int s = splits_of(M, N, K);
  return s > 1 ? 4ll * s * M * N : 0;
}

// Parts of the workspace, each on a 256-byte boundary.
struct Work {
  long long mid, norm, q, k, v, rot, att, gate, up, act, rstd, lse, lo, hi, solid, split, total;
  explicit Work(const Sizes& z) {
    long long at = 0;
    auto take = [&](long long bytes) {
      const long long here = at;
      at += (bytes + 255) / 256 * 256;
      return here;
    };
    const long long M = z.M();
    const int nq = z.hq * z.D, nk = z.hkv * z.D;
    mid = take(2 * M * z.dim), norm = take(2 * M * z.dim);
    q = take(2 * M * nq), k = take(2 * M * nk), v = take(2 * M * nk), rot = take(2 * M * nq), att = take(2 * M * nq);
    const bool fused = runs_rows(z.M(), z.hidden, z.dim) || gates_in_pairs(z.M(), z.hidden, z.dim, sm_pairs());
    gate = take(fused ? 0 : 2 * M * z.hidden), up = take(fused ? 0 : 2 * M * z.hidden), act = take(2 * M * z.hidden);
    rstd = take(4 * M);
    const bool tiles = !decodes(z);
    lse = take(tiles ? 4 * M * z.hq : 0);
    lo = take(tiles ? 4 * M : 0), hi = take(tiles ? 4 * M : 0), solid = take(tiles ? M : 0);
    long long most = 0;
    const int shapes[][2] = {{nq, z.dim}, {nk, z.dim}, {z.dim, nq}, {z.hidden, z.dim}, {z.dim, z.hidden}};
    for (const auto& n : shapes) {
      const long long need = split_bytes(z.M(), n[0], n[1]);
      most = need > most ? need : most;
    }
    split = take(most);
    total = at;
  }
};

struct Call {
  float* split;
  int* err;
  cudaStream_t st;
  int rc = kOk;
  bool ok(int r) {
    if (rc == kOk) rc = r;
    return rc == kOk;
  }
  // y[M, N] = x[M, K] · w[N, K]ᵀ (+ bias) (+ residual), as gemm and gemm_residual
  void product(const void* x, const void* w, const void* bias, const void* residual, void* y, int M, int N, int K) {
    if (rc != kOk) return;
    if (runs_rows(M, N, K)) {
      const long long ldw = K, ldy = N;
      ok(ttb_gemm_rows(x, K, M, K, 1, &w, &ldw, &N, &y, &ldy, bias == nullptr ? nullptr : &bias, residual, residual == nullptr ? 0 : N, 0, 1.f, st));
    } else if (const int splits = splits_of(M, N, K); splits > 1) {
      ok(ttb_gemm_bf16_splitk(x, w, split, y, M, N, K, 0, 0, K, K, N, 0, 0, bias, residual, residual == nullptr ? 0 : N, splits, 1.f, err, st));
    } else if (fills_pairs(M, N, K, sm_pairs())) {
      ok(residual == nullptr ? ttb_gemm_bf16_2sm(x, w, y, M, N, K, 0, 0, K, K, N, 0, bias, 1.f, err, st)
                             : ttb_gemm_bf16_2sm_residual(x, w, y, residual, M, N, K, 0, K, K, N, N, bias, err, st));
    } else if (ok(ttb_gemm_bf16(x, w, y, M, N, K, 0, 0, K, K, N, 0, 0, bias, 1.f, err, st)) && residual != nullptr) {
      const long long n = static_cast<long long>(M) * N / 8, blocks = (n + 255) / 256;
      TTB_COUNT_LAUNCH(1);
      add_kernel<<<static_cast<int>(blocks < 8ll * sm_count() ? blocks : 8ll * sm_count()), 256, 0, st>>>(static_cast<uint4*>(y), static_cast<const uint4*>(residual), n);
      ok(cudaGetLastError() == cudaSuccess ? kOk : kErrDriver);
    }
  }
};

static bool takes(const Sizes& z) {
  if (z.count <= 0 || z.b <= 0 || z.s <= 0 || z.hkv <= 0 || z.hq <= 0 || z.hq % z.hkv || (z.D != 64 && z.D != 128) || z.max_seq <= 0) return false;
  if (z.dim <= 0 || z.dim % 8 || z.dim > 16384 || z.hidden <= 0 || z.hidden % 8) return false;
  return static_cast<long long>(z.b) * z.s * (z.hidden > z.dim ? z.hidden : z.dim) < (1ll << 31) && z.b <= 65535;
}

}  // namespace layers
}  // namespace ttb

// What the rules above say of a product on a device of `pairs` SM pairs: rows, ranges, pairs, gated pairs.  No device is needed.
extern "C" void ttb_product_rules(int M, int N, int K, int pairs, int* out) {
  using namespace ttb::layers;
  out[0] = runs_rows(M, N, K), out[1] = splits_of(M, N, K), out[2] = fills_pairs(M, N, K, pairs), out[3] = gates_in_pairs(M, N, K, pairs);
}

// Bytes of workspace of a pass over b rows of s new tokens; 0 for sizes that it does not take.
extern "C" long long ttb_decoder_layers_workspace(int count, int b, int s, int dim, int hq, int hkv, int D, int hidden, int max_seq) {
  const ttb::layers::Sizes z{count, b, s, dim, hq, hkv, D, hidden, max_seq};
  return ttb::layers::takes(z) ? ttb::layers::Work(z).total : 0;
}

// h[b * s, dim] (embedded tokens; overwritten) through `count` layers and the final norm into y[b * s, dim].  `words`: per layer, in host memory, the addresses in
// struct Layer (biases may be 0); weights [rows, columns] contiguous, caches [>= b, max_seq, hkv, D], all 16-byte aligned.  pos int32 [b, s]; mask: nonzero byte =
// visible, row (b, i) at mask + b * mask_b + i * mask_r (mask_b 0: the same for all rows), max_seq bytes each.
extern "C" int ttb_decoder_layers(const long long* words, int count, int b, int s, int dim, int hq, int hkv, int D, int hidden, int max_seq, float eps, float scale, int interleaved, void* h,
                                  void* y, const void* norm, const int* pos, const void* mask, long long mask_b, long long mask_r, void* work, int* err, void* stream) {
  using namespace ttb;
  using namespace ttb::layers;
  const Sizes z{count, b, s, dim, hq, hkv, D, hidden, max_seq};
  if (!takes(z) || words == nullptr || scale <= 0.f) return kErrBadShape;
  const Work at(z);
  uint8_t* base = static_cast<uint8_t*>(work);
  auto part = [&](long long off) { return static_cast<void*>(base + off); };
  const int M = z.M(), nq = hq * D, nk = hkv * D;
  auto st = static_cast<cudaStream_t>(stream);
  Call c{static_cast<float*>(part(at.split)), err, st};
  float* rstd = static_cast<float*>(part(at.rstd));
  void *mid = part(at.mid), *xn = part(at.norm), *q = part(at.q), *k = part(at.k), *v = part(at.v), *rot = part(at.rot), *att = part(at.att), *act = part(at.act);
  int *lo = static_cast<int*>(part(at.lo)), *hi = static_cast<int*>(part(at.hi));
  const bool few = decodes(z), norms = ttb_gemm_rows_norms(M, dim) != 0;
  if (!few) c.ok(ttb_mask_bounds(mask, mask_b, mask_r, mask_b != 0 ? b : 1, s, max_seq, lo, hi, part(at.solid), st));
  for (int i = 0; i < count && c.rc == kOk; ++i) {
    const Layer& l = reinterpret_cast<const Layer*>(words)[i];
    const bool joined = runs_rows(M, nq, dim) && runs_rows(M, nk, dim), gated = runs_rows(M, hidden, dim);
    if (!(norms && joined)) c.ok(ttb_rmsnorm_fwd(h, l.sa_scale, xn, rstd, M, dim, eps, st));
    if (c.rc == kOk && joined) {
      const void *w[] = {l.wq, l.wk, l.wv}, *bias[] = {l.bq, l.bk, l.bv};
      void* out[] = {q, k, v};
      const long long ldw[] = {dim, dim, dim}, ldy[] = {nq, nk, nk};
      const int n[] = {nq, nk, nk};
      const bool biased = l.bq != nullptr || l.bk != nullptr || l.bv != nullptr;
      c.ok(norms ? ttb_gemm_rows_normed(h, dim, l.sa_scale, eps, M, dim, 3, w, ldw, n, out, ldy, biased ? bias : nullptr, st)
                 : ttb_gemm_rows(xn, dim, M, dim, 3, w, ldw, n, out, ldy, biased ? bias : nullptr, nullptr, 0, 0, 1.f, st));
    } else {
      c.product(xn, l.wq, l.bq, nullptr, q, M, nq, dim);
      c.product(xn, l.wk, l.bk, nullptr, k, M, nk, dim);
      c.product(xn, l.wv, l.bv, nullptr, v, M, nk, dim);
    }
    const int rope_len = static_cast<int>(l.rope_len);
    if (c.rc == kOk && few && s == 1) {
      c.ok(ttb_attn_decode_append(q, k, v, att, l.k_cache, l.v_cache, l.rope, pos, l.slots, mask, mask_b, b, max_seq, hq, hkv, D, interleaved, rope_len, scale, st));
    } else if (c.rc == kOk && c.ok(ttb_rope_append(q, k, v, rot, l.k_cache, l.v_cache, l.rope, pos, l.slots, M, hq, hkv, D, s, max_seq, interleaved, rope_len, st))) {
      c.ok(few ? ttb_attn_decode(rot, l.k_cache, l.v_cache, att, mask, mask_b, mask_r, nullptr, nullptr, b, s, max_seq, hq, hkv, D, scale, st)
               : ttb_attn_fwd2_masked(rot, l.k_cache, l.v_cache, att, static_cast<float*>(part(at.lse)), lo, hi, part(at.solid), mask_b != 0 ? s : 0, mask, mask_b, mask_r, b, s, max_seq, hq,
                                      hkv, D, scale, err, st));
    }
    c.product(att, l.wo, nullptr, h, mid, M, dim, nq);
    if (c.rc == kOk && !(norms && gated)) c.ok(ttb_rmsnorm_fwd(mid, l.mlp_scale, xn, rstd, M, dim, eps, st));
    if (c.rc != kOk) break;
    if (norms && gated) {
      c.ok(ttb_gemm_rows_gated_normed(mid, dim, l.mlp_scale, eps, l.w1, l.w3, dim, act, hidden, M, hidden, dim, st));
    } else if (gated) {
      c.ok(ttb_gemm_rows_gated(xn, dim, l.w1, l.w3, dim, act, hidden, M, hidden, dim, 0.f, 0.f, st));
    } else if (gates_in_pairs(M, hidden, dim, sm_pairs())) {
      c.ok(ttb_gemm_swiglu_bf16_2sm(xn, l.w1, l.w3, act, nullptr, nullptr, M, hidden, dim, dim, dim, hidden, 0.f, 0.f, err, st));
    } else {
      c.product(xn, l.w1, nullptr, nullptr, part(at.gate), M, hidden, dim);
      c.product(xn, l.w3, nullptr, nullptr, part(at.up), M, hidden, dim);
      if (c.rc == kOk) c.ok(ttb_swiglu_fwd(part(at.gate), part(at.up), act, M, hidden, hidden, hidden, hidden, st));
    }
    c.product(act, l.w2, nullptr, mid, h, M, dim, hidden);
  }
  if (c.rc == kOk) c.ok(ttb_rmsnorm_fwd(h, norm, y, rstd, M, dim, eps, st));
  return c.rc;
}
