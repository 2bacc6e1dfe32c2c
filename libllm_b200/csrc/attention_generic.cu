// Causal grouped-query attention over the paged cache, any head size up to 1,024 (values may
// have another width than keys, or be the first channels of the key rows themselves: v_ld), any number of heads and groups; optional sliding window,
// optional block mask (a query sees only keys of its own block of `block` positions, blocks
// counted from position 0), optionally the first `sink` positions of the sequence kept visible
// beyond the window (at their true positions), optional gate per (token, head) on the result (multiplied by
// sigmoid(gate)); element type float or bfloat16, arithmetic in 32-bit.  A CTA of four warps serves one (token, head): the
// warps take blocks of 32 keys in turn, lanes a key each for the scores, then 32 channels at a time for the
// weighted sum, with a running maximum and sum per warp (the online form of softmax,
// src/flint/cpu/softmax.cc:31-60); the four are joined in warp order.
//
// What bounds it is a warp's chain of loads, a few hundred keys long in a decoding step whose 64 or so (token, head) pairs
// leave most SMs without a warp: hence four warps to a pair, eight value rows asked for before the first is
// used, a key's place in the pages worked out once by the lane that scores it, and loops over
// channels no longer than the head (instantiations for heads up to 64, 128, 256 and 1,024).
// 32 heads of 64 over 8 key heads, two sequences of some 150 keys: 158 -> 17 us a launch (prompt and single tokens together).
//
// This is the attention of the true 32-bit path and of head sizes the fast bfloat16
// kernels do not take.  It serves prompts and single tokens alike: the keys of the
// step's own tokens are already in the cache when it runs, and the token at position p
// reads keys 0..p (or the last `window` of them), which is the bottom-right aligned
// causal mask of the reference (src/flint/operators.cc:119-124).  Head h reads
// key/value head h / (heads / kv_heads) (src/flint/operators.cc:43-56); scores are
// scaled by 1/sqrt(d) (src/flint/operators.cc:115-117).
//
// A token's result depends only on its own sequence: the order of additions is fixed by
// the position, not by the batch.
#include "common.cuh"
#include <math.h>

LLM_DEFINE_LAST_ERROR(llm_attention_generic_last_error)

constexpr int WARPS = 4;
constexpr int MAX_D_LARGE = 1024;

__device__ __forceinline__ float dot_row(const float *q, const float *k, int d, bool vec) {
  float acc = 0.f;
  if (!vec) {
    for (int c = 0; c < d; ++c) acc = fmaf(q[c], k[c], acc);
    return acc;
  }
#pragma unroll 4
  for (int c = 0; c < d; c += 4) {
    const float4 v = *reinterpret_cast<const float4 *>(k + c);
    acc = fmaf(q[c], v.x, acc);
    acc = fmaf(q[c + 1], v.y, acc);
    acc = fmaf(q[c + 2], v.z, acc);
    acc = fmaf(q[c + 3], v.w, acc);
  }
  return acc;
}
__device__ __forceinline__ float dot_row(const float *q, const __nv_bfloat16 *k, int d, bool vec) {
  float acc = 0.f;
  if (!vec) {
    for (int c = 0; c < d; ++c) acc = fmaf(q[c], __bfloat162float(k[c]), acc);
    return acc;
  }
#pragma unroll 2
  for (int c = 0; c < d; c += 8) {
    const uint4 raw = *reinterpret_cast<const uint4 *>(k + c);
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      acc = fmaf(q[c + 2 * i], f.x, acc);
      acc = fmaf(q[c + 2 * i + 1], f.y, acc);
    }
  }
  return acc;
}

// Weights that stand for themselves instead of a softmax's (SIG): a visible key's weight is sigmoid(cap tanh(temp s / cap) + bias)
// with a temperature and a bias per head (cap 0: no bound); the result is multiplied by out_scale.
struct SigmoidWeights {
  const float *temp, *bias;
  float cap, out_scale;
};

template <typename T, int MAX_D, bool SIG>
__global__ void __launch_bounds__(WARPS * 32)
attention_generic_kernel(const T *q, long long q_stride, T *__restrict__ out,
                         long long out_stride, const T *kcache,
                         const T *vcache, const int *tok_seq,
                         const int *tok_pos, const int *page_table,
                         int pt_stride, int n_heads, int n_kv, int d, int dv, int page_size,
                         int window, int block, int sink, float scale, const float *gate,
                         long long gate_stride, int vec, int v_ld, float null_score, const float *__restrict__ null_scores,
                         SigmoidWeights sig) {
  __shared__ __align__(16) float q_s[MAX_D];
  __shared__ float acc_s[WARPS][MAX_D];
  __shared__ float m_s[WARPS], l_s[WARPS];
  constexpr int NI = MAX_D / 32, AHEAD = MAX_D <= 256 ? 8 : 2;     // value rows on their way at once
  grid_dependents_launch();
  grid_dependency_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int token = (int)(blockIdx.x / (unsigned)n_heads), h = (int)(blockIdx.x % (unsigned)n_heads);
  const int p = tok_pos[token];
  const int *pt = page_table + (size_t)tok_seq[token] * pt_stride;
  const int kvh = h / (n_heads / n_kv);
  const T *qrow = q + (size_t)token * q_stride + (size_t)h * d;
  for (int c = threadIdx.x; c < d; c += WARPS * 32) q_s[c] = to_float(qrow[c]);
  __syncthreads();

  int kstart = window > 0 ? max(0, p - window + 1) : 0;
  if (block > 0) kstart = max(kstart, p / block * block);
  float m = -INFINITY, l = 0.f;
  const float temp = SIG ? sig.temp[h] : 0.f, bias = SIG ? sig.bias[h] : 0.f;
  float acc[NI];
#pragma unroll
  for (int i = 0; i < NI; ++i) acc[i] = 0.f;

  // two runs of keys: the kept first positions that lie before the window, then the window
  const int sink_end = (window > 0 && block == 0) ? min(sink, kstart) : 0;
  for (int run = sink_end > 0 ? 0 : 1; run < 2; ++run) {
    const int k0 = run == 0 ? 0 : kstart, k1 = run == 0 ? sink_end : p + 1;
    for (int kb = k0 + warp * 32; kb < k1; kb += WARPS * 32) {
      const int j = min(kb + lane, k1 - 1);
      const bool valid = kb + lane < k1;
      const long long at = ((long long)pt[j / page_size] * n_kv + kvh) * page_size + j % page_size;   // this lane's key's row
      float s = -INFINITY;
      if (valid) s = dot_row(q_s, kcache + at * d, d, vec != 0) * scale;
      float pj;
      if (SIG) {
        s *= temp;
        if (sig.cap > 0.f) s = sig.cap * tanhf(s / sig.cap);
        pj = valid ? 1.f / (1.f + expf(-(s + bias))) : 0.f;
      } else {
        // minus infinity while this warp has met no other score (a product that overflows): such keys weigh nothing, they are not NaN
        const float m_new = fmaxf(m, warp_max(s)), ref = m_new == -INFINITY ? 0.f : m_new;
        pj = valid ? expf(s - ref) : 0.f;
        const float alpha = expf(m - ref);                  // 0 on the first block (m = -inf)
        l = l * alpha + warp_sum(pj);
#pragma unroll
        for (int i = 0; i < NI; ++i) acc[i] *= alpha;
        m = m_new;
      }
      const int nvalid = min(32, k1 - kb);
      for (int j0 = 0; j0 < nvalid; j0 += AHEAD) {
        float v[AHEAD][NI];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          const T *vrow = vcache + __shfl_sync(0xffffffffu, at, j0 + u) * v_ld;       // beyond nvalid: the last key's row, not used
#pragma unroll
          for (int i = 0; i < NI; ++i) v[u][i] = lane + 32 * i < dv ? to_float(vrow[lane + 32 * i]) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          const float pv = __shfl_sync(0xffffffffu, pj, j0 + u);
          if (j0 + u < nvalid) {
#pragma unroll
            for (int i = 0; i < NI; ++i) acc[i] = fmaf(pv, v[u][i], acc[i]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) acc_s[warp][lane + 32 * i] = acc[i];
  if (lane == 0) {
    m_s[warp] = m;
    l_s[warp] = l;
  }
  __syncthreads();
  if (null_scores) null_score = null_scores[h];
  float top = -INFINITY;
  if (!SIG) {
#pragma unroll
    for (int w = 0; w < WARPS; ++w) top = fmaxf(top, m_s[w]);
    top = fmaxf(top, null_score);           // one more key whose score is null_score and whose value is nought, if above -inf
  }
  float f[WARPS], sum = !SIG && null_score > -INFINITY ? expf(null_score - top) : 0.f;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    f[w] = SIG ? 1.f : m_s[w] == -INFINITY ? 0.f : expf(m_s[w] - top);
    sum += l_s[w] * f[w];
  }
  float inv = SIG ? sig.out_scale : 1.f / sum;
  if (gate) inv *= 1.f / (1.f + expf(-gate[(size_t)token * gate_stride + h]));
  T *orow = out + (size_t)token * out_stride + (size_t)h * dv;
  for (int c = threadIdx.x; c < dv; c += WARPS * 32) {
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) o = fmaf(acc_s[w][c], f[w], o);
    orow[c] = from_float<T>(o * inv);
  }
}

// v_ld: channels between two value rows of the value storage (dv for a storage of its own; the key rows' width
// when the values are the first dv channels of the keys and vcache is kcache).
static int launch_generic(int dtype, const void *q, long long q_stride, void *out,
                          long long out_stride, const void *kcache, const void *vcache,
                          const int *tok_seq, const int *tok_pos, const int *page_table,
                          int pt_stride, int n_tokens, int n_heads, int n_kv, int d, int dv, int v_ld,
                          int page_size, int window, int block, int sink, float scale, const float *gate,
                          long long gate_stride, float null_score, const float *null_scores, const SigmoidWeights *sig,
                          cudaStream_t stream) {
  if (n_tokens == 0) return LLM_OK;
  LLM_REQUIRE(n_tokens > 0 && n_heads > 0 && n_kv > 0 && n_heads % n_kv == 0, "attention: bad head counts %d/%d", n_heads, n_kv);
  LLM_REQUIRE(d > 0 && d <= MAX_D_LARGE && dv > 0 && dv <= MAX_D_LARGE, "attention: head sizes %d / %d are not supported (up to %d)", d, dv,
              MAX_D_LARGE);
  LLM_REQUIRE(v_ld >= dv, "attention: value rows of %d channels in a storage of %d a row", dv, v_ld);
  LLM_REQUIRE(window >= 0 && block >= 0 && sink >= 0, "attention: bad window, block or number of kept first positions");
  LLM_REQUIRE(sink == 0 || block == 0, "attention: kept first positions go with a window, not with a block mask");
  // 16-byte loads of key rows where rows start on such a boundary
  const int vec = (dtype == LLM_F32 ? d % 4 == 0 : d % 8 == 0) && (uintptr_t)kcache % 16 == 0;
  // a CTA to a (token, head): launches of as many tokens as a grid has room for
  const int tokens = n_tokens < 2147483647LL / n_heads ? n_tokens : (int)(2147483647LL / n_heads);
  LLM_REQUIRE(((long long)n_tokens * n_heads + WARPS - 1) / WARPS < 2147483647LL, "attention: too many tokens");
  const int widest = d > dv ? d : dv;
  const SigmoidWeights sw = sig ? *sig : SigmoidWeights{};
#define GENERIC_RUN(T, MAXD, SIG)                                                                                        \
  for (long long t0 = 0; t0 < n_tokens; t0 += tokens)                                                                     \
    LLM_CHECK_CUDA(llm_launch(attention_generic_kernel<T, MAXD, SIG>, dim3((unsigned)((n_tokens - t0 < tokens ? n_tokens - t0 : tokens) * n_heads)), \
                              dim3(WARPS * 32), 0, stream, (const T *)q + t0 * q_stride, q_stride, (T *)out + t0 * out_stride, out_stride,     \
                              (const T *)kcache, (const T *)vcache, tok_seq + t0, tok_pos + t0, page_table, pt_stride, n_heads, n_kv, d, dv,  \
                              page_size, window, block, sink, scale, gate ? gate + t0 * gate_stride : gate, gate_stride, vec, v_ld, null_score, \
                              null_scores, sw),                                                                           \
                   "attention_generic")
#define GENERIC_GO(T, MAXD)                                                                                              \
  do {                                                                                                                   \
    if (sig) GENERIC_RUN(T, MAXD, true);                                                                                 \
    else GENERIC_RUN(T, MAXD, false);                                                                                    \
    return LLM_OK;                                                                                                       \
  } while (0)
#define GENERIC_TYPE(T)                                                                                                  \
  do {                                                                                                                   \
    if (widest <= 64) GENERIC_GO(T, 64);                                                                                 \
    if (widest <= 128) GENERIC_GO(T, 128);                                                                               \
    if (widest <= 256) GENERIC_GO(T, 256);                                                                               \
    GENERIC_GO(T, MAX_D_LARGE);                                                                                          \
  } while (0)
  if (dtype == LLM_F32) GENERIC_TYPE(float);
  if (dtype == LLM_BF16) GENERIC_TYPE(__nv_bfloat16);
  LLM_FAIL("attention: unknown dtype %d", dtype);
#undef GENERIC_TYPE
#undef GENERIC_GO
#undef GENERIC_RUN
}

LLM_EXPORT int llm_attention_generic_ld(int dtype, const void *q, long long q_stride, void *out,
                                        long long out_stride, const void *kcache, const void *vcache,
                                        const int *tok_seq, const int *tok_pos, const int *page_table,
                                        int pt_stride, int n_tokens, int n_heads, int n_kv, int d, int dv, int v_ld,
                                        int page_size, int window, int block, int sink, float scale, const float *gate,
                                        long long gate_stride, float null_score, cudaStream_t stream) {
  return launch_generic(dtype, q, q_stride, out, out_stride, kcache, vcache, tok_seq, tok_pos, page_table, pt_stride, n_tokens, n_heads,
                        n_kv, d, dv, v_ld, page_size, window, block, sink, scale, gate, gate_stride, null_score, nullptr, nullptr, stream);
}

// The same with a null score per head (32-bit, device; null: none).
LLM_EXPORT int llm_attention_generic_sinks(int dtype, const void *q, long long q_stride, void *out, long long out_stride,
                                           const void *kcache, const void *vcache, const int *tok_seq, const int *tok_pos,
                                           const int *page_table, int pt_stride, int n_tokens, int n_heads, int n_kv, int d, int dv,
                                           int v_ld, int page_size, int window, int block, int sink, float scale, const float *gate,
                                           long long gate_stride, float null_score, const float *null_scores, cudaStream_t stream) {
  return launch_generic(dtype, q, q_stride, out, out_stride, kcache, vcache, tok_seq, tok_pos, page_table, pt_stride, n_tokens, n_heads,
                        n_kv, d, dv, v_ld, page_size, window, block, sink, scale, gate, gate_stride, null_score, null_scores, nullptr,
                        stream);
}

// The weights of SigmoidWeights instead of a softmax's.
LLM_EXPORT int llm_attention_generic_sigmoid(int dtype, const void *q, long long q_stride, void *out, long long out_stride,
                                             const void *kcache, const void *vcache, const int *tok_seq, const int *tok_pos,
                                             const int *page_table, int pt_stride, int n_tokens, int n_heads, int n_kv, int d, int dv,
                                             int page_size, int window, float scale, const float *temp, const float *bias, float cap,
                                             float out_scale, cudaStream_t stream) {
  LLM_REQUIRE(temp && bias && cap >= 0.f, "attention: sigmoid weights need a temperature and a bias per head");
  const SigmoidWeights sig{temp, bias, cap, out_scale};
  return launch_generic(dtype, q, q_stride, out, out_stride, kcache, vcache, tok_seq, tok_pos, page_table, pt_stride, n_tokens, n_heads,
                        n_kv, d, dv, dv, page_size, window, 0, 0, scale, nullptr, 0, -INFINITY, nullptr, &sig, stream);
}

LLM_EXPORT int llm_attention_generic(int dtype, const void *q, long long q_stride, void *out,
                                     long long out_stride, const void *kcache, const void *vcache,
                                     const int *tok_seq, const int *tok_pos, const int *page_table,
                                     int pt_stride, int n_tokens, int n_heads, int n_kv, int d, int dv,
                                     int page_size, int window, int block, int sink, float scale, const float *gate,
                                     long long gate_stride, cudaStream_t stream) {
  return llm_attention_generic_ld(dtype, q, q_stride, out, out_stride, kcache, vcache, tok_seq, tok_pos, page_table, pt_stride,
                                  n_tokens, n_heads, n_kv, d, dv, dv, page_size, window, block, sink, scale, gate, gate_stride, -INFINITY, stream);
}
