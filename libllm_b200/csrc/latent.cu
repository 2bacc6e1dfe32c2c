// Kernels of latent attention: keys and values of all heads are functions of one cached vector
// per position, c (kv_rank channels, RMS-normed), plus one rotated key part (rot_dim channels)
// that all heads share.  A head's unrotated key is W_uk c and its value W_uv c, so
//   score = q_n . (W_uk c) + q_r . k_r = (W_uk^T q_n) . c + q_r . k_r
//   head  = sum_j p_j W_uv c_j        = W_uv (sum_j p_j c_j)
// and attention runs over the cached rows [c | k_r] themselves, as one key/value head that every
// query head reads: the query is [W_uk^T q_n | q_r] (kv_rank + rot_dim channels), the values are
// the first kv_rank channels of the key rows, and the head's result is expanded by W_uv after.
// Here: the placement of a step's tokens (both latents' norms, the rotation, the append to the
// cache), the queries' absorption of W_uk, and the expansion of the heads' results by W_uv.  The
// attention itself is attention_generic.cu (value rows with the key rows' stride).  No
// counterpart in the reference, whose one mixer caches keys and values per head
// (src/libllm/llama.cc:178-225).
//
// 32-bit: norms (sums over the product's 32-bit result), rotation, every accumulation.
#include "common.cuh"
#include <math.h>
#include <algorithm>

LLM_DEFINE_LAST_ERROR(llm_latent_last_error)

// One pair of a rotation table row: cs = [cosines (rot/2) | sines (rot/2)]; pair i is channels (2i, 2i + 1) when
// interleaved, (i, i + rot/2) otherwise.  (u, v) -> (u cos - v sin, v cos + u sin).
__device__ __forceinline__ void rotate_pair(const float *x, const float *cs, int rot, int i, int interleaved, int *ca, int *cb, float *ra,
                                            float *rb) {
  const int half = rot / 2;
  const int a = interleaved ? 2 * i : i, b = interleaved ? 2 * i + 1 : i + half;
  const float u = x[a], v = x[b], c = cs[i], s = cs[half + i];
  *ca = a, *cb = b;
  *ra = u * c - v * s;
  *rb = v * c + u * s;
}

// ---------------------------------------------------------------- placement
// proj rows (32-bit): the query latent (q_rank values at off_q; q_rank 0: none) and, when the run has a latent projection of
// its own (off_kv >= 0), kv_rank + rot_dim values at off_kv.  cq_out = rms(query latent) * q_weight in the
// engine's type; cache row of the token = [rms(first kv_rank) * kv_weight | rotated last rot_dim].
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS)
latent_place_kernel(const float *proj, long long ld, int off_q, int q_rank, const float *__restrict__ q_weight,
                    T *__restrict__ cq_out, long long ldq, int off_kv, int kv_rank, int rot, const float *__restrict__ kv_weight,
                    float eps, const float *__restrict__ table, int table_rows, int interleaved, const int *tok_seq,
                    const int *tok_pos, const int *page_table, int pt_stride, T *__restrict__ cache,
                    int page_size) {
  __shared__ float scratch[THREADS / 32 + 1];
  grid_dependents_launch();
  grid_dependency_wait();
  const int t = blockIdx.x;
  const float *row = proj + (size_t)t * ld;
  if (q_rank > 0) {
    float ss = 0.f;
    for (int c = threadIdx.x; c < q_rank; c += THREADS) ss = fmaf(row[off_q + c], row[off_q + c], ss);
    const float inv = rsqrtf(block_sum<THREADS>(ss, scratch) / (float)q_rank + eps);
    for (int c = threadIdx.x; c < q_rank; c += THREADS) cq_out[(size_t)t * ldq + c] = from_float<T>(row[off_q + c] * inv * q_weight[c]);
  }
  if (off_kv < 0) return;
  const int pos = tok_pos[t];
  const int page = page_table[(size_t)tok_seq[t] * pt_stride + pos / page_size];
  T *dst = cache + ((size_t)page * page_size + (pos % page_size)) * (size_t)(kv_rank + rot);
  const float *kv = row + off_kv;
  float ss = 0.f;
  for (int c = threadIdx.x; c < kv_rank; c += THREADS) ss = fmaf(kv[c], kv[c], ss);
  const float inv = rsqrtf(block_sum<THREADS>(ss, scratch) / (float)kv_rank + eps);
  for (int c = threadIdx.x; c < kv_rank; c += THREADS) dst[c] = from_float<T>(kv[c] * inv * kv_weight[c]);
  const float *cs = table + (size_t)(pos < table_rows ? pos : table_rows - 1) * rot;
  for (int i = threadIdx.x; i < rot / 2; i += THREADS) {
    int a, b;
    float ra, rb;
    rotate_pair(kv + kv_rank, cs, rot, i, interleaved, &a, &b, &ra, &rb);
    dst[kv_rank + a] = from_float<T>(ra);
    dst[kv_rank + b] = from_float<T>(rb);
  }
}

LLM_EXPORT int llm_latent_place(int dtype, const float *proj, long long ld, int n_tokens, int off_q, int q_rank, const float *q_weight,
                                void *cq_out, long long ldq, int off_kv, int kv_rank, int rot, const float *kv_weight, float eps,
                                const float *table, int table_rows, int interleaved, const int *tok_seq, const int *tok_pos,
                                const int *page_table, int pt_stride, void *cache, int page_size, cudaStream_t stream) {
  if (n_tokens == 0) return LLM_OK;
  LLM_REQUIRE(n_tokens > 0 && q_rank >= 0 && off_q >= 0 && (q_rank == 0 || (q_weight && cq_out)), "latent_place: bad sizes");
  if (off_kv >= 0)
    LLM_REQUIRE(kv_rank > 0 && rot >= 0 && rot % 2 == 0 && kv_weight && cache && page_table && (rot == 0 || (table && table_rows > 0)),
                "latent_place: bad sizes of the key/value latent");
  constexpr int THREADS = 256;
  if (dtype == LLM_F32)
    llm_launch(latent_place_kernel<float, THREADS>, dim3(n_tokens), dim3(THREADS), 0, stream, proj, ld, off_q, q_rank, q_weight,
               (float *)cq_out, ldq, off_kv, kv_rank, rot, kv_weight, eps, table, table_rows, interleaved, tok_seq, tok_pos, page_table,
               pt_stride, (float *)cache, page_size);
  else if (dtype == LLM_BF16)
    llm_launch(latent_place_kernel<__nv_bfloat16, THREADS>, dim3(n_tokens), dim3(THREADS), 0, stream, proj, ld, off_q, q_rank, q_weight,
               (__nv_bfloat16 *)cq_out, ldq, off_kv, kv_rank, rot, kv_weight, eps, table, table_rows, interleaved, tok_seq, tok_pos,
               page_table, pt_stride, (__nv_bfloat16 *)cache, page_size);
  else LLM_FAIL("latent_place: unknown dtype %d", dtype);
  LLM_CHECK_LAUNCH("latent_place");
  return LLM_OK;
}

// ---------------------------------------------------------------- the queries take in W_uk
// q rows (32-bit) [heads, d + rot]: out[t, h] = [sum_i q[t, h, i] * w_uk[h * d + i, :] (kv_rank) | rotated q[t, h, d:] (rot)]
// in the engine's type.  A CTA takes one head and TT tokens: the tokens' unrotated parts lie in shared memory, a
// thread owns V neighbouring output channels and walks the head's d rows of w_uk (its neighbours read the neighbouring channels);
// the channels are shared out over blockIdx.z so that a step of few tokens still fills the device.
// What bounds a decoding step here is the chain of waits, not the 2 MB of w_uk: so the first rows of w_uk (64 in 16 bits: a whole head of
// 64) are in registers before the kernel before has finished, and no more tokens are multiplied than there are.  (With latent_expand
// and the decode kernel's loads below: two prompts and twelve tokens of a model with latent layers 14.82 -> 14.18 ms.)
constexpr int LAT_TT = 16;
template <typename T, int THREADS, int TT, int V>
__global__ void __launch_bounds__(THREADS)
latent_absorb_kernel(const float *q, long long ldq, const T *__restrict__ w_uk, T *__restrict__ out, long long ldo,
                     int n_tokens, int d, int rot, int kv_rank, const float *__restrict__ table, int table_rows, int interleaved,
                     const int *tok_pos) {
  extern __shared__ float qs[];                        // [TT][d]
  struct alignas(sizeof(T) * V) Piece { T v[V]; };
  constexpr int ROWS = sizeof(T) == 2 ? 64 : 32;       // rows of w_uk held at once
  grid_dependents_launch();
  const int t0 = blockIdx.x * TT, h = blockIdx.y;
  const int nt = min(TT, n_tokens - t0);
  const int c = (blockIdx.z * THREADS + threadIdx.x) * V;
  const T *w = w_uk + (size_t)h * d * kv_rank + (c < kv_rank ? c : 0);
  Piece held[ROWS];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) held[i] = *reinterpret_cast<const Piece *>(w + (size_t)min(i0 + i, d - 1) * kv_rank);
  };
  fetch(0);
  grid_dependency_wait();
  for (int i = threadIdx.x; i < TT * d; i += THREADS) {
    const int t = i / d, k = i - t * d;
    qs[i] = t < nt ? q[(size_t)(t0 + t) * ldq + (size_t)h * (d + rot) + k] : 0.f;
  }
  __syncthreads();
  float acc[TT][V];
#pragma unroll
  for (int t = 0; t < TT; ++t)
#pragma unroll
    for (int v = 0; v < V; ++v) acc[t][v] = 0.f;
  for (int i0 = 0; i0 < d; i0 += ROWS) {
    if (i0 > 0) fetch(i0);
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
      if (i0 + i < d) {
#pragma unroll
        for (int t = 0; t < TT; ++t)
#pragma unroll
          for (int v = 0; v < V; ++v) acc[t][v] = fmaf(qs[t * d + i0 + i], to_float(held[i].v[v]), acc[t][v]);
      }
  }
  if (c < kv_rank) {
#pragma unroll
    for (int t = 0; t < TT; ++t)
      if (t < nt) {
        T *dst = out + (size_t)(t0 + t) * ldo + (size_t)h * (kv_rank + rot) + c;
#pragma unroll
        for (int v = 0; v < V; ++v) dst[v] = from_float<T>(acc[t][v]);
      }
  }
  const int half = rot / 2;
  if (blockIdx.z != 0) return;
  for (int i = threadIdx.x; i < nt * half; i += THREADS) {
    const int t = i / half, pr = i - t * half;
    const int pos = tok_pos[t0 + t];
    const float *cs = table + (size_t)(pos < table_rows ? pos : table_rows - 1) * rot;
    int a, b;
    float ra, rb;
    rotate_pair(q + (size_t)(t0 + t) * ldq + (size_t)h * (d + rot) + d, cs, rot, pr, interleaved, &a, &b, &ra, &rb);
    T *dst = out + (size_t)(t0 + t) * ldo + (size_t)h * (kv_rank + rot) + kv_rank;
    dst[a] = from_float<T>(ra);
    dst[b] = from_float<T>(rb);
  }
}

LLM_EXPORT int llm_latent_absorb(int dtype, const float *q, long long ldq, const void *w_uk, void *out, long long ldo, int n_tokens,
                                 int n_heads, int d, int rot, int kv_rank, const float *table, int table_rows, int interleaved,
                                 const int *tok_pos, cudaStream_t stream) {
  if (n_tokens == 0) return LLM_OK;
  LLM_REQUIRE(n_tokens > 0 && n_heads > 0 && n_heads <= 65535 && d > 0 && kv_rank > 0 && rot >= 0 && rot % 2 == 0, "latent_absorb: bad sizes");
  LLM_REQUIRE(rot == 0 || (table && table_rows > 0), "latent_absorb: a rotation needs its table");
  constexpr int THREADS = 64;
  const int tt = n_tokens <= 1 ? 1 : n_tokens <= 2 ? 2 : n_tokens <= 4 ? 4 : n_tokens <= 8 ? 8 : LAT_TT;
  const size_t smem = (size_t)tt * d * sizeof(float);
  LLM_REQUIRE((size_t)LAT_TT * d * sizeof(float) <= 96 * 1024, "latent_absorb: heads of %d channels are not supported", d);
  // two channels to a thread where rows of w_uk start on their boundary
  const int v = kv_rank % 2 == 0 && (uintptr_t)w_uk % (dtype == LLM_F32 ? 8 : 4) == 0 ? 2 : 1;
  const dim3 grid((n_tokens + tt - 1) / tt, n_heads, (kv_rank + THREADS * v - 1) / (THREADS * v));
#define ABSORB_GO(T, TT, V)                                                                                                  \
  do {                                                                                                                       \
    LLM_CHECK_CUDA(llm_allow_smem(latent_absorb_kernel<T, THREADS, TT, V>, smem), "latent_absorb attribute");                 \
    llm_launch(latent_absorb_kernel<T, THREADS, TT, V>, grid, dim3(THREADS), smem, stream, q, ldq, (const T *)w_uk, (T *)out, ldo, \
               n_tokens, d, rot, kv_rank, table, table_rows, interleaved, tok_pos);                                          \
  } while (0)
#define ABSORB_TYPE(T, V)                                                                                                    \
  do {                                                                                                                       \
    if (tt == 1) ABSORB_GO(T, 1, V);                                                                                         \
    else if (tt == 2) ABSORB_GO(T, 2, V);                                                                                    \
    else if (tt == 4) ABSORB_GO(T, 4, V);                                                                                    \
    else if (tt == 8) ABSORB_GO(T, 8, V);                                                                                    \
    else ABSORB_GO(T, LAT_TT, V);                                                                                            \
  } while (0)
  if (dtype == LLM_F32 && v == 2) ABSORB_TYPE(float, 2);
  else if (dtype == LLM_F32) ABSORB_TYPE(float, 1);
  else if (dtype == LLM_BF16 && v == 2) ABSORB_TYPE(__nv_bfloat16, 2);
  else if (dtype == LLM_BF16) ABSORB_TYPE(__nv_bfloat16, 1);
  else LLM_FAIL("latent_absorb: unknown dtype %d", dtype);
#undef ABSORB_TYPE
#undef ABSORB_GO
  LLM_CHECK_LAUNCH("latent_absorb");
  return LLM_OK;
}

// ---------------------------------------------------------------- the heads' results are expanded by W_uv
// x [tokens, heads, kv_rank] (the weighted sums of cached latents), w_uv [heads * dv, kv_rank]:
// out[t, h, j] = sum_c x[t, h, c] * w_uv[h * dv + j, c].  A CTA takes one head and TT tokens; a warp owns output
// channels, its lanes walk a row of w_uv together (in lane order, then the shuffle tree); blockIdx.z shares the
// output channels out, eight to a CTA.  `gate` (32-bit, one value per token and head, rows gate_stride apart; null: none): the
// head's result is multiplied by sigmoid(gate).
// As above: sixteen pieces of the row (a whole latent of 512) are on their way before the dependency is waited for, and a CTA takes
// ET tokens, no more than there are.
constexpr int LAT_ET = 8;
template <typename T, int THREADS, int ET>
__global__ void __launch_bounds__(THREADS)
latent_expand_kernel(const T *x, long long ldx, const T *__restrict__ w_uv, T *__restrict__ out, long long ldo, int n_tokens,
                     int kv_rank, int dv, const float *gate, long long gate_stride) {
  extern __shared__ float xs[];                        // [ET][kv_rank]
  constexpr int HELD = 16;
  grid_dependents_launch();
  const int t0 = blockIdx.x * ET, h = blockIdx.y;
  const int nt = min(ET, n_tokens - t0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float held[HELD];
  auto fetch = [&](int j, int c0) {
    const T *w = w_uv + ((size_t)h * dv + j) * kv_rank;
#pragma unroll
    for (int i = 0; i < HELD; ++i) held[i] = c0 + i * 32 + lane < kv_rank ? to_float(w[c0 + i * 32 + lane]) : 0.f;
  };
  const int j0 = blockIdx.z * (THREADS / 32) + warp;
  if (j0 < dv) fetch(j0, 0);
  grid_dependency_wait();
  for (int i = threadIdx.x; i < ET * kv_rank; i += THREADS) {
    const int t = i / kv_rank, c = i - t * kv_rank;
    xs[i] = t < nt ? to_float(x[(size_t)(t0 + t) * ldx + (size_t)h * kv_rank + c]) : 0.f;
  }
  __syncthreads();
  for (int j = j0; j < dv; j += THREADS / 32 * gridDim.z) {
    float acc[ET];
#pragma unroll
    for (int t = 0; t < ET; ++t) acc[t] = 0.f;
    for (int c0 = 0; c0 < kv_rank; c0 += 32 * HELD) {
      if (j != j0 || c0 > 0) fetch(j, c0);
#pragma unroll
      for (int i = 0; i < HELD; ++i) {
        const int c = c0 + i * 32 + lane;
        if (c < kv_rank) {
#pragma unroll
          for (int t = 0; t < ET; ++t) acc[t] = fmaf(xs[t * kv_rank + c], held[i], acc[t]);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < ET; ++t) {
      float s = warp_sum(acc[t]);
      if (gate && t < nt) s *= 1.f / (1.f + expf(-gate[(size_t)(t0 + t) * gate_stride + h]));
      if (lane == 0 && t < nt) out[(size_t)(t0 + t) * ldo + (size_t)h * dv + j] = from_float<T>(s);
    }
  }
}

LLM_EXPORT int llm_latent_expand_gated(int dtype, const void *x, long long ldx, const void *w_uv, void *out, long long ldo, int n_tokens,
                                       int n_heads, int kv_rank, int dv, const float *gate, long long gate_stride, cudaStream_t stream) {
  if (n_tokens == 0) return LLM_OK;
  LLM_REQUIRE(n_tokens > 0 && n_heads > 0 && n_heads <= 65535 && kv_rank > 0 && dv > 0, "latent_expand: bad sizes");
  constexpr int THREADS = 256;
  const int et = n_tokens <= 1 ? 1 : n_tokens <= 2 ? 2 : n_tokens <= 4 ? 4 : LAT_ET;
  const size_t smem = (size_t)et * kv_rank * sizeof(float);
  LLM_REQUIRE((size_t)LAT_ET * kv_rank * sizeof(float) <= 96 * 1024, "latent_expand: a latent of %d channels is not supported", kv_rank);
  const dim3 grid((n_tokens + et - 1) / et, n_heads, std::min(64, (dv + THREADS / 32 - 1) / (THREADS / 32)));
#define EXPAND_GO(T, ET)                                                                                                  \
  do {                                                                                                                    \
    LLM_CHECK_CUDA(llm_allow_smem(latent_expand_kernel<T, THREADS, ET>, smem), "latent_expand attribute");                 \
    llm_launch(latent_expand_kernel<T, THREADS, ET>, grid, dim3(THREADS), smem, stream, (const T *)x, ldx, (const T *)w_uv, \
               (T *)out, ldo, n_tokens, kv_rank, dv, gate, gate_stride);                                                  \
  } while (0)
#define EXPAND_TYPE(T)                                                                                                    \
  do {                                                                                                                    \
    if (et == 1) EXPAND_GO(T, 1);                                                                                         \
    else if (et == 2) EXPAND_GO(T, 2);                                                                                    \
    else if (et == 4) EXPAND_GO(T, 4);                                                                                    \
    else EXPAND_GO(T, LAT_ET);                                                                                            \
  } while (0)
  if (dtype == LLM_F32) EXPAND_TYPE(float);
  else if (dtype == LLM_BF16) EXPAND_TYPE(__nv_bfloat16);
  else LLM_FAIL("latent_expand: unknown dtype %d", dtype);
#undef EXPAND_TYPE
#undef EXPAND_GO
  LLM_CHECK_LAUNCH("latent_expand");
  return LLM_OK;
}

LLM_EXPORT int llm_latent_expand(int dtype, const void *x, long long ldx, const void *w_uv, void *out, long long ldo, int n_tokens,
                                 int n_heads, int kv_rank, int dv, cudaStream_t stream) {
  return llm_latent_expand_gated(dtype, x, ldx, w_uv, out, ldo, n_tokens, n_heads, kv_rank, dv, nullptr, 0, stream);
}
