// Plain matrix product C[M,N] = A[M,K] * W[N,K]^T (+ bias) on the CUDA cores, 32-bit
// accumulate.  This is the matrix product of the true 32-bit path (no tensor cores, no
// reduced-precision mode) and the yardstick the fast bfloat16 products are tested
// against.  The order in which an output's K products are added is fixed by K alone, so a row's
// result does not depend on how many rows the call has or on where the row lies in the batch:
// 32-bit operands whose rows start on 16 bytes are added in eight parts of K (runs of whole
// blocks of 32), in each the even and the odd k by an accumulator each, ascending, and the parts in order;
// everything else in the order k = 0, 1, 2, ... with one accumulator.
//
// Reference counterpart: the fp32 GEMM of the CPU backend (src/flint/cpu/matmul.cc:56-259)
// and cublasGemmEx with CUBLAS_COMPUTE_32F on CUDA (src/flint/cuda/gemm_cublas.cc:160-197).
#include "common.cuh"

LLM_DEFINE_LAST_ERROR(llm_gemm_plain_last_error)

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

// ---------------------------------------------------------------- 32-bit operands, rows on 16 bytes
constexpr int PARTS = 8, PART_BLOCK = 32;      // parts of K, each a run of whole blocks of 32

__device__ __forceinline__ int part_length(int K) { return ((K + PART_BLOCK - 1) / PART_BLOCK + PARTS - 1) / PARTS * PART_BLOCK; }
// 16 bytes to shared memory, zeros where `in` does not hold (the address is then not read)
__device__ __forceinline__ void copy16(float *dst, const float *src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Two products added to two sums in one instruction: the packed form, with which the loops below spend their issue slots on
// half as many multiplications as one value at a time would need.
__device__ __forceinline__ void fma_pair(unsigned long long &acc, unsigned long long a, unsigned long long w) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(w));
}
__device__ __forceinline__ float add_pair(unsigned long long acc) {
  return __uint_as_float((unsigned)acc) + __uint_as_float((unsigned)(acc >> 32));
}
__device__ __forceinline__ ulonglong2 ld_pairs(const float *p) { return *reinterpret_cast<const ulonglong2 *>(p); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Few rows of A (single-token steps; MT of them to a blockIdx.y): bound by the stream of W.  A CTA takes 16 rows of W, two
// parts of K to each of its four warps and a lane to each (row of W, part), so that a matrix of 2,048 rows still gives
// 128 CTAs and an output's chain of additions is an eighth of K long.  A warp fills a ring of its own
// (128 bytes of each row and part a stage, 16-byte asynchronous copies), so no barrier is met
// before the parts are added.  A row's pitch of 36 floats spreads eight lanes' 16-byte reads over all banks.
// W does not depend on the kernel before and is on its way before that has finished.
// [2, 2,048] x [16,384, 2,048]^T: 285 -> 31 us (4.4 TB/s of W); [2, 8,192] x [2,048, 8,192]^T: 927 -> 20 us.
template <int MT>
struct FewShape {
  static constexpr int PITCH = PART_BLOCK + 4;
  static constexpr int W_FLOATS = 2 * 16 * PITCH, A_FLOATS = 2 * MT * PITCH;      // a warp's stage: two parts
  static constexpr int STAGES = 5;
  static constexpr size_t SMEM = (size_t)STAGES * 4 * (W_FLOATS + A_FLOATS) * sizeof(float);
};
template <int MT>
__global__ void __launch_bounds__(128)
gemm_few_kernel(const float *A, long long lda, const float *__restrict__ W, long long ldw,
                const float *__restrict__ bias, float *__restrict__ C, long long ldc, int M, int N, int K) {
  using S = FewShape<MT>;
  constexpr int PITCH = S::PITCH, STAGES = S::STAGES;
  extern __shared__ __align__(16) float smem[];
  grid_dependents_launch();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = blockIdx.x * 16;
  const int plen = part_length(K);
  A += (size_t)blockIdx.y * MT * lda;
  C += (size_t)blockIdx.y * MT * ldc;
  M = min(M - (int)blockIdx.y * MT, MT);
  float *ring = smem + (size_t)warp * STAGES * (S::W_FLOATS + S::A_FLOATS);
  const int n_blocks = plen / PART_BLOCK;
  auto load_w = [&](int blk, int stage) {
    float *dst = ring + (size_t)stage * (S::W_FLOATS + S::A_FLOATS);
#pragma unroll
    for (int i = 0; i < 8; ++i) {                       // 2 parts x 16 rows x 8 pieces of 16 bytes
      const int e = i * 32 + lane, piece = e & 7, row = (e >> 3) & 15, half = e >> 7;
      const int k0 = (warp * 2 + half) * plen, k = k0 + blk * PART_BLOCK + piece * 4;
      const bool in = k < K && n0 + row < N;
      copy16(dst + (half * 16 + row) * PITCH + piece * 4, in ? W + (size_t)(n0 + row) * ldw + k : W, in);
    }
  };
  auto load_a = [&](int blk, int stage) {
    float *dst = ring + (size_t)stage * (S::W_FLOATS + S::A_FLOATS) + S::W_FLOATS;
#pragma unroll
    for (int e = lane; e < 2 * MT * 8; e += 32) {
      const int piece = e & 7, row = (e >> 3) % MT, half = (e >> 3) / MT;
      const int k = (warp * 2 + half) * plen + blk * PART_BLOCK + piece * 4;
      const bool in = k < K && row < M;
      copy16(dst + (half * MT + row) * PITCH + piece * 4, in ? A + (size_t)row * lda + k : A, in);
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s)
    if (s < n_blocks) load_w(s, s);
  grid_dependency_wait();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < n_blocks) load_a(s, s);
    copy_commit();
  }
  unsigned long long acc[MT];                           // sums over even and odd k
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m] = 0ull;
  const int row = lane & 15, half = lane >> 4;
  for (int blk = 0; blk < n_blocks; ++blk) {
    copy_wait<STAGES - 2>();
    __syncwarp();
    {                                                   // the stage that was read in the round before
      const int ahead = blk + STAGES - 1;
      if (ahead < n_blocks) {
        load_w(ahead, ahead % STAGES);
        load_a(ahead, ahead % STAGES);
      }
      copy_commit();
    }
    const float *st = ring + (size_t)(blk % STAGES) * (S::W_FLOATS + S::A_FLOATS);
    const float *sw = st + (half * 16 + row) * PITCH, *sa = st + S::W_FLOATS + half * MT * PITCH;
#pragma unroll
    for (int k4 = 0; k4 < PART_BLOCK; k4 += 4) {
      const ulonglong2 w = ld_pairs(sw + k4);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const ulonglong2 a = ld_pairs(sa + m * PITCH + k4);
        fma_pair(acc[m], a.x, w.x);
        fma_pair(acc[m], a.y, w.y);
      }
    }
  }
  copy_wait<0>();
  __syncthreads();
  float *red = smem;                                    // [PARTS][MT][16], over the rings
#pragma unroll
  for (int m = 0; m < MT; ++m) red[((warp * 2 + half) * MT + m) * 16 + row] = add_pair(acc[m]);
  __syncthreads();
  for (int e = threadIdx.x; e < MT * 16; e += 128) {
    const int m = e / 16, r = e % 16;
    if (m >= M || n0 + r >= N) continue;
    float v = red[m * 16 + r];
#pragma unroll
    for (int p = 1; p < PARTS; ++p) v += red[(p * MT + m) * 16 + r];
    if (bias) v += bias[n0 + r];
    C[(size_t)m * ldc + n0 + r] = v;
  }
}

// More rows of A: bound by the FMA pipe.  A CTA of eight warps computes 32 x 64 outputs, each warp the
// whole tile over its own part of K from a ring of its own (no barriers), a lane 8 x 8 outputs: 16 reads of
// 16 bytes for 128 packed multiplications and additions; and matrices of 2,048 rows, whose tiles alone would not
// fill the SMs with warps, do.  Lanes take every fourth row of A and every eighth of W: with a pitch of 20 floats their reads meet no
// bank twice.  [213, 2,048] x [16,384, 2,048]^T: 780 -> 416 us (34 TFLOP/s; tiles of 64 x 64 with single
// multiplications 463).
struct TileShape {
  static constexpr int RM = 32, KS = 16, PITCH = KS + 4;
  static constexpr int STAGES = 3;
  static constexpr int FLOATS = (RM + 64) * PITCH;
  static constexpr size_t RING = (size_t)PARTS * STAGES * FLOATS * sizeof(float), SUMS = (size_t)PARTS * RM * 64 * sizeof(float);
  static constexpr size_t SMEM = RING > SUMS ? RING : SUMS;
};
__global__ void __launch_bounds__(256, 1)
gemm_tile_kernel(const float *A, long long lda, const float *__restrict__ W, long long ldw,
                 const float *__restrict__ bias, float *__restrict__ C, long long ldc, int M, int N, int K) {
  using S = TileShape;
  constexpr int RM = S::RM, PITCH = S::PITCH, KS = S::KS, STAGES = S::STAGES, LM = RM / 4;
  extern __shared__ __align__(16) float smem[];
  grid_dependents_launch();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m0 = blockIdx.y * RM, n0 = blockIdx.x * 64;
  const int plen = part_length(K), k0 = warp * plen, k1 = min(K, k0 + plen);
  const int n_blocks = k1 > k0 ? (k1 - k0 + KS - 1) / KS : 0;
  float *ring = smem + (size_t)warp * STAGES * S::FLOATS;
  auto load_w = [&](int blk, int stage) {
    float *dst = ring + (size_t)stage * S::FLOATS + RM * PITCH;
#pragma unroll
    for (int i = 0; i < 8; ++i) {                       // 64 rows x 4 pieces of 16 bytes
      const int e = i * 32 + lane, piece = e & 3, row = e >> 2, k = k0 + blk * KS + piece * 4;
      const bool in = k < k1 && n0 + row < N;
      copy16(dst + row * PITCH + piece * 4, in ? W + (size_t)(n0 + row) * ldw + k : W, in);
    }
  };
  auto load_a = [&](int blk, int stage) {
    float *dst = ring + (size_t)stage * S::FLOATS;
#pragma unroll
    for (int i = 0; i < RM / 8; ++i) {
      const int e = i * 32 + lane, piece = e & 3, row = e >> 2, k = k0 + blk * KS + piece * 4;
      const bool in = k < k1 && m0 + row < M;
      copy16(dst + row * PITCH + piece * 4, in ? A + (size_t)(m0 + row) * lda + k : A, in);
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s)
    if (s < n_blocks) load_w(s, s);
  grid_dependency_wait();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < n_blocks) load_a(s, s);
    copy_commit();
  }
  unsigned long long acc[LM][8];                        // sums over even and odd k
#pragma unroll
  for (int i = 0; i < LM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  const int ma = lane >> 3, nb = lane & 7;              // this lane's rows of A: ma + 4 i; of W: nb + 8 j
  for (int blk = 0; blk < n_blocks; ++blk) {
    copy_wait<STAGES - 2>();
    __syncwarp();
    {
      const int ahead = blk + STAGES - 1;
      if (ahead < n_blocks) {
        load_w(ahead, ahead % STAGES);
        load_a(ahead, ahead % STAGES);
      }
      copy_commit();
    }
    const float *sa = ring + (size_t)(blk % STAGES) * S::FLOATS + ma * PITCH;
    const float *sw = ring + (size_t)(blk % STAGES) * S::FLOATS + (RM + nb) * PITCH;
#pragma unroll 2
    for (int k4 = 0; k4 < KS; k4 += 4) {
      ulonglong2 w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = ld_pairs(sw + j * 8 * PITCH + k4);
#pragma unroll
      for (int i = 0; i < LM; ++i) {
        const ulonglong2 a = ld_pairs(sa + i * 4 * PITCH + k4);
#pragma unroll
        for (int j = 0; j < 8; ++j) fma_pair(acc[i][j], a.x, w[j].x);
#pragma unroll
        for (int j = 0; j < 8; ++j) fma_pair(acc[i][j], a.y, w[j].y);
      }
    }
  }
  copy_wait<0>();
  __syncthreads();
  float *red = smem + (size_t)warp * RM * 64;           // [PARTS][RM][64], over the rings
#pragma unroll
  for (int i = 0; i < LM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) red[(ma + 4 * i) * 64 + nb + 8 * j] = add_pair(acc[i][j]);
  __syncthreads();
  for (int e = threadIdx.x; e < RM * 64; e += 256) {
    const int m = m0 + e / 64, n = n0 + e % 64;
    if (m >= M || n >= N) continue;
    float v = smem[e];
#pragma unroll
    for (int p = 1; p < PARTS; ++p) v += smem[(size_t)p * RM * 64 + e];
    if (bias) v += bias[n];
    C[(size_t)m * ldc + n] = v;
  }
}

template <int MT>
static int launch_few(const float *A, long long lda, const float *W, long long ldw, const float *bias, float *C, long long ldc, int M, int N,
                      int K, cudaStream_t stream) {
  auto kern = gemm_few_kernel<MT>;
  LLM_CHECK_CUDA(llm_allow_smem(kern, FewShape<MT>::SMEM), "gemm_plain attribute");
  LLM_CHECK_CUDA(llm_launch(kern, dim3((N + 15) / 16, (M + MT - 1) / MT), dim3(128), FewShape<MT>::SMEM, stream, A, lda, W, ldw, bias, C, ldc, M, N, K),
                 "gemm_plain launch");
  return LLM_OK;
}
static int launch_tile(const float *A, long long lda, const float *W, long long ldw, const float *bias, float *C, long long ldc, int M, int N,
                       int K, cudaStream_t stream) {
  using S = TileShape;
  LLM_CHECK_CUDA(llm_allow_smem(gemm_tile_kernel, S::SMEM), "gemm_plain attribute");
  LLM_REQUIRE(M <= 65535 * BM, "gemm_plain: %d rows are too many", M);        // as for the tiles of 64 rows below
  constexpr int MOST = 65535 * S::RM;          // rows of one launch
  for (long long m0 = 0; m0 < M; m0 += MOST) {
    const int m = (int)(M - m0 < MOST ? M - m0 : MOST);
    LLM_CHECK_CUDA(llm_launch(gemm_tile_kernel, dim3((N + 63) / 64, (m + S::RM - 1) / S::RM), dim3(256), S::SMEM, stream, A + m0 * lda, lda, W, ldw,
                              bias, C + m0 * ldc, ldc, m, N, K),
                   "gemm_plain launch");
  }
  return LLM_OK;
}
// Both kernels give a row the same bits, so the choice may look at everything.  Eight rows on the kernel for few cost 59 us at a W of
// [16,384, 2,048] and 31 at [2,048, 8,192], the tile's kernel 76 and 119 whatever the rows up to 32: with tiles for
// less than half of the SMs it is better to stream W twice.
static int launch_f32(const float *A, long long lda, const float *W, long long ldw, const float *bias, float *C, long long ldc, int M, int N,
                      int K, cudaStream_t stream) {
  if (M == 1) return launch_few<1>(A, lda, W, ldw, bias, C, ldc, M, N, K, stream);
  if (M == 2) return launch_few<2>(A, lda, W, ldw, bias, C, ldc, M, N, K, stream);
  if (M <= 4) return launch_few<4>(A, lda, W, ldw, bias, C, ldc, M, N, K, stream);
  if (M <= 8 || (M <= 16 && (N + 63) / 64 <= sm_count() / 2)) return launch_few<8>(A, lda, W, ldw, bias, C, ldc, M, N, K, stream);
  return launch_tile(A, lda, W, ldw, bias, C, ldc, M, N, K, stream);
}
// Whether rows start on 16 bytes and hold whole pieces of 16: a question of the matrices, never of the number of rows.
static bool takes_f32(const void *A, long long lda, const void *W, long long ldw, int K) {
  return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
}

// ---------------------------------------------------------------- every type and alignment

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(const TA *__restrict__ A, long long lda, const TW *__restrict__ W, long long ldw,
                  const float *__restrict__ bias, TC *__restrict__ C, long long ldc, int M, int N, int K) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;          // 16 x 16 threads, each 4 x 4 outputs
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64 x 16 tile of each operand: 1024 values, 4 per thread; k is the fast index of
    // the load so that reads of a row are contiguous.
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const int e = tid + l * 256;
      const int r = e / BK, kk = e % BK;
      const int gm = m0 + r, gn = n0 + r, gk = k0 + kk;
      As[kk][r] = (gm < M && gk < K) ? to_float(A[(size_t)gm * lda + gk]) : 0.f;
      Ws[kk][r] = (gn < N && gk < K) ? to_float(W[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[gn];
      C[(size_t)gm * ldc + gn] = from_float<TC>(v);
    }
  }
}

template <typename TA, typename TW, typename TC>
static int launch(const void *A, long long lda, const void *W, long long ldw, const float *bias, void *C,
                  long long ldc, int M, int N, int K, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  LLM_REQUIRE(grid.y <= 65535, "gemm_plain: %d rows are too many for one launch", M);
  gemm_plain_kernel<TA, TW, TC><<<grid, 256, 0, stream>>>((const TA *)A, lda, (const TW *)W, ldw, bias,
                                                         (TC *)C, ldc, M, N, K);
  LLM_CHECK_LAUNCH("gemm_plain");
  return LLM_OK;
}

// in_dtype is the type of A and W, out_dtype that of C.  Leading dimensions in elements.
LLM_EXPORT int llm_gemm_plain(int in_dtype, int out_dtype, const void *A, long long lda, const void *W,
                              long long ldw, const float *bias, void *C, long long ldc, int M, int N,
                              int K, cudaStream_t stream) {
  if (M == 0) return LLM_OK;
  LLM_REQUIRE(M > 0 && N > 0 && K > 0 && lda >= K && ldw >= K && ldc >= N, "gemm_plain: bad sizes");
  if (in_dtype == LLM_F32 && out_dtype == LLM_F32 && takes_f32(A, lda, W, ldw, K))
    return launch_f32((const float *)A, lda, (const float *)W, ldw, bias, (float *)C, ldc, M, N, K, stream);
  if (in_dtype == LLM_F32 && out_dtype == LLM_F32)
    return launch<float, float, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, stream);
  if (in_dtype == LLM_BF16 && out_dtype == LLM_BF16)
    return launch<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(A, lda, W, ldw, bias, C, ldc, M, N, K, stream);
  if (in_dtype == LLM_BF16 && out_dtype == LLM_F32)
    return launch<__nv_bfloat16, __nv_bfloat16, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, stream);
  LLM_FAIL("gemm_plain: unsupported dtypes in %d out %d", in_dtype, out_dtype);
}
