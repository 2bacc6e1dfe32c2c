// The 32-bit product on the 5th-generation tensor cores: out[M, N] = x[M, K] * W[N, K]^T (+ bias), 32-bit operands and sums.
//
// A tensor core takes 11 significant bits of a 32-bit operand (kind::tf32).  So each operand is split, in the kernel, into what such
// a value holds and what such a value holds of the rest: x = h + l, |l| <= 2^-11 |x|, and what is left of l is about
// 2^-22 |x| at most.  A product is l h' + h l' + h h': three tensor-core products, the small ones first; l l' (2^-22 of the product at most, of
// either sign) is left out.  The tensor cores' own sums are kept short, because they do not round to nearest: 32 of K, then a warp takes the sum
// out of tensor memory and adds it to its registers in 32-bit arithmetic.
//
// W's rows are the 128-row operand and the rows of x its N operand, as in gemm_tc.cu; the walk over K is in stages of 32:
//   loader       TMA boxes of [128 x 32] of W and [TN x 32] of x (128-byte swizzle) into a ring; W's before the kernel before is waited for;
//   converters   split W's tile and put both parts into tensor memory, as the A operand (a lane a row: shared memory, which the products and
//                the copies keep busy, is read once for it), and split x's tile within shared memory;
//   issuer       twelve tcgen05.mma a stage, into one of two accumulators (at TN = 128 a stage takes 0.9 us: 0.6 of products, 0.45 to split x, and three
//                stages in the ring do not hide them and a load behind one another);
//   adders       the sum of a stage (tcgen05.ld) to their registers.
// K is cut into `parts` runs, one or two to each CTA of a cluster, whose sums meet through distributed shared memory and are added in order.
// Two where TN is 128: such a CTA fills an SM, and sixteen clusters of eight do not find room at once.
// The number of parts and the stages depend on N and K alone, so a row's bits do not depend on how many rows the call has.
//
// Infinities and values that are no number have no such parts: where a sum is not finite its CTA adds that run of K again, product by product.
// Every wait has a time limit, as in gemm_tc.cu.
#pragma once
#include "tc_common.cuh"

namespace {

constexpr int FS_BK = 32;                      // of K to a stage: 128 bytes, one swizzle row
constexpr int FS_W_BYTES = 128 * FS_BK * 4;

template <int TN>
struct FsShape {
  static constexpr int X_BYTES = TN * FS_BK * 4;                // x's tile, and once more for its second part
  static constexpr int STAGE_BYTES = FS_W_BYTES + 2 * X_BYTES;
  static constexpr int GROUPS = TN == 128 ? 1 : 2;              // of four converter warps of W, a stage to each in turn
  static constexpr int XCONV = TN >= 64 ? TN / 32 : TN / 16;    // converter warps of x
  static constexpr int ADD = TN >= 64 ? 8 : 4;                  // adder warps
  static constexpr int COLS = TN / (ADD / 4);                   // rows of x to an adder's lane
  static constexpr int XCONV0 = 2 + 4 * GROUPS, ADD0 = XCONV0 + XCONV;      // their first warps
  static constexpr int THREADS = 32 * (ADD0 + ADD);
  // few rows of x: half of an SM's shared memory, so that the next product's CTA fills its ring while this one finishes
  static constexpr int CTAS = TN <= 32 ? 2 : 1;                 // on an SM at once
  static constexpr int SUB = TN == 128 ? 2 : 1;                 // parts of K to a CTA, one behind the other
  static constexpr int STAGES = TN <= 32 ? 102 * 1024 / STAGE_BYTES : TN == 64 ? 6 : 3;
  static constexpr int SUM_BYTES = TN * 128 * 4;                // a part's sums
  static constexpr int SLOTS = TN == 128 ? 4 : TN == 64 ? 2 : 3;                       // of the A operand in tensor memory
  static constexpr int ACC0 = SLOTS * 64;                       // columns: SLOTS x [h | l], then two accumulators
  static constexpr int TMEM = TN == 128 ? 512 : 256;
  // behind the ring: with two parts to a CTA the first one's sums (the last one's lie over the ring), else what the CTAs of the
  // cluster bring for this one to add
  static constexpr int KEPT = STAGES * STAGE_BYTES;
  static constexpr int BARS = KEPT + SUM_BYTES;
  static constexpr size_t SMEM = 1024 + (size_t)BARS + 512;
  static_assert(ACC0 + 2 * TN <= TMEM, "tensor memory");
  static_assert(SUM_BYTES <= STAGES * STAGE_BYTES, "the sums fit the ring");
};

__device__ __forceinline__ void fs_mma(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// The two parts of a value.  h: rounded to 11 bits (half away).  l: the rest, exact; the tensor cores read 11 bits of
// it, and the addition makes up for what that takes off on average.  Not a number in, not a number in l.
__device__ __forceinline__ void fs_split(float x, unsigned &h, unsigned &l) {
  h = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  const float rest = x - __uint_as_float(h);
  l = __float_as_uint(fmaf(rest, 0x1.6p-12f, rest));
}
__device__ __forceinline__ float fs_peer(unsigned addr, unsigned rank) {           // a value in the shared memory of a CTA of the cluster
  float v;
  asm volatile("{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %1, %2;\nld.shared::cluster.f32 %0, [a];\n}" : "=f"(v) : "r"(addr), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ void fs_put(unsigned addr, unsigned rank, float v) {
  asm volatile("{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %0, %1;\nst.shared::cluster.f32 [a], %2;\n}" ::"r"(addr), "r"(rank), "f"(v) : "memory");
}
__device__ __forceinline__ void fs_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void fs_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void fs_cluster_sync() {
  fs_cluster_arrive();
  fs_cluster_wait();
}

template <int TN>
__global__ void __launch_bounds__(FsShape<TN>::THREADS, FsShape<TN>::CTAS)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const float *A, long long lda,
                   const float *__restrict__ W, long long ldw, const float *__restrict__ bias, float *__restrict__ C, long long ldc, int M, int N,
                   int K, int parts, int stages_per_part, int *status) {
  using S = FsShape<TN>;
  constexpr int STAGES = S::STAGES, SLOTS = S::SLOTS, COLS = S::COLS, SUB = S::SUB;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned long long *bars = (unsigned long long *)(smem + S::BARS);
  const unsigned bar_w = smem_u32(bars), bar_x = bar_w + 8 * STAGES, bar_xready = bar_x + 8 * STAGES, bar_empty = bar_xready + 8 * STAGES;   // of a stage
  const unsigned bar_ready = bar_empty + 8 * STAGES, bar_used = bar_ready + 8 * SLOTS;                  // of a slot of A
  const unsigned bar_full = bar_used + 8 * SLOTS, bar_added = bar_full + 16;                            // of an accumulator
  unsigned *tmem_slot = (unsigned *)(bars + 4 * STAGES + 2 * SLOTS + 4);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  grid_dependents_launch();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_w + 8 * s, 1);
      mbar_init(bar_x + 8 * s, 1);
      mbar_init(bar_xready + 8 * s, S::XCONV);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(bar_ready + 8 * s, 4);
      mbar_init(bar_used + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar_full + 8 * a, 1);
      mbar_init(bar_added + 8 * a, S::ADD);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tma_prefetch_map(&map_w);
    tma_prefetch_map(&map_x);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((unsigned)S::TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = *tmem_slot;
  // A CTA's shared memory may be written by another one only when it is known to run: all say so here, and wait for it where the adders put their
  // sums (the other warps where the parts meet), when it has long been so.
  if (parts > 1) fs_cluster_arrive();

  const int tok0 = blockIdx.y * TN, row0 = blockIdx.z * 128;
  const int sub = parts > 1 ? SUB : 1;                          // parts of this CTA; the CTAs of a cluster share a tile's parts
  const int n_stages = (K + FS_BK - 1) / FS_BK;
  const int st0 = blockIdx.x * sub * stages_per_part;
  const int n = max(0, min(n_stages, st0 + sub * stages_per_part) - st0);      // 0: nothing is left for these parts
  const int quarter = warp & 3;                // the 32 lanes of tensor memory that a warp may use

  if (warp == 0) {
    // ------------------------------------------------------------ loader
    const bool leader = elect_one();
    auto load_w = [&](int i) {
      if (!leader) return;
      const int s = i % STAGES;
      mbar_expect_tx(bar_w + 8 * s, FS_W_BYTES);
      tma_load_2d(smem_u32(smem + s * S::STAGE_BYTES), &map_w, (st0 + i) * FS_BK, row0, bar_w + 8 * s);
    };
    auto load_x = [&](int i) {
      if (!leader) return;
      const int s = i % STAGES;
      mbar_expect_tx(bar_x + 8 * s, S::X_BYTES);
      tma_load_2d(smem_u32(smem + s * S::STAGE_BYTES) + FS_W_BYTES, &map_x, (st0 + i) * FS_BK, tok0, bar_x + 8 * s);
    };
    const int first = min(n, STAGES);
    for (int i = 0; i < first; ++i) load_w(i);
    grid_dependency_wait();
    for (int i = 0; i < first; ++i) load_x(i);
    bool ok = true;
    for (int i = first; i < n; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * (i % STAGES), (i / STAGES & 1) ^ 1, abort_flag, status, 1));
      if (!ok) break;
      load_w(i);
      load_x(i);
    }
    if (leader && (!ok || *abort_flag)) {      // given up: let the loads that are in flight land before the CTA goes away
      const unsigned long long t0 = globaltimer();
      while (globaltimer() - t0 < 2000000ull) {
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ products
    const bool leader = elect_one();
    // D in 32-bit floats, A and B tf32 (format 2), both K-major
    constexpr unsigned IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(TN >> 3) << 17) | ((128u >> 4) << 24);
    for (int i = 0; i < n; ++i) {
      const int s = i % STAGES, a = i % SLOTS, acc = i & 1;
      const bool ok = mbar_wait(bar_ready + 8 * a, i / SLOTS & 1, abort_flag, status, 3) &&
                      mbar_wait(bar_xready + 8 * s, i / STAGES & 1, abort_flag, status, 3) &&
                      mbar_wait(bar_added + 8 * acc, (i / 2 & 1) ^ 1, abort_flag, status, 2);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const unsigned x_addr = smem_u32(smem + s * S::STAGE_BYTES) + FS_W_BYTES;
      const unsigned long long xh = smem_desc(x_addr), xl = smem_desc(x_addr + S::X_BYTES);
      const unsigned wh = tmem + a * 64, wl = wh + 32, d = tmem + S::ACC0 + acc * TN;
      if (leader) {
#pragma unroll
        for (int k = 0; k < 12; ++k)           // 8 of K: 32 bytes of a row
          fs_mma(d, (k < 4 ? wl : wh) + (k & 3) * 8, (k < 4 || k >= 8 ? xh : xl) + (unsigned long long)((k & 3) * 2), IDESC, k > 0 ? 1u : 0u);
        tc_commit(bar_empty + 8 * s);
        tc_commit(bar_used + 8 * a);
        tc_commit(bar_full + 8 * acc);
      }
      __syncwarp();
    }
    grid_dependency_wait();
  } else if (warp < S::XCONV0) {
    // ------------------------------------------------------------ W's converters
    const int row = quarter * 32 + lane;
    for (int i = (warp - 2) / 4; i < n; i += S::GROUPS) {
      const int s = i % STAGES, a = i % SLOTS;
      const unsigned char *st = smem + s * S::STAGE_BYTES + row * 128;
      const bool ok = mbar_wait(bar_used + 8 * a, (i / SLOTS & 1) ^ 1, abort_flag, status, 4) && mbar_wait(bar_w + 8 * s, i / STAGES & 1, abort_flag, status, 4);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const unsigned dst = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)(a * 64);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        unsigned h[16], l[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {          // 16-byte pieces of the row, where the swizzle has put them
          const float4 v = *reinterpret_cast<const float4 *>(st + (((half * 4 + c) ^ (row & 7)) << 4));
          fs_split(v.x, h[4 * c], l[4 * c]);
          fs_split(v.y, h[4 * c + 1], l[4 * c + 1]);
          fs_split(v.z, h[4 * c + 2], l[4 * c + 2]);
          fs_split(v.w, h[4 * c + 3], l[4 * c + 3]);
        }
        tc_st16(dst + half * 16, h);
        tc_st16(dst + 32 + half * 16, l);
      }
      tc_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ready + 8 * a);
    }
    grid_dependency_wait();
  } else if (warp < S::ADD0) {
    // ------------------------------------------------------------ x's converters
    const int tid = threadIdx.x - 32 * S::XCONV0;
    for (int i = 0; i < n; ++i) {
      const int s = i % STAGES;
      if (!__all_sync(0xffffffffu, mbar_wait(bar_x + 8 * s, i / STAGES & 1, abort_flag, status, 5))) break;
      float4 *xt = reinterpret_cast<float4 *>(smem + s * S::STAGE_BYTES + FS_W_BYTES), *xl = xt + S::X_BYTES / 16;
#pragma unroll 4
      for (int e = tid; e < TN * 8; e += 32 * S::XCONV) {      // place by place: both tiles are swizzled alike
        const float4 v = xt[e];
        uint4 vh, vl;
        fs_split(v.x, vh.x, vl.x);
        fs_split(v.y, vh.y, vl.y);
        fs_split(v.z, vh.z, vl.z);
        fs_split(v.w, vh.w, vl.w);
        *reinterpret_cast<uint4 *>(xt + e) = vh;
        *reinterpret_cast<uint4 *>(xl + e) = vl;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // the products read shared memory by another path than these stores
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_xready + 8 * s);
    }
    grid_dependency_wait();
  } else {
    // ------------------------------------------------------------ adders
    const int col0 = (warp - S::ADD0) / 4 * COLS, row = row0 + quarter * 32 + lane;
    const unsigned src = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)(S::ACC0 + col0);
    bool ok = true;
    for (int p = 0, i0 = 0; p < sub; ++p) {
      const int i1 = p == sub - 1 ? n : min(n, stages_per_part);
      float sum[COLS];
#pragma unroll
      for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
      for (int i = i0; i < i1; ++i) {
        const int acc = i & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * acc, i / 2 & 1, abort_flag, status, 6));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < COLS; c += 16) {
          float v[16];
          tc_ld16(src + (unsigned)(acc * TN + c), v);
#pragma unroll
          for (int j = 0; j < 16; ++j) sum[c + j] += v[j];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_added + 8 * acc);
      }
      // the part's sums: to the result, or to shared memory, the last part's over the ring
      if (p == 0) grid_dependency_wait();
      bool odd = false;                        // something that is not finite
#pragma unroll
      for (int j = 0; j < COLS; ++j) odd = odd || !(fabsf(sum[j]) <= 3.402823466e38f);
      float *mine = reinterpret_cast<float *>(smem + (p == sub - 1 ? 0 : S::KEPT)) + (size_t)col0 * 128 + quarter * 32 + lane;
      const int n_tok = min(COLS, M - tok0 - col0);
      float *c = C + (size_t)(tok0 + col0) * ldc + row;
      if (parts > 1) {
#pragma unroll
        for (int j = 0; j < COLS; ++j) mine[j * 128] = sum[j];
      } else if (row < N) {
        const float add = bias ? bias[row] : 0.f;
#pragma unroll
        for (int j = 0; j < COLS; ++j)
          if (j < n_tok) c[(size_t)j * ldc] = bias ? sum[j] + add : sum[j];
      }
      if (odd && ok && row < N) {
        const int k0 = (st0 + i0) * FS_BK, k1 = min(K, (st0 + i1) * FS_BK);
#pragma unroll 1
        for (int j = 0; j < n_tok; ++j) {
          float *y = parts > 1 ? mine + j * 128 : c + (size_t)j * ldc;
          if (fabsf(*y) <= 3.402823466e38f) continue;
          const float *x = A + (size_t)(tok0 + col0 + j) * lda, *w = W + (size_t)row * ldw;
          float v = 0.f;
#pragma unroll 1
          for (int k = k0; k < k1; ++k) v = fmaf(x[k], w[k], v);
          *y = parts == 1 && bias ? v + bias[row] : v;
        }
      }
      if (parts > 1 && p == 0) {
        __syncwarp();
        fs_cluster_wait();
      }
      if (parts > 1 && SUB == 1) {             // to the CTA that adds this row of x
        const int n_ctas = parts, most = (TN + n_ctas - 1) / n_ctas;
        const unsigned there = smem_u32(smem) + S::KEPT + (unsigned)((int)blockIdx.x * most * 128 + quarter * 32 + lane) * 4;
#pragma unroll 1
        for (int j = 0; j < n_tok; ++j)
          fs_put(there + (unsigned)((col0 + j) / n_ctas * 512), (unsigned)((col0 + j) % n_ctas), mine[j * 128]);
      }
      i0 = i1;
    }
  }

  // ---------------------------------------------------------------- the parts' sums, in order
  if (parts > 1) {
    __syncwarp();
    if (warp < S::ADD0) fs_cluster_wait();     // for the CTAs' start: the adders have
    fs_cluster_sync();
    const int n_ctas = parts / sub, rank = blockIdx.x;         // the grid's first dimension is one cluster
    const unsigned base = smem_u32(smem);
    const int n_tok = min(TN, M - tok0), r = threadIdx.x & 127, at = threadIdx.x >> 7;
    constexpr int AT = S::THREADS / 128;                       // a token to each 128 threads; what is left of the block has none
    if (at < AT && row0 + r < N) {
      const float add = bias ? bias[row0 + r] : 0.f;
      const int most = (TN + n_ctas - 1) / n_ctas;
      const float *here = reinterpret_cast<const float *>(smem + S::KEPT) + r;
      for (int c = rank + at * n_ctas; c < n_tok; c += AT * n_ctas) {
        float v[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          if (SUB == 1) v[p] = p < parts ? here[(p * most + c / n_ctas) * 128] : 0.f;
          else v[p] = p < parts ? fs_peer(base + (unsigned)(p % SUB == SUB - 1 ? 0 : S::KEPT) + (unsigned)(c * 128 + r) * 4, p / SUB) : 0.f;
        }
        float y = v[0];
#pragma unroll
        for (int p = 1; p < 8; ++p)
          if (p < parts) y += v[p];
        C[(size_t)(tok0 + c) * ldc + row0 + r] = bias ? y + add : y;
      }
    }
    if (SUB > 1) {
      __syncwarp();
      fs_cluster_sync();                       // nobody leaves while another reads its sums
    }
  }

  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)S::TMEM) : "memory");
  }
}

// A map over a row-major 32-bit matrix [rows, cols] with row stride ld: boxes of [box_rows x 32], 128-byte swizzle, zeros outside.
int fs_map(const void *ptr, long long rows, long long cols, long long ld, int box_rows, CUtensorMap *out) {
  EncodeTiledFn fn = encode_fn();
  LLM_REQUIRE(fn != nullptr, "tensor map: the driver does not offer cuTensorMapEncodeTiled");
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
  const cuuint32_t box[2] = {(cuuint32_t)FS_BK, (cuuint32_t)box_rows}, elem[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  LLM_REQUIRE(r == CUDA_SUCCESS, "tensor map: cuTensorMapEncodeTiled failed (%d) for a 32-bit matrix of %lld x %lld", (int)r, rows, cols);
  return LLM_OK;
}

// Parts of K: as many as give every SM a tile, by the matrix alone.
inline int fs_parts(int N, int K) {
  const int tiles = (N + 127) / 128, stages = (K + FS_BK - 1) / FS_BK;
  int parts = 1;
  while (parts < 8 && tiles * parts * 2 <= sm_count() && stages / (parts * 2) >= 4) parts *= 2;
  return parts;
}

template <int TN>
int launch_f32_tc(const float *A, long long lda, const float *W, long long ldw, const float *bias, float *C, long long ldc, int M, int N, int K,
                  int *status, cudaStream_t stream) {
  using S = FsShape<TN>;
  CUtensorMap map_w, map_x;
  int rc = fs_map(W, N, K, ldw, 128, &map_w);
  if (rc == LLM_OK) rc = fs_map(A, M, K, lda, TN, &map_x);
  if (rc != LLM_OK) return rc;
  const int stages = (K + FS_BK - 1) / FS_BK, parts = fs_parts(N, K), per = (stages + parts - 1) / parts;
  auto kern = gemm_f32_tc_kernel<TN>;
  LLM_CHECK_CUDA(llm_allow_smem(kern, S::SMEM), "gemm_f32_tc attribute");
  cudaLaunchConfig_t cfg = {};
  const int ctas = parts > 1 ? parts / S::SUB : 1;              // of a cluster
  cfg.gridDim = dim3(ctas, (M + TN - 1) / TN, (N + 127) / 128);
  cfg.blockDim = dim3(S::THREADS);
  cfg.dynamicSmemBytes = S::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = llm_pdl_enabled() ? 2 : 1;
  LLM_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, map_w, map_x, A, lda, W, ldw, bias, C, ldc, M, N, K, parts, per, status), "gemm_f32_tc launch");
  return LLM_OK;
}

}  // namespace
