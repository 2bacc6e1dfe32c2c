// Matrix product on the 5th-generation tensor cores: out[M, N] = x[M, K] * W[N, K]^T, bfloat16
// operands, 32-bit accumulation in tensor memory, optional fused SwiGLU and partial products
// over parts of K.  One kernel serves a decoding step of a few tokens, where it streams W once
// from HBM, and a prompt step of thousands.
//
// W's rows are the 128-row operand of tcgen05.mma and the tokens its N operand ("swap AB"): the
// accumulator of a tile is D[128 rows of W][TN tokens] with TN = 16 .. 256, so that a step of 8
// tokens costs no more than one of 16 and the instruction shape is full at any batch.  A CTA is
// persistent (one per SM) and walks over its tiles with three kinds of warps:
//   warp 0   one lane issues TMA loads (cp.async.bulk.tensor, 128-byte swizzle) of [64 rows x 64 k]
//            boxes of W and a [TN x 64 k] box of x into a ring of shared-memory stages;
//   warp 1   allocates tensor memory; one lane issues tcgen05.mma (four k-steps of 16 per stage)
//            and commits each stage back to the loader and each finished tile to the epilogue;
//   warps 2-5 read the accumulator with tcgen05.ld (each warp its quarter of the 128 lanes),
//            apply the epilogue and store out[token][row], while the next tile's products run
//            into the other accumulator buffer.
// 90 KB (few tokens) to 200 KB (prompts) of loads are in flight per SM, which is what a stream from
// HBM needs.
//
// SwiGLU, or any gated unit of GluShape: W is the stacked gate|up matrix [2I, K], and the stacked product never reaches memory (the
// reference runs a separate launch, src/flint/cuda/swiglu.cu:29-59, after cuBLAS, src/flint/cuda/gemm_cublas.cc:160-197).  Which form
// a launch takes (dispatch_tc):
//   up to 64 tokens      a tile of 64 features, gate and up rows in turns of 16, traded by shuffles within an epilogue warp; where I is
//                        no multiple of 16, gate rows in lanes 0-63 and up rows in lanes 64-127, handed over through shared memory;
//   prompts, takes_pair  two SMs to a tile (gated_pair_kernel, below), rows in turns as above;
//   other prompts        a tile of 128 gate rows and one of 128 up rows with an accumulator each.
//
// Rows of W, tokens and K beyond the matrices are zero-filled by TMA and never stored, so every
// size is taken (K a multiple of 8: rows must start on 16 bytes).  Every wait on a barrier has a
// time limit; when it runs out the CTA records a code in `status`, waits for its loads in flight,
// frees its tensor memory and returns.  Weights are loaded before the programmatic dependency on
// the previous kernel is waited for, tokens after it.
#include "common.cuh"
#include "tc_common.cuh"

LLM_DEFINE_LAST_ERROR(llm_gemm_tc_last_error)

namespace {

constexpr int TC_THREADS = 192;
constexpr int TC_ROWS = 128;                   // rows of W per tile (UMMA M)
constexpr int TC_A_BYTES = TC_ROWS * TC_BK * 2;

// SW: 0 plain product; 1 SwiGLU with gate and up rows interleaved in one 128-row tile (64 + 64,
// handed over between epilogue warps: steps of few tokens, where a tile per SM matters); 2 SwiGLU with
// a tile of 128 gate rows and one of 128 up rows per stage and an accumulator for each, so that a
// lane holds both values of a feature (prompt steps); 3 like 1 with gate and up rows in turns of 16 (the map of get_gated_map: I a
// multiple of 16), so that a warp has both halves of its features and trades them by shuffles: 64 tokens x 16,384
// rows 19.7 -> 16.1 us, 8 tokens 14.4 -> 13.1.
//
// R, KBS (plain products): a matrix with few tiles of 128 rows leaves most SMs idle, and the others' time goes by the stages that a loader and an
// issuer get through one by one, some 0.2 us each beyond the ring, whatever a stage holds (at K = 2,048 five ready stages of 32: 8.8 us for 6 tiles, 9.2
// for 25).  There a tile has R = 32 or 64 rows and a stage KBS = 4 or 2 blocks of 64 of K, so that four or two times as many SMs each
// get through a quarter or half of the stages.  The instruction keeps its 128 rows: those beyond R are whatever lies behind the
// block in shared memory, and nobody reads their sums.  A row's sum is the same whatever R.  In steps of a few requests, K = 2,048: 3,104 rows
// x 4 tokens 9.2 -> 7.2 us, 8,192 x 2 9.8 -> 7.5.  Every CTA brings the tokens too: from 33 tokens on 32 rows to a tile lose, and beyond 48 so do 64
// (a prompt of 37 tokens, tiles of 128 / 64 / 32 rows: 1,054 / 1,043 / 1,070 us; a step of 64 50.0 / 50.6 ms a pass).
template <int TN, int SW, int R = TC_ROWS, int KBS = 1>
struct TcShape {
  static_assert(SW == 0 || (R == TC_ROWS && (KBS == 1 || SW == 3)), "gated units have tiles of 128 rows");
  static constexpr int A_TILES = SW == 2 ? 2 : 1;
  static constexpr int A_BYTES = A_TILES * R * TC_BK * 2;
  static constexpr int B_BYTES = TN * TC_BK * 2;
  static constexpr int BLOCK_BYTES = A_BYTES + B_BYTES;                  // 64 of K
  static constexpr int STAGE_BYTES = KBS * BLOCK_BYTES;
  // Steps of few tokens (TN <= 32) take half of an SM's shared memory, so that the CTA of the next
  // product in the stream can move in beside this one and fill its ring with weights while this
  // one finishes; larger steps take a ring as deep as fits (measured: equal at 1 and 8 tokens,
  // 5 % faster at 64 with the deep ring).  Tiles of fewer rows take BEYOND besides: with 32 rows, and with 64 rows and up to 16 tokens, that makes 116,224
  // bytes, of which two lack 1 KB of an SM; such a CTA has room beside tiles of 128 rows or the gated unit, not beside one of its kind.  The
  // gated unit of up to 16 tokens, the widest product, takes stages of two blocks and as much as two CTAs
  // of an SM can have: 8 tokens, 16 steps 14.35 -> 14.23 ms a pass (the other products too: 13.97, but decoders with more and smaller launches
  // lose 1.5 %, whose kernels then find less room beside them; stages of two blocks in 73 KB: 15.5).
  static constexpr int BUDGET = SW == 3 && TN == 16 ? 108 * 1024 : TN <= 32 ? 100 * 1024 : 200 * 1024;
  static constexpr int STAGES = BUDGET / STAGE_BYTES;
  static constexpr int ACC_COLS = A_TILES * TN;                          // columns of one accumulator buffer
  static constexpr int TMEM_COLS = 2 * ACC_COLS < 32 ? 32 : 2 * ACC_COLS;  // two buffers; a power of two
  // SwiGLU hand-over: 64 rows x 16 tokens (+1 pad).  Plain products have no use for it, but with 4 KB less of shared memory a third kernel's CTAs
  // find room beside two of these, which costs a step of few tokens 1 to 2 % (tiles of 128 rows, 8 tokens: 14.28 -> 14.41 ms a pass; not tried with tiles of fewer).
  static constexpr int XCH_BYTES = SW <= 1 ? 64 * 17 * 4 : 0;
  static constexpr int BEYOND = (TC_ROWS - R) * TC_BK * 2;              // read behind the last block by the instruction's other rows
  static constexpr size_t SMEM = 1024 + (size_t)STAGES * STAGE_BYTES + BEYOND + XCH_BYTES + 256;
  static_assert(TMEM_COLS <= 512, "the accumulators do not fit tensor memory");
};

// 64 of K of the gate and up rows of four groups of 16 features, in turns (get_gated_map)
__device__ __forceinline__ void tma_load_turns(unsigned dst, const CUtensorMap *map, int k, int group, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(k), "r"(0), "r"(group), "r"(bar) : "memory");
}
// A warp's 16 gate and 16 up rows of 16 tokens, a row to a lane (gates in lanes 0-15): the gate's lane keeps the even tokens, the
// up's lane the odd ones, and each stores the gated unit of its eight.
template <typename TO>
__device__ __forceinline__ void store_turns(const float (&v)[16], TO *__restrict__ out, long long ldo, int f, int n_out, int tok0, int M,
                                            const GluShape &glu) {
  const bool up = (threadIdx.x & 31) >= 16;
  TO y[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float even = v[2 * i], odd = v[2 * i + 1];
    const float got = __shfl_xor_sync(0xffffffffu, up ? even : odd, 16);
    y[i] = from_float<TO>(glu_value(up ? got : even, up ? odd : got, glu));
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int tok = tok0 + 2 * i + (up ? 1 : 0);
    if (f < n_out && tok < M) out[(size_t)tok * ldo + f] = y[i];
  }
}

template <int TN, int SW, typename TO, int R = TC_ROWS, int KBS = 1>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
               TO *__restrict__ out, long long ldo, int M, int n_out, int K, int row_tiles, int tok_tiles,
               int k_parts, int kb_per_part, long long part_stride, int group_tiles, int group_rows, GluShape glu, int *status) {
  using S = TcShape<TN, SW, R, KBS>;
  constexpr bool SWIGLU = SW == 1;                      // the interleaved tile with the hand-over
  constexpr int STAGES = S::STAGES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char *xch_raw = smem + (size_t)STAGES * S::STAGE_BYTES + S::BEYOND;
  unsigned long long *bars = (unsigned long long *)(xch_raw + S::XCH_BYTES);
  // bars: full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], hand-over full and empty;
  // then the TMEM address and the abort flag
  const unsigned bar_full = smem_u32(bars), bar_empty = smem_u32(bars + STAGES);
  const unsigned bar_tfull = smem_u32(bars + 2 * STAGES), bar_tempty = smem_u32(bars + 2 * STAGES + 2);
  const unsigned bar_xfull = smem_u32(bars + 2 * STAGES + 4), bar_xempty = smem_u32(bars + 2 * STAGES + 5);
  unsigned *tmem_slot = (unsigned *)(bars + 2 * STAGES + 6);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

  // The warp's number comes out of a shuffle so that the compiler knows it is the same in all of
  // a warp's lanes: the loader's and the issuer's loops then run in all 32 lanes (address and
  // descriptor arithmetic in the uniform datapath), and only the copy, product and commit
  // instructions themselves are one lane's.  Issued from inside a one-lane branch, a product cost
  // about 115 cycles of that lane, more than it takes the tensor core at 16 to 128 tokens.
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  grid_dependents_launch();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar_tfull + 8 * a, 1);
      mbar_init(bar_tempty + 8 * a, 4);
    }
    mbar_init(bar_xfull, 2);
    mbar_init(bar_xempty, 2);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((unsigned)S::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = *tmem_slot;

  const int n_tiles = row_tiles * tok_tiles * k_parts;
  const int n_kblocks_total = (K + TC_BK - 1) / TC_BK;
  constexpr int ROWS_OUT = SW == 1 || SW == 3 ? 64 : R;  // output features per tile

  if (warp == 0) {
    // ------------------------------------------------------------ loader
    const bool leader = elect_one();
    // The walk over this CTA's (tile, k block) pairs, one per stage filled.
    struct Walk {
      int tile, kb, kb1, x_row, row_a, row_b;
      bool valid;
    };
    auto start = [&](Walk &w, int tile) {
      w.tile = tile;
      w.valid = tile < n_tiles;
      if (!w.valid) return;
      const int part = tile % k_parts, row_tile = tile / (k_parts * tok_tiles);
      w.x_row = (tile / k_parts) % tok_tiles * TN + row_tile / group_tiles * group_rows;
      w.kb = part * kb_per_part;
      w.kb1 = min(n_kblocks_total, w.kb + kb_per_part);
      w.row_a = row_tile * ROWS_OUT;
      w.row_b = SW != 0 ? n_out + w.row_a : w.row_a + 64;
    };
    auto next = [&](Walk &w) {
      w.kb += KBS;
      if (w.kb >= w.kb1) start(w, w.tile + gridDim.x);
    };
    auto load_w = [&](const Walk &w, int stage) {
      const unsigned dst = smem_u32(smem + (size_t)stage * S::STAGE_BYTES);
      if (leader && (R < TC_ROWS || KBS > 1)) {
        const int n = min(KBS, w.kb1 - w.kb);           // the part's last stage may have fewer blocks
        mbar_expect_tx(bar_full + 8 * stage, n * S::BLOCK_BYTES);
#pragma unroll
        for (int j = 0; j < KBS; ++j)
          if (j < n) {
            if (SW == 3) tma_load_turns(dst + j * S::BLOCK_BYTES, &map_w, (w.kb + j) * TC_BK, w.row_a / 16, bar_full + 8 * stage);
            else tma_load_2d(dst + j * S::BLOCK_BYTES, &map_w, (w.kb + j) * TC_BK, w.row_a, bar_full + 8 * stage);
          }
      } else if (leader) {
        mbar_expect_tx(bar_full + 8 * stage, S::STAGE_BYTES);
        if (SW == 2) {                    // 128 gate rows, then 128 up rows: the map's boxes are 128 rows here
          tma_load_2d(dst, &map_w, w.kb * TC_BK, w.row_a, bar_full + 8 * stage);
          tma_load_2d(dst + TC_A_BYTES, &map_w, w.kb * TC_BK, w.row_b, bar_full + 8 * stage);
        } else if (SW == 3) {
          tma_load_turns(dst, &map_w, w.kb * TC_BK, w.row_a / 16, bar_full + 8 * stage);
        } else {
          tma_load_2d(dst, &map_w, w.kb * TC_BK, w.row_a, bar_full + 8 * stage);
          tma_load_2d(dst + TC_A_BYTES / 2, &map_w, w.kb * TC_BK, w.row_b, bar_full + 8 * stage);
        }
      }
    };
    auto load_x = [&](const Walk &w, int stage) {
      if (leader)
#pragma unroll
        for (int j = 0; j < KBS; ++j)
          if (j == 0 || w.kb + j < w.kb1)
            tma_load_2d(smem_u32(smem + (size_t)stage * S::STAGE_BYTES) + j * S::BLOCK_BYTES + S::A_BYTES, &map_x, (w.kb + j) * TC_BK,
                        w.x_row, bar_full + 8 * stage);
    };
    // Weights first: they do not depend on the kernel before this one, so the whole ring
    // is filled with them while that kernel still runs.  Then the wait, then the tokens of
    // the same stages, then the rest of the walk stage by stage.
    Walk w, w2;
    start(w, blockIdx.x);
    int n_pre = 0;
    for (; w.valid && n_pre < STAGES; next(w), ++n_pre) load_w(w, n_pre);
    start(w2, blockIdx.x);
    grid_dependency_wait();
    for (int s = 0; s < n_pre; ++s, next(w2)) load_x(w2, s);
    int stage = n_pre % STAGES;
    unsigned phase = n_pre == STAGES ? 1u : 0u;
    bool ok = true;
    for (; w.valid; next(w)) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, status, 1));
      if (!ok) break;
      load_w(w, stage);
      load_x(w, stage);
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
    if (leader && (!ok || *abort_flag)) {
      // given up: let the loads that are in flight land before the CTA goes away
      const unsigned long long t0 = globaltimer();
      for (int s = 0; s < STAGES; ++s)
        while (!mbar_try(bar_full + 8 * s, 0) && !mbar_try(bar_full + 8 * s, 1) && globaltimer() - t0 < 2000000ull) {
        }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ tensor-core issue
    const bool leader = elect_one();
    constexpr unsigned IDESC = instr_desc(TC_ROWS, TN);
    int stage = 0;
    unsigned phase = 0;
    int iter = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++iter) {
      const int part = tile % k_parts;
      const int kb0 = part * kb_per_part, kb1 = min(n_kblocks_total, kb0 + kb_per_part);
      const int acc = iter & 1;
      const unsigned acc_phase = (iter >> 1) & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(bar_tempty + 8 * acc, acc_phase ^ 1, abort_flag, status, 2));
      if (!ok) break;
      tc_fence_after();
      const unsigned d_tmem = tmem_base + acc * S::ACC_COLS;
      for (int kb = kb0; kb < kb1; kb += KBS) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * stage, phase, abort_flag, status, 3));
        if (!ok) break;
        tc_fence_after();
        const unsigned a_addr = smem_u32(smem + (size_t)stage * S::STAGE_BYTES);
        const unsigned long long a_desc = smem_desc(a_addr), b_desc = smem_desc(a_addr + S::A_BYTES);
        const unsigned long long a2_desc = smem_desc(a_addr + TC_A_BYTES);
        const unsigned first = kb > kb0 ? 1u : 0u;
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < TC_BK / 16; ++kk) {  // 16 k = 32 bytes further along the swizzled row
            tc_mma(d_tmem, a_desc + (unsigned long long)(kk * 2), b_desc + (unsigned long long)(kk * 2), IDESC,
                   kk > 0 ? 1u : first);
            if (SW == 2)                             // the up rows into the accumulator beside
              tc_mma(d_tmem + TN, a2_desc + (unsigned long long)(kk * 2), b_desc + (unsigned long long)(kk * 2), IDESC,
                     kk > 0 ? 1u : first);
          }
#pragma unroll
          for (int j = 1; j < KBS; ++j)
            if (kb + j < kb1) {
              const unsigned long long step = (unsigned long long)(j * (S::BLOCK_BYTES >> 4));
#pragma unroll
              for (int kk = 0; kk < TC_BK / 16; ++kk)
                tc_mma(d_tmem, a_desc + step + (unsigned long long)(kk * 2), b_desc + step + (unsigned long long)(kk * 2), IDESC, 1u);
            }
          tc_commit(bar_empty + 8 * stage);          // the stage is free when these products have read it
        }
        __syncwarp();
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok && leader) tc_commit(bar_tfull + 8 * acc);      // the tile's accumulator is complete
      __syncwarp();
    }
    grid_dependency_wait();
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5)
    grid_dependency_wait();
    const int quarter = warp & 3;                    // the 32 lanes of tensor memory this warp may read
    float *xch = (float *)xch_raw;
    int iter = 0;
    unsigned n_chunk = 0;                            // hand-overs so far (SwiGLU)
    bool ok = true;
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++iter) {
      const int part = tile % k_parts, tok_tile = (tile / k_parts) % tok_tiles, row_tile = tile / (k_parts * tok_tiles);
      const int acc = iter & 1;
      const unsigned acc_phase = (iter >> 1) & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag, status, 4));
      if (!ok) break;
      tc_fence_after();
      TO *o = out + (size_t)part * part_stride;
      const int row_in_tile = quarter * 32 + lane;
      const int tok0 = tok_tile * TN;
#pragma unroll 1
      for (int c0 = 0; c0 < TN && ok && (SW == 1 || tok0 + c0 < M) && quarter * 32 < R; c0 += 16, ++n_chunk) {
        float v[16];
        tc_ld16(tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)(acc * S::ACC_COLS + c0), v);
        if (SW == 3) {
          store_turns(v, o, ldo, row_tile * 64 + quarter * 16 + (lane & 15), n_out, tok0 + c0, M, glu);
        } else if (SW == 2) {
          float u[16];
          tc_ld16(tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)(acc * S::ACC_COLS + TN + c0), u);
          const int f = row_tile * 128 + row_in_tile;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int tok = tok0 + c0 + i;
            const float g = v[i];
            if (f < n_out && tok < M) o[(size_t)tok * ldo + f] = from_float<TO>(glu_value(g, u[i], glu));
          }
        } else if (SWIGLU) {
          // The upper two warps (up rows) hand their values to the lower two (gate rows of the
          // same features) through shared memory; both directions are barriers with a time limit.
          if (quarter >= 2) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_xempty, (n_chunk & 1) ^ 1, abort_flag, status, 5));
            if (!ok) break;
#pragma unroll
            for (int i = 0; i < 16; ++i) xch[(row_in_tile - 64) * 17 + i] = v[i];
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_xfull);
          } else {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_xfull, n_chunk & 1, abort_flag, status, 6));
            if (!ok) break;
            const int f = row_tile * 64 + row_in_tile;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int tok = tok0 + c0 + i;
              const float up = xch[row_in_tile * 17 + i];
              const float g = v[i];
              if (f < n_out && tok < M) o[(size_t)tok * ldo + f] = from_float<TO>(glu_value(g, up, glu));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_xempty);
          }
        } else {
          const int f = row_tile * R + row_in_tile;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int tok = tok0 + c0 + i;
            if (f < n_out && tok < M) o[(size_t)tok * ldo + f] = from_float<TO>(v[i]);
          }
        }
      }
      if (!ok) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_tempty + 8 * acc);
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((unsigned)S::TMEM_COLS)
                 : "memory");
  }
}

// A map over the stacked gate|up matrix [2 I, K] as [I / 16][gate, up][16][K]: a box is 64 of K of 64 features' rows, gate and up in
// turns of 16.
int get_gated_map(const void *W, long long I, long long K, CUtensorMap *out) {
  EncodeTiledFn fn = encode_fn();
  LLM_REQUIRE(fn != nullptr, "tensor map: the driver does not offer cuTensorMapEncodeTiled");
  const cuuint64_t dims[4] = {(cuuint64_t)K, 16, 2, (cuuint64_t)(I / 16)};
  const cuuint64_t strides[3] = {(cuuint64_t)K * 2, (cuuint64_t)(I * K) * 2, (cuuint64_t)K * 32};
  const cuuint32_t box[4] = {(cuuint32_t)TC_BK, 16, 2, 4};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(W), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  LLM_REQUIRE(r == CUDA_SUCCESS, "tensor map: cuTensorMapEncodeTiled failed (%d) for a gated matrix of %lld x %lld", (int)r, I, K);
  return LLM_OK;
}

template <int TN, int SW, typename TO, int R = TC_ROWS, int KBS = 1>
int launch_tc(const void *x, long long ldx, const void *W, void *out, long long ldo, int M, int N, int K, int k_parts,
              long long part_stride, const GluShape &glu, int *status, cudaStream_t stream, int n_groups = 1, int group_n = 0) {
  using S = TcShape<TN, SW, R, KBS>;
  const int n_out = SW != 0 ? N / 2 : N;
  const int rows_out = SW == 1 || SW == 3 ? 64 : R;
  const int row_tiles = (n_out + rows_out - 1) / rows_out;
  const int tok_tiles = (M + TN - 1) / TN;
  const int n_kblocks = (K + TC_BK - 1) / TC_BK;
  const int kb_per_part = (n_kblocks + k_parts - 1) / k_parts;
  LLM_REQUIRE((long long)(k_parts - 1) * kb_per_part < n_kblocks, "gemm_tc: %d parts leave one of them without work (K = %d)", k_parts, K);
  CUtensorMap map_w, map_x;
  int rc = SW == 3 ? get_gated_map(W, n_out, K, &map_w) : get_map(W, N, K, K, SW == 2 || KBS > 1 ? R : 64, &map_w);
  if (rc != LLM_OK) return rc;
  rc = get_map(x, (long long)n_groups * M, K, ldx, TN, &map_x);
  if (rc != LLM_OK) return rc;
  auto kern = gemm_tc_kernel<TN, SW, TO, R, KBS>;
  LLM_CHECK_CUDA(llm_allow_smem(kern, S::SMEM), "gemm_tc attribute");
  const long long tiles = (long long)row_tiles * tok_tiles * k_parts;
  LLM_REQUIRE(tiles < (1ll << 30), "gemm_tc: too many tiles");
  const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
  LLM_CHECK_CUDA(llm_launch(kern, dim3(grid), dim3(TC_THREADS), S::SMEM, stream, map_w, map_x, (TO *)out, ldo, M, n_out, K,
                            row_tiles, tok_tiles, k_parts, kb_per_part, part_stride, n_groups > 1 ? group_n / 128 : row_tiles,
                            n_groups > 1 ? M : 0, glu, status),
                 "gemm_tc launch");
  return LLM_OK;
}

// ---------------------------------------------------------------- the gated unit of a prompt step, two SMs to a tile
// At thousands of tokens a tile's operands, not its products, are what one SM cannot bring in fast enough: 256 rows of W x
// 128 tokens need 48 KB per 64 of K, 94 bytes a cycle at the tensor cores' rate, and an SM's loads end at 64.  Here a
// cluster of two CTAs works on one tile of 256 rows of W x 256 tokens (tcgen05 cta_group::2): each brings half of the
// rows and half of the tokens, 32 KB for the same products, 64 bytes a cycle, and each holds the accumulator of its own 128 rows.
// The CTA of even rank issues the products of both; its barriers count what both have loaded and read.
//
// A CTA's 128 rows are gate and up rows of 64 features in turns of 16 (one four-dimensional box of the map), so that the
// epilogue's warps hold a feature's gate in lane l < 16 and its up in lane l + 16: the two trade every other
// token by shuffles, each lane then has both values of 8 tokens in 16, and nothing passes through shared memory.
// 2,048 tokens x [16,384, 2,048]: 118 us on one SM a tile, 92 here (1.49 PFLOP/s; the library product and its pass 136); 8,192 x
// [28,672, 4,096]: 1,247 (the library's 1,544 + 215).
constexpr int GP_FEATURES = 64;                // of one CTA; a pair has 128
constexpr int GP_TOKENS = 256;                 // of the pair; each CTA loads 128
constexpr int GP_HALF_BYTES = 128 * TC_BK * 2; // a CTA's rows, or its tokens, of one stage
constexpr int GP_STAGES = 6;
// Eight epilogue warps, two to a quarter of the lanes (128 tokens each): with four, the gated unit of a tile (an exponential, a
// division, a shuffle and a store for each of 16,384 values) took longer than its products at K = 2,048 (115.7 us a launch at
// 2,048 tokens instead of 92).
constexpr int GP_THREADS = 64 + 256;
constexpr size_t GP_SMEM = 1024 + (size_t)GP_STAGES * 2 * GP_HALF_BYTES + 256;

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned in_cta(unsigned addr, unsigned rank) {      // the same place in the shared memory of a CTA of the cluster
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename TO>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
gated_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, TO *__restrict__ out, long long ldo,
                  int M, int n_out, int K, int row_tiles, int tok_tiles, GluShape glu, int *status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned long long *bars = (unsigned long long *)(smem + (size_t)GP_STAGES * 2 * GP_HALF_BYTES);
  const unsigned bar_full = smem_u32(bars), bar_empty = smem_u32(bars + GP_STAGES);
  const unsigned bar_tfull = smem_u32(bars + 2 * GP_STAGES), bar_tempty = smem_u32(bars + 2 * GP_STAGES + 2);
  unsigned *tmem_slot = (unsigned *)(bars + 2 * GP_STAGES + 4);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const unsigned rank = cluster_rank();
  grid_dependents_launch();
  if (threadIdx.x == 0) {
    for (int s = 0; s < GP_STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);          // rank 0's: its loader, and the bytes of both
      mbar_init(bar_empty + 8 * s, 1);         // each CTA's own: the products that read the stage, committed to both
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar_tfull + 8 * a, 1);         // each CTA's own
      mbar_init(bar_tempty + 8 * a, 16);       // rank 0's: the epilogue warps of both
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tma_prefetch_map(&map_w);
    tma_prefetch_map(&map_x);
  }
  if (warp == 1) {                             // in both CTAs: the pair's tensor memory is allocated together
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                              // both CTAs' barriers are there before anyone signals the other's
  tc_fence_after();
  const unsigned tmem_base = *tmem_slot;

  const int n_tiles = row_tiles * tok_tiles, n_kblocks = (K + TC_BK - 1) / TC_BK;
  const int first = blockIdx.x / 2, step = gridDim.x / 2;      // this pair's tiles

  if (warp == 0) {
    // ------------------------------------------------------------ loader: this CTA's half of both operands
    const bool leader = elect_one();
    struct Walk {
      int tile, kb;
      bool valid;
    };
    auto next = [&](Walk &w) {
      if (++w.kb >= n_kblocks) {
        w.tile += step;
        w.kb = 0;
        w.valid = w.tile < n_tiles;
      }
    };
    auto load_w = [&](const Walk &w, int stage) {
      if (!leader) return;
      const unsigned full = in_cta(bar_full + 8 * stage, 0);
      if (rank == 0) mbar_expect_tx(bar_full + 8 * stage, 4 * GP_HALF_BYTES);
      const int group = ((w.tile / tok_tiles) * 2 + (int)rank) * (GP_FEATURES / 16);
      asm volatile(
          "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %3, %4}], [%5];"
          ::"r"(smem_u32(smem + (size_t)stage * 2 * GP_HALF_BYTES)), "l"(&map_w), "r"(w.kb * TC_BK), "r"(0), "r"(group), "r"(full) : "memory");
    };
    auto load_x = [&](const Walk &w, int stage) {
      if (!leader) return;
      const unsigned full = in_cta(bar_full + 8 * stage, 0);
      asm volatile(
          "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
          ::"r"(smem_u32(smem + (size_t)stage * 2 * GP_HALF_BYTES) + GP_HALF_BYTES), "l"(&map_x), "r"(w.kb * TC_BK),
          "r"(w.tile % tok_tiles * GP_TOKENS + (int)rank * 128), "r"(full) : "memory");
    };
    // weights before the dependency is waited for, tokens after it
    Walk w{first, 0, first < n_tiles}, w2 = w;
    int n_pre = 0;
    for (; w.valid && n_pre < GP_STAGES; next(w), ++n_pre) load_w(w, n_pre);
    grid_dependency_wait();
    for (int s = 0; s < n_pre; ++s, next(w2)) load_x(w2, s);
    int stage = n_pre % GP_STAGES;
    unsigned phase = n_pre == GP_STAGES ? 1u : 0u;
    bool ok = true;
    for (; w.valid; next(w)) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, status, 1));
      if (!ok) break;
      load_w(w, stage);
      load_x(w, stage);
      if (++stage == GP_STAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
    if (!ok) {                                 // given up: what is in flight lands within this time, whoever's barrier it signals
      const unsigned long long t0 = globaltimer();
      while (globaltimer() - t0 < 2000000ull) {
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ products of both CTAs, issued by rank 0
    const bool leader = elect_one();
    constexpr unsigned IDESC = instr_desc(256, GP_TOKENS);
    auto commit = [&](unsigned bar) {          // arrives at this barrier in both CTAs when the products so far are done
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                   ::"r"(bar), "h"((unsigned short)3) : "memory");
    };
    int stage = 0, iter = 0;
    unsigned phase = 0;
    bool ok = rank == 0;
    for (int tile = first; tile < n_tiles && ok; tile += step, ++iter) {
      const int acc = iter & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(bar_tempty + 8 * acc, ((iter >> 1) & 1) ^ 1, abort_flag, status, 2));
      if (!ok) break;
      tc_fence_after();
      const unsigned d_tmem = tmem_base + acc * GP_TOKENS;
      for (int kb = 0; kb < n_kblocks; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * stage, phase, abort_flag, status, 3));
        if (!ok) break;
        tc_fence_after();
        const unsigned a_addr = smem_u32(smem + (size_t)stage * 2 * GP_HALF_BYTES);
        const unsigned long long a_desc = smem_desc(a_addr), b_desc = smem_desc(a_addr + GP_HALF_BYTES);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < TC_BK / 16; ++kk)
            asm volatile(
                "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
                ::"r"(d_tmem), "l"(a_desc + (unsigned long long)(kk * 2)), "l"(b_desc + (unsigned long long)(kk * 2)), "r"(IDESC),
                "r"(kk > 0 || kb > 0 ? 1u : 0u) : "memory");
          commit(bar_empty + 8 * stage);
        }
        __syncwarp();
        if (++stage == GP_STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok && leader) commit(bar_tfull + 8 * acc);
      __syncwarp();
    }
    grid_dependency_wait();
  } else {
    // ------------------------------------------------------------ epilogue of this CTA's 128 rows (warps 2..9)
    grid_dependency_wait();
    const int quarter = warp & 3, half = (warp - 2) / 4;       // the lanes of tensor memory the warp may read; its half of the tokens
    constexpr int CHUNKS = GP_TOKENS / 32;
    int iter = 0;
    for (int tile = first; tile < n_tiles; tile += step, ++iter) {
      const int acc = iter & 1, tok0 = tile % tok_tiles * GP_TOKENS + half * (GP_TOKENS / 2);
      if (!__all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * acc, (iter >> 1) & 1, abort_flag, status, 4))) break;
      tc_fence_after();
      const int f = ((tile / tok_tiles) * 2 + (int)rank) * GP_FEATURES + quarter * 16 + (lane & 15);
      const unsigned taddr = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)(acc * GP_TOKENS + half * (GP_TOKENS / 2));
      float even[16], odd[16];
#pragma unroll 1
      for (int c = 0; c < CHUNKS; c += 2) {          // two loads on their way, none from one round to the next
        tc_ld16_issue(taddr + c * 16, even);
        tc_ld16_issue(taddr + (c + 1) * 16, odd);
        tc_ld_wait();
        tc_ld_ready(even);
        tc_ld_ready(odd);
        store_turns(even, out, ldo, f, n_out, tok0 + c * 16, M, glu);
        store_turns(odd, out, ldo, f, n_out, tok0 + (c + 1) * 16, M, glu);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_cta(bar_tempty + 8 * acc, 0)) : "memory");
    }
  }

  // ---------------------------------------------------------------- teardown: neither CTA leaves while the other may signal it
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

template <typename TO>
int launch_gated_pair(const void *x, long long ldx, const void *W, void *out, long long ldo, int M, int n_out, int K, const GluShape &glu,
                      int *status, cudaStream_t stream) {
  CUtensorMap map_w, map_x;
  int rc = get_gated_map(W, n_out, K, &map_w);
  if (rc != LLM_OK) return rc;
  rc = get_map(x, M, K, ldx, 128, &map_x);
  if (rc != LLM_OK) return rc;
  const int row_tiles = (n_out + 2 * GP_FEATURES - 1) / (2 * GP_FEATURES), tok_tiles = (M + GP_TOKENS - 1) / GP_TOKENS;
  const long long tiles = (long long)row_tiles * tok_tiles;
  LLM_REQUIRE(tiles < (1ll << 30), "gemm_tc: too many tiles");
  const int pairs = (int)(tiles < sm_count() / 2 ? tiles : sm_count() / 2);
  auto kern = gated_pair_kernel<TO>;
  LLM_CHECK_CUDA(llm_allow_smem(kern, GP_SMEM), "gemm_tc attribute");
  LLM_CHECK_CUDA(llm_launch(kern, dim3(2 * pairs), dim3(GP_THREADS), GP_SMEM, stream, map_w, map_x, (TO *)out, ldo, M, n_out, K, row_tiles,
                            tok_tiles, glu, status),
                 "gemm_tc launch");
  return LLM_OK;
}

// Whether the gated unit of M tokens and a stacked matrix of N rows runs two SMs to a tile: whole groups of 16 features (the map),
// tiles for most pairs of SMs, and 512 tokens or more of which the last tile does not waste a fifth.  Measured against the library product and
// its pass ([16,384, 2,048]): 300 tokens 45 us against 28, 512 34 against 40, 773 (of 1,024) 66 against 59, 1,024 56 against 72; with tiles for
// half of the pairs ([2,048, 512], 1,024 tokens) 15 against 12.
bool takes_pair(int M, int N) {
  const long long tok_tiles = (M + GP_TOKENS - 1) / GP_TOKENS, row_tiles = (N / 2 + 2 * GP_FEATURES - 1) / (2 * GP_FEATURES);
  return N % 32 == 0 && M >= 512 && tok_tiles * GP_TOKENS * 4 <= (long long)M * 5 && tok_tiles * row_tiles * 2 >= sm_count();
}

// Rows of W to a tile of a plain product of few tokens: as many fewer than 128 as still leave every SM at most one tile (TcShape).
int tile_rows(int N, int k_parts) {
  const long long tiles = (long long)((N + TC_ROWS - 1) / TC_ROWS) * k_parts;
  return tiles * 4 <= sm_count() ? 32 : tiles * 2 <= sm_count() ? 64 : TC_ROWS;
}

template <bool SWIGLU, typename TO>
int dispatch_tc(const void *x, long long ldx, const void *W, void *out, long long ldo, int M, int N, int K, int k_parts,
                long long part_stride, const GluShape &glu, int *status, cudaStream_t stream) {
#define TC_GO(TN, SW) return launch_tc<TN, SW, TO>(x, ldx, W, out, ldo, M, N, K, k_parts, part_stride, glu, status, stream)
  if (SWIGLU) {
    if (M <= 64 && N / 2 % 16 == 0) {
      if (M <= 16) return launch_tc<16, 3, TO, TC_ROWS, 2>(x, ldx, W, out, ldo, M, N, K, k_parts, part_stride, glu, status, stream);
      if (M <= 32) TC_GO(32, 3);
      TC_GO(64, 3);
    }
    if (M <= 16) TC_GO(16, 1);
    if (M <= 32) TC_GO(32, 1);
    if (M <= 64) TC_GO(64, 1);
    if (takes_pair(M, N)) return launch_gated_pair<TO>(x, ldx, W, out, ldo, M, N / 2, K, glu, status, stream);
    TC_GO(128, 2);
  }
#define TC_NARROW(TN, R, KBS) return launch_tc<TN, 0, TO, R, KBS>(x, ldx, W, out, ldo, M, N, K, k_parts, part_stride, glu, status, stream)
  const int rows = M <= 48 ? tile_rows(N, k_parts) : TC_ROWS;
  if (rows == 32 && M <= 16) TC_NARROW(16, 32, 4);
  if (rows == 32 && M <= 32) TC_NARROW(32, 32, 4);
  if (rows == 64 && M <= 16) TC_NARROW(16, 64, 2);
  if (rows == 64 && M <= 32) TC_NARROW(32, 64, 2);
  if (rows <= 64) TC_NARROW(64, 64, 2);
#undef TC_NARROW
  if (M <= 16) TC_GO(16, 0);
  if (M <= 32) TC_GO(32, 0);
  if (M <= 64) TC_GO(64, 0);
  if (M <= 128) TC_GO(128, 0);
  TC_GO(256, 0);
#undef TC_GO
}

}  // namespace

// How many parts of K a product with this few rows of W should be cut into so that most SMs have a
// tile; 1 when the matrix has tiles enough.  The caller adds the parts (32-bit) in order.
LLM_EXPORT int llm_gemm_tc_suggest_parts(int M, int N, int K) {
  const int tok_tiles = M <= 256 ? 1 : (M + 255) / 256;
  const int tiles = ((N + 127) / 128) * tok_tiles;
  const int kblocks = (K + TC_BK - 1) / TC_BK;
  // the most parts (up to 8) that still leave every SM at most one tile and every part at least
  // four K blocks, none of them empty
  // Above 32 tokens the parts themselves weigh (8 parts of 64 tokens x 2,048 features are 4 MB to
  // write and to read again): four at most (batch 64: 1.735 -> 1.687 ms a step; at 32 tokens eight
  // are still better, 1.297 against 1.350 ms).
  const int cap = M > 32 ? 4 : 8;
  const int most = sm_count() / (tiles > 0 ? tiles : 1) < cap ? sm_count() / (tiles > 0 ? tiles : 1) : cap;
  int parts = 1;
  for (int p = 2; p <= most; ++p) {
    const int per = (kblocks + p - 1) / p;
    if (per >= 4 && (p - 1) * per < kblocks) parts = p;
  }
  return parts;
}

// 1 if the gated unit of these sizes runs two SMs to a tile.
LLM_EXPORT int llm_gemm_tc_pairs(int M, int N) { return takes_pair(M, N); }

// x [M, K] bfloat16 (row stride ldx elements), W [N, K] bfloat16 contiguous, out [M, N] of out_dtype,
// or [M, N/2] with swiglu (W = stacked gate|up).  With k_parts > 1 (plain product, 32-bit out) part p
// writes its share of K to out + p * part_stride.  `status` (device int, may be null) receives a
// non-zero code if a wait inside the kernel ran out of time.  With swiglu the gated unit is (limit, slope, shift)'s (GluShape).
LLM_EXPORT int llm_gemm_tc_glu(const void *x, long long ldx, const void *W, void *out, long long ldo, int out_dtype,
                               int M, int N, int K, int swiglu, float limit, float slope, float shift, int k_parts, long long part_stride,
                               int *status, cudaStream_t stream) {
  const GluShape glu{limit, slope, shift};
  if (M == 0 || N == 0) return LLM_OK;
  LLM_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_tc: bad sizes %d x %d x %d", M, N, K);
  LLM_REQUIRE(K % 8 == 0 && ldx % 8 == 0, "gemm_tc: K = %d and the row stride %lld must be multiples of 8 (rows start on 16 bytes)", K, ldx);
  LLM_REQUIRE((uintptr_t)x % 16 == 0 && (uintptr_t)W % 16 == 0, "gemm_tc: operands must be 16-byte aligned");
  LLM_REQUIRE(!swiglu || N % 2 == 0, "gemm_tc: a stacked gate|up matrix has an even number of rows");
  LLM_REQUIRE(k_parts >= 1 && k_parts <= 64 && (k_parts == 1 || (!swiglu && out_dtype == LLM_F32)),
              "gemm_tc: parts of K need a plain product with 32-bit output");
  if (swiglu) {
    if (out_dtype == LLM_BF16) return dispatch_tc<true, __nv_bfloat16>(x, ldx, W, out, ldo, M, N, K, k_parts, part_stride, glu, status, stream);
    if (out_dtype == LLM_F32) return dispatch_tc<true, float>(x, ldx, W, out, ldo, M, N, K, k_parts, part_stride, glu, status, stream);
  } else {
    if (out_dtype == LLM_BF16) return dispatch_tc<false, __nv_bfloat16>(x, ldx, W, out, ldo, M, N, K, k_parts, part_stride, glu, status, stream);
    if (out_dtype == LLM_F32) return dispatch_tc<false, float>(x, ldx, W, out, ldo, M, N, K, k_parts, part_stride, glu, status, stream);
  }
  LLM_FAIL("gemm_tc: unknown output dtype %d", out_dtype);
}

LLM_EXPORT int llm_gemm_tc(const void *x, long long ldx, const void *W, void *out, long long ldo, int out_dtype,
                           int M, int N, int K, int swiglu, int k_parts, long long part_stride, int *status,
                           cudaStream_t stream) {
  return llm_gemm_tc_glu(x, ldx, W, out, ldo, out_dtype, M, N, K, swiglu, __builtin_huge_valf(), 1.f, 0.f, k_parts, part_stride, status, stream);
}

// Several products of as many inputs in one launch: x [n_groups * M, K] (input g's rows from g * M on), W the matrices one
// behind the other, each but the last of group_n rows (a multiple of 128, so that a tile has one input), N rows in all;
// out [M, N] 32-bit.
LLM_EXPORT int llm_gemm_tc_grouped(const void *x, long long ldx, const void *W, float *out, long long ldo, int M, int N, int K, int n_groups,
                                   int group_n, int *status, cudaStream_t stream) {
  if (M == 0 || N == 0) return LLM_OK;
  LLM_REQUIRE(M > 0 && N > 0 && K > 0 && n_groups >= 1, "gemm_tc_grouped: bad sizes %d x %d x %d", M, N, K);
  LLM_REQUIRE(n_groups == 1 || (group_n > 0 && group_n % 128 == 0 && (long long)(n_groups - 1) * group_n < N && (long long)n_groups * group_n >= N),
              "gemm_tc_grouped: %d matrices of %d rows do not make %d", n_groups, group_n, N);
  LLM_REQUIRE(K % 8 == 0 && ldx % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)W % 16 == 0, "gemm_tc_grouped: rows must start on 16 bytes");
#define TC_GROUP(TN) return launch_tc<TN, 0, float>(x, ldx, W, out, ldo, M, N, K, 1, 0, GluShape{}, status, stream, n_groups, group_n)
  if (M <= 16) TC_GROUP(16);
  if (M <= 32) TC_GROUP(32);
  if (M <= 64) TC_GROUP(64);
  if (M <= 128) TC_GROUP(128);
  TC_GROUP(256);
#undef TC_GROUP
}

// ---------------------------------------------------------------- a wait that runs out, for tests
// One warp waits, through the same bounded wait as the product's warps, on a barrier that nobody
// arrives on: no copy and no tensor memory is in flight.  After `limit_ns` the wait gives up,
// records code 9 in `status` and the kernel returns by itself.  It shows that a wait that runs out
// leaves the device usable and is seen by the host; nothing else launches it.
__global__ void wait_probe_kernel(unsigned long long limit_ns, int *status) {
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  mbar_wait_limit(smem_u32(&bar), 0, &abort_flag, status, 9, limit_ns);
}

LLM_EXPORT int llm_gemm_tc_wait_probe(long long limit_ns, int *status, cudaStream_t stream) {
  LLM_REQUIRE(limit_ns > 0 && limit_ns <= 100000000ll, "wait_probe: the limit must lie in (0, 100 ms]");
  LLM_REQUIRE(status != nullptr, "wait_probe: no status word");
  wait_probe_kernel<<<1, 32, 0, stream>>>((unsigned long long)limit_ns, status);
  LLM_CHECK_LAUNCH("wait_probe");
  return LLM_OK;
}
