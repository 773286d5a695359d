// C[M,N] = A[M,K] . W[N,K]^T in bfloat16 on the 5th-generation tensor cores (tcgen05), for many rows
// (prefill).  Blocks are persistent: as many as the GPU holds, each walking tiles of 128 x BN of C
// (BN 256, 192, 160 or 128, see tc_tile_columns), in bands of 8 n-tiles (n-tile fastest
// inside a band, see tc_tile), so that blocks running side by side share operand tiles:
//
//   warp 0, one lane   TMA producer: 128x64 tiles of A and BNx64 tiles of W into a ring of shared-memory
//                      stages (cp.async.bulk.tensor, 128-byte swizzle, completion counted on an mbarrier)
//   warp 1             MMA issuer (one lane issues): per stage four tcgen05.mma (M 128, N BN, K 16) straight from shared
//                      memory into a float accumulator in tensor memory; tcgen05.commit hands the stage
//                      back to the producer and, after the last k-block, the accumulator to the epilogue
//   warps 2..9         epilogue: tcgen05.ld of the accumulator (each warp its 32 lanes = 32 rows of C, and one half of
//                      the columns; warps 2..5 of a split product all of them), conversion, guarded stores
//
// There are two accumulators in tensor memory (2 x BN columns): the epilogue of one tile runs while
// the next tile's products are issued.
//
// Both operands are K-major, which is how activations and checkpoint weights already lie in memory,
// so nothing is re-tiled at load.  Rows past M (or past a group's end) and k past K are zero-filled
// by TMA and masked at the store.
//
// Grouped form (routed experts): rows of A are already sorted by group and contiguous; group e owns
// rows [offsets[e], offsets[e+1]) and multiplies them with W[e].  Row tiles are counted per group, so
// a tile never mixes groups in its stored rows.
//
// Every wait on an mbarrier is bounded by wall time: when it runs out the block records an error
// code (see snk_gemm_tc_status), issues no more loads and products, gives the copies in flight a moment
// to land, frees its tensor memory and returns.  snk_gemm_tc_test_lose_loads makes that happen for a test:
// the producers then issue no loads, so the waits for operands run out.
// (the role of snowllm/ops/gemm.py:33-41 and the expert products of snowllm/ops/inference.py:60-76
// at prefill shapes)
#include "tma.cuh"
#include "tcgen05.cuh"

#define TC_BM 128
#define TC_BK 64
// Epilogue warps: two to each 32 lanes of tensor memory, which share a tile's columns; one where a product is split along K, whose
// blocks have one short tile each and are soon followed by other kernels' on the same SMs (with two the kernel alone is as fast, but
// in a chain of norm, gated product and product, us, two / one: 2,048 x 1,536 200 rows 26.1 / 23.8, 2,048 x 1,024 129 rows 24.1 / 22.0, 1,024 x
// 1,408 64 rows 17.3 / 18.1).
#define TC_EPI_WARPS 8
#define TC_SPLIT_EPI_WARPS 4
#define TC_SMEM_TILES (192 * 1024)    // bytes of shared memory given to the operand stages
#ifndef TC_BAND
#define TC_BAND 8                     // n-tiles in a band of the tile order (8, 16 and 28 measured; 8 is best or equal everywhere)
#endif
#define TC_WAIT_NS 1500000000ull      // 1.5 s per wait before giving up

enum { TC_ERR_WAIT_FULL = 1, TC_ERR_WAIT_EMPTY = 2, TC_ERR_WAIT_ACC = 3, TC_ERR_WAIT_ACC_FREE = 4 };

__device__ int g_tc_status;            // 0, or the first error code a block recorded
__device__ int g_tc_lose_loads;        // test hook: producers issue no loads (the operands then never arrive)

// Wait for a phase, for TC_WAIT_NS at most.  False: the wait ran out, or another one of the block has (`aborted`, shared).
__device__ __noinline__ bool mbar_wait_long(uint64_t* bar, uint32_t parity, volatile int* aborted, int code) {
  const uint64_t start = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (*aborted) return false;
    if (global_ns() - start > TC_WAIT_NS) {
      *aborted = 1;
      atomicCAS(&g_tc_status, 0, code);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* aborted, int code) {
  return mbar_try_wait(bar, parity) || mbar_wait_long(bar, parity, aborted, code);
}
// The same by all lanes of a warp, which come out together and with one answer.  Lanes that waited each for itself could fall
// apart (nothing joins them again in a loop that is left by a failed wait): one that comes two phases late waits for a phase that
// never comes, and the aligned instructions behind the loops want whole warps.  (One vote a k-block, for the 512 cycles of its products:
// in turn with the loop of one issuing lane, us, that / so, 8,192 x 6,144 x 2,048 169 / 159, 1,024 x 2,048 x 8,192 54.1 / 49.2.)
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* aborted, int code) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, aborted, code));
}

#define TC_MAX_STAGES 6

template <int EPI>
struct __align__(16) TcShared {
  uint64_t full[TC_MAX_STAGES];
  uint64_t empty[TC_MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int aborted;
  __align__(16) float stage_out[EPI][TC_STAGE_FLOATS];    // one staging tile per epilogue warp (tc_store_piece)
};

// Rows of C and rows of W that tile `tile` covers.  Plain: tiles = row_tiles * n_tiles, row tile fastest.
// Grouped: row tiles are counted group by group (a tile never spans two groups).
struct TcTile {
  int row0, row_end, w_row0, n0;
  bool valid;
};

__device__ __forceinline__ TcTile tc_tile(int tile, int row_tiles, int M, int N, int BN, const int* offsets,
                                          int groups) {
  TcTile t;
  // Tiles are numbered in bands of up to TC_BAND n-tiles: inside a band the n-tile runs fastest, then the row
  // tile; then the next band.  Blocks that run side by side so share a row tile of A and read neighbouring
  // tiles of W (measured against row tiles fastest: +6 % on 2048 x 6144 x 2048, +6 to +8 % on the experts'
  // products; one band over all of a wide N lost 8 % on 2048 x 14336 x 2048).
  const int n_tiles = (N + BN - 1) / BN;
  const int bands = (n_tiles + TC_BAND - 1) / TC_BAND;
  const int band_w = (n_tiles + bands - 1) / bands;
  const int per_band = row_tiles * band_w;
  const int band = tile / per_band, in_band = tile % per_band;
  const int w_here = min(band_w, n_tiles - band * band_w);   // the last band may be narrower
  const int rt = in_band / w_here, nt = band * band_w + in_band % w_here;
  t.n0 = nt * BN;
  t.valid = t.n0 < N;
  if (!offsets) {
    t.row0 = rt * TC_BM;
    t.row_end = M;
    t.w_row0 = 0;
    return t;
  }
  int left = rt;
  t.valid = false;
  t.row0 = t.row_end = t.w_row0 = 0;
  if (nt * BN >= N) return t;
  for (int e = 0; e < groups; ++e) {
    const int begin = offsets[e], cnt = offsets[e + 1] - begin;
    const int tiles_e = (cnt + TC_BM - 1) / TC_BM;
    if (left < tiles_e) {
      t.row0 = begin + left * TC_BM;
      t.row_end = begin + cnt;
      t.w_row0 = e * N;
      t.valid = true;
      return t;
    }
    left -= tiles_e;
  }
  return t;
}

// SWIGLU: W holds gate and up rows interleaved in blocks of 8 (rows 16j..16j+7: gate of features
// 8j..8j+7, rows 16j+8..16j+15: their up rows); the store is act(gate) * up into C[M, N/2], act by the code
// that the entry point's `swiglu` argument carries (1 silu, 2 relu, 3 gelu in its tanh form).
// ADD (float): the product is added to what C holds (the stream that a sublayer's output belongs to).
template <int BN, typename OutT, bool SWIGLU, bool ADD, int EPI>
__global__ void __launch_bounds__(64 + 32 * EPI, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
               OutT* __restrict__ C, int M, int N, int K, const int* __restrict__ offsets, int groups,
               int row_tiles_bound, int splits, int act, int w_ahead) {
  constexpr int STAGE_BYTES = (TC_BM + BN) * TC_BK * 2;
  constexpr int STAGES = TC_SMEM_TILES / STAGE_BYTES < TC_MAX_STAGES ? TC_SMEM_TILES / STAGE_BYTES : TC_MAX_STAGES;
  constexpr uint32_t TMEM_COLS = BN <= 128 ? 256 : 512;    // two accumulators, in a power of two of columns
  static_assert(BN % 32 == 0 && BN <= 256, "pieces of 32 columns");
  extern __shared__ unsigned char smem_raw[];
  // tiles need 1024-byte alignment for the 128-byte swizzle
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  TcShared<EPI>* sh = reinterpret_cast<TcShared<EPI>*>(tiles + (size_t)STAGES * STAGE_BYTES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_tiles = (K + TC_BK - 1) / TC_BK;

  // Barriers and tensor memory are set up before the wait for the kernel in front: none of it touches
  // global memory, and it then overlaps with that kernel's tail.
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->acc_full[b], 1);
      mbar_init(&sh->acc_empty[b], EPI);                 // one arrival per epilogue warp
    }
    sh->aborted = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {                                       // one warp allocates both accumulators
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&sh->tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_acc = sh->tmem_base;
  volatile int* aborted = &sh->aborted;
  // w_ahead (plain products): W was there before the kernel in front of this launch began, so its tiles of the first
  // ring of k-blocks are on their way before the wait, and only A's follow after it.  Replayed chains of a norm and the
  // product, without / with: 17 rows 2,048 x 1,792 11.4 / 10.4 us, 64 rows 2,048 x 2,048 11.6 / 11.5, gate|up and down of 1,024 and 2,816
  // 23.6 / 22.4, but 6,144 x 2,048 14.1 / 14.5; over 150 sizes of 17 to 1,024 rows 1.2 % less, 9 % at best, 4 % more at worst;
  // the 64-request decode step of the 8B-A1B sizes 4,890 / 4,868 us.
  int early = 0;
  if (w_ahead && !offsets && threadIdx.x == 0 && *const_cast<volatile int*>(&g_tc_lose_loads) == 0) {
    const int total = row_tiles_bound * ((N + BN - 1) / BN), k_per = (k_tiles + splits - 1) / splits;
    if ((int)blockIdx.x < total * splits) {
      const TcTile t = tc_tile(blockIdx.x % total, row_tiles_bound, M, N, BN, offsets, groups);
      const int kt_begin = (blockIdx.x / total) * k_per, kt_end = min(k_tiles, kt_begin + k_per);
      for (; t.valid && early < STAGES && kt_begin + early < kt_end; ++early) {
        mbar_expect_tx(&sh->full[early], STAGE_BYTES);
        tma_load_2d(tiles + (size_t)early * STAGE_BYTES + TC_BM * TC_BK * 2, &map_w, &sh->full[early],
                    (kt_begin + early) * TC_BK, t.w_row0 + t.n0);
      }
    }
  }
  pdl_begin();
  // number of row tiles: known for the plain product, counted from the offsets for the grouped one
  int row_tiles = row_tiles_bound;
  if (offsets) {
    row_tiles = 0;
    for (int e = 0; e < groups; ++e) row_tiles += (offsets[e + 1] - offsets[e] + TC_BM - 1) / TC_BM;
  }
  const int n_tiles = (N + BN - 1) / BN;
  const int total = row_tiles * n_tiles;
  // splits > 1 (plain products with few tiles): work item w is tile w % total over the k-blocks of part
  // w / total, and the partial product goes to plane w / total of C, which then is float [splits, M, N]
  const int items = total * splits;
  const int k_per = (k_tiles + splits - 1) / splits;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;                                        // k-blocks issued so far, over all tiles
      const bool lose_loads = *const_cast<volatile int*>(&g_tc_lose_loads) != 0;
      for (int item = blockIdx.x; item < items && !*aborted; item += gridDim.x) {
        const TcTile t = tc_tile(item % total, row_tiles, M, N, BN, offsets, groups);
        if (!t.valid) continue;
        const int kt_begin = (item / total) * k_per, kt_end = min(k_tiles, kt_begin + k_per);
        for (int kt = kt_begin; kt < kt_end; ++kt, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(&sh->empty[s], ((it / STAGES) & 1) ^ 1, aborted, TC_ERR_WAIT_EMPTY)) break;   // nothing more is issued
          if (lose_loads) continue;
          unsigned char* stage = tiles + (size_t)s * STAGE_BYTES;
          if (it >= early) mbar_expect_tx(&sh->full[s], STAGE_BYTES);
          tma_load_2d(stage, &map_a, &sh->full[s], kt * TC_BK, t.row0);
          if (it >= early) tma_load_2d(stage + TC_BM * TC_BK * 2, &map_w, &sh->full[s], kt * TC_BK, t.w_row0 + t.n0);
        }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_bf16(TC_BM, BN), elected = elect_lane();
    const uint32_t ring_lo = smem_desc_lo(smem_u32(tiles)), empty0 = smem_u32(&sh->empty[0]);
    int s = 0, local = 0;
    uint32_t lap = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const TcTile t = tc_tile(item % total, row_tiles, M, N, BN, offsets, groups);
      if (!t.valid) continue;
      const int kt_begin = (item / total) * k_per, kt_end = min(k_tiles, kt_begin + k_per);
      const int buf = local & 1;
      if (!mbar_wait_warp(&sh->acc_empty[buf], ((local >> 1) & 1) ^ 1, aborted, TC_ERR_WAIT_ACC_FREE)) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_acc + (uint32_t)(buf * BN);
      int kt = kt_begin;
      for (; kt < kt_end; ++kt) {
        if (!mbar_wait_warp(&sh->full[s], lap, aborted, TC_ERR_WAIT_FULL)) break;
        tc_fence_after();
        const uint32_t a_lo = ring_lo + s * (STAGE_BYTES >> 4), w_lo = a_lo + (TC_BM * TC_BK * 2 >> 4);
#pragma unroll
        for (int k = 0; k < TC_BK / 16; ++k)             // 16 k-values: 32 bytes further along the swizzled rows
          umma_bf16_lo(d_tmem, a_lo + 2 * k, w_lo + 2 * k, idesc, (kt > kt_begin || k > 0) ? 1u : 0u, elected);
        umma_commit_if(empty0 + s * 8, elected);         // the stage is free once these MMAs have read it
        if (++s == STAGES) {
          s = 0;
          lap ^= 1;
        }
      }
      if (kt < kt_end) break;                            // a wait ran out
      umma_commit_if(smem_u32(&sh->acc_full[buf]), elected);
      ++local;
    }
  } else {
    const int lane_group = warp & 3;                     // a warp reads the 32 tensor-memory lanes 32*(warp%4)..
    constexpr int STEP = EPI * 8;                        // the warps of 32 lanes take the tile's pieces of 32 columns in turns
    const int c_begin = (warp - 2) / 4 * 32;
    float* stage_out = sh->stage_out[warp - 2];
    int local = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const TcTile t = tc_tile(item % total, row_tiles, M, N, BN, offsets, groups);
      if (!t.valid) continue;
      OutT* Cp = C + (size_t)(item / total) * M * N;        // the part's plane (C itself without a split)
      const int buf = local & 1;
      TcOld<ADD> old;
      tc_load_old<ADD>(old, lane, Cp, t.row0 + lane_group * 32, t.row_end, t.n0 + c_begin, N);
      if (!mbar_wait_warp(&sh->acc_full[buf], (local >> 1) & 1, aborted, TC_ERR_WAIT_ACC)) break;
      tc_fence_after();
#pragma unroll 1
      for (int c0 = c_begin; c0 < BN; c0 += STEP) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)(buf * BN + c0), r);
        if (c0 + STEP >= BN) {                            // everything of this warp's part is in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->acc_empty[buf]);
        }
        if (!*aborted)
          tc_store_piece<OutT, SWIGLU, ADD>(r, stage_out, lane, Cp, t.row0 + lane_group * 32, t.row_end, t.n0 + c0, N, act, old);
        if (c0 + STEP < BN) tc_load_old<ADD>(old, lane, Cp, t.row0 + lane_group * 32, t.row_end, t.n0 + c0 + STEP, N);
      }
      ++local;
    }
  }
  if (*aborted) drain_after_abort();
  __syncwarp();                                          // (the deallocation wants the whole warp)
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(TMEM_COLS)
                 : "memory");
  }
}

template <int BN, typename OutT, bool SWIGLU, bool ADD = false, int EPI = TC_EPI_WARPS>
static int launch_tc(const CUtensorMap& map_a, const CUtensorMap& map_w, void* C, int M, int N, int K,
                     const int* offsets, int groups, int row_tiles, int splits, int w_ahead, cudaStream_t stream,
                     int act = SNK_GLU_SILU) {
  constexpr int STAGE_BYTES = (TC_BM + BN) * TC_BK * 2;
  constexpr int STAGES = TC_SMEM_TILES / STAGE_BYTES < TC_MAX_STAGES ? TC_SMEM_TILES / STAGE_BYTES : TC_MAX_STAGES;
  const size_t smem = 1024 + (size_t)STAGES * STAGE_BYTES + sizeof(TcShared<EPI>);
  static std::atomic<int> ready[SNK_MAX_DEVICES];
  int sms = 0;
  const int rc = snk_kernel_ready(ready, gemm_tc_kernel<BN, OutT, SWIGLU, ADD, EPI>, smem, &sms);
  if (rc) return rc;
  const long long tiles = (long long)row_tiles * ((N + BN - 1) / BN) * splits;
  const int blocks = (int)(tiles < sms ? tiles : sms);     // one block per SM (shared memory), persistent
  snk_launch(gemm_tc_kernel<BN, OutT, SWIGLU, ADD, EPI>, dim3(blocks), dim3(64 + 32 * EPI), smem, stream, map_a, map_w, static_cast<OutT*>(C), M, N, K,
                                                                 offsets, groups, row_tiles, splits, act, w_ahead);
  SNK_LAUNCH_CHECK();
  return 0;
}

// ---------------------------------------------------------------------------------------------
// Products with few tiles (one row tile, a narrow N: the projections of a 64-row decode step) would leave
// most SMs idle behind a long serial walk over K.  They are split along K into parts that run side by
// side; each part leaves its float partial product in a plane of scratch, and a second kernel adds the
// planes in part order and stores C (converted, or through SwiGLU).
template <typename OutT, bool SWIGLU, bool ADD = false>
__global__ void splitk_reduce_kernel(const float* __restrict__ parts, OutT* __restrict__ C, int M, int N, int splits,
                                     int act) {
  pdl_begin();
  const size_t plane = (size_t)M * N;
  if constexpr (SWIGLU) {
    // blocks of 16 columns: 8 gate columns, then the 8 up columns of the same features
    const size_t blocks = plane / 16;
    const size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= blocks) return;
    float g[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, u[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // four planes' vectors on their way at a time (one by one 64 rows of 3,072 columns came to 15.2 us, product and this, 13.5 so)
#pragma unroll 4
    for (int p = 0; p < splits; ++p) {
      const float4* src = reinterpret_cast<const float4*>(parts + (size_t)p * plane + b * 16);
      const float4 g0 = src[0], g1 = src[1], u0 = src[2], u1 = src[3];
      g[0] += g0.x; g[1] += g0.y; g[2] += g0.z; g[3] += g0.w; g[4] += g1.x; g[5] += g1.y; g[6] += g1.z; g[7] += g1.w;
      u[0] += u0.x; u[1] += u0.y; u[2] += u0.z; u[3] += u0.w; u[4] += u1.x; u[5] += u1.y; u[6] += u1.z; u[7] += u1.w;
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 v = __floats2bfloat162_rn(glu_out(g[2 * j], u[2 * j], act),
                                                     glu_out(g[2 * j + 1], u[2 * j + 1], act));
      o[j] = *reinterpret_cast<const uint32_t*>(&v);
    }
    *reinterpret_cast<uint4*>(C + b * 8) = make_uint4(o[0], o[1], o[2], o[3]);   // row m, features 8*(b % (N/16))..
  } else {
    const size_t vecs = plane / 4;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= vecs) return;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), old = acc;
    if constexpr (ADD) old = reinterpret_cast<const float4*>(C)[i];
    for (int p = 0; p < splits; ++p) {
      const float4 v = reinterpret_cast<const float4*>(parts + (size_t)p * plane)[i];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    if constexpr (ADD) {
      acc.x += old.x; acc.y += old.y; acc.z += old.z; acc.w += old.w;
    }
    store4<OutT>(C + 4 * i, acc.x, acc.y, acc.z, acc.w);
  }
}

// How many parts along K a plain product of these sizes is split into (1: none).
static int tc_splits(int M, int N, int K, const int* offsets) {
  static const bool off = [] {
    const char* e = getenv("SNOWLLM_B200_TC_SPLIT");
    return e && e[0] == '0';
  }();
  int sms = 0;
  if (offsets || off || N % 16 || snk_device_sms(&sms)) return 1;
  const int k_tiles = (K + TC_BK - 1) / TC_BK;
  const int tiles = ((M + TC_BM - 1) / TC_BM) * ((N + 127) / 128);
  int splits = sms / tiles;                                   // parts that still find an SM each
  if (splits > 8) splits = 8;
  if (splits > k_tiles / 4) splits = k_tiles / 4;             // a part walks at least four k-blocks
  if (splits < 2) return 1;
  const int k_per = (k_tiles + splits - 1) / splits;
  return (k_tiles + k_per - 1) / k_per;                       // no part without k-blocks
}

// Columns of an unsplit plain product's tiles: the fewest rounds of tiles over the SMs, a tile counted by the operand bytes that it
// takes in (128 rows of A and its columns of W, per k-block); a narrower tile has to win by 3 %, as wide ones share more of
// what they read.  The line lies where the rounds change, so no two sizes have the same reason.  Measured, us, tiles of 256 (from 120
// of them on, else 128) before / with this rule, in replayed chains over rotating weights:
//   160 columns  21,504 x 2,048: 24 rows 30.0 / 26.7, 128 rows 26.8 / 21.7 (135 tiles, one round, for two of 168), 200 rows 36.0 / 27.7;
//                14,336 x 2,048: 300 rows 33.6 / 25.8
//   192 columns  6,144 x 2,048: 438 rows 21.5 / 16.4, 1,024 rows 29.1 / 26.0; 3,072 x 2,048: 1,024 rows 21.2 / 15.9, 2,048 rows 28.9 / 24.8;
//                2,048 x 8,192: 1,536 rows 65 / 50; 2,048 x 2,048: 1,536 rows 21.6 / 15.8
//   128 columns  16,384 x 2,048: 300 rows 34.2 / 30.5
// Over 96 sizes (24 to 3,000 rows of eight products) the rule's choice was within 2 % of the fastest of the four at all but
// one, 16,384 columns of 1,536 rows, which the 3 % keep with 256.
static int tc_tile_columns(int M, int N, int sms, double* its_cost = nullptr) {
  static const int columns[4] = {256, 192, 160, 128};
  const long long row_tiles = (M + TC_BM - 1) / TC_BM;
  int best = 256;
  double least = 0.0;
  for (int bn : columns) {
    const long long tiles = row_tiles * ((N + bn - 1) / bn);
    const double cost = (double)((tiles + sms - 1) / sms) * (TC_BM + bn);
    if (bn == 256 || cost < 0.97 * least) {
      best = bn;
      least = cost;
    }
  }
  if (its_cost) *its_cost = least;
  return best;
}
// For tests: what an unsplit plain product of these sizes takes on a device of that many SMs.
SNK_API int snk_gemm_tc_tile(int M, int N, int sms) { return tc_tile_columns(M, N, sms); }

// Whether a plain product of these sizes is better off on pairs of SMs (gemm_tc2.cu, 256 x 256 tiles a pair): by the same count of
// rounds, a pair's tile at 340, what its 256 rows and columns came to against the tiles here.  Products split along K stay here.
// Measured, us, one SM / pairs: 16,384 x 2,048: 300 rows 31.1 / 29.5, 512 rows 35.4 / 30.9, 1,024 rows 60.6 / 54.5, 2,048 rows 109 / 98, 3,500 rows
// 185 / 166; 6,144 x 2,048: 512 rows 16.8 / 18.7, 1,024 rows 26.2 / 27.2, 2,048 rows 42.9 / 39.1; 3,072 x 2,048: 2,048 rows 25.1 / 27.3, 2,560 rows
// 29.1 / 27.6; 2,048 x 8,192: 1,024 rows 39.3 / 47.1, 2,048 rows 61.2 / 54.5, 2,560 rows 81.9 / 87.5.  Over 99 sizes (300 to 3,500 rows of nine
// products) the slower one was chosen at seven, by 2 to 6 %.
#define TC_PAIR_TILE_COST 340.0
SNK_API int snk_gemm_tc_pairs_pay(int M, int N, int K, int sms) {
  if (sms < 2) return 0;
  double here = 0.0;
  tc_tile_columns(M, N, sms, &here);
  const long long tiles = ((M + 255ll) / 256) * ((N + 255) / 256), pairs = sms / 2;
  return tc_splits(M, N, K, nullptr) == 1 && (double)((tiles + pairs - 1) / pairs) * TC_PAIR_TILE_COST < 0.97 * here;
}
// Grouped products on one SM: wide tiles where they still give every SM work.
static int tc_grouped_tile(int M, int N) { return (long long)((M + TC_BM - 1) / TC_BM) * ((N + 255) / 256) >= 120 ? 256 : 128; }

// Bytes of scratch snk_gemm_tc wants for these sizes (0: none).
SNK_API long long snk_gemm_tc_scratch_bytes(int M, int N, int K, int grouped) {
  if (grouped) return 0;
  const int splits = tc_splits(M, N, K, nullptr);
  return splits > 1 ? (long long)splits * M * N * (long long)sizeof(float) : 0;
}

// M: rows of A (all groups together).  Grouped: offsets[groups+1] on the device, W = [groups, N, K];
// max_row_tiles bounds the number of 128-row tiles over all groups (M/128 + groups is always enough).
// out_f32: 0 bfloat16, 1 float, 2 float added to what C holds (plain products).
// scratch: snk_gemm_tc_scratch_bytes of device memory (may be null when that is 0).  w_ahead (plain products): W was
// there before the kernel in front of this launch began, and may be read ahead of the wait for it.
SNK_API int snk_gemm_tc(const void* A, const void* W, void* C, int M, int N, int K, const int* offsets,
                        int groups, int max_row_tiles, int out_f32, int swiglu, void* scratch, int w_ahead,
                        cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 8) return SNK_ERR_SIZE;                   // TMA: the row pitch is a multiple of 16 bytes
  if (swiglu && (N % 16 || out_f32 || swiglu == SNK_ACT_RELU2)) return SNK_ERR_SIZE;
  const bool add = out_f32 == 2;
  if (add && offsets) return SNK_ERR_SIZE;
  if (((uintptr_t)A % 16) || ((uintptr_t)W % 16) || ((uintptr_t)C % 16)) return SNK_ERR_ALIGN;
  const int row_tiles = offsets ? max_row_tiles : (M + TC_BM - 1) / TC_BM;
  if (row_tiles <= 0) return SNK_ERR_SIZE;
  int sms = 0, rc = snk_device_sms(&sms);
  if (rc) return rc;
  const int splits = tc_splits(M, N, K, offsets);
  const int bn = splits > 1 ? 128 : offsets ? tc_grouped_tile(M, N) : tc_tile_columns(M, N, sms);
  if (splits > 1 && (scratch == nullptr || ((uintptr_t)scratch % 16))) return SNK_ERR_ALIGN;
  CUtensorMap map_a, map_w;
  rc = tensor_map(A, M, K, TC_BM, TC_BK, &map_a);
  if (rc) return rc;
  rc = tensor_map(W, (long long)(offsets ? groups : 1) * N, K, bn, TC_BK, &map_w);
  if (rc) return rc;
  if (splits > 1) {
    rc = launch_tc<128, float, false, false, TC_SPLIT_EPI_WARPS>(map_a, map_w, scratch, M, N, K, nullptr, 1, row_tiles, splits, w_ahead, stream);
    if (rc) return rc;
    const float* parts = static_cast<const float*>(scratch);
    const size_t work = swiglu ? (size_t)M * N / 16 : (size_t)M * N / 4;
    const dim3 grid((unsigned)((work + 255) / 256)), block(256);
    if (swiglu) snk_launch(splitk_reduce_kernel<bf16, true>, grid, block, 0, stream, parts, static_cast<bf16*>(C), M, N, splits, swiglu);
    else if (add) snk_launch(splitk_reduce_kernel<float, false, true>, grid, block, 0, stream, parts, static_cast<float*>(C), M, N, splits, 0);
    else if (out_f32) snk_launch(splitk_reduce_kernel<float, false>, grid, block, 0, stream, parts, static_cast<float*>(C), M, N, splits, 0);
    else snk_launch(splitk_reduce_kernel<bf16, false>, grid, block, 0, stream, parts, static_cast<bf16*>(C), M, N, splits, 0);
    SNK_LAUNCH_CHECK();
    return 0;
  }
#define TC_GO(T_, S_, ADD_)                                                                                                \
  (bn == 256 ? launch_tc<256, T_, S_, ADD_>(map_a, map_w, C, M, N, K, offsets, groups, row_tiles, 1, w_ahead, stream, swiglu) : \
   bn == 192 ? launch_tc<192, T_, S_, ADD_>(map_a, map_w, C, M, N, K, offsets, groups, row_tiles, 1, w_ahead, stream, swiglu) : \
   bn == 160 ? launch_tc<160, T_, S_, ADD_>(map_a, map_w, C, M, N, K, offsets, groups, row_tiles, 1, w_ahead, stream, swiglu) : \
               launch_tc<128, T_, S_, ADD_>(map_a, map_w, C, M, N, K, offsets, groups, row_tiles, 1, w_ahead, stream, swiglu))
  if (swiglu) return TC_GO(bf16, true, false);
  if (add) return TC_GO(float, false, true);
  return out_f32 ? TC_GO(float, false, false) : TC_GO(bf16, false, false);
#undef TC_GO
}

// The product split along K with the sum left to the caller: `parts` receives the float planes
// [splits][M][N], to be added in plane order (what splitk_reduce_kernel does).  Returns the number of planes
// through *splits_out; products that are not split (see snk_gemm_tc_scratch_bytes) give SNK_ERR_SIZE.
SNK_API int snk_gemm_tc_parts(const void* A, const void* W, void* parts, int M, int N, int K, int* splits_out,
                              int w_ahead, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || K % 8) return SNK_ERR_SIZE;
  if (((uintptr_t)A % 16) || ((uintptr_t)W % 16) || parts == nullptr || ((uintptr_t)parts % 16)) return SNK_ERR_ALIGN;
  const int splits = tc_splits(M, N, K, nullptr);
  if (splits <= 1) return SNK_ERR_SIZE;
  CUtensorMap map_a, map_w;
  int rc = tensor_map(A, M, K, TC_BM, TC_BK, &map_a);
  if (rc) return rc;
  rc = tensor_map(W, N, K, 128, TC_BK, &map_w);
  if (rc) return rc;
  *splits_out = splits;
  return launch_tc<128, float, false, false, TC_SPLIT_EPI_WARPS>(map_a, map_w, parts, M, N, K, nullptr, 1, (M + TC_BM - 1) / TC_BM, splits, w_ahead, stream);
}

// Test hook: with on != 0 the producers of later launches issue no loads, so that the bounded waits run out
// (about 1.5 s) and the launches return with an error status instead of a product.  Synchronises.
SNK_API int snk_gemm_tc_test_lose_loads(int on) {
  return (int)cudaMemcpyToSymbol(g_tc_lose_loads, &on, sizeof(int));
}

// Queue a copy of the status word into ``host`` (pinned host memory, one int) on ``stream`` without waiting
// for it and without clearing it: a caller that synchronises with the stream anyway (an event, a read-back)
// learns of a wait that ran out at no cost.  Not for use inside a stream capture.
SNK_API int snk_gemm_tc_status_peek(int* host, void* stream) {
  return (int)cudaMemcpyFromSymbolAsync(host, g_tc_status, sizeof(int), 0, cudaMemcpyDeviceToHost, (cudaStream_t)stream);
}

// 0, or the first error a block of any earlier launch recorded (a wait that ran out); reading clears
// it.  Synchronises the device.
SNK_API int snk_gemm_tc_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int));
  return v;
}

// ---------------------------------------------------------------------------------------------
// out[r, :] = in[rows[r] / div, :]  (bfloat16 rows of K elements, K a multiple of 8)
#define GATHER_ROWS_PER_BLOCK 8
__global__ void gather_rows_kernel(const uint4* __restrict__ in, uint4* __restrict__ out,
                                   const int* __restrict__ rows, int div, int vecs, int R) {
  pdl_begin();
  // a block copies GATHER_ROWS_PER_BLOCK rows; every thread has one vector of each row in flight
  const int r0 = blockIdx.x * GATHER_ROWS_PER_BLOCK;
  for (int i = threadIdx.x; i < vecs; i += blockDim.x) {
    uint4 v[GATHER_ROWS_PER_BLOCK];
#pragma unroll
    for (int j = 0; j < GATHER_ROWS_PER_BLOCK; ++j)
      if (r0 + j < R) v[j] = in[(size_t)(rows[r0 + j] / div) * vecs + i];
#pragma unroll
    for (int j = 0; j < GATHER_ROWS_PER_BLOCK; ++j)
      if (r0 + j < R) out[(size_t)(r0 + j) * vecs + i] = v[j];
  }
}

SNK_API int snk_gather_rows_bf16(const void* in, void* out, const int* rows, int div, int R, int K,
                                 cudaStream_t stream) {
  if (R <= 0) return 0;
  if (K % 8 || ((uintptr_t)in % 16) || ((uintptr_t)out % 16)) return SNK_ERR_ALIGN;
  snk_launch(gather_rows_kernel, dim3((R + GATHER_ROWS_PER_BLOCK - 1) / GATHER_ROWS_PER_BLOCK), dim3(256), 0, stream,
             static_cast<const uint4*>(in), static_cast<uint4*>(out), rows, div <= 0 ? 1 : div, K / 8, R);
  SNK_LAUNCH_CHECK();
  return 0;
}
