// C[M,N] = A[M,K] . W[N,K]^T in bfloat16 on the tcgen05 tensor cores with PAIRS of SMs (cta_group::2), for
// many rows (prefill).  The one-SM kernel of gemm_tc.cu is bound by what L2 feeds an SM: 48 KB of operands per
// k-block of a 128 x 256 tile.  Here a cluster of two blocks owns a 256 x 256 tile of C: each block loads its own
// 128 rows of A and HALF of the 256 rows of W (32 KB per k-block), the leader block issues one MMA of M 256 for
// both, and the tensor cores of the two SMs read the other block's half of W across the pair.  A third less
// operand traffic per product.
//
//   warp 0, one lane   TMA producer (both blocks): 128x64 of A and 128x64 of W into this block's stage ring; the
//                      bytes of both blocks count towards the LEADER's stage barrier (cta_group::2 loads)
//   warp 1             leader only: waits for the stage, one lane issues four tcgen05.mma.cta_group::2; a multicast commit
//                      frees the stage in both blocks and, after the last k-block, hands the accumulator to both
//                      epilogues
//   warps 2..5 or 9    epilogue (both blocks): tcgen05.ld of this block's 128 accumulator rows, stores; then an
//                      arrival on the leader's accumulator-free barrier (remote from the peer)
//
// Row tiles are 256 rows.  Grouped products run the kernel further down, with the operands changed round.
// Every mbarrier wait is bounded by wall time (see snk_gemm_tc2_status); when one runs out both blocks of the pair
// stop issuing loads and products, give the copies in flight a moment to land, free their tensor memory and
// return.  No TMA load is multicast: each block loads what it owns.
#include "tcgen05.cuh"

#define T2_BM 128                     // rows of A per block (256 per pair)
#define T2_BN 256                     // columns of C per pair; each block loads T2_BN / 2 rows of W
#define T2_BK 64
// Epilogue warps of each block: two to each 32 lanes of tensor memory, which share a tile's columns, where one was what a tile
// waited for: the gated store (8,192 x 16,384 x 2,048, one / two warps: 405 / 342 us alone) and the grouped products (2,048
// tokens, down 78.4 / 73.4 us).  The plain stores of the ungrouped product stay behind its products with one (8,192 x 6,144 x 2,048
// 136.5 / 136.7 us).
#define T2_EPI_WARPS 8
#define T2_PLAIN_EPI_WARPS 4
#define T2_STAGE_BYTES ((T2_BM + T2_BN / 2) * T2_BK * 2)
#ifndef T2_STAGES
#define T2_STAGES 6
#endif
#define T2_MAX_STAGES 11              // (grouped products with few rows a group)
static_assert(T2_STAGES <= T2_MAX_STAGES, "barriers");
#ifndef T2_BAND
#define T2_BAND 8
#endif
#define T2_WAIT_NS 1500000000ull
#ifndef T2_ACC_BUFFERS
#define T2_ACC_BUFFERS 2              // accumulators in tensor memory: the epilogue of a tile overlaps the next tile's products
#endif

enum { T2_ERR_FULL = 1, T2_ERR_EMPTY = 2, T2_ERR_ACC = 3, T2_ERR_ACC_FREE = 4, T2_ERR_PEER = 5 };

__device__ int g_t2_status;
__device__ int g_t2_lose_loads;      // test hook: producers issue no loads (the operands then never arrive)
__device__ unsigned int g_t2_tmem[2];  // the tensor-memory base addresses the two blocks of cluster 0 were given (a probe)

// The long way of a wait: polls for T2_WAIT_NS at most.  False: the wait ran out, or another one of the pair has.
__device__ __noinline__ bool t2_wait_long(uint64_t* bar, uint32_t parity, volatile int* aborted, int code) {
  const uint64_t start = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (*aborted) return false;
    if (global_ns() - start > T2_WAIT_NS) {
      *aborted = 1;
      st_cluster_u32(const_cast<int*>(aborted), cluster_ctarank() ^ 1u, 1u);   // the other block of the pair stops too
      atomicCAS(&g_t2_status, 0, code);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool t2_wait(uint64_t* bar, uint32_t parity, volatile int* aborted, int code) {
  return mbar_try_wait(bar, parity) || t2_wait_long(bar, parity, aborted, code);
}
// The same by all lanes of a warp (mbar_wait_warp of gemm_tc.cu).
__device__ __forceinline__ bool t2_wait_warp(uint64_t* bar, uint32_t parity, volatile int* aborted, int code) {
  return __all_sync(0xffffffffu, t2_wait(bar, parity, aborted, code));
}

struct __align__(16) T2Shared {
  uint64_t full[T2_MAX_STAGES];     // (leader) both blocks' stages hold their operands
  uint64_t empty[T2_MAX_STAGES];    // the MMAs that read the stage have completed (both blocks)
  uint64_t acc_full[2];             // the tile's products have completed (both blocks)
  uint64_t acc_empty[2];            // (leader) both epilogues have read the accumulator: an arrival a warp
  uint32_t tmem_base;
  int aborted;
};
struct __align__(16) T2Staging {
  float tile[T2_PLAIN_EPI_WARPS][TC_STAGE_FLOATS];            // one per epilogue warp (tc_store_piece)
};

struct T2Tile {
  int row0, row_end, w_row0, n0;
  bool valid;
};

// Pair tile `tile`: 256 rows x 256 columns.
__device__ __forceinline__ T2Tile t2_tile(int tile, int row_tiles, int M, int N) {
  T2Tile t;
  // bands of up to T2_BAND n-tiles, the n-tile fastest inside a band, then the row tile (as in gemm_tc.cu)
  const int n_tiles = (N + T2_BN - 1) / T2_BN;
  const int bands = (n_tiles + T2_BAND - 1) / T2_BAND;
  const int band_w = (n_tiles + bands - 1) / bands;
  const int per_band = row_tiles * band_w;
  const int band = tile / per_band, in_band = tile % per_band;
  const int w_here = min(band_w, n_tiles - band * band_w);
  const int rt = in_band / w_here, nt = band * band_w + in_band % w_here;
  t.n0 = nt * T2_BN;
  t.valid = t.n0 < N;
  t.row0 = rt * 2 * T2_BM;
  t.row_end = M;
  t.w_row0 = 0;
  return t;
}

// ADD (float): the product is added to what C holds.
template <typename OutT, bool SWIGLU, bool ADD>
__global__ void __launch_bounds__(64 + 32 * (SWIGLU ? T2_EPI_WARPS : T2_PLAIN_EPI_WARPS))
gemm_tc2_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                OutT* __restrict__ C, int M, int N, int K, int row_tiles, int act) {
  constexpr int EPI_WARPS = SWIGLU ? T2_EPI_WARPS : T2_PLAIN_EPI_WARPS, EPI_COLS = T2_BN * 4 / EPI_WARPS;   // columns a warp takes
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  T2Shared* sh = reinterpret_cast<T2Shared*>(tiles + (size_t)T2_STAGES * T2_STAGE_BYTES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();               // 0: leader, 1: peer
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;     // pairs lie along x
  const int k_tiles = (K + T2_BK - 1) / T2_BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < T2_STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->acc_full[b], 1);
      mbar_init(&sh->acc_empty[b], 2 * EPI_WARPS);       // the epilogue warps of both blocks
    }
    sh->aborted = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&sh->tmem_base)), "r"((uint32_t)(T2_ACC_BUFFERS * T2_BN)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync();                                        // both blocks' barriers and tensor memory are set up
  tc_fence_after();
  // the accumulator's address is the leader's: the MMA writes rows 128..255 at the same columns of the peer
  const uint32_t tmem_acc = rank == 0 ? sh->tmem_base : ld_cluster_u32(&sh->tmem_base, 0);
  if (pair == 0 && threadIdx.x == 0) g_t2_tmem[rank] = sh->tmem_base;
  volatile int* aborted = &sh->aborted;
  pdl_begin();
  const int n_tiles = (N + T2_BN - 1) / T2_BN;
  const int total = row_tiles * n_tiles;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      const bool lose_loads = *const_cast<volatile int*>(&g_t2_lose_loads) != 0;
      for (int tile = pair; tile < total && !*aborted; tile += pairs) {
        const T2Tile t = t2_tile(tile, row_tiles, M, N);
        if (!t.valid) continue;
        for (int kt = 0; kt < k_tiles; ++kt, ++it) {
          const int s = it % T2_STAGES;
          if (!t2_wait(&sh->empty[s], ((it / T2_STAGES) & 1) ^ 1, aborted, T2_ERR_EMPTY)) break;   // nothing more is issued
          if (lose_loads) continue;
          // both blocks' bytes count towards the leader's barrier: it is the leader that issues the MMAs
          if (rank == 0) mbar_expect_tx(&sh->full[s], 2 * T2_STAGE_BYTES);
          const uint32_t bar = cluster_addr(&sh->full[s], 0);
          unsigned char* stage = tiles + (size_t)s * T2_STAGE_BYTES;
          tma2_load_2d(stage, &map_a, bar, kt * T2_BK, t.row0 + (int)rank * T2_BM);
          tma2_load_2d(stage + T2_BM * T2_BK * 2, &map_w, bar, kt * T2_BK, t.w_row0 + t.n0 + (int)rank * (T2_BN / 2));
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {                                     // the leader issues for the pair; the peer's warp rests
      const uint32_t idesc = instr_desc_bf16(2 * T2_BM, T2_BN), elected = elect_lane();
      const uint32_t ring_lo = smem_desc_lo(smem_u32(tiles)), empty0 = smem_u32(&sh->empty[0]);
      int s = 0, local = 0;
      uint32_t lap = 0;
      for (int tile = pair; tile < total; tile += pairs) {
        const T2Tile t = t2_tile(tile, row_tiles, M, N);
        if (!t.valid) continue;
        const int buf = local % T2_ACC_BUFFERS;
        const int use = local / T2_ACC_BUFFERS;          // how often this accumulator was used before
        if (!t2_wait_warp(&sh->acc_empty[buf], (use & 1) ^ 1, aborted, T2_ERR_ACC_FREE)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_acc + (uint32_t)(buf * T2_BN);
        int kt = 0;
        for (; kt < k_tiles; ++kt) {
          if (!t2_wait_warp(&sh->full[s], lap, aborted, T2_ERR_FULL)) break;        // both blocks' stage s
          tc_fence_after();
          const uint32_t a_lo = ring_lo + s * (T2_STAGE_BYTES >> 4), w_lo = a_lo + (T2_BM * T2_BK * 2 >> 4);
#pragma unroll
          for (int k = 0; k < T2_BK / 16; ++k)           // 16 k-values: 32 bytes further along the swizzled rows
            umma2_bf16_lo(d_tmem, a_lo + 2 * k, w_lo + 2 * k, idesc, (kt > 0 || k > 0) ? 1u : 0u, elected);
          umma2_commit_if(empty0 + s * 8, 3, elected);   // the stage is free in both blocks once these MMAs have read it
          if (++s == T2_STAGES) {
            s = 0;
            lap ^= 1;
          }
        }
        if (kt < k_tiles) break;                         // a wait ran out
        umma2_commit_if(smem_u32(&sh->acc_full[buf]), 3, elected);
        ++local;
      }
    }
  } else {
    const int lane_group = warp & 3, c_begin = (warp - 2) / 4 * EPI_COLS;
    float* stage_out = SWIGLU ? nullptr : reinterpret_cast<T2Staging*>(sh + 1)->tile[warp - 2];
    int local = 0;
    for (int tile = pair; tile < total; tile += pairs) {
      const T2Tile t = t2_tile(tile, row_tiles, M, N);
      if (!t.valid) continue;
      const int buf = local % T2_ACC_BUFFERS;
      const int use = local / T2_ACC_BUFFERS;
      const int first_row = t.row0 + (int)rank * T2_BM + lane_group * 32;
      TcOld<ADD> old;
      tc_load_old<ADD>(old, lane, C, first_row, t.row_end, t.n0 + c_begin, N);
      if (!t2_wait_warp(&sh->acc_full[buf], use & 1, aborted, T2_ERR_ACC)) break;
      tc_fence_after();
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_begin + EPI_COLS; c0 += 32) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)(buf * T2_BN + c0), r);
        if (c0 + 32 >= c_begin + EPI_COLS) {             // everything of this warp's part is in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0 && !*aborted) {
            if (rank == 0) mbar_arrive(&sh->acc_empty[buf]);
            else mbar_arrive_remote(&sh->acc_empty[buf], 0);
          }
        }
        if (!*aborted)
          tc_store_piece<OutT, SWIGLU, ADD>(r, stage_out, lane, C, first_row, t.row_end, t.n0 + c0, N, act, old);
        if (c0 + 32 < c_begin + EPI_COLS) tc_load_old<ADD>(old, lane, C, first_row, t.row_end, t.n0 + c0 + 32, N);
      }
      ++local;
    }
  }
  if (*aborted) drain_after_abort();
  tc_fence_before();
  __syncwarp();
  cluster_sync();                                        // nobody of the pair touches tensor memory or barriers any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;"
                 ::"r"(sh->tmem_base), "r"((uint32_t)(T2_ACC_BUFFERS * T2_BN)) : "memory");
  }
}

template <typename OutT, bool SWIGLU, bool ADD = false>
static int launch_tc2(const CUtensorMap& map_a, const CUtensorMap& map_w, void* C, int M, int N, int K,
                      int row_tiles, cudaStream_t stream, int act) {
  const size_t smem = 1024 + (size_t)T2_STAGES * T2_STAGE_BYTES + sizeof(T2Shared) + sizeof(T2Staging);
  static std::atomic<int> ready[SNK_MAX_DEVICES];
  int sms = 0;
  const int rc = snk_kernel_ready(ready, gemm_tc2_kernel<OutT, SWIGLU, ADD>, smem, &sms);
  if (rc) return rc;
  const long long tiles = (long long)row_tiles * ((N + T2_BN - 1) / T2_BN);
  const int pairs = (int)(tiles < sms / 2 ? tiles : sms / 2);
  const dim3 block(64 + 32 * (SWIGLU ? T2_EPI_WARPS : T2_PLAIN_EPI_WARPS));
  snk_launch_cluster3(gemm_tc2_kernel<OutT, SWIGLU, ADD>, dim3(2 * pairs), block, smem, stream, dim3(2, 1, 1),
                      map_a, map_w, static_cast<OutT*>(C), M, N, K, row_tiles, act);
  SNK_LAUNCH_CHECK();
  return 0;
}

// ---------------------------------------------------------------------------------------------
// Grouped products (experts): the operands change places.  With rows of A as the 128-row operand a group of
// 270 rows costs three one-SM tiles (two pair tiles), each as dear as a full one, and what bounds a tile is
// the operand bytes an SM takes in.  Here W is the 256-row operand of the pair (each block loads 128 rows of
// W: 16 KB per k-block) and the group's ROWS are the N side of the MMA, which may be any multiple of 16 up
// to 256: a tile is 256 columns of C by up to 256 rows, a group's last tile is as wide as it needs, and each
// block loads half of the tile's rows of A.  The accumulator holds C transposed (lanes: columns of C); the
// epilogue turns it back.
//
// Items in order: group, then 256-column tile of C, then the group's row tiles, so that the pairs that
// read the same rows of W run side by side; item i goes to pair i % pairs.  (Measured and dropped: runs of
// neighbouring items of equal modelled cost per pair, 157 -> 180 us on the experts' gate|up product of 2,048
// tokens, as pairs side by side then read far-apart memory; items drawn from a counter as pairs get free,
// 159 us; L2 prefetch of an item's rows of W in one piece, 184 to 198 us.)
//
// Up to 32 groups come in the order of their row tiles' length, longest first: a round of items then has one length, and the
// shortest make the last, partly filled one.
//
// Groups of few rows are bound by the read of W, and that by the bytes an SM keeps on their way: a stage's part for A
// is as large as the longest row tile of the launch needs, and the ring has as many stages as then fit (11 of 20 KB,
// 9 of 24 KB, 6 of 32 KB; a plain TMA read loop: 5.3 TB/s with 64 KB of an SM in flight, 6.4 with 128 KB).
// Measured in turn, 32 groups, gate|up of 2,048 x 3,584 with its gate, tokens with the top 4 of 32, us (an issuing lane, one epilogue
// warp to 32 lanes, the offsets read for each item / so): 16 tokens 64.9 / 62.1, 64 87.0 / 80.4 = 5.8 TB/s, 276 89.0 / 83.3, 1,024 121 / 99.8, 2,048 210 /
// 155, 4,096 349 / 254; down of 1,792 x 2,048 37.5 / 35.2, 47.7 / 45.4, 49.9 / 47.1, 59.7 / 52.9, 83.4 / 74.4, 129 / 116.  (Also tried: tiles of 224
// or 240 columns where they fill the last round better, 89.5 us at 8 rows and slower from 256 rows on, where an item costs its
// full M of 256 whatever it keeps.)
#define T2G_MAX_GROUPS 256
#define T2G_W_BYTES (T2_BM * T2_BK * 2)               // of a stage: 128 rows of W, then 128, 64 or 32 of the tile's rows of A
#define T2G_RING_BYTES (11 * (T2G_W_BYTES + 32 * T2_BK * 2))     // the largest of the three rings
#define T2G_BOXES 5                  // tensor maps of A with boxes of 128, 64, 32, 16 and 8 rows

struct T2GMaps {
  CUtensorMap a[T2G_BOXES];
};
// What every block works out of the offsets: the groups in the order they are taken, and the items before each.
struct T2GPlan {
  int first[T2G_MAX_GROUPS + 1];     // by place in the order: items before the group,
  int order[T2G_MAX_GROUPS];         // its number,
  int begin[T2G_MAX_GROUPS], cnt[T2G_MAX_GROUPS];   // its rows (an item is looked up here alone: from the offsets in global
                                     // memory a pair stood 1,080 cycles between two items, 5 % of one)
  int longest;                       // rows of the longest row tile
};

// A group's rows are dealt evenly to its row tiles (in steps of 16): every tile streams the same rows of W,
// so a group of 270 rows as 144 + 128 costs two half-length products, where 256 + 16 costs a full one and
// a second pass over W for 16 rows (with 2,048 tokens, top 4 of 32 experts, half the groups are just
// above 256 rows).
__device__ __forceinline__ int t2g_row_tiles(int cnt) { return (cnt + 2 * T2_BM - 1) / (2 * T2_BM); }
__device__ __forceinline__ int t2g_tile_rows(int cnt) {
  const int row_tiles = t2g_row_tiles(cnt);
  return row_tiles ? ((cnt + row_tiles - 1) / row_tiles + 15) & ~15 : 0;
}

// By all threads of the block; ends with a barrier.  Up to 32 groups are put in order, equal lengths in the groups' own order (every
// block comes to the same plan), by a lane per group that compares its own with all others in registers.  More groups stay in
// their own order: what the other order gains there, 0 to 3 %, is less than it costs.  Measured, us: groups in their own order
// for all, their sum by one thread / every group in order, compared through shared memory / so: 256 groups of 512 x 512, 1,032 rows
// 35.5 / 41.5 / 35.1; 40 of 512 x 1,024, half of 8,192 rows in one group 28.1 / 32.4 / 28.7; 64 of 768 x 2,048, 16,384 rows 87.4 /
// 85.6 / 88.2; 8 of 512 x 256, 128 rows 8.2 / 8.5 / 8.4.
__device__ __forceinline__ void t2g_plan(T2GPlan* plan, const int* __restrict__ offsets, int groups, int n_tiles) {
  if (groups <= 32) {
    const int lane = threadIdx.x;                        // (only the first warp's threads have a group)
    const int begin = lane < groups ? offsets[lane] : 0, cnt = lane < groups ? offsets[lane + 1] - begin : 0;
    const int mine = t2g_tile_rows(cnt), items = t2g_row_tiles(cnt) * n_tiles;
    int place = 0, before = 0, all = 0;
    for (int o = 0; o < groups && threadIdx.x < 32; ++o) {
      const int rows = __shfl_sync(0xffffffffu, mine, o), its = __shfl_sync(0xffffffffu, items, o);
      if (rows > mine || (rows == mine && o < lane)) {
        ++place;
        before += its;
      }
      all += its;
    }
    if (lane < groups) {
      plan->order[place] = lane;
      plan->begin[place] = begin;
      plan->cnt[place] = cnt;
      plan->first[place] = before;
      if (place == 0) plan->longest = mine;
    }
    if (lane == 0) plan->first[groups] = all;
    __syncthreads();
    return;
  }
  for (int e = threadIdx.x; e < groups; e += blockDim.x) {
    const int begin = offsets[e], cnt = offsets[e + 1] - begin;
    plan->begin[e] = begin;
    plan->cnt[e] = cnt;
    plan->order[e] = e;
    plan->first[e] = t2g_row_tiles(cnt) * n_tiles;       // the group's items, for now
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int run = 0, longest = 0;
    for (int e = threadIdx.x; e - (int)threadIdx.x < groups; e += 32) {
      const int items = e < groups ? plan->first[e] : 0;
      int upto = items;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int before = __shfl_up_sync(0xffffffffu, upto, o);
        if ((int)threadIdx.x >= o) upto += before;
      }
      if (e < groups) {
        plan->first[e] = run + upto - items;
        longest = max(longest, t2g_tile_rows(plan->cnt[e]));
      }
      run += __shfl_sync(0xffffffffu, upto, 31);
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    if (threadIdx.x == 0) {
      plan->first[groups] = run;
      plan->longest = longest;
    }
  }
  __syncthreads();
}

struct T2GItem {
  int row0, row_end, nt, w_row0, f0;  // rows row0 .. of A (nt of them in the MMA, a multiple of 16), W rows w_row0 + f0 ..
};

__device__ __forceinline__ T2GItem t2g_item(int item, const T2GPlan* plan, int groups, int N) {
  T2GItem t;
  int lo = 0, hi = groups;                               // the place lo with first[lo] <= item < first[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (plan->first[mid] <= item) lo = mid; else hi = mid;
  }
  const int e = plan->order[lo], begin = plan->begin[lo], cnt = plan->cnt[lo];
  const int row_tiles = t2g_row_tiles(cnt), per = t2g_tile_rows(cnt);
  const int in_group = item - plan->first[lo];
  const int ft = in_group / row_tiles, tt = in_group % row_tiles;
  t.row0 = begin + tt * per;
  t.row_end = min(begin + cnt, t.row0 + per);
  const int left = t.row_end - t.row0;
  t.nt = left <= 0 ? 16 : (left + 15) & ~15;
  t.w_row0 = e * N;
  t.f0 = ft * T2_BN;
  return t;
}

// The box of A for nt / 2 rows per block: the smallest of 128, 64, 32, 16, 8 that holds them.
__device__ __forceinline__ int t2g_box(int half_rows) {
  int b = 0, rows = 128;
  while (b + 1 < T2G_BOXES && (rows >> 1) >= half_rows) { rows >>= 1; ++b; }
  return b;
}

// The gated store of a grouped piece of `rows` (up to 32) rows.  Lanes 0..7 and 16..23 hold a column of gates each, the eight behind each
// their ups: of rows 2 j and 2 j + 1 a gate's lane gives the second for its up's first, and each then has both of one row.  A store
// writes 16 neighbouring columns of two rows.  Four pairs of rows at a time, their exchanges ahead of their activations and those ahead of
// their stores, and no more than there are rows: with halves of 16 rows exchanged, activated and stored one after the other
// an item's epilogue was one chain of 16, and longer than its products where K or the rows were few.  Measured, us, so before / now, 128
// groups of 768 x 512 and the top 8 of them: 200 tokens 38.2 / 31.7, 1,024 46.8 / 41.3; 32 groups of 3,584 x 2,048, top 4: 64 tokens 84 /
// 82, 276 92.9 / 88.4, 2,048 195 / 161, 4,096 304 / 272.  Eight pairs at a time 83.8 and 167 instead of 83.6 and 161 (100 and 2,048
// tokens), all sixteen 86.5 and 172.
template <typename OutT>
__device__ __forceinline__ void t2g_glu_store(uint32_t (&r)[32], int lane, OutT* __restrict__ dst, int ld, int mine, int rows, int act) {
  const int up = (lane >> 3) & 1;
  dst += (size_t)up * ld + (lane & 7) + ((lane >> 4) << 3);
  mine -= up;
#pragma unroll
  for (int j0 = 0; j0 < 16; j0 += 4) {
    if (2 * j0 >= rows) break;                           // (the same for all lanes)
#pragma unroll
    for (int j = j0; j < j0 + 4; ++j) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, up ? r[2 * j] : r[2 * j + 1], 8);
      if (up) r[2 * j] = other;
      else r[2 * j + 1] = other;
    }
#pragma unroll
    for (int j = j0; j < j0 + 4; ++j) r[2 * j] = __float_as_uint(glu_out(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]), act));
#pragma unroll
    for (int j = j0; j < j0 + 4; ++j)
      if (2 * j < mine) dst[(size_t)(2 * j) * ld] = from_f<OutT>(__uint_as_float(r[2 * j]));
  }
}

template <typename OutT, bool SWIGLU>
__global__ void __launch_bounds__(64 + 32 * T2_EPI_WARPS)
gemm_tc2_grouped_kernel(const __grid_constant__ T2GMaps maps, const __grid_constant__ CUtensorMap map_w,
                        OutT* __restrict__ C, int N, int K, const int* __restrict__ offsets, int groups, int act) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  T2Shared* sh = reinterpret_cast<T2Shared*>(tiles + T2G_RING_BYTES);
  T2GPlan* plan = reinterpret_cast<T2GPlan*>(sh + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int k_tiles = (K + T2_BK - 1) / T2_BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < T2_MAX_STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->acc_full[b], 1);
      mbar_init(&sh->acc_empty[b], 2 * T2_EPI_WARPS);
    }
    sh->aborted = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&sh->tmem_base)), "r"((uint32_t)(T2_ACC_BUFFERS * T2_BN)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_acc = rank == 0 ? sh->tmem_base : ld_cluster_u32(&sh->tmem_base, 0);
  volatile int* aborted = &sh->aborted;
  pdl_begin();                                           // offsets are written by the kernel before this one
  t2g_plan(plan, offsets, groups, (N + T2_BN - 1) / T2_BN);
  const int total = plan->first[groups];
  // the ring: both blocks of a pair, and every thread, come to the same one
  const int stages = plan->longest <= 64 ? 11 : plan->longest <= 128 ? 9 : 6;
  const int stage_bytes = T2G_W_BYTES + (plan->longest <= 64 ? 32 : plan->longest <= 128 ? 64 : 128) * T2_BK * 2;

  int s = 0;                                             // the stage of the next k-block (producer and MMA thread)
  uint32_t lap = 0;                                      // the parity of the ring's rounds so far
  auto next_stage = [&]() {
    if (++s == stages) {
      s = 0;
      lap ^= 1;
    }
  };
  const bool lose_loads = *const_cast<volatile int*>(&g_t2_lose_loads) != 0;
  auto issue_loads = [&](int item) {
    const T2GItem t = t2g_item(item, plan, groups, N);
    const int half = t.nt >> 1, box = t2g_box(half);
    const uint32_t bytes = (uint32_t)(T2G_W_BYTES + (128 >> box) * T2_BK * 2);
    for (int kt = 0; kt < k_tiles; ++kt, next_stage()) {
      if (!t2_wait(&sh->empty[s], lap ^ 1, aborted, T2_ERR_EMPTY)) return;     // a wait ran out: nothing more is issued
      if (lose_loads) continue;
      if (rank == 0) mbar_expect_tx(&sh->full[s], 2 * bytes);
      const uint32_t bar = cluster_addr(&sh->full[s], 0);
      unsigned char* stage = tiles + (size_t)s * stage_bytes;
      tma2_load_2d(stage, &map_w, bar, kt * T2_BK, t.w_row0 + t.f0 + (int)rank * T2_BM);
      tma2_load_2d(stage + T2G_W_BYTES, &maps.a[box], bar, kt * T2_BK, t.row0 + (int)rank * half);
    }
  };

  if (warp == 0) {
    if (lane == 0)
      for (int item = pair; item < total && !*aborted; item += pairs) issue_loads(item);
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t elected = elect_lane();
      const uint32_t ring_lo = smem_desc_lo(smem_u32(tiles)), empty0 = smem_u32(&sh->empty[0]);
      int local = 0;
      for (int item = pair; item < total; item += pairs, ++local) {
        const T2GItem t = t2g_item(item, plan, groups, N);
        const uint32_t idesc = instr_desc_bf16(2 * T2_BM, t.nt);
        const int buf = local % T2_ACC_BUFFERS;
        const int use = local / T2_ACC_BUFFERS;
        if (!t2_wait_warp(&sh->acc_empty[buf], (use & 1) ^ 1, aborted, T2_ERR_ACC_FREE)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_acc + (uint32_t)(buf * T2_BN);
        int kt = 0;
        for (; kt < k_tiles; ++kt, next_stage()) {
          if (!t2_wait_warp(&sh->full[s], lap, aborted, T2_ERR_FULL)) break;
          tc_fence_after();
          const uint32_t w_lo = ring_lo + s * (stage_bytes >> 4), a_lo = w_lo + (T2G_W_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < T2_BK / 16; ++k)
            umma2_bf16_lo(d_tmem, w_lo + 2 * k, a_lo + 2 * k, idesc, (kt > 0 || k > 0) ? 1u : 0u, elected);
          umma2_commit_if(empty0 + s * 8, 3, elected);
        }
        if (kt < k_tiles) break;                         // a wait ran out
        umma2_commit_if(smem_u32(&sh->acc_full[buf]), 3, elected);
      }
    }
  } else {
    // two warps to each 32 lanes (columns of C): they take the item's pieces of 32 rows in turns
    const int lane_group = warp & 3, c_begin = (warp - 2) / 4 * 32;
    int local = 0;
    for (int item = pair; item < total; item += pairs, ++local) {
      const T2GItem t = t2g_item(item, plan, groups, N);
      const int buf = local % T2_ACC_BUFFERS;
      const int use = local / T2_ACC_BUFFERS;
      if (!t2_wait_warp(&sh->acc_full[buf], use & 1, aborted, T2_ERR_ACC)) break;
      tc_fence_after();
      const int col0 = t.f0 + (int)rank * T2_BM + lane_group * 32;     // this warp's 32 columns of C: one per lane
      auto release = [&]() {                             // all that this warp reads of the accumulator is in registers
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && !*aborted) {
          if (rank == 0) mbar_arrive(&sh->acc_empty[buf]);
          else mbar_arrive_remote(&sh->acc_empty[buf], 0);
        }
      };
      if (c_begin >= t.nt) release();
#pragma unroll 1
      for (int c0 = c_begin; c0 < t.nt; c0 += 64) {
        uint32_t r[32];                                  // this lane's column of C at rows row0 + c0 ..
        tmem_ld32(tmem_acc + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)(buf * T2_BN + c0), r);
        if (c0 + 64 >= t.nt) release();
        const int rows = t.row_end - (t.row0 + c0);      // of this piece and the ones behind it
        if constexpr (SWIGLU) {
          t2g_glu_store(r, lane, C + (size_t)(t.row0 + c0) * (N / 2) + col0 / 2, N / 2, col0 + (lane & 16) + 16 <= N ? rows : 0, rows, act);
        } else if (col0 + lane < N) {
          // a warp's store writes 32 neighbouring columns of one row
          OutT* dst = C + (size_t)(t.row0 + c0) * N + col0 + lane;
          auto store = [&](int j) {
            float v = __uint_as_float(r[j]);
            if constexpr (sizeof(OutT) == 2) v = unary_out(v, act);
            dst[(size_t)j * N] = from_f<OutT>(v);
          };
          if (rows >= 32) {
#pragma unroll
            for (int j = 0; j < 32; ++j) store(j);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < rows) store(j);
          }
        }
      }
    }
  }
  if (*aborted) drain_after_abort();
  tc_fence_before();
  __syncwarp();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;"
                 ::"r"(sh->tmem_base), "r"((uint32_t)(T2_ACC_BUFFERS * T2_BN)) : "memory");
  }
}

template <typename OutT, bool SWIGLU>
static int launch_tc2_grouped(const T2GMaps& maps, const CUtensorMap& map_w, void* C, int M, int N, int K,
                              const int* offsets, int groups, cudaStream_t stream, int act) {
  const size_t smem = 1024 + T2G_RING_BYTES + sizeof(T2Shared) + sizeof(T2GPlan);
  static std::atomic<int> ready[SNK_MAX_DEVICES];
  int sms = 0;
  const int rc = snk_kernel_ready(ready, gemm_tc2_grouped_kernel<OutT, SWIGLU>, smem, &sms);
  if (rc) return rc;
  // at most M / 256 full row tiles and one partial tile per group
  const long long items = ((long long)M / (2 * T2_BM) + groups) * ((N + T2_BN - 1) / T2_BN);
  const int pairs = (int)(items < sms / 2 ? items : sms / 2);
  snk_launch_cluster3(gemm_tc2_grouped_kernel<OutT, SWIGLU>, dim3(2 * pairs), dim3(64 + 32 * T2_EPI_WARPS), smem, stream,
                      dim3(2, 1, 1), maps, map_w, static_cast<OutT*>(C), N, K, offsets, groups, act);
  SNK_LAUNCH_CHECK();
  return 0;
}

// M: rows of A (all groups together).  Grouped: offsets[groups+1] on the device, W = [groups, N, K].  out_f32: 0 bfloat16, 1 float,
// 2 float added to what C holds (plain products).
SNK_API int snk_gemm_tc2(const void* A, const void* W, void* C, int M, int N, int K, const int* offsets,
                         int groups, int out_f32, int swiglu, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 8) return SNK_ERR_SIZE;
  const int unary = swiglu == SNK_ACT_RELU2 ? swiglu : 0;  // (grouped products only)
  if (unary) swiglu = 0;
  if ((swiglu && N % 16) || ((swiglu || unary) && out_f32) || (unary && !offsets) || (out_f32 == 2 && offsets)) return SNK_ERR_SIZE;
  if (((uintptr_t)A % 16) || ((uintptr_t)W % 16) || ((uintptr_t)C % 16)) return SNK_ERR_ALIGN;
  if (offsets) {
    if (groups <= 0 || groups > T2G_MAX_GROUPS) return SNK_ERR_SIZE;
    T2GMaps maps;
    for (int b = 0; b < T2G_BOXES; ++b) {
      const int rc = tensor_map(A, M, K, 128 >> b, T2_BK, &maps.a[b]);
      if (rc) return rc;
    }
    CUtensorMap gw;
    const int rc = tensor_map(W, (long long)groups * N, K, T2_BM, T2_BK, &gw);
    if (rc) return rc;
    if (swiglu) return launch_tc2_grouped<bf16, true>(maps, gw, C, M, N, K, offsets, groups, stream, swiglu);
    if (out_f32) return launch_tc2_grouped<float, false>(maps, gw, C, M, N, K, offsets, groups, stream, 0);
    return launch_tc2_grouped<bf16, false>(maps, gw, C, M, N, K, offsets, groups, stream, unary);
  }
  const int row_tiles = (M + 2 * T2_BM - 1) / (2 * T2_BM);
  if (row_tiles <= 0) return SNK_ERR_SIZE;
  CUtensorMap map_a, map_w;
  int rc = tensor_map(A, M, K, T2_BM, T2_BK, &map_a);
  if (rc) return rc;
  rc = tensor_map(W, N, K, T2_BN / 2, T2_BK, &map_w);
  if (rc) return rc;
  if (swiglu) return launch_tc2<bf16, true>(map_a, map_w, C, M, N, K, row_tiles, stream, swiglu);
  if (out_f32 == 2) return launch_tc2<float, false, true>(map_a, map_w, C, M, N, K, row_tiles, stream, 0);
  if (out_f32) return launch_tc2<float, false>(map_a, map_w, C, M, N, K, row_tiles, stream, 0);
  return launch_tc2<bf16, false>(map_a, map_w, C, M, N, K, row_tiles, stream, 0);
}

// Test hook: with on != 0 the producers of later launches issue no loads, so that the bounded waits run out
// (about 1.5 s) and the launches return with an error status instead of a product.  Synchronises.
SNK_API int snk_gemm_tc2_test_lose_loads(int on) {
  return (int)cudaMemcpyToSymbol(g_t2_lose_loads, &on, sizeof(int));
}

// Queue a copy of the status word into ``host`` (pinned host memory, one int) on ``stream`` without waiting
// for it and without clearing it: a caller that synchronises with the stream anyway (an event, a read-back)
// learns of a wait that ran out at no cost.  Not for use inside a stream capture.
SNK_API int snk_gemm_tc2_status_peek(int* host, void* stream) {
  return (int)cudaMemcpyFromSymbolAsync(host, g_t2_status, sizeof(int), 0, cudaMemcpyDeviceToHost, (cudaStream_t)stream);
}

// 0, or the first error a block of any earlier launch recorded (a wait that ran out); reading clears it.
// tmem (may be null): the tensor-memory addresses the two blocks of the first pair were given.  Synchronises.
SNK_API int snk_gemm_tc2_status(unsigned int* tmem) {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_t2_status, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_t2_status, &zero, sizeof(int));
  if (tmem && cudaMemcpyFromSymbol(tmem, g_t2_tmem, 2 * sizeof(unsigned int)) != cudaSuccess) return -1;
  return v;
}
