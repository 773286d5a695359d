// C[M,N] = A[M,K] . W[N,K]^T in bfloat16 for few rows (decode: M up to 64), bound by the read of W.
//
// Two kernels, which come to the same bits.  The first one's weights stream from HBM exactly once, straight into tensor-core
// fragments; the second one (further down: plain products of up to 16 rows, where stream_pays says so) brings W through a
// ring in shared memory.  A block of the first owns 16 rows of W (16 output features).  Its 8 warps split K in
// interleaved 32-element blocks; a warp multiplies its 16x32 piece of W with up to 64 tokens by
// mma.sync m16n8k16 (W as the 16-row operand, 8 tokens as the 8-column operand) and the 8 partial
// sums meet in shared memory, added in warp order: no atomics, the same bits every run, and a
// token's result does not depend on which other tokens the launch holds.
//
// Fragment trick: lane (g, t) loads 16 contiguous bytes (8 k-values at k0 + 8t) of W rows g and
// g + 8 and of token row g.  The first four values feed one MMA, the last four a second one; the
// two MMAs see a permutation of the 32 k-values, the same one for both operands, which a dot
// product does not mind.  So every global load is a full 16-byte vector and no shuffle is needed.
//
// Few output features (N/16 blocks would leave SMs idle): a thread-block cluster of S blocks along z
// shares one 16-row strip of W and splits K S ways more; the S partial sums meet in the first block
// through distributed shared memory, added in rank order.  S depends on N and K alone.
//
// Grouped form (routed experts): rows are sorted by group; group e owns rows
// [offsets[e], offsets[e+1]) and uses W + e*N*K; a_rows gathers A (row r reads A[a_rows[r] / a_div]).
// A group with more than 64 rows is walked in passes of 64 (W is then re-read from L2).
// (the role of snowllm/ops/gemm.py:33-41 and the expert products of snowllm/ops/inference.py:60-76
// at decode shapes)
#include "tma.cuh"

#ifndef SK_WARPS
#define SK_WARPS 8
#endif
#define SK_ROWS 16
#define SK_KBLOCK 32
#ifndef SK_UNROLL
#define SK_UNROLL 4
#endif
#ifndef SK_PREFETCH_LINES
#define SK_PREFETCH_LINES 4    // rounds of 16 lines of 128 bytes per row that a block asks L2 for ahead of its wait
                               // (measured in the decode step of one request while all its plain products ran here, 0 / 2 / 4
                               // rounds: 1.497 / 1.482 / 1.476 ms; now its dense gate|up and its head do)
#endif

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// SWIGLU: W holds gate and up rows interleaved in blocks of 8 (rows 16j..16j+7: gate of features
// 8j..8j+7, rows 16j+8..16j+15: their up rows), so a block's 16 rows are 8 features' gate and up; the
// store is then silu(gate) * up into C[M, N/2].
template <int MT, typename OutT, bool SWIGLU>
__global__ void __launch_bounds__(SK_WARPS * 32)
gemm_skinny_kernel(const bf16* __restrict__ A, const bf16* __restrict__ W, OutT* __restrict__ C, int M,
                   int N, int K, const int* __restrict__ a_rows, int a_div,
                   const int* __restrict__ offsets, int groups, int act, int w_ahead) {
#if SK_PREFETCH_LINES > 0
  if (w_ahead && offsets == nullptr) {
    // W is a weight (the caller says so) and this block's 16 rows of it are known from the block's number
    // alone: while the kernel before this one ends, ask L2 for the first lines of each row (128 bytes a
    // thread and round; no register is held, nothing is read into the SM).  A grouped product does not
    // know before the wait which groups own rows.  (Told by the caller that the offsets are older than the kernel in
    // front, the experts' second product of one token asked for its rows while the first one ran: it took as long as
    // without, 9 us, and the first one 25 us instead of 16.)
    const int row = min((int)(blockIdx.x * SK_ROWS + (threadIdx.x >> 4)), N - 1);
    const char* base = reinterpret_cast<const char*>(W + (size_t)row * K);
    const int row_bytes = K * 2;
    const int first = blockIdx.z * (row_bytes / (int)gridDim.z) & ~127;      // a cluster's blocks split K
#pragma unroll
    for (int i = 0; i < SK_PREFETCH_LINES; ++i) {
      const int off = first + ((threadIdx.x & 15) + 16 * i) * 128;
      if (off < row_bytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(base + off));
    }
  }
#endif
  pdl_begin();
  __shared__ float red[SK_WARPS][MT * 8][SK_ROWS + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * SK_ROWS;
  int row_begin = 0, row_end = M;
  const bf16* Wg = W;
  if (offsets) {
    // groups > gridDim.y: there are fewer rows than groups, and block y takes the y-th group that owns any (every warp
    // looks it up for itself).  One token with the top 4 of 32 experts then starts 896 blocks and not 7,168 of which
    // 6,272 end at once: 18.8 -> 16 us of the gate|up product in the decode step.  (With as many rows as groups, 8 such
    // tokens, the look-up cost as much as it saved.)  The look-up has the group's rows in its registers: no second read.
    int e = blockIdx.y;
    if (groups > (int)gridDim.y) {
      int left = blockIdx.y;
      e = -1;
      for (int e0 = 0; e0 < groups; e0 += 32) {
        const bool in = e0 + lane < groups;
        const int begin = in ? offsets[e0 + lane] : 0, end = in ? offsets[e0 + lane + 1] : 0;
        const bool owns = end > begin;
        const unsigned own = __ballot_sync(0xffffffffu, owns);
        const unsigned it = __ballot_sync(0xffffffffu, owns && __popc(own & ((1u << lane) - 1)) == left);
        if (it) {
          const int from = __ffs(it) - 1;
          e = e0 + from;
          row_begin = __shfl_sync(0xffffffffu, begin, from);
          row_end = __shfl_sync(0xffffffffu, end, from);
          break;
        }
        left -= __popc(own);
      }
      if (e < 0) return;
    } else {
      row_begin = offsets[e];
      row_end = offsets[e + 1];
    }
    Wg = W + (size_t)e * N * K;
  }
  if (row_begin >= row_end) return;
  // the two W rows of this lane (rows past N read row N-1 and are dropped at the store)
  const bf16* w_lo = Wg + (size_t)min(n0 + g, N - 1) * K + 8 * t;
  const bf16* w_hi = Wg + (size_t)min(n0 + g + 8, N - 1) * K + 8 * t;
  const int kblocks = (K + SK_KBLOCK - 1) / SK_KBLOCK;
  const int split = gridDim.z, rank = blockIdx.z;         // the cluster spans z: S blocks split K further
  const int vwarp = rank * SK_WARPS + warp, vwarps = split * SK_WARPS;

  for (int m0 = row_begin; m0 < row_end; m0 += MT * 8) {
    const bf16* a_ptr[MT];
    bool a_ok[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      const int r = m0 + i * 8 + g;
      a_ok[i] = r < row_end;
      const int src = a_ok[i] ? (a_rows ? a_rows[r] / a_div : r) : 0;
      a_ptr[i] = A + (size_t)src * K + 8 * t;
    }
    float acc[MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int kb0 = vwarp; kb0 < kblocks; kb0 += vwarps * SK_UNROLL) {
      uint4 wl[SK_UNROLL], wh[SK_UNROLL];
#pragma unroll
      for (int u = 0; u < SK_UNROLL; ++u) {
        const int kb = kb0 + u * vwarps;
        const int k = kb * SK_KBLOCK + 8 * t;
        if (kb < kblocks && k < K) {              // K is a multiple of 8: a lane's 8 values are all in or all out
          wl[u] = ldg_stream(w_lo + (size_t)kb * SK_KBLOCK);
          wh[u] = ldg_stream(w_hi + (size_t)kb * SK_KBLOCK);
        } else {
          wl[u] = make_uint4(0, 0, 0, 0);
          wh[u] = make_uint4(0, 0, 0, 0);
        }
      }
#pragma unroll
      for (int u = 0; u < SK_UNROLL; ++u) {
        const int kb = kb0 + u * vwarps;
        const int k = kb * SK_KBLOCK + 8 * t;
        const bool k_ok = kb < kblocks && k < K;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          uint4 x = make_uint4(0, 0, 0, 0);
          if (k_ok && a_ok[i]) x = *reinterpret_cast<const uint4*>(a_ptr[i] + (size_t)kb * SK_KBLOCK);
          mma_bf16(acc[i], wl[u].x, wh[u].x, wl[u].y, wh[u].y, x.x, x.y);
          mma_bf16(acc[i], wl[u].z, wh[u].z, wl[u].w, wh[u].w, x.z, x.w);
        }
      }
    }
    // acc[i] = {(row g, token 2t), (row g, token 2t+1), (row g+8, token 2t), (row g+8, token 2t+1)}
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      red[warp][i * 8 + 2 * t][g] = acc[i][0];
      red[warp][i * 8 + 2 * t + 1][g] = acc[i][1];
      red[warp][i * 8 + 2 * t][g + 8] = acc[i][2];
      red[warp][i * 8 + 2 * t + 1][g + 8] = acc[i][3];
    }
    __syncthreads();
    if (split > 1) {
      // this block's sum over its warps goes to red[0]; the first block then adds the blocks' sums in rank order
      for (int idx = threadIdx.x; idx < MT * 8 * SK_ROWS; idx += SK_WARPS * 32) {
        const int tok = idx / SK_ROWS, r = idx % SK_ROWS;
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < SK_WARPS; ++w) sum += red[w][tok][r];
        red[0][tok][r] = sum;                               // read and written by this thread alone
      }
      cluster_sync();
      if (rank == 0) {
        for (int idx = threadIdx.x; idx < MT * 8 * SK_ROWS; idx += SK_WARPS * 32) {
          const int tok = idx / SK_ROWS, r = idx % SK_ROWS;
          float sum = red[0][tok][r];
          for (int q = 1; q < split; ++q) sum += ld_cluster_f32(&red[0][tok][r], q);
          red[1][tok][r] = sum;
        }
        __syncthreads();
        if constexpr (SWIGLU) {
          for (int idx = threadIdx.x; idx < MT * 8 * (SK_ROWS / 2); idx += SK_WARPS * 32) {
            const int tok = idx / (SK_ROWS / 2), r = idx % (SK_ROWS / 2);
            const int m = m0 + tok, n = n0 + r;
            if (m < row_end && n + 8 < N) {
              const float gate = red[1][tok][r], up = red[1][tok][r + 8];
              C[(size_t)m * (N / 2) + n0 / 2 + r] = from_f<OutT>(glu_out(gate, up, act));
            }
          }
        } else {
          for (int idx = threadIdx.x; idx < MT * 8 * SK_ROWS; idx += SK_WARPS * 32) {
            const int tok = idx / SK_ROWS, r = idx % SK_ROWS;
            const int m = m0 + tok, n = n0 + r;
            if (m < row_end && n < N) C[(size_t)m * N + n] = from_f<OutT>(unary_out(red[1][tok][r], act));
          }
        }
      }
      cluster_sync();                                       // the others' shared memory lives until it has been read
      continue;
    }
    if constexpr (SWIGLU) {
      for (int idx = threadIdx.x; idx < MT * 8 * (SK_ROWS / 2); idx += SK_WARPS * 32) {
        const int tok = idx / (SK_ROWS / 2), r = idx % (SK_ROWS / 2);
        const int m = m0 + tok, n = n0 + r;
        if (m < row_end && n + 8 < N) {
          float gate = 0.f, up = 0.f;
#pragma unroll
          for (int w = 0; w < SK_WARPS; ++w) {
            gate += red[w][tok][r];
            up += red[w][tok][r + 8];
          }
          C[(size_t)m * (N / 2) + n0 / 2 + r] = from_f<OutT>(glu_out(gate, up, act));
        }
      }
    } else {
      for (int idx = threadIdx.x; idx < MT * 8 * SK_ROWS; idx += SK_WARPS * 32) {
        const int tok = idx / SK_ROWS, r = idx % SK_ROWS;
        const int m = m0 + tok, n = n0 + r;
        if (m < row_end && n < N) {
          float s = 0.f;
#pragma unroll
          for (int w = 0; w < SK_WARPS; ++w) s += red[w][tok][r];
          C[(size_t)m * N + n] = from_f<OutT>(unary_out(s, act));
        }
      }
    }
  }
}

// How many blocks share one strip of W (a cluster along z).  A plain product with fewer strips than
// the GPU has SMs is split 4 ways, as long as every warp of the cluster keeps two k-blocks of its own.
// Measured in a replayed chain of launches at 8 rows: 2048 x 2048 6.8 -> 5.1 us, 2048 x 7168 20.6 -> 9.2 us;
// with 384 strips (6144 x 2048) any split lost (8.1 -> 11.0 us), and so did 8 ways everywhere.
// Depends on N and K alone, so a row's sum has the same order whatever else the launch holds.
#define SK_SPLIT 4
#define SK_SPLIT_MAX_STRIPS 148
static int skinny_split(int N, int K, const int* offsets) {
  static int off = -1;                                     // SNOWLLM_B200_SKINNY_SPLIT=0 in the environment: never split
  if (off < 0) {
    const char* e = getenv("SNOWLLM_B200_SKINNY_SPLIT");
    off = (e && e[0] == '0') ? 1 : 0;
  }
  if (offsets || off) return 1;                            // grouped: the groups already multiply the blocks
  const int strips = (N + SK_ROWS - 1) / SK_ROWS, kblocks = (K + SK_KBLOCK - 1) / SK_KBLOCK;
  return (strips <= SK_SPLIT_MAX_STRIPS && kblocks >= 2 * SK_SPLIT * SK_WARPS) ? SK_SPLIT : 1;
}

// ---------------------------------------------------------------------------------------------
// Plain products of up to 16 rows: the same, with W streamed through shared memory.  What bounds them is the read of W,
// and most of what a small one takes beside it is the way from the end of the kernel before to the first bytes of W.  Where
// W is a weight (the caller says so: w_ahead) one block per SM keeps a ring of stages (16 rows x 512 columns each, one TMA
// box, filled by a ninth warp) that starts to fill while the kernel before still runs, and goes on across the block's
// strips of 16 rows; eight warps multiply out of it.  Ring and sums take less than half of an SM's shared memory, so that
// the next product can start beside this one.
//
// The numbers are the same bits as above: warp w takes the 32-column runs w, w + 8, .. of a strip in order, the same MMAs,
// the same order of the warps' sums (SPLIT 4: four sums a warp, as the cluster's blocks held them).  A box brings 64
// columns of a row at a time (128 bytes, swizzled), so two warps share a block of 16 x 128 bytes.  Lane g of the MMA
// holds row st_row(g), an order in which the eight lanes that read shared memory together find their 16 bytes in
// different banks.
//
// Measured, 1 row, in a replayed chain of the product alone (the kernel above): 2,048 x 2,048 5.3 -> 3.0 us, 6,144 x 2,048 8.5 ->
// 7.0, 4,096 x 4,096 14.0 -> 8.7; in the decode steps, where the ring fills ahead, 4.1 -> 2.7 us from the end of the kernel
// before to the end of 2,048 x 2,048 and 7.0 -> 5.6 of 6,144 x 2,048.  Sizes at which it loses: see stream_pays.
// Grouped products stay above: a group's strips are few and each has other rows of A to fetch, so the eight warps of the
// one block cannot hide that as eight blocks an SM do (20 of 32 experts with a row each: 72 us here, 54 above).
#define ST_RUNS 16                              // runs of 32 columns of a stage (8 blocks of 64 columns)
#define ST_BYTES (SK_ROWS * ST_RUNS * 64)
#define ST_MAX_ROWS 16
#define ST_WAIT_NS 1500000000ull

__device__ int g_sk_status;
static int sk_lose_loads = 0;        // test hook: producers issue no loads (the stages then never fill)

__device__ __forceinline__ int st_row(int g) { return (g >> 1) | ((g & 1) << 2); }

struct StShared {
  uint64_t full[8], empty[8];
  int aborted;
};

__device__ __forceinline__ void st_wait(uint64_t* bar, uint32_t parity, volatile int* aborted, int code) {
  if (*aborted || mbar_try_wait(bar, parity)) return;
  const uint64_t start = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (*aborted) return;
    if (global_ns() - start > ST_WAIT_NS) {
      *aborted = 1;
      atomicCAS(&g_sk_status, 0, code);
      return;
    }
  }
}

template <int MT, typename OutT, bool SWIGLU, int SPLIT>
__global__ void __launch_bounds__((SK_WARPS + 1) * 32)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map, const bf16* __restrict__ A, OutT* __restrict__ C, int M, int N,
                   int K, int stages, int act, int w_ahead, int lose_loads) {
  extern __shared__ unsigned char raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  // two sets of sums, so that one barrier a strip is enough (one where four sums a warp would take the ring's room)
  constexpr int SETS = SPLIT == 1 ? 2 : 1;
  float(*red)[SPLIT * SK_WARPS][MT * 8][SK_ROWS + 1] =
      reinterpret_cast<float(*)[SPLIT * SK_WARPS][MT * 8][SK_ROWS + 1]>(ring + (size_t)stages * ST_BYTES);
  StShared* sh = reinterpret_cast<StShared*>(red + SETS);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int strips = (N + SK_ROWS - 1) / SK_ROWS, runs = K / 32, boxes = (runs + ST_RUNS - 1) / ST_RUNS;
  volatile int* aborted = &sh->aborted;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], SK_WARPS);
    }
    sh->aborted = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  int s = 0;
  uint32_t lap = 0;
  auto next_stage = [&]() {
    if (++s == stages) {
      s = 0;
      lap ^= 1;
    }
  };

  if (warp == SK_WARPS) {                                // the producer: reads W alone
    if (lane == 0) {
      // Boxes that go out ahead of the wait for the kernel in front: one ring, whose stages are empty.  The next one waits
      // for warps that wait for that kernel, and its time is not to run while they do.
      int ahead = w_ahead ? stages : 0;
      for (int strip = blockIdx.x; strip < strips && !*aborted; strip += gridDim.x) {
        for (int box = 0; box < boxes; ++box, next_stage()) {
          if (ahead-- == 0) pdl_wait();
          st_wait(&sh->empty[s], lap ^ 1, aborted, 2);
          if (*aborted) break;
          if (lose_loads) continue;
          mbar_expect_tx(&sh->full[s], ST_BYTES);        // a box that reaches past the last run is filled up with zeros
          tma_load_3d(ring + (size_t)s * ST_BYTES, &map, &sh->full[s], 0, strip * SK_ROWS, box * (ST_RUNS / 2));
        }
      }
    }
    if (*aborted) drain_after_abort();
    return;
  }

  pdl_begin();
  const int g = lane >> 2, t = lane & 3, row_g = st_row(g);
  // this lane's 16 bytes of row row_g in its warp's half of a block of 64 columns (rows 8..15 follow 1 KB further on)
  const int place = (warp >> 1) * 2048 + row_g * 128 + ((((warp & 1) * 4 + t) ^ row_g) << 4);
  const bf16* a_ptr[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i) a_ptr[i] = A + (size_t)(i * 8 + g < M ? i * 8 + g : 0) * K + 8 * t;
  int turn = 0;
  for (int strip = blockIdx.x; strip < strips; strip += gridDim.x, turn ^= SETS - 1) {
    uint4 x[2][MT];                                      // this lane's values of A for the two runs of the next box
    auto load_x = [&](int box) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int run = box * ST_RUNS + h * SK_WARPS + warp;
#pragma unroll
        for (int i = 0; i < MT; ++i)
          x[h][i] = i * 8 + g < M && run < runs ? *reinterpret_cast<const uint4*>(a_ptr[i] + (size_t)run * 32)
                                                : make_uint4(0, 0, 0, 0);
      }
    };
    float acc[SPLIT][MT][4];
#pragma unroll
    for (int q = 0; q < SPLIT; ++q)
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[q][i][j] = 0.f;
    auto multiply = [&](int box, float (&lo)[MT][4], float (&hi)[MT][4]) {
      uint4 now[2][MT];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < MT; ++i) now[h][i] = x[h][i];
      load_x(box + 1);                                   // (past the last box: zeros)
      st_wait(&sh->full[s], lap, aborted, 1);
      const unsigned char* stage = ring + (size_t)s * ST_BYTES + place;
      uint4 wl[2], wh[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        wl[h] = *reinterpret_cast<const uint4*>(stage + h * (ST_BYTES / 2));
        wh[h] = *reinterpret_cast<const uint4*>(stage + h * (ST_BYTES / 2) + 1024);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->empty[s]);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        mma_bf16(lo[i], wl[0].x, wh[0].x, wl[0].y, wh[0].y, now[0][i].x, now[0][i].y);
        mma_bf16(lo[i], wl[0].z, wh[0].z, wl[0].w, wh[0].w, now[0][i].z, now[0][i].w);
      }
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        mma_bf16(hi[i], wl[1].x, wh[1].x, wl[1].y, wh[1].y, now[1][i].x, now[1][i].y);
        mma_bf16(hi[i], wl[1].z, wh[1].z, wl[1].w, wh[1].w, now[1][i].z, now[1][i].w);
      }
      next_stage();
    };
    load_x(0);
    if constexpr (SPLIT == 1) {
      for (int box = 0; box < boxes; ++box) multiply(box, acc[0], acc[0]);
    } else {
      static_assert(SPLIT == 1 || SPLIT == 4, "runs 8 q .. 8 q + 7 of every 32 are sum q's");
      for (int box = 0; box < boxes; box += 2) {
        multiply(box, acc[0], acc[1]);
        if (box + 1 < boxes) multiply(box + 1, acc[2], acc[3]);
      }
    }
#pragma unroll
    for (int q = 0; q < SPLIT; ++q)
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        float(*mine)[SK_ROWS + 1] = red[turn][q * SK_WARPS + warp];
        mine[i * 8 + 2 * t][row_g] = acc[q][i][0];
        mine[i * 8 + 2 * t + 1][row_g] = acc[q][i][1];
        mine[i * 8 + 2 * t][row_g + 8] = acc[q][i][2];
        mine[i * 8 + 2 * t + 1][row_g + 8] = acc[q][i][3];
      }
    asm volatile("bar.sync 1, %0;" ::"n"(SK_WARPS * 32) : "memory");
    auto sum_of = [&](int tok, int r) {
      float total = 0.f;
#pragma unroll
      for (int q = 0; q < SPLIT; ++q) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < SK_WARPS; ++w) sum += red[turn][q * SK_WARPS + w][tok][r];
        total = q == 0 ? sum : total + sum;
      }
      return total;
    };
    const int n0 = strip * SK_ROWS, toks = min(MT * 8, M);
    if constexpr (SWIGLU) {
      for (int idx = threadIdx.x; idx < toks * (SK_ROWS / 2); idx += SK_WARPS * 32) {
        const int tok = idx / (SK_ROWS / 2), r = idx % (SK_ROWS / 2);
        if (n0 + r + 8 < N)
          C[(size_t)tok * (N / 2) + n0 / 2 + r] = from_f<OutT>(glu_out(sum_of(tok, r), sum_of(tok, r + 8), act));
      }
    } else {
      for (int idx = threadIdx.x; idx < toks * SK_ROWS; idx += SK_WARPS * 32) {
        const int tok = idx / SK_ROWS, r = idx % SK_ROWS;
        if (n0 + r < N) C[(size_t)tok * N + n0 + r] = from_f<OutT>(unary_out(sum_of(tok, r), act));
      }
    }
    if constexpr (SETS == 1) asm volatile("bar.sync 1, %0;" ::"n"(SK_WARPS * 32) : "memory");
  }
  // the producer may have issued its last box and gone before a wait ran out here: the warp that gave up keeps the
  // block's shared memory until the boxes on their way have landed
  if (*aborted) drain_after_abort();
}

// Where the ring is the faster of the two kernels.  It gains at the start of a product and where N gives the kernel above
// one to three blocks an SM, too few loads on their way; it loses where that one fills the SMs (4 and more strips an SM: 16 KB
// a stage and 0.5 us of multiplying 8 rows hold a block to 4.9 TB/s of all SMs, there 5.9), where a strip is a short walk
// (a round of strips costs more than its bytes), and where few strips are long walks, which the cluster above divides by four.
// Measured in replayed chains of a norm and the product, M 1 / 4 / 8 / 16, us here (there):
//   one round   2,048 x 2,048 5.7 (6.5) / 5.7 (6.6) / 5.9 (7.1) / 6.7 (8.9); 512 x 1,024 3.5 (4.0) / 3.8 (4.6) / 4.0 (4.7) / 4.2 (6.2);
//               512 x 4,096 1.04 to 1.15 times there, 256 x 16,384 1.23 to 1.47, 2,048 x 10,752 0.94 / 1.04 / 1.04 / 0.89,
//               2,048 x 20,480 1.04 to 1.18
//   two         4,096 x 4,096 0.69 / 0.75 / 0.80 / 0.75 times there, x 1,024 0.98 / 0.99 / 1.02 / 0.90, x 256 1.07 / 1.04 / 1.05 / 0.99
//   three       6,144 x 2,048 0.96 / 0.98 / 1.03 / 1.00, x 4,096 0.82 / 0.90 / 0.96 / 0.96, x 1,024 1.05 / 1.07 / 1.14 / 1.06,
//               x 20,480 0.84 / 1.05 / 1.12 / 1.07
//   more        8,192 x 2,048 1.02 / 1.06 / 1.13 / 1.11, 16,384 x 2,048 0.91 / 0.99 / 1.08 / 1.04 (but gate|up and down of 2,048 and 7,168
//               together 25.7 / 27.8 / 29.8 / 35.3 us with gate|up here, 24.1 / 25.0 / 25.7 / 31.4 with it there), 65,536 x 2,048 1.12 /
//               1.12 / 1.28 / 1.26, 128,256 x 1,024 1.39 to 1.51
static bool stream_pays(int N, int K, int sms) {
  const int strips = (N + SK_ROWS - 1) / SK_ROWS, rounds = (strips + sms - 1) / sms;
  if (rounds <= 1) return K <= 2560 || (strips >= sms * 3 / 4 && K <= 12288);
  if (rounds == 2) return K >= 512;
  return rounds == 3 && K >= 2048 && K <= 16384;
}

// For tests: whether a plain product of these sizes streams W through shared memory on a device of that many SMs.
SNK_API int snk_gemm_skinny_streams(int M, int N, int K, int sms) {
  return M <= ST_MAX_ROWS && K % 64 == 0 && stream_pays(N, K, sms);
}

template <int MT, typename OutT, bool SWIGLU, int SPLIT>
static int launch_stream(const CUtensorMap& map, const bf16* A, void* C, int M, int N, int K, int act, int w_ahead, int sms,
                         cudaStream_t stream) {
  constexpr int sums = (SPLIT == 1 ? 2 : 1) * SPLIT * SK_WARPS * MT * 8 * (SK_ROWS + 1) * (int)sizeof(float);
  // two products' rings on one SM: 6 stages of 16 KB, fewer where the sums take the room
  constexpr int room = (110 * 1024 - sums - (int)sizeof(StShared)) / ST_BYTES, stages = room < 6 ? room : 6;
  constexpr int smem = 1024 + stages * ST_BYTES + sums + (int)sizeof(StShared);
  static std::atomic<int> limit_set[SNK_MAX_DEVICES];
  int device = 0, set = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  const int rc = snk_per_device(limit_set, device, &set, [&](int* n) {
    *n = 1;
    return (int)cudaFuncSetAttribute(gemm_stream_kernel<MT, OutT, SWIGLU, SPLIT>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (rc) return rc;
  const int strips = (N + SK_ROWS - 1) / SK_ROWS;
  snk_launch(gemm_stream_kernel<MT, OutT, SWIGLU, SPLIT>, dim3(strips < sms ? strips : sms), dim3((SK_WARPS + 1) * 32), smem,
             stream, map, A, static_cast<OutT*>(C), M, N, K, stages, act, w_ahead, sk_lose_loads);
  SNK_LAUNCH_CHECK();
  return 0;
}

template <int MT>
static int stream_product(const CUtensorMap& map, const void* A, void* C, int M, int N, int K, int out_f32, int swiglu,
                          int split, int w_ahead, int sms, cudaStream_t stream) {
  const bf16* a = static_cast<const bf16*>(A);
  if (swiglu && swiglu != SNK_ACT_RELU2)
    return split > 1 ? launch_stream<MT, bf16, true, SK_SPLIT>(map, a, C, M, N, K, swiglu, w_ahead, sms, stream)
                     : launch_stream<MT, bf16, true, 1>(map, a, C, M, N, K, swiglu, w_ahead, sms, stream);
  if (out_f32)
    return split > 1 ? launch_stream<MT, float, false, SK_SPLIT>(map, a, C, M, N, K, 0, w_ahead, sms, stream)
                     : launch_stream<MT, float, false, 1>(map, a, C, M, N, K, 0, w_ahead, sms, stream);
  return split > 1 ? launch_stream<MT, bf16, false, SK_SPLIT>(map, a, C, M, N, K, swiglu, w_ahead, sms, stream)
                   : launch_stream<MT, bf16, false, 1>(map, a, C, M, N, K, swiglu, w_ahead, sms, stream);
}

template <int MT>
static int launch_skinny(const void* A, const void* W, void* C, int M, int N, int K, const int* a_rows,
                         int a_div, const int* offsets, int groups, int out_f32, int swiglu, int split,
                         int w_ahead, cudaStream_t stream) {
  // Fewer rows than groups: a block per row and strip, which looks its group up, unless the blocks of all groups are on the SMs
  // at once (8 to each) and the idle ones cost nothing (8 groups of 512 x 256, one token with two of them: 3.0 / 2.8 us).
  const int strips = (N + SK_ROWS - 1) / SK_ROWS;
  int sms = 0, per_group = groups;
  if (offsets && groups > M) {
    const int rc = snk_device_sms(&sms);
    if (rc) return rc;
    if ((long long)strips * groups > 8ll * sms) per_group = M;
  }
  dim3 grid(strips, offsets ? per_group : 1, split);
  const dim3 block(SK_WARPS * 32);
  const bf16 *a = static_cast<const bf16*>(A), *w = static_cast<const bf16*>(W);
  const int unary = swiglu == SNK_ACT_RELU2 ? swiglu : 0;
  if (swiglu && !unary)
    snk_launch_cluster(gemm_skinny_kernel<MT, bf16, true>, grid, block, 0, stream, split, a, w,
                       static_cast<bf16*>(C), M, N, K, a_rows, a_div, offsets, groups, swiglu, w_ahead);
  else if (out_f32)
    snk_launch_cluster(gemm_skinny_kernel<MT, float, false>, grid, block, 0, stream, split, a, w,
                       static_cast<float*>(C), M, N, K, a_rows, a_div, offsets, groups, 0, w_ahead);
  else
    snk_launch_cluster(gemm_skinny_kernel<MT, bf16, false>, grid, block, 0, stream, split, a, w,
                       static_cast<bf16*>(C), M, N, K, a_rows, a_div, offsets, groups, unary, w_ahead);
  SNK_LAUNCH_CHECK();
  return 0;
}

// rows_hint: the most rows one group (or the whole product) is expected to hold; picks how many
// 8-token tiles a pass covers.  More rows than that still give the right result, in more passes.
// swiglu: W is gate/up interleaved in blocks of 8 rows and C is [M, N/2] bfloat16 = silu(gate) * up (or, SNK_ACT_RELU2:
// C is [M, N] bfloat16, the square of relu of the product).
// w_ahead: W was there before the kernel in front of this launch began, and may be read ahead of the wait for it.
SNK_API int snk_gemm_skinny(const void* A, const void* W, void* C, int M, int N, int K, const int* a_rows,
                            int a_div, const int* offsets, int groups, int rows_hint, int out_f32, int swiglu,
                            int w_ahead, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 8) return SNK_ERR_SIZE;
  if (swiglu && ((swiglu != SNK_ACT_RELU2 && N % 16) || out_f32)) return SNK_ERR_SIZE;
  if (((uintptr_t)A % 16) || ((uintptr_t)W % 16)) return SNK_ERR_ALIGN;
  if (groups > 65535) return SNK_ERR_SIZE;
  if (a_div <= 0) a_div = 1;
  const int split = skinny_split(N, K, offsets);
  // K in whole blocks of 64 columns, one pass: W through shared memory, where that is the faster way
  if (!offsets && !a_rows && M <= ST_MAX_ROWS && K % 64 == 0) {
    int sms = 0;
    int rc = snk_device_sms(&sms);
    if (rc) return rc;
    if (stream_pays(N, K, sms)) {
      CUtensorMap map;
      rc = tensor_map(W, N, K, SK_ROWS, 0, &map, ST_RUNS / 2);
      if (rc) return rc;
      if (M <= 8) return stream_product<1>(map, A, C, M, N, K, out_f32, swiglu, split, w_ahead, sms, stream);
      return stream_product<2>(map, A, C, M, N, K, out_f32, swiglu, split, w_ahead, sms, stream);
    }
  }
  if (rows_hint <= 8) return launch_skinny<1>(A, W, C, M, N, K, a_rows, a_div, offsets, groups, out_f32, swiglu, split, w_ahead, stream);
  if (rows_hint <= 16) return launch_skinny<2>(A, W, C, M, N, K, a_rows, a_div, offsets, groups, out_f32, swiglu, split, w_ahead, stream);
  if (rows_hint <= 32) return launch_skinny<4>(A, W, C, M, N, K, a_rows, a_div, offsets, groups, out_f32, swiglu, split, w_ahead, stream);
  return launch_skinny<8>(A, W, C, M, N, K, a_rows, a_div, offsets, groups, out_f32, swiglu, split, w_ahead, stream);
}

// Test hook: with on != 0 the producers of later launches issue no loads, so that the bounded waits run out
// (about 1.5 s) and the launches return with an error status instead of a product.
SNK_API int snk_gemm_skinny_test_lose_loads(int on) {
  sk_lose_loads = on;
  return 0;
}

// Queue a copy of the status word into ``host`` (pinned host memory, one int) on ``stream`` without waiting
// for it and without clearing it.  Not for use inside a stream capture.
SNK_API int snk_gemm_skinny_status_peek(int* host, void* stream) {
  return (int)cudaMemcpyFromSymbolAsync(host, g_sk_status, sizeof(int), 0, cudaMemcpyDeviceToHost, (cudaStream_t)stream);
}

// 0, or the code of a wait that ran out in any earlier launch (1: a stage never filled, 2: one never came back);
// reading clears it.  Synchronises.
SNK_API int snk_gemm_skinny_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_sk_status, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_sk_status, &zero, sizeof(int));
  return v;
}
