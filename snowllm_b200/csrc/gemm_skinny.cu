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

struct __align__(16) StShared {      // (the rows of a norm, read 16 bytes at a time, lie behind it)
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

// What a step of a few one-token rows has its products do beside the multiplying (ST_NORM, ST_CONV of FUSE).  Such a step is
// a chain of small launches, and from the end of one kernel to the end of a next that does next to nothing are 3 to 4 us.
//
// ST_NORM: the rows of A are not there yet, but a residual, what is added to it, and the weight of an RMS norm.  Every block
// forms the rows for itself in shared memory (the sum, its mean square, the rounded row: add_rmsnorm_kernel's arithmetic in its
// order, so that a request's rows are the same bits whether one, two or more requests are in the step) and
// writes its share of the new residual, to other memory than it is read from, as other blocks may still be reading.
// ST_CONV: W is [B | C | x], three times H rows, and every row of A is one token of a request of its own.  A unit of 16
// channels is their three strips, one after the other by the same block, whose threads keep the strips' sums, and the store is
// the gated convolution over the channel's history (short_conv_decode_kernel's arithmetic), which it brings up to date.
// Measured, a decode step before / with both, us: 1.2B sizes 1 request 759 / 672, 2 requests 780 / 692; 2.6B sizes 1 request 1,502 / 1,365;
// 8B-A1B sizes 1 request 1,288 / 1,219, 2 requests 1,637 / 1,613.  With the norm's weight loaded behind the sum 707 of 759; the
// convolution alone gains nothing at 8 rows.  The squares summed in an order of the block's own / in the norm's: 670.1 / 670.6 and 1,226 /
// 1,215.
enum { ST_NORM = 1, ST_CONV = 2 };
#define ST_FUSE_ROWS 2                          // rows a launch may have
#define ST_NORM_VECS 4                          // vectors of four a thread may hold of a row
#define ST_NORM_SMEM (2 * (2048 + 8) * 2)       // bytes of shared memory for the rows: 2 of 2,048, or one of 4,096
#define ST_CONV_TAPS 4
struct StFuse {
  // ST_NORM: residual [M, K], plus delta [M, K] or the routed experts' weighted sum (as add_rmsnorm_kernel takes it)
  const float *residual, *delta, *moe_y, *topk_w;
  const int* pair_pos;
  float* new_residual;
  SmallVec gamma;
  int k;
  float eps;
  // ST_CONV: state [slots, taps - 1, H]
  SmallVec taps;
  bf16* state;
  const int *seg_start, *seg_slot;
  int L;
};

// By the eight multiplying warps: rows of the norm into xs [M][pitch].  Two rows share the warps evenly; a thread has all its
// loads on their way before the first is used.  ST_GAMMA loads its values of the norm's weight (ahead of the wait for the kernel
// in front, where the caller says so: it is a weight as W is).
struct StNormPart {
  int row, tid, threads, n4;
  __device__ __forceinline__ StNormPart(int M, int K) {
    const int per_row = M == 1 ? SK_WARPS : SK_WARPS / 2;
    row = (threadIdx.x >> 5) / per_row;
    threads = per_row * 32;
    tid = threadIdx.x - row * threads;
    n4 = K / 4;
  }
};
__device__ __forceinline__ void st_gamma(const StFuse& f, const StNormPart& p, float4 (&g)[ST_NORM_VECS]) {
#pragma unroll
  for (int j = 0; j < ST_NORM_VECS; ++j) {
    const int i = p.tid + j * p.threads;
    g[j] = i < p.n4 ? make_float4(f.gamma[4 * i], f.gamma[4 * i + 1], f.gamma[4 * i + 2], f.gamma[4 * i + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
__device__ __forceinline__ void st_norm_rows(const StFuse& f, const StNormPart& p, const float4 (&g)[ST_NORM_VECS], bf16* xs, int pitch,
                                             float* red, int M, int K) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per_row = p.threads / 32;
  const int chains = max(norm_threads(K) / p.threads, 1);                   // 1, 2 or 4
  const bool mine = p.row < M;
  float4 v[ST_NORM_VECS];
  float squares[ST_NORM_VECS] = {};
  if (mine) {
    const float4* res4 = reinterpret_cast<const float4*>(f.residual + (size_t)p.row * K);
#pragma unroll
    for (int j = 0; j < ST_NORM_VECS; ++j) {
      const int i = p.tid + j * p.threads;
      v[j] = i < p.n4 ? res4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (f.moe_y) {
      float4 acc[ST_NORM_VECS];
#pragma unroll
      for (int j = 0; j < ST_NORM_VECS; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int q = 0; q < f.k; ++q) {
        const float w = f.topk_w[p.row * f.k + q];
        const float4* y4 = reinterpret_cast<const float4*>(f.moe_y + (size_t)f.pair_pos[p.row * f.k + q] * K);
#pragma unroll
        for (int j = 0; j < ST_NORM_VECS; ++j) {
          const int i = p.tid + j * p.threads;
          if (i < p.n4) {
            const float4 y = y4[i];
            acc[j].x = fmaf(w, y.x, acc[j].x); acc[j].y = fmaf(w, y.y, acc[j].y);
            acc[j].z = fmaf(w, y.z, acc[j].z); acc[j].w = fmaf(w, y.w, acc[j].w);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < ST_NORM_VECS; ++j) {
        v[j].x += acc[j].x; v[j].y += acc[j].y; v[j].z += acc[j].z; v[j].w += acc[j].w;
      }
    } else if (f.delta) {
      const float4* d4 = reinterpret_cast<const float4*>(f.delta + (size_t)p.row * K);
#pragma unroll
      for (int j = 0; j < ST_NORM_VECS; ++j) {
        const int i = p.tid + j * p.threads;
        if (i < p.n4) {
          const float4 d = d4[i];
          v[j].x += d.x; v[j].y += d.y; v[j].z += d.z; v[j].w += d.w;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < ST_NORM_VECS; ++j) {             // a thread here is `chains` of the norm's kernel, of every chains-th vector each
      float ss = 0.f;
      if (j >= 1 && chains == 1) ss = squares[j - (j >= 1)];
      if (j >= 2 && chains == 2) ss = squares[j - 2 * (j >= 2)];
      ss = fmaf(v[j].x, v[j].x, ss); ss = fmaf(v[j].y, v[j].y, ss);
      ss = fmaf(v[j].z, v[j].z, ss); ss = fmaf(v[j].w, v[j].w, ss);
      squares[j] = ss;
    }
  }
  // block_sum of those threads: a sum a warp of theirs, and then the warps'
#pragma unroll
  for (int j = 0; j < ST_NORM_VECS; ++j) {
    if (j < ST_NORM_VECS - chains) continue;             // (continued by a later vector's)
    const float ss = warp_sum(squares[j]);
    if (lane == 0) red[p.row * 16 + (j - (ST_NORM_VECS - chains)) * per_row + warp - p.row * per_row] = ss;
  }
  asm volatile("bar.sync 1, %0;" ::"n"(SK_WARPS * 32) : "memory");
  if (mine) {
    const float sum = warp_sum(lane < chains * per_row ? red[p.row * 16 + lane] : 0.f);
    const float inv = rsqrtf(sum / (float)K + f.eps);
#pragma unroll
    for (int j = 0; j < ST_NORM_VECS; ++j) {
      const int i = p.tid + j * p.threads;
      if (i < p.n4) {
        store4<bf16>(xs + (size_t)p.row * pitch + 4 * i, v[j].x * inv * g[j].x, v[j].y * inv * g[j].y, v[j].z * inv * g[j].z,
                     v[j].w * inv * g[j].w);
        if (f.new_residual && i % gridDim.x == blockIdx.x)
          reinterpret_cast<float4*>(f.new_residual + (size_t)p.row * K)[i] = v[j];
      }
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(SK_WARPS * 32) : "memory");
}

__host__ __device__ constexpr int st_norm_pitch(int K) { return K + 8; }     // bf16 of a row in shared memory (banks shift by 16 bytes)

template <int MT, typename OutT, bool SWIGLU, int SPLIT, int FUSE>
__global__ void __launch_bounds__((SK_WARPS + 1) * 32, (FUSE & ST_NORM) ? 2 : MT == 1 ? 3 : SPLIT == 1 ? 2 : 0)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map, const bf16* __restrict__ A, OutT* __restrict__ C, int M, int N,
                   int K, int stages, int act, int w_ahead, int lose_loads, const StFuse f) {
  extern __shared__ unsigned char raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  // two sets of sums, so that one barrier a strip is enough (one where four sums a warp would take the ring's room)
  constexpr int SETS = SPLIT == 1 ? 2 : 1;
  float(*red)[SPLIT * SK_WARPS][MT * 8][SK_ROWS + 1] =
      reinterpret_cast<float(*)[SPLIT * SK_WARPS][MT * 8][SK_ROWS + 1]>(ring + (size_t)stages * ST_BYTES);
  StShared* sh = reinterpret_cast<StShared*>(red + SETS);
  bf16* xs = reinterpret_cast<bf16*>(sh + 1);            // ST_NORM: the rows of A
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int strips = (N + SK_ROWS - 1) / SK_ROWS, runs = K / 32, boxes = (runs + ST_RUNS - 1) / ST_RUNS;
  // this block's strips: every gridDim.x-th, or (ST_CONV) the three strips of every gridDim.x-th unit
  constexpr int PARTS = FUSE & ST_CONV ? 3 : 1;
  const int H = N / PARTS, units = strips / PARTS;
  const int walk = ((units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * PARTS;
  auto first_row = [&](int i) { return (i % PARTS) * H + ((int)blockIdx.x + i / PARTS * (int)gridDim.x) * SK_ROWS; };
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
      for (int i = 0; i < walk && !*aborted; ++i) {
        const int w_row = first_row(i);
        for (int box = 0; box < boxes; ++box, next_stage()) {
          if (ahead-- == 0) pdl_wait();
          st_wait(&sh->empty[s], lap ^ 1, aborted, 2);
          if (*aborted) break;
          if (lose_loads) continue;
          mbar_expect_tx(&sh->full[s], ST_BYTES);        // a box that reaches past the last run is filled up with zeros
          tma_load_3d(ring + (size_t)s * ST_BYTES, &map, &sh->full[s], 0, w_row, box * (ST_RUNS / 2));
        }
      }
    }
    if (*aborted) drain_after_abort();
    return;
  }

  const StNormPart norm_part(M, K);
  float4 gamma[ST_NORM_VECS];
  if constexpr (FUSE & ST_NORM) {
    if (w_ahead) st_gamma(f, norm_part, gamma);
  }
  pdl_begin();
  if constexpr (FUSE & ST_NORM) {
    if (!w_ahead) st_gamma(f, norm_part, gamma);
  }
  const int g = lane >> 2, t = lane & 3, row_g = st_row(g);
  // this lane's 16 bytes of row row_g in its warp's half of a block of 64 columns (rows 8..15 follow 1 KB further on)
  const int place = (warp >> 1) * 2048 + row_g * 128 + ((((warp & 1) * 4 + t) ^ row_g) << 4);
  const int toks = min(MT * 8, M);
  // ST_CONV: this thread's token and channel of a unit, what it needs of the channel's history, and the strips' sums
  const int my_tok = threadIdx.x / SK_ROWS, my_r = threadIdx.x % SK_ROWS;
  const bool conv_mine = (FUSE & ST_CONV) && my_tok < toks;
  bf16* hist_at = nullptr;
  bool has_state = false;
  float tap[ST_CONV_TAPS], hist[ST_CONV_TAPS - 1], gate_b = 0.f, gate_c = 0.f;
  if constexpr (FUSE & ST_CONV) {
    if (conv_mine) {
      has_state = f.seg_start[my_tok] > 0;
      hist_at = f.state + (size_t)f.seg_slot[my_tok] * (f.L - 1) * H;
    }
  }
  if constexpr (FUSE & ST_NORM) {
    st_norm_rows(f, norm_part, gamma, xs, st_norm_pitch(K), &red[0][0][0][0], M, K);
    A = xs;
  }
  const int a_pitch = FUSE & ST_NORM ? st_norm_pitch(K) : K;
  const bf16* a_ptr[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i) a_ptr[i] = A + (size_t)(i * 8 + g < M ? i * 8 + g : 0) * a_pitch + 8 * t;
  int turn = 0;
  for (int i_strip = 0; i_strip < walk; ++i_strip, turn ^= SETS - 1) {
    const int n0 = first_row(i_strip), part = i_strip % PARTS;
    if constexpr (FUSE & ST_CONV) {
      if (part == 0 && conv_mine) {                      // on their way while the first strip is multiplied
        const int c = n0 + my_r;
#pragma unroll
        for (int j = 0; j < ST_CONV_TAPS; ++j)
          if (j < f.L) tap[j] = f.taps[(size_t)c * f.L + j];
#pragma unroll
        for (int j = 0; j < ST_CONV_TAPS - 1; ++j)
          if (j < f.L - 1) hist[j] = has_state ? to_f<bf16>(hist_at[(size_t)j * H + c]) : 0.f;
      }
    }
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
    if constexpr (FUSE & ST_CONV) {
      if (conv_mine) {
        const float v = round_f<bf16>(sum_of(my_tok, my_r));             // as the product's store leaves it
        if (part == 0) gate_b = v;
        else if (part == 1) gate_c = v;
        else {
          const int c = n0 - 2 * H + my_r;
          const float now = round_f<bf16>(gate_b * v);
          float acc = 0.f, last = 0.f;                   // taps in order: oldest first, the current token last
#pragma unroll
          for (int j = 0; j < ST_CONV_TAPS; ++j) {
            if (j < f.L - 1) acc = fmaf(tap[j], hist[j < ST_CONV_TAPS - 1 ? j : 0], acc);
            else if (j == f.L - 1) last = tap[j];
          }
          acc = fmaf(last, now, acc);
          C[(size_t)my_tok * H + c] = from_f<OutT>(gate_c * acc);
#pragma unroll
          for (int j = 0; j < ST_CONV_TAPS - 1; ++j)
            if (j < f.L - 1)
              hist_at[(size_t)j * H + c] = from_f<bf16>(j + 1 < f.L - 1 ? hist[j + 1 < ST_CONV_TAPS - 1 ? j + 1 : 0] : now);
        }
      }
    } else if constexpr (SWIGLU) {
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

template <int MT, typename OutT, bool SWIGLU, int SPLIT, int FUSE = 0>
static int launch_stream(const CUtensorMap& map, const bf16* A, void* C, int M, int N, int K, int act, int w_ahead, int sms,
                         cudaStream_t stream, const StFuse& f = StFuse{}) {
  constexpr int sums = (SPLIT == 1 ? 2 : 1) * SPLIT * SK_WARPS * MT * 8 * (SK_ROWS + 1) * (int)sizeof(float);
  // two products' rings on one SM: 6 stages of 16 KB, fewer where the sums (or the rows of a norm) take the room
  constexpr int rows_of_norm = FUSE & ST_NORM ? ST_NORM_SMEM : 0, most = 110 * 1024;
  constexpr int room = (most - sums - rows_of_norm - (int)sizeof(StShared)) / ST_BYTES, stages = room < 6 ? room : 6;
  constexpr int smem = 1024 + stages * ST_BYTES + sums + rows_of_norm + (int)sizeof(StShared);
  static std::atomic<int> limit_set[SNK_MAX_DEVICES];
  int device = 0, set = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  const int rc = snk_per_device(limit_set, device, &set, [&](int* n) {
    *n = 1;
    return (int)cudaFuncSetAttribute(gemm_stream_kernel<MT, OutT, SWIGLU, SPLIT, FUSE>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (rc) return rc;
  const int units = (N + SK_ROWS - 1) / SK_ROWS / (FUSE & ST_CONV ? 3 : 1);
  snk_launch(gemm_stream_kernel<MT, OutT, SWIGLU, SPLIT, FUSE>, dim3(units < sms ? units : sms), dim3((SK_WARPS + 1) * 32), smem,
             stream, map, A, static_cast<OutT*>(C), M, N, K, stages, act, w_ahead, sk_lose_loads, f);
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

// Whether M rows of one token each pass the gated convolution at the store of its input product (ST_CONV), on a device of that
// many SMs: where the product streams W, and three strips a unit give no SM more strips than dealing them one by one does
// (2,048 channels: 128 units, 3 strips at the most either way).
static bool conv_pays(int M, int K, int H, int L, int sms) {
  if (M < 1 || M > ST_FUSE_ROWS || K < 64 || K % 64 || H < SK_ROWS || H % SK_ROWS || L < 2 || L > ST_CONV_TAPS || sms < 1)
    return false;
  const int units = H / SK_ROWS, strips = 3 * units;
  return skinny_split(3 * H, K, nullptr) == 1 && stream_pays(3 * H, K, sms) && 3 * ((units + sms - 1) / sms) <= (strips + sms - 1) / sms;
}

SNK_API int snk_conv_step_ok(int M, int K, int H, int L) {
  int sms = 0;
  return snk_device_sms(&sms) == 0 && conv_pays(M, K, H, L, sms);
}

static int stream_map(const void* W, int N, int K, CUtensorMap* map) {
  if ((uintptr_t)W % 16) return SNK_ERR_ALIGN;
  return tensor_map(W, N, K, SK_ROWS, 0, map, ST_RUNS / 2);
}

static void conv_args(StFuse* f, const void* taps, int taps_f32, void* state, const int* seg_start, const int* seg_slot, int L) {
  f->taps = SmallVec{taps, taps_f32};
  f->state = static_cast<bf16*>(state);
  f->seg_start = seg_start;
  f->seg_slot = seg_slot;
  f->L = L;
}

// y [M, H] = the gated short convolution of A . W^T, W = [B | C | x] ([3 H, K]), for M rows that are one token of a request
// each; state [slots, L - 1, H] is brought up to date.  snk_conv_step_ok says which sizes it takes.
SNK_API int snk_conv_step(const void* A, const void* W, const void* taps, int taps_f32, void* state, const int* seg_start,
                          const int* seg_slot, void* out, int M, int K, int H, int L, int w_ahead, cudaStream_t stream) {
  if (M <= 0) return 0;
  if ((uintptr_t)A % 16) return SNK_ERR_ALIGN;
  int sms = 0;
  int rc = snk_device_sms(&sms);
  if (rc) return rc;
  if (!conv_pays(M, K, H, L, sms)) return SNK_ERR_SIZE;
  CUtensorMap map;
  rc = stream_map(W, 3 * H, K, &map);
  if (rc) return rc;
  StFuse f = {};
  conv_args(&f, taps, taps_f32, state, seg_start, seg_slot, L);
  return launch_stream<1, bf16, false, 1, ST_CONV>(map, static_cast<const bf16*>(A), out, M, 3 * H, K, 0, w_ahead, sms, stream, f);
}

// Whether M rows of a norm over K columns are formed by the blocks of the product behind it (ST_NORM): few rows of few bytes
// (``pieces``: the float rows that are added to a residual's row), as every block reads them all, and a product whose K is not
// split.
#define ST_NORM_BYTES (40 * 1024)
#define ST_NORM_STRIPS_PER_SM 10
static bool norm_pays(int M, int N, int K, int pieces, int sms) {
  if (M < 1 || M > ST_FUSE_ROWS || K < 64 || K % 64 || N < 1 || sms < 1 || M * st_norm_pitch(K) * 2 > ST_NORM_SMEM) return false;
  const int per_row = M == 1 ? SK_WARPS : SK_WARPS / 2;
  const int strips = (N + SK_ROWS - 1) / SK_ROWS;
  return K / 4 <= ST_NORM_VECS * 32 * per_row && (long long)M * (1 + pieces) * K * 4 <= ST_NORM_BYTES &&
         skinny_split(N, K, nullptr) == 1 && strips >= sms && strips <= ST_NORM_STRIPS_PER_SM * sms;
}

SNK_API int snk_norm_product_ok(int M, int N, int K, int pieces) {
  int sms = 0;
  return snk_device_sms(&sms) == 0 && norm_pays(M, N, K, pieces, sms);
}

// C = norm(residual + what is added) . W^T in bfloat16: the RMS norm (add_rmsnorm's arguments) of M rows and the product behind
// it.  new_residual [M, K] (other memory than residual; may be null where nothing is added) receives the sum.  swiglu: as
// snk_gemm_skinny.  L > 0: the product is a gated short convolution's input product, and C [M, N / 3] its output, as in
// snk_conv_step.
SNK_API int snk_norm_product(const float* residual, const float* delta, const float* moe_y, const int* pair_pos,
                             const float* topk_w, int k, const void* gamma, int gamma_f32, float eps, float* new_residual,
                             const void* W, void* C, int M, int N, int K, int swiglu, const void* taps, int taps_f32,
                             void* state, const int* seg_start, const int* seg_slot, int L, int w_ahead, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (((uintptr_t)residual % 16) || ((uintptr_t)delta % 16) || ((uintptr_t)moe_y % 16) || ((uintptr_t)new_residual % 16))
    return SNK_ERR_ALIGN;
  int sms = 0;
  int rc = snk_device_sms(&sms);
  if (rc) return rc;
  if ((delta && moe_y) || (moe_y && k < 1) || ((delta || moe_y) && (!new_residual || new_residual == residual)) ||
      !norm_pays(M, N, K, moe_y ? k : delta ? 1 : 0, sms))
    return SNK_ERR_SIZE;
  if (L > 0 ? (swiglu || N % 3 || !conv_pays(M, K, N / 3, L, sms)) : (swiglu && (N % 16 || swiglu == SNK_ACT_RELU2)))
    return SNK_ERR_SIZE;
  CUtensorMap map;
  rc = stream_map(W, N, K, &map);
  if (rc) return rc;
  StFuse f = {};
  f.residual = residual;
  f.delta = delta;
  f.moe_y = moe_y;
  f.pair_pos = pair_pos;
  f.topk_w = topk_w;
  f.k = k;
  f.gamma = SmallVec{gamma, gamma_f32};
  f.eps = eps;
  f.new_residual = delta || moe_y ? new_residual : nullptr;
  if (L > 0) {
    conv_args(&f, taps, taps_f32, state, seg_start, seg_slot, L);
    return launch_stream<1, bf16, false, 1, ST_NORM | ST_CONV>(map, nullptr, C, M, N, K, 0, w_ahead, sms, stream, f);
  }
  if (swiglu) return launch_stream<1, bf16, true, 1, ST_NORM>(map, nullptr, C, M, N, K, swiglu, w_ahead, sms, stream, f);
  return launch_stream<1, bf16, false, 1, ST_NORM>(map, nullptr, C, M, N, K, 0, w_ahead, sms, stream, f);
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
