// C[M,N] = A[M,K] . W[N,K]^T on the CUDA cores, with float accumulation in k order.
//
// This is the matrix product of the true 32-bit path (plain FFMA: no TF32, no split
// tricks), and the reference kernel that the tensor-core products are checked against.
// Each output element is one thread's sum over k = 0..K-1 in ascending order, so a row's
// result does not depend on how many other rows the launch holds, nor on which of the two
// kernels below forms it.
//
// Grouped form (routed experts): rows are sorted by group; group e owns rows
// [offsets[e], offsets[e+1]) and multiplies them with W + e*N*K.  `a_rows` gathers A: the
// A row of output row r is a_rows[r] / a_div (a_rows == nullptr: row r itself).
// (the role of snowllm/ops/gemm.py:33-41 and of the expert products in
// snowllm/ops/inference.py:60-76)
#include "common.cuh"

// Four values of a row as they are fetched, to be turned into floats where they are used: what is computed from a load ends
// the time in which the load may be on its way.  (bfloat16, K = 2,044, converted at the fetch / at the store to shared memory: 17 x
// 2,048 225 / 102 us, 512 x 2,048 414 / 140 us; 190 and 194 us with the 64 x 64 tile before.)
template <typename T> struct Vec4;
template <> struct Vec4<float> {
  typedef float Raw;
  static __device__ __forceinline__ void fetch(const float* p, float (&r)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    r[0] = t.x; r[1] = t.y; r[2] = t.z; r[3] = t.w;
  }
  static __device__ __forceinline__ float raw(const float* p) { return *p; }
  static __device__ __forceinline__ void floats(const float (&r)[4], bool vec, float (&v)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = r[i];
  }
};
template <> struct Vec4<bf16> {
  typedef uint32_t Raw;              // vec: two values each in the first two, otherwise one in the low half of each
  static __device__ __forceinline__ void fetch(const bf16* p, uint32_t (&r)[4]) {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    r[0] = t.x; r[1] = t.y; r[2] = r[3] = 0u;
  }
  static __device__ __forceinline__ uint32_t raw(const bf16* p) { return *reinterpret_cast<const unsigned short*>(p); }
  static __device__ __forceinline__ void floats(const uint32_t (&r)[4], bool vec, float (&v)[4]) {
    v[0] = __uint_as_float(r[0] << 16);
    v[1] = __uint_as_float(vec ? r[0] & 0xffff0000u : r[1] << 16);
    v[2] = __uint_as_float(vec ? r[1] << 16 : r[2] << 16);
    v[3] = __uint_as_float(vec ? r[1] & 0xffff0000u : r[3] << 16);
  }
};

// Four values from k on of a row (not ok: zeros), zeros past K; vec (K is a multiple of 4): by one vector load.
template <typename T>
__device__ __forceinline__ void load4(const T* row, int k, int K, bool ok, bool vec, typename Vec4<T>::Raw (&r)[4]) {
  if (!ok) { r[0] = r[1] = r[2] = r[3] = 0; return; }
  if (vec && k + 3 < K) { Vec4<T>::fetch(row + k, r); return; }
#pragma unroll
  for (int i = 0; i < 4; ++i) r[i] = (k + i < K) ? Vec4<T>::raw(row + k + i) : typename Vec4<T>::Raw(0);
}

// Two independent fused multiply-adds by one instruction (fma.rn.f32x2), each rounded as fmaf rounds: acc += (a, a) * w.
__device__ __forceinline__ void fma2(unsigned long long& acc, float a, unsigned long long w) {
  unsigned long long aa;
  asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(aa), "l"(w));
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// ---------------------------------------------------------------------------------------
// Many rows: tiles of BM x BN, a thread owns TM x TN outputs (TN columns as runs of four, BN / (TN / 4) apart, so that
// a warp's shared-memory reads are consecutive).  Bound by the FMA pipe; the multiply-adds go two to an instruction,
// which leaves half of the issue slots to the loads from shared memory.  The next BK columns of both operands are on
// their way to registers while the current ones are multiplied; shared memory is double buffered, one barrier a step.
// Measured (TFLOP/s; 74 is the pipe's rate, 34 the 64 x 64 single-buffered tile before): 2,048 x 16,384 x 2,048 53, 509 x 16,384
// x 2,048 49, 509 x 2,048 x 2,048 32 (128 tiles: one a SM).  Tried and slower: A stored twice for the paired operand
// (40), single multiply-adds (47), 8 columns a step (49), 16 x 8 outputs a thread.
#define BK 16

template <typename T, typename OutT, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__(BM * BN / (TM * TN), BM * BN / (TM * TN) >= 256 ? 2 : (TM * TN >= 64 ? 3 : 4))
gemm_tile_kernel(const T* __restrict__ A, const T* __restrict__ W, OutT* __restrict__ C, int M,
                 int N, int K, const int* __restrict__ a_rows, int a_div,
                 const int* __restrict__ offsets, int vec) {
  constexpr int THREADS = BM * BN / (TM * TN), TX = BN / TN, RUNS = TN / 4;
  constexpr int A4 = BM * (BK / 4) / THREADS, W4 = BN * (BK / 4) / THREADS;       // vectors a thread brings in a step
  static_assert(A4 * THREADS == BM * (BK / 4) && W4 * THREADS == BN * (BK / 4) && TN % 4 == 0 && TM % 4 == 0, "tile");
  pdl_begin();
  __shared__ __align__(16) float As[2][BK][BM + 4];
  __shared__ __align__(16) float Ws[2][BK][BN + 4];
  int row_begin = 0, row_end = M;
  const T* Wg = W;
  if (offsets) {
    row_begin = offsets[blockIdx.z];
    row_end = offsets[blockIdx.z + 1];
    Wg = W + (size_t)blockIdx.z * N * K;
  }
  const int m0 = row_begin + blockIdx.y * BM;
  if (m0 >= row_end) return;
  const int n0 = blockIdx.x * BN;
  const int tid = threadIdx.x;
  const int lr = tid / (BK / 4), lk = (tid % (BK / 4)) * 4;       // tile-load coordinates
  const int ty = tid / TX, tx = tid % TX;

  int a_row[A4];                                     // -1: past the rows
#pragma unroll
  for (int i = 0; i < A4; ++i) {
    const int r = m0 + lr + i * (THREADS / (BK / 4));
    a_row[i] = r < row_end ? (a_rows ? a_rows[r] / a_div : r) : -1;
  }
  const T* w_ptr = Wg + (size_t)(n0 + lr) * K;
  typename Vec4<T>::Raw av[A4][4], wv[W4][4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < A4; ++i) load4<T>(A + (size_t)a_row[i] * K, k0 + lk, K, a_row[i] >= 0, vec, av[i]);
#pragma unroll
    for (int i = 0; i < W4; ++i)
      load4<T>(w_ptr + (size_t)(i * (THREADS / (BK / 4))) * K, k0 + lk, K, n0 + lr + i * (THREADS / (BK / 4)) < N, vec, wv[i]);
  };
  auto stage = [&](int b) {
    float v[4];
#pragma unroll
    for (int i = 0; i < A4; ++i) {
      Vec4<T>::floats(av[i], vec, v);
#pragma unroll
      for (int j = 0; j < 4; ++j) As[b][lk + j][lr + i * (THREADS / (BK / 4))] = v[j];
    }
#pragma unroll
    for (int i = 0; i < W4; ++i) {
      Vec4<T>::floats(wv[i], vec, v);
#pragma unroll
      for (int j = 0; j < 4; ++j) Ws[b][lk + j][lr + i * (THREADS / (BK / 4))] = v[j];
    }
  };

  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

  fetch(0);
  stage(0);
  __syncthreads();
  const int steps = (K + BK - 1) / BK;
  for (int s = 0; s < steps; ++s) {
    const int b = s & 1;
    if (s + 1 < steps) fetch((s + 1) * BK);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[TM];
      unsigned long long w[TN / 2];
#pragma unroll
      for (int i = 0; i < TM / 4; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(&As[b][k][ty * TM + 4 * i]);
        a[4 * i] = v.x; a[4 * i + 1] = v.y; a[4 * i + 2] = v.z; a[4 * i + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < RUNS; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[b][k][j * (BN / RUNS) + tx * 4]);
        w[2 * j] = v.x; w[2 * j + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], a[i], w[j]);
    }
    if (s + 1 < steps) {
      stage(b ^ 1);                                   // read last before the barrier of the step before
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = m0 + ty * TM + i;
    if (r >= row_end) continue;
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      const int c = n0 + (j / 2) * (BN / RUNS) + tx * 4 + (j & 1) * 2;
      float lo, hi;
      unpack2(acc[i][j], lo, hi);
      if (c < N) C[(size_t)r * N + c] = from_f<OutT>(lo);
      if (c + 1 < N) C[(size_t)r * N + c + 1] = from_f<OutT>(hi);
    }
  }
}

// ---------------------------------------------------------------------------------------
// Few rows (decode), float: bound by the read of W.  A block owns FR_COLS columns (rows of W) and FR_STAGES chunks of
// FR_K of their values, which four warps of its own bring in by cp.async (a row of a chunk is one instruction of a warp),
// W's first chunks from before the wait for the kernel before where W is a weight (w_ahead).  The other warps multiply: a lane owns one column and R
// rows, half-warps rows of their own.  The sum over k stays one thread's, in order: with K chained multiply-adds of four
// cycles a block cannot end sooner than 4 K cycles (4.3 us at K = 2,048), so nothing but them and the reads of their
// operands is left to those warps, and the narrow blocks of 16 columns share the columns out over as many SMs as N gives.
// Measured, 4 rows (in a replayed chain; the 64 x 64 tile before): 2,048 x 2,048 9.4 us (146), 14,336 x 2,048 31 us (190),
// 2,048 x 7,168 28 us (523), 65,536 x 2,048 108 us = 5.0 TB/s; with the loads in the warps that multiply 19, 41, 66, 130 us.
#define FR_COLS 16
#define FR_K 128
#define FR_STAGES 4
#define FR_PITCH (FR_K + 4)        // an odd number of 16-byte units: eight lanes on eight rows hit different banks
#define FR_LOADERS 4               // warps that load

__device__ __forceinline__ void cp_async16(float* smem, const float* gmem, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               :: "r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(ok ? 16 : 0));
}

template <int R, int WARPS>
__global__ void __launch_bounds__((WARPS + FR_LOADERS) * 32)
gemm_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                const int* __restrict__ a_rows, int a_div, const int* __restrict__ offsets, int groups, int w_ahead) {
  constexpr int ROWS = 2 * R * WARPS;
  constexpr int W_EACH = FR_COLS / FR_LOADERS, A_EACH = (ROWS + FR_LOADERS - 1) / FR_LOADERS;
  extern __shared__ __align__(16) float sm[];          // per stage: FR_COLS rows of W, then ROWS rows of A
  constexpr int STAGE = (FR_COLS + ROWS) * FR_PITCH;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n0 = blockIdx.x * FR_COLS;
  const int loader = warp - WARPS;                     // 0..3: a warp that loads
  const int chunks = (K + FR_K - 1) / FR_K;
  int row_begin = 0, row_end = M;
  const float* w_src[W_EACH];                          // a loader's rows of W (a row past N loads zeros)
  auto point_w = [&](const float* Wg) {
#pragma unroll
    for (int i = 0; i < W_EACH; ++i)
      w_src[i] = Wg + (size_t)min(n0 + loader + i * FR_LOADERS, N - 1) * K + lane * 4;
  };
  auto load_w = [&](int c) {
    float* to = sm + (c % FR_STAGES) * STAGE + loader * FR_PITCH + lane * 4;
    const bool in = c * FR_K + lane * 4 < K;           // K is a multiple of 4
#pragma unroll
    for (int i = 0; i < W_EACH; ++i)
      cp_async16(to + i * (FR_LOADERS * FR_PITCH), w_src[i] + (in ? c * FR_K : -lane * 4),
                 in && n0 + loader + i * FR_LOADERS < N);
  };
  bool w_there = offsets == nullptr && w_ahead;        // W is a weight: its first chunks need not wait
  if (w_there && loader >= 0) {
    point_w(W);
#pragma unroll
    for (int c = 0; c < FR_STAGES - 1; ++c)
      if (c < chunks) load_w(c);
  }
  pdl_begin();
  if (offsets) {
    int e = blockIdx.y;
    if (groups > (int)gridDim.y) {
      // fewer rows than groups: block y takes the y-th group that owns any (every warp looks it up for itself), and no block
      // is started for a group without rows (see launch_few)
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
    if (row_begin >= row_end) return;
    point_w(W + (size_t)e * N * K);
  } else if (!w_there) {
    point_w(W);
  }
  const int col = lane & 15;
  const int first = (warp * 2 + (lane >> 4)) * R;      // a multiplying lane's rows of a pass
  for (int m0 = row_begin; m0 < row_end; m0 += ROWS) {
    const float* a_src[A_EACH];
    bool a_ok[A_EACH];
#pragma unroll
    for (int i = 0; i < A_EACH; ++i) {
      const int r = loader + i * FR_LOADERS;
      a_ok[i] = loader >= 0 && r < ROWS && m0 + r < row_end;
      a_src[i] = A + (a_ok[i] ? (size_t)(a_rows ? a_rows[m0 + r] / a_div : m0 + r) * K + lane * 4 : 0);
    }
    auto load_a = [&](int c) {
      float* to = sm + (c % FR_STAGES) * STAGE + (FR_COLS + loader) * FR_PITCH + lane * 4;
      const bool in = c * FR_K + lane * 4 < K;
#pragma unroll
      for (int i = 0; i < A_EACH; ++i)
        if (loader + i * FR_LOADERS < ROWS)
          cp_async16(to + i * (FR_LOADERS * FR_PITCH), in && a_ok[i] ? a_src[i] + c * FR_K : A, in && a_ok[i]);
    };
    if (loader >= 0) {
#pragma unroll
      for (int c = 0; c < FR_STAGES - 1; ++c) {
        if (c < chunks) {
          if (!w_there) load_w(c);
          load_a(c);
        }
        asm volatile("cp.async.commit_group;");
      }
    }
    w_there = false;
    float acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0.f;
    for (int c = 0; c < chunks; ++c) {
      if (loader >= 0) asm volatile("cp.async.wait_group %0;" :: "n"(FR_STAGES - 2));
      __syncthreads();                                 // chunk c is there, and everyone is done with chunk c - 1
      if (loader >= 0) {
        if (c + FR_STAGES - 1 < chunks) {
          load_w(c + FR_STAGES - 1);
          load_a(c + FR_STAGES - 1);
        }
        asm volatile("cp.async.commit_group;");
        continue;
      }
      const float* ws = sm + (c % FR_STAGES) * STAGE + col * FR_PITCH;
      const float* as = sm + (c % FR_STAGES) * STAGE + (FR_COLS + first) * FR_PITCH;
#pragma unroll
      for (int k = 0; k < FR_K; k += 4) {              // past K both operands are zeros
        const float4 w = *reinterpret_cast<const float4*>(ws + k);
        float4 a[R];
#pragma unroll
        for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * FR_PITCH + k);
#pragma unroll
        for (int i = 0; i < R; ++i) acc[i] = fmaf(a[i].x, w.x, acc[i]);
#pragma unroll
        for (int i = 0; i < R; ++i) acc[i] = fmaf(a[i].y, w.y, acc[i]);
#pragma unroll
        for (int i = 0; i < R; ++i) acc[i] = fmaf(a[i].z, w.z, acc[i]);
#pragma unroll
        for (int i = 0; i < R; ++i) acc[i] = fmaf(a[i].w, w.w, acc[i]);
      }
    }
    if (loader < 0) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int r = m0 + first + i;
        if (r < row_end && n0 + col < N) C[(size_t)r * N + n0 + col] = acc[i];
      }
    } else {
      asm volatile("cp.async.wait_group 0;");
    }
    __syncthreads();                                   // the next pass writes the stages again
  }
}

struct SimtArgs {
  const void *A, *W;
  void* C;
  int M, N, K;
  const int* a_rows;
  int a_div;
  const int* offsets;
  int groups, rows, vec;           // rows: the most that one group (or the product) can own
  int w_ahead;
  cudaStream_t stream;
};

template <typename T, typename OutT, int BM, int BN, int TM, int TN>
static int launch_tile(const SimtArgs& p) {
  dim3 grid((p.N + BN - 1) / BN, (p.rows + BM - 1) / BM, p.offsets ? p.groups : 1);
  if (grid.y > 65535u || grid.z > 65535u) return SNK_ERR_SIZE;
  snk_launch(gemm_tile_kernel<T, OutT, BM, BN, TM, TN>, grid, dim3(BM * BN / (TM * TN)), 0, p.stream,
             static_cast<const T*>(p.A), static_cast<const T*>(p.W), static_cast<OutT*>(p.C), p.M, p.N, p.K, p.a_rows,
             p.a_div, p.offsets, p.vec);
  SNK_LAUNCH_CHECK();
  return 0;
}

template <int R, int WARPS>
static int launch_few(const SimtArgs& p) {
  constexpr int smem = FR_STAGES * (FR_COLS + 2 * R * WARPS) * FR_PITCH * (int)sizeof(float);
  static_assert(smem <= 227 * 1024, "stages");
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel<R, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
  }
  // Fewer rows than groups: a block per row and strip, which looks its group up, unless the blocks of all groups are on the SMs at
  // once (five to each) and the idle ones cost nothing.  Measured, us, a block per group / per row: 32 groups of 2,048 x 1,792, 4 rows 19.7 / 14.3, 8
  // 26.7 / 24.2, 16 42.0 / 39.4, 28 59.8 / 58.3; of 3,584 x 2,048, 16 rows 75.4 / 73.1; of 384 x 512 (768 blocks, just above the line), 4 rows 4.4 /
  // 3.5, 16 5.4 / 5.4; 128 groups of 768 x 512, 4 rows 9.3 / 4.2, 64 24.1 / 21.8; 256 of 256 x 512, 8 rows 7.0 / 4.8, 128 18.6 / 17.7, but 248, with
  // nearly a row to a group, 25.9 / 26.5.
  const long long strips = (p.N + FR_COLS - 1) / FR_COLS;
  int sms = 0, per_group = p.offsets ? p.groups : 1;
  if (p.offsets && p.M <= p.groups - (p.groups + 15) / 16) {
    const int rc = snk_device_sms(&sms);
    if (rc) return rc;
    if (strips * p.groups > 5ll * sms) per_group = p.M;
  }
  snk_launch(gemm_few_kernel<R, WARPS>, dim3((unsigned)strips, per_group), dim3((WARPS + FR_LOADERS) * 32), smem,
             p.stream, static_cast<const float*>(p.A), static_cast<const float*>(p.W), static_cast<float*>(p.C), p.M, p.N,
             p.K, p.a_rows, p.a_div, p.offsets, p.groups, p.w_ahead);
  SNK_LAUNCH_CHECK();
  return 0;
}

// Up to here W's read is the bound.  Measured, in replayed chains over rotating weights, this kernel / the tiles, us: 2,048 x 2,048 1 row
// 8.6 / 95, 4 rows 10.0 / 95, 8 rows 12.6 / 95, 16 rows 21.5 / 95; 6,144 x 2,048 14 / 87, 19 / 88, 22 / 89, 45 / 88; 16,384 x 2,048
// 27 / 94, 35 / 95, 50 / 94, 91 / 95; 65,536 x 2,048 96 / 272, 111 / 274, 165 / 275, 316 / 279 (there the tiles are ahead from 10 rows on);
// 20 rows 58 / 89 at 6,144 x 2,048 and 118 / 97 at 16,384 x 2,048.
// Grouped, up to 4 rows a group on average (32 groups, 3,584 x 2,048, each token in 4 of them at random): 4 tokens 80 / 240 us, 8 128 / 313,
// 16 174 / 421, 32 272 / 461; 128 groups of 768 x 512: 16 tokens 25 / 58, 100 74 / 102.  A group far above the average is walked in
// passes that read W again: all 32 tokens in the same 4 of 32 groups 195 / 174 us, 100 tokens in the same 4 of 128 groups 69 / 36,
// all 400 rows in one of 128 groups 250 / 54 (such a group would need tiles of its own: a second launch whose blocks find no such
// group in every ordinary step).
#define FR_MAX_ROWS 16

// The tile with the least work on the busiest SM: rounds of tiles over the SMs times the tile's area, over the share of
// the FMA rate that its shared-memory reads leave.  The shares are those at 4,096 x 16,384 x 2,048 (128 x 128 5.16 ms, 64 x 128 5.28,
// 64 x 64 6.64, 32 x 64 8.56).  Against all four tiles at 135 sizes (17 to 8,192 rows; N 64 to 16,384; K 640 to 8,192) the
// choice was within 2 % of the fastest at 127, 3 to 6 % off at six, 9 and 12 % off at one each.
// rows: the most that one group can own, which the grid's 65,535 blocks along y have to hold (a lower tile that would not is
// left out); mean: rows of a group (of the product); sms: the device's.  0 to 3: 128 x 128, 64 x 128, 64 x 64, 32 x 64.
static int pick_tile(int groups, int rows, long long mean, int N, int sms) {
  static const int bm[4] = {128, 64, 64, 32}, bn[4] = {128, 128, 64, 64};
  static const double rate[4] = {1.0, 0.95, 0.8, 0.6};
  int best = 0;
  double least = 0.0;
  for (int t = 0; t < 4; ++t) {
    if (t > 0 && (rows + bm[t] - 1ll) / bm[t] > 65535) continue;
    const long long tiles = (long long)groups * ((mean + bm[t] - 1) / bm[t]) * ((N + bn[t] - 1) / bn[t]);
    const double cost = (double)((tiles + sms - 1) / sms) * bm[t] * bn[t] / rate[t];
    if (t == 0 || cost < least) {
      best = t;
      least = cost;
    }
  }
  return best;
}

// For tests: the tile that a product of M rows takes on a device of that many SMs (groups 0: plain; otherwise one group owns
// `rows` rows at most).
SNK_API int snk_gemm_simt_tile(int M, int N, int groups, int rows, int sms) {
  return groups ? pick_tile(groups, rows, (M + groups - 1) / groups, N, sms) : pick_tile(1, M, M, N, sms);
}

template <typename T, typename OutT>
static int launch_tiles(const SimtArgs& p) {
  int sms = 0;
  const int rc = snk_device_sms(&sms);
  if (rc) return rc;
  const int G = p.offsets ? p.groups : 1;
  switch (pick_tile(G, p.rows, p.offsets ? (p.M + G - 1) / G : p.M, p.N, sms)) {
    case 0: return launch_tile<T, OutT, 128, 128, 8, 8>(p);
    case 1: return launch_tile<T, OutT, 64, 128, 8, 8>(p);
    case 2: return launch_tile<T, OutT, 64, 64, 4, 8>(p);
    default: return launch_tile<T, OutT, 32, 64, 4, 4>(p);
  }
}

// out_f32: C is float whatever the compute dtype.  groups <= 1 and offsets == nullptr: plain
// product.  max_rows_per_group bounds the rows any one group can own (for the grid).  w_ahead (plain products): W was
// there before the kernel in front of this launch began, and may be read ahead of the wait for it.
SNK_API int snk_gemm_simt(const void* A, const void* W, void* C, int M, int N, int K,
                          const int* a_rows, int a_div, const int* offsets, int groups,
                          int max_rows_per_group, int out_f32, int dtype, int w_ahead, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return SNK_ERR_SIZE;
  const int rows = offsets ? max_rows_per_group : M;
  if (rows <= 0) return 0;
  const size_t esz = dtype == SNK_F32 ? 4 : 2;
  const int vec = (K % 4 == 0) && ((uintptr_t)A % 16 == 0) && ((uintptr_t)W % 16 == 0) &&
                  (((size_t)K * esz) % 8 == 0);
  const SimtArgs p{A, W, C, M, N, K, a_rows, a_div <= 0 ? 1 : a_div, offsets, groups, rows, vec, w_ahead, stream};
  if (dtype == SNK_F32 && vec && (offsets ? (long long)M <= 4ll * groups : M <= FR_MAX_ROWS) && (!offsets || groups <= 65535)) {
    // Rows of a pass: those of the product, or about twice a group's mean (fuller groups take more passes).  32 groups of 3,584 x 2,048,
    // passes of 2 / 4 / 8 / 16 rows: 1 row a group on average 128 / 128 / 186 / 364 us, 2 rows 194 / 174 / 252 / 498, 4 rows 325 / 244 /
    // 272 / 539; plain 2,048 x 2,048 of 4 rows 15.6 / 10.0 / 12.6 / 21.5, of 8 rows 28.8 / 18.2 / 12.6 / 21.8.
    const int pass = offsets ? 2 * ((M + groups - 1) / groups) : M;
    if (pass <= 2) return launch_few<1, 1>(p);
    if (pass <= 4) return launch_few<2, 1>(p);
    if (pass <= 8) return launch_few<2, 2>(p);
    return launch_few<4, 2>(p);
  }
  SNK_DISPATCH(dtype, {
    if (out_f32 || dtype == SNK_F32) return launch_tiles<T, float>(p);
    return launch_tiles<T, T>(p);
  });
  return 0;
}
