// tcgen05 (5th-generation tensor cores): operand descriptors, MMA issue, commit, tensor-memory loads and
// fences, for one SM (cta_group::1) and for a pair of SMs (cta_group::2).
#pragma once
#include "tma.cuh"

// Shared-memory matrix descriptor of a tile whose rows are 128 bytes, written by TMA with the 128-byte swizzle, in two words.
// The low one: start address in steps of 16 bytes, bits [0, 14); leading byte offset (not used by swizzled K-major layouts), bits
// [16, 30).  A tile or 16 columns further on is an addition; shared memory ends far below the field's 2^14 steps.  The high one
// is the same for every such tile: stride byte offset (8-row groups lie 1024 bytes apart), bits [32, 46); version 1, bits [46, 48);
// layout type 2 = 128-byte swizzle, bits [61, 64).
#define TC_DESC_HI ((uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29))
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t smem_addr) { return (smem_addr >> 4) | (1u << 16); }

// Instruction descriptor of kind::f16: D float, A and B bfloat16, both K-major, M m (128; 256 for a pair of
// SMs), N n.
__device__ __forceinline__ uint32_t instr_desc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// D += A B, both operands by the low words of their descriptors.  For a loop that a whole warp walks with one lane issuing
// (`elected`): the instruction carries the lane's predicate, so that no branch stands around it, and all that leads up to it is the
// same in every lane; the loop's waits are the warp's (mbar_wait_warp).  An issuing lane of its own, with its branch, descriptors
// formed for each instruction and three reads of the abort word a k-block, took 620 cycles per k-block of 64 whatever the tile: more than
// the 512 that the products of a 256-column tile take.  Measured in turn, us, such a lane / so, on pairs of SMs: 8,192 x 6,144 x 2,048 160 /
// 142, 8,192 x 2,048 x 8,192 207 / 191, 4,096 x 6,144 x 2,048 86.8 / 83.4; on one: 8,192 x 6,144 x 2,048 169 / 159, 1,024 x 2,048 x 8,192 54.1 / 49.2.
__device__ __forceinline__ void umma_bf16_lo(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate,
                                             uint32_t elected) {
  asm volatile(
      "{\n .reg .pred p, q;\n .reg .b64 a, b;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
      " mov.b64 a, {%1, %6};\n mov.b64 b, {%2, %6};\n"
      " @q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}"
      ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(elected), "r"(TC_DESC_HI) : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t bar, uint32_t elected) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
      " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar), "r"(elected) : "memory");
}
// One lane of the (converged) warp: 1 there, 0 elsewhere.
__device__ __forceinline__ uint32_t elect_lane() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(e));
  return e;
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }


// ---------------------------------------------------------------------------------------------
// The store of a 32 x 32 piece of an accumulator that tcgen05.ld left with one ROW per lane (r[0..31]: the
// row's 32 columns).  Stored straight from there, a warp's instruction would touch 32 rows, 16 bytes each.
// So the piece goes through shared memory (rows of 128 bytes, whose 16-byte vectors change places by the row's number:
// stores and loads without bank conflicts) and comes back with 8 lanes side by side along a row: every store instruction then
// writes whole 128-byte (float) or 64-byte (bfloat16) runs of 4 rows.  (With SwiGLU a lane's row shrinks to 32 bytes, which two
// 16-byte stores from the registers write faster.)
//   first_row: row of C of lane 0; rows >= row_end are not stored; col0: first column of the piece (a multiple
//   of 32); N: columns of the product (SwiGLU: C has N / 2).  Pieces that reach past N take the slow path.
//   ADD (float): the piece is added to what C holds, whose values tc_load_old has brought in for the lanes that store them: the
//   first piece's while the tile's products still run, each other one's behind the stores of the piece before.
#define TC_STAGE_FLOATS (32 * 32)

template <bool ADD> struct TcOld { float4 v[ADD ? 8 : 1]; };
template <bool ADD, typename OutT>
__device__ __forceinline__ void tc_load_old(TcOld<ADD>& old, int lane, const OutT* C, int first_row, int row_end, int col0, int N) {
  if constexpr (ADD) {
    const bool in = col0 + 32 <= N && (N % 8) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = first_row + 4 * i + (lane >> 3);
      old.v[i] = in && row < row_end ? *reinterpret_cast<const float4*>(C + (size_t)row * N + col0 + (lane & 7) * 4)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

template <typename OutT, bool SWIGLU, bool ADD = false>
__device__ __forceinline__ void tc_store_piece(const uint32_t (&r)[32], float* stage, int lane, OutT* __restrict__ C,
                                               int first_row, int row_end, int col0, int N,
                                               int act, const TcOld<ADD>& old) {
  if constexpr (SWIGLU) {
    // columns: 8 gates, their 8 ups, 8 gates, their 8 ups -> 16 outputs of this lane's row, two 16-byte stores
    // (measured: faster from the registers than through the staging tile, 106 against 123 us on 2048 x 14336 x 2048)
    const int row = first_row + lane;
    if (row >= row_end) return;
    OutT* dst = C + (size_t)row * (N / 2) + col0 / 2;
#pragma unroll
    for (int blk = 0; blk < 2; ++blk) {
      if (col0 + blk * 16 + 16 <= N) {
        uint32_t p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float g0 = __uint_as_float(r[blk * 16 + 2 * j]), g1 = __uint_as_float(r[blk * 16 + 2 * j + 1]);
          const float u0 = __uint_as_float(r[blk * 16 + 8 + 2 * j]), u1 = __uint_as_float(r[blk * 16 + 9 + 2 * j]);
          const __nv_bfloat162 v = __floats2bfloat162_rn(glu_out(g0, u0, act), glu_out(g1, u1, act));
          p[j] = *reinterpret_cast<const uint32_t*>(&v);
        }
        *reinterpret_cast<uint4*>(dst + blk * 8) = make_uint4(p[0], p[1], p[2], p[3]);
      }
    }
    return;
  } else {
    static_assert(!ADD || sizeof(OutT) == 4, "the stream is float");
    if (col0 + 32 <= N && (N % 8) == 0) {
      uint4* mine = reinterpret_cast<uint4*>(stage + lane * 32);
#pragma unroll
      for (int c = 0; c < 8; ++c) mine[c ^ (lane & 7)] = make_uint4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int rr = 4 * i + (lane >> 3), row = first_row + rr;
        float4 v = *reinterpret_cast<const float4*>(stage + rr * 32 + (((lane ^ rr) & 7) << 2));
        if constexpr (ADD) {
          v.x += old.v[i].x; v.y += old.v[i].y; v.z += old.v[i].z; v.w += old.v[i].w;
        }
        if (row < row_end) store4<OutT>(C + (size_t)row * N + col0 + (lane & 7) * 4, v.x, v.y, v.z, v.w);
      }
      __syncwarp();
      return;
    }
    // a piece at the right edge, or a width the vector stores do not take: this lane's row, element by element
    const int row = first_row + lane;
    if (row >= row_end) return;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (col0 + i < N) {
        OutT& c = C[(size_t)row * N + col0 + i];
        c = from_f<OutT>(__uint_as_float(r[i]) + (ADD ? to_f<OutT>(c) : 0.f));
      }
  }
}

// ---- a pair of SMs (cta_group::2): the leader block issues; operands lie at the same shared-memory
// offsets in both blocks (each block its 128 rows of A and its half of B's rows), the accumulator rows
// 0..127 in the leader's tensor memory and 128..255 in the peer's, at the same columns.
// By the elected lane of a warp, as umma_bf16_lo.
__device__ __forceinline__ void umma2_bf16_lo(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                              uint32_t accumulate, uint32_t elected) {
  asm volatile(
      "{\n .reg .pred p, q;\n .reg .b64 a, b;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
      " mov.b64 a, {%1, %6};\n mov.b64 b, {%2, %6};\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n}"
      ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(elected), "r"(TC_DESC_HI) : "memory");
}
// Arrives once on the barrier at this shared-memory offset in every block of `cta_mask` when the MMAs issued so
// far have completed.
__device__ __forceinline__ void umma2_commit_if(uint32_t bar, uint16_t cta_mask, uint32_t elected) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n"
      " @q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}"
      ::"r"(bar), "h"(cta_mask), "r"(elected) : "memory");
}
// A tile load whose bytes count towards a barrier that may lie in the peer block of the pair (`cluster_bar`: the
// barrier's shared::cluster address, from cluster_addr); not a multicast: the data goes to this block only.
__device__ __forceinline__ void tma2_load_2d(void* smem_dst, const CUtensorMap* map, uint32_t cluster_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(x), "r"(y)
      : "memory");
}
// The shared::cluster address of the variable at this shared-memory offset in block `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void* local, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
  return remote;
}
// One arrival on the barrier at the same offset in block `rank` of the cluster.
__device__ __forceinline__ void mbar_arrive_remote(uint64_t* bar, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(bar)), "r"(rank));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
__device__ __forceinline__ uint32_t ld_cluster_u32(const uint32_t* local, uint32_t rank) {
  uint32_t remote, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster_u32(const void* local, uint32_t rank, uint32_t v) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
