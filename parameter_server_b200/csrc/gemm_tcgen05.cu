// Dense layer GEMM on the 5th-generation tensor cores: D[M,N] = act(A[M,K] · B[N,K]ᵀ), fp32 in
// memory, TF32 multiply, fp32 accumulate in tensor memory (TMEM).
//
// Small and medium problems: one CTA (128 threads) per 128x128 output tile:
//   warp 0, one lane   TMA producer: cp.async.bulk.tensor 2-D tiles of A and B (128 rows x 32 floats =
//                      one 128-byte swizzle row each, two spans per stage) into a 3-stage shared-memory
//                      ring, completion on the stage's "full" mbarrier
//   warp 1, one lane   MMA issuer: tcgen05.mma.cta_group::1.kind::tf32, eight K=8 steps per stage (with
//                      four, the barriers' round trips were a third of the time), the accumulator lives in 128 TMEM columns; tcgen05.commit releases the stage
//                      ("empty" mbarrier) and finally signals "accumulator complete"
//   all 4 warps        epilogue: tcgen05.ld 32 lanes x 32 columns per warp and step, activation, store
// Both operands are K-major (row-major with K contiguous), which is how the layers keep their data:
// activations [batch, features] and weights [out, in]; the products of the backward pass read transposes that
// an epilogue, the activation's slope or the tiled transpose kernel wrote.  No load is a multicast.
//
// This is the framework's replacement of the Eigen GEMMs of the reference's fully connected
// layer (src/neural_network/fully_connected_layer.h:27-65); the activation functions are those
// of src/neural_network/activation_function.h:39-99.
//
// Every mbarrier wait is bounded.  If one runs out, the CTA records it in the status word, stops
// issuing work, waits a bounded time for copies in flight, frees its TMEM and returns.
#include <cuda.h>

#include "psb_common.cuh"

namespace psb {

constexpr int kBM = 128, kBN = 128, kBK = 32;       // tile; kBK floats = 128 bytes = swizzle span
constexpr int kStages = 3, kSpans = 2;
constexpr int kUmmaK = 8;                            // K per tcgen05.mma for tf32
constexpr uint32_t kTmemCols = 128;
constexpr uint32_t kWaitLimit = 4u * 1000u * 1000u;   // polls of try_wait before giving up

enum Activation : int { kActIdentity = 0, kActRelu = 1, kActScaledTanh = 2, kActSigmoid = 3 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// bounded wait for the phase with the given parity; false when the limit is hit
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < kWaitLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}

// K-major operand tile in shared memory, 128-byte swizzle: rows of 128 bytes, groups of 8 rows
// (1024 bytes) are the swizzle atoms.  start address >> 4 in bits 0-13, stride byte offset
// (1024 >> 4) in bits 32-45, descriptor version 1 in bits 46-47, layout type 2 (128B swizzle)
// in bits 61-63; the leading byte offset is not used for swizzled K-major tiles.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// instruction descriptor for kind::tf32: D fp32 (1 at bits 4-5), A and B tf32 (2 at bits 7-9 and
// 10-12), both K-major (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28
__host__ __device__ constexpr uint32_t make_idesc(int m, int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ float apply_act(float x, int act) {
  switch (act) {
    case kActRelu: return fmaxf(x, 0.f);
    case kActScaledTanh: return 1.7159f * tanhf(0.6666667f * x);
    case kActSigmoid: return 1.f / (1.f + __expf(-x));
    default: return x;
  }
}

// 32 columns of one row (lane = row, registers = columns) through the activation to out and, when out_t is given,
// to its transpose [N, M]: for a fixed column the lanes of a warp hold consecutive rows, so those stores are
// whole 128-byte lines and cost no second pass over the matrix.
__device__ __forceinline__ void store_chunk(const uint32_t (&r)[32], float* __restrict__ out, float* __restrict__ out_t, int row, int col,
                                            int M, int N, int ldo, int act) {
  if (row >= M || col >= N) return;
  float* dst = out + (size_t)row * ldo + col;
  float* dst_t = out_t != nullptr ? out_t + (size_t)col * M + row : nullptr;
  const int ncol = N - col;
  if (ncol >= 32 && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      float4 v;
      v.x = apply_act(__uint_as_float(r[j]), act);
      v.y = apply_act(__uint_as_float(r[j + 1]), act);
      v.z = apply_act(__uint_as_float(r[j + 2]), act);
      v.w = apply_act(__uint_as_float(r[j + 3]), act);
      *reinterpret_cast<float4*>(dst + j) = v;
      if (dst_t != nullptr) {
        dst_t[(size_t)j * M] = v.x;
        dst_t[(size_t)(j + 1) * M] = v.y;
        dst_t[(size_t)(j + 2) * M] = v.z;
        dst_t[(size_t)(j + 3) * M] = v.w;
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < ncol) {
        const float v = apply_act(__uint_as_float(r[j]), act);
        dst[j] = v;
        if (dst_t != nullptr) dst_t[(size_t)j * M] = v;
      }
  }
}

struct __align__(1024) GemmSmem {
  float a[kStages][kSpans][kBM * kBK];
  float b[kStages][kSpans][kBN * kBK];
  uint64_t full[kStages], empty[kStages], acc_full;
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
};

// kRows: rows of A that exist and are loaded (the tile's other rows are whatever shared memory holds: rows do not
// mix, and theirs are not stored); kCols: columns of the tile.  The weight gradient of a layer with one output is
// [1, batch] · [batch, in]: a few CTAs walk all of K one block after the other.  With 8 rows and 32 columns a block
// is an eighth of the loads and there are four times the CTAs; the sums and their order stay the same.
// B200, L2 flushed, before and after (one 32-deep block per barrier, square tiles): 1x1024x8192 106 -> 64 us,
// 1024x1024x8192 107 -> 80, 4096x1024x8192 211 -> 154.
constexpr int kThinRows = 8, kThinCols = 32;
template <int kRows, int kCols>
__global__ void __launch_bounds__(128, 1)
gemm_tf32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         float* __restrict__ out, float* __restrict__ out_t, int M, int N, int K, int ldo, int act, uint32_t* status) {
  extern __shared__ uint8_t smem_raw[];
  GemmSmem& s = *reinterpret_cast<GemmSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kCols;
  const int nkb = (K + kSpans * kBK - 1) / (kSpans * kBK);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) { mbar_init(&s.full[i], 1); mbar_init(&s.empty[i], 1); }
    mbar_init(&s.acc_full, 1);
    s.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {   // one warp allocates the accumulator columns
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s.tmem_base;

  if (warp == 0 && lane == 0) {
    // ---------------- TMA producer
    for (int kb = 0; kb < nkb; ++kb) {
      const int st = kb % kStages;
      if (kb >= kStages && !mbar_wait(&s.empty[st], ((kb / kStages) - 1) & 1)) { s.abort_flag = 1; break; }
      mbar_expect_tx(&s.full[st], (uint32_t)(kRows + kCols) * kSpans * kBK * 4);
#pragma unroll
      for (int h = 0; h < kSpans; ++h) {       // a span past the end of K is filled with zeros
        tma_load_2d(s.a[st][h], &map_a, &s.full[st], (kb * kSpans + h) * kBK, m0);
        tma_load_2d(s.b[st][h], &map_b, &s.full[st], (kb * kSpans + h) * kBK, n0);
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer
    constexpr uint32_t idesc = make_idesc(kBM, kCols);
    for (int kb = 0; kb < nkb; ++kb) {
      const int st = kb % kStages;
      if (!mbar_wait(&s.full[st], (kb / kStages) & 1)) { s.abort_flag = 1; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int h = 0; h < kSpans; ++h) {
        const uint64_t da = make_smem_desc(smem_u32(s.a[st][h]));
        const uint64_t db = make_smem_desc(smem_u32(s.b[st][h]));
#pragma unroll
        for (int k = 0; k < kBK / kUmmaK; ++k) {
          const uint32_t accumulate = (kb > 0 || h > 0 || k > 0) ? 1u : 0u;
          const uint64_t adv = (uint64_t)((k * kUmmaK * 4) >> 4);   // 32 bytes per K step inside the swizzle row
          asm volatile(
              "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
              ::"r"(tmem), "l"(da + adv), "l"(db + adv), "r"(idesc), "r"(accumulate) : "memory");
        }
      }
      // release the stage once the MMAs that read it have completed
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&s.empty[st])) : "memory");
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&s.acc_full)) : "memory");
  }
  __syncwarp();

  // ---------------- epilogue (all four warps; warp w owns TMEM lanes 32w .. 32w+31)
  int ok = 1;
  if (lane == 0) {
    ok = mbar_wait(&s.acc_full, 0) ? 1 : 0;
    if (!ok) s.abort_flag = 1;
    if (s.abort_flag) ok = 0;
  }
  ok = __shfl_sync(0xffffffffu, ok, 0);   // warp-uniform: the TMEM loads below are warp-collective
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    const int row = m0 + warp * 32 + lane;
#pragma unroll 1
    for (int c0 = 0; c0 < kCols; c0 += 32) {
      uint32_t r[32];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
          "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
          "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
            "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
            "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
          : "r"(taddr) : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      store_chunk(r, out, out_t, row, n0 + c0, M, N, ldo, act);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s.abort_flag) {
    if (threadIdx.x == 0) set_status(status, kWaitTimeout, blockIdx.x, 100 + blockIdx.y);
    // give copies that may still be in flight a bounded time to land before the shared memory goes away
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ------------------------------------------------------------------ CTA pairs
// Large problems: persistent pairs of SMs, each pair on one 256x256 tile at a time (cta_group::2): a CTA holds 128
// rows of A and 128 of the 256 rows of B, and the tensor cores of both read B from both shared memories, so an SM
// loads 32 KB per 32-deep K block instead of the 48 KB that a 128x256 tile of its own takes, and six stages fit.
// The accumulator is double-buffered in TMEM (2 x 256 columns): the epilogue of a tile runs under the next tile's
// main loop.  What bounds it is how fast one thread gets K blocks through its barriers (a read of the abort flag per K
// block cost a seventh of the rate at K = 8192) and, for short K, writing the result.  TF32 rates on B200, L2 flushed
// between calls, against 128x256 tiles on single persistent CTAs: 4096x1024x8192 524 -> 645 TFLOP/s, 8192x4096x1024
// 513 -> 550, 3000x3000x2044 370 -> 472.
//   both CTAs   warp 0: TMA loads of the CTA's own halves, completion counted on the LEADER's "full" barrier
//   leader      warp 1: tcgen05.mma for the pair; its commits release the stage ("empty") and publish the
//               accumulator ("tfull") in both CTAs
//   both CTAs   warps 2-5: epilogue of the CTA's 128 rows; they hand the accumulator back on the leader's "tempty"
// Every CTA loads its own rows: no multicast load.
constexpr int kDTile = 256, kDHalf = 128, kDStages = 6, kPThreads = 192;
constexpr uint32_t kDHalfBytes = kDHalf * kBK * 4;

struct __align__(1024) GemmSmemD {
  float a[kDStages][kDHalf * kBK];
  float b[kDStages][kDHalf * kBK];
  uint64_t full[kDStages], empty[kDStages], tfull[2], tempty[2];
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
};

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank)); return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// bar: shared::cluster address of a barrier in either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// arrive on the barrier at this offset in both CTAs once the MMAs issued so far have completed
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPThreads, 1)
gemm_tf32_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                      float* __restrict__ out, float* __restrict__ out_t, int M, int N, int K, int ldo, int act, uint32_t* status) {
  extern __shared__ uint8_t smem_raw[];
  GemmSmemD& s = *reinterpret_cast<GemmSmemD*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const int nbm = (M + kDTile - 1) / kDTile, nbn = (N + kDTile - 1) / kDTile;
  const int ntiles = nbm * nbn, pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int nkb = (K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kDStages; ++i) { mbar_init(&s.full[i], 1); mbar_init(&s.empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s.tfull[i], 1); mbar_init(&s.tempty[i], 8); }
    s.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();       // the peer's barriers are ready before anything is signalled there
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s.tmem_base;

  if (warp == 0 && lane == 0) {
    // ---------------- TMA producer, tiles m-fastest
    uint32_t g = 0;
    for (int t = pair; t < ntiles && !s.abort_flag; t += npairs) {
      const int m0 = (t % nbm) * kDTile + rank * kDHalf, n0 = (t / nbm) * kDTile + rank * kDHalf;
      for (int kb = 0; kb < nkb; ++kb, ++g) {
        const int st = g % kDStages;
        if (g >= (uint32_t)kDStages && !mbar_wait(&s.empty[st], ((g / kDStages) - 1) & 1)) { s.abort_flag = 1; break; }
        if (rank == 0) mbar_expect_tx(&s.full[st], 4 * kDHalfBytes);
        const uint32_t bar = mapa_u32(smem_u32(&s.full[st]), 0);
        tma_load_2d_pair(s.a[st], &map_a, bar, kb * kBK, m0);
        tma_load_2d_pair(s.b[st], &map_b, bar, kb * kBK, n0);
      }
    }
    // the last releases must have landed here before this CTA's shared memory may go away
    for (uint32_t u = g > (uint32_t)kDStages ? g - kDStages : 0; u < g && !s.abort_flag; ++u)
      if (!mbar_wait(&s.empty[u % kDStages], (u / kDStages) & 1)) s.abort_flag = 1;
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---------------- MMA issuer of the pair
    constexpr uint32_t idesc = make_idesc(kDTile, kDTile);
    uint32_t g = 0, it = 0;
    for (int t = pair; t < ntiles && !s.abort_flag; t += npairs, ++it) {
      const uint32_t acc = it & 1u;
      if (it >= 2 && !mbar_wait(&s.tempty[acc], ((it >> 1) - 1) & 1)) { s.abort_flag = 1; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d_tmem = tmem + acc * (uint32_t)kDTile;
      for (int kb = 0; kb < nkb; ++kb, ++g) {
        const int st = g % kDStages;
        if (!mbar_wait(&s.full[st], (g / kDStages) & 1)) { s.abort_flag = 1; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t da = make_smem_desc(smem_u32(s.a[st]));
        const uint64_t db = make_smem_desc(smem_u32(s.b[st]));
#pragma unroll
        for (int k = 0; k < kBK / kUmmaK; ++k) {
          const uint32_t accumulate = (kb > 0 || k > 0) ? 1u : 0u;
          const uint64_t adv = (uint64_t)((k * kUmmaK * 4) >> 4);
          asm volatile(
              "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
              ::"r"(d_tmem), "l"(da + adv), "l"(db + adv), "r"(idesc), "r"(accumulate) : "memory");
        }
        commit_pair(&s.empty[st]);
      }
      commit_pair(&s.tfull[acc]);
    }
  } else if (warp >= 2) {
    // ---------------- epilogue warps of both CTAs
    const int q = warp & 3;
    uint32_t it = 0;
    for (int t = pair; t < ntiles; t += npairs, ++it) {
      const uint32_t acc = it & 1u;
      int ok = 1;
      if (lane == 0) {
        ok = mbar_wait(&s.tfull[acc], (it >> 1) & 1) ? 1 : 0;
        if (!ok) s.abort_flag = 1;
        if (s.abort_flag) ok = 0;
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int m0 = (t % nbm) * kDTile + rank * kDHalf, n0 = (t / nbm) * kDTile;
      const int row = m0 + q * 32 + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < kDTile; c0 += 32) {
        uint32_t r[32];
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + acc * (uint32_t)kDTile + (uint32_t)c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr) : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 32 >= kDTile) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa_u32(smem_u32(&s.tempty[acc]), 0)) : "memory");
        }
        store_chunk(r, out, out_t, row, n0 + c0, M, N, ldo, act);
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s.abort_flag) {
    if (threadIdx.x == 0) set_status(status, kWaitTimeout, blockIdx.x, 300);
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();       // neither CTA frees its accumulators or leaves while the other still works
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ------------------------------------------------------------------ outer products
// The input gradient of a net's last layer, [batch, 1] · [1, in], is an outer product: no contraction for the tensor
// cores, and a K padded to 4 takes four more launches.  The operands are cut to TF32 as the tensor cores cut them.
__device__ __forceinline__ float tf32_cut(float x) { return __uint_as_float(__float_as_uint(x) & 0xFFFFE000u); }

// K <= 4: every element is a sum of at most four products.  A thread keeps four columns' operands and walks rows.
// Bound by writing the result: 8192x1024x1 on B200 40 -> 12 us (33 MB).
constexpr int kRankRows = 16;
__global__ void __launch_bounds__(256)
k_gemm_rank4(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, float* __restrict__ out_t, int M, int N,
             int K, int lda, int ldb, int ldo, int act) {
  const int n0 = (int)(blockIdx.x * 256 + threadIdx.x) * 4;
  if (n0 >= N) return;
  float w[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) w[j][k] = n0 + j < N && k < K ? tf32_cut(b[(size_t)(n0 + j) * ldb + k]) : 0.f;
  // groups of kRankRows rows, gridDim.y apart (a grid has at most 65,535 of them)
  for (int64_t g = (int64_t)blockIdx.y * kRankRows; g < M; g += (int64_t)gridDim.y * kRankRows)
  for (int m = (int)g, m1 = M - m > kRankRows ? m + kRankRows : M; m < m1; ++m) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float x = k < K ? tf32_cut(a[(size_t)m * lda + k]) : 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = k < K ? v[j] + x * w[j][k] : v[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = apply_act(v[j], act);
    float* dst = out + (size_t)m * ldo + n0;
    if (n0 + 4 <= N && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
      *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) if (n0 + j < N) dst[j] = v[j];
    }
    if (out_t != nullptr)
#pragma unroll
      for (int j = 0; j < 4; ++j) if (n0 + j < N) out_t[(size_t)(n0 + j) * M + m] = v[j];
  }
}

// ------------------------------------------------------------------ elementwise / layout kernels of the NN app
// tiled transpose of a small matrix, out[c][r] = in[r][c]   (src/base/dense_matrix.h:87-104)
__global__ void k_transpose(const float* __restrict__ in, float* __restrict__ out, int rows, int cols) {
  __shared__ float tile[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x, r0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y)
    if (r0 + j < rows && c < cols) tile[j][threadIdx.x] = in[(size_t)(r0 + j) * cols + c];
  __syncthreads();
  const int r = blockIdx.y * 32 + threadIdx.x, c0 = blockIdx.x * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y)
    if (c0 + j < cols && r < rows) out[(size_t)(c0 + j) * rows + r] = tile[threadIdx.x][j];
}
// A minibatch in one launch: rows sel[] of x, their labels, and (unless null) the transposed rows that the first
// layer's weight gradient reads.  For 256 rows of 64 floats the three index and transpose launches it stands for are
// host time.
__global__ void k_gather_minibatch(const float* __restrict__ x, const float* __restrict__ y, const int64_t* __restrict__ sel, int rows,
                                   int cols, float* __restrict__ xb, float* __restrict__ xbt, float* __restrict__ yb) {
  __shared__ float tile[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x, r0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int r = r0 + j;
    if (r >= rows) continue;
    const size_t from = (size_t)sel[r];
    if (c < cols) {
      const float v = x[from * cols + c];
      xb[(size_t)r * cols + c] = v;
      tile[j][threadIdx.x] = v;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) yb[r] = y[from];
  }
  if (xbt == nullptr) return;
  __syncthreads();
  const int r = r0 + threadIdx.x, c0 = blockIdx.x * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y)
    if (c0 + j < cols && r < rows) xbt[(size_t)(c0 + j) * rows + r] = tile[threadIdx.x][j];
}
// act'(y) expressed through the activation output y
__device__ __forceinline__ float act_slope(float yv, int act) {
  if (act == kActRelu) return yv > 0.f ? 1.f : 0.f;
  if (act == kActScaledTanh) { const float t = yv / 1.7159f; return 1.7159f * 0.6666667f * (1.f - t * t); }
  if (act == kActSigmoid) return yv * (1.f - yv);
  return 1.f;
}
// z = g ∘ act'(y) with act' expressed through the activation output y
__global__ void k_act_backward(const float* __restrict__ g, const float* __restrict__ y, float* __restrict__ z, size_t n, int act) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    z[i] = g[i] * act_slope(y[i], act);
  }
}
// z = g ∘ act'(y) (unless null) and its transpose in one pass over g and y: the weight gradient needs zᵀ, the
// input gradient z.  64 x 64 tiles: 16-byte global accesses both ways where rows and columns are multiples of 4
// (kVec), one float at a time otherwise; the tile's odd row length keeps the transposed reads free of bank conflicts.
// Without kAct the plain transpose of g.
constexpr int kActTile = 64;
template <bool kVec, bool kAct>
__global__ void __launch_bounds__(256)
k_act_backward_t(const float* __restrict__ g, const float* __restrict__ y, float* __restrict__ z, float* __restrict__ zt, int rows,
                 int cols, int act) {
  __shared__ float tile[kActTile][kActTile + 1];
  const int r0 = blockIdx.y * kActTile, c0 = blockIdx.x * kActTile;
  constexpr int kW = kVec ? 4 : 1, kLine = kActTile / kW;
  for (int i = threadIdx.x; i < kActTile * kLine; i += 256) {
    const int r = i / kLine, c = (i % kLine) * kW;
    if (r0 + r >= rows || c0 + c >= cols) continue;
    const size_t at = (size_t)(r0 + r) * cols + c0 + c;
    if (kVec) {
      float4 v = *reinterpret_cast<const float4*>(g + at);
      if (kAct) {
        const float4 yv = *reinterpret_cast<const float4*>(y + at);
        v.x *= act_slope(yv.x, act); v.y *= act_slope(yv.y, act);
        v.z *= act_slope(yv.z, act); v.w *= act_slope(yv.w, act);
      }
      if (z != nullptr) *reinterpret_cast<float4*>(z + at) = v;
      tile[r][c] = v.x; tile[r][c + 1] = v.y; tile[r][c + 2] = v.z; tile[r][c + 3] = v.w;
    } else {
      const float v = kAct ? g[at] * act_slope(y[at], act) : g[at];
      if (z != nullptr) z[at] = v;
      tile[r][c] = v;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kActTile * kLine; i += 256) {
    const int c = i / kLine, r = (i % kLine) * kW;
    if (r0 + r >= rows || c0 + c >= cols) continue;
    float* dst = zt + (size_t)(c0 + c) * rows + r0 + r;
    if (kVec) *reinterpret_cast<float4*>(dst) = make_float4(tile[r][c], tile[r + 1][c], tile[r + 2][c], tile[r + 3][c]);
    else *dst = tile[r][c];
  }
}
// logistic loss layer: loss += Σ log(1+e^{-x y}); grad = -y/(1+e^{x y})   (src/neural_network/loss_layer.h:39-58)
__global__ void k_logistic_loss(const float* __restrict__ x, const float* __restrict__ y, float* __restrict__ grad, size_t n, double* loss) {
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float m = x[i] * y[i];
    acc += (double)log1pexp(-m);
    if (grad) grad[i] = -y[i] / (1.f + __expf(m));
  }
  acc = warp_sum_d(acc);
  if ((threadIdx.x & 31) == 0 && acc != 0.0) atomicAdd(loss, acc);
}
// SGD: w -= α g / (β + sqrt(t));  AdaGrad: h += g², w -= α g / (β + sqrt(h))   (src/neural_network/sgd_solver.h:11-36)
// Bound by reading w, g, h and writing w, h: 16-byte accesses where the arrays allow them (4 M weights, AdaGrad, L2
// flushed: 26.7 -> 20.5 us on B200).
__device__ __forceinline__ void sgd_one(float& w, float g, float& h, float alpha, float beta, float iter, int adagrad) {
  float denom;
  if (adagrad) { const float hv = h + g * g; h = hv; denom = beta + sqrtf(hv); }
  else denom = beta + sqrtf(iter);
  w -= alpha * g / denom;
}
template <bool kVec>
__global__ void k_sgd_update(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ h, size_t n, float alpha, float beta,
                             float iter, int adagrad) {
  const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  if (kVec) {
    for (size_t i = first; i < n / 4; i += step) {
      float4 wv = reinterpret_cast<const float4*>(w)[i], hv = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 gv = reinterpret_cast<const float4*>(g)[i];
      if (adagrad) hv = reinterpret_cast<const float4*>(h)[i];
      sgd_one(wv.x, gv.x, hv.x, alpha, beta, iter, adagrad);
      sgd_one(wv.y, gv.y, hv.y, alpha, beta, iter, adagrad);
      sgd_one(wv.z, gv.z, hv.z, alpha, beta, iter, adagrad);
      sgd_one(wv.w, gv.w, hv.w, alpha, beta, iter, adagrad);
      if (adagrad) reinterpret_cast<float4*>(h)[i] = hv;
      reinterpret_cast<float4*>(w)[i] = wv;
    }
  }
  for (size_t i = (kVec ? n / 4 * 4 : 0) + first; i < n; i += step) {
    float hv = adagrad ? h[i] : 0.f;
    float wv = w[i];
    sgd_one(wv, g[i], hv, alpha, beta, iter, adagrad);
    if (adagrad) h[i] = hv;
    w[i] = wv;
  }
}
// per-column mean-centre and scale to norm sqrt(rows)   (src/neural_network/data_layer.h:25-31)
__global__ void k_col_normalize(float* __restrict__ x, int rows, int cols) {
  const int c = blockIdx.x;
  __shared__ double sh[64];
  double s = 0.0;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) s += x[(size_t)r * cols + c];
  s = warp_sum_d(s);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) { double t = 0; for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += sh[i]; sh[32] = t / rows; }
  __syncthreads();
  const float mean = (float)sh[32];
  double q = 0.0;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) { const float d = x[(size_t)r * cols + c] - mean; q += (double)d * d; }
  q = warp_sum_d(q);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = q;
  __syncthreads();
  if (threadIdx.x == 0) { double t = 0; for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += sh[i]; sh[33] = t; }
  __syncthreads();
  const float nrm = (float)sqrt(sh[33]);
  const float scale = nrm > 0.f ? sqrtf((float)rows) / nrm : 0.f;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) x[(size_t)r * cols + c] = (x[(size_t)r * cols + c] - mean) * scale;
}

}  // namespace psb

using namespace psb;

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}
// 2-D map over a row-major [rows, k] fp32 matrix with row stride ld (floats), box = box_rows rows x 32 floats, 128B swizzle
int make_map(CUtensorMap* map, const float* base, int rows, int k, int ld, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return -1;
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)r;
}
// 256x256 tiles from which on CTA pairs are faster than one 128x128 tile per CTA: 2048x1024x2048 (32 tiles) takes 31 us in
// tiles and 41 in pairs, 2048x2048x512 (64 tiles) 34 and 27
constexpr long kPairTiles = 48;
template <int kRows, int kCols>
int launch_tile(const float* a, const float* b, float* out, float* out_t, int M, int N, int K, int lda, int ldb, int ldo, int act,
                uint32_t* status, cudaStream_t stream) {
  CUtensorMap ma, mb;
  int r = make_map(&ma, a, M, K, lda, kRows);
  if (r == 0) r = make_map(&mb, b, N, K, ldb, kCols);
  if (r) return r;
  const size_t smem = sizeof(GemmSmem) + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tf32_tcgen05_kernel<kRows, kCols>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const dim3 grid((M + kBM - 1) / kBM, (N + kCols - 1) / kCols);
  gemm_tf32_tcgen05_kernel<kRows, kCols><<<grid, 128, smem, stream>>>(ma, mb, out, out_t, M, N, K, ldo, act, status);
  return (int)cudaGetLastError();
}
inline int egrid(size_t n) { size_t b = (n + 255) / 256; if (b < 1) b = 1; if (b > 148 * 8) b = 148 * 8; return (int)b; }

}  // namespace

extern "C" {

// out[M,N] (row stride ldo) = act(a[M,K] (row stride lda) · b[N,K]ᵀ (row stride ldb)); out_t, when not null,
// receives the transpose [N,M] too.  variant: 0 by size, 1 one tile per CTA, 2 CTA pairs, 3 K of at most four.
// Requirements: a, b 16-byte aligned; lda, ldb multiples of 4 floats (variant 3: none).  Returns 0, a CUDA error, or
// -1 when tensor maps cannot be created (no driver entry point).
int psb_gemm_tn_tf32(const float* a, const float* b, float* out, float* out_t, int M, int N, int K, int lda, int ldb, int ldo, int act,
                     int variant, uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const bool aligned = ((lda | ldb) & 3) == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
  if (variant == 3 ? K > 4 : !aligned) return (int)cudaErrorInvalidValue;
  const unsigned row_groups = ((unsigned)M + kRankRows - 1) / kRankRows;
  const dim3 rank_grid((N + 1023) / 1024, row_groups < 65535u ? row_groups : 65535u);
  const long tiles_d = (long)((M + kDTile - 1) / kDTile) * ((N + kDTile - 1) / kDTile);
  if (variant == 0) variant = K <= 4 ? 3 : tiles_d >= kPairTiles ? 2 : 1;
  if (variant == 3) {
    k_gemm_rank4<<<rank_grid, 256, 0, stream>>>(a, b, out, out_t, M, N, K, lda, ldb, ldo, act);
    return (int)cudaGetLastError();
  }
  if (variant == 2) {
    CUtensorMap ma, mb;
    int r = make_map(&ma, a, M, K, lda, kDHalf);
    if (r == 0) r = make_map(&mb, b, N, K, ldb, kDHalf);
    if (r) return r;
    static int sms = 0;
    if (sms == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
    const size_t smem_d = sizeof(GemmSmemD) + 1024;
    static bool attr_d = false;
    if (!attr_d) {
      cudaError_t e = cudaFuncSetAttribute(gemm_tf32_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_d);
      if (e != cudaSuccess) return (int)e;
      attr_d = true;
    }
    const int pairs = (int)(tiles_d < sms / 2 ? tiles_d : sms / 2);
    gemm_tf32_pair_kernel<<<2 * pairs, kPThreads, smem_d, stream>>>(ma, mb, out, out_t, M, N, K, ldo, act, status);
    return (int)cudaGetLastError();
  }
  if (M <= kThinRows) return launch_tile<kThinRows, kThinCols>(a, b, out, out_t, M, N, K, lda, ldb, ldo, act, status, stream);
  return launch_tile<kBM, kBN>(a, b, out, out_t, M, N, K, lda, ldb, ldo, act, status, stream);
}
// An empty matrix is refused here and in psb_act_backward_t: it is a minibatch without rows, whose gradients nothing would write.
int psb_transpose(const float* in, float* out, int rows, int cols, cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return (int)cudaErrorInvalidConfiguration;
  const dim3 grid((cols + kActTile - 1) / kActTile, (rows + kActTile - 1) / kActTile);
  if (grid.y > 65535u) return (int)cudaErrorInvalidValue;
  // 32 x 32 tiles of single floats / 64 x 64 tiles of float4 on B200, L2 flushed: 256x64 6.2 / 8.2 us (few blocks, each with a
  // longer chain), 3000x700 10.2 / 10.2, 1024x4096 16.4 / 12.3, 8192x1024 24.6 / 18.4
  if ((size_t)rows * cols < (size_t)1 << 20) {
    const dim3 small((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
    k_transpose<<<small, block, 0, s>>>(in, out, rows, cols);
    return (int)cudaGetLastError();
  }
  const uintptr_t all = reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out);
  if (((rows | cols) & 3) == 0 && (all & 15) == 0) k_act_backward_t<true, false><<<grid, 256, 0, s>>>(in, nullptr, nullptr, out, rows, cols, 0);
  else k_act_backward_t<false, false><<<grid, 256, 0, s>>>(in, nullptr, nullptr, out, rows, cols, 0);
  return (int)cudaGetLastError();
}
// sel: rows indices into x [*, cols] and y; xbt may be null
int psb_gather_minibatch(const float* x, const float* y, const int64_t* sel, int rows, int cols, float* xb, float* xbt, float* yb,
                         cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return 0;
  const dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
  if (grid.y > 65535u) return (int)cudaErrorInvalidValue;
  k_gather_minibatch<<<grid, block, 0, s>>>(x, y, sel, rows, cols, xb, xbt, yb);
  return (int)cudaGetLastError();
}
int psb_act_backward(const float* g, const float* y, float* z, size_t n, int act, cudaStream_t s) {
  k_act_backward<<<egrid(n), 256, 0, s>>>(g, y, z, n, act);
  return (int)cudaGetLastError();
}
// z (may be null) and its transpose zt [cols, rows]
int psb_act_backward_t(const float* g, const float* y, float* z, float* zt, int rows, int cols, int act, cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return (int)cudaErrorInvalidConfiguration;
  const uintptr_t all = reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(zt);
  const dim3 grid((cols + kActTile - 1) / kActTile, (rows + kActTile - 1) / kActTile);
  if (grid.y > 65535u) return (int)cudaErrorInvalidValue;
  if (((rows | cols) & 3) == 0 && (all & 15) == 0) k_act_backward_t<true, true><<<grid, 256, 0, s>>>(g, y, z, zt, rows, cols, act);
  else k_act_backward_t<false, true><<<grid, 256, 0, s>>>(g, y, z, zt, rows, cols, act);
  return (int)cudaGetLastError();
}
int psb_logistic_loss(const float* x, const float* y, float* grad, size_t n, double* loss, cudaStream_t s) {
  k_logistic_loss<<<egrid(n), 256, 0, s>>>(x, y, grad, n, loss);
  return (int)cudaGetLastError();
}
int psb_sgd_update(float* w, const float* g, float* h, size_t n, float alpha, float beta, float iter, int adagrad, cudaStream_t s) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(h);
  if ((all & 15) == 0) k_sgd_update<true><<<egrid((n + 3) / 4), 256, 0, s>>>(w, g, h, n, alpha, beta, iter, adagrad);
  else k_sgd_update<false><<<egrid(n), 256, 0, s>>>(w, g, h, n, alpha, beta, iter, adagrad);
  return (int)cudaGetLastError();
}
int psb_col_normalize(float* x, int rows, int cols, cudaStream_t s) {
  k_col_normalize<<<cols, 256, 0, s>>>(x, rows, cols);
  return (int)cudaGetLastError();
}

}  // extern "C"
