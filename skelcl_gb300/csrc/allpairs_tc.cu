// AllPairs zip(x*y) / reduce(x+y) over float on the 5th-generation tensor
// cores: P = A (M x K) * B (K x N), both row-major, FP32 in and out.
//
// Precision: "3xBF16" (Henry, Tang & Heinecke, "Leveraging the bfloat16
// Artificial Intelligence Datatype for Higher-Precision Computations",
// ARITH 2019).  Each FP32 operand is split into bf16 parts
//   x = hi + mid + lo (+ O(2^-24 |x|)),  hi = bf16(x), mid = bf16(x - hi),
//   lo = bf16(x - hi - mid)
// and the products whose magnitude can reach FP32 precision are accumulated
// in FP32 in tensor memory, smallest terms first:
//   kind 6: lo*hi + hi*lo + mid*mid + mid*hi + hi*mid + hi*hi   (3 parts)
//   kind 3: mid*hi + hi*mid + hi*hi                              (2 parts)
// The reference's semantics (AllPairsKernel.cl:47-135: P = sum over k of
// A[i][k]*B[k][j], identity 0) are kept; only the order of the FP32 sums
// differs from the sequential fold of the CUDA-core kernel.
// Three parts hold every bit of an FP32 operand (24, of elements that are
// neither tiny nor huge), so that products with one-hot rows and of whole
// numbers below 2^12 are exact, as the sequential fold's are.  (Two FP16 parts
// and three products ran 8192 x 4096 x 8192 in 1.1 ms against 2.0, but hold 22
// or 23 bits: a quarter of all elements times 1 came out changed.)
//
// Shape of the bf16 kernel: 128 x 128 output tile per CTA.  Warp 0 (one thread) streams k-blocks
// of 64 with TMA (3D tensor maps over the split parts, SWIZZLE_128B, one
// mbarrier per stage); warp 1 allocates 2 x 128 TMEM columns and one thread
// issues tcgen05.mma.kind::f16 (M=128, N=128, K=16; both operands K-major in
// shared memory), committing each stage back to the producer.  Each k-block
// is accumulated into one of two TMEM accumulators (ping-pong) and drained
// by warps 2-5 with tcgen05.ld into FP32 registers, where the k-block
// partials are summed with round-to-nearest adds.  Measured on GB300: letting
// the tensor core chain all 1536 MMAs of K = 4096 into one accumulator gave
// a normwise error of 2.6e-5 against FP64, growing about linearly with K (the
// accumulator's additions are not round-to-nearest); draining per k-block
// keeps each chain at 24 MMAs.  Every mbarrier wait is bounded; a wait that
// gives up raises the device status word and the CTA still frees its tensor
// memory before it returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "internal.h"

namespace scl {
namespace tc {

constexpr int BM = 128;
constexpr int MPAD = 256;                        // M padding: whole tiles of CTA pairs
constexpr int NPAD = 256;                        // N padding: fits both tile widths
constexpr int KPAD = 64;                         // K padding: whole k-blocks of both shapes

// Tile shape by output-tile width BN_T: 128 x 128 tiles take k-blocks of 64
// (one 128-byte SWIZZLE_128B row of bf16) with 4 epilogue warps; 128 x 256
// tiles take k-blocks of 32 (one 64-byte SWIZZLE_64B row, so that three
// stages of six parts fit in shared memory) with 8 epilogue warps, and read
// each A tile for twice as many columns.
template <int BN_T>
struct Shape {
  static constexpr int BN = BN_T;
  static constexpr int BK = BN_T == 256 ? 32 : 64;
  static constexpr int A_TILE = BM * BK * 2;     // bytes of one A part per stage
  static constexpr int B_TILE = BN * BK * 2;     // bytes of one B part per stage
  static constexpr int EPI_WARPS = BN / 32;      // each drains 32 rows x 128 columns
  static constexpr int THREADS = 64 + 32 * EPI_WARPS;
  static constexpr uint32_t TMEM_COLS = 2 * BN;  // two FP32 accumulators (ping-pong)
  static constexpr uint32_t SBO = 8 * BK * 2;    // bytes between 8-row groups
  static constexpr uint64_t LAYOUT = BK == 64 ? 2u : 4u;  // SWIZZLE_128B : SWIZZLE_64B
  // Instruction descriptor, kind::f16: D = F32 (bits 4-5 = 1), A = B = BF16
  // (bits 7-9 = 1, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 in bits
  // 17-22, M >> 4 in bits 24-28.
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) |
                                    ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
};

// Shared-memory matrix descriptor for a K-major swizzled tile (rows of BK
// 16-bit parts, 8-row groups SBO bytes apart): start address >> 4 (bits 0-13),
// leading-byte offset 1 (unused for swizzled K-major), stride-byte offset >> 4
// (bits 32-45), descriptor version 1 (bits 46-47), layout (bits 61-63).
template <typename SH>
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;
  d |= (uint64_t)(SH::SBO >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= SH::LAYOUT << 61;
  return d;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;"
      " selp.u32 %0, 1, 0, p; }"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}

// Bounded wait; false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
  uint32_t polls = 0;
  while (!mbar_test(bar, parity)) {
    if (++polls > limit) return false;
    if (polls > 64) __nanosleep(32);
  }
  return true;
}

// 32 / 16 consecutive tensor-memory columns of this warp's 32 lanes (complete
// after tcgen05.wait::ld).
__device__ __forceinline__ void tmem_load32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10,"
      " %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27,"
      " %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10,"
      " %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// The address of `addr` (shared memory) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned; barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void raise(unsigned int* err) {
  if (err) atomicOr(err, 1u);
}

// One operand of the split pass: X, `rows` x K row-major (kmajor) or K x
// `rows` row-major, into planes [part][rp][Kp] of bf16 parts.  Only the first
// `rows` rows of a plane are written (the rest only reach outputs that are
// not stored); k is zero-filled to Kp.
struct Operand {
  const float* x;
  __nv_bfloat16* out;
  uint32_t rows, rp;
  int kmajor;
};

// X tile of 64 rows x KT k (128, or 64: split_depth) at (r0, k0): KT / 8
// neighbouring lanes hold 8 consecutive k each of a row and store 2 * KT
// contiguous bytes per part.
template <int KT>
__device__ __forceinline__ void split_tile(const Operand& op, uint32_t K, uint32_t Kp, uint32_t r0, uint32_t k0,
                                           int parts, float (*tile)[65]) {
  const uint64_t plane = (uint64_t)op.rp * Kp;
  const uint32_t R = op.rows;
  if (!op.kmajor) {
    // K x R: through shared memory, [k][row]; 16-byte loads when rows allow
    // it (r0 and R multiples of 4: a load is wholly in or out)
    if ((R % 4u) == 0 && (reinterpret_cast<uintptr_t>(op.x) & 15u) == 0) {
      const uint32_t c4 = threadIdx.x % 16, kr = threadIdx.x / 16;
      float4 q[KT / 16];
#pragma unroll
      for (int i = 0; i < KT / 16; ++i) {
        const uint32_t k = k0 + kr + 16 * i, n = r0 + c4 * 4;
        q[i] = (k < K && n < R) ? *reinterpret_cast<const float4*>(op.x + (uint64_t)k * R + n)
                                : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < KT / 16; ++i) {
        float* t = &tile[kr + 16 * i][c4 * 4];
        t[0] = q[i].x;
        t[1] = q[i].y;
        t[2] = q[i].z;
        t[3] = q[i].w;
      }
    } else {
#pragma unroll 8
      for (int i = threadIdx.x; i < KT * 64; i += 256) {
        const uint32_t kk = (uint32_t)i / 64, nn = (uint32_t)i % 64;
        const uint32_t k = k0 + kk, n = r0 + nn;
        tile[kk][nn] = (k < K && n < R) ? op.x[(uint64_t)k * R + n] : 0.0f;
      }
    }
    __syncthreads();
  }
  const bool vec = op.kmajor && (K % 4u) == 0 && (reinterpret_cast<uintptr_t>(op.x) & 15u) == 0;
  constexpr int LANES = KT / 8, AT_ONCE = 256 / LANES, PASSES = 64 / AT_ONCE;
  const uint32_t kc = (threadIdx.x % LANES) * 8, k = k0 + kc;
  float x[PASSES][8];
#pragma unroll
  for (int c = 0; c < PASSES; ++c) {
    const uint32_t rr = threadIdx.x / LANES + AT_ONCE * c, row = r0 + rr;
    if (!op.kmajor) {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[c][e] = tile[kc + e][rr];
    } else if (vec && row < R && k + 8 <= K) {
      const float4 a = *reinterpret_cast<const float4*>(op.x + (uint64_t)row * K + k);
      const float4 b = *reinterpret_cast<const float4*>(op.x + (uint64_t)row * K + k + 4);
      x[c][0] = a.x; x[c][1] = a.y; x[c][2] = a.z; x[c][3] = a.w;
      x[c][4] = b.x; x[c][5] = b.y; x[c][6] = b.z; x[c][7] = b.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[c][e] = (row < R && k + e < K) ? op.x[(uint64_t)row * K + k + e] : 0.0f;
    }
  }
#pragma unroll
  for (int c = 0; c < PASSES; ++c) {
    const uint32_t row = r0 + threadIdx.x / LANES + AT_ONCE * c;
    __align__(16) __nv_bfloat16 h[8], m[8], l[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      h[e] = __float2bfloat16_rn(x[c][e]);
      const float r1 = x[c][e] - __bfloat162float(h[e]);
      m[e] = __float2bfloat16_rn(r1);
      l[e] = __float2bfloat16_rn(r1 - __bfloat162float(m[e]));
    }
    if (row < R && k < Kp) {
      __nv_bfloat16* out = op.out + ((uint64_t)row * Kp + k);
      *reinterpret_cast<uint4*>(out) = *reinterpret_cast<const uint4*>(h);
      *reinterpret_cast<uint4*>(out + plane) = *reinterpret_cast<const uint4*>(m);
      if (parts > 2) *reinterpret_cast<uint4*>(out + 2 * plane) = *reinterpret_cast<const uint4*>(l);
    }
  }
}

// Splits both operands, one 64 x KT tile per step (grid-stride over A's tiles,
// then B's).  Bound by memory: reads 4 bytes, writes 6 (three parts)
// per element.  A row-major operand's tiles are taken along k, a transposed
// one's along its rows, so neighbouring blocks read neighbouring memory.
template <int KT>
__global__ void __launch_bounds__(256)
split_kernel(const Operand a, const Operand b, uint32_t K, uint32_t Kp, int parts) {
  __shared__ float tile[KT][65];
  // the contraction's blocks may start setting up once every block here runs
  // (they wait for this grid's end before they read): 2-4 % of a small product
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  dependency_wait();
  const uint32_t kt = (Kp + KT - 1) / KT;
  const uint32_t rta = (a.rows + 63) / 64, rtb = (b.rows + 63) / 64;
  const uint64_t na = (uint64_t)rta * kt, n = na + (uint64_t)rtb * kt;
  for (uint64_t t = blockIdx.x; t < n; t += gridDim.x) {
    const bool second = t >= na;
    const Operand& op = second ? b : a;
    const uint64_t i = second ? t - na : t;
    const uint32_t rt = second ? rtb : rta;
    const uint32_t r0 = (uint32_t)(op.kmajor ? i / kt : i % rt) * 64;
    const uint32_t k0 = (uint32_t)(op.kmajor ? i % kt : i / rt) * KT;
    split_tile<KT>(op, K, Kp, r0, k0, parts, tile);
    if (n > gridDim.x) __syncthreads();  // (block-uniform: the tile is filled again)
  }
}

// Whether 16-byte stores fit every row of P: it may be a view that starts at
// any element.
__device__ __forceinline__ bool rows_aligned(const float* P, uint32_t N) {
  return (N % 4u) == 0u && (reinterpret_cast<uintptr_t>(P) & 15u) == 0;
}

// A 128 x 128 tile's sums lie in the shared memory of the cluster's `ranks`
// blocks (16-byte chunk c of row r at chunk c ^ (r % 32) of the row's 512
// bytes): this block adds up its share of the rows, in block order, and stores
// them, a warp per row.  us, against a thread storing its own row's 128 sums:
// 1400 x 300 x 1400 14.7 -> 13.5, x 1401 23.7 -> 14.4, 1500 x 2000 x 1499 57.7 ->
// 48.8.
template <int THREADS>
__device__ __forceinline__ void store_sums(uint32_t base, uint32_t ranks, uint32_t rank, uint32_t m0, uint32_t n0,
                                           uint32_t M, uint32_t N, float* P) {
  const uint32_t rows = BM / ranks, first = rank * rows;
  const bool vec = rows_aligned(P, N);
  for (uint32_t i = threadIdx.x; i < rows * 32u; i += THREADS) {
    const uint32_t r = first + i / 32u, c = i % 32u;
    const uint32_t at = base + r * 512u + ((c ^ (r & 31u)) * 16u);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t p = 0; p < ranks; ++p) {
      float4 o;
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(cluster_addr(at, p)) : "memory");
      v.x += o.x;
      v.y += o.y;
      v.z += o.z;
      v.w += o.w;
    }
    const uint32_t row = m0 + r, col = n0 + c * 4u;
    if (row < M) {
      float* dst = P + (uint64_t)row * N + col;
      if (vec && col + 4u <= N) {
        *reinterpret_cast<float4*>(dst) = v;
      } else {
        if (col < N) dst[0] = v.x;
        if (col + 1u < N) dst[1] = v.y;
        if (col + 2u < N) dst[2] = v.z;
        if (col + 3u < N) dst[3] = v.w;
      }
    }
  }
}

// G = k-blocks accumulated in tensor memory between two drains into the
// epilogue's FP32 registers (1: every k-block; larger G drains less often at
// a longer in-TMEM accumulation chain).
//
// Output tiles are numbered in groups of `group_m` tile rows: block b of the
// 1D grid takes tile row first + (b mod group) mod rows and tile column
// (b mod group) div rows of its group, so consecutive blocks share one
// column of B's parts while cycling over a few rows of A's.  A wave of one
// block per SM then reads about group_m rows of A and SMs / group_m columns
// of B, which stay in L2 for the whole wave (row-major order read every
// column of B in every wave: at 4096^3, 2.5x the parts' bytes from DRAM).
// SPLIT: the blocks of a cluster share one output tile, each taking a share of
// its k-blocks; their sums meet in shared memory, where every block adds up
// its share of the tile's rows, in block order.
template <int PARTS, int STAGES, int G, int BN_T, bool SPLIT = false>
__global__ void __launch_bounds__(Shape<BN_T>::THREADS, 1)
gemm_3xbf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   float* P, uint32_t M, uint32_t N, uint32_t Kp, uint32_t spin_limit,
                   unsigned int* err, uint32_t tiles_n, uint32_t group_m) {
  using SH = Shape<BN_T>;
  constexpr int BN = SH::BN, BK = SH::BK;
  constexpr int STAGE_BYTES = PARTS * (SH::A_TILE + SH::B_TILE);
  constexpr uint32_t TMEM_COLS = SH::TMEM_COLS;
  constexpr uint32_t IDESC = SH::IDESC;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t acc_full[2];   // MMA -> epilogue: k-block partial ready
  __shared__ __align__(8) uint64_t acc_empty[2];  // epilogue -> MMA: accumulator drained
  __shared__ __align__(8) uint64_t drain_bar;     // all issued MMAs have finished
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;  // 1024-aligned stage ring
  uint32_t n0, m0, ranks = 1, rank = 0;
  if constexpr (SPLIT) {
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  }
  {
    const uint32_t tile = blockIdx.x / ranks;
    const uint32_t tiles_m = gridDim.x / ranks / tiles_n, per_group = group_m * tiles_n;
    const uint32_t grp = tile / per_group, r = tile % per_group;
    const uint32_t first = grp * group_m;
    const uint32_t rows = tiles_m - first < group_m ? tiles_m - first : group_m;
    m0 = (first + r % rows) * BM;
    n0 = (r / rows) * BN;
  }
  // this block's k-blocks: nk from k0 on
  const uint32_t all_k = Kp / BK, k0 = all_k * rank / ranks, nk = all_k * (rank + 1) / ranks - k0;

  if (threadIdx.x == 0) {
    s_fail = 0;
    for (int s = 0; s < STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&full_bar[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&empty_bar[s])));
    }
    for (int a = 0; a < 2; ++a) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&acc_full[a])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;"
                   :: "r"(smem_u32(&acc_empty[a])), "r"(SH::EPI_WARPS));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&drain_bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" :: "l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" :: "l"(&tmB) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  dependency_wait();  // (the barriers and tensor memory above need nothing of the split)
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    // ---- TMA producer
    if (lane == 0) {
      for (uint32_t kb = 0; kb < nk; ++kb) {
        const int s = (int)(kb % STAGES);
        const uint32_t round = kb / STAGES;
        if (round > 0 && !mbar_wait(smem_u32(&empty_bar[s]), (round - 1) & 1u, spin_limit)) {
          raise(err);
          s_fail = 1;
          break;
        }
        const uint32_t fb = smem_u32(&full_bar[s]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     :: "r"(fb), "r"((uint32_t)STAGE_BYTES) : "memory");
        const uint32_t stage = base + (uint32_t)s * STAGE_BYTES;
        const int kx = (int)((k0 + kb) * BK);
#pragma unroll
        for (int p = 0; p < PARTS; ++p) {
          asm volatile(
              "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
              " [%0], [%1, {%2, %3, %4}], [%5];"
              :: "r"(stage + (uint32_t)p * SH::A_TILE), "l"(&tmA), "r"(kx), "r"((int)m0), "r"(p),
                 "r"(fb)
              : "memory");
          asm volatile(
              "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
              " [%0], [%1, {%2, %3, %4}], [%5];"
              :: "r"(stage + (uint32_t)(PARTS * SH::A_TILE + p * SH::B_TILE)), "l"(&tmB), "r"(kx),
                 "r"((int)n0), "r"(p), "r"(fb)
              : "memory");
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer
    if (lane == 0) {
      // (a part, b part) products, smallest first
      constexpr int NPROD = PARTS == 3 ? 6 : 3;
      int prod_a[NPROD], prod_b[NPROD];
      if (PARTS == 3) {  // lo*hi, hi*lo, mid*mid, mid*hi, hi*mid, hi*hi
        const int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
        for (int q = 0; q < NPROD; ++q) { prod_a[q] = pa[q]; prod_b[q] = pb[q]; }
      } else {           // mid*hi, hi*mid, hi*hi
        const int pa[3] = {1, 0, 0}, pb[3] = {0, 1, 0};
        for (int q = 0; q < NPROD; ++q) { prod_a[q] = pa[q]; prod_b[q] = pb[q]; }
      }
      for (uint32_t kb = 0; kb < nk; ++kb) {
        const int s = (int)(kb % STAGES);
        const uint32_t grp = kb / G;          // drain group of this k-block
        const bool first_in_grp = kb % G == 0;
        const bool last_in_grp = kb % G == G - 1 || kb + 1 == nk;
        const int acc_i = (int)(grp & 1u);
        const uint32_t use = grp >> 1;  // how often this accumulator was used before
        if (first_in_grp && use > 0 &&
            !mbar_wait(smem_u32(&acc_empty[acc_i]), (use - 1) & 1u, spin_limit)) {
          raise(err);
          s_fail = 1;
          break;
        }
        if (!mbar_wait(smem_u32(&full_bar[s]), (kb / STAGES) & 1u, spin_limit)) {
          raise(err);
          s_fail = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t stage = base + (uint32_t)s * STAGE_BYTES;
        const uint32_t dtm = tmem + (uint32_t)(acc_i * BN);
#pragma unroll
        for (int q = 0; q < NPROD; ++q) {
          const uint64_t ad = smem_desc<SH>(stage + (uint32_t)prod_a[q] * SH::A_TILE);
          const uint64_t bd =
              smem_desc<SH>(stage + (uint32_t)(PARTS * SH::A_TILE + prod_b[q] * SH::B_TILE));
#pragma unroll
          for (int ks = 0; ks < BK / 16; ++ks) {
            // advance 16 bf16 = 32 bytes along K inside the swizzle row
            const uint64_t a = ad + (uint64_t)(ks * 2);
            const uint64_t b = bd + (uint64_t)(ks * 2);
            const uint32_t acc = (!first_in_grp || q > 0 || ks > 0) ? 1u : 0u;  // fresh per group
            asm volatile(
                "{ .reg .pred p; setp.ne.b32 p, %4, 0;"
                " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
                :: "r"(dtm), "l"(a), "l"(b), "r"(IDESC), "r"(acc)
                : "memory");
          }
        }
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
            :: "r"(smem_u32(&empty_bar[s])) : "memory");
        if (last_in_grp)
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
              :: "r"(smem_u32(&acc_full[acc_i])) : "memory");
      }
      // no MMA may still run when the tensor memory is freed (also after a
      // failed wait above)
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
          :: "r"(smem_u32(&drain_bar)) : "memory");
      if (!mbar_wait(smem_u32(&drain_bar), 0, spin_limit)) raise(err);
    }
  } else {
    // ---- epilogue: warp w (2 .. 1 + EPI_WARPS) owns TMEM lanes 32*(w % 4) ..
    //      and columns 128*((w - 2) / 4) ..; each thread keeps its row's 128
    //      partial sums in registers
    constexpr int CW = 128;  // columns per epilogue warp
    const int q = warp & 3;
    const int h = (warp - 2) >> 2;
    float sum[CW];
#pragma unroll
    for (int j = 0; j < CW; ++j) sum[j] = 0.0f;
    bool ok = true;
    const uint32_t ngrp = (nk + G - 1) / G;
    for (uint32_t grp = 0; grp < ngrp; ++grp) {
      const int acc_i = (int)(grp & 1u);
      if (!mbar_wait(smem_u32(&acc_full[acc_i]), (grp >> 1) & 1u, spin_limit)) {
        if (lane == 0) raise(err);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < CW / 32; ++c) {
        uint32_t r[32];
        tmem_load32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc_i * BN + h * CW + c * 32), r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[c * 32 + j] += __uint_as_float(r[j]);
      }
      // accumulator drained: hand it back to the MMA issuer (one arrive per warp)
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];"
                     :: "r"(smem_u32(&acc_empty[acc_i])) : "memory");
    }
    if (BN == 128) {
      // (every MMA that reads the stages has completed)  16-byte chunk c of
      // row r at chunk c ^ (r % 32): a warp's accesses meet all banks
      const uint32_t r = (uint32_t)(q * 32 + lane);
#pragma unroll
      for (int c = 0; c < CW / 4; ++c)
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};"
                     :: "r"(base + r * (CW * 4) + (((uint32_t)c ^ (r & 31u)) * 16u)), "f"(sum[c * 4]),
                        "f"(sum[c * 4 + 1]), "f"(sum[c * 4 + 2]), "f"(sum[c * 4 + 3])
                     : "memory");
    } else if (ok) {
      const uint32_t row = m0 + (uint32_t)(q * 32 + lane);
      if (row < M) {
        const bool vec = rows_aligned(P, N);
#pragma unroll
        for (int c = 0; c < CW / 32; ++c) {
          const uint32_t col0 = n0 + (uint32_t)(h * CW + c * 32);
          float* dst = P + (uint64_t)row * N + col0;
          if (vec && col0 + 32 <= N) {
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              *reinterpret_cast<float4*>(dst + j) =
                  make_float4(sum[c * 32 + j], sum[c * 32 + j + 1], sum[c * 32 + j + 2],
                              sum[c * 32 + j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (col0 + j < N) dst[j] = sum[c * 32 + j];
          }
        }
      }
    }
  }

  static_assert(!SPLIT || BN == 128, "one epilogue warp per 32 rows: its sums are whole rows");
  if constexpr (BN == 128) {
    __syncthreads();
    if constexpr (SPLIT) cluster_sync();
    store_sums<SH::THREADS>(base, ranks, rank, m0, n0, M, N, P);
    if constexpr (SPLIT) {
      __syncthreads();
      cluster_sync();  // no block leaves while another may still read its sums
    }
  }

  // ---- teardown: wait for the copies a failed pipeline may still have in
  //      flight (bounded), then free the tensor memory
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_fail && threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_wait(smem_u32(&full_bar[s]), 0, spin_limit);
      mbar_wait(smem_u32(&full_bar[s]), 1, spin_limit);
    }
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 :: "r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// ---- CTA pairs --------------------------------------------------------------------
// 256 x 256 output tiles, each by a pair of CTAs (cta_group::2, M = 256, N =
// 256, K = 16): k-blocks of 32, four stages of 48 KB per CTA.  Each CTA of the
// pair holds 128 rows of A and 128 of the 256 columns of B per stage and the
// accumulators of its 128 rows x 256 columns; the pair's first CTA issues the
// MMAs.  Two 256-column accumulators in tensor memory alternate (ping-pong),
// drained every 64 of K by 8 epilogue warps of 32 rows x 128 columns into FP32
// registers.  The products of a k-block of 32 follow one another as in
// gemm_3xbf16_kernel's 256-column tiles, or (SMALLEST_FIRST) those of a drain's
// two together as in its 128-column tiles: the same sums in the same order, so
// the same bits.
// Against gemm_3xbf16_kernel a pair reads each operand for twice the outputs.
// Bound by the tensor cores, then by the way round an accumulator (MMAs, commit,
// drain, arrival from the other CTA).  16 epilogue warps of 64 columns and two
// half-tiles of N = 128 with their own accumulators were a tenth and a fifth
// slower.
// WALK: as many pairs as the device holds, each over several tiles, so that one
// tile's way out overlaps the next one's products (allpairs_pair_launch says
// when).
constexpr int kPairCols = 256;  // tile columns; the tile has 2 * BM rows
constexpr int kPairCW = 128;    // columns per epilogue warp
constexpr int kPairThreads = 64 + 32 * 4 * (kPairCols / kPairCW);
struct PairShape {
  static constexpr int PARTS = 3;
  static constexpr int STAGES = 4;
  static constexpr int G = 2;  // k-blocks per drain
  static constexpr int BK = 32;
  static constexpr int TILE = BM * BK * 2;       // bytes of one part of either operand per CTA
  static constexpr int STAGE_BYTES = 2 * PARTS * TILE;
  static constexpr uint32_t SBO = 8 * BK * 2;
  static constexpr uint64_t LAYOUT = 4u;         // SWIZZLE_64B
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kPairCols >> 3) << 17) |
                                    ((uint32_t)(2 * BM >> 4) << 24);
};
constexpr int kPairOut = 4 * (kPairCols / kPairCW) * 2048;  // an epilogue warp's way out
constexpr size_t kPairSmem = (size_t)PairShape::STAGES * PairShape::STAGE_BYTES + kPairOut + 1024;

struct PairArgs {
  float* P;
  unsigned int* err;
  uint32_t M, N, Kp, spin_limit, tiles_n, tiles_m, group_m;
};

// Bounded wait for arrivals from both CTAs.  ACQUIRE: for what they wrote to
// shared memory (the operands' copies, read by MMAs that nothing else orders
// after them); without it for the accumulators, which the tcgen05 fences on
// either side of the hand-over order.
template <bool ACQUIRE>
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, uint32_t limit) {
  uint32_t polls = 0;
  for (;;) {
    uint32_t ok;
    if (ACQUIRE)
      asm volatile(
          "{ .reg .pred p; mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;"
          " selp.u32 %0, 1, 0, p; }"
          : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    else
      asm volatile(
          "{ .reg .pred p; mbarrier.test_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;"
          " selp.u32 %0, 1, 0, p; }"
          : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
    if (++polls > limit) return false;
    if (polls > 64) __nanosleep(32);
  }
}
// Arrives on `bar` of both CTAs of the pair once every MMA issued so far has
// completed.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      :: "r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}

struct PairBarriers {
  uint64_t full[4];       // operands of a stage landed, both CTAs' (used in the first CTA)
  uint64_t empty[4];      // the MMAs reading a stage completed (each CTA)
  uint64_t acc_full[2];   // accumulator ready (each CTA)
  uint64_t acc_empty[2];  // accumulator drained by both CTAs' epilogues (first CTA)
  uint64_t drain;         // all issued MMAs completed (each CTA)
};

template <bool WALK, bool SMALLEST_FIRST>
__device__ __forceinline__ void pair_body(const CUtensorMap& tmA, const CUtensorMap& tmB, const PairArgs& g,
                                          uint32_t base, uint32_t stage_out, PairBarriers* bars, uint32_t tmem,
                                          uint32_t rank, int* s_fail) {
  using SH = PairShape;
  constexpr int EPI_WARPS = 4 * (kPairCols / kPairCW);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t nk = g.Kp / SH::BK, tiles = g.tiles_m * g.tiles_n;
  // WALK: the pair takes tiles pair, pair + pairs, ... of all; else tile `pair`
  const uint32_t pair = blockIdx.x / 2, pairs = WALK ? gridDim.x / 2 : 1, end = WALK ? tiles : pair + 1;
  // this CTA's rows m0 .. and the tile's columns n0 .. of tile t: tiles in
  // groups of group_m tile rows (see gemm_3xbf16_kernel)
  auto place = [&](uint32_t t, uint32_t* m0, uint32_t* n0) {
    const uint32_t per_group = g.group_m * g.tiles_n;
    const uint32_t grp = t / per_group, r = t % per_group, first = grp * g.group_m;
    const uint32_t rows = g.tiles_m - first < g.group_m ? g.tiles_m - first : g.group_m;
    *m0 = ((first + r % rows) * 2 + rank) * BM;
    *n0 = (r / rows) * kPairCols;
  };
  // the roles' counters run on across the tiles, so that a tile's first operands
  // and MMAs overlap the last one's way out
  if (warp == 0) {
    // ---- TMA producer (both CTAs): its 128 rows of A and of B's columns, counted
    //      on the first CTA's barrier
    if (lane == 0) {
      uint32_t m0, n0, it = 0;  // k-blocks so far
      bool landed = true;
      for (uint32_t t = pair; landed && t < end; t += pairs) {
        place(t, &m0, &n0);
        for (uint32_t kb = 0; kb < nk; ++kb, ++it) {
          const uint32_t s = it % SH::STAGES, round = it / SH::STAGES;
          if (round > 0 && !mbar_wait(smem_u32(&bars->empty[s]), (round - 1) & 1u, g.spin_limit)) {
            raise(g.err);
            *s_fail = 1;
            landed = false;
            break;
          }
          const uint32_t fb = smem_u32(&bars->full[s]);
          if (rank == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                         :: "r"(fb), "r"((uint32_t)(2 * SH::STAGE_BYTES)) : "memory");
          const uint32_t first_fb = cluster_addr(fb, 0);
          const uint32_t stage = base + s * SH::STAGE_BYTES;
          const int kx = (int)(kb * SH::BK);
#pragma unroll
          for (int p = 0; p < SH::PARTS; ++p) {
            asm volatile(
                "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                " [%0], [%1, {%2, %3, %4}], [%5];"
                :: "r"(stage + (uint32_t)(p * SH::TILE)), "l"(&tmA), "r"(kx), "r"((int)m0), "r"(p), "r"(first_fb)
                : "memory");
            asm volatile(
                "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                " [%0], [%1, {%2, %3, %4}], [%5];"
                :: "r"(stage + (uint32_t)((SH::PARTS + p) * SH::TILE)), "l"(&tmB), "r"(kx),
                   "r"((int)(n0 + rank * 128u)), "r"(p), "r"(first_fb)
                : "memory");
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer (first CTA)
    if (lane == 0) {
      if (rank == 0) {
        // the products of one k-block: part pa of A times part pb of B
        auto mma = [&](uint32_t dtm, uint32_t stage, int pa, int pb, bool fresh) {
          const uint64_t ad = smem_desc<SH>(stage + (uint32_t)(pa * SH::TILE));
          const uint64_t bd = smem_desc<SH>(stage + (uint32_t)((SH::PARTS + pb) * SH::TILE));
#pragma unroll
          for (int ks = 0; ks < SH::BK / 16; ++ks) {
            // 16 elements = 32 bytes along K inside the swizzle row
            const uint64_t a = ad + (uint64_t)(ks * 2), b = bd + (uint64_t)(ks * 2);
            const uint32_t acc = fresh && ks == 0 ? 0u : 1u;
            asm volatile(
                "{ .reg .pred p; setp.ne.b32 p, %4, 0;"
                " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p; }"
                :: "r"(dtm), "l"(a), "l"(b), "r"(SH::IDESC), "r"(acc)
                : "memory");
          }
        };
        // lo*hi, hi*lo, mid*mid, mid*hi, hi*mid, hi*hi: smallest first
        constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
        bool landed = true;
        uint32_t it = 0, grp = 0;  // k-blocks and drain groups so far
        for (uint32_t t = pair; landed && t < end; t += pairs) {
          for (uint32_t kb = 0; landed && kb < nk; kb += SH::G, it += SH::G, ++grp) {  // one drain group
            const uint32_t acc_i = grp & 1u, use = grp >> 1;
            const uint32_t dtm = tmem + acc_i * kPairCols;
            if (use > 0)
              landed = mbar_wait_cluster<false>(smem_u32(&bars->acc_empty[acc_i]), (use - 1) & 1u, g.spin_limit);
            if constexpr (SMALLEST_FIRST) {
              // the whole drain group product by product, the smallest first,
              // as gemm_3xbf16_kernel does with its k-blocks of 64
#pragma unroll
              for (int j = 0; j < SH::G; ++j)
                landed = landed && mbar_wait_cluster<true>(smem_u32(&bars->full[(it + j) % SH::STAGES]),
                                                     ((it + j) / SH::STAGES) & 1u, g.spin_limit);
              if (!landed) break;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
              for (int q = 0; q < 6; ++q)
#pragma unroll
                for (int j = 0; j < SH::G; ++j)
                  mma(dtm, base + (it + j) % SH::STAGES * SH::STAGE_BYTES, pa[q], pb[q], q == 0 && j == 0);
#pragma unroll
              for (int j = 0; j < SH::G; ++j) commit_pair(smem_u32(&bars->empty[(it + j) % SH::STAGES]));
            } else {
#pragma unroll
              for (int j = 0; j < SH::G; ++j) {
                const uint32_t s = (it + j) % SH::STAGES, stage = base + s * SH::STAGE_BYTES;
                landed = landed && mbar_wait_cluster<true>(smem_u32(&bars->full[s]), ((it + j) / SH::STAGES) & 1u,
                                                     g.spin_limit);
                if (!landed) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int q = 0; q < 6; ++q) mma(dtm, stage, pa[q], pb[q], q == 0 && j == 0);
                commit_pair(smem_u32(&bars->empty[s]));
              }
            }
            if (landed) commit_pair(smem_u32(&bars->acc_full[acc_i]));
          }
        }
        if (!landed) {
          raise(g.err);
          *s_fail = 1;
        }
        // no MMA may still run when the tensor memory is freed (also after a
        // failed wait above)
        commit_pair(smem_u32(&bars->drain));
      }
      if (!mbar_wait(smem_u32(&bars->drain), 0, g.spin_limit)) raise(g.err);
    }
  } else {
    // ---- epilogue (both CTAs): warp w (2 .. 9) owns tensor-memory lanes
    //      32 * (w % 4) .. and columns 128 * ((w - 2) / 4) ..
    const int q = warp & 3;
    const uint32_t tile_col = (uint32_t)(((warp - 2) >> 2) * kPairCW);
    bool ok = true;
    uint32_t grp = 0;  // drain groups so far
    for (uint32_t t = pair; ok && t < end; t += pairs) {
      uint64_t sum[kPairCW / 2];  // pairs of neighbouring columns
#pragma unroll
      for (int j = 0; j < kPairCW / 2; ++j) sum[j] = 0ull;
      const uint32_t last = grp + nk / SH::G;
      for (; grp != last; ++grp) {
        const uint32_t acc_i = grp & 1u;
        if (!mbar_wait(smem_u32(&bars->acc_full[acc_i]), (grp >> 1) & 1u, g.spin_limit)) {
          if (lane == 0) raise(g.err);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tm = tmem + ((uint32_t)(q * 32) << 16) + acc_i * kPairCols + tile_col;
#pragma unroll
        for (int c = 0; c < kPairCW / 16; ++c) {
          uint32_t r[16];
          tmem_load16(tm + (uint32_t)(c * 16), r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum[c * 8 + j]) : "l"(pack2(r[2 * j], r[2 * j + 1])));
        }
        // accumulator drained: hand it back to the MMA issuer (one arrive per warp)
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];"
                       :: "r"(cluster_addr(smem_u32(&bars->acc_empty[acc_i]), 0)) : "memory");
      }
      // The sums leave 16 columns at a time through shared memory (16-byte chunk
      // c of row r at chunk c ^ (r / 2 % 4)), four lanes to a row, so that a
      // store covers 64 bytes of eight rows instead of 16 bytes of 32 (with three
      // products in place of six, 8192 x 256 x 8192 245 -> 171 us, K = 4096 1.14 ->
      // 1.11 ms).
      if (ok) {
        const uint32_t st = stage_out + (uint32_t)(warp - 2) * 2048u;
        const bool vec = rows_aligned(g.P, g.N);
        uint32_t m0, n0;
        place(t, &m0, &n0);
#pragma unroll
        for (int c = 0; c < kPairCW / 16; ++c) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            asm volatile("st.shared.v2.u64 [%0], {%1, %2};"
                         :: "r"(st + (uint32_t)lane * 64u + (((uint32_t)j ^ ((uint32_t)lane >> 1 & 3u)) * 16u)),
                            "l"(sum[c * 8 + 2 * j]), "l"(sum[c * 8 + 2 * j + 1])
                         : "memory");
          __syncwarp();
          const uint32_t col0 = n0 + tile_col + (uint32_t)(c * 16);
          if (vec) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t r = (uint32_t)(i * 8 + (lane >> 2)), ch = (uint32_t)(lane & 3);
              float4 v;
              asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                           : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                           : "r"(st + r * 64u + ((ch ^ (r >> 1 & 3u)) * 16u))
                           : "memory");
              const uint32_t row = m0 + (uint32_t)(q * 32) + r, col = col0 + ch * 4u;
              if (row < g.M && col < g.N) *reinterpret_cast<float4*>(g.P + (uint64_t)row * g.N + col) = v;
            }
          } else {
            // sixteen lanes to a row: 8000 x 256 x 8001 212 -> 166 us (three
            // products), 2001 x 1000 x 2003 48 -> 41 against four 4-byte stores of
            // four lanes to a row
            const uint32_t cc = (uint32_t)(lane & 15), col = col0 + cc;
#pragma unroll 4
            for (int i = 0; i < 16; ++i) {
              const uint32_t r = (uint32_t)(i * 2 + (lane >> 4)), row = m0 + (uint32_t)(q * 32) + r;
              float v;
              asm volatile("ld.shared.f32 %0, [%1];"
                           : "=f"(v) : "r"(st + r * 64u + (((cc >> 2) ^ (r >> 1 & 3u)) * 16u) + (cc & 3u) * 4u)
                           : "memory");
              if (row < g.M && col < g.N) g.P[(uint64_t)row * g.N + col] = v;
            }
          }
          __syncwarp();
        }
      }
    }
  }
  static_assert(EPI_WARPS * 32 + 64 == kPairThreads, "");
}

// WALK, SMALLEST_FIRST: see above.
template <bool WALK, bool SMALLEST_FIRST>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const PairArgs g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) PairBarriers bars;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail;
  const int warp = threadIdx.x >> 5;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;  // 1024-aligned stage ring
  const uint32_t stage_out = base + PairShape::STAGES * PairShape::STAGE_BYTES;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  if (threadIdx.x == 0) {
    s_fail = 0;
    auto init = [](uint64_t* b, uint32_t count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(b)), "r"(count));
    };
    for (int s = 0; s < 4; ++s) {
      init(&bars.full[s], 1);
      init(&bars.empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      init(&bars.acc_full[a], 1);
      init(&bars.acc_empty[a], 2 * 4 * (kPairCols / kPairCW));
    }
    init(&bars.drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  dependency_wait();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // both CTAs' barriers are initialised, both hold tensor memory
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  pair_body<WALK, SMALLEST_FIRST>(tmA, tmB, g, base, stage_out, &bars, tmem, rank, &s_fail);

  // ---- teardown: wait for the copies a failed pipeline may still have in
  //      flight (bounded), then, both CTAs together, free the tensor memory
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_fail && threadIdx.x == 0) {
    for (int s = 0; s < 4; ++s) {
      mbar_wait(smem_u32(&bars.full[s]), 0, g.spin_limit);
      mbar_wait(smem_u32(&bars.full[s]), 1, g.spin_limit);
    }
  }
  __syncthreads();
  cluster_sync();  // neither CTA leaves while the other may still signal it
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
  }
}

// ---- One wave of 128 x 128 tiles, the split fused -----------------------------------
// Blocks that read the operands themselves: 512 threads load a k-block of 64 as
// FP32 into registers, split it into three bf16 parts and store those where
// gemm_3xbf16_kernel's TMA would have put them, while the tensor cores work on
// the k-block before and the sums of the one before that are drained.  No split
// pass, no planes written and read back, 64 instead of 96 KB per k-block from
// L2; but every tile splits its own rows and columns, at 1.7 us per k-block (2.1
// with an operand whose k are not contiguous, 2.5 with both) against 1.2 of
// the kernel that reads parts: bound by the conversions, and by shared memory,
// which the tensor cores' operand reads alone keep at 90 %.  It wins while the
// k-blocks are few.  us, split pass and kernel / fused: 500 x K x 600 K = 40
// 9.4 / 6.1, 128 10.9 / 7.9, 190 11.7 / 10.7, 256 12.7 / 11.9, 300 14.0 / 14.1;
// 1000 x K x 1100 K = 128 10.2 / 8.0, 256 12.2 / 12.0, 300 13.4 / 14.4; left
// operand transposed K = 190 11.3 / 11.3, 256 12.4 / 13.7.  (256 threads: 2.4
// us per k-block.)  The same parts in the same order: the same bits.
struct Fused {
  Operand a, b;
  float* P;
  unsigned int* err;
  uint32_t M, N, K, spin_limit, tiles_n, group_m;
};
constexpr int kFusedThreads = 512;
constexpr int kFusedChunks = 1024 / kFusedThreads;     // of either operand per thread
constexpr int kFusedCols = 128 * 128 / kFusedThreads;  // of sums per thread

// The operand's k-block of 64 at k0, rows r0 .. + 127, 8 consecutive k (a
// 16-byte chunk of a part) at a time: chunk c of row
// c / 8 where k is contiguous, else of row c % 128, so that lanes read
// neighbouring memory.
struct FusedPlace {
  uint32_t row, kc;
};
__device__ __forceinline__ FusedPlace fused_place(int kmajor, int i) {
  const uint32_t c = threadIdx.x + (uint32_t)i * kFusedThreads;
  return kmajor ? FusedPlace{c / 8u, c % 8u} : FusedPlace{c % 128u, c / 128u};
}
__device__ __forceinline__ void fused_load(const Operand& op, uint32_t K, uint32_t r0, uint32_t k0, bool vec,
                                           float (&x)[kFusedChunks][8]) {
#pragma unroll
  for (int i = 0; i < kFusedChunks; ++i) {
    const FusedPlace at = fused_place(op.kmajor, i);
    const uint32_t row = r0 + at.row, k = k0 + at.kc * 8u;
    const bool in = row < op.rows;
    if (op.kmajor) {
      const float* src = op.x + (in ? (uint64_t)row * K + k : 0u);
      if (vec && in && k + 8u <= K) {
        const float4 u = *reinterpret_cast<const float4*>(src), v = *reinterpret_cast<const float4*>(src + 4);
        x[i][0] = u.x; x[i][1] = u.y; x[i][2] = u.z; x[i][3] = u.w;
        x[i][4] = v.x; x[i][5] = v.y; x[i][6] = v.z; x[i][7] = v.w;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[i][e] = in && k + e < K ? src[e] : 0.0f;
      }
    } else {
      const float* src = op.x + (in ? (uint64_t)k * op.rows + row : 0u);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[i][e] = in && k + e < K ? src[(uint64_t)e * op.rows] : 0.0f;
    }
  }
}
__device__ __forceinline__ void fused_store(int kmajor, const float (&x)[kFusedChunks][8], uint32_t tile) {
#pragma unroll
  for (int i = 0; i < kFusedChunks; ++i) {
    const FusedPlace at = fused_place(kmajor, i);
    uint32_t part[3][4];
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      float u = x[i][e], v = x[i][e + 1];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(u, v);
        part[p][e / 2] = *reinterpret_cast<const uint32_t*>(&h);
        u -= __low2float(h);
        v -= __high2float(h);
      }
    }
    // (SWIZZLE_128B: 16-byte chunk kc of row r at chunk kc ^ (r % 8))
    const uint32_t dst = tile + at.row * 128u + ((at.kc ^ (at.row & 7u)) * 16u);
#pragma unroll
    for (int p = 0; p < 3; ++p)
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                   :: "r"(dst + (uint32_t)p * Shape<128>::A_TILE), "r"(part[p][0]), "r"(part[p][1]), "r"(part[p][2]),
                      "r"(part[p][3])
                   : "memory");
  }
}

// SPLIT: the blocks of a cluster share an output tile's k-blocks.
template <bool SPLIT>
__global__ void __launch_bounds__(kFusedThreads, 1) gemm_fused_kernel(const Fused g) {
  using SH = Shape<128>;
  constexpr int STAGE_BYTES = 3 * (SH::A_TILE + SH::B_TILE);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t done[2];  // the MMAs of k-blocks 0, 2, ... / 1, 3, ... completed
  __shared__ uint32_t tmem_slot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint32_t ranks = 1, rank = 0;
  if constexpr (SPLIT) {
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  }
  uint32_t m0, n0;
  {
    // tiles in groups of group_m tile rows (see gemm_3xbf16_kernel)
    const uint32_t tile = blockIdx.x / ranks, tiles_m = gridDim.x / ranks / g.tiles_n, per_group = g.group_m * g.tiles_n;
    const uint32_t grp = tile / per_group, r = tile % per_group, first = grp * g.group_m;
    const uint32_t rows = tiles_m - first < g.group_m ? tiles_m - first : g.group_m;
    m0 = (first + r % rows) * BM;
    n0 = (r / rows) * 128u;
  }
  const uint32_t all_k = (g.K + 63u) / 64u, k0 = all_k * rank / ranks, nk = all_k * (rank + 1) / ranks - k0;
  if (threadIdx.x == 0) {
    for (int a = 0; a < 2; ++a)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&done[a])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&tmem_slot)), "r"(SH::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  dependency_wait();
  const bool vec = (g.K % 4u) == 0u;
  const bool vec_a = vec && (reinterpret_cast<uintptr_t>(g.a.x) & 15u) == 0,
             vec_b = vec && (reinterpret_cast<uintptr_t>(g.b.x) & 15u) == 0;
  float xa[kFusedChunks][8], xb[kFusedChunks][8];
  fused_load(g.a, g.K, m0, k0 * 64u, vec_a, xa);
  fused_load(g.b, g.K, n0, k0 * 64u, vec_b, xb);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  // warp w owns tensor-memory lanes 32 * (w % 4) .. (rows) and columns kFusedCols * (w / 4) ..
  const int q = warp & 3, h = warp >> 2;
  float sum[kFusedCols];
#pragma unroll
  for (int j = 0; j < kFusedCols; ++j) sum[j] = 0.0f;
  bool ok = true;
  auto drain = [&](uint32_t kb) {  // adds k-block kb's products to the sums
    const uint32_t a = kb & 1u;
    if (ok && !mbar_wait(smem_u32(&done[a]), (kb >> 1) & 1u, g.spin_limit)) {
      ok = false;
      if (lane == 0) raise(g.err);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int c = 0; c < kFusedCols / 32; ++c) {
      uint32_t r[32];
      tmem_load32(tmem + ((uint32_t)(q * 32) << 16) + a * 128u + (uint32_t)(h * kFusedCols + c * 32), r);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; ++j) sum[c * 32 + j] += __uint_as_float(r[j]);
    }
  };
  for (uint32_t kb = 0; kb < nk; ++kb) {
    // Stage and accumulator kb % 2 were last used for k-block kb - 2, whose
    // MMAs this thread has seen complete (drain).
    const uint32_t stage = base + (kb & 1u) * STAGE_BYTES;
    fused_store(g.a.kmajor, xa, stage);
    fused_store(g.b.kmajor, xb, stage + 3 * SH::A_TILE);
    if (kb + 1 < nk) {
      fused_load(g.a, g.K, m0, (k0 + kb + 1) * 64u, vec_a, xa);
      fused_load(g.b, g.K, n0, (k0 + kb + 1) * 64u, vec_b, xb);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};  // smallest first
#pragma unroll
      for (int p = 0; p < 6; ++p) {
        const uint64_t ad = smem_desc<SH>(stage + (uint32_t)pa[p] * SH::A_TILE);
        const uint64_t bd = smem_desc<SH>(stage + (uint32_t)(3 * SH::A_TILE + pb[p] * SH::B_TILE));
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint32_t acc = p > 0 || ks > 0 ? 1u : 0u;
          asm volatile(
              "{ .reg .pred p; setp.ne.b32 p, %4, 0;"
              " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
              :: "r"(tmem + (kb & 1u) * 128u), "l"(ad + (uint64_t)(ks * 2)), "l"(bd + (uint64_t)(ks * 2)),
                 "r"(SH::IDESC), "r"(acc)
              : "memory");
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                   :: "r"(smem_u32(&done[kb & 1u])) : "memory");
    }
    __syncwarp();
    if (kb > 0) drain(kb - 1);
  }
  if (nk > 0) drain(nk - 1);

  // the sums through shared memory: no MMA reads the stages any more (after a
  // wait that gave up, another one is made: the status says the outputs are void)
  if (!ok) mbar_wait(smem_u32(&done[(nk - 1) & 1u]), ((nk - 1) >> 1) & 1u, g.spin_limit);
  __syncwarp();
  const uint32_t r = (uint32_t)(q * 32 + lane);
#pragma unroll
  for (int c = 0; c < kFusedCols / 4; ++c)
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};"
                 :: "r"(base + r * 512u + (((uint32_t)(h * (kFusedCols / 4) + c) ^ (r & 31u)) * 16u)), "f"(sum[c * 4]),
                    "f"(sum[c * 4 + 1]), "f"(sum[c * 4 + 2]), "f"(sum[c * 4 + 3])
                 : "memory");
  __syncthreads();
  if constexpr (SPLIT) cluster_sync();
  store_sums<kFusedThreads>(base, ranks, rank, m0, n0, g.M, g.N, g.P);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (SPLIT) cluster_sync();  // no block leaves while another may still read its sums
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(SH::TMEM_COLS) : "memory");
  }
}

inline uint32_t round_up(uint32_t v, uint32_t m) { return (v + m - 1) / m * m; }

}  // namespace tc

size_t allpairs_tc_scratch_bytes(uint32_t M, uint32_t N, uint32_t K, int parts) {
  const uint64_t Mp = tc::round_up(M, tc::MPAD), Np = tc::round_up(N, tc::NPAD),
                 Kp = tc::round_up(K, tc::KPAD);
  return (size_t)parts * (Mp + Np) * Kp * 2 + 1024;
}

bool allpairs_tc_supported(uint32_t M, uint32_t N, uint32_t K, const void*, const void*,
                           const void*) {
  // the split arrays' row pitch (Kp * 2 bytes) and plane sizes stay far below
  // the tensor-map limits for any 32-bit shape; tiny products are not worth
  // the split
  return (uint64_t)M * N >= 128ull * 128ull && K >= 16 && rt().cc_major == 10;
}

static int encode_parts(CUtensorMap* tm, const void* base, uint64_t rows, uint64_t Kp, int parts,
                        uint32_t box_rows, uint32_t box_k) {
  cuuint64_t dims[3] = {Kp, rows, (cuuint64_t)parts};
  cuuint64_t strides[2] = {Kp * 2, rows * Kp * 2};
  cuuint32_t box[3] = {box_k, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = rt().drv.cuTensorMapEncodeTiled(
      tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
      box_k == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cu_fail(r, "cuTensorMapEncodeTiled(split parts)");
  return SCL_OK;
}

namespace {
// Blocks that share an output tile of 128 x 128 (a cluster): as many as leave
// no SM without a block, with at least four k-blocks of 64 each.  Splitting
// the operands included, with one block per tile and so: 1000 x 500 x 1100 (72
// tiles on 152 SMs) 16.5 -> 15.9 us, 1000 x 1100 x 500 (32 tiles) 27.9 -> 16.3
// us, 64 x 4096 x 512 (4 tiles) 72.9 -> 19.0 us; 256 x 256 x 256 with two
// k-blocks each 11.2 -> 12.1 us.
uint32_t split_of_k(uint64_t tiles, uint32_t Kp) {
  const uint64_t sms = sm_count();
  uint32_t s = 1;
  while (s < 8 && tiles * s * 2 <= sms && Kp / 64 >= 8 * s) s *= 2;
  return s;
}

template <int PARTS, int STAGES, int G, int BN_T>
cudaError_t launch_gemm(dim3 grid, cudaStream_t stream, const CUtensorMap& tmA, const CUtensorMap& tmB,
                        float* P, uint32_t M, uint32_t N, uint32_t Kp, uint32_t spin_limit,
                        unsigned int* err, uint32_t tiles_n, uint32_t group_m) {
  using SH = tc::Shape<BN_T>;
  const size_t smem = (size_t)STAGES * PARTS * (SH::A_TILE + SH::B_TILE) + 1024;
  return launch_overlapped(tc::gemm_3xbf16_kernel<PARTS, STAGES, G, BN_T>, grid, dim3(SH::THREADS), smem, stream,
                           tmA, tmB, P, M, N, Kp, spin_limit, err, tiles_n, group_m);
}

// Both operands' split descriptors for planes of `parts` parts from `scratch`
// (1024-aligned inside it).
struct Split {
  uint32_t Mp, Np, Kp;
  tc::Operand a, b;
};
Split split_of(const float* A, const float* B, uint32_t M, uint32_t N, uint32_t K, int parts, int trans,
               void* scratch) {
  Split s;
  s.Mp = tc::round_up(M, tc::MPAD);
  s.Np = tc::round_up(N, tc::NPAD);
  s.Kp = tc::round_up(K, tc::KPAD);
  __nv_bfloat16* base = reinterpret_cast<__nv_bfloat16*>(((uintptr_t)scratch + 1023) & ~(uintptr_t)1023);
  s.a = {A, base, M, s.Mp, (trans & 1) ? 0 : 1};
  s.b = {B, base + (size_t)parts * s.Mp * s.Kp, N, s.Np, (trans & 2) ? 1 : 0};
  return s;
}
// k of a tile of the split pass: 64 (more blocks an SM, and none half empty where
// Kp is an odd number of 64s), but 128 for operands of over 2^25 elements, whose
// stores go to memory and want to be long.  us of a call, 128 / 64: 2000 x K x
// 2000 K = 64 10.8 / 10.0, 1000 39.0 / 37.6; 1 x K x 62000 K = 16 18.5 / 14.9, 192
// 41.3 / 37.7, 4096 664 / 680; 100 x 4096 x 39680 518 / 533.
uint32_t split_depth(const Split& s) {
  const uint64_t elements = ((uint64_t)s.a.rows + s.b.rows) * s.Kp;
  return elements < (1ull << 25) || (s.Kp % 128 == 64 && s.Kp <= 320) ? 64 : 128;
}
cudaError_t launch_split(const Split& s, uint32_t K, int parts, cudaStream_t stream) {
  const uint32_t depth = split_depth(s);
  const uint64_t tiles = (uint64_t)((s.a.rows + 63) / 64 + (s.b.rows + 63) / 64) * ((s.Kp + depth - 1) / depth);
  return launch_overlapped(depth == 64 ? tc::split_kernel<64> : tc::split_kernel<128>,
                           dim3((unsigned)std::min<uint64_t>(tiles, 0x7fffffffull)), dim3(256), 0, stream, s.a, s.b, K,
                           s.Kp, parts);
}

// The output tiles (rows x cols each), numbered in groups of tile rows; the
// default is a group whose rows of A and columns of B for one wave of one
// block per SM fit in L2 together.
struct Tiles {
  uint32_t m, n, group;
};
int tiles_of(uint32_t M, uint32_t N, uint32_t rows, uint32_t cols, uint32_t group_rows, Tiles* t) {
  const uint64_t tn = ((uint64_t)N + cols - 1) / cols, tm = ((uint64_t)M + rows - 1) / rows;
  if (tn * tm * (rows / tc::BM) > 0x7fffffffull) return fail(SCL_ERR_ARG, "tensor-core AllPairs: too many output tiles");
  uint32_t g = (group_rows ? group_rows : 16) / (rows / tc::BM);
  if (g < 1) g = 1;
  if (g > tm) g = (uint32_t)tm;
  *t = {(uint32_t)tm, (uint32_t)tn, g};
  return SCL_OK;
}
}  // namespace

// bf16 parts: `parts` 3 (six products) or 2 (three), each drained every
// `drain` k-blocks.
int allpairs_tc_launch(const float* A, const float* B, float* P, uint32_t M, uint32_t N,
                       uint32_t K, int parts, int trans, int drain, int wide, uint32_t group_rows,
                       void* scratch, size_t scratch_bytes, cudaStream_t stream, uint32_t spin_limit,
                       unsigned int* err) {
  if (parts != 2 && parts != 3) return fail(SCL_ERR_ARG, "3xBF16: parts must be 2 or 3");
  if (scratch_bytes < allpairs_tc_scratch_bytes(M, N, K, parts))
    return fail(SCL_ERR_ARG, "3xBF16: scratch too small");
  const Split sp = split_of(A, B, M, N, K, parts, trans, scratch);
  const uint32_t Kp = sp.Kp;
  const uint32_t bn = wide ? 256 : 128, bk = wide ? 32 : 64;
  Tiles tiles;
  if (int st = tiles_of(M, N, tc::BM, bn, group_rows, &tiles)) return st;
  const dim3 grid(tiles.m * tiles.n);
  const uint32_t tn = tiles.n, group_m = tiles.group;
  alignas(64) CUtensorMap tmA, tmB;
  if (int st = encode_parts(&tmA, sp.a.out, sp.Mp, Kp, parts, tc::BM, bk)) return st;
  if (int st = encode_parts(&tmB, sp.b.out, sp.Np, Kp, parts, bn, bk)) return st;
  cudaError_t e = launch_split(sp, K, parts, stream);
  if (e != cudaSuccess) return cuda_fail(e, "split launch");
  if (wide) {
    // 128 x 256 tiles, k-blocks of 32: drains every 2 k-blocks (64 K, as the
    // narrow shape's default); parts 3: 3 stages of 72 KB; parts 2: 4 of 48 KB
    e = parts == 3 ? launch_gemm<3, 3, 2, 256>(grid, stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m)
                   : launch_gemm<2, 4, 2, 256>(grid, stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m);
  } else if (parts == 3) {
    // parts 3: 2 stages of 96 KB; parts 2: 3 stages of 64 KB
    const uint32_t split = drain >= 2 ? 1 : split_of_k(grid.x, Kp);
    e = drain >= 4  ? launch_gemm<3, 2, 4, 128>(grid, stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m)
      : drain == 2  ? launch_gemm<3, 2, 2, 128>(grid, stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m)
      : split == 1  ? launch_gemm<3, 2, 1, 128>(grid, stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m)
                    : launch_clustered(tc::gemm_3xbf16_kernel<3, 2, 1, 128, true>, split, dim3(grid.x * split),
                                       dim3(tc::Shape<128>::THREADS),
                                       (size_t)2 * 3 * (tc::Shape<128>::A_TILE + tc::Shape<128>::B_TILE) + 1024,
                                       stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m);
  } else {
    e = drain >= 4 ? launch_gemm<2, 3, 4, 128>(grid, stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m)
      : drain == 2 ? launch_gemm<2, 3, 2, 128>(grid, stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m)
                   : launch_gemm<2, 3, 1, 128>(grid, stream, tmA, tmB, P, M, N, Kp, spin_limit, err, tn, group_m);
  }
  if (e != cudaSuccess) return cuda_fail(e, "3xBF16 launch");
  return SCL_OK;
}

namespace {
// CTA pairs the device holds at once.
uint64_t resident_pairs() {
  int n = rt().pair_clusters;
  if (n == 0) {
    const int half = (int)(sm_count() / 2);
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(2 * half));
    cfg.blockDim = dim3(tc::kPairThreads);
    cfg.dynamicSmemBytes = tc::kPairSmem;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(tc::gemm_pair_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)tc::kPairSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, tc::gemm_pair_kernel<true, false>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = half;
    }
    rt().pair_clusters = n;
  }
  return (uint64_t)n;
}
}  // namespace

namespace {
// While a tile has few k-blocks, its start and its way out weigh more than its
// products: each pair then walks over the tiles.  us, one tile per pair and
// walking: 8192 x K x 8192 K = 64 124 / 64, 512 298 / 248, 1000 519 / 482, 2500
// 1193 / 1178, 4096 1853 / 1904 (dealt out in advance, the tiles do not follow
// the pairs' speeds); 2600 x K x 4000 K = 512 65.9 / 56.5, 1500 156 / 147; 2600 x
// 3000 x 20000 1191 / 1216.
bool pair_walks(uint64_t tiles, uint32_t Kp) { return Kp <= 2560 && tiles > resident_pairs(); }
}  // namespace

// One wave of 128 x 128 tiles (or of clusters that share one), few k-blocks a
// block: the operands split where they are used (gemm_fused_kernel).
bool allpairs_fused_wins(uint32_t M, uint32_t N, uint32_t K, int trans) {
  const uint64_t sms = sm_count();
  const uint64_t tiles = (uint64_t)((M + 127) / 128) * ((N + 127) / 128);
  const uint32_t all_k = (K + 63) / 64, split = split_of_k(tiles, tc::round_up(K, tc::KPAD));
  const bool strided = trans == 1;  // both operands
  return tiles <= sms && (all_k + split - 1) / split <= (strided ? 3u : 4u);
}
int allpairs_fused_launch(const float* A, const float* B, float* P, uint32_t M, uint32_t N, uint32_t K, int trans,
                          uint32_t group_rows, cudaStream_t stream, uint32_t spin_limit, unsigned int* err) {
  Tiles tiles;
  if (int st = tiles_of(M, N, tc::BM, 128, group_rows, &tiles)) return st;
  const tc::Fused args = {{A, nullptr, M, M, (trans & 1) ? 0 : 1},
                          {B, nullptr, N, N, (trans & 2) ? 1 : 0},
                          P, err, M, N, K, spin_limit, tiles.n, tiles.group};
  const uint32_t split = split_of_k((uint64_t)tiles.m * tiles.n, tc::round_up(K, tc::KPAD));
  const dim3 grid(tiles.m * tiles.n * split);
  const size_t smem = (size_t)2 * 3 * (tc::Shape<128>::A_TILE + tc::Shape<128>::B_TILE) + 1024;
  const cudaError_t e =
      split == 1 ? launch_overlapped(tc::gemm_fused_kernel<false>, grid, dim3(tc::kFusedThreads), smem, stream, args)
                 : launch_clustered(tc::gemm_fused_kernel<true>, split, grid, dim3(tc::kFusedThreads), smem, stream, args);
  if (e != cudaSuccess) return cuda_fail(e, "tensor-core AllPairs launch");
  return SCL_OK;
}

// CTA pairs, three bf16 parts.  `small`: the products in the order of 128-column
// tiles, else of 256-column ones.
int allpairs_pair_launch(const float* A, const float* B, float* P, uint32_t M, uint32_t N, uint32_t K, int trans,
                         bool small, uint32_t group_rows, void* scratch, size_t scratch_bytes, cudaStream_t stream,
                         uint32_t spin_limit, unsigned int* err) {
  if (scratch_bytes < allpairs_tc_scratch_bytes(M, N, K, 3))
    return fail(SCL_ERR_ARG, "tensor-core AllPairs: scratch too small");
  const Split sp = split_of(A, B, M, N, K, 3, trans, scratch);
  const uint32_t Kp = sp.Kp;
  Tiles tiles;
  if (int st = tiles_of(M, N, 2 * tc::BM, tc::kPairCols, group_rows, &tiles)) return st;
  alignas(64) CUtensorMap tmA, tmB;
  if (int st = encode_parts(&tmA, sp.a.out, sp.Mp, Kp, 3, tc::BM, 32)) return st;
  if (int st = encode_parts(&tmB, sp.b.out, sp.Np, Kp, 3, 128, 32)) return st;
  cudaError_t e = launch_split(sp, K, 3, stream);
  if (e != cudaSuccess) return cuda_fail(e, "split launch");
  const tc::PairArgs args = {P, err, M, N, Kp, spin_limit, tiles.n, tiles.m, tiles.group};
  const uint64_t all = (uint64_t)tiles.m * tiles.n;
  const bool walk = !small && pair_walks(all, Kp);
  e = launch_overlapped(small  ? tc::gemm_pair_kernel<false, true>
                        : walk ? tc::gemm_pair_kernel<true, false>
                               : tc::gemm_pair_kernel<false, false>,
                        dim3((unsigned)(2 * (walk ? resident_pairs() : all))), dim3(tc::kPairThreads), tc::kPairSmem,
                        stream, tmA, tmB, args);
  if (e != cudaSuccess) return cuda_fail(e, "tensor-core AllPairs launch");
  return SCL_OK;
}

// Whether CTA pairs take the place of 128 x 128 tiles: where those take two
// waves of the SMs and 256 x 256 tiles one of the pairs.  A k-block of 64 takes
// 1.2 us in the former (its 96 KB per SM come at 12 TB/s, from L2) and 1.9 us in
// the latter, for twice the outputs per SM, with the same products in the same
// order and so the same bits.  us, 128 x 128 tiles and so, the split included:
// 2000 x K x 2000 K = 64 15.3 / 11.9, 500 32.1 / 24.8, 2000 90.1 / 71.8, 4000
// 166 / 132; 300 x 1000 x 8000 55.8 / 47.3.
bool allpairs_pair_replaces_small(uint32_t M, uint32_t N) {
  const uint64_t sms = sm_count(), pairs = resident_pairs();
  const uint64_t small = (uint64_t)((M + 127) / 128) * ((N + 127) / 128);
  const uint64_t large = (uint64_t)((M + 255) / 256) * ((N + 255) / 256);
  return small > sms && large <= pairs;
}

// ... and of 128 x 256 tiles: nearly always.  us, 128 x 256 tiles and so, the
// split included: 8192 x K x 8192 K = 64 167 / 64, 256 247 / 132, 1000 575 /
// 482, 4096 2072 / 1902; 2560 x 512 x 2048 48.3 / 39.9; 4000 x 1000 x 3000 121 /
// 104; 2500 x 1000 x 2305 109 / 75.  Not where the pairs' 256 rows hold so much
// more padding that it shows: as rows take more pair tiles for their wide ones,
// 1100 x K x 20000 (1.11) K = 512 139 / 113, 1500 321 / 320, 3000 604 / 618; 300
// x K x 60000 (1.33) K = 256 113 / 92, 1500 405 / 437; 128 x K x 100000 (2) K =
// 64 55 / 47, 512 171 / 180, 3000 821 / 978.  With as many waves the padding
// costs nothing: 640 x 1500 x 7936 124 / 110.  A few rows write next to nothing,
// and what is left is the pairs' start: 1 x 50 x 62000 20.7 / 23.7, 100 x 128 x
// 39680 32.2 / 28.3.
bool allpairs_pair_replaces_wide(uint32_t M, uint32_t N, uint32_t K) {
  const uint64_t sms = sm_count(), pairs = resident_pairs();
  const uint64_t wide = (uint64_t)((M + 127) / 128) * ((N + 255) / 256);
  const uint64_t large = (uint64_t)((M + 255) / 256) * ((N + 255) / 256);
  if ((K <= 128 && M >= 100) || (K <= 256 && 3 * large <= 2 * wide)) return true;
  return 20 * large <= 11 * wide || (large + pairs - 1) / pairs <= (wide + sms - 1) / sms;
}

}  // namespace scl

using namespace scl;

extern "C" int scl_debug_allpairs_split(const float* A, const float* B, uint32_t M, uint32_t N,
                                        uint32_t K, int parts, int trans, void* scratch,
                                        size_t scratch_bytes, size_t* needed) {
  if (parts != 2 && parts != 3) return fail(SCL_ERR_ARG, "split: parts must be 2 or 3");
  const size_t need = allpairs_tc_scratch_bytes(M, N, K, parts);
  if (needed) *needed = need;
  if (!scratch) return SCL_OK;
  if (int st = require_init()) return st;
  if (!A || !B || scratch_bytes < need) return fail(SCL_ERR_ARG, "split: null operand or scratch too small");
  const Split sp = split_of(A, B, M, N, K, parts, trans, scratch);
  SCL_CUDA(launch_split(sp, K, parts, rt().stream));
  return SCL_OK;
}
