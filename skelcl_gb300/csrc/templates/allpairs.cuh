// ---------------------------------------------------------------------------
// AllPairs for sm_103a on CUDA cores.
//
// SCL_KIND 12 (Reduce + Zip pair, include/SkelCL/detail/AllPairsKernel.cl:47-135):
//   P[i][j] = id (+) z(A[i][0],B[0][j]) (+) ... (+) z(A[i][K-1],B[K-1][j])
// folded strictly in k order (AllPairsKernel.cl:89-91); the right operand is
// K x N row-major (AllPairsKernel.cl:72).  Extra arguments: the Reduce's
// first, then the Zip's (AllPairsDef.h:265-269).
// Shape: BM x BN outputs per block, TM x TN accumulators per thread, k-tiles
// copied into a ring in shared memory with cp.async.  Unlike the reference, P
// is written once (the reference re-reads and re-writes P every 32-wide k
// segment, AllPairsKernel.cl:77-78,95-96).
// A fold runs along k in one thread, so a block's time is that of its K steps
// whatever the size of the output: small outputs are bound by how many blocks
// share them and by a step's latency, large ones by the arithmetic (FP32: two
// instructions per pair of |x - y| and +).  Hence four tiles, chosen by the
// number of blocks (scl_launch_allpairs).  us against one tile of 128 x 128
// with register prefetch: |x - y|, K = 255 97 x 97 46.7 -> 5.9, 500 x 500
// 46.7 -> 11.4, 1001 x 1001 51 -> 30, 2700 x 2700 170 -> 144, 4096 x 4096 (K =
// 256) 289 -> 287 (bound by issue; 3.8 % of it the last wave); double x * y,
// K = 128 97 x 97 517 -> 10.6, 1400 x 1400 524 -> 417, 3000 x 3000 2086 ->
// 1876 (FP64 pipe: 1840).
//
// SCL_KIND 13 (user f(lmatrix_t*, rmatrix_t*, dim, ...),
// include/SkelCL/detail/AllPairsKernel2.cl:42-65): one output per thread in
// 16 x 16 blocks; when 16 rows of A and 16 columns of B fit in shared memory
// they are staged there and the accessors read the staged copies.
// ---------------------------------------------------------------------------
#if SCL_KIND == 12
typedef SCL_TYPE_0 scl_L;
typedef SCL_TYPE_1 scl_Rt;
typedef SCL_TYPE_2 scl_O;

template <typename T> struct scl_ap_real { static constexpr bool value = false; };
template <> struct scl_ap_real<float> { static constexpr bool value = true; };
template <> struct scl_ap_real<double> { static constexpr bool value = true; };

// BYTES to shared memory, complete after cp.async.wait_group.
template <int BYTES>
__device__ __forceinline__ void scl_ap_copy(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;"
               :: "r"((unsigned int)__cvta_generic_to_shared(dst)), "l"(src), "n"(BYTES) : "memory");
}

// k-tiles of BK4 in STAGES buffers, BK4 / 2 where an operand is wider than 4
// bytes.  Thread (tx, ty) owns groups of four (or all) consecutive rows and
// columns, the groups spread over the tile: its shared-memory reads are
// 16-byte loads that a warp spreads over all banks.  The block's tile is
// blockIdx.x in rows of tiles_n.
template <int BM, int BN, int TM, int TN, int BK4, int STAGES, int PER_SM>
__global__ void __launch_bounds__(BM / TM * (BN / TN), PER_SM)
scl_allpairs_simt(const scl_L* A, const scl_Rt* B, scl_O* P, unsigned int M, unsigned int N,
                  unsigned int K, unsigned int tiles_n, int vec_b SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  // operands are scalars (a zero of each is well-formed): vector types, which sit
  // on the size of their components, would want other copies
  static_assert(sizeof((scl_L)0) + sizeof((scl_Rt)0) > 0, "AllPairs: scalar operands");
  // wider values take tiles of at most four outputs per thread
  if constexpr (TM * TN > 4 && (sizeof(scl_L) > 4 || sizeof(scl_Rt) > 4 || sizeof(scl_O) > 4)) return;
  constexpr int BK = sizeof(scl_L) <= 4 && sizeof(scl_Rt) <= 4 ? BK4 : BK4 / 2;
  constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
  constexpr int VA = TM < 4 ? TM : 4, VB = TN < 4 ? TN : 4;
  constexpr bool ASYNC = (sizeof(scl_L) == 4 || sizeof(scl_L) == 8) && (sizeof(scl_Rt) == 4 || sizeof(scl_Rt) == 8);
  constexpr int AHEAD = ASYNC ? STAGES - 1 : 1;
  constexpr int LDA = BM + 4;  // (the transposed stores of A meet two to a bank)
  // 8 x 8 accumulators: 64 x 128 of |x - y| at 4096 x 256 x 4096 307 us with all
  // 16 steps unrolled, 287 with four; int x * y at 4001 x 255 x 4001 264 and 269
  constexpr int UNR = TM == 8 && scl_ap_real<scl_O>::value ? 4 : BK;
  constexpr int TAIL = TM * TN >= 32 ? 1 : 4;
  __shared__ __align__(16) scl_L As[STAGES][BK][LDA];
  __shared__ __align__(16) scl_Rt Bs[STAGES][BK][BN];
  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;
  const unsigned int m0 = blockIdx.x / tiles_n * BM, n0 = blockIdx.x % tiles_n * BN;
  // global -> shared: a thread brings A[row ra + i * RS][k ka] and
  // B[k kb + i * KS][column cb]; rows and columns past the matrix are read from
  // its last, for outputs that are not stored, and k past K are left out
  static_assert(THREADS % BK == 0 && THREADS % BN == 0, "");
  constexpr int RS = THREADS / BK, AE = BM / RS, KS = THREADS / BN, BE = BK / KS, KSV = THREADS / (BN / 4);
  const int ra = tid / BK, ka = tid % BK;
  const bool rows_in = m0 + BM <= M;
  scl_L va[ASYNC ? 1 : AE];
  scl_Rt vb[ASYNC ? 1 : BE];
  auto fetch = [&](unsigned int kt) {
    const unsigned int k0 = kt * BK;
    const int buf = (int)(kt % STAGES);
    if (k0 + ka < K) {
      const scl_L* src = A + (scl_u64)(m0 + ra) * K + (k0 + ka);
#pragma unroll
      for (int i = 0; i < AE; ++i) {
        if (!rows_in) src = A + (scl_u64)min(m0 + ra + i * RS, M - 1) * K + (k0 + ka);
        if constexpr (ASYNC) scl_ap_copy<(int)sizeof(scl_L)>(&As[buf][ka][ra + i * RS], src);
        else va[i] = *src;
        src += (scl_u64)RS * K;
      }
    }
    if constexpr (ASYNC && sizeof(scl_Rt) == 4) {
      if (vec_b) {
        const int c = tid % (BN / 4) * 4, k = tid / (BN / 4);
        const scl_Rt* src = B + (scl_u64)(k0 + k) * N + (n0 + c < N ? n0 + c : 0);
#pragma unroll
        for (int i = 0; i < (BK + KSV - 1) / KSV; ++i, src += (scl_u64)KSV * N)
          if (k + i * KSV < BK && k0 + k + i * KSV < K) scl_ap_copy<16>(&Bs[buf][k + i * KSV][c], src);
        return;
      }
    }
    const int cb = tid % BN, kb = tid / BN;
    const scl_Rt* src = B + (scl_u64)(k0 + kb) * N + min(n0 + cb, N - 1);
#pragma unroll
    for (int i = 0; i < BE; ++i, src += (scl_u64)KS * N) {
      if (k0 + kb + i * KS < K) {
        if constexpr (ASYNC) scl_ap_copy<(int)sizeof(scl_Rt)>(&Bs[buf][kb + i * KS][cb], src);
        else vb[i] = *src;
      }
    }
  };
  auto put = [&](unsigned int kt) {
    if constexpr (!ASYNC) {
      const int buf = (int)(kt % STAGES);
#pragma unroll
      for (int i = 0; i < AE; ++i) As[buf][ka][ra + i * RS] = va[i];
#pragma unroll
      for (int i = 0; i < BE; ++i) Bs[buf][tid / BN + i * KS][tid % BN] = vb[i];
    }
  };
  auto commit = [&]() {
    if constexpr (ASYNC) asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto step = [&](scl_O (&acc)[TM][TN], int cur, int kk) {
    scl_L a[TM];
    scl_Rt b[TN];
#pragma unroll
    for (int g = 0; g < TM / VA; ++g) {
      const scl_pack<scl_L, VA> q = scl_load<scl_L, VA>(&As[cur][kk][g * (BM / (TM / VA)) + ty * VA]);
#pragma unroll
      for (int i = 0; i < VA; ++i) a[g * VA + i] = q.v[i];
    }
#pragma unroll
    for (int g = 0; g < TN / VB; ++g) {
      const scl_pack<scl_Rt, VB> q = scl_load<scl_Rt, VB>(&Bs[cur][kk][g * (BN / (TN / VB)) + tx * VB]);
#pragma unroll
      for (int i = 0; i < VB; ++i) b[g * VB + i] = q.v[i];
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
        acc[i][j] = USR_REDUCE(acc[i][j], USR_ZIP(a[i], b[j] SCL_ZIP_ARGS) SCL_REDUCE_ARGS);
  };

  scl_O acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = (scl_O)(SCL_IDENTITY);

  const unsigned int ktiles = (K + BK - 1) / BK;
#pragma unroll
  for (int t = 0; t < AHEAD; ++t) {
    if (t < ktiles) {
      fetch(t);
      put(t);
    }
    commit();
  }
  for (unsigned int kt = 0; kt < ktiles; ++kt) {
    if constexpr (ASYNC) asm volatile("cp.async.wait_group %0;" :: "n"(AHEAD - 1) : "memory");
    __syncthreads();
    if (kt + AHEAD < ktiles) fetch(kt + AHEAD);
    commit();
    const int cur = (int)(kt % STAGES);
    const unsigned int kmax = min((unsigned int)BK, K - kt * BK);
    if (kmax == BK) {
#pragma unroll UNR
      for (int kk = 0; kk < BK; ++kk) step(acc, cur, kk);
    } else {
#pragma unroll TAIL
      for (unsigned int kk = 0; kk < kmax; ++kk) step(acc, cur, (int)kk);
    }
    if (kt + AHEAD < ktiles) put(kt + AHEAD);
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const unsigned int gm = m0 + (i / VA) * (BM / (TM / VA)) + ty * VA + i % VA;
    if (gm >= M) continue;
#pragma unroll
    for (int h = 0; h < TN / VB; ++h) {
      const unsigned int gn = n0 + h * (BN / (TN / VB)) + tx * VB;
      scl_O* dst = P + (scl_u64)gm * N + gn;
      if (sizeof(scl_O) == 4 && (N % VB) == 0 && gn + VB - 1 < N && (((scl_u64)dst) & (VB * 4 - 1u)) == 0) {
        scl_pack<scl_O, VB> o;
#pragma unroll
        for (int j = 0; j < VB; ++j) o.v[j] = acc[i][h * VB + j];
        scl_store<scl_O, VB>(dst, o);
      } else {
#pragma unroll
        for (int j = 0; j < VB; ++j)
          if (gn + j < N) dst[j] = acc[i][h * VB + j];
      }
    }
  }
}

#elif SCL_KIND == 13
extern "C" __global__ void __launch_bounds__(256)
scl_allpairs_generic(const SCL_TYPE_0* A, const SCL_TYPE_1* B, SCL_TYPE_2* P,
                     unsigned int dimension, unsigned int height, unsigned int width,
                     int staged SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  const unsigned int col = blockIdx.x * 16 + threadIdx.x;
  const unsigned int row = blockIdx.y * 16 + threadIdx.y;
  SCL_TYPE_0* As = reinterpret_cast<SCL_TYPE_0*>(scl_dyn_smem);
  SCL_TYPE_1* Bs = reinterpret_cast<SCL_TYPE_1*>(
      scl_dyn_smem + (((size_t)16 * dimension * sizeof(SCL_TYPE_0) + 15) & ~(size_t)15));
  lmatrix_t Mm;
  Mm.data = A;
  Mm.dimension = dimension;
  Mm.row = row;
  rmatrix_t Nm;
  Nm.data = B;
  Nm.width = width;
  Nm.column = col;
  if (staged) {
    const int t = threadIdx.y * 16 + threadIdx.x;
    const unsigned int r0 = blockIdx.y * 16, c0 = blockIdx.x * 16;
    for (unsigned int k = t; k < 16u * dimension; k += 256) {
      const unsigned int rr = k / dimension, kk = k % dimension;
      As[k] = (r0 + rr < height) ? A[(scl_u64)(r0 + rr) * dimension + kk] : (SCL_TYPE_0)0;
    }
    for (unsigned int k = t; k < 16u * dimension; k += 256) {
      const unsigned int kk = k / 16, cc = k % 16;
      Bs[k] = (c0 + cc < width) ? B[(scl_u64)kk * width + c0 + cc] : (SCL_TYPE_1)0;
    }
    __syncthreads();
    Mm.scl_row = As + (size_t)threadIdx.y * dimension;
    Nm.scl_col = Bs + threadIdx.x;
    Nm.scl_stride = 16;
  } else {
    Mm.scl_row = A + (scl_u64)row * dimension;
    Nm.scl_col = B + col;
    Nm.scl_stride = width;
  }
  if (row < height && col < width)
    P[(scl_u64)row * width + col] = USR_FUNC(&Mm, &Nm, dimension SCL_EXTRA_ARGS);
}
#endif
