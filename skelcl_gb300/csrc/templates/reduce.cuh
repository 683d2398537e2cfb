// ---------------------------------------------------------------------------
// Reduce for sm_103a: ONE launch.  Replaces the reference's two kernels
// SCL_REDUCE_1 (8192 work-items, strided fold) and SCL_REDUCE_2 (one work-group
// tree) of include/SkelCL/detail/ReduceKernel.cl:51-128 and
// include/SkelCL/detail/ReduceDef.h:98-245.
//
// Semantics kept from the reference:
//  * the identity is not used to seed the fold: every partial starts from a
//    real element (ReduceKernel.cl:60-61), so a non-neutral `id` string has
//    no effect, as in the reference;
//  * the operator is assumed associative and commutative (the reference folds
//    element j, j+8192, j+2*8192 ... and then a tree);
//  * the result is a one-element vector (ReduceDef.h:113-121).
// Empty input (the reference reads out of bounds there) yields SCL_IDENTITY.
//
// Shape: grid-stride 16-byte loads, per-thread fold in T, then warp-shuffle
// and block folds in the carry type SCL_CARRY_T (double for float element
// types: "cross-block carries in FP64"), one partial per block, and the last
// block to finish (atomic ticket) folds the partials in block order and
// resets the ticket for the next launch.
// ---------------------------------------------------------------------------

template <typename T>
__device__ __forceinline__ T scl_shfl_down(const T& v, int off) {
  constexpr int W = (int)((sizeof(T) + 3) / 4);
  unsigned int w[W];
  memcpy(w, &v, sizeof(T));
#pragma unroll
  for (int i = 0; i < W; ++i) w[i] = __shfl_down_sync(0xffffffffu, w[i], off);
  T r;
  memcpy(&r, w, sizeof(T));
  return r;
}
template <typename T>
__device__ __forceinline__ T scl_shfl_up(const T& v, int off) {
  constexpr int W = (int)((sizeof(T) + 3) / 4);
  unsigned int w[W];
  memcpy(w, &v, sizeof(T));
#pragma unroll
  for (int i = 0; i < W; ++i) w[i] = __shfl_up_sync(0xffffffffu, w[i], off);
  T r;
  memcpy(&r, w, sizeof(T));
  return r;
}
template <typename T>
__device__ __forceinline__ T scl_shfl_idx(const T& v, int src) {
  constexpr int W = (int)((sizeof(T) + 3) / 4);
  unsigned int w[W];
  memcpy(w, &v, sizeof(T));
#pragma unroll
  for (int i = 0; i < W; ++i) w[i] = __shfl_sync(0xffffffffu, w[i], src);
  T r;
  memcpy(&r, w, sizeof(T));
  return r;
}
// Coherent (L1-bypassing) copy of a value written by another block.
template <typename T>
__device__ __forceinline__ T scl_ld_cg(const T* p) {
  T r;
  if constexpr (sizeof(T) % 4 == 0) {
    unsigned int w[sizeof(T) / 4];
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 4); ++i)
      w[i] = *((const volatile unsigned int*)p + i);
    memcpy(&r, w, sizeof(T));
  } else {
    unsigned char b[sizeof(T)];
#pragma unroll
    for (int i = 0; i < (int)sizeof(T); ++i) b[i] = *((const volatile unsigned char*)p + i);
    memcpy(&r, b, sizeof(T));
  }
  return r;
}
template <typename T>
__device__ __forceinline__ void scl_st_cg(T* p, const T& v) {
  if constexpr (sizeof(T) % 4 == 0) {
    unsigned int w[sizeof(T) / 4];
    memcpy(w, &v, sizeof(T));
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 4); ++i) *((volatile unsigned int*)p + i) = w[i];
  } else {
    unsigned char b[sizeof(T)];
    memcpy(b, &v, sizeof(T));
#pragma unroll
    for (int i = 0; i < (int)sizeof(T); ++i) *((volatile unsigned char*)p + i) = b[i];
  }
}

#if SCL_KIND == 9 || SCL_KIND == 16
#if SCL_KIND == 16
typedef SCL_TYPE_2 scl_T;  // the zipped element type folded by the Reduce
#else
typedef SCL_TYPE_0 scl_T;
#endif
typedef SCL_CARRY_T scl_C;

// Fold (have, value) pairs across a warp; lane 0 ends with the warp's fold.
__device__ __forceinline__ void scl_warp_fold(bool& have, scl_C& c SCL_USER_PARAMS) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    scl_C o = scl_shfl_down(c, off);
    bool oh = __shfl_down_sync(0xffffffffu, have ? 1 : 0, off) != 0;
    if ((threadIdx.x & 31) + off < 32 && oh) {
      c = have ? (scl_C)SCL_FUNC_C(c, o SCL_OP_ARGS) : o;
      have = true;
    }
  }
}

// Block fold; the result is valid in thread 0.
__device__ __forceinline__ void scl_block_fold(bool& have, scl_C& c SCL_USER_PARAMS) {
  __shared__ scl_C s_val[32];
  __shared__ int s_have[32];
  scl_warp_fold(have, c SCL_EXTRA_ARGS);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  if (lane == 0) {
    s_val[warp] = c;
    s_have[warp] = have ? 1 : 0;
  }
  __syncthreads();
  if (warp == 0) {
    have = lane < nwarps && s_have[lane];
    if (have) c = s_val[lane];
    scl_warp_fold(have, c SCL_EXTRA_ARGS);
  }
  __syncthreads();
}

#if SCL_KIND == 9
template <int U>
__global__ void scl_reduce_k(const scl_T* in, scl_T* out, scl_u64 n, int aligned,
                             scl_C* partials, unsigned int* ticket,
                             unsigned int* err SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  constexpr int V = scl_vec_width<sizeof(scl_T)>::value;
  const scl_u64 tid = SCL_TID(), nth = SCL_NTH();
  if (n == 0) {
    if (tid == 0) out[0] = (scl_T)(SCL_IDENTITY);
    return;
  }
  const scl_u64 nvec = aligned ? n / V : 0;
  bool have = false;
  scl_T acc;
  scl_u64 j = tid;
  if (j < nvec) {
    scl_pack<scl_T, V> p = scl_load<scl_T, V>(in + j * V);
    acc = p.v[0];
#pragma unroll
    for (int e = 1; e < V; ++e) acc = SCL_FUNC(acc, p.v[e] SCL_OP_ARGS);
    have = true;
    j += nth;
  }
  for (; j < nvec; j += nth * U) {
    scl_pack<scl_T, V> a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const scl_u64 k = j + (scl_u64)u * nth;
      if (k < nvec) a[u] = scl_load<scl_T, V>(in + k * V);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const scl_u64 k = j + (scl_u64)u * nth;
      if (k < nvec) {
#pragma unroll
        for (int e = 0; e < V; ++e) acc = SCL_FUNC(acc, a[u].v[e] SCL_OP_ARGS);
      }
    }
  }
  for (scl_u64 i = nvec * V + tid; i < n; i += nth) {
    acc = have ? SCL_FUNC(acc, in[i] SCL_OP_ARGS) : in[i];
    have = true;
  }
  scl_C c;
  if (have) c = (scl_C)acc;
  scl_block_fold(have, c SCL_EXTRA_ARGS);

  if (gridDim.x == 1) {  // no other block's partials to wait for
    if (threadIdx.x == 0) out[0] = (scl_T)c;
    return;
  }
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    // every block holds at least one element (the host sizes the grid so)
    scl_st_cg(&partials[blockIdx.x], c);
    __threadfence();
    const unsigned int t = atomicAdd(ticket, 1u);
    s_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  have = false;
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
    scl_C v = scl_ld_cg(&partials[b]);
    c = have ? (scl_C)SCL_FUNC_C(c, v SCL_OP_ARGS) : v;
    have = true;
  }
  scl_block_fold(have, c SCL_EXTRA_ARGS);
  if (threadIdx.x == 0) {
    out[0] = (scl_T)c;
    *ticket = 0u;  // ready for the next launch on this workspace
  }
}

// Segments of at most short_max elements (empty ones included: SCL_IDENTITY):
// one warp each, warps striding over the segments (warp `wid` of `nw`), U
// elements per lane in flight, folded in the element type (no block boundary
// is crossed; FP64 folds here would make the FP64 pipe the bound for tiny
// segments); longer segments are left to the tiles.
template <int U>
__device__ __forceinline__ void scl_reduce_short_run(const scl_T* in, scl_T* out, const scl_u64* seg_off,
                                                     scl_u64 n_seg, scl_u64 short_max, scl_u64 wid,
                                                     scl_u64 nw SCL_USER_PARAMS) {
  const int lane = threadIdx.x & 31;
  scl_u64 sg = wid;
  // the next segment's offsets are loaded while this one is folded
  scl_u64 lo_next = sg < n_seg ? seg_off[sg] : 0, hi_next = sg < n_seg ? seg_off[sg + 1] : 0;
  for (; sg < n_seg; sg += nw) {
    const scl_u64 lo = lo_next;
    const scl_u64 len = hi_next > lo ? hi_next - lo : 0;
    if (sg + nw < n_seg) {
      lo_next = seg_off[sg + nw];
      hi_next = seg_off[sg + nw + 1];
    }
    if (len > short_max) continue;
    bool have = false;
    scl_T acc;
    for (scl_u64 b = 0; b < len; b += 32 * U) {
      scl_T v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const scl_u64 e = b + (scl_u64)(u * 32 + lane);
        if (e < len) v[u] = in[lo + e];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (b + (scl_u64)(u * 32 + lane) < len) {
          acc = have ? SCL_FUNC(acc, v[u] SCL_OP_ARGS) : v[u];
          have = true;
        }
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const scl_T o = scl_shfl_down(acc, off);
      const bool oh = __shfl_down_sync(0xffffffffu, have ? 1 : 0, off) != 0;
      if (lane + off < 32 && oh) {
        acc = have ? SCL_FUNC(acc, o SCL_OP_ARGS) : o;
        have = true;
      }
    }
    if (lane == 0) out[sg] = have ? acc : (scl_T)(SCL_IDENTITY);
  }
}

// The warp-per-segment kernel on its own (segmented launches without a
// segment plan; with one, scl_reduce_seg<R, 1> runs the same code in the
// blocks past the tiles).
template <int U>
__global__ void __launch_bounds__(256)
scl_reduce_short(const scl_T* in, scl_T* out, const scl_u64* seg_off, scl_u64 n_seg,
                 scl_u64 short_max SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  scl_reduce_short_run<U>(in, out, seg_off, n_seg, short_max,
                          ((scl_u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                          ((scl_u64)gridDim.x * blockDim.x) >> 5 SCL_EXTRA_ARGS);
}

// Window role of a planned segmented Reduce (the blocks past the tiles):
// block r takes window record r of the plan, {first vector, end vector,
// first element, elements}: consecutive vectors of at most short_max elements
// that start in one window of short_max elements (all but the last end
// inside it, so the record spans at most 2 * short_max = WT elements).  The
// record's elements are brought into shared memory by bulk asynchronous
// copies (element e0 + p at ts[p + shift]; bounded wait) while each thread
// reads its first vector's offsets.  Then every vector is folded by a group of
// G threads, G the power of two that gives the record's vectors all 256
// threads: thread l of the group folds elements l, l + G, ... (in four chains
// side by side where vectors are long or G is small: chains no longer than a
// warp's, or a quarter of a vector of up to 256), the group's folds combine in a
// shuffle tree (a strided fold and a tree, as in the flat reduce; the operator is
// taken to be commutative).  A long vector among so many that G < 8 is left to a
// warp: its few threads would hold up the block, and their chains round more
// often (20,000 vectors of 4000 floats beside 300 empty ones each 0.69 -> 0.08
// ms).  An empty vector yields SCL_IDENTITY.  Folds in the element type.  10^6
// vectors of 1..199 floats 0.143 -> 0.081 ms, 10^7 of 0..2 0.323 -> 0.041 ms,
// 3.3 * 10^5 of 200..399 0.134 -> 0.075 ms against a thread per vector of up to
// 256 elements (about 40 busy threads of a block's 256) and a warp per longer one.
// A warp takes each vector of a record that has at most eight (groups of two and
// more warps waited for one another: 10^5 vectors of 500..1499 floats 75.6 -> 64.7
// us, of doubles 69 -> 58 a fifth of it), and of one of up to 32 whose vectors
// are long (450 elements on average) or uneven (the longest over three times the
// average: 40,000 log-uniform of 1..4096 floats 20.4 -> 15.5 us, of shorts 18.8 ->
// 11.8; even ones of 200..399 floats 14.6 by groups, 15.3 by warps).
#define SCL_REDUCE_AHEAD (2 * SCL_SMS)
// A vector among many is long from here on.  (Of single bytes a record holds four
// times as many, and groups of few threads fold whole numbers as exactly as a
// warp: 32 % faster for vectors of 200..399.)
constexpr bool kWinBytes = sizeof(scl_T) == 1;
#define SCL_WIN_LONG (kWinBytes ? 512 : 256)
// Elements first, first + step, ... below n (first < n) of v, in four chains
// side by side.
__device__ __forceinline__ scl_T scl_fold_chains(const scl_T* v, int first, int n, int step SCL_USER_PARAMS) {
  scl_T acc = v[first];
  int e = first + step;
  if (e + 2 * step < n) {
    scl_T c1 = v[e], c2 = v[e + step], c3 = v[e + 2 * step];
    for (e += 3 * step; e + 3 * step < n; e += 4 * step) {
      acc = SCL_FUNC(acc, v[e] SCL_OP_ARGS);
      c1 = SCL_FUNC(c1, v[e + step] SCL_OP_ARGS);
      c2 = SCL_FUNC(c2, v[e + 2 * step] SCL_OP_ARGS);
      c3 = SCL_FUNC(c3, v[e + 3 * step] SCL_OP_ARGS);
    }
    if (e < n) acc = SCL_FUNC(acc, v[e] SCL_OP_ARGS);
    if (e + step < n) c1 = SCL_FUNC(c1, v[e + step] SCL_OP_ARGS);
    if (e + 2 * step < n) c2 = SCL_FUNC(c2, v[e + 2 * step] SCL_OP_ARGS);
    return SCL_FUNC(SCL_FUNC(acc, c1 SCL_OP_ARGS), SCL_FUNC(c2, c3 SCL_OP_ARGS) SCL_OP_ARGS);
  }
  for (; e < n; e += step) acc = SCL_FUNC(acc, v[e] SCL_OP_ARGS);
  return acc;
}

// The folds of a record (elements e0 .. at ts) by groups of G = 2^glog < 32
// threads in four chains each, and of the vectors too long for so few threads by
// a warp each.  A function of its own: it keeps its registers off the other path.
__device__ __noinline__ void scl_reduce_window_chains(scl_T* out, const scl_u64* seg_off, scl_u64 lo, scl_u64 top,
                                                      scl_u64 e0, int len, const scl_T* ts, int glog,
                                                      unsigned int longest SCL_USER_PARAMS) {
  constexpr int B = 256;
  const int G = 1 << glog, gl = (int)threadIdx.x & (G - 1), lane = threadIdx.x & 31;
  const int most = kWinBytes ? SCL_WIN_LONG : (G >= 8 ? len : SCL_WIN_LONG);
  for (scl_u64 base = lo; base < top; base += B >> glog) {
    const scl_u64 sg = base + (threadIdx.x >> glog);
    scl_u64 a = 0, b = 0;
    if (sg < top) {
      a = seg_off[sg];
      b = seg_off[sg + 1];
    }
    const bool mine = sg < top && (b <= a || (a >= e0 && b <= e0 + (scl_u64)len));
    const int nv = mine && b > a ? (int)(b - a) : 0;
    scl_T acc = (scl_T)(SCL_IDENTITY);
    if (gl < nv && nv <= most) acc = scl_fold_chains(ts + (int)(a - e0), gl, nv, G SCL_EXTRA_ARGS);
    for (int off = G >> 1; off > 0; off >>= 1) {
      // (threads of the group below nv hold a fold)
      const scl_T o = scl_shfl_down(acc, off);
      if (gl + off < G && gl + off < nv) acc = SCL_FUNC(acc, o SCL_OP_ARGS);
    }
    if (gl == 0 && mine && nv <= most) out[sg] = acc;
  }
  if ((int)longest <= most) return;  // (block-uniform)
  // warp w takes the long ones of vectors lo + w, lo + w + 8, ... (an offset pair
  // per lane)
  for (scl_u64 g = lo + (threadIdx.x >> 5); g < top; g += B) {
    const scl_u64 mine = g + (scl_u64)(B / 32 * lane);
    scl_u64 a = 0, b = 0;
    if (mine < top) {
      a = seg_off[mine];
      b = seg_off[mine + 1];
    }
    unsigned int todo =
        __ballot_sync(0xffffffffu, b > a && b - a > (scl_u64)most && a >= e0 && b <= e0 + (scl_u64)len);
    while (todo) {
      const int k = __ffs((int)todo) - 1;
      todo &= todo - 1u;
      const int p = __shfl_sync(0xffffffffu, (int)(a - e0), k), n = __shfl_sync(0xffffffffu, (int)(b - a), k);
      scl_T acc = scl_fold_chains(ts + p, lane, n, 32 SCL_EXTRA_ARGS);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const scl_T o = scl_shfl_down(acc, off);
        if (lane + off < 32) acc = SCL_FUNC(acc, o SCL_OP_ARGS);
      }
      if (lane == 0) out[g + (scl_u64)(B / 32 * k)] = acc;
    }
  }
}

// (CHAINS: a warp's fold of a vector in four chains too.)
template <int WT, bool CHAINS>
__device__ __forceinline__ void scl_reduce_window_run(const scl_T* in, scl_T* out, const scl_u64* seg_off,
                                                      const scl_u64* win_rec, scl_u64 r, scl_u64 n_rec,
                                                      scl_T* ts, unsigned int spin_limit,
                                                      unsigned int* err SCL_USER_PARAMS) {
  constexpr int B = 256;
  const scl_T ident = (scl_T)(SCL_IDENTITY);
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int s_ok;
  const unsigned int bar_s = (unsigned int)__cvta_generic_to_shared(&bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar_s));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const scl_u64 lo = win_rec[4 * r], top = win_rec[4 * r + 1], e0 = win_rec[4 * r + 2];
  const scl_u64 w3 = win_rec[4 * r + 3], ln = SCL_WIN_ELEMENTS(w3);
  const int len = (int)(ln < (scl_u64)WT ? ln : (scl_u64)WT);  // (more only for bad offsets)
  const unsigned int longest = (unsigned int)(w3 >> 32);
  // the record two per SM further on is asked into L2 ahead of its block, which
  // makes two dependent trips there (the record, then what it names): 10^6
  // vectors of 1..199 floats 95.4 -> 87.1 us (152 records ahead 89.1, 912 87.7)
  if (threadIdx.x == 32 && r + SCL_REDUCE_AHEAD < n_rec) {
    const scl_u64* nr = win_rec + 4 * (r + SCL_REDUCE_AHEAD);
    const scl_u64 nl = SCL_WIN_ELEMENTS(nr[3]);
    const scl_u64 a0 = (scl_u64)in + nr[2] * sizeof(scl_T), l0 = nl < (scl_u64)WT ? nl : (scl_u64)WT;
    scl_prefetch_l2(a0, a0 + l0 * sizeof(scl_T));
    scl_prefetch_l2((scl_u64)(seg_off + nr[0]), (scl_u64)(seg_off + nr[1] + 1));
  }
  unsigned int tx;
  const int shift = scl_stage_bulk<scl_T, B>(in + e0, len, ts, bar_s, &tx);
  const scl_u64 nvec = top - lo;
  const unsigned int share = nvec < B ? B / (unsigned int)nvec : 1u;  // threads per vector
  const int glog = 31 - __clz((int)share);
  const int G = 1 << glog, gl = (int)threadIdx.x & (G - 1);
  const scl_u64 step = (scl_u64)(B >> glog);
  const unsigned int few = nvec < B ? (unsigned int)nvec : B;
  const bool warps = G >= 32 || (G >= 8 && ((unsigned int)len >= 450u * few || longest * few > 3u * (unsigned int)len));
  const bool chains = longest > SCL_WIN_LONG || (G < 4 && longest >= 8);
  // this group's first vector's offsets are read while the copy lands
  scl_u64 sg = lo + (threadIdx.x >> (warps ? 5 : glog));
  scl_u64 a = 0, b = 0;
  if (sg < top) {
    a = seg_off[sg];
    b = seg_off[sg + 1];
  }
  if (threadIdx.x == 0) {
    bool ok = tx == 0u || scl_mbar_wait(bar_s, spin_limit);
    if (!ok) {
      scl_raise(err, SCL_DEV_ERR_TIMEOUT);
      scl_mbar_wait(bar_s, 1u << 21);  // the copy may still land here: stay (bounded) until it has
    }
    s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  if (!s_ok) return;
  if (warps) {  // (block-uniform; sg, a, b are the warp's first vector)
    const int lane = threadIdx.x & 31;
    for (; sg < top; sg += B / 32) {
      // (outside the record only for offsets changed since the plan)
      const bool mine = b <= a || (a >= e0 && b <= e0 + (scl_u64)len);
      const int nv = mine && b > a ? (int)(b - a) : 0;
      const scl_T* v = ts + (nv ? (int)(a - e0) + shift : 0);
      const scl_u64 cur = sg;
      if (sg + B / 32 < top) {
        a = seg_off[sg + B / 32];
        b = seg_off[sg + B / 32 + 1];
      }
      scl_T acc = ident;
      if constexpr (CHAINS) {
        if (lane < nv) acc = scl_fold_chains(v, lane, nv, 32 SCL_EXTRA_ARGS);
      } else if (lane < nv) {
        acc = v[lane];
        for (int e = lane + 32; e < nv; e += 32) acc = SCL_FUNC(acc, v[e] SCL_OP_ARGS);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        // (lanes below nv hold a fold)
        const scl_T o = scl_shfl_down(acc, off);
        if (lane + off < 32 && lane + off < nv) acc = SCL_FUNC(acc, o SCL_OP_ARGS);
      }
      if (lane == 0 && mine) out[cur] = acc;
    }
    return;
  }
  if (chains) {  // (block-uniform)
    scl_reduce_window_chains(out, seg_off, lo, top, e0, len, ts + shift, glog, longest SCL_EXTRA_ARGS);
    return;
  }
  for (scl_u64 base = lo; base < top; base += step) {  // (block-uniform)
    // (outside the record only for offsets changed since the plan)
    const bool mine = sg < top && (b <= a || (a >= e0 && b <= e0 + (scl_u64)len));
    const int nv = mine && b > a ? (int)(b - a) : 0;
    const scl_T* v = ts + (nv ? (int)(a - e0) + shift : 0);
    const scl_u64 cur = sg;
    sg += step;
    if (sg < top) {
      a = seg_off[sg];
      b = seg_off[sg + 1];
    }
    scl_T acc = ident;
    if (gl < nv) {
      acc = v[gl];
#pragma unroll 4
      for (int e = gl + G; e < nv; e += G) acc = SCL_FUNC(acc, v[e] SCL_OP_ARGS);
    }
    for (int off = G >> 1; off > 0; off >>= 1) {
      // (threads of the group below nv hold a fold)
      const scl_T o = scl_shfl_down(acc, off);
      if (gl + off < G && gl + off < nv) acc = SCL_FUNC(acc, o SCL_OP_ARGS);
    }
    if (gl == 0 && mine) out[cur] = acc;
  }
}

// A function of its own beside the tiles, whose registers and order of loads its
// code would change (250 log-uniform vectors of 64..2^20 floats 12.3 us, inlined
// 13.8, with CHAINS 15.7).
template <int WT>
__device__ __noinline__ void scl_reduce_window_apart(const scl_T* in, scl_T* out, const scl_u64* seg_off,
                                                     const scl_u64* win_rec, scl_u64 r, scl_u64 n_rec, scl_T* ts,
                                                     unsigned int spin_limit, unsigned int* err SCL_USER_PARAMS) {
  scl_reduce_window_run<WT, false>(in, out, seg_off, win_rec, r, n_rec, ts, spin_limit, err SCL_EXTRA_ARGS);
}

// Segmented Reduce (no counterpart in the reference): out[s] = the fold of
// segment [seg_off[s], seg_off[s+1]) of the flat vector, for every segment,
// in one launch.  Tiles of R x 256 vectors never span segments (segment s
// owns tiles tile_start[s] .. tile_start[s+1]-1, at least one); each tile
// folds its elements into partials[tile], and the last tile of a segment to
// finish (per-segment ticket, reset afterwards) folds that segment's
// partials.  An empty segment yields SCL_IDENTITY.  Blocks past the last
// tile (the grid is an upper bound) return at once; with MERGED (a segment
// plan numbered the tiles) they fold the segments of at most short_max
// elements instead, one window of them per block (scl_reduce_window_run):
// one launch for a whole segmented Reduce.
template <int R, int MERGED = 0, int PER_SM = 0>
__global__ void __launch_bounds__(256, PER_SM)
scl_reduce_seg(const scl_T* in, scl_T* out, const scl_u64* seg_off,
               const unsigned int* tile_start, scl_u64 n_seg, int aligned, scl_C* partials,
               unsigned int* tickets, unsigned int* err, scl_u64 short_max,
               const scl_u64* win_rec, unsigned int spin_limit,
               const unsigned int* tile_seg, unsigned int n_tiles SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  (void)short_max;
  (void)win_rec;
  (void)spin_limit;
  // the tile count, from the host when a plan knows it (~0u: read it)
  const unsigned int nt = n_tiles != ~0u ? n_tiles : tile_start[n_seg];
  if constexpr (MERGED != 0) {
    if (blockIdx.x >= nt) {  // (block-uniform: the whole block takes the window role)
      constexpr int WT = 8 * 256 * scl_vec_width<sizeof(scl_T)>::value;  // 32 KB of elements
      scl_T* ts = reinterpret_cast<scl_T*>(scl_dyn_smem);
      if constexpr (PER_SM != 0)
        scl_reduce_window_run<WT, true>(in, out, seg_off, win_rec, blockIdx.x - nt, gridDim.x - nt, ts, spin_limit,
                                        err SCL_EXTRA_ARGS);
      else
        scl_reduce_window_apart<WT>(in, out, seg_off, win_rec, blockIdx.x - nt, gridDim.x - nt, ts, spin_limit,
                                    err SCL_EXTRA_ARGS);
      return;
    }
  }
  constexpr int V = scl_vec_width<sizeof(scl_T)>::value;
  constexpr int B = 256;
  constexpr scl_u64 TILE = (scl_u64)R * B * V;
  const unsigned int tile = blockIdx.x;
  __shared__ long long s_seg;
  if (threadIdx.x == 0) {
    long long sg = -1;
    if (tile < nt) {
      if (tile_seg) {  // (a segment plan's table)
        sg = (long long)tile_seg[tile];
      } else {
        scl_u64 lo = 0, hi = n_seg - 1;
        while (lo < hi) {
          const scl_u64 mid = (lo + hi + 1) / 2;
          if (tile_start[mid] <= tile) lo = mid; else hi = mid - 1;
        }
        sg = (long long)lo;
      }
    }
    s_seg = sg;
  }
  __syncthreads();
  if (s_seg < 0) return;
  const scl_u64 sg = (scl_u64)s_seg;
  const unsigned int first = tile_start[sg], count = tile_start[sg + 1] - first;
  const scl_u64 off = seg_off[sg], len = seg_off[sg + 1] > off ? seg_off[sg + 1] - off : 0;
  if (len == 0) {
    if (threadIdx.x == 0) out[sg] = (scl_T)(SCL_IDENTITY);
    return;
  }
  const scl_T* src = in + off;
  const scl_u64 begin = (scl_u64)(tile - first) * TILE;
  const scl_u64 end = begin + TILE < len ? begin + TILE : len;
  bool have = false;
  scl_T acc;
  const bool vec = aligned && ((off * sizeof(scl_T)) % 16 == 0) && end - begin == TILE;
  if (vec) {  // R vectors per thread, loaded 8 at a time
    constexpr int G = R < 8 ? R : 8;
#pragma unroll 1
    for (int r0 = 0; r0 < R; r0 += G) {
      scl_pack<scl_T, V> a[G];
#pragma unroll
      for (int r = 0; r < G; ++r)
        a[r] = scl_load<scl_T, V>(src + begin + ((scl_u64)(r0 + r) * B + threadIdx.x) * V);
#pragma unroll
      for (int r = 0; r < G; ++r)
#pragma unroll
        for (int e = 0; e < V; ++e) {
          acc = have ? SCL_FUNC(acc, a[r].v[e] SCL_OP_ARGS) : a[r].v[e];
          have = true;
        }
    }
  } else {
    // ragged or unaligned: scalar head up to the first 16-byte boundary,
    // 16-byte body, scalar tail
    scl_u64 h = begin, bend = begin;
    if (V > 1 && ((scl_u64)(src + begin)) % sizeof(scl_T) == 0) {
      const scl_u64 mis = ((scl_u64)(src + begin)) & 15u;
      h = begin + (mis ? (16u - mis) / sizeof(scl_T) : 0);
      if (h > end) h = end;
      bend = h + (end - h) / V * V;
    }
    for (scl_u64 i = begin + threadIdx.x; i < h; i += B) {
      acc = have ? SCL_FUNC(acc, src[i] SCL_OP_ARGS) : src[i];
      have = true;
    }
    for (scl_u64 i = h + (scl_u64)threadIdx.x * V; i < bend; i += (scl_u64)B * V) {
      scl_pack<scl_T, V> a = scl_load<scl_T, V>(src + i);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        acc = have ? SCL_FUNC(acc, a.v[e] SCL_OP_ARGS) : a.v[e];
        have = true;
      }
    }
    for (scl_u64 i = (bend > h ? bend : h) + threadIdx.x; i < end; i += B) {
      acc = have ? SCL_FUNC(acc, src[i] SCL_OP_ARGS) : src[i];
      have = true;
    }
  }
  scl_C c;
  if (have) c = (scl_C)acc;
  scl_block_fold(have, c SCL_EXTRA_ARGS);
  if (count == 1) {  // the segment's only tile
    if (threadIdx.x == 0) out[sg] = (scl_T)c;
    return;
  }
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    scl_st_cg(&partials[tile], c);
    __threadfence();
    s_last = (atomicAdd(&tickets[sg], 1u) == count - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  have = false;
  for (unsigned int b = threadIdx.x; b < count; b += B) {
    scl_C v = scl_ld_cg(&partials[first + b]);
    c = have ? (scl_C)SCL_FUNC_C(c, v SCL_OP_ARGS) : v;
    have = true;
  }
  scl_block_fold(have, c SCL_EXTRA_ARGS);
  if (threadIdx.x == 0) {
    out[sg] = (scl_T)c;
    tickets[sg] = 0u;
  }
}

#endif  // SCL_KIND == 9

#if SCL_KIND == 16
// Fused Zip -> Reduce (no counterpart in the reference, which materialises
// the zipped vector): out[0] = fold over i of USR_ZIP(left[i], right[i]),
// in one pass over both inputs with the single-pass reduce above (per-thread
// fold, FP64 carries for float, last-block combine).  Extra arguments: the
// Reduce's first, then the Zip's.
template <int U>
__global__ void scl_zipreduce_k(const SCL_TYPE_0* left, const SCL_TYPE_1* right, scl_T* out,
                                scl_u64 n, int aligned, scl_C* partials, unsigned int* ticket,
                                unsigned int* err SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  constexpr int V = scl_vec_width<sizeof(SCL_TYPE_0), sizeof(SCL_TYPE_1)>::value;
  const scl_u64 tid = SCL_TID(), nth = SCL_NTH();
  if (n == 0) {
    if (tid == 0) out[0] = (scl_T)(SCL_IDENTITY);
    return;
  }
  const scl_u64 nvec = aligned ? n / V : 0;
  bool have = false;
  scl_T acc;
  for (scl_u64 j = tid; j < nvec; j += nth * U) {
    scl_pack<SCL_TYPE_0, V> a[U];
    scl_pack<SCL_TYPE_1, V> b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const scl_u64 k = j + (scl_u64)u * nth;
      if (k < nvec) {
        a[u] = scl_load<SCL_TYPE_0, V>(left + k * V);
        b[u] = scl_load<SCL_TYPE_1, V>(right + k * V);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const scl_u64 k = j + (scl_u64)u * nth;
      if (k < nvec) {
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const scl_T z = USR_ZIP(a[u].v[e], b[u].v[e] SCL_SECOND_ARGS);
          acc = have ? SCL_FUNC(acc, z SCL_OP_ARGS) : z;
          have = true;
        }
      }
    }
  }
  for (scl_u64 i = nvec * V + tid; i < n; i += nth) {
    const scl_T z = USR_ZIP(left[i], right[i] SCL_SECOND_ARGS);
    acc = have ? SCL_FUNC(acc, z SCL_OP_ARGS) : z;
    have = true;
  }
  scl_C c;
  if (have) c = (scl_C)acc;
  scl_block_fold(have, c SCL_EXTRA_ARGS);

  if (gridDim.x == 1) {
    if (threadIdx.x == 0) out[0] = (scl_T)c;
    return;
  }
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    scl_st_cg(&partials[blockIdx.x], c);  // every block holds at least one element
    __threadfence();
    const unsigned int t = atomicAdd(ticket, 1u);
    s_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  have = false;
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
    scl_C v = scl_ld_cg(&partials[b]);
    c = have ? (scl_C)SCL_FUNC_C(c, v SCL_OP_ARGS) : v;
    have = true;
  }
  scl_block_fold(have, c SCL_EXTRA_ARGS);
  if (threadIdx.x == 0) {
    out[0] = (scl_T)c;
    *ticket = 0u;
  }
}
#endif  // SCL_KIND == 16
#endif
