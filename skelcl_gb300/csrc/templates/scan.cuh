// ---------------------------------------------------------------------------
// Scan for sm_103a: single-pass decoupled look-back (Merrill & Garland,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back", NVIDIA 2016).
//
// Replaces the reference's recursive Blelloch scan (SCL_SCAN, ceil(log_256 N)
// passes) and its uniform-add passes (SCL_UNIFORM_COMBINATION) of
// include/SkelCL/detail/ScanKernel.cl:74-250 / ScanDef.h:91-259.
//
// Semantics kept from the reference: the output is the EXCLUSIVE scan seeded
// with the identity (out[0] = id, out[i] = x[0] + ... + x[i-1]; ScanKernel.cl
// clears the last element to SCL_IDENTITY before the down-sweep and pads
// partial blocks with it), and the operator must be associative (the
// reference combines in tree order).  Extensions: SCL_SHAPE_INCLUSIVE gives
// the inclusive scan, SCL_SHAPE_REVERSE scans from the last element (the
// adjoint of a forward sum-scan is a reverse scan).
//
// Tile = R rows x 256 threads x V elements (V = 16 bytes / sizeof T), loaded
// with coalesced 16-byte accesses: row r of the tile is one contiguous span of
// 256*V elements, thread t holds elements [r*256*V + t*V, +V).  The staged
// kernel's tiles are numbered by block index: blocks are dispatched in index
// order, so a tile only waits on tiles whose blocks have started, and the
// tile's copy is issued at once (an atomic ticket taken first, as the
// register kernel still does, put one L2 round trip in front of every tile's
// copy: 2^26 floats 102.4 against 98.2 us).  Were that order ever broken,
// the bounded waits below would end the launch with SCL_DEV_ERR_TIMEOUT
// instead of a hang.
// In-tile: per-thread sequential fold, warp shuffles, one warp scans the R*8
// warp totals, publishes the tile aggregate and looks back over up to 32
// predecessors per round trip (one lane per predecessor).  Every wait is
// bounded by `spin_limit` polls, after which the tile raises
// SCL_DEV_ERR_TIMEOUT and proceeds, so a launch always terminates.  Carries
// across tiles are held in SCL_CARRY_T (double for float element types).
//
// Tile status: one 16-byte slot {aggregate word, inclusive word} per tile,
// each slot alone on a 128-byte line (SCL_SLOT_STRIDE words apart), so a poll
// is one 16-byte load and publishers and pollers of different tiles never
// share a line (measured on GB300: sharing lines cost about a third of the
// scan's bandwidth).
//   mode 1, carry <= 4 bytes: word = 1<<32 | value bits; 0 = not published
//   mode 2, carry is double : word = ~(value bits); 0 = not published
//   mode 0, other carries   : flag word (release/acquire) + separate values
// ---------------------------------------------------------------------------

#if SCL_KIND == 10 || SCL_KIND == 17
typedef SCL_TYPE_0 scl_T;
typedef SCL_CARRY_T scl_C;
#if SCL_KIND == 17
// Fused Scan -> Map (no counterpart in the reference, which materialises the
// scanned vector): the staged kernel stores USR_MAP(scan value) instead of
// the scan value.  Extra arguments: the Scan's first, then the Map's.
typedef SCL_TYPE_1 scl_O;
#define SCL_EPILOGUE(v) USR_MAP(v SCL_SECOND_ARGS)
#else
typedef scl_T scl_O;
#define SCL_EPILOGUE(v) (v)
#endif

// A staged tile asks for the tile this many after it to be brought into L2, one
// per SM (152 here): its successors' copies then take an L2 round trip instead
// of one through DRAM under load, and the look-back, which waits for the slowest
// of its predecessors, ends sooner.  2^28 int 359.8 -> 332.3 us, 2^26 97.0 ->
// 89.6 (the transfers 317 and 79); 2^26 float 98.6 -> 94.5.  76 tiles ahead
// 92.1 us at 2^26, 304 90.4, 912 (a whole wave of resident tiles) 104.1; asked
// for before the tile's own copy, 94.5.
#define SCL_SCAN_AHEAD SCL_SMS
#define SCL_SCAN_B 256
#define SCL_SCAN_W 8
#define SCL_SLOT_STRIDE 16  // 64-bit words between tile slots (128 bytes)
#define SCL_FLAG_AGG 1u
#define SCL_FLAG_INC 2u

template <typename A, typename B> struct scl_same { static constexpr bool value = false; };
template <typename A> struct scl_same<A, A> { static constexpr bool value = true; };
template <typename C> struct scl_status_mode {
  static constexpr int value = sizeof(C) <= 4 ? 1 : (scl_same<C, double>::value ? 2 : 0);
};

// Staged kernel: when carries are wider than the elements (FP64 carries of a
// float scan), each thread folds its lane prefix into the staged tile before
// the look-back instead of keeping R warp prefixes in registers across it
// (measured on GB300, f32 2^26: 40 registers with spills -> 29 without, 4.5 %
// faster; for 4-byte carries keeping them is 1 % faster).
constexpr bool kLocalPrefix = !scl_same<scl_C, scl_T>::value;

// Adjacent 16-byte vectors of a lane in one row of a staged tile.  A row costs
// every lane five folds across the warp and two more for its prefix; doubles,
// whose additions this device does at a sixty-fourth of the rate of single
// precision, take four vectors a lane (2.75 folds an element instead of 5, for
// four-way bank conflicts): 2^25 doubles 344.5 -> 204.2 us (two vectors 243.7,
// eight 260.3; floats with two 94.5 -> 102.8 at 2^26).
constexpr int kLaneVectors = scl_same<scl_T, double>::value ? 4 : 1;
// In a branch that folds: keeps the fold of doubles in the branch, which few
// warps may take, where it would be made in any case and its result selected (2 *
// 10^7 doubles in vectors of 1..199 156 -> 133 us).
__device__ __forceinline__ void scl_costly_fold() {
  if constexpr (kLaneVectors > 1) asm volatile("");
}
// A lane's vectors in shared memory.
template <typename T, int V, int M>
__device__ __forceinline__ scl_pack<T, V * M> scl_load_lane(const T* p) {
  if constexpr (M == 1) return scl_load<T, V>(p);
  scl_pack<T, V * M> r;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const scl_pack<T, V> q = scl_load<T, V>(p + m * V);
#pragma unroll
    for (int e = 0; e < V; ++e) r.v[m * V + e] = q.v[e];
  }
  return r;
}
template <typename T, int V, int M>
__device__ __forceinline__ void scl_store_lane(T* p, const scl_pack<T, V * M>& r) {
  if constexpr (M == 1) {
    scl_store<T, V>(p, r);
    return;
  }
#pragma unroll
  for (int m = 0; m < M; ++m) {
    scl_pack<T, V> q;
#pragma unroll
    for (int e = 0; e < V; ++e) q.v[e] = r.v[m * V + e];
    scl_store<T, V>(p + m * V, q);
  }
}

__device__ __forceinline__ unsigned long long scl_ld_relaxed64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void scl_st_relaxed64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}

template <typename C>
__device__ __forceinline__ unsigned long long scl_pack_word(const C& v) {
  if constexpr (scl_status_mode<C>::value == 1) {
    unsigned int bits = 0;
    memcpy(&bits, &v, sizeof(C));
    return (1ull << 32) | bits;
  } else {
    unsigned long long bits;
    memcpy(&bits, &v, 8);
    return ~bits;  // all-ones bits (never produced by arithmetic) would read as "not published"
  }
}
template <typename C>
__device__ __forceinline__ C scl_unpack_word(unsigned long long w) {
  C v;
  if constexpr (scl_status_mode<C>::value == 1) {
    unsigned int bits = (unsigned int)w;
    memcpy(&v, &bits, sizeof(C));
  } else {
    const unsigned long long bits = ~w;
    memcpy(&v, &bits, 8);
  }
  return v;
}

// Ordered inclusive warp scan: lane l gets x[0] + ... + x[l].
template <typename T>
__device__ __forceinline__ T scl_warp_incl(T v SCL_USER_PARAMS) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    T o = scl_shfl_up(v, off);
    if (lane >= off) v = SCL_FUNC(o, v SCL_OP_ARGS);
  }
  return v;
}

// Status storage of one launch (device pointers into the workspace).
struct scl_scan_status {
  unsigned long long* slots;  // modes 1, 2: slot of tile t at slots[t * SCL_SLOT_STRIDE]
  unsigned int* flags;        // mode 0
  scl_C* agg;                 // mode 0
  scl_C* incl;                // mode 0
};

// What a launch clears for the next one: the slots (or flags) [0, n) of the
// status region the previous launch used, and that region's ticket word.
// The host alternates launches between two regions, so no launch needs a
// separate clear before it (a launch recorded in a graph uses a third
// region that the graph clears itself).
struct scl_scan_clear {
  unsigned long long* slots;  // modes 1, 2
  unsigned int* flags;        // mode 0
  unsigned int* ticket;       // reset to 0 (block 0), or null
  unsigned long long n;
};

__device__ __forceinline__ void scl_scan_clear_other(const scl_scan_clear& c) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && c.ticket) *c.ticket = 0u;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < c.n;
       i += stride) {
    if constexpr (scl_status_mode<scl_C>::value != 0) {
      asm volatile("st.global.v2.u64 [%0], {%1, %1};" :: "l"(c.slots + i * SCL_SLOT_STRIDE), "l"(0ull)
                   : "memory");
    } else {
      c.flags[i] = 0u;
    }
  }
}

__device__ __forceinline__ void scl_publish(const scl_scan_status& st, unsigned int tile,
                                            bool inclusive, const scl_C& v) {
  if constexpr (scl_status_mode<scl_C>::value != 0) {
    scl_st_relaxed64(st.slots + (size_t)tile * SCL_SLOT_STRIDE + (inclusive ? 1 : 0),
                     scl_pack_word(v));
  } else {
    scl_st_cg(inclusive ? &st.incl[tile] : &st.agg[tile], v);
    scl_st_release(&st.flags[tile], inclusive ? SCL_FLAG_INC : SCL_FLAG_AGG);
  }
}

// Poll predecessor `idx` until it published something (or the wait gives up).
// Returns 2 = inclusive prefix, 1 = aggregate, 0 = gave up; value in *v.
__device__ __forceinline__ int scl_poll(const scl_scan_status& st, long long idx,
                                        unsigned int spin_limit, scl_C* v) {
  unsigned int polls = 0;
  while (true) {
    if constexpr (scl_status_mode<scl_C>::value != 0) {
      unsigned long long wa, wi;
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                   : "=l"(wa), "=l"(wi) : "l"(st.slots + (size_t)idx * SCL_SLOT_STRIDE) : "memory");
      if (wi != 0ull) { *v = scl_unpack_word<scl_C>(wi); return 2; }
      if (wa != 0ull) { *v = scl_unpack_word<scl_C>(wa); return 1; }
    } else {
      const unsigned int f = scl_ld_acquire(&st.flags[idx]);
      if (f == SCL_FLAG_INC) { *v = scl_ld_cg(&st.incl[idx]); return 2; }
      if (f == SCL_FLAG_AGG) { *v = scl_ld_cg(&st.agg[idx]); return 1; }
    }
    if (++polls > spin_limit) return 0;
    if (polls > 32) scl_nanosleep(32);
  }
}

// Decoupled look-back of warp 0 (all 32 lanes) for tile number `tile`, whose
// sequence starts at tile `first`: returns the fold of every
// earlier tile of the sequence, combined as f(earlier, later).  Each round
// reads 32 predecessors (one per lane, lane l = tile - 1 - l); a round that
// finds an inclusive prefix ends the look-back, otherwise its aggregates are
// folded in and the next 32 are read.  (Measured on GB300 and not kept:
// 64 or 128 predecessors per round, several loads in flight per lane, in
// every round, or only after a first round without an inclusive prefix, or
// only for the first two waves of tiles -- all slower, 1.5-18 %; with the
// code present but never taken the time is unchanged.)
__device__ __forceinline__ scl_C scl_lookback(const scl_scan_status& st, long long tile, long long first,
                                              unsigned int spin_limit, unsigned int* err
                                                  SCL_USER_PARAMS) {
  const int lane = threadIdx.x & 31;
  const scl_C cid = (scl_C)(scl_T)(SCL_IDENTITY);
  scl_C running = cid;  // fold of the tiles already visited (later ones)
  long long pred = tile - 1;
  bool first_round = true;
  while (true) {
    const long long idx = pred - lane;
    scl_C v = cid;
    int kind = 2;  // before the sequence's first tile: nothing to add, stop here
    if (idx >= first) {
      kind = scl_poll(st, idx, spin_limit, &v);
      if (kind == 0) {
        scl_raise(err, SCL_DEV_ERR_TIMEOUT);
        v = cid;
        kind = 2;
      }
    }
    const unsigned int pmask = __ballot_sync(0xffffffffu, kind == 2);
    // the usual case: the nearest predecessor already holds its inclusive
    // prefix, and nothing needs folding (the fold below costs five shuffle
    // rounds, in FP64 for float carries)
    if (pmask & 1u) {
      const scl_C w = scl_shfl_idx(v, 0);
      return first_round ? w : (scl_C)SCL_FUNC_C(w, running SCL_OP_ARGS);
    }
    const int first_inc = pmask ? __ffs(pmask) - 1 : 31;  // nearest inclusive prefix
    if (lane > first_inc) v = cid;
    // ordered fold over lanes: higher lane = earlier tile
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      scl_C o = scl_shfl_down(v, off);
      if (lane + off < 32) v = (scl_C)SCL_FUNC_C(o, v SCL_OP_ARGS);
    }
    const scl_C window = scl_shfl_idx(v, 0);
    running = (scl_C)SCL_FUNC_C(window, running SCL_OP_ARGS);
    if (pmask) return running;
    pred -= 32;
    first_round = false;
  }
}

template <int R, int MINB>
__global__ void __launch_bounds__(SCL_SCAN_B, MINB)  // MINB resident tiles per SM at least
scl_scan_k(const scl_T* in, scl_T* out, scl_u64 n, unsigned int flags, int aligned,
           unsigned int* tile_counter, scl_scan_status st, scl_scan_clear clr,
           unsigned int spin_limit, unsigned int* err SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  constexpr int B = SCL_SCAN_B, W = SCL_SCAN_W;
  constexpr int V = scl_vec_width<sizeof(scl_T)>::value;
  constexpr int TILE = R * B * V;
  const bool inclusive = (flags & 1u) != 0, reverse = (flags & 2u) != 0;
  const scl_T ident = (scl_T)(SCL_IDENTITY);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  __shared__ unsigned int s_tile;
  __shared__ scl_T s_wsum[R * W];
  __shared__ scl_T s_carry;  // the tile's prefix, converted once to the element type
  if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1u);
  scl_scan_clear_other(clr);
  __syncthreads();
  const unsigned int tile = s_tile;
  const scl_u64 base = (scl_u64)tile * TILE;

  // ---- load (logical order; reverse maps logical i to physical n-1-i)
  scl_T x[R][V];
  const bool full = aligned && base + TILE <= n && (!reverse || n % V == 0);
  if (full) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const scl_u64 q = (scl_u64)r * B + threadIdx.x;
      if (!reverse) {
        scl_pack<scl_T, V> p = scl_load<scl_T, V>(in + base + q * V);
#pragma unroll
        for (int e = 0; e < V; ++e) x[r][e] = p.v[e];
      } else {
        scl_pack<scl_T, V> p = scl_load<scl_T, V>(in + (n - base - (q + 1) * V));
#pragma unroll
        for (int e = 0; e < V; ++e) x[r][e] = p.v[V - 1 - e];
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const scl_u64 i = base + ((scl_u64)r * B + threadIdx.x) * V + e;
        x[r][e] = i < n ? in[reverse ? n - 1 - i : i] : ident;
      }
  }

  // ---- in-thread inclusive scan of each vector, then warp scans of totals
  scl_T wincl[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int e = 1; e < V; ++e) x[r][e] = SCL_FUNC(x[r][e - 1], x[r][e] SCL_OP_ARGS);
    wincl[r] = scl_warp_incl(x[r][V - 1] SCL_EXTRA_ARGS);
    if (lane == 31) s_wsum[r * W + warp] = wincl[r];
  }
  __syncthreads();

  // ---- warp 0: exclusive prefixes of the R*W warp totals (row-major = tile
  //      order), the tile aggregate, then the look-back for the tile prefix
  if (warp == 0) {
    scl_T carry = ident;
#pragma unroll
    for (int c = 0; c < (R * W + 31) / 32; ++c) {
      const int q = c * 32 + lane;
      scl_T v = q < R * W ? s_wsum[q] : ident;
      scl_T vi = scl_warp_incl(v SCL_EXTRA_ARGS);
      scl_T ve = scl_shfl_up(vi, 1);
      if (lane == 0) ve = ident;
      if (q < R * W) s_wsum[q] = SCL_FUNC(carry, ve SCL_OP_ARGS);
      scl_T total = scl_shfl_idx(vi, 31);
      carry = SCL_FUNC(carry, total SCL_OP_ARGS);
    }
    const scl_C aggc = (scl_C)carry;
    scl_C prefix = (scl_C)ident;
    if (lane == 0) scl_publish(st, tile, tile == 0, aggc);
    if (tile != 0) {
      prefix = scl_lookback(st, (long long)tile, 0, spin_limit, err SCL_EXTRA_ARGS);
      if (lane == 0) scl_publish(st, tile, true, (scl_C)SCL_FUNC_C(prefix, aggc SCL_OP_ARGS));
    }
    if (lane == 0) s_carry = (scl_T)prefix;
  }
  __syncthreads();

  // ---- outputs (computed in place in x)
  const scl_T tile_carry = s_carry;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    scl_T lane_excl = scl_shfl_up(wincl[r], 1);
    if (lane == 0) lane_excl = ident;
    const scl_T pre = SCL_FUNC(SCL_FUNC(tile_carry, s_wsum[r * W + warp] SCL_OP_ARGS),
                               lane_excl SCL_OP_ARGS);
    if (inclusive) {
#pragma unroll
      for (int e = 0; e < V; ++e) x[r][e] = SCL_FUNC(pre, x[r][e] SCL_OP_ARGS);
    } else {
#pragma unroll
      for (int e = V - 1; e > 0; --e) x[r][e] = SCL_FUNC(pre, x[r][e - 1] SCL_OP_ARGS);
      x[r][0] = pre;
    }
  }
  if (full) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const scl_u64 q = (scl_u64)r * B + threadIdx.x;
      scl_pack<scl_T, V> p;
      if (!reverse) {
#pragma unroll
        for (int e = 0; e < V; ++e) p.v[e] = x[r][e];
        scl_store<scl_T, V>(out + base + q * V, p);
      } else {
#pragma unroll
        for (int e = 0; e < V; ++e) p.v[V - 1 - e] = x[r][e];
        scl_store<scl_T, V>(out + (n - base - (q + 1) * V), p);
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const scl_u64 i = base + ((scl_u64)r * B + threadIdx.x) * V + e;
        if (i < n) out[reverse ? n - 1 - i : i] = x[r][e];
      }
  }
}

// ---------------------------------------------------------------------------
// Shared-memory staged variant.  One elected thread brings the tile into
// shared memory with bulk asynchronous copies (completion counted on an
// mbarrier), threads scan it there, and only the R warp totals per thread stay
// in registers while warp 0 looks back: about 40 registers per thread, so the
// SM holds as many tiles as its shared memory allows (6 of 32 KB) instead of
// as many as the register file allows with the tile in registers (4).
// Reverse, ragged and unaligned tiles are staged with ordinary loads.
// ---------------------------------------------------------------------------

// Segmented scan of the segments of at most short_max elements: one warp per
// segment, warps striding over the segments (warp `wid` of `nw`); per round
// each lane scans U contiguous elements serially, a warp scan combines the
// lanes' totals, and rounds are chained through a carry in the element type
// (no block boundary is crossed, as inside one tile of the tiled kernel; FP64
// carries here would make the FP64 pipe the bound for tiny segments); longer
// segments (and empty ones, which have nothing to write) are left to the
// tiles.  Operand order and identity handling are those of the tiled kernel:
// f(earlier, later), the exclusive form starts from SCL_IDENTITY.
template <int U>
__device__ __forceinline__ void scl_scan_short_run(const scl_T* in, scl_O* out, const scl_u64* seg_off,
                                                   scl_u64 n_seg, unsigned int flags, scl_u64 short_max,
                                                   scl_u64 wid, scl_u64 nw SCL_USER_PARAMS) {
  const int lane = threadIdx.x & 31;
  const bool inclusive = (flags & 1u) != 0, reverse = (flags & 2u) != 0;
  const scl_T ident = (scl_T)(SCL_IDENTITY);
  // round b of a segment [lo, hi): lane l holds the logical elements
  // b + l*U .. b + l*U + U-1, which sit at lo + e, or at hi - 1 - e reversed
  // (identity past the end, and nothing loaded for segments left to tiles)
  auto load = [&](scl_T (&v)[U], scl_u64 lo, scl_u64 hi, scl_u64 b) {
    const scl_u64 len = hi - lo;
    const bool mine = len <= short_max;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const scl_u64 e = b + (scl_u64)lane * U + k;
      v[k] = (mine && e < len) ? in[reverse ? hi - 1 - e : lo + e] : ident;
    }
  };
  auto bounds = [&](scl_u64 sg, scl_u64* lo, scl_u64* hi) {
    *lo = 0;
    *hi = 0;
    if (sg < n_seg) {
      *lo = seg_off[sg];
      const scl_u64 h = seg_off[sg + 1];
      *hi = h > *lo ? h : *lo;
    }
  };
  // software pipeline: the next segment's first round and the offsets of
  // the one after are loaded while this segment is scanned
  scl_u64 sg = wid;
  scl_u64 lo, hi, lo_n, hi_n;
  bounds(sg, &lo, &hi);
  bounds(sg + nw, &lo_n, &hi_n);
  scl_T v[U];
  load(v, lo, hi, 0);
  for (; sg < n_seg; sg += nw) {
    scl_u64 lo_nn, hi_nn;
    bounds(sg + 2 * nw, &lo_nn, &hi_nn);
    scl_T vn[U];
    load(vn, lo_n, hi_n, 0);
    const scl_u64 len = hi - lo;
    if (len > 0 && len <= short_max) {
      scl_T carry = ident;
      for (scl_u64 b = 0; b < len; b += 32 * U) {
        if (b > 0) load(v, lo, hi, b);
        const scl_u64 e0 = b + (scl_u64)lane * U;
#pragma unroll
        for (int k = 1; k < U; ++k) v[k] = SCL_FUNC(v[k - 1], v[k] SCL_OP_ARGS);
        const scl_T tot = scl_warp_incl(v[U - 1] SCL_EXTRA_ARGS);
        scl_T lane_excl = scl_shfl_up(tot, 1);
        if (lane == 0) lane_excl = ident;
        const scl_T pre = SCL_FUNC(carry, lane_excl SCL_OP_ARGS);
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const scl_u64 e = e0 + k;
          if (e < len) {
            const scl_T r = inclusive ? SCL_FUNC(pre, v[k] SCL_OP_ARGS)
                                      : (k == 0 ? pre : SCL_FUNC(pre, v[k - 1] SCL_OP_ARGS));
            out[reverse ? hi - 1 - e : lo + e] = SCL_EPILOGUE(r);
          }
        }
        carry = SCL_FUNC(carry, scl_shfl_idx(tot, 31) SCL_OP_ARGS);
      }
    }
    lo = lo_n;
    hi = hi_n;
    lo_n = lo_nn;
    hi_n = hi_nn;
#pragma unroll
    for (int k = 0; k < U; ++k) v[k] = vn[k];
  }
}

// ---- windows of short segments (planned segmented Scan) --------------------
// One block takes one window record r of the plan, {first vector, end vector,
// first element, elements}: consecutive vectors of at most a quarter of a
// tile that start in one window of 47/64 of a tile (half a tile of each for
// elements of 8 bytes and more), all but the last ending inside it, so that the
// record fits in one staged tile.
// The record's elements come into shared memory by bulk asynchronous copies
// (element e0 + p at ts[p + shift]; bounded wait) while the threads mark, in
// a bit mask, where the vectors start in logical order (their last elements
// for a reverse scan).  Then the whole record is scanned at once as one
// segmented scan, whatever the vectors' lengths: rows of 32 x E elements, one
// per warp at a time, E consecutive ones per lane (two 16-byte vectors), a
// start bit cutting the running fold; the lanes' tails are scanned across
// the warp back to the nearest lane that holds a start, the rows' tails
// across one warp, and an element before its row's first start takes the
// row's carry when it is read back.  f(earlier, later) throughout, in the
// element type; the identity only fills positions outside the record.
// Bound by memory (8 bytes an element), then by issue: 10^6 vectors of 1..199
// floats 0.211 -> 0.133 ms (flat 0.142), 10^7 of 0..2 0.352 -> 0.048 ms,
// 66,666 of 1000..1999 0.284 -> 0.133 ms against one thread per vector of up
// to 256 elements (about 40 busy threads of a block's 256, each a chain of
// shared-memory round trips) and a warp per longer one.
template <typename T, int TILE>
struct scl_win {
  static constexpr int V = scl_vec_width<sizeof(T)>::value;
  // elements per lane and row (more of doubles, as in a staged tile: 2 * 10^7 in
  // vectors of 1..199 170 -> 150 us)
  static constexpr int E = (kLaneVectors > 1 ? 4 : 2) * V;
  static constexpr int ROW = 32 * E;
  static constexpr int ROWS = TILE / ROW + 1;  // (a record keeps its 16-byte phase)
  unsigned int mask[ROWS * ROW / 32];       // bit p: a vector starts at ts[p]
  T carry[ROWS];                            // a row's tail, then the carry into it
  int head[ROWS];                           // the row's first start (ROW: none)
};

// The block's record in shared memory, its starts marked; false after a
// wait that gave up.  Ends with a block barrier.
template <typename T, int TILE, int B>
__device__ __forceinline__ bool scl_win_open(const T* in, const scl_u64* seg_off, scl_u64 lo, scl_u64 top,
                                             scl_u64 e0, int len, bool reverse, const T& ident, T* ts,
                                             scl_win<T, TILE>& w, unsigned int bar_s, unsigned int spin_limit,
                                             unsigned int* err, int* shift_out) {
  typedef scl_win<T, TILE> W;
  __shared__ int s_ok;
  unsigned int tx;
  const int shift = scl_stage_bulk<T, B>(in + e0, len, ts, bar_s, &tx);
  *shift_out = shift;
  // this thread's first vector's offsets are read while the copy lands
  scl_u64 sg = lo + threadIdx.x;
  scl_u64 a = 0, b = 0;
  if (sg < top) {
    a = seg_off[sg];
    b = seg_off[sg + 1];
  }
  for (int i = threadIdx.x; i < W::ROWS * W::ROW / 32; i += B) w.mask[i] = 0u;
  const int P = shift + len, PT = (P + W::E - 1) / W::E * W::E;
  if ((int)threadIdx.x < shift) ts[threadIdx.x] = ident;
  if ((int)threadIdx.x < PT - P) ts[P + threadIdx.x] = ident;
  __syncthreads();
  while (sg < top) {
    // (outside the record only for offsets changed since the plan)
    if (b > a && a >= e0 && b <= e0 + (scl_u64)len) {
      const int p = (int)((reverse ? b - 1 : a) - e0) + shift;
      atomicOr(&w.mask[p >> 5], 1u << (p & 31));
    }
    sg += B;
    if (sg < top) {
      a = seg_off[sg];
      b = seg_off[sg + 1];
    }
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
  return s_ok != 0;
}

// Segmented scan across a warp: lane l's t becomes the fold of the t of lanes
// start .. l, start = the nearest lane at or below l whose bit is set in
// `starts` (0 if none).
template <typename T>
__device__ __forceinline__ T scl_warp_segscan(T t, unsigned int starts SCL_USER_PARAMS) {
  const int lane = threadIdx.x & 31;
  const unsigned int below = starts & (0xffffffffu >> (31 - lane));
  const int start = below ? 31 - __clz((int)below) : 0;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const T o = scl_shfl_up(t, off);
    if (lane - off >= start) t = SCL_FUNC(o, t SCL_OP_ARGS);
  }
  return t;
}

// Scans positions 0 .. P - 1 of the record in place (REV: from the end), up
// to the carries into the rows (scl_win_at applies them).  Ends with a block
// barrier.
template <int REV, typename T, int TILE, int B>
__device__ __forceinline__ void scl_win_scan(T* ts, unsigned int P, const T& ident,
                                             scl_win<T, TILE>& w SCL_USER_PARAMS) {
  typedef scl_win<T, TILE> W;
  constexpr int V = W::V, E = W::E;
  const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const unsigned int chunks = (P + E - 1) / E, rows = (chunks + 31u) / 32u;
  for (unsigned int row = warp; row < rows; row += B / 32) {
    const unsigned int j = row * 32u + lane;
    const unsigned int pos = (REV ? chunks - 1u - j : j) * E;
    T x[E];  // in logical order
    unsigned int hd = 0;
    if (j < chunks) {
      scl_pack<T, V> p[E / V];
#pragma unroll
      for (int c = 0; c < E / V; ++c) p[c] = scl_load<T, V>(ts + pos + c * V);
#pragma unroll
      for (int e = 0; e < V; ++e)
#pragma unroll
        for (int c = 0; c < E / V; ++c) x[REV ? E - 1 - c * V - e : c * V + e] = p[c].v[e];
      hd = w.mask[pos >> 5] >> (pos & 31u);
      if (REV) hd = __brev(hd << (32 - E));
      else if (E < 32) hd &= (1u << (E & 31)) - 1u;
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) x[e] = ident;
    }
#pragma unroll
    for (int e = 1; e < E; ++e)
      if (!((hd >> e) & 1u)) x[e] = SCL_FUNC(x[e - 1], x[e] SCL_OP_ARGS);
    const unsigned int starts = __ballot_sync(0xffffffffu, hd != 0u);
    const T t = scl_warp_segscan(x[E - 1], starts SCL_EXTRA_ARGS);
    const T cin = scl_shfl_up(t, 1);
    const int first = hd ? __ffs((int)hd) - 1 : E;  // elements the lanes before reach into
    if (lane != 0) {
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (e < first) {
          scl_costly_fold();
          x[e] = SCL_FUNC(cin, x[e] SCL_OP_ARGS);
        }
    }
    if (j < chunks) {
      scl_pack<T, V> p[E / V];
#pragma unroll
      for (int e = 0; e < V; ++e)
#pragma unroll
        for (int c = 0; c < E / V; ++c) p[c].v[e] = x[REV ? E - 1 - c * V - e : c * V + e];
#pragma unroll
      for (int c = 0; c < E / V; ++c) scl_store<T, V>(ts + pos + c * V, p[c]);
    }
    const int fl = starts ? __ffs((int)starts) - 1 : 0;
    const int fe = __shfl_sync(0xffffffffu, first, fl);
    if (lane == 31u) {
      w.carry[row] = t;
      w.head[row] = starts ? fl * E + fe : W::ROW;
    }
  }
  __syncthreads();
  if (warp == 0) {
    T carry = ident;
    for (unsigned int r0 = 0; r0 < rows; r0 += 32) {
      const unsigned int r = r0 + lane;
      const bool in_row = r < rows;
      T t = in_row ? w.carry[r] : ident;
      const unsigned int starts = __ballot_sync(0xffffffffu, in_row && w.head[in_row ? r : 0] < W::ROW);
      t = scl_warp_segscan(t, starts SCL_EXTRA_ARGS);
      const unsigned int below = starts & (0xffffffffu >> (31u - lane));
      if (r0 > 0 && below == 0u) t = SCL_FUNC(carry, t SCL_OP_ARGS);
      const T prev = scl_shfl_up(t, 1);
      if (in_row) w.carry[r] = lane == 0 ? carry : prev;
      carry = scl_shfl_idx(t, 31);
    }
  }
  __syncthreads();
}

// The scanned value at ts[p].
template <int REV, typename T, int TILE>
__device__ __forceinline__ T scl_win_at(const T* ts, unsigned int p, unsigned int P,
                                        const scl_win<T, TILE>& w SCL_USER_PARAMS) {
  typedef scl_win<T, TILE> W;
  const unsigned int l = REV ? (P + W::E - 1) / W::E * W::E - 1 - p : p;
  const unsigned int row = l / W::ROW;
  T v = ts[p];
  if ((int)(l % W::ROW) < w.head[row]) {
    scl_costly_fold();
    v = SCL_FUNC(w.carry[row], v SCL_OP_ARGS);
  }
  return v;
}

// Scans the opened record and stores it: out[e0 - shift + p] for position p,
// 16 bytes at a time where `out` shares the input's 16-byte phase.
template <int REV, int TILE>
__device__ __forceinline__ void scl_scan_window_store(scl_T* ts, scl_u64 e0, int shift, int len, bool inclusive,
                                                      scl_win<scl_T, TILE>& w, scl_O* out SCL_USER_PARAMS) {
  constexpr int B = SCL_SCAN_B;
  typedef scl_win<scl_T, TILE> W;
  constexpr int V = W::V;
  const scl_T ident = (scl_T)(SCL_IDENTITY);
  const unsigned int P = (unsigned int)(shift + len), PT = (P + W::E - 1) / W::E * W::E;
  scl_win_scan<REV, scl_T, TILE, B>(ts, P, ident, w SCL_EXTRA_ARGS);
  const scl_u64 ob = (scl_u64)out + e0 * sizeof(scl_O) - (scl_u64)shift * sizeof(scl_O);
  const bool ovec = sizeof(scl_O) == sizeof(scl_T) && (ob & 15u) == 0;
  for (unsigned int p0 = threadIdx.x * V; p0 < P; p0 += B * V) {
    // (V positions of one lane's chunk: one row; they take the row's carry
    // up to its first start)
    const unsigned int l0 = REV ? PT - 1u - p0 : p0, row = l0 / W::ROW;
    const int d = w.head[row] - (int)(l0 % W::ROW);
    scl_pack<scl_T, V> v = scl_load<scl_T, V>(ts + p0);
    if (REV ? d > 1 - V : d > 0) {
      const scl_T c = w.carry[row];
#pragma unroll
      for (int e = 0; e < V; ++e)
        if (REV ? d > -e : d > e) {
          scl_costly_fold();
          v.v[e] = SCL_FUNC(c, v.v[e] SCL_OP_ARGS);
        }
    }
    scl_pack<scl_O, V> m;
    if (inclusive) {
#pragma unroll
      for (int e = 0; e < V; ++e) m.v[e] = SCL_EPILOGUE(v.v[e]);
    } else {
      // the value before (after, for a reverse scan), or the identity at a start
      scl_T prev = ident;
      if (REV ? p0 + V < P : p0 > 0)
        prev = scl_win_at<REV>(ts, REV ? p0 + V : p0 - 1u, P, w SCL_EXTRA_ARGS);
      const unsigned int bits = w.mask[p0 >> 5] >> (p0 & 31u);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const scl_T before = REV ? (e + 1 < V ? v.v[e + 1 < V ? e + 1 : e] : prev)
                                 : (e > 0 ? v.v[e > 0 ? e - 1 : 0] : prev);
        const scl_T val = (bits >> e) & 1u ? ident : before;
        m.v[e] = SCL_EPILOGUE(val);
      }
    }
    if (ovec && p0 >= (unsigned int)shift && p0 + V <= P) {
      scl_store<scl_O, V>(reinterpret_cast<scl_O*>(ob) + p0, m);
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e)
        if (p0 + e >= (unsigned int)shift && p0 + e < P) out[e0 + (p0 + e - (unsigned int)shift)] = m.v[e];
    }
  }
}

// Window role of a planned segmented scan (the blocks past the tiles; see
// scl_win): the record's vectors are scanned in place and stored in order
// (they cover the record).  The exclusive form starts from SCL_IDENTITY.
template <int TILE>
__device__ __forceinline__ void scl_scan_window_run(const scl_T* in, scl_O* out, const scl_u64* seg_off,
                                                    const scl_u64* win_rec, scl_u64 r, scl_u64 n_rec,
                                                    unsigned int flags, scl_T* ts, unsigned int bar_s,
                                                    unsigned int spin_limit,
                                                    unsigned int* err SCL_USER_PARAMS) {
  constexpr int B = SCL_SCAN_B;
  typedef scl_win<scl_T, TILE> W;
  const bool inclusive = (flags & 1u) != 0, reverse = (flags & 2u) != 0;
  const scl_T ident = (scl_T)(SCL_IDENTITY);
  __shared__ W w;
  const scl_u64 lo = win_rec[4 * r], top = win_rec[4 * r + 1], e0 = win_rec[4 * r + 2];
  const scl_u64 ln = SCL_WIN_ELEMENTS(win_rec[4 * r + 3]);
  const int len = (int)(ln < (scl_u64)TILE ? ln : (scl_u64)TILE);  // (more only for bad offsets)
  if (threadIdx.x == 32 && r + SCL_SCAN_AHEAD < n_rec) {  // (see SCL_SCAN_AHEAD)
    const scl_u64* nr = win_rec + 4 * (r + SCL_SCAN_AHEAD);
    const scl_u64 nl = SCL_WIN_ELEMENTS(nr[3]);
    const scl_u64 a0 = (scl_u64)in + nr[2] * sizeof(scl_T), l0 = nl < (scl_u64)TILE ? nl : (scl_u64)TILE;
    scl_prefetch_l2(a0, a0 + l0 * sizeof(scl_T));
    scl_prefetch_l2((scl_u64)(seg_off + nr[0]), (scl_u64)(seg_off + nr[1] + 1));
  }
  if (len == 0) return;  // (block-uniform) nothing to write for empty vectors
  int shift;
  if (!scl_win_open<scl_T, TILE, B>(in, seg_off, lo, top, e0, len, reverse, ident, ts, w, bar_s, spin_limit,
                                    err, &shift))
    return;
  if (reverse) scl_scan_window_store<1, TILE>(ts, e0, shift, len, inclusive, w, out SCL_EXTRA_ARGS);
  else scl_scan_window_store<0, TILE>(ts, e0, shift, len, inclusive, w, out SCL_EXTRA_ARGS);
}

// The warp-per-segment kernel on its own (segmented launches without a
// segment plan; with one, scl_scan_s<R, MINB, 2> runs the same code in the
// blocks past the tiles).
template <int U>
__global__ void __launch_bounds__(256)
scl_scan_short(const scl_T* in, scl_O* out, const scl_u64* seg_off, scl_u64 n_seg,
               unsigned int flags, scl_u64 short_max SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  scl_scan_short_run<U>(in, out, seg_off, n_seg, flags, short_max,
                        ((scl_u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                        ((scl_u64)gridDim.x * blockDim.x) >> 5 SCL_EXTRA_ARGS);
}
//
// Tiles lie on the 16-byte grid of `in`: with `a` the first element index on
// a 16-byte boundary, a (forward) sequence [lo, hi) starts its first tile at
// lo rounded down onto the grid, and a reverse sequence ends its first tile
// at hi rounded up; elements of a tile outside the sequence are masked with
// the identity (which must be neutral, as for the reference's padding).  So
// every tile's shared-memory image has position p <-> element tile_lo + p,
// 16-byte vector slots, and one bulk copy of the tile's elements, rounded
// out to 16 bytes, when that stays inside the vector.  Elements that cannot
// be aligned (sizes other than 4, 8, 16 bytes, or a misaligned pointer) use
// ordinary loads.  The host counts tiles with the same rule (scl_scan_tiles).
//
// SEG = 1: a segmented scan, one independent scan per segment
// [seg_off[s], seg_off[s+1]) of the flat vector.  Segment s owns the tiles
// tile_start[s] .. tile_start[s+1]-1 (at least one), and the look-back stops
// at the segment's first tile.  Blocks past the last tile (the grid is an
// upper bound) return at once.
// SEG = 2: the same (a segment plan numbered the tiles), and the blocks past
// the tiles scan the segments of at most short_max elements, one window of
// them per block (scl_scan_window_run): one launch for a whole segmented
// scan.
template <int R, int MINB, int SEG = 0>
__global__ void __launch_bounds__(SCL_SCAN_B, MINB)
scl_scan_s(const scl_T* in, scl_O* out, scl_u64 n, unsigned int flags, int aligned,
           unsigned int* tile_counter, scl_scan_status st, scl_scan_clear clr, unsigned int spin_limit,
           unsigned int* err, const scl_u64* seg_off, const unsigned int* tile_start,
           scl_u64 n_seg, scl_u64 short_max, const scl_u64* win_rec,
           const unsigned int* tile_seg, unsigned int n_tiles SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  (void)aligned;
  (void)short_max;
  (void)win_rec;
  (void)tile_seg;
  (void)tile_counter;
  // segmented: the tile count, from the host when a plan knows it (~0u:
  // read it from tile_start[n_seg])
  unsigned int nt = 0;
  if constexpr (SEG != 0) nt = n_tiles != ~0u ? n_tiles : tile_start[n_seg];
  (void)n_tiles;  // (the register kernel's ticket; the host passes both kernels the same arguments)
  constexpr int B = SCL_SCAN_B, W = SCL_SCAN_W;
  constexpr int V = scl_vec_width<sizeof(scl_T)>::value;
  constexpr int TILE = R * B * V;
  // rows of the in-tile scan and a lane's elements in each
  constexpr int M = R % kLaneVectors == 0 ? kLaneVectors : 1, RR = R / M, VV = V * M;
  constexpr unsigned int ROW_BYTES = B * V * sizeof(scl_T);
  constexpr bool natural = sizeof(scl_T) == 4 || sizeof(scl_T) == 8 || sizeof(scl_T) == 16;
  const bool inclusive = (flags & 1u) != 0, reverse = (flags & 2u) != 0;
  const scl_T ident = (scl_T)(SCL_IDENTITY);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  scl_T* ts = reinterpret_cast<scl_T*>(scl_dyn_smem);  // position p <-> element tile_lo + p

  __shared__ __align__(8) unsigned long long bar;
  __shared__ unsigned int s_tile;
  __shared__ int s_ok;
  __shared__ scl_T s_wsum[RR * W];
  __shared__ scl_T s_carry;  // the tile's prefix, converted once to the element type
  const unsigned int bar_s = (unsigned int)__cvta_generic_to_shared(&bar);
  if (threadIdx.x == 0) {
    // the block index is the tile; segmented, the grid is an upper bound
    // and blocks at or past the tile count take no tile
    if constexpr (SEG == 0) {
      s_tile = blockIdx.x;
    } else {
      s_tile = blockIdx.x < nt ? blockIdx.x : 0xffffffffu;
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar_s));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  scl_scan_clear_other(clr);
  if constexpr (SEG == 2) {
    if (blockIdx.x >= nt) {  // (block-uniform: the whole block takes the window role)
      scl_scan_window_run<TILE>(in, out, seg_off, win_rec, blockIdx.x - nt, gridDim.x - nt, flags, ts, bar_s, spin_limit,
                                err SCL_EXTRA_ARGS);
      return;
    }
  }
  __syncthreads();
  const unsigned int tile = s_tile;
  unsigned int first = 0;  // number of the first tile of this tile's sequence
  long long lo = 0, hi = (long long)n;  // the sequence's elements
  if constexpr (SEG != 0) {
    __shared__ long long s_seg;
    if (threadIdx.x == 0) {
      long long sg = -1;
      if (tile < nt) {
        if (tile_seg) {  // (a segment plan's table)
          sg = (long long)tile_seg[tile];
        } else {
          scl_u64 l = 0, h = n_seg - 1;  // largest s with tile_start[s] <= tile
          while (l < h) {
            const scl_u64 mid = (l + h + 1) / 2;
            if (tile_start[mid] <= tile) l = mid; else h = mid - 1;
          }
          sg = (long long)l;
        }
      }
      s_seg = sg;
    }
    __syncthreads();
    if (s_seg < 0) return;
    const scl_u64 sg = (scl_u64)s_seg;
    first = tile_start[sg];
    lo = (long long)seg_off[sg];
    hi = (long long)seg_off[sg + 1];
    if (hi < lo) hi = lo;  // a decreasing offset (reported by the pre-pass)
    if (lo == hi) return;  // an empty segment's only tile: nobody looks back at it
  }
  const long long local = (long long)(tile - first);

  // ---- the tile's place on the grid, its valid elements [c_lo, c_hi)
  const bool grid = natural && ((scl_u64)in % sizeof(scl_T)) == 0;
  const long long vg = grid ? V : 1;
  const long long a = grid ? (long long)(((16u - ((scl_u64)in & 15u)) & 15u) / sizeof(scl_T)) : 0;
  long long tile_lo;
  if (!reverse) {
    const long long m = (((lo - a) % vg) + vg) % vg;
    tile_lo = lo - m + local * TILE;
  } else {
    const long long m = (((a - hi) % vg) + vg) % vg;
    tile_lo = hi + m - (local + 1) * TILE;
  }
  const long long c_lo = tile_lo > lo ? tile_lo : lo;
  const long long c_hi = tile_lo + TILE < hi ? tile_lo + TILE : hi;
  const bool full = c_lo == tile_lo && c_hi == tile_lo + TILE;

  // ---- stage: one bulk copy of [c_lo, c_hi) rounded out to 16 bytes, or loads
  const scl_u64 tbase = (scl_u64)in + (scl_u64)(tile_lo * (long long)sizeof(scl_T));
  const scl_u64 g0 = (scl_u64)in + (scl_u64)c_lo * sizeof(scl_T);
  const scl_u64 g1 = (scl_u64)in + (scl_u64)c_hi * sizeof(scl_T);
  const scl_u64 a0 = g0 & ~(scl_u64)15, a1 = (g1 + 15) & ~(scl_u64)15;
  const scl_u64 vlo = ((scl_u64)in + 15) & ~(scl_u64)15;
  const scl_u64 vhi = ((scl_u64)in + (scl_u64)n * sizeof(scl_T)) & ~(scl_u64)15;
  const bool bulk = grid && a0 >= vlo && a1 <= vhi;
  if (bulk) {
    if (threadIdx.x == 0) {
      const unsigned int bytes = (unsigned int)(a1 - a0);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                   :: "r"(bar_s), "r"(bytes) : "memory");
      const unsigned int dst = (unsigned int)__cvta_generic_to_shared(ts) + (unsigned int)(a0 - tbase);
      if (full) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
              :: "r"(dst + r * ROW_BYTES), "l"((const void*)(a0 + r * ROW_BYTES)), "r"(ROW_BYTES),
                 "r"(bar_s)
              : "memory");
      } else {
        for (unsigned int o = 0; o < bytes; o += ROW_BYTES) {
          const unsigned int sz = bytes - o < ROW_BYTES ? bytes - o : ROW_BYTES;
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
              :: "r"(dst + o), "l"((const void*)(a0 + o)), "r"(sz), "r"(bar_s)
              : "memory");
        }
      }
      // (segments lie in order, so in a segmented scan of either direction the
      // tiles to come lie about as far ahead, once segments fill their tiles)
      if (SEG == 0 || (SEG == 2 && full)) {
        const long long ahead = reverse && SEG == 0 ? tile_lo - (long long)SCL_SCAN_AHEAD * TILE
                                                    : tile_lo + (long long)SCL_SCAN_AHEAD * TILE;
        if (ahead >= 0 && ahead + TILE <= (long long)n) {
          const scl_u64 pa = (scl_u64)in + (scl_u64)ahead * sizeof(scl_T);
          scl_prefetch_l2(pa, pa + TILE * sizeof(scl_T));
        }
      }
      const bool ok = scl_mbar_wait(bar_s, spin_limit);
      if (!ok) {
        scl_raise(err, SCL_DEV_ERR_TIMEOUT);
        // The copies may still land in this block's shared memory: the block
        // stays until they have (bounded by about 0.1 s, whatever the
        // caller's poll limit), and the tile is not used.
        scl_mbar_wait(bar_s, 1u << 21);
      }
      s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    if (!s_ok) return;  // successors time out too and see the error flag
  } else {
    for (int k = threadIdx.x; k < TILE; k += B) {
      const long long i = tile_lo + k;
      ts[k] = (i >= c_lo && i < c_hi) ? in[i] : ident;
    }
    __syncthreads();
  }
  const bool mask = bulk && !full;  // positions outside [c_lo, c_hi) hold other data

  // ---- in-thread inclusive scan of each lane's VV elements (written back to
  //      their slots in logical order), warp scans of the totals.  Logical
  //      group q sits at q*VV, or at TILE-(q+1)*VV reversed for a reverse scan.
  scl_T wincl[RR];  // (unused with local prefixes)
#pragma unroll
  for (int r = 0; r < RR; ++r) {
    const int q = r * B + threadIdx.x;
    const int pos = reverse ? TILE - (q + 1) * VV : q * VV;
    scl_pack<scl_T, VV> p = scl_load_lane<scl_T, V, M>(ts + pos);
    if (mask) {
#pragma unroll
      for (int e = 0; e < VV; ++e) {
        const long long i = tile_lo + pos + e;
        if (i < c_lo || i >= c_hi) p.v[e] = ident;
      }
    }
    if (reverse) {
#pragma unroll
      for (int e = 0; e < VV / 2; ++e) {
        const scl_T t = p.v[e];
        p.v[e] = p.v[VV - 1 - e];
        p.v[VV - 1 - e] = t;
      }
    }
#pragma unroll
    for (int e = 1; e < VV; ++e) p.v[e] = SCL_FUNC(p.v[e - 1], p.v[e] SCL_OP_ARGS);
    if constexpr (kLocalPrefix) {
      const scl_T tot = scl_warp_incl(p.v[VV - 1] SCL_EXTRA_ARGS);
      scl_T lx = scl_shfl_up(tot, 1);
      if (lane == 0) lx = ident;
      if (lane == 31) s_wsum[r * W + warp] = tot;
#pragma unroll
      for (int e = 0; e < VV; ++e) p.v[e] = SCL_FUNC(lx, p.v[e] SCL_OP_ARGS);
      scl_store_lane<scl_T, V, M>(ts + pos, p);
    } else {
      scl_store_lane<scl_T, V, M>(ts + pos, p);
      wincl[r] = scl_warp_incl(p.v[VV - 1] SCL_EXTRA_ARGS);
      if (lane == 31) s_wsum[r * W + warp] = wincl[r];
    }
  }
  __syncthreads();

  // ---- warp 0: tile aggregate, publication and look-back (as scl_scan_k)
  if (warp == 0) {
    scl_T carry = ident;
#pragma unroll
    for (int c = 0; c < (RR * W + 31) / 32; ++c) {
      const int q = c * 32 + lane;
      scl_T v = q < RR * W ? s_wsum[q] : ident;
      scl_T vi = scl_warp_incl(v SCL_EXTRA_ARGS);
      scl_T ve = scl_shfl_up(vi, 1);
      if (lane == 0) ve = ident;
      if (q < RR * W) s_wsum[q] = SCL_FUNC(carry, ve SCL_OP_ARGS);
      scl_T total = scl_shfl_idx(vi, 31);
      carry = SCL_FUNC(carry, total SCL_OP_ARGS);
    }
    const scl_C aggc = (scl_C)carry;
    scl_C prefix = (scl_C)ident;
    if (lane == 0) scl_publish(st, tile, tile == first, aggc);
    if (tile != first) {
      prefix = scl_lookback(st, (long long)tile, (long long)first, spin_limit, err SCL_EXTRA_ARGS);
      if (lane == 0) scl_publish(st, tile, true, (scl_C)SCL_FUNC_C(prefix, aggc SCL_OP_ARGS));
    }
    if (lane == 0) s_carry = (scl_T)prefix;
  }
  __syncthreads();

  // ---- outputs: 16-byte stores for whole slots when `out` shares the grid
  const scl_T tile_carry = s_carry;
  // (whole-slot stores need the output elements the size of the scanned ones)
  const bool ovec = sizeof(scl_O) == sizeof(scl_T) && full &&
                    (((scl_u64)out + (scl_u64)(tile_lo * (long long)sizeof(scl_O))) & 15u) == 0;
#pragma unroll
  for (int r = 0; r < RR; ++r) {
    const int q = r * B + threadIdx.x;
    const int pos = reverse ? TILE - (q + 1) * VV : q * VV;
    scl_pack<scl_T, VV> p = scl_load_lane<scl_T, V, M>(ts + pos);
    scl_pack<scl_T, VV> o;  // logical order
    if constexpr (kLocalPrefix) {
      // the slot holds the warp-local inclusive values
      const scl_T pre = SCL_FUNC(tile_carry, s_wsum[r * W + warp] SCL_OP_ARGS);
      if (inclusive) {
#pragma unroll
        for (int e = 0; e < VV; ++e) o.v[e] = SCL_FUNC(pre, p.v[e] SCL_OP_ARGS);
      } else {
        const scl_T lx = scl_shfl_up(p.v[VV - 1], 1);  // the previous lane's last value
        o.v[0] = lane == 0 ? pre : SCL_FUNC(pre, lx SCL_OP_ARGS);
#pragma unroll
        for (int e = 1; e < VV; ++e) o.v[e] = SCL_FUNC(pre, p.v[e - 1] SCL_OP_ARGS);
      }
    } else {
      scl_T lane_excl = scl_shfl_up(wincl[r], 1);
      if (lane == 0) lane_excl = ident;
      const scl_T pre = SCL_FUNC(SCL_FUNC(tile_carry, s_wsum[r * W + warp] SCL_OP_ARGS),
                                 lane_excl SCL_OP_ARGS);
      if (inclusive) {
#pragma unroll
        for (int e = 0; e < VV; ++e) o.v[e] = SCL_FUNC(pre, p.v[e] SCL_OP_ARGS);
      } else {
        o.v[0] = pre;
#pragma unroll
        for (int e = 1; e < VV; ++e) o.v[e] = SCL_FUNC(pre, p.v[e - 1] SCL_OP_ARGS);
      }
    }
    if (reverse) {  // back to physical order
#pragma unroll
      for (int e = 0; e < VV / 2; ++e) {
        const scl_T t = o.v[e];
        o.v[e] = o.v[VV - 1 - e];
        o.v[VV - 1 - e] = t;
      }
    }
    scl_pack<scl_O, VV> m;
#pragma unroll
    for (int e = 0; e < VV; ++e) m.v[e] = SCL_EPILOGUE(o.v[e]);
    if (ovec) {
      scl_store_lane<scl_O, V, M>(out + (tile_lo + pos), m);
    } else {
#pragma unroll
      for (int e = 0; e < VV; ++e) {
        const long long i = tile_lo + pos + e;
        if (i >= c_lo && i < c_hi) out[i] = m.v[e];
      }
    }
  }
}

#endif
