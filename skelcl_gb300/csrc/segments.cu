// Segmented launches (no counterpart in the reference): thousands of
// vectors of uneven length stored back to back in one flat buffer, segment s
// = [seg_offsets[s], seg_offsets[s+1]), processed by one launch per skeleton
// and length class.
//
// segments_prepare() is the pre-pass of the segmented Scan and Reduce, three
// small launches: it copies the caller's offsets into the program workspace
// clamped to the buffer (raising a device status bit if an offset lies past
// the buffer or decreases; every consumer reads segment s as
// [off[s], max(off[s], off[s+1])), so no access leaves the buffer), and
// numbers the tiles of the segments longer than `short_max` elements:
// segment s owns tiles tile_start[s] .. tile_start[s+1]-1, so no tile spans
// two segments: ceil(len / tile) of them, or, for tiles laid on a grid of vg
// elements with phase a (the scan's 16-byte grid), as many as cover the
// segment once its start (end, for a reverse scan) is rounded onto the grid.
// Shorter segments, empty ones included, get no tiles: one warp each handles
// them in a separate kernel.  tile_start[n_segments] is the tile count.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>

#include "internal.h"

namespace scl {
namespace {

constexpr int kPrepThreads = 1024;

__device__ __forceinline__ uint64_t warp_incl_max(uint64_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o && u > v) v = u;
  }
  return v;
}
__device__ __forceinline__ uint64_t warp_incl_sum(uint64_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}
// Block-wide inclusive scan (max or sum) of one value per thread.
template <bool MAX>
__device__ uint64_t block_incl(uint64_t v, uint64_t* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = MAX ? warp_incl_max(v) : warp_incl_sum(v);
  if (lane == 31) s_warp[warp] = v;
  __syncthreads();
  if (warp == 0) {
    uint64_t w = s_warp[lane];
    w = MAX ? warp_incl_max(w) : warp_incl_sum(w);
    s_warp[lane] = w;
  }
  __syncthreads();
  if (warp > 0) {
    const uint64_t p = s_warp[warp - 1];
    v = MAX ? (p > v ? p : v) : v + p;
  }
  __syncthreads();
  return v;
}

constexpr int kSegThreads = 256, kSegPerThread = 8;
constexpr uint64_t kSegPerBlock = (uint64_t)kSegThreads * kSegPerThread;

// Tiles of a segment [lo, hi) (hi >= lo): none when it is short.
__device__ __forceinline__ uint64_t seg_tiles(uint64_t lo, uint64_t hi, uint64_t tile, uint64_t vg,
                                              uint64_t a, int reverse, uint64_t short_max) {
  const uint64_t len = hi - lo;
  if (len <= short_max) return 0;
  // the segment's first tile starts (ends, reverse) on the grid {a + k*vg}
  const uint64_t m = reverse ? (a + vg - hi % vg) % vg : (lo + vg - a) % vg;
  return (len + m + tile - 1) / tile;
}

// 1. clamp the offsets (written to off_out unless it is null), count each
//    segment's tiles, one sum per block
__global__ void __launch_bounds__(kSegThreads)
seg_clamp_count_kernel(const uint64_t* off_in, uint64_t n_seg, uint64_t n_total, uint64_t tile,
                       uint64_t vg, uint64_t a, int reverse, uint64_t short_max, uint64_t* off_out,
                       uint64_t* block_sums, unsigned int* err) {
  __shared__ uint64_t s_warp[32];
  const uint64_t s0 = (uint64_t)blockIdx.x * kSegPerBlock + (uint64_t)threadIdx.x * kSegPerThread;
  uint64_t sum = 0;
  bool bad = false;
#pragma unroll
  for (int k = 0; k < kSegPerThread; ++k) {
    const uint64_t sg = s0 + k;
    if (sg >= n_seg) break;
    const uint64_t rlo = off_in[sg], rhi = off_in[sg + 1];
    bad = bad || rlo > n_total || rhi < rlo;
    const uint64_t lo = rlo < n_total ? rlo : n_total;
    uint64_t hi = rhi < n_total ? rhi : n_total;
    if (hi < lo) hi = lo;
    if (off_out) off_out[sg] = lo;
    if (sg + 1 == n_seg) {
      if (off_out) off_out[n_seg] = rhi < n_total ? rhi : n_total;
      bad = bad || rhi > n_total;
    }
    sum += seg_tiles(lo, hi, tile, vg, a, reverse, short_max);
  }
  if (bad && err) atomicOr(err, kDevErrSegments);
  const uint64_t incl = block_incl<false>(sum, s_warp);
  if (threadIdx.x == kSegThreads - 1) block_sums[blockIdx.x] = incl;
}

// 2. exclusive sum over the blocks' sums (one block); the total at [nb]
__global__ void __launch_bounds__(kPrepThreads)
seg_scan_sums_kernel(uint64_t* block_sums, uint64_t nb) {
  __shared__ uint64_t s_warp[32];
  __shared__ uint64_t s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (uint64_t c = 0; c < nb; c += kPrepThreads) {
    const uint64_t b = c + threadIdx.x;
    const uint64_t v = b < nb ? block_sums[b] : 0;
    const uint64_t incl = block_incl<false>(v, s_warp);
    const uint64_t carry = s_carry;
    if (b < nb) block_sums[b] = carry + incl - v;
    __syncthreads();
    if (threadIdx.x == kPrepThreads - 1) s_carry = carry + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) block_sums[nb] = s_carry;
}

// 3. every segment's first tile
__global__ void __launch_bounds__(kSegThreads)
seg_tile_start_kernel(const uint64_t* off, uint64_t n_seg, uint64_t tile, uint64_t vg, uint64_t a,
                      int reverse, uint64_t short_max, const uint64_t* block_sums, uint64_t nb,
                      unsigned int* tile_start) {
  __shared__ uint64_t s_warp[32];
  const uint64_t s0 = (uint64_t)blockIdx.x * kSegPerBlock + (uint64_t)threadIdx.x * kSegPerThread;
  uint64_t cnt[kSegPerThread], sum = 0;
#pragma unroll
  for (int k = 0; k < kSegPerThread; ++k) {
    const uint64_t sg = s0 + k;
    cnt[k] = 0;
    if (sg < n_seg) {
      const uint64_t lo = off[sg];
      uint64_t hi = off[sg + 1];
      if (hi < lo) hi = lo;
      cnt[k] = seg_tiles(lo, hi, tile, vg, a, reverse, short_max);
    }
    sum += cnt[k];
  }
  const uint64_t incl = block_incl<false>(sum, s_warp);
  uint64_t start = block_sums[blockIdx.x] + incl - sum;
#pragma unroll
  for (int k = 0; k < kSegPerThread; ++k) {
    const uint64_t sg = s0 + k;
    if (sg < n_seg) tile_start[sg] = (unsigned int)start;
    start += cnt[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) tile_start[n_seg] = (unsigned int)block_sums[nb];
}

// gx[i] (+)= g[s] for every element i of segment s (elements outside every
// segment are left alone).  A block takes a run of consecutive chunks of CH
// elements.  It finds the last segment starting at or before the run (256
// probes per round) and then walks the segments from chunk to chunk: it marks
// in a bit mask where the chunk's non-empty segments start, keeps their values
// in order, and gives every element the value of the last start at or below
// it: the mask's running count, one count per word and a popcount.  The next
// chunk's first 256 segments are read while this one is stored.  Bound by
// memory (4 bytes an element): 10^6 vectors of 1..199 floats 0.123 -> 0.081 ms,
// 10^7 of 0..2 0.651 -> 0.116 ms, against broadcast_long_segments_kernel (a
// search per chunk instead of per run: 0.107 and 0.137 ms).
template <typename T>
struct BroadcastChunk {
  static constexpr int WORDS = 1024 / sizeof(T);  // mask words, one per thread at most
  static constexpr int CH = WORDS * 32 - 32;      // a word to spare for gx's 16-byte phase
};
template <typename T>
__global__ void __launch_bounds__(256)
broadcast_segments_kernel(const T* g, T* gx, const uint64_t* off,
                          uint64_t n_seg, uint64_t n_total, int acc, uint64_t run) {
  constexpr int WORDS = BroadcastChunk<T>::WORDS, CH = BroadcastChunk<T>::CH, V = 16 / sizeof(T);
  __shared__ unsigned int mask[WORDS];  // bit p: a segment starts at position p
  __shared__ int before[WORDS];         // starts below the word
  __shared__ int warp_sum[8];
  __shared__ int cov_lo, cov_hi;        // positions covered by segments
  __shared__ unsigned long long last;   // last segment that starts in or before the chunk
  __shared__ T val[CH];                 // the segments' values, in order
  const int tid = threadIdx.x, lane = tid & 31;
  // position p = element c0 + p - phase, so that positions and gx share
  // their 16-byte phase (CH is a multiple of V)
  const int phase = (int)((reinterpret_cast<uintptr_t>(gx) & 15u) / sizeof(T));
  dependency_wait();
  uint64_t c0 = (uint64_t)blockIdx.x * run * CH;
  const uint64_t end = c0 + run * CH < n_total ? c0 + run * CH : n_total;
  if (c0 >= end) return;  // (block-uniform)
  // last segment with off[s] <= c0 (0 if none): each round 256 offsets spread
  // over [lo, hi] are probed and the count at or below c0 narrows it
  // (decreasing offsets still end the search)
  uint64_t lo = 0, hi = n_seg - 1;
  while (lo < hi) {  // (block-uniform)
    const uint64_t span = hi - lo;
    const int below = __syncthreads_count(off[lo + 1 + span * (uint64_t)tid / 256] <= c0);
    if (below == 0) {
      hi = lo;
    } else {
      const uint64_t at = lo + 1 + span * (uint64_t)(below - 1) / 256;
      hi = below < 256 ? lo + span * (uint64_t)below / 256 : hi;
      lo = at;
    }
  }
  // segment lo + tid: its offsets and value
  uint64_t a = ~0ull, b = 0;
  T v = T(0);
  auto fetch = [&](uint64_t s) {
    a = ~0ull;
    if (s < n_seg) {
      a = off[s];
      b = off[s + 1];
      v = g[s];
    }
  };
  fetch(lo + tid);
  for (; c0 < end; c0 += CH) {  // (block-uniform)
    const uint64_t c1 = c0 + CH < end ? c0 + CH : end;
    if (tid < WORDS) mask[tid] = 0u;
    if (tid == 0) {
      cov_lo = CH + V;
      cov_hi = 0;
      last = lo;
    }
    __syncthreads();
    // the part [i0, i1) of the chunk, as positions, of the segment at hand
    auto part = [&](int* i0, int* i1) {
      *i0 = *i1 = 0;
      if (a >= c1) return;
      const uint64_t x0 = a > c0 ? a : c0, x1 = b < c1 ? b : c1;
      if (x0 < x1) {
        *i0 = (int)(x0 - c0) + phase;
        *i1 = (int)(x1 - c0) + phase;
      }
    };
    int f0 = 0, f1 = 0;  // this thread's first segment
    const T fv = v;
    bool many = false;   // more than 256 segments
    for (uint64_t base = lo;; base += 256) {  // (block-uniform)
      int i0, i1;
      part(&i0, &i1);
      if (base == lo) {
        f0 = i0;
        f1 = i1;
      }
      if (i0 < i1) atomicOr(&mask[i0 >> 5], 1u << (i0 & 31));
      const int wl = __reduce_min_sync(0xffffffffu, i0 < i1 ? i0 : CH + V);
      const int wh = __reduce_max_sync(0xffffffffu, i1);
      const unsigned int starts = __ballot_sync(0xffffffffu, a < c1);
      if (lane == 0) {
        if (wh > 0) {
          atomicMin(&cov_lo, wl);
          atomicMax(&cov_hi, wh);
        }
        if (starts) atomicMax(&last, (unsigned long long)(base + tid + 31 - __clz((int)starts)));
      }
      if (!__syncthreads_or(tid == 255 && a < c1)) break;
      many = true;
      fetch(base + 256 + tid);
    }
    // starts below each word
    const int cnt = tid < WORDS ? __popc(mask[tid]) : 0;
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    if (lane == 31) warp_sum[tid >> 5] = incl;
    __syncthreads();
    int base_cnt = 0;
    for (int w = 0; w < (tid >> 5); ++w) base_cnt += warp_sum[w];
    if (tid < WORDS) before[tid] = base_cnt + incl - cnt;
    __syncthreads();
    // the last start at or below position p
    auto rank = [&](int p) { return before[p >> 5] + __popc(mask[p >> 5] & (0xffffffffu >> (31 - (p & 31)))) - 1; };
    if (f0 < f1) val[rank(f0)] = fv;
    const uint64_t next = last;
    if (many) {
      for (uint64_t base = lo + 256; base <= next; base += 256) {  // (block-uniform)
        fetch(base + tid);
        int i0, i1;
        part(&i0, &i1);
        if (i0 < i1) val[rank(i0)] = v;
      }
    }
    lo = next;
    fetch(lo + tid);  // the next chunk's
    __syncthreads();
    T* const out = gx + c0 - phase;
    const int lo_p = cov_lo, hi_p = cov_hi;
    for (int p = (lo_p / V + tid) * V; p < hi_p; p += 256 * V) {
      if (p >= lo_p && p + V <= hi_p) {
        int r = rank(p);
        const unsigned int starts = (mask[p >> 5] >> (p & 31)) >> 1;  // at p + 1 ..
        T x[V];
        x[0] = val[r];
#pragma unroll
        for (int e = 1; e < V; ++e) {
          r += (int)((starts >> (e - 1)) & 1u);
          x[e] = val[r];
        }
        if (acc) {
          const uint4 w = *reinterpret_cast<const uint4*>(out + p);
          T y[V];
          memcpy(y, &w, 16);
#pragma unroll
          for (int e = 0; e < V; ++e) x[e] += y[e];
        }
        uint4 w;
        memcpy(&w, x, 16);
        *reinterpret_cast<uint4*>(out + p) = w;
      } else {
        for (int e = 0; e < V; ++e)
          if (p + e >= lo_p && p + e < hi_p) {
            const T u = val[rank(p + e)];
            out[p + e] = acc ? out[p + e] + u : u;
          }
      }
    }
    __syncthreads();
  }
}

// The same for long segments: each warp takes a chunk of CH elements: it finds
// the last segment starting at or before the chunk (a search of the warp, 32
// probes per round), then walks the segments that start before the chunk's
// end, the offsets and values of 32 of them read at once, and writes each
// one's part of the chunk with lane-strided stores (16 bytes at a time when
// gx is 16-byte aligned, single elements at the part's ragged ends).
constexpr int kBroadcastWarp = 1024;
template <typename T>
__global__ void __launch_bounds__(256)
broadcast_long_segments_kernel(const T* g, T* gx, const uint64_t* off,
                          uint64_t n_seg, uint64_t n_total, int acc, int aligned) {
  constexpr int CH = kBroadcastWarp, V = 16 / sizeof(T);
  dependency_wait();
  const int lane = threadIdx.x & 31;
  const uint64_t c0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * CH;
  if (c0 >= n_total) return;  // (warp-uniform)
  const uint64_t c1 = c0 + CH < n_total ? c0 + CH : n_total;
  // last segment with off[s] <= c0 (0 if none): each round the lanes probe 32
  // offsets spread over [lo, hi] and the count at or below c0 narrows it (by
  // 32 for increasing offsets; decreasing ones still end the search)
  uint64_t lo = 0, hi = n_seg - 1;
  while (lo < hi) {  // (warp-uniform)
    const uint64_t span = hi - lo;
    const uint64_t p = lo + 1 + span * (uint64_t)lane / 32;
    const int below = __popc(__ballot_sync(0xffffffffu, off[p] <= c0));
    if (below == 0) {
      hi = lo;
    } else {
      const uint64_t p_last = lo + 1 + span * (uint64_t)(below - 1) / 32;
      hi = below < 32 ? lo + span * (uint64_t)below / 32 : hi;
      lo = p_last;
    }
  }
  // this warp's part [r0, r1) of one segment, value v, as offsets from c0
  // (a multiple of CH, so offsets and indices share their 16-byte phase)
  T* const base = gx + c0;
  auto one = [&](int r, T v) { base[r] = acc ? base[r] + v : v; };
  auto put = [&](int r0, int r1, T v) {
    if (!aligned) {
      for (int r = r0 + lane; r < r1; r += 32) one(r, v);
      return;
    }
    const int h0 = (r0 + V - 1) & ~(V - 1);
    const int h = h0 < r1 ? h0 : r1;                        // end of the ragged head
    const int t0 = r1 & ~(V - 1), t = t0 > h ? t0 : h;      // start of the ragged tail
    if (r0 + lane < h) one(r0 + lane, v);
    for (int q = h + lane * V; q < t; q += 32 * V) {
      T r[V];
      if (acc) {
        const uint4 w = *reinterpret_cast<const uint4*>(base + q);
        memcpy(r, &w, 16);
#pragma unroll
        for (int e = 0; e < V; ++e) r[e] += v;
      } else {
#pragma unroll
        for (int e = 0; e < V; ++e) r[e] = v;
      }
      uint4 w;
      memcpy(&w, r, 16);
      *reinterpret_cast<uint4*>(base + q) = w;
    }
    if (t + lane < r1) one(t + lane, v);
  };
  for (uint64_t sb = lo; sb < n_seg; sb += 32) {
    const uint64_t my = sb + lane;
    uint64_t a_l = n_total, b_l = n_total;
    T v_l = T(0);
    if (my < n_seg) {
      a_l = off[my];
      b_l = off[my + 1];
      v_l = g[my];
    }
    const int cnt = n_seg - sb < 32 ? (int)(n_seg - sb) : 32;
    bool past = false;
    for (int k = 0; k < cnt; ++k) {
      const uint64_t a = __shfl_sync(0xffffffffu, a_l, k), b0 = __shfl_sync(0xffffffffu, b_l, k);
      const T v = __shfl_sync(0xffffffffu, v_l, k);
      if (a >= c1) {  // this and (for increasing offsets) every later segment start past the chunk
        past = true;
        break;
      }
      const uint64_t b = b0 > a ? b0 : a;
      const uint64_t i0 = a > c0 ? a : c0, i1 = b < c1 ? b : c1;
      if (i0 < i1) put((int)(i0 - c0), (int)(i1 - c0), v);
    }
    if (past) break;
  }
}

// tile_seg[t] = s for every tile t of segment s (tiles tile_start[s] ..
// tile_start[s+1]-1), one thread per segment.
__global__ void __launch_bounds__(256) seg_tile_owner_kernel(const unsigned int* __restrict__ tile_start,
                                                             uint64_t n_seg, unsigned int* __restrict__ tile_seg) {
  for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n_seg;
       s += (uint64_t)gridDim.x * blockDim.x)
    for (unsigned int t = tile_start[s]; t < tile_start[s + 1]; ++t) tile_seg[t] = (unsigned int)s;
}

}  // namespace

size_t segments_prepare_scratch(uint64_t n_seg) {
  return ((n_seg + kSegPerBlock - 1) / kSegPerBlock + 1) * sizeof(uint64_t);
}

int segments_prepare(const uint64_t* seg_offsets, uint64_t n_seg, uint64_t n_total, uint64_t tile,
                     uint64_t vg, uint64_t a, int reverse, uint64_t short_max, uint64_t* off_out,
                     unsigned int* tile_start, uint64_t* scratch, cudaStream_t stream) {
  const uint64_t nb = (n_seg + kSegPerBlock - 1) / kSegPerBlock;
  if (nb == 0) return SCL_OK;
  if (nb > 0x7fffffffull) return fail(SCL_ERR_ARG, "too many segments");
  // off_out == seg_offsets: the offsets are already clamped; number the
  // tiles without writing them again
  seg_clamp_count_kernel<<<(unsigned)nb, kSegThreads, 0, stream>>>(
      seg_offsets, n_seg, n_total, tile, vg, a, reverse, short_max,
      off_out == seg_offsets ? nullptr : off_out, scratch, rt().dev_err);
  seg_scan_sums_kernel<<<1, kPrepThreads, 0, stream>>>(scratch, nb);
  seg_tile_start_kernel<<<(unsigned)nb, kSegThreads, 0, stream>>>(off_out, n_seg, tile, vg, a, reverse,
                                                                  short_max, scratch, nb, tile_start);
  SCL_CUDA(cudaGetLastError());
  rt().launches += 3;
  return SCL_OK;
}

// ---- segment plans ------------------------------------------------------------
namespace {
std::mutex g_plan_mu;
std::map<uint32_t, std::unique_ptr<SegPlan>> g_plans;
uint32_t g_next_plan = 1;

void free_plan(SegPlan* p) {
  if (!rt().initialized) return;
  cudaStreamSynchronize(rt().stream);
  cudaFree(p->off);
  cudaFree(p->tickets);
  cudaFree(p->scratch);
  for (auto& c : p->cfgs) {
    cudaFree(c.tile_start);
    cudaFree(c.tile_seg);
  }
  for (auto& r : p->records) cudaFree(r.rec);
}
}  // namespace

// Window records of the short segments: consecutive segments of at most
// short_max elements that start in the same window of `window` >= short_max
// elements form one record {first segment, end segment, first element,
// elements}; longer segments belong to the tiles and end the record before
// them.  All but the last segment of a record end inside its window, so a
// record spans less than window + short_max elements.  Records whose segments
// are all empty stay (the Reduce writes their identities); windows that own
// no segment get none.  `off` holds n_seg + 1 clamped offsets.
// each(first, end, first element, elements, longest segment's length).
template <typename Each>
static void walk_window_records(const uint64_t* off, uint64_t n_seg, uint64_t short_max, uint64_t window,
                                const Each& each) {
  for (uint64_t sg = 0; sg < n_seg;) {
    const uint64_t e0 = off[sg];
    uint64_t lo = e0, hi = off[sg + 1];  // the segment at hand
    uint64_t len = hi > lo ? hi - lo : 0;
    if (len > short_max) {
      ++sg;
      continue;
    }
    const uint64_t w0 = e0 / window * window;
    uint64_t top = sg + 1, last = lo + len, longest = len;
    while (top < n_seg) {
      lo = hi;
      hi = off[top + 1];
      len = hi > lo ? hi - lo : 0;
      if (lo - w0 >= window || len > short_max) break;
      last = lo + len;
      longest = std::max(longest, len);
      ++top;
    }
    each(sg, top, e0, last > e0 ? last - e0 : 0, longest);
    sg = top;
  }
}
void segplan_window_records(const uint64_t* off, uint64_t n_seg, uint64_t short_max, uint64_t window,
                            std::vector<uint64_t>* rec) {
  rec->clear();
  walk_window_records(off, n_seg, short_max, window,
                      [&](uint64_t first, uint64_t end, uint64_t e0, uint64_t elements, uint64_t) {
                        rec->insert(rec->end(), {first, end, e0, elements});
                      });
}

namespace {
// The plan's records for these limits, built on the host at first use.
int segplan_records(SegPlan* p, uint64_t short_max, uint64_t window, const SegPlanRecords** out) {
  for (auto& r : p->records)
    if (r.short_max == short_max && r.window == window) {
      *out = &r;
      return SCL_OK;
    }
  if (p->host_off.empty()) {
    std::vector<uint64_t> off(p->n_seg + 1);
    SCL_CUDA(cudaMemcpyAsync(off.data(), p->off, off.size() * sizeof(uint64_t), cudaMemcpyDeviceToHost,
                             rt().stream));
    SCL_CUDA(cudaStreamSynchronize(rt().stream));
    p->host_off.swap(off);
  }
  std::vector<uint64_t> rec;
  // the kernels find the longest vector's length above the elements (below 2^32:
  // a tile's)
  walk_window_records(p->host_off.data(), p->n_seg, short_max, window,
                      [&](uint64_t first, uint64_t end, uint64_t e0, uint64_t elements, uint64_t longest) {
                        rec.insert(rec.end(), {first, end, e0, elements | longest << 32});
                      });
  SegPlanRecords r;
  r.short_max = short_max;
  r.window = window;
  r.n_rec = rec.size() / 4;
  if (r.n_rec) {
    rt().device_allocs++;
    cudaError_t e = cudaMalloc(&r.rec, rec.size() * sizeof(uint64_t));
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(r.rec, rec.data(), rec.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, rt().stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(rt().stream);
    if (e != cudaSuccess) {
      cudaFree(r.rec);
      return cuda_fail(e, "segment plan: window records");
    }
  }
  p->records.push_back(r);
  *out = &p->records.back();
  return SCL_OK;
}
}  // namespace

SegPlan* segplan_find(uint32_t id) {
  std::lock_guard<std::mutex> g(g_plan_mu);
  auto it = g_plans.find(id);
  return it == g_plans.end() ? nullptr : it->second.get();
}

int segplan_config(SegPlan* p, uint64_t tile, uint64_t vg, uint64_t a, int reverse, uint64_t short_max,
                   uint64_t window, const SegPlanCfg** out) {
  for (auto& c : p->cfgs)
    if (c.tile == tile && c.vg == vg && c.a == a && c.reverse == reverse && c.short_max == short_max &&
        c.window == window) {
      *out = &c;
      return SCL_OK;
    }
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  SCL_CUDA(cudaStreamIsCapturing(rt().stream, &capture));
  if (capture != cudaStreamCaptureStatusNone)
    return fail(SCL_ERR_ARG,
                "segment plan: this tile shape is first used inside a stream capture; make the call "
                "once before capturing (building its tile numbering reads the tile count back)");
  SegPlanCfg c;
  c.tile = tile;
  c.vg = vg;
  c.a = a;
  c.reverse = reverse;
  c.short_max = short_max;
  c.window = window;
  const SegPlanRecords* rec = nullptr;
  if (int st = segplan_records(p, short_max, window, &rec)) return st;
  c.n_rec = rec->n_rec;
  c.win_rec = rec->rec;
  rt().device_allocs++;
  SCL_CUDA(cudaMalloc(&c.tile_start, (p->n_seg + 1) * sizeof(unsigned int)));
  if (int st = segments_prepare(p->off, p->n_seg, p->n_total, tile, vg, a, reverse, short_max, p->off,
                                c.tile_start, p->scratch, rt().stream)) {
    cudaFree(c.tile_start);
    return st;
  }
  unsigned int tiles = 0;
  SCL_CUDA(cudaMemcpyAsync(&tiles, c.tile_start + p->n_seg, sizeof(tiles), cudaMemcpyDeviceToHost,
                           rt().stream));
  SCL_CUDA(cudaStreamSynchronize(rt().stream));
  c.tiles = tiles;
  // each tile's segment, so that a tile finds its segment with one load
  if (tiles) {
    rt().device_allocs++;
    cudaError_t e = cudaMalloc(&c.tile_seg, (size_t)tiles * sizeof(unsigned int));
    if (e == cudaSuccess) {
      const uint64_t nb = std::min<uint64_t>((p->n_seg + 255) / 256, 65535);
      seg_tile_owner_kernel<<<(unsigned)nb, 256, 0, rt().stream>>>(c.tile_start, p->n_seg, c.tile_seg);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
      cudaFree(c.tile_start);
      cudaFree(c.tile_seg);
      return cuda_fail(e, "segment plan: tile owners");
    }
  }
  p->cfgs.push_back(c);
  *out = &p->cfgs.back();
  return SCL_OK;
}

}  // namespace scl

using namespace scl;

extern "C" int scl_segplan_create(const uint64_t* seg_offsets, uint64_t n_segments, uint64_t n,
                                  uint32_t* plan) {
  if (int st = require_init()) return st;
  if (!plan) return fail(SCL_ERR_ARG, "scl_segplan_create: null plan");
  *plan = 0;
  if (!seg_offsets || n_segments == 0) return fail(SCL_ERR_ARG, "scl_segplan_create: no segments");
  const uint64_t nb = (n_segments + kSegPerBlock - 1) / kSegPerBlock;
  if (nb > 0x7fffffffull) return fail(SCL_ERR_ARG, "scl_segplan_create: too many segments");
  std::unique_ptr<SegPlan> p(new SegPlan);
  p->n_seg = n_segments;
  p->n_total = n;
  rt().device_allocs += 3;
  cudaError_t e = cudaMalloc(&p->off, (n_segments + 1) * sizeof(uint64_t));
  if (e == cudaSuccess) e = cudaMalloc(&p->tickets, n_segments * sizeof(unsigned int));
  if (e == cudaSuccess) e = cudaMalloc(&p->scratch, segments_prepare_scratch(n_segments));
  if (e == cudaSuccess) e = cudaMemsetAsync(p->tickets, 0, n_segments * sizeof(unsigned int), rt().stream);
  if (e != cudaSuccess) {
    free_plan(p.get());
    cudaGetLastError();
    return fail(SCL_ERR_OOM, "scl_segplan_create: device memory for the plan");
  }
  // the clamped copy of the offsets (no tiles counted yet)
  seg_clamp_count_kernel<<<(unsigned)nb, kSegThreads, 0, rt().stream>>>(
      seg_offsets, n_segments, n, ~0ull, 1, 0, 0, ~0ull, p->off, p->scratch, rt().dev_err);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    free_plan(p.get());
    return cuda_fail(e, "segment plan: clamp kernel");
  }
  ++rt().launches;
  std::lock_guard<std::mutex> g(g_plan_mu);
  p->id = g_next_plan++;
  if (g_next_plan == 0) g_next_plan = 1;
  *plan = p->id;
  g_plans[p->id] = std::move(p);
  return SCL_OK;
}

extern "C" int scl_segplan_release(uint32_t plan) {
  std::unique_ptr<SegPlan> p;
  {
    std::lock_guard<std::mutex> g(g_plan_mu);
    auto it = g_plans.find(plan);
    if (it == g_plans.end()) return plan == 0 ? SCL_OK : fail(SCL_ERR_ARG, "scl_segplan_release: no such plan");
    p = std::move(it->second);
    g_plans.erase(it);
  }
  free_plan(p.get());
  return SCL_OK;
}

extern "C" int scl_adjoint_broadcast_segments(const void* g, void* gx, const uint64_t* seg_offsets,
                                              uint64_t n_segments, uint64_t n, int dtype,
                                              int accumulate) {
  if (int st = require_init()) return st;
  if (dtype != SCL_DTYPE_F32 && dtype != SCL_DTYPE_F64)
    return fail(SCL_ERR_ARG, "segmented broadcast: dtype must be SCL_DTYPE_F32 or _F64");
  if (n == 0 || n_segments == 0) return SCL_OK;
  if (!g || !gx || !seg_offsets) return fail(SCL_ERR_ARG, "segmented broadcast: null pointer");
  const int acc = accumulate ? 1 : 0;
  // a warp per 1024 elements walks long segments at the speed of plain stores,
  // but spends 40 instructions an element on short ones: 10^8 floats in
  // vectors of 100 on average 123 us against 81 for the chunks, of 300 64
  // against 70, of 1500 62 against 70.  Of doubles, whose chunks have half as many
  // elements, plain stores win from 48 on (10^7 in vectors of 32 on average 37
  // against 27, of 50 26.3 / 26.9, of 100 15.7 / 26.4), added ones later (of 50 59
  // against 32, of 150 37 / 31)
  const bool long_segments = n / n_segments >= (dtype == SCL_DTYPE_F64 && !acc ? 48u : 200u);
  if (long_segments) {
    const uint64_t blocks = (n + 8 * kBroadcastWarp - 1) / (8 * kBroadcastWarp);
    if (blocks > 0x7fffffffull) return fail(SCL_ERR_ARG, "segmented broadcast: vector too large");
    const dim3 grid((unsigned)blocks);
    const int aligned = (reinterpret_cast<uintptr_t>(gx) & 15u) == 0 ? 1 : 0;
    SCL_CUDA(dtype == SCL_DTYPE_F32
                 ? launch_overlapped(broadcast_long_segments_kernel<float>, grid, dim3(256), 0, rt().stream,
                                     (const float*)g, (float*)gx, seg_offsets, n_segments, n, acc, aligned)
                 : launch_overlapped(broadcast_long_segments_kernel<double>, grid, dim3(256), 0, rt().stream,
                                     (const double*)g, (double*)gx, seg_offsets, n_segments, n, acc, aligned));
    return SCL_OK;
  }
  // one wave of blocks (6 per SM by their shared memory), each a run of chunks
  const uint64_t chunk = dtype == SCL_DTYPE_F32 ? BroadcastChunk<float>::CH : BroadcastChunk<double>::CH;
  const uint64_t chunks = (n + chunk - 1) / chunk, wave = sm_count() * 6;
  const uint64_t run = (chunks + wave - 1) / wave, blocks = (chunks + run - 1) / run;
  const dim3 grid((unsigned)blocks);
  SCL_CUDA(dtype == SCL_DTYPE_F32
               ? launch_overlapped(broadcast_segments_kernel<float>, grid, dim3(256), 0, rt().stream,
                                   (const float*)g, (float*)gx, seg_offsets, n_segments, n, acc, run)
               : launch_overlapped(broadcast_segments_kernel<double>, grid, dim3(256), 0, rt().stream,
                                   (const double*)g, (double*)gx, seg_offsets, n_segments, n, acc, run));
  return SCL_OK;
}

extern "C" int scl_debug_window_records(const uint64_t* offsets, uint64_t n_segments, uint64_t short_max,
                                        uint64_t* records, uint64_t capacity, uint64_t* count) {
  if (!offsets || !count) return fail(SCL_ERR_ARG, "scl_debug_window_records: null argument");
  if (short_max == 0) return fail(SCL_ERR_ARG, "scl_debug_window_records: short_max must be positive");
  std::vector<uint64_t> rec;
  segplan_window_records(offsets, n_segments, short_max, short_max, &rec);
  *count = rec.size() / 4;
  if (records) {
    if (capacity < *count) return fail(SCL_ERR_ARG, "scl_debug_window_records: capacity too small");
    std::memcpy(records, rec.data(), rec.size() * sizeof(uint64_t));
  }
  return SCL_OK;
}
