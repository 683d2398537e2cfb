// ---------------------------------------------------------------------------
// MapOverlap for sm_103a: 2D stencil over a row-major matrix.
//
// Reference: SCL_MAPOVERLAP (include/SkelCL/detail/MapOverlapKernel.cl:59-148)
// with the OL distribution's host-built padding rows
// (include/SkelCL/detail/OLDistributionDef.h:264-343).  Net semantics:
//   out[y][x] = f(view), getData(view, dx, dy) = in'[y+dy][x+dx]
// where in' is `in` extended by R on every side with
//   NEAREST: in[clamp(y+dy)][clamp(x+dx)]  (corners included)
//   NEUTRAL: the neutral element.
// dx runs along columns, dy along rows (test/MapOverlapTests.cpp:187-216).
// Here both axes are padded in-kernel; no padded copy of the matrix exists.
//
// Shape: a block of 32 x 8 threads owns a 32-column x (8*PY)-row output tile
// and stages the (8*PY+2R) x SCL_WIN_W input window in shared memory, either
// with one TMA 2D tile load (OOB elements filled with zero, then patched for
// NEAREST / non-zero NEUTRAL) or with cooperative coalesced loads.  Each
// thread computes PY vertically adjacent outputs; with the user loops
// unrolled, taps shared between those outputs and the user's weight loads
// are read once per thread instead of once per output.
// Generated names: SCL_OVERLAP_RANGE, SCL_PADDING (0 neutral, 1 nearest),
// SCL_NEUTRAL, SCL_NEUTRAL_IS_ZERO.
// ---------------------------------------------------------------------------
#if SCL_KIND == 11

__device__ __forceinline__ scl_u64 scl_clampi(long long v, long long hi) {
  return (scl_u64)(v < 0 ? 0 : (v > hi ? hi : v));
}

// Fill the positions of the window that lie outside the matrix: a warp takes a
// row of the window at a time, all of it for a row outside, else the columns
// left and right of the matrix, several loads in flight.
template <int WIN_H>
__device__ __forceinline__ void scl_patch_border(SCL_TYPE_0* win, long long x_org, long long y_org,
                                                 scl_u64 rows, scl_u64 cols) {
  // (the window overlaps the matrix: these fit in an int)
  const int left = x_org < 0 ? (int)-x_org : 0, top = y_org < 0 ? (int)-y_org : 0;
  const int right = (long long)cols - x_org < SCL_WIN_W ? (int)((long long)cols - x_org) : SCL_WIN_W;
  const int bottom = (long long)rows - y_org < WIN_H ? (int)((long long)rows - y_org) : WIN_H;
#pragma unroll 1
  for (int ly = threadIdx.y; ly < WIN_H; ly += 8) {
    const bool inside = ly >= top && ly < bottom;
    SCL_TYPE_0* row = win + ly * SCL_WIN_W;
#if SCL_PADDING == 1
    // (the clamped positions lie inside both the matrix and the window)
    const SCL_TYPE_0* from = win + (inside ? ly : (ly < top ? top : bottom - 1)) * SCL_WIN_W;
#endif
#pragma unroll
    for (int c = 0; c < SCL_WIN_W; c += 32) {
      const int lx = c + (int)threadIdx.x;
      if (lx >= SCL_WIN_W || (inside && lx >= left && lx < right)) continue;
#if SCL_PADDING == 1
      row[lx] = from[lx < left ? left : (lx >= right ? right - 1 : lx)];
#else
      row[lx] = (SCL_TYPE_0)(SCL_NEUTRAL);
#endif
    }
  }
}

// Each thread computes PY vertically adjacent outputs in each of SCL_PX
// adjacent columns: with the user loops unrolled, the taps those outputs
// share are read once.
template <int PY>
__device__ __forceinline__ void scl_compute_tile(const SCL_TYPE_0* win,
                                                 SCL_TYPE_1 (&res)[PY][SCL_PX] SCL_USER_PARAMS) {
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int p = 0; p < PY; ++p) {
    const int ly = ty * PY + p;
#pragma unroll
    for (int c = 0; c < SCL_PX; ++c) {
      const int lx = tx * SCL_PX + c;
      input_matrix_t m;
      m.data = win + (ly + SCL_R) * SCL_WIN_W + SCL_XLEAD + lx;
      m.local_row = ly;
      m.local_column = lx;
      res[p][c] = USR_FUNC(m SCL_EXTRA_ARGS);
    }
  }
}

// One element of 4 or 8 bytes to shared memory (complete after
// cp.async.wait_all).
__device__ __forceinline__ void scl_stage_element(SCL_TYPE_0* dst, const SCL_TYPE_0* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;"
               :: "r"((unsigned int)__cvta_generic_to_shared(dst)), "l"(src), "n"((int)sizeof(SCL_TYPE_0))
               : "memory");
}

// A window that lies inside the matrix, at (x_org, y_org), a warp per row.
template <int WIN_H>
__device__ __forceinline__ void scl_stage_window(SCL_TYPE_0* win, const SCL_TYPE_0* in, long long x_org,
                                                 long long y_org, scl_u64 cols) {
  const int tx = threadIdx.x, ty = threadIdx.y;
  const SCL_TYPE_0* src = in + (scl_u64)(y_org + ty) * cols + (scl_u64)(x_org + tx);
  SCL_TYPE_0* dst = win + ty * SCL_WIN_W + tx;
  for (int ly = ty; ly < WIN_H; ly += 8, src += 8 * cols, dst += 8 * SCL_WIN_W) {
#pragma unroll
    for (int c = 0; c < SCL_WIN_W; c += 32)
      if (c + 32 <= SCL_WIN_W || tx < SCL_WIN_W - c) scl_stage_element(dst + c, src + c);
  }
}

// The window through registers, padded outside the matrix, for elements that
// cp.async does not take and for windows that reach outside (asynchronous copies
// of the nearest elements: 20,000 x 33 floats, clamped, R = 1 14.0 us against 5.6):
// the loads of several rows are in flight before their stores.  Sobel on unsigned
// char, 1000 x 1001 7.0 -> 3.4 us, 3000 x 2999 15.5 -> 12.9, against loading and
// storing an element at a time in border tiles and a row at a time elsewhere
// (a window is a chain of 5 to 25 load latencies then).  Rows brought as words
// and shifted into place ran 7.2 and 15.2 us, stores in words 7.4 and 16.8.
template <int WIN_H, bool WHOLE>
__device__ __forceinline__ void scl_stage_registers(SCL_TYPE_0* win, const SCL_TYPE_0* in, long long x_org,
                                                    long long y_org, scl_u64 rows, scl_u64 cols) {
  constexpr int NR = (WIN_H + 7) / 8, NC = (SCL_WIN_W + 31) / 32, BATCH = NR * NC <= 16 ? NR : (NC < 16 ? 16 / NC : 1);
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll 1
  for (int r0 = 0; r0 < NR; r0 += BATCH) {
    SCL_TYPE_0 v[BATCH][NC];
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      const int ly = (r0 + i) * 8 + ty;
      if (ly >= WIN_H) break;
      const long long gy = y_org + ly;
      const SCL_TYPE_0* row = in + (WHOLE ? (scl_u64)gy : scl_clampi(gy, (long long)rows - 1)) * cols;
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const long long gx = x_org + j * 32 + tx;
        if ((j + 1) * 32 > SCL_WIN_W && tx >= SCL_WIN_W - j * 32) continue;
        if (WHOLE) {
          v[i][j] = row[gx];
          continue;
        }
#if SCL_PADDING == 1
        v[i][j] = row[scl_clampi(gx, (long long)cols - 1)];
#else
        const bool inside = gy >= 0 && gy < (long long)rows && gx >= 0 && gx < (long long)cols;
        v[i][j] = inside ? row[gx] : (SCL_TYPE_0)(SCL_NEUTRAL);
#endif
      }
    }
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      const int ly = (r0 + i) * 8 + ty;
      if (ly >= WIN_H) break;
#pragma unroll
      for (int j = 0; j < NC; ++j)
        if ((j + 1) * 32 <= SCL_WIN_W || tx < SCL_WIN_W - j * 32) win[ly * SCL_WIN_W + j * 32 + tx] = v[i][j];
    }
  }
}

// Cooperative-load variant: any shape, any alignment.  A warp brings a row of
// the window at a time, coalesced; the outputs go back through shared memory
// (the window's place, once every thread has read it) so that a warp stores
// rows as well, not every SCL_PX-th element.  6000 x 5999 floats, clamped, R =
// 1 108.4 -> 59.6 us, R = 5 280.5 -> 171.3 us against staging by a division per
// element and stores SCL_PX elements apart (which remain where the outputs do
// not fit beside Local arguments: ROWS_OUT 0, a kernel of its own since the
// branch alone cost the others 3 to 13 %).
template <int PY, int ROWS_OUT = 1>
__global__ void __launch_bounds__(256)
scl_mapoverlap_ldst(const SCL_TYPE_0* in, SCL_TYPE_1* out, scl_u64 rows, scl_u64 cols SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  constexpr int TH = 8 * PY, WIN_H = TH + 2 * SCL_R;
  SCL_TYPE_0* win = reinterpret_cast<SCL_TYPE_0*>(scl_dyn_smem);  // WIN_H x SCL_WIN_W
  const scl_u64 x0 = (scl_u64)blockIdx.x * SCL_TW, y0 = (scl_u64)blockIdx.y * TH;
  const long long x_org = (long long)x0 - SCL_XLEAD, y_org = (long long)y0 - SCL_R;
  const int tx = threadIdx.x, ty = threadIdx.y;
  constexpr bool sized = sizeof(SCL_TYPE_0) == 4 || sizeof(SCL_TYPE_0) == 8;
  const bool whole = x_org >= 0 && y_org >= 0 && x_org + SCL_WIN_W <= (long long)cols && y_org + WIN_H <= (long long)rows;
  bool async = false;
  if constexpr (sized) {
    async = whole && (scl_u64)in % sizeof(SCL_TYPE_0) == 0;
    if (async) scl_stage_window<WIN_H>(win, in, x_org, y_org, cols);
  }
  if (!async) {
    if (whole) scl_stage_registers<WIN_H, true>(win, in, x_org, y_org, rows, cols);
    else scl_stage_registers<WIN_H, false>(win, in, x_org, y_org, rows, cols);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  SCL_TYPE_1 res[PY][SCL_PX];
  scl_compute_tile<PY>(win, res SCL_EXTRA_ARGS);
  if constexpr (!ROWS_OUT) {
#pragma unroll
    for (int p = 0; p < PY; ++p) {
      const scl_u64 y = y0 + ty * PY + p, x = x0 + (scl_u64)tx * SCL_PX;
      if (y >= rows) break;
#pragma unroll
      for (int c = 0; c < SCL_PX; ++c)
        if (x + c < cols) out[y * cols + x + c] = res[p][c];
    }
    return;
  }
  __syncthreads();
  SCL_TYPE_1* mine = reinterpret_cast<SCL_TYPE_1*>(scl_dyn_smem) + ty * PY * SCL_TW;  // this warp's rows
#pragma unroll
  for (int p = 0; p < PY; ++p) {
    scl_pack<SCL_TYPE_1, SCL_PX> v;
#pragma unroll
    for (int c = 0; c < SCL_PX; ++c) v.v[c] = res[p][c];
    scl_store<SCL_TYPE_1, SCL_PX>(mine + p * SCL_TW + tx * SCL_PX, v);
  }
  __syncwarp();
#pragma unroll
  for (int p = 0; p < PY; ++p) {
    const scl_u64 y = y0 + ty * PY + p;
    if (y >= rows) break;
#pragma unroll
    for (int c = 0; c < SCL_PX; ++c) {
      const scl_u64 x = x0 + c * 32 + tx;
      if (x < cols) out[y * cols + x] = mine[p * SCL_TW + c * 32 + tx];
    }
  }
}

// TMA variant: one elected thread loads the whole window with
// cp.async.bulk.tensor.2d (zero fill outside the matrix); border tiles are
// patched afterwards.  Requires cols * sizeof(T) % 16 == 0 (tensor-map stride
// rule) and a 16-byte aligned base; the host checks both.  With `ovec` (the
// host's word that rows of `out` sit on the size of SCL_PX elements) a thread
// stores its adjacent columns at once.  8192^2 floats, with that and the border
// patched by rows: clamped R = 1 91.3 -> 78.7 us, R = 2 100.6 -> 87.6, R = 5
// 299.8 -> 283.2; neutral R = 5 287.4 -> 276.2 us (79 us are the transfer).
// (A resident grid whose blocks fetch their next window while computing took
// 100.6 and 327 us clamped: tiles are best handed out as blocks end.)
struct __align__(64) scl_tmap { unsigned long long v[16]; };

template <int PY>
__global__ void __launch_bounds__(256)
scl_mapoverlap_tma(const __grid_constant__ scl_tmap tmap, SCL_TYPE_1* out, scl_u64 rows,
                   scl_u64 cols, unsigned int spin_limit, unsigned int* err, int ovec SCL_EXTRA_PARAMS) {
  SCL_EXTRA_SETUP
  constexpr int TH = 8 * PY, WIN_H = TH + 2 * SCL_R;
  SCL_TYPE_0* win = reinterpret_cast<SCL_TYPE_0*>(scl_dyn_smem);  // WIN_H x SCL_WIN_W
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int s_ok;
  const scl_u64 x0 = (scl_u64)blockIdx.x * SCL_TW, y0 = (scl_u64)blockIdx.y * TH;
  const long long x_org = (long long)x0 - SCL_XLEAD, y_org = (long long)y0 - SCL_R;
  const unsigned int bar_s = (unsigned int)__cvta_generic_to_shared(&bar);
  const int t = threadIdx.y * blockDim.x + threadIdx.x;
  constexpr unsigned int bytes = WIN_H * SCL_WIN_W * sizeof(SCL_TYPE_0);
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar_s));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (t == 0) {
    const unsigned int dst = (unsigned int)__cvta_generic_to_shared(win);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(bar_s), "r"(bytes) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];"
        :: "r"(dst), "l"(&tmap), "r"((int)x_org), "r"((int)y_org), "r"(bar_s)
        : "memory");
    // Bounded wait on phase 0 by thread 0 only; the verdict is block-uniform.
    unsigned int done = 0, polls = 0;
    while (!done) {
      asm volatile(
          "{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], 0;"
          " selp.u32 %0, 1, 0, p; }"
          : "=r"(done) : "r"(bar_s) : "memory");
      if (!done) {
        if (++polls > spin_limit) break;
        scl_nanosleep(32);
      }
    }
    s_ok = done ? 1 : 0;
    if (!done) {
      scl_raise(err, SCL_DEV_ERR_TIMEOUT);
      // The copy may still land in this block's shared memory: thread 0 keeps
      // the block alive (bounded again) before it returns.
      for (unsigned int k = 0; k < spin_limit && !done; ++k) {
        scl_nanosleep(64);
        asm volatile(
            "{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], 0;"
            " selp.u32 %0, 1, 0, p; }"
            : "=r"(done) : "r"(bar_s) : "memory");
      }
    }
  }
  __syncthreads();
  if (!s_ok) return;
  const bool border = x_org < 0 || y_org < 0 || x_org + SCL_WIN_W > (long long)cols ||
                      y_org + WIN_H > (long long)rows;
#if SCL_PADDING == 1 || SCL_NEUTRAL_IS_ZERO == 0
  if (border) scl_patch_border<WIN_H>(win, x_org, y_org, rows, cols);
#endif
  __syncthreads();
  SCL_TYPE_1 res[PY][SCL_PX];
  scl_compute_tile<PY>(win, res SCL_EXTRA_ARGS);
#pragma unroll
  for (int p = 0; p < PY; ++p) {
    const scl_u64 y = y0 + threadIdx.y * PY + p, x = x0 + (scl_u64)threadIdx.x * SCL_PX;
    if (y >= rows) break;
    if (ovec) {
      scl_pack<SCL_TYPE_1, SCL_PX> v;
#pragma unroll
      for (int c = 0; c < SCL_PX; ++c) v.v[c] = res[p][c];
      if (x < cols) scl_store<SCL_TYPE_1, SCL_PX>(out + y * cols + x, v);
    } else {
#pragma unroll
      for (int c = 0; c < SCL_PX; ++c)
        if (x + c < cols) out[y * cols + x + c] = res[p][c];
    }
  }
}
#endif
