// Weighted-minhash hash kernels for sm_100a.
//
// Replaces weighted_minhash_cuda (kernel.cu:56-112 of src-d/minhashcuda) and
// the host-side binpacking that fed it (minhashcuda.cc:457-528).
//
// Per (row, sample) the value computed is the reference's (kernel.cu:95-110):
//   w = logf(weight); t = floorf(w / r + beta);
//   ln_a = ln_c - (t - beta) * r - r;  keep the first strict minimum.
// Each operation is spelled with an explicit round-to-nearest intrinsic so the
// compiler cannot re-associate or contract differently from the reference
// build: the multiply-subtract of kernel.cu:104-105 is one fused multiply-add
// (the form the reference build evaluates; pinned on a B200 by the tests).
//
// Layout and mapping (B200-first, not the reference's):
//  - a column's parameters are contiguous, in sample pairs (r r c c b b): one
//    nnz's for a tile of 32*SPL samples are three vector loads per lane over
//    one contiguous block (SPL=4: 1536 B),
//  - a warp owns one (chunk, sample tile) item; each lane keeps SPL running
//    minima in registers (no shared-memory spill as in kernel.cu:72-74),
//    each with the position of its entry and, for short rows, its t; what is
//    missing of (k, t) is recovered once per (row, sample) at the row's end,
//  - each warp stages its CSR positions in 256-entry windows with TMA bulk
//    copies (cp.async.bulk, mbarrier completion, double-buffered), turns the
//    weights into ln(weight) in place once per nnz, lane-parallel (the
//    reference evaluates logf once per thread, :95), validates the window's
//    columns once, and reads them back as shared-memory broadcasts,
//  - parameters for the next nnz are loaded into a second register set while
//    the current one is evaluated (ping-pong, no register copies); the loop
//    has no branch per nnz, samples are evaluated in pairs with packed f32x2
//    arithmetic, and the running minimum is updated with selects,
//  - work is cut by nnz, not by rows, so one 50k-nnz row and many 5-nnz rows
//    cost the same per item; rows that cross a chunk boundary are merged by
//    a finalize pass (tie -> earlier position, as the strict '<' scan).
#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <cstdlib>

#include "hash_device.cuh"
#include "wmh_internal.h"

namespace mhb {
namespace {

// chunk_row[c] = first row whose first position is >= c*chunk (rows if none),
// for the chunks whose first owned row is row i (i == rows: the chunks past
// the last row start); also validates the offsets.
__device__ __forceinline__ void plan_row(const HashArgs &a, uint32_t i) {
  const uint32_t base = a.indptr[0];
  uint32_t start, c_hi;
  if (i < a.rows) {
    const uint32_t s = a.indptr[i], e = a.indptr[i + 1];
    if (e < s || s < base) atomicOr(a.status, kStatusBadIndptr);
    start = s - base;
    c_hi = min(start / a.chunk, a.nchunks - 1);
  } else {
    if (a.indptr[a.rows] - base != a.nnz || a.indptr[a.rows] < base)
      atomicOr(a.status, kStatusBadIndptr);
    start = 0xFFFFFFFFu;
    c_hi = a.nchunks - 1;
  }
  uint32_t c_lo = 0;
  if (i > 0) {
    const uint32_t prev = a.indptr[i - 1] - base;
    c_lo = prev / a.chunk + 1;
  }
  for (uint32_t c = c_lo; c <= c_hi && c < a.nchunks; ++c) a.chunk_row[c] = i;
  (void)start;
}

// clear: the launch's one block clears the status word first, in place of a
// memset of its own (launches of few rows are bound by their launch count).
__global__ void plan_kernel(const HashArgs a, bool clear) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (clear) {
    if (threadIdx.x == 0) *a.status = 0;
    __syncthreads();
  }
  if (i == 0 && a.next_item) *a.next_item = 0;
  if (i <= a.rows) plan_row(a, i);
}

// Parameter sets a warp keeps in registers for register budget MINB
// (resident blocks per SM).  The gathers are latency-bound; with 2 blocks per
// SM there are half the warps of the 4-block budget to hide them, and 128
// registers per thread, room for a third set (12 registers at 4 samples per
// lane) that keeps two positions' gathers in flight: 111-122 registers, no
// spills.  524,288 rows of the 1,000,000-dim Zipf(1.1) matrix take 106.3 ms
// with it (3 and 4 blocks: 108.4 and 109.5), of uniform columns over 12,000,000
// dims 66.0 ms (64.7 and 62.6); with two sets (compared before the samples lay
// in pairs) the 2-block kernel took 6% and 16% longer.  The 3- and 4-block
// budgets (85 and 64 registers) have no room for it.
__host__ __device__ constexpr int param_depth(int minb) { return minb == 2 ? 3 : 2; }

// One (chunk c, sample tile) item over the CSR of `a`: finishes the rows
// that lie inside chunk c and leaves partial minima for the rows that cross
// its ends.  Returns false after an error exit (status flagged, in-flight
// staging copies drained); the warp must then stop.
// SPAD: the generator's s_pad when it is known at compile time (0: read it
// from the arguments), which turns the parameter-block addressing into one
// wide multiply-add and immediate load offsets.
// DEPTH: parameter sets in registers, 2 (the next position is loaded while
// one is evaluated) or 3 (the next two are), see param_depth.
template <int SPL, int SPAD, bool PACKED, int DEPTH, bool KEEP>
__device__ __forceinline__ bool hash_item(const HashArgs &a, uint32_t c, uint32_t tile,
                                          WarpCtx &wc) {
  const uint32_t lane = wc.lane;
  WarpStage &stg = *wc.stg;
  PackedStage *pk = wc.pk;
  uint32_t &parity = wc.parity;
  const uint32_t base = a.indptr[0];
  const uint32_t spad = SPAD ? static_cast<uint32_t>(SPAD) : a.s_pad;
  const size_t col_stride = static_cast<size_t>(3) * (SPAD ? static_cast<uint32_t>(SPAD) : a.s_pad);
  // Bulk copies only from device memory; mapped host CSR is read by the lanes.
  const uintptr_t col_addr =
      PACKED ? (reinterpret_cast<uintptr_t>(a.cols_lo) | reinterpret_cast<uintptr_t>(a.cols_hi))
             : reinterpret_cast<uintptr_t>(a.cols);
  const bool bulk_ok =
      !a.host_csr && ((reinterpret_cast<uintptr_t>(a.weights) | col_addr) & 15u) == 0;
  {
    const uint32_t s0 = tile * (32u * SPL) + lane * SPL;
    const bool active = s0 < spad;
    // Lanes past the last sample read the tile's first samples (in bounds)
    // and never store, so parameter loads need no branch.
    const float *__restrict__ pbase = a.params + param_index(active ? s0 : tile * (32u * SPL));
    const uint32_t cs = c * a.chunk;
    const uint32_t ce = cs + min(a.chunk, a.nnz - cs);  // no uint32 overflow near 2^32
    uint32_t r_next = a.chunk_row[c];
    const uint32_t r_stop = (c + 1 < a.nchunks) ? a.chunk_row[c + 1] : a.rows;

    // The row being accumulated: kNone, the row running in from the previous
    // chunk (head), or an owned row.
    uint32_t row = kNone, row_end = cs;
    bool head = false;
    if (r_next > 0) {
      const uint32_t e = a.indptr[r_next] - base;
      if (e > cs) {
        row = r_next - 1;
        row_end = e;
        head = true;
      }
    }
    RowState<SPL, KEEP> st;
    st.reset();
    const uint32_t *win = stg.c[0];  // the window last staged and its first position
    uint32_t win_at = cs;

    auto flush = [&]() {
      if (row == kNone || !active) return;
      if (head) {
        store_partial(a, 2 * c, s0, st);
      } else if (row_end > ce) {
        store_partial(a, 2 * c + 1, s0, st);
      } else {
        store_final(a, row, s0, st, win, win_at);
      }
    };

    const uint32_t nwin = (ce - cs + kWin - 1) / kWin;
    if (nwin > 0) issue_window<PACKED>(a, stg, pk, 0, cs, min(kWin, ce - cs), bulk_ok, lane);
    if (nwin > 1)
      issue_window<PACKED>(a, stg, pk, 1, cs + kWin, min(kWin, ce - cs - kWin), bulk_ok, lane);

    // Error exits wait (bounded) for the windows still in flight into this
    // warp's staging buffers before leaving: windows [from, min(from+2, nwin)).
    auto drain = [&](uint32_t from) {
      for (uint32_t kk = from; kk < nwin && kk < from + 2; ++kk) {
        const uint32_t bb = kk & 1u;
        for (uint32_t spins = 0; !mbar_try_wait(&stg.bar[bb], (parity >> bb) & 1u);)
          if (++spins > kSpinLimit) break;
        parity ^= 1u << bb;
      }
    };

    for (uint32_t k = 0; k < nwin; ++k) {
      const uint32_t b = k & 1u;
      const uint32_t ws = cs + k * kWin;
      const uint32_t n = min(kWin, ce - ws);
      if (!finish_window<PACKED>(a, stg, pk, b, (parity >> b) & 1u, ws, n, bulk_ok, lane)) {
        if (lane == 0) atomicOr(a.status, kStatusStall);
        drain(k);
        return false;
      }
      parity ^= 1u << b;
      const float *__restrict__ lw = stg.w[b];
      const uint32_t *__restrict__ cl = stg.c[b];
      win = stg.c[b];
      win_at = ws;

      // Columns in the window are < dim, and slots n and n + 1 hold column 0
      // (finish_window).
      if constexpr (DEPTH == 3) {
        // Three parameter sets: at each segment's start A holds position i
        // and B position i + 1; positions up to n + 1 read the zero column
        // slots past the window.
        Params<SPL> A, B, C;
        A.load(pbase + cl[0] * col_stride);
        B.load(pbase + cl[1] * col_stride);
        uint32_t i = 0;
        while (i < n) {
          while (ws + i >= row_end) {
            flush();
            if (r_next >= r_stop) {  // only reachable with inconsistent offsets
              if (lane == 0) atomicOr(a.status, kStatusBadIndptr);
              drain(k + 1);
              return false;
            }
            row = r_next++;
            row_end = a.indptr[row + 1] - base;
            head = false;
            st.reset();
          }
          const uint32_t seg = min(row_end - ws, n);
          while (i + 3 <= seg) {  // prefetches reach i + 4 <= n + 1
            C.load(pbase + cl[i + 2] * col_stride);
            eval_all(A, lw[i], ws + i, active, st);
            A.load(pbase + cl[i + 3] * col_stride);
            eval_all(B, lw[i + 1], ws + i + 1, active, st);
            B.load(pbase + cl[i + 4] * col_stride);
            eval_all(C, lw[i + 2], ws + i + 2, active, st);
            i += 3;
          }
          if (i + 2 == seg) {
            C.load(pbase + cl[i + 2] * col_stride);
            eval_all(A, lw[i], ws + i, active, st);
            eval_all(B, lw[i + 1], ws + i + 1, active, st);
            i += 2;
            A = C;
            B.load(pbase + cl[i + 1] * col_stride);
          } else if (i + 1 == seg) {
            eval_all(A, lw[i], ws + i, active, st);
            i += 1;
            A = B;
            B.load(pbase + cl[i + 1] * col_stride);
          }
        }
        if (k + 2 < nwin) {
          const uint32_t ws2 = ws + 2 * kWin;
          issue_window<PACKED>(a, stg, pk, b, ws2, min(kWin, ce - ws2), bulk_ok, lane);
        }
        continue;
      }
      Params<SPL> A, B;
      uint32_t dA = cl[0], dB = 0;
      A.load(pbase + dA * col_stride);
      uint32_t i = 0;
      while (i < n) {
        // Row boundaries (warp-uniform): finish rows, start the next owned one.
        while (ws + i >= row_end) {
          flush();
          if (r_next >= r_stop) {  // only reachable with inconsistent offsets
            if (lane == 0) atomicOr(a.status, kStatusBadIndptr);
            drain(k + 1);
            return false;
          }
          row = r_next++;
          row_end = a.indptr[row + 1] - base;
          head = false;
          st.reset();
        }
        const uint32_t seg = min(row_end - ws, n);
        // Pairs: A holds position i, B is loaded for i+1 while A is
        // evaluated, A for i+2 while B is evaluated.
        while (i + 1 < seg) {  // i + 2 <= n
          dB = cl[i + 1];
          B.load(pbase + dB * col_stride);
          eval_all(A, lw[i], ws + i, active, st);
          dA = cl[i + 2];
          A.load(pbase + dA * col_stride);
          eval_all(B, lw[i + 1], ws + i + 1, active, st);
          i += 2;
        }
        if (i < seg) {  // i + 1 <= n
          dB = cl[i + 1];
          B.load(pbase + dB * col_stride);
          eval_all(A, lw[i], ws + i, active, st);
          ++i;
          A = B;
          dA = dB;
        }
      }
      if (k + 2 < nwin) {
        const uint32_t ws2 = ws + 2 * kWin;
        issue_window<PACKED>(a, stg, pk, b, ws2, min(kWin, ce - ws2), bulk_ok, lane);
      }
    }
    flush();
    // Remaining owned rows are empty and start at ce (only possible in the
    // last chunk: trailing empty rows).
    while (r_next < r_stop) {
      row = r_next++;
      row_end = ce;
      head = false;
      st.reset();
      flush();
    }
  }
  return true;
}

// PACKED: the columns arrive as cols_lo/cols_hi (HashArgs::col_hi_bits).
template <int SPL, int MINB, int SPAD, bool PACKED, bool KEEP>
__global__ void __launch_bounds__(kHashBlock, MINB) hash_kernel(const HashArgs a) {
  __shared__ WarpStage stage_all[kHashBlock / 32];
  PackedStage *packed = nullptr;
  if constexpr (PACKED) {
    __shared__ PackedStage packed_stage[kHashBlock / 32];
    packed = &packed_stage[threadIdx.x >> 5];
  }
  if (*a.status & kStatusBadIndptr) return;
  WarpCtx wc;
  warp_ctx_init(wc, &stage_all[threadIdx.x >> 5], packed);
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t items = a.nchunks * a.ntiles;
  for (uint32_t item = gw; item < items; item += nw) {
    const uint32_t c = item / a.ntiles;
    if (!hash_item<SPL, SPAD, PACKED, param_depth(MINB), KEEP>(a, c, item - c * a.ntiles, wc)) return;
  }
}

// Merge the partials of every row that leaves its own chunk: one warp per
// (chunk owning such a row, tile of 32 samples), lanes over samples.  The
// chunks the row runs through are read in position order with unconditional
// loads, kFinalizeUnroll in flight (a row of 50,000 nnz cut into 64-nnz
// chunks has ~780 partials), and a strict '<' keeps the earliest position on
// ties, as the scan of kernel.cu:106 does.
constexpr uint32_t kFinalizeUnroll = 8;

// Merges, for sample s, the partials of the row that leaves chunk c (if one
// does) and writes its output pair.
__device__ __forceinline__ void finalize_item(const HashArgs &a, uint32_t c, uint32_t s) {
  const uint32_t base = a.indptr[0];
  const uint32_t r0 = a.chunk_row[c];
  const uint32_t r1 = (c + 1 < a.nchunks) ? a.chunk_row[c + 1] : a.rows;
  if (r1 <= r0) return;
  const uint32_t row = r1 - 1;
  const uint32_t end = a.indptr[row + 1] - base;
  const uint32_t ce = chunk_begin(a, c + 1, base);
  if (end <= ce || s >= a.samples) return;
  uint32_t c_last = (end - 1) / a.chunk;
  while (chunk_begin(a, c_last, base) >= end) --c_last;  // begins at the next row
  const size_t stride = 2 * static_cast<size_t>(a.s_pad);  // one chunk's two slots
  size_t off = static_cast<size_t>(2 * c + 1) * a.s_pad + s;
  float mn = a.part_ln[off];
  uint2 kt = a.part_kt[off];  // position and t
  off = static_cast<size_t>(2 * (c + 1)) * a.s_pad + s;
  uint32_t cc = c + 1;
  for (; cc + kFinalizeUnroll - 1 <= c_last; cc += kFinalizeUnroll) {
    float m[kFinalizeUnroll];
    uint2 k[kFinalizeUnroll];
#pragma unroll
    for (uint32_t u = 0; u < kFinalizeUnroll; ++u) {
      m[u] = a.part_ln[off + u * stride];
      k[u] = a.part_kt[off + u * stride];
    }
#pragma unroll
    for (uint32_t u = 0; u < kFinalizeUnroll; ++u) {
      const bool lt = m[u] < mn;
      mn = lt ? m[u] : mn;
      kt.x = lt ? k[u].x : kt.x;
      kt.y = lt ? k[u].y : kt.y;
    }
    off += kFinalizeUnroll * stride;
  }
  for (; cc <= c_last; ++cc, off += stride) {
    const float m2 = a.part_ln[off];
    const uint2 k2 = a.part_kt[off];
    const bool lt = m2 < mn;
    mn = lt ? m2 : mn;
    kt = lt ? k2 : kt;
  }
  uint32_t *o = a.out + (static_cast<size_t>(row) * a.samples + s) * 2;
  if (!a.part_t) {
    kt = resolve(a, kt.x, s);
  } else if (kt.x >= a.nnz) {
    kt = make_uint2(kNone, kNone);
  } else {
    kt.x = a.col_hi_bits ? packed_col(a, kt.x) : a.cols[kt.x];
  }
  *reinterpret_cast<uint2 *>(o) = kt;
}

__global__ void finalize_kernel(const HashArgs a) {
  // Any failure (invalid CSR, a staging copy that gave up) fails the call;
  // the partials a failed hash launch left may be stale, so none is merged.
  if (*a.status != 0) return;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t gw = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5;
  const uint64_t nw = (gridDim.x * static_cast<uint64_t>(blockDim.x)) >> 5;
  const uint32_t stiles = (a.samples + 31) / 32;
  const uint64_t items = static_cast<uint64_t>(a.nchunks) * stiles;
  for (uint64_t it = gw; it < items; it += nw) {
    const uint32_t c = static_cast<uint32_t>(it / stiles);
    const uint32_t s = static_cast<uint32_t>(it - static_cast<uint64_t>(c) * stiles) * 32 + lane;
    finalize_item(a, c, s);
  }
}

// ---- Device-resident batches ----------------------------------------------
// Many CSR matrices hashed against one generator by one persistent launch.
// Every matrix is cut into chunks of the same size; the batch's chunks are
// numbered matrix after matrix, and a warp item is (batch chunk, sample
// tile).  chunk_owner maps a batch chunk to its matrix, whose CSR, output and
// slice of the chunk table and partials the item then works on exactly as a
// single-matrix launch would: results equal one launch per matrix bit for bit
// (a row's arg-min and its ties do not depend on how positions are cut).

constexpr int kSetupThreads = 1024;

// Exclusive prefix sum over the block of one value per thread; returns this
// thread's offset and writes the total to *total.
__device__ __forceinline__ uint64_t block_exclusive_scan(uint64_t x, uint64_t *total) {
  __shared__ uint64_t warp_sums[kSetupThreads / 32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint64_t incl = x;
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= static_cast<uint32_t>(o)) incl += y;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint64_t w = lane < kSetupThreads / 32 ? warp_sums[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= static_cast<uint32_t>(o)) w += y;
    }
    warp_sums[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  const uint64_t before_warp = warp ? warp_sums[warp - 1] : 0;
  *total = warp_sums[kSetupThreads / 32 - 1];
  __syncthreads();
  return before_warp + incl - x;
}

// One block of kSetupThreads: per-matrix nnz (validating the end offsets),
// the batch's chunk size (the planner's rule applied to the whole batch, and
// large enough that the chunks fit max_chunks), each matrix's chunk range
// and the chunk -> matrix table.
__global__ void __launch_bounds__(kSetupThreads) batch_setup_kernel(const BatchArgs b) {
  const uint32_t t = threadIdx.x;
  const uint32_t per = (b.count + kSetupThreads - 1) / kSetupThreads;
  const uint32_t m0 = min(b.count, t * per), m1 = min(b.count, m0 + per);
  uint64_t nnz_sum = 0, rows_sum = 0, nonempty = 0;
  for (uint32_t m = m0; m < m1; ++m) {
    BatchMatrix &mt = b.mats[m];
    uint32_t n = 0;
    if (mt.rows) {
      const uint32_t s0 = mt.indptr[0], e = mt.indptr[mt.rows];
      if (e < s0) {
        atomicOr(b.base.status, kStatusBadIndptr);
      } else {
        n = e - s0;
      }
      ++nonempty;
    }
    mt.nnz = n;
    nnz_sum += n;
    rows_sum += mt.rows;
  }
  uint64_t total_nnz, total_rows, total_nonempty;
  block_exclusive_scan(nnz_sum, &total_nnz);
  block_exclusive_scan(rows_sum, &total_rows);
  block_exclusive_scan(nonempty, &total_nonempty);
  __shared__ uint32_t s_chunk;
  if (t == 0) {
    const uint32_t f = b.filter_min_row && total_nnz >= b.filter_min_nnz &&
                       total_nnz >= total_rows * filter_row(b.filter_min_row, total_nnz * b.base.s_pad / 2);
    b.plan->filter = f;
    const uint64_t ntiles = b.ntiles[f], target = b.warps[f] * b.waves, want = b.warps[f] * 8;
    uint64_t chunk = (total_nnz * ntiles + target - 1) / target;
    const uint64_t avg_row = total_rows ? (total_nnz + total_rows - 1) / total_rows : 1;
    chunk = max(chunk, min(4 * avg_row, static_cast<uint64_t>(1024)));
    b.plan->snap = 0;
    if (f) {
      const FilterSplit sp = filter_split(total_nnz * ntiles, b.warps[1], b.waves, avg_row);
      chunk = sp.chunk;
      b.plan->snap = sp.snap;
      *b.base.next_item = 0;
    } else {
      chunk = min(chunk, max(static_cast<uint64_t>(64), (total_nnz * ntiles + want - 1) / want));
    }
    // sum over matrices of ceil(nnz_m / chunk) <= total_nnz / chunk + nonempty
    const uint64_t avail = b.max_chunks > total_nonempty ? b.max_chunks - total_nonempty : 1;
    chunk = max(chunk, (total_nnz + avail - 1) / avail);
    if (!f && total_nnz * ntiles <= 8 * b.warps[0]) {  // tiny, as in make_plan
      const uint64_t one = (total_nnz * ntiles + b.warps[0] - 1) / b.warps[0];
      chunk = max(static_cast<uint64_t>(8), (one + 7) & ~static_cast<uint64_t>(7));
    } else {
      chunk = max(static_cast<uint64_t>(64), (chunk + 31) & ~static_cast<uint64_t>(31));
    }
    if (chunk > (1u << 24)) {
      chunk = 1u << 24;
      if (total_nnz / chunk + total_nonempty > b.max_chunks) atomicOr(b.base.status, kStatusBadIndptr);
    }
    s_chunk = static_cast<uint32_t>(chunk);
  }
  __syncthreads();
  const uint32_t chunk = s_chunk;
  uint64_t my_chunks = 0;
  for (uint32_t m = m0; m < m1; ++m) {
    const BatchMatrix &mt = b.mats[m];
    if (mt.rows) my_chunks += max(static_cast<uint64_t>(1), (static_cast<uint64_t>(mt.nnz) + chunk - 1) / chunk);
  }
  uint64_t total_chunks;
  uint64_t cb = block_exclusive_scan(my_chunks, &total_chunks);
  const bool fits = total_chunks <= b.max_chunks;
  for (uint32_t m = m0; m < m1; ++m) {
    BatchMatrix &mt = b.mats[m];
    const uint32_t nc = mt.rows ? static_cast<uint32_t>(max(
        static_cast<uint64_t>(1), (static_cast<uint64_t>(mt.nnz) + chunk - 1) / chunk)) : 0u;
    mt.chunk_base = static_cast<uint32_t>(cb);
    mt.nchunks = fits ? nc : 0u;
    if (fits)
      for (uint32_t c = 0; c < nc; ++c) b.chunk_owner[cb + c] = m;
    cb += nc;
  }
  if (t == 0) {
    if (!fits) atomicOr(b.base.status, kStatusBadIndptr);
    b.plan->chunk = chunk;
    b.plan->nchunks = fits ? static_cast<uint32_t>(total_chunks) : 0u;
  }
}

// Matrix owning plan thread g: the last one whose plan_base is <= g (matrices
// without rows own no threads and share the next matrix's plan_base).
__device__ __forceinline__ uint32_t plan_owner(const BatchArgs &b, uint32_t g) {
  uint32_t lo = 0, hi = b.count;  // answer in [lo, hi)
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (b.plan_base[mid] <= g) lo = mid; else hi = mid;
  }
  return lo;
}

__global__ void batch_plan_kernel(const BatchArgs b, uint32_t plan_threads) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= plan_threads || (*b.base.status & kStatusBadIndptr)) return;
  const uint32_t m = plan_owner(b, g);
  const BatchMatrix mt = b.mats[m];
  if (!mt.rows || !mt.nchunks) return;
  const HashArgs v = matrix_view(b, mt, b.plan->chunk);
  plan_row(v, g - b.plan_base[m]);
}

// The matrix view of an item is kept in shared memory, one per warp: its
// fields are read where the item needs them (per row or window), so the
// evaluation loop's registers are the single-matrix kernel's.
template <int SPL, int MINB, int SPAD>
__global__ void __launch_bounds__(kHashBlock, MINB) hash_batch_kernel(const BatchArgs b) {
  __shared__ WarpStage stage_all[kHashBlock / 32];
  __shared__ HashArgs views[kHashBlock / 32];
  if ((*b.base.status & kStatusBadIndptr) || b.plan->filter) return;
  WarpCtx wc;
  warp_ctx_init(wc, &stage_all[threadIdx.x >> 5]);
  HashArgs &view = views[threadIdx.x >> 5];
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t ntiles = b.ntiles[0];
  const uint32_t chunk = b.plan->chunk;
  const uint32_t items = b.plan->nchunks * ntiles;
  for (uint32_t item = gw; item < items; item += nw) {
    const uint32_t gc = item / ntiles;
    const uint32_t m = b.chunk_owner[gc];
    const uint32_t base = b.mats[m].chunk_base;
    __syncwarp();
    if (wc.lane == 0) view = matrix_view(b, b.mats[m], chunk);
    __syncwarp();
    if (!hash_item<SPL, SPAD, false, param_depth(MINB), false>(view, gc - base, item - gc * ntiles, wc))
      return;
  }
}

__global__ void finalize_batch_kernel(const BatchArgs b) {
  if (*b.base.status != 0) return;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t gw = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5;
  const uint64_t nw = (gridDim.x * static_cast<uint64_t>(blockDim.x)) >> 5;
  const uint32_t stiles = (b.base.samples + 31) / 32;
  const uint32_t chunk = b.plan->chunk;
  const uint64_t items = static_cast<uint64_t>(b.plan->nchunks) * stiles;
  for (uint64_t it = gw; it < items; it += nw) {
    const uint32_t gc = static_cast<uint32_t>(it / stiles);
    const uint32_t s = static_cast<uint32_t>(it - static_cast<uint64_t>(gc) * stiles) * 32 + lane;
    const BatchMatrix mt = b.mats[b.chunk_owner[gc]];
    if (mt.nchunks < 2) continue;  // a matrix of one chunk has no partials to merge
    const HashArgs v = matrix_view(b, mt, chunk);
    finalize_item(v, gc - mt.chunk_base, s);
  }
}

__global__ void logf_kernel(const float *in, float *out, size_t n) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[i] = logf(in[i]);
}

}  // namespace

cudaError_t launch_plan(const HashArgs &a, cudaStream_t stream, bool clear_status) {
  const uint32_t threads = clear_status && a.rows < 1024 ? 1024 : 256;
  const uint32_t blocks = a.rows / threads + 1;
  if (clear_status && blocks > 1) {
    const cudaError_t e = cudaMemsetAsync(a.status, 0, sizeof(uint32_t), stream);
    if (e != cudaSuccess) return e;
  }
  plan_kernel<<<blocks, threads, 0, stream>>>(a, clear_status && blocks == 1);
  return cudaGetLastError();
}

namespace {

using HashFn = void (*)(const HashArgs);
using BatchFn = void (*)(const BatchArgs);

// Instantiated (samples per lane, minimum resident blocks per SM) variants,
// with s_pad compiled in for the common sample counts.  The 4-block ones come
// with and without KEEP.
#define MHB_PICK(PICKED)                          \
  switch (spl * 100000 + minb * 10000 + s_pad) {  \
    case 440128: return PICKED(4, 4, 128, KEEP);  \
    case 440256: return PICKED(4, 4, 256, KEEP);  \
    case 240064: return PICKED(2, 4, 64, KEEP);   \
    case 430128: return PICKED(4, 3, 128, false); \
    case 420128: return PICKED(4, 2, 128, false); \
    case 430256: return PICKED(4, 3, 256, false); \
    case 420256: return PICKED(4, 2, 256, false); \
    default: break;                               \
  }                                               \
  switch (spl * 10 + minb) {                      \
    case 44: return PICKED(4, 4, 0, KEEP);        \
    case 24: return PICKED(2, 4, 0, KEEP);        \
    case 14: return PICKED(1, 4, 0, KEEP);        \
    case 43: return PICKED(4, 3, 0, false);       \
    case 42: return PICKED(4, 2, 0, false);       \
    default: return nullptr;                      \
  }
#define MHB_BATCH(SPL, MINB, SPAD, KEEP) hash_batch_kernel<SPL, MINB, SPAD>
#define MHB_HASH(SPL, MINB, SPAD, KEEP) hash_kernel<SPL, MINB, SPAD, PACKED, KEEP>

BatchFn pick_batch(uint32_t spl, uint32_t minb, uint32_t s_pad) { MHB_PICK(MHB_BATCH) }
template <bool PACKED, bool KEEP>
HashFn pick_hash(uint32_t spl, uint32_t minb, uint32_t s_pad) {
  MHB_PICK(MHB_HASH)
}
#undef MHB_HASH
#undef MHB_BATCH
#undef MHB_PICK

HashFn pick_hash(uint32_t spl, uint32_t minb, uint32_t s_pad, bool packed, bool keep) {
  if (packed)
    return keep ? pick_hash<true, true>(spl, minb, s_pad) : pick_hash<true, false>(spl, minb, s_pad);
  return keep ? pick_hash<false, true>(spl, minb, s_pad) : pick_hash<false, false>(spl, minb, s_pad);
}

}  // namespace

cudaError_t launch_hash(const HashArgs &a, const HashPlan &plan, cudaStream_t stream) {
  if (plan.filter) return launch_filter(a, plan, stream);
  const HashFn fn = pick_hash(plan.spl, plan.minb, a.s_pad, a.col_hi_bits != 0, plan.keep != 0);
  if (!fn) return cudaErrorInvalidValue;
  fn<<<plan.grid, kHashBlock, 0, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_finalize(const HashArgs &a, cudaStream_t stream) {
  const uint64_t warps_per_block = 8;
  const uint64_t items = static_cast<uint64_t>(a.nchunks) * ((a.samples + 31) / 32);
  uint64_t blocks = (items + warps_per_block - 1) / warps_per_block;
  if (blocks > 8192) blocks = 8192;
  finalize_kernel<<<static_cast<unsigned>(blocks), 32 * warps_per_block, 0, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_batch(const BatchArgs &b, const HashPlan &dense, const HashPlan &filtered,
                         uint32_t plan_threads, cudaStream_t stream) {
  const BatchFn fn = pick_batch(dense.spl, dense.minb, b.base.s_pad);
  if (!fn || b.count == 0 || b.max_chunks == 0) return cudaErrorInvalidValue;
  batch_setup_kernel<<<1, kSetupThreads, 0, stream>>>(b);
  if (plan_threads)
    batch_plan_kernel<<<(plan_threads + 255) / 256, 256, 0, stream>>>(b, plan_threads);
  if (b.filter_min_row) {
    const cudaError_t e = launch_filter_batch(b, filtered, stream);
    if (e != cudaSuccess) return e;
  }
  fn<<<dense.grid, kHashBlock, 0, stream>>>(b);
  const uint64_t stiles = (b.base.samples + 31) / 32;
  uint64_t blocks = (static_cast<uint64_t>(b.max_chunks) * stiles + 7) / 8;
  blocks = std::min<uint64_t>(std::max<uint64_t>(blocks, 1), 8192);
  finalize_batch_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(b);
  return cudaGetLastError();
}

int hash_blocks_per_sm(uint32_t spl, uint32_t minb, uint32_t s_pad) {
  const HashFn fn = pick_hash(spl, minb, s_pad, false, false);
  int n = 0;
  if (!fn || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kHashBlock, 0) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return n > 0 ? n : 1;
}

int plan_blocks_per_sm(const HashPlan &plan, uint32_t s_pad) {
  return plan.filter ? filter_blocks_per_sm(s_pad, plan.filter) : hash_blocks_per_sm(plan.spl, plan.minb, s_pad);
}

size_t hash_kernel_registers(uint32_t spl, uint32_t minb, uint32_t s_pad) {
  const HashFn fn = pick_hash(spl, minb, s_pad, false, false);
  cudaFuncAttributes attr{};
  if (!fn || cudaFuncGetAttributes(&attr, fn) != cudaSuccess) return 0;
  return attr.numRegs;
}

cudaError_t launch_logf(const float *in, float *out, size_t n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  size_t blocks = (n + 255) / 256;
  if (blocks > 65535) blocks = 65535;
  logf_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(in, out, n);
  return cudaGetLastError();
}

}  // namespace mhb
