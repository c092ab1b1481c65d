// Bound-filtered weighted-minhash kernels for sm_100a.
//
// The dense kernels (hash_kernels.cu) evaluate every (entry, sample) of a
// row from 12 bytes of parameters, although only a sample's running minimum
// matters.  These kernels read one byte per (entry, sample) and evaluate only
// the entries that byte cannot rule out.
//
// With u = t - beta the evaluated value (kernel.cu:101-105 of
// src-d/minhashcuda) is ln_a = ln_c - u*r - r, and t = floor(w/r + beta)
// gives w - r < u*r <= w, so
//     ln_c - r - w <= ln_a < ln_c - w.
// ln_c - r depends on the table alone: the byte table `bounds` holds it
// rounded down in steps of 1/20.  An entry is skipped when its bound minus w
// is above a threshold that the sample's minimum does not exceed; the others
// go through the dense kernels' evaluation in float32 with the exact quotient.
// A skipped entry could not have replaced the minimum, so the hashes are the
// dense kernels' bit for bit.
//
// The threshold is the sample's running minimum or, while that is higher, a
// guess: a row's minimum of ln_a is distributed as ln(Exp(1) / sum of weights)
// whatever the weights, so ln(kGuess / sum) is exceeded by one sample in
// e^kGuess.  Samples that end above the guess are found at the end of the row
// and scanned again without it (rescan).  With the generator's distributions
// (r ~ Gamma(2), c ~ Gamma(2)) the share of entries whose c * e^-r lies below
// x is x * (ln(1/x) + 0.42); counted on the device, 17 candidates per sample
// are evaluated in a 1400-entry row, 13 in one of 300 (42 in the former
// without the guess, when a row's first entries all pass).
//
// What bounds it.  Per entry a 128-byte line of bounds and per candidate a
// 12-byte triple in a 32- or 64-byte sector somewhere in the table.  On uniform
// columns over 12M that is HBM: 3.9 bytes per eval (12 in the dense kernel) at
// 86% of the measured copy rate.  On Zipf columns, whose bounds stay in L2 (0.73
// bytes per eval from HBM), it is the warps' waits for gathers at 5 instructions
// per eval and 54% of the issue slots; candidates take a third of the time.
// Against the dense kernels, device-resident, same box: 524,288 Zipf rows of
// 1400 entries 98.1 -> 27.7 ms (3.4e12 evals/s), 131,072 ragged rows over 12M
// columns 16.0 -> 5.3 ms, 256 uneven matrices at 256 samples 12.8 -> 5.9 ms,
// 20,011 rows of 300 entries 855 -> 418 us.  filter_rule in wmh_internal.h says
// which launches come here.
//
// Rounding.  In float32 the computed ln_a may lie below the real
// ln_c - r - w by at most 2^-24 * (6|w| + 5 r (1 + |beta|) + 3|ln_c|) (one
// relative error of 2^-24 per operation; the quotient's and the sum's enter
// through t <= RN(RN(w/r) + beta)).  |w| <= 104 for a finite nonzero float32
// weight; with r <= 64, |beta| <= 2 and |ln_c| <= 64 that is below 2^-13, and
// kBoundSlack = 2^-9 is subtracted before the bound is rounded down.  A
// parameter outside those ranges (assigned tables; r = 0, NaN) or a bound
// below the byte's range gets byte 0, which always passes.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "hash_device.cuh"
#include "wmh_internal.h"

namespace mhb {
namespace {

// ---- Threshold arithmetic --------------------------------------------------
// In units of 1/20 with everything rounded up: entry i passes for a sample
// when byte <= m + l + 240, m = ceil(20 * threshold), l = ceil(20 * w_i).
// Two samples share a register as 16-bit halves; the halves' signed sums are
// formed by one 32-bit addition each because the biased total
//     D = filter_diff(byte, m, l) = 0x8000 + byte - T,  T = m + l + 241,
// stays within 16 bits; bit 15 of D is clear exactly when byte < T.

constexpr uint32_t kThrOpen = kThrLimit + kThrBias;  // every entry passes
// 7 was the fastest of 5 (20% slower on 1400-entry rows: one sample in 150 is
// scanned again), 7, 8 and 10 (8% slower on 200-entry rows: more candidates).
constexpr float kGuess = 7.0f;
// A threshold is kept within this of the row's guess (3 in ln_a).  The few
// samples with a lower minimum let a few entries more pass; the lower end of
// the byte's range (T >= 1) would otherwise be set for all samples by the one
// with the least minimum.
constexpr uint32_t kThrSpread = 60;

// ceil(20 * x); 0.01 covers the product's rounding.  NaN gives 0, infinities
// the ends of int.
__device__ __forceinline__ int quant_up(float x) {
  return __float2int_ru(__fmaf_rn(x, kBoundScale, 0.01f));
}
// m and l (the clamps' reasons are at their definitions).
__device__ __forceinline__ int quant_min(float mn) { return clamp_min(quant_up(mn)); }
__device__ __forceinline__ int quant_weight(float w) { return clamp_weight(quant_up(w)); }
__device__ __forceinline__ uint32_t threshold(float mn) {
  return static_cast<uint32_t>(quant_min(mn) + kThrBias);
}

// Minima as (monotone image of ln_a, position).  The smallest pair is the
// smallest ln_a and, among equal ones, the earliest position: the first strict
// minimum of kernel.cu:106, in whatever order it is combined.
__device__ __forceinline__ uint32_t ordered(float x) {
  const uint32_t u = __float_as_uint(__fadd_rn(x, 0.0f));  // -0 -> +0: equal as floats
  return u ^ (static_cast<uint32_t>(static_cast<int32_t>(u) >> 31) | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t k) {
  return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xFFFFFFFFu));
}
__device__ __forceinline__ unsigned long long make_key(float x, uint32_t pos) {
  return static_cast<unsigned long long>(ordered(x)) << 32 | pos;
}

// ln_a of one (entry, sample), kernel.cu:101-105, and its t.
__device__ __forceinline__ float exact_ln_a(float w, float r, float c, float b, float &t) {
  t = exact_t(w, r, b);
  return __fsub_rn(__fmaf_rn(-__fsub_rn(t, b), r, c), r);
}
// The sign bits of the four halves of (d0, d1), each spread over a byte (prmt
// with the replicate-sign bit of its selectors, which __byte_perm masks off).
__device__ __forceinline__ uint32_t half_signs(uint32_t d0, uint32_t d1) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, 0xFDB9;" : "=r"(r) : "r"(d0), "r"(d1));
  return r;
}

// 24 warps per SM at 80 registers, with the seldom used state of an item in
// shared memory: 131,072 Zipf rows of 1400 entries take 7.3 ms, 7.7 with 20
// warps (96 registers), 7.6 with 28 (72), 7.5 with 32 (64).
constexpr int kFilterBlocks = 6;
// Candidates evaluated at a time per lane: 1 / 2 / 3 take 7.9 / 7.3 / 7.8 ms
// there, and 7.5 / 6.6 / 6.6 ms on 256 uneven matrices at 256 samples.
constexpr uint32_t kEvalDepth = 2;
// Queue length at which a batch is followed by an evaluation.  Fresh thresholds
// pay: at 128 a 300-entry row has 13 candidates per sample, evaluated only at
// the end of its windows 17.
constexpr uint32_t kEvalAt = 128;
constexpr uint32_t kFWin = 128;    // CSR positions per staged window
// Candidates a warp holds: at least 127 left over and 512 more.  Shared memory
// is taken from L1, which has to hold a candidate's sector between its three
// loads: 1024 measured 4% slower on 1400-entry rows.
constexpr uint32_t kQueue = 768;

// One warp's shared memory; TILE samples per tile.
template <uint32_t TILE>
struct alignas(16) FilterStage {
  WarpStageT<kFWin> st;
  int32_t l[kFWin];              // l of the window's entries in both halves (l * 65537)
  // The tile's samples: the running minimum (ordered), its position, and the
  // pair it gives (kernel.cu:108).
  uint32_t val[TILE], pos[TILE], k[TILE], t[TILE];
  uint16_t thr[TILE];            // their thresholds, m + kThrBias
  uint16_t queue[kQueue];        // candidates: window position | sample << 8
  // Of the item, seldom read (registers are short): its chunk, the end of the
  // rows it owns, and the first position of the current row in the chunk.
  uint32_t chunk, r_stop, row_begin;
};

// Inclusive prefix sum over the warp.
__device__ __forceinline__ uint32_t warp_prefix(uint32_t x, uint32_t lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    x += lane >= static_cast<uint32_t>(o) ? y : 0u;
  }
  return x;
}

// One (chunk c, sample tile) item, as hash_item of the dense kernels: the
// rows inside chunk c are finished, partial minima of the rows that cross its
// ends are left for the finalize pass.  Chunks begin at a row where one
// starts soon enough (chunk_begin).
//
// LN lanes hold 16 samples each of one entry, so a tile is 16 * LN samples
// and one warp load fetches the bytes of 32 / LN entries (16 per lane; with 4
// samples per lane addresses and loads cost four times as much per sample).  A
// batch is 8 such loads, kept four ahead (eight ahead measured the same); its
// candidates go to a queue in shared memory.  Once it holds 128, and at the end of a window or row, the
// queue is evaluated, two candidates per lane at a time so that their
// parameter gathers overlap, and the thresholds are updated.
template <int LN, int SPAD, bool PACKED>
__device__ __forceinline__ bool filter_item(const HashArgs &a, uint32_t c, uint32_t tile,
                                            WarpCtxT<kFWin> &wc, FilterStage<16 * LN> &fs) {
  constexpr uint32_t TILE = 16 * LN;
  constexpr uint32_t GRP = 8 * (32 / LN);  // entries per batch
  const uint32_t lane = wc.lane;
  const uint32_t sub8 = lane / LN * 8;     // the lane's eight entries of a batch
  const uint32_t sl = lane % LN * 16;      // and its samples in the tile
  WarpStageT<kFWin> &stg = fs.st;
  uint32_t &parity = wc.parity;
  const uint32_t base = a.indptr[0];
  const uint32_t spad = SPAD ? static_cast<uint32_t>(SPAD) : a.s_pad;
  const uint32_t bstride = SPAD ? bound_stride(SPAD) : a.b_stride;
  const uintptr_t col_addr =
      PACKED ? (reinterpret_cast<uintptr_t>(a.cols_lo) | reinterpret_cast<uintptr_t>(a.cols_hi))
             : reinterpret_cast<uintptr_t>(a.cols);
  const bool bulk_ok =
      !a.host_csr && ((reinterpret_cast<uintptr_t>(a.weights) | col_addr) & 15u) == 0;
  const uint32_t t0 = tile * TILE;         // first sample of the tile
  const uint32_t width = min(TILE, a.samples - t0);  // samples of the tile that exist
  // Lanes past the last sample read the tile's first bytes; their candidate
  // bits are masked off.
  const uint32_t qoff = t0 + (t0 + sl < bstride ? sl : 0);
  const float *__restrict__ ptile = a.params + param_index(t0);

  const uint32_t cs = chunk_begin(a, c, base);
  const uint32_t ce = chunk_begin(a, c + 1, base);
  uint32_t r_next = a.chunk_row[c];
  __syncwarp();
  if (lane == 0) {
    fs.chunk = c;
    fs.r_stop = (c + 1 < a.nchunks) ? a.chunk_row[c + 1] : a.rows;
    fs.row_begin = cs;
  }
  __syncwarp();
  uint32_t row = kNone, row_end = cs;
  bool head = false, fresh = true;  // fresh: none of the row's entries has been looked at
  if (r_next > 0) {
    const uint32_t e = a.indptr[r_next] - base;
    if (e > cs) {
      row = r_next - 1;
      row_end = e;
      head = true;
    }
  }
  uint32_t thr[8];         // thresholds of the lane's 16 samples, two per register
  uint32_t thr_min = 0;    // the least of the tile's
  uint32_t thr_guess = kThrOpen;
  bool guessing = true;

  // Thresholds from the minima, to shared memory and to the lanes that use them.
  auto refresh = [&]() {
    const uint32_t thr_floor = thr_guess == kThrOpen ? 0 : thr_guess - kThrSpread;
    uint32_t least = kThrOpen;
#pragma unroll
    for (uint32_t v = 0; v < TILE / 32; ++v) {
      const uint32_t hi = fs.val[v * 32 + lane];
      const uint32_t t = max(min(thr_guess, threshold(unordered(hi))), thr_floor);
      fs.thr[v * 32 + lane] = static_cast<uint16_t>(t);
      least = min(least, t);
    }
    thr_min = __reduce_min_sync(0xFFFFFFFFu, least);
    __syncwarp();
    const uint4 x = *reinterpret_cast<const uint4 *>(&fs.thr[sl]);
    const uint4 y = *reinterpret_cast<const uint4 *>(&fs.thr[sl + 8]);
    thr[0] = x.x; thr[1] = x.y; thr[2] = x.z; thr[3] = x.w;
    thr[4] = y.x; thr[5] = y.y; thr[6] = y.z; thr[7] = y.w;
  };

  // Scans the row's entries [row_begin, end) again for every sample whose
  // minimum is above the guess, one sample at a time, lanes over entries.
  auto rescan = [&](uint32_t end) {
    uint32_t failed = 0;
    for (uint32_t s1 = 0; s1 < width; s1 += 32) {
      const bool above =
          s1 + lane < width &&
          threshold(unordered(fs.val[s1 + lane])) > thr_guess;
      uint32_t todo = __ballot_sync(0xFFFFFFFFu, above);
      while (todo) {
        const uint32_t s = s1 + __ffs(todo) - 1;
        todo &= todo - 1;
        ++failed;
        uint32_t best_k = fs.k[s], best_t = fs.t[s];
        unsigned long long best = static_cast<unsigned long long>(fs.val[s]) << 32 | fs.pos[s];
        const uint32_t begin = fs.row_begin, len = end - begin;  // p + 32 could wrap near 2^32
        for (uint32_t o = lane; o < len; o += 32) {
          const uint32_t p = begin + o;
          uint32_t col = PACKED ? packed_col(a, p) : a.cols[p];
          if (col >= a.dim) col = 0;
          const float w = logf(a.weights[p]);
          const uint32_t byte = a.bounds[static_cast<size_t>(col) * bstride + t0 + s];
          const int m = quant_min(unordered(static_cast<uint32_t>(best >> 32)));
          if (static_cast<int>(byte) > max(m + quant_weight(w) + 240, 0)) continue;
          const float *p3 = ptile + static_cast<size_t>(col) * 3 * spad + param_index(s);
          float t;
          const float x = exact_ln_a(w, __ldg(p3), __ldg(p3 + 2), __ldg(p3 + 4), t);
          if (x < FLT_MAX && make_key(x, p) < best) {
            best = make_key(x, p);
            best_k = col;
            best_t = whole(t);
          }
        }
        unsigned long long least = best;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          least = min(least, __shfl_xor_sync(0xFFFFFFFFu, least, o));
        __syncwarp();
        if (best == least) {  // lanes that share it hold the same pair
          fs.val[s] = static_cast<uint32_t>(least >> 32);
          fs.pos[s] = static_cast<uint32_t>(least);
          fs.k[s] = best_k;
          fs.t[s] = best_t;
        }
      }
    }
    // A table of other distributions, for which the guess does not hold.
    if (failed > TILE / 8) guessing = false;
    __syncwarp();
  };

  // Leaves the row that ends (in this chunk) at `end`.
  auto flush = [&](uint32_t end) {
    if (row == kNone) return;
    if (!fresh) rescan(end);
    const bool partial = head || row_end > ce;
    for (uint32_t s = lane; s < width; s += 32) {
      if (partial) {
        const size_t off = static_cast<size_t>(2 * fs.chunk + (head ? 0 : 1)) * spad + t0 + s;
        a.part_ln[off] = fresh ? FLT_MAX : unordered(fs.val[s]);
        a.part_kt[off] = make_uint2(fresh ? kNone : fs.pos[s], fresh ? kNone : fs.t[s]);
      } else {
        reinterpret_cast<uint2 *>(a.out)[static_cast<size_t>(row) * a.samples + t0 + s] =
            fresh ? make_uint2(kNone, kNone) : make_uint2(fs.k[s], fs.t[s]);
      }
    }
    __syncwarp();
  };

  // Windows start at multiples of 32 positions (16-byte aligned bulk copies
  // of every array), the first one possibly before the chunk.
  const uint32_t w0 = cs & ~31u;
  // Offsets from w0, which stay far from 2^32 where positions may not.
  const uint32_t span = ce > cs ? ce - w0 : 0;
  auto issue = [&](uint32_t at, uint32_t buf) {
    if (at < span)
      issue_window<PACKED>(a, stg, wc.pk, buf, w0 + at, min(kFWin, span - at), bulk_ok, lane);
  };
  issue(0, 0);
  issue(kFWin, 1);
  // Error exits wait (bounded) for the copies still in flight, those of the
  // windows at offset `from` and behind it.
  auto drain_copies = [&](uint32_t from, uint32_t buf) {
    for (uint32_t kk = 0; kk < 2 && from < span; ++kk, from += kFWin, buf ^= 1u) {
      for (uint32_t spins = 0; !mbar_try_wait(&stg.bar[buf], (parity >> buf) & 1u);)
        if (++spins > kSpinLimit) break;
      parity ^= 1u << buf;
    }
  };

  uint32_t b = 0;
  uint32_t i = cs - w0;
  for (uint32_t off = 0; off < span; off += kFWin, b ^= 1u, i = 0) {
    const uint32_t ws = w0 + off;
    const uint32_t n = min(kFWin, span - off);
    if (!finish_window<PACKED>(a, stg, wc.pk, b, (parity >> b) & 1u, ws, n, bulk_ok, lane)) {
      if (lane == 0) atomicOr(a.status, kStatusStall);
      drain_copies(off, b);
      return false;
    }
    parity ^= 1u << b;
    const float *__restrict__ lw = stg.w[b];
    uint32_t *__restrict__ cl = stg.c[b];
    for (uint32_t p = lane; p < n; p += 32) fs.l[p] = quant_weight(lw[p]) * 65537;
    // Entries past the window's end in its last batch: column 0, masked off.
    for (uint32_t p = n + lane; p < ((n + GRP - 1) & ~(GRP - 1)); p += 32) cl[p] = 0;
    __syncwarp();

    // Evaluates queued candidates from the end, kEvalDepth per lane at a time,
    // until at most `leave` are left.
    uint32_t count = 0;
    auto evaluate = [&](uint32_t leave) {
      do {
        const uint32_t from = count > 32 * kEvalDepth ? count - 32 * kEvalDepth : 0;
        uint32_t e[kEvalDepth];
        float r[kEvalDepth], lc[kEvalDepth], be[kEvalDepth];
#pragma unroll
        for (uint32_t j = 0; j < kEvalDepth; ++j) {
          // Lanes past the end repeat the last candidate's loads.
          e[j] = fs.queue[min(from + 32 * j + lane, count - 1)];
          const float *p = ptile + static_cast<size_t>(cl[e[j] & 0xFFu]) * 3 * spad + param_index(e[j] >> 8);
          r[j] = __ldg(p);
          lc[j] = __ldg(p + 2);
          be[j] = __ldg(p + 4);
        }
        // The minimum first, then position and pair of whoever holds it: the one
        // lane that brought the value stores its own; of equal values (ties, also
        // with an earlier minimum) the earliest position stores over it.
        uint32_t x[kEvalDepth];
        float t[kEvalDepth];
        bool brought[kEvalDepth];
#pragma unroll
        for (uint32_t j = 0; j < kEvalDepth; ++j) {
          const float ln_a = exact_ln_a(lw[e[j] & 0xFFu], r[j], lc[j], be[j], t[j]);
          x[j] = from + 32 * j + lane < count && ln_a < FLT_MAX ? ordered(ln_a) : 0xFFFFFFFFu;
          brought[j] = x[j] < atomicMin(&fs.val[e[j] >> 8], x[j]);
        }
        __syncwarp();
        auto store = [&](uint32_t j) {
          fs.pos[e[j] >> 8] = ws + (e[j] & 0xFFu);
          fs.k[e[j] >> 8] = cl[e[j] & 0xFFu];
          fs.t[e[j] >> 8] = whole(t[j]);
        };
        bool tie = false;
#pragma unroll
        for (uint32_t j = 0; j < kEvalDepth; ++j) {
          const bool holds = fs.val[e[j] >> 8] == x[j];
          if (holds && brought[j]) store(j);
          brought[j] = holds && !brought[j];
          tie |= brought[j];
        }
        if (__any_sync(0xFFFFFFFFu, tie)) {
          __syncwarp();
#pragma unroll
          for (uint32_t j = 0; j < kEvalDepth; ++j) {
            const uint32_t pos = ws + (e[j] & 0xFFu);
            if (brought[j]) brought[j] = pos < atomicMin(&fs.pos[e[j] >> 8], pos);
          }
          __syncwarp();
#pragma unroll
          for (uint32_t j = 0; j < kEvalDepth; ++j)
            if (brought[j] && fs.pos[e[j] >> 8] == ws + (e[j] & 0xFFu)) store(j);
        }
        __syncwarp();
        count = from;
      } while (count > leave);
    };

    while (i < n) {
      while (ws + i >= row_end) {
        flush(row_end);
        if (r_next >= fs.r_stop) {  // only reachable with inconsistent offsets
          if (lane == 0) atomicOr(a.status, kStatusBadIndptr);
          drain_copies(off + kFWin, b ^ 1u);
          return false;
        }
        row = r_next++;
        if (lane == 0) fs.row_begin = row_end;
        __syncwarp();
        row_end = a.indptr[row + 1] - a.indptr[0];
        head = false;
        fresh = true;
      }
      const uint32_t seg = min(row_end - ws, n);
      if (fresh) {
        // First look at the row: no minima yet, thresholds at the guess.
        fresh = false;
        thr_guess = kThrOpen;
        if (guessing) {
          float sum = 0.0f;
          const uint32_t len = min(row_end, ce) - fs.row_begin;
          const float *__restrict__ weights = a.weights + fs.row_begin;
#pragma unroll 8
          for (uint32_t o = lane; o < len; o += 32) sum += fmaxf(weights[o], 0.0f);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
          if (sum > 0.0f && sum < FLT_MAX) thr_guess = threshold(__logf(kGuess / sum));
        }
        thr_min = thr_guess;
#pragma unroll
        for (int v = 0; v < 8; ++v) thr[v] = thr_guess * 65537u;
#pragma unroll
        for (uint32_t v = 0; v < TILE / 32; ++v) {
          fs.val[v * 32 + lane] = ordered(FLT_MAX);
          fs.pos[v * 32 + lane] = kNone;
          fs.k[v * 32 + lane] = kNone;
          fs.t[v * 32 + lane] = kNone;
        }
        __syncwarp();
      }
      uint32_t g = i & ~(GRP - 1);
      uint4 q[4];  // bytes of four entries ahead
      // The table is at most 2 GiB: 32-bit byte offsets.
      auto load = [&](uint32_t col) {
        return __ldg(reinterpret_cast<const uint4 *>(a.bounds + (col * bstride + qoff)));
      };
      {
        const uint4 c0 = *reinterpret_cast<const uint4 *>(&cl[g + sub8]);
        q[0] = load(c0.x);
        q[1] = load(c0.y);
        q[2] = load(c0.z);
        q[3] = load(c0.w);
      }
      while (g < seg) {
        const uint32_t h = g + sub8;
        const int32_t l_lo = (1 + 16384 - static_cast<int32_t>(thr_min)) * 65537;
        uint32_t miss[4] = {0, 0, 0, 0};  // byte j of [v], bit x: entry h + x cannot win 4v + j
        // Entry h + x against the lane's 16 samples.
        auto compare = [&](int x, int32_t lx) {
          // l is kept above the value at which some T would drop below 1.
          const uint32_t l = static_cast<uint32_t>(max(lx, l_lo));
          const uint4 qx = q[x % 4];
          const uint32_t qq[4] = {qx.x, qx.y, qx.z, qx.w};
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const uint32_t d0 = __byte_perm(qq[v], 0xC0C0C0C0u, 0x4140) - thr[2 * v] - l;
            const uint32_t d1 = __byte_perm(qq[v], 0xC0C0C0C0u, 0x4342) - thr[2 * v + 1] - l;
            miss[v] |= half_signs(d0, d1) & (0x01010101u << x);
          }
        };
        const int4 la = *reinterpret_cast<const int4 *>(&fs.l[h]);
        const uint4 ca = *reinterpret_cast<const uint4 *>(&cl[h + 4]);
        compare(0, la.x);
        q[0] = load(ca.x);
        compare(1, la.y);
        q[1] = load(ca.y);
        compare(2, la.z);
        q[2] = load(ca.z);
        compare(3, la.w);
        q[3] = load(ca.w);
        const int4 lb = *reinterpret_cast<const int4 *>(&fs.l[h + 4]);
        if (g + GRP < seg) {  // with the loads of the next batch
          const uint4 cb = *reinterpret_cast<const uint4 *>(&cl[h + GRP]);
          compare(4, lb.x);
          q[0] = load(cb.x);
          compare(5, lb.y);
          q[1] = load(cb.y);
          compare(6, lb.z);
          q[2] = load(cb.z);
          compare(7, lb.w);
          q[3] = load(cb.w);
        } else {
          compare(4, lb.x);
          compare(5, lb.y);
          compare(6, lb.z);
          compare(7, lb.w);
        }
        uint32_t in_row = 0xFFFFFFFFu;  // entries of the row
        if (g < i || g + GRP > seg) {
          const uint32_t up = min(max(static_cast<int>(seg) - static_cast<int>(h), 0), 8);
          const uint32_t lo = min(max(static_cast<int>(i) - static_cast<int>(h), 0), 8);
          in_row = (((1u << up) - 1u) & ~((1u << lo) - 1u)) * 0x01010101u;
        }
        uint32_t hits[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          hits[v] = ~miss[v] & in_row;
          if (SPAD == 0 || (SPAD % TILE) != 0 || a.samples != spad) {  // samples that do not exist
            const int left = static_cast<int>(width) - static_cast<int>(sl + 4 * v);
            hits[v] &= left >= 4 ? 0xFFFFFFFFu : left <= 0 ? 0u : (1u << (8 * left)) - 1u;
          }
        }
        auto push = [&](uint32_t m, uint32_t v, uint32_t at) {
          const uint32_t code = h | (sl + 4 * v) << 8;
          while (m) {
            uint32_t bit;  // the highest set bit: entry bit % 8, sample bit / 8
            asm("bfind.u32 %0, %1;" : "=r"(bit) : "r"(m));
            m ^= 1u << bit;
            fs.queue[at++] = static_cast<uint16_t>(code + (bit & 7u) + (bit >> 3 << 8));
          }
          return at;
        };
        const uint32_t mine =
            __popc(hits[0]) + __popc(hits[1]) + __popc(hits[2]) + __popc(hits[3]);
        const uint32_t incl = warp_prefix(mine, lane);
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        if (count + total <= kQueue) {
          uint32_t at = count + incl - mine;
#pragma unroll
          for (uint32_t v = 0; v < 4; ++v) at = push(hits[v], v, at);
          count += total;
          if (count >= kEvalAt) {
            __syncwarp();
            evaluate(32 * kEvalDepth - 1);
            refresh();
          }
        } else {
          // More than the queue has room for: at most 512 at a time, four
          // entries of four samples per lane.
#pragma unroll 1
          for (uint32_t part = 0; part < 8; ++part) {
            const uint32_t v = part >> 1;
            const uint32_t m = (v == 0 ? hits[0] : v == 1 ? hits[1] : v == 2 ? hits[2] : hits[3]) &
                               (part & 1u ? 0xF0F0F0F0u : 0x0F0F0F0Fu);
            const uint32_t in2 = warp_prefix(__popc(m), lane);
            const uint32_t sum2 = __shfl_sync(0xFFFFFFFFu, in2, 31);
            if (count + sum2 > kQueue) {
              __syncwarp();
              evaluate(0);
            }
            push(m, v, count + in2 - __popc(m));
            count += sum2;
          }
        }
        g += GRP;
      }
      if (count) {
        __syncwarp();
        evaluate(0);
        if (ws + seg < row_end) refresh();  // the row goes on
      }
      i = seg;
    }
    issue(off + 2 * kFWin, b);
  }
  flush(min(row_end, ce));
  while (r_next < fs.r_stop) {  // trailing empty rows of the last chunk
    row = r_next++;
    row_end = ce;
    head = false;
    fresh = true;
    flush(ce);
  }
  return true;
}

// The next item beyond each warp's first, taken in order of demand (lane 0
// holds it): rows, and so items, differ in length, and the last items of a
// launch go to the warps that are done.
__device__ __forceinline__ uint32_t take_item(uint32_t *next_item, uint32_t lane) {
  return lane == 0 ? atomicAdd(next_item, 1u) : 0u;
}

template <int LN, int SPAD, bool PACKED>
__global__ void __launch_bounds__(kFilterBlock, kFilterBlocks) filter_kernel(const HashArgs a) {
  __shared__ FilterStage<16 * LN> stage_all[kFilterBlock / 32];
  PackedStageT<kFWin> *packed = nullptr;
  if constexpr (PACKED) {
    __shared__ PackedStageT<kFWin> packed_stage[kFilterBlock / 32];
    packed = &packed_stage[threadIdx.x >> 5];
  }
  if (*a.status & kStatusBadIndptr) return;
  FilterStage<16 * LN> &fs = stage_all[threadIdx.x >> 5];
  WarpCtxT<kFWin> wc;
  warp_ctx_init(wc, &fs.st, packed);
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t items = a.nchunks * a.ntiles;
  for (uint32_t item = gw; item < items;) {
    const uint32_t next = take_item(a.next_item, wc.lane);  // in flight during this item
    const uint32_t c = item / a.ntiles;
    if (!filter_item<LN, SPAD, PACKED>(a, c, item - c * a.ntiles, wc, fs)) return;
    item = nw + __shfl_sync(0xFFFFFFFFu, next, 0);
  }
}

template <int LN, int SPAD>
__global__ void __launch_bounds__(kFilterBlock, kFilterBlocks) filter_batch_kernel(const BatchArgs b) {
  __shared__ FilterStage<16 * LN> stage_all[kFilterBlock / 32];
  __shared__ HashArgs views[kFilterBlock / 32];
  if ((*b.base.status & kStatusBadIndptr) || !b.plan->filter) return;
  FilterStage<16 * LN> &fs = stage_all[threadIdx.x >> 5];
  WarpCtxT<kFWin> wc;
  warp_ctx_init(wc, &fs.st);
  HashArgs &view = views[threadIdx.x >> 5];
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t ntiles = b.ntiles[1];
  const uint32_t chunk = b.plan->chunk;
  const uint32_t items = b.plan->nchunks * ntiles;
  for (uint32_t item = gw; item < items;) {
    const uint32_t next = take_item(b.base.next_item, wc.lane);
    const uint32_t gc = item / ntiles;
    const uint32_t m = b.chunk_owner[gc];
    const uint32_t base = b.mats[m].chunk_base;
    __syncwarp();
    if (wc.lane == 0) view = matrix_view(b, b.mats[m], chunk);
    __syncwarp();
    if (!filter_item<LN, SPAD, false>(view, gc - base, item - gc * ntiles, wc, fs)) return;
    item = nw + __shfl_sync(0xFFFFFFFFu, next, 0);
  }
}

using FilterFn = void (*)(const HashArgs);
using FilterBatchFn = void (*)(const BatchArgs);

FilterFn pick_filter(uint32_t s_pad, uint32_t lanes, bool packed) {
  if (lanes == 8 && s_pad == 128)
    return packed ? filter_kernel<8, 128, true> : filter_kernel<8, 128, false>;
  if (lanes == 8 && s_pad == 256)
    return packed ? filter_kernel<8, 256, true> : filter_kernel<8, 256, false>;
  switch (lanes) {
    case 8: return packed ? filter_kernel<8, 0, true> : filter_kernel<8, 0, false>;
    case 4: return packed ? filter_kernel<4, 0, true> : filter_kernel<4, 0, false>;
    default: return packed ? filter_kernel<2, 0, true> : filter_kernel<2, 0, false>;
  }
}

FilterBatchFn pick_filter_batch(uint32_t s_pad) {
  if (s_pad == 128) return filter_batch_kernel<8, 128>;
  if (s_pad == 256) return filter_batch_kernel<8, 256>;
  switch (filter_lanes(s_pad)) {
    case 8: return filter_batch_kernel<8, 0>;
    case 4: return filter_batch_kernel<4, 0>;
    default: return filter_batch_kernel<2, 0>;
  }
}

}  // namespace

cudaError_t launch_filter(const HashArgs &a, const HashPlan &plan, cudaStream_t stream) {
  pick_filter(a.s_pad, plan.filter, a.col_hi_bits != 0)<<<plan.grid, kFilterBlock, 0, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_filter_batch(const BatchArgs &b, const HashPlan &plan, cudaStream_t stream) {
  pick_filter_batch(b.base.s_pad)<<<plan.grid, kFilterBlock, 0, stream>>>(b);
  return cudaGetLastError();
}

int filter_blocks_per_sm(uint32_t s_pad, uint32_t lanes) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pick_filter(s_pad, lanes, false), kFilterBlock, 0) !=
      cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return n > 0 ? n : 1;
}

}  // namespace mhb
