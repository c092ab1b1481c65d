// Device code shared by the dense hash kernels (hash_kernels.cu) and the
// bound-filtered ones (filter_kernels.cu): one evaluation of the weighted
// MinHash, the TMA-staged CSR windows, and the result of a (row, sample).
#ifndef MHCUDA_B200_HASH_DEVICE_CUH
#define MHCUDA_B200_HASH_DEVICE_CUH
#include <cfloat>
#include <cstdint>

#include "wmh_internal.h"

namespace mhb {
namespace {

// Index of sample s's r inside a column of the parameter table; its ln_c and
// beta are 2 and 4 floats further (samples are stored in pairs, r r c c b b).
__device__ __forceinline__ uint32_t param_index(uint32_t s) { return (s >> 1) * 6 + (s & 1u); }

// The byte table of the filtered kernels: ln_c - r in steps of 1/kBoundScale
// from -kBoundOffset, rounded down after kBoundSlack is taken off (see
// filter_kernels.cu for what it bounds and why the slack is enough).  0 for
// what lies below the range and for parameters outside those the slack was
// derived for.
constexpr float kBoundScale = 20.0f;
constexpr float kBoundOffset = 12.0f;
constexpr float kBoundSlack = 0x1p-9f;

__device__ __forceinline__ uint32_t bound_byte(float r, float c, float b) {
  const bool known = r >= 0x1p-60f && r <= 64.0f && fabsf(c) <= 64.0f && fabsf(b) <= 2.0f;
  if (!known) return 0;  // NaN too
  const float x = floorf((c - r - kBoundSlack + kBoundOffset) * kBoundScale);
  return static_cast<uint32_t>(fminf(fmaxf(x, 0.0f), 255.0f));
}

// t of kernel.cu:103 exactly as the reference computes it: IEEE quotient,
// rounded sum, floor.
__device__ __forceinline__ float exact_t(float w, float r, float b) {
  return floorf(__fadd_rn(__fdiv_rn(w, r), b));
}

// Margin of the fast t below, relative to |w/r| + |beta| + 1.
constexpr float kTMargin = 0x1p-18f;

// Fast t.  Only floor(v) with v = RN(RN(w/r) + beta) is needed, and it only
// depends on the exact quotient when v lies close to an integer.  With
// y = rcp.approx(r) (documented error 1 ulp; 2^-22 relative assumed) and
// va = RN(RN(w*y) + beta):
//   |va - v| <= |w/r| * 2^-20.6 + |beta| * 2^-23 < m,
//   m = (|w*y| + |beta| + 1) * 2^-18,
// so when va is more than m away from every integer, floor(va) = floor(v).
// Returns false (t undecided) otherwise, and for every non-finite or
// flushed case (w = +-inf/NaN, r = 0/denormal/huge, |va| >= 2^22: m >= 16).
__device__ __forceinline__ bool fast_t(float w, float r, float b, float &t) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(r));
  const float qa = __fmul_rn(w, y);
  const float va = __fadd_rn(qa, b);
  t = floorf(va);
  const float f = __fsub_rn(va, t);  // exact for |va| >= 1; 1.0 or exact for va in (-1, 1)
  const float m = __fmaf_rn(__fadd_rn(fabsf(qa), fabsf(b)), kTMargin, kTMargin);
  return fabsf(__fsub_rn(f, 0.5f)) < __fsub_rn(0.5f, m);  // NaN -> false
}

// First position of chunk c (c == nchunks: nnz): c * chunk or, when a row
// starts at most `snap` positions further, that row's start (the filtered
// kernels, whose rows are dearer in pieces).  Chunks inside a row that is kept
// whole are empty.
__device__ __forceinline__ uint32_t chunk_begin(const HashArgs &a, uint32_t c, uint32_t base) {
  if (c >= a.nchunks) return a.nnz;
  const uint32_t at = c * a.chunk;
  if (!a.snap) return at;
  const uint32_t e = a.indptr[a.chunk_row[c]] - base;
  return e - at <= a.snap ? e : at;
}

// Column of relative position p in a packed CSR.
__device__ __forceinline__ uint32_t packed_col(const HashArgs &a, uint32_t p) {
  const uint32_t h = a.col_hi_bits == 4 ? (a.cols_hi[p >> 1] >> ((p & 1u) * 4)) & 15u
                                        : a.cols_hi[p];
  return static_cast<uint32_t>(a.cols_lo[p]) | (h << 16);
}

// (uint32)(int32)t as kernel.cu:108; the GPU conversion saturates.
__device__ __forceinline__ uint32_t whole(float t) {
  return static_cast<uint32_t>(static_cast<int32_t>(t));
}

// The output pair of kernel.cu:108 for sample s whose minimum came from the
// entry at relative position `pos`: k = cols[pos] and t recomputed from the
// entry with the exact quotient.  Every evaluation used that same t (fast_t
// only decides t when it equals the exact one), so tracking the position
// instead of (k, t) changes nothing but the work per evaluation.
// A position outside [0, nnz) (none found, or a partial that a failed launch
// left unwritten) yields kNone and reads nothing.
__device__ __forceinline__ uint2 resolve(const HashArgs &a, uint32_t pos, uint32_t s) {
  if (pos >= a.nnz) return make_uint2(kNone, kNone);
  const uint32_t k = a.col_hi_bits ? packed_col(a, pos) : a.cols[pos];
  // An invalid column was evaluated as column 0 and failed the call: keep
  // the parameter reads in bounds.
  if (k >= a.dim) return make_uint2(kNone, kNone);
  const float w = logf(a.weights[pos]);
  const float *col = a.params + static_cast<size_t>(k) * 3 * a.s_pad + param_index(s);
  const float t = exact_t(w, col[0], col[4]);
  return make_uint2(k, whole(t));
}

// KEEP: the minimum's t is kept beside its position (one select per
// evaluation, a register per sample), so that the end of a row does not
// recompute it: three gathers, a logarithm and a division per (row, sample).
template <int SPL, bool KEEP>
struct RowState {
  float mn[SPL];
  uint32_t pos[SPL];  // relative position of the minimum, kNone if none
  float t[KEEP ? SPL : 1];
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int j = 0; j < SPL; ++j) {
      mn[j] = FLT_MAX;
      pos[j] = kNone;
      if constexpr (KEEP) t[j] = 0.0f;
    }
  }
  // One (nnz, sample) evaluation, kernel.cu:106-109, given ln_a.
  __device__ __forceinline__ void update(int j, float ln_a, float tj, uint32_t p) {
    const bool lt = ln_a < mn[j];
    mn[j] = lt ? ln_a : mn[j];
    pos[j] = lt ? p : pos[j];
    if constexpr (KEEP) t[j] = lt ? tj : t[j];
  }
};

// win: the staged columns of the positions from `ws` on.
template <int SPL, bool KEEP>
__device__ __forceinline__ void store_final(const HashArgs &a, uint32_t row, uint32_t s0,
                                            const RowState<SPL, KEEP> &st,
                                            const uint32_t *__restrict__ win, uint32_t ws) {
  uint32_t *o = a.out + (static_cast<size_t>(row) * a.samples + s0) * 2;
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    uint2 kt;
    if constexpr (KEEP) {
      kt = make_uint2(kNone, kNone);
      if (st.pos[j] < a.nnz) {
        const uint32_t k = st.pos[j] >= ws ? win[st.pos[j] - ws]
                           : a.col_hi_bits ? packed_col(a, st.pos[j])
                                           : a.cols[st.pos[j]];
        kt = make_uint2(k, whole(st.t[j]));
      }
    } else {
      kt = resolve(a, st.pos[j], s0 + j);
    }
    if (s0 + j < a.samples) *reinterpret_cast<uint2 *>(o + 2 * j) = kt;
  }
}

template <int SPL, bool KEEP>
__device__ __forceinline__ void store_partial(const HashArgs &a, uint32_t slot, uint32_t s0,
                                              const RowState<SPL, KEEP> &st) {
  const size_t off = static_cast<size_t>(slot) * a.s_pad + s0;
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    uint32_t t = 0;  // without KEEP the merge recomputes it (HashArgs::part_t)
    if constexpr (KEEP) t = whole(st.t[j]);
    a.part_ln[off + j] = st.mn[j];
    a.part_kt[off + j] = make_uint2(st.pos[j], t);
  }
}

// ---- TMA bulk staging of the CSR (per warp, double-buffered) -------------

constexpr uint32_t kWin = 256;  // CSR positions per staged window of the dense kernels
constexpr uint32_t kSpinLimit = 1u << 22;

// One warp's staging area: two windows of weights (turned into ln w in
// place) and column indices, each with its own transaction barrier.  Column
// slots n and n + 1 of a window of n positions hold column 0, so the loop may
// prefetch two positions past the window without a bounds branch (the row stride of c,
// WIN + 4 words, keeps both windows 16-byte aligned for the bulk copies).
template <uint32_t WIN>
struct alignas(16) WarpStageT {
  float w[2][WIN];
  uint32_t c[2][WIN + 4];
  unsigned long long bar[2];
};
using WarpStage = WarpStageT<kWin>;

// Landing area of packed columns (HashArgs::col_hi_bits != 0): the low 16
// bits and the high nibbles or bytes of each window's columns, rebuilt into
// WarpStage::c by finish_window.
template <uint32_t WIN>
struct alignas(16) PackedStageT {
  uint16_t lo[2][WIN];
  uint8_t hi[2][WIN];
};
using PackedStage = PackedStageT<kWin>;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Global -> this CTA's shared memory, completion counted on `bar`.  Both
// addresses 16-byte aligned, bytes a multiple of 16.  No multicast.
__device__ __forceinline__ void bulk_copy_g2s(void *dst, const void *src, uint32_t bytes,
                                              unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// Positions of a window that arrive by bulk copy: a multiple of 4 (16 bytes
// of weights and of columns), or of 32 with packed columns (16 bytes of high
// nibbles); window starts are multiples of 32.
template <bool PACKED>
__device__ __forceinline__ uint32_t bulk_positions(uint32_t n, bool bulk_ok) {
  return bulk_ok ? (n & (PACKED ? ~31u : ~3u)) : 0u;
}

// Lane 0 starts the copy of positions [ws, ws + n) into buffer `b`: the
// 16-byte-aligned body by bulk copies, the ragged tail is left to
// finish_window's plain loads.
template <bool PACKED, uint32_t WIN>
__device__ __forceinline__ void issue_window(const HashArgs &a, WarpStageT<WIN> &st,
                                             PackedStageT<WIN> *pk,
                                             uint32_t b, uint32_t ws, uint32_t n, bool bulk_ok,
                                             uint32_t lane) {
  // Order this warp's earlier generic accesses of the buffer before the
  // asynchronous writes that are about to land in it.
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    const uint32_t nb = bulk_positions<PACKED>(n, bulk_ok);
    if (nb) {
      if constexpr (PACKED) {
        const uint32_t hi_bytes = a.col_hi_bits == 4 ? nb / 2 : nb;
        const uint32_t hi_off = a.col_hi_bits == 4 ? ws / 2 : ws;
        mbar_arrive_expect_tx(&st.bar[b], 6u * nb + hi_bytes);
        bulk_copy_g2s(st.w[b], a.weights + ws, 4u * nb, &st.bar[b]);
        bulk_copy_g2s(pk->lo[b], a.cols_lo + ws, 2u * nb, &st.bar[b]);
        bulk_copy_g2s(pk->hi[b], a.cols_hi + hi_off, hi_bytes, &st.bar[b]);
      } else {
        mbar_arrive_expect_tx(&st.bar[b], 8u * nb);
        bulk_copy_g2s(st.w[b], a.weights + ws, 4u * nb, &st.bar[b]);
        bulk_copy_g2s(st.c[b], a.cols + ws, 4u * nb, &st.bar[b]);
      }
    } else {
      mbar_arrive(&st.bar[b]);
    }
  }
}

// Waits for buffer `b` (bounded), loads the tail, turns weights into
// ln(weight) in place -- once per nnz, lane-parallel -- and validates the
// columns: a column >= dim flags kStatusBadColumn (the call then fails, its
// hashes are not valid output) and is replaced by column 0, so the
// evaluation loop reads only in-bounds parameters without a check per nnz.
// Returns false if the copy did not complete within the spin limit.
template <bool PACKED, uint32_t WIN>
__device__ __forceinline__ bool finish_window(const HashArgs &a, WarpStageT<WIN> &st,
                                              PackedStageT<WIN> *pk,
                                              uint32_t b, uint32_t parity, uint32_t ws,
                                              uint32_t n, bool bulk_ok, uint32_t lane) {
  uint32_t spins = 0;
  while (!mbar_try_wait(&st.bar[b], parity)) {
    if (++spins > kSpinLimit) return false;
  }
  const uint32_t nb = bulk_positions<PACKED>(n, bulk_ok);
  bool bad = false;
  for (uint32_t i = lane; i < n; i += 32) {
    float x;
    uint32_t col;
    if constexpr (PACKED) {
      if (i < nb) {
        x = st.w[b][i];
        const uint32_t h = a.col_hi_bits == 4 ? (pk->hi[b][i >> 1] >> ((i & 1u) * 4)) & 15u
                                              : pk->hi[b][i];
        col = static_cast<uint32_t>(pk->lo[b][i]) | (h << 16);
      } else {
        x = __ldg(a.weights + ws + i);
        col = packed_col(a, ws + i);
      }
    } else if (i < nb) {
      x = st.w[b][i];
      col = st.c[b][i];
    } else if (a.host_csr) {  // mapped host memory: plain loads
      x = a.weights[ws + i];
      col = a.cols[ws + i];
    } else {
      x = __ldg(a.weights + ws + i);
      col = __ldg(a.cols + ws + i);
    }
    if (col >= a.dim) {
      bad = true;
      col = 0;
    }
    st.c[b][i] = col;
    st.w[b][i] = logf(x);
  }
  if (__any_sync(0xFFFFFFFFu, bad) && lane == 0) atomicOr(a.status, kStatusBadColumn);
  if (lane == 0) st.c[b][n] = st.c[b][n + 1] = 0;  // the prefetch slots past the window
  __syncwarp();
  return true;
}

// One position's parameters for the lane's SPL samples.  p: param_index of the
// first (a multiple of SPL, so the three 128- or 64-bit loads are aligned and
// every sample pair lands in adjacent registers for the f32x2 arithmetic).
template <int SPL>
struct Params {
  struct {
    float v[SPL];
  } r, c, b;
  __device__ __forceinline__ void load(const float *__restrict__ p) {
    if constexpr (SPL == 4) {
      const float4 x = __ldg(reinterpret_cast<const float4 *>(p));
      const float4 y = __ldg(reinterpret_cast<const float4 *>(p) + 1);
      const float4 z = __ldg(reinterpret_cast<const float4 *>(p) + 2);
      r.v[0] = x.x; r.v[1] = x.y; c.v[0] = x.z; c.v[1] = x.w;
      b.v[0] = y.x; b.v[1] = y.y; r.v[2] = y.z; r.v[3] = y.w;
      c.v[2] = z.x; c.v[3] = z.y; b.v[2] = z.z; b.v[3] = z.w;
    } else if constexpr (SPL == 2) {
      const float2 x = __ldg(reinterpret_cast<const float2 *>(p));
      const float2 y = __ldg(reinterpret_cast<const float2 *>(p) + 1);
      const float2 z = __ldg(reinterpret_cast<const float2 *>(p) + 2);
      r.v[0] = x.x; r.v[1] = x.y; c.v[0] = y.x; c.v[1] = y.y; b.v[0] = z.x; b.v[1] = z.y;
    } else {
      r.v[0] = __ldg(p);
      c.v[0] = __ldg(p + 2);
      b.v[0] = __ldg(p + 4);
    }
  }
};

// ---- Packed pairs of float32 (sm_100 f32x2 arithmetic) --------------------
// One add/sub/mul/fma.rn.f32x2 applies the IEEE round-to-nearest operation
// to both halves independently, so a pair computes exactly what two
// __fadd_rn / __fsub_rn / __fmul_rn / __fmaf_rn calls compute, in one issue.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void split(F2 x, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x.v));
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

template <int SPL, bool KEEP>
__device__ __forceinline__ void eval_all(const Params<SPL> &p, float w, uint32_t pos, bool active,
                                         RowState<SPL, KEEP> &st) {
  float t[SPL];
  bool undecided = false;
  if constexpr (SPL % 2 == 0) {
    // fast_t on sample pairs.  The bound is fast_t's; the limit 0.5 - m is
    // one fma, (|qa| + |b|) * -2^-18 + (0.5 - 2^-18), whose single rounding
    // (<= 2^-26) is covered by the additive 2^-18 in m.
    const F2 ww = f2(w, w);
#pragma unroll
    for (int j = 0; j < SPL; j += 2) {
      float y0, y1;
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(p.r.v[j]));
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(p.r.v[j + 1]));
      const F2 qa = mul2(ww, f2(y0, y1));
      const F2 va = add2(qa, f2(p.b.v[j], p.b.v[j + 1]));
      float q0, q1;
      split(qa, q0, q1);
      float v0, v1;
      split(va, v0, v1);
      t[j] = floorf(v0);
      t[j + 1] = floorf(v1);
      const F2 fr = sub2(va, f2(t[j], t[j + 1]));
      const F2 s = f2(__fadd_rn(fabsf(q0), fabsf(p.b.v[j])),
                      __fadd_rn(fabsf(q1), fabsf(p.b.v[j + 1])));
      const F2 lim = fma2(s, f2(-kTMargin, -kTMargin), f2(0.5f - kTMargin, 0.5f - kTMargin));
      const F2 dv = sub2(fr, f2(0.5f, 0.5f));
      float d0, d1, l0, l1;
      split(dv, d0, d1);
      split(lim, l0, l1);
      undecided |= !(fabsf(d0) < l0) || !(fabsf(d1) < l1);  // NaN -> undecided
    }
  } else {
#pragma unroll
    for (int j = 0; j < SPL; ++j) undecided |= !fast_t(w, p.r.v[j], p.b.v[j], t[j]);
  }
  // Rare: some lane's t sits within the margin of an integer; the warp takes
  // the exact quotient for all its samples (warp-uniform branch).
  if (__any_sync(0xFFFFFFFFu, undecided && active)) {
#pragma unroll
    for (int j = 0; j < SPL; ++j) t[j] = exact_t(w, p.r.v[j], p.b.v[j]);
  }
  if constexpr (SPL % 2 == 0) {
    // ln_a = fma(-(t - beta), r, ln_c) - r on pairs; beta - t is -(t - beta)
    // exactly (round-to-nearest is symmetric).
#pragma unroll
    for (int j = 0; j < SPL; j += 2) {
      const F2 rr = f2(p.r.v[j], p.r.v[j + 1]);
      const F2 nb = sub2(f2(p.b.v[j], p.b.v[j + 1]), f2(t[j], t[j + 1]));
      const F2 ln_a = sub2(fma2(nb, rr, f2(p.c.v[j], p.c.v[j + 1])), rr);
      float l0, l1;
      split(ln_a, l0, l1);
      st.update(j, l0, t[j], pos);
      st.update(j + 1, l1, t[j + 1], pos);
    }
  } else {
#pragma unroll
    for (int j = 0; j < SPL; ++j) {
      const float tb = __fsub_rn(t[j], p.b.v[j]);
      st.update(j, __fsub_rn(__fmaf_rn(-tb, p.r.v[j], p.c.v[j]), p.r.v[j]), t[j], pos);
    }
  }
}

// Per-warp state of the hash kernels: the staging buffers, their barrier
// phases and the launch-wide constants of the item loop.
template <uint32_t WIN>
struct WarpCtxT {
  WarpStageT<WIN> *stg;
  PackedStageT<WIN> *pk;  // packed-column landing area (packed kernels only)
  uint32_t parity;  // bit b: phase parity to wait for on buffer b
  uint32_t lane;
};
using WarpCtx = WarpCtxT<kWin>;

// The warp's staging buffers: its own `stg` and (packed kernels) `pk`.
template <uint32_t WIN>
__device__ __forceinline__ void warp_ctx_init(WarpCtxT<WIN> &w, WarpStageT<WIN> *stg,
                                              PackedStageT<WIN> *pk = nullptr) {
  w.lane = threadIdx.x & 31u;
  w.stg = stg;
  w.pk = pk;
  if (w.lane == 0) {
    mbar_init(&w.stg->bar[0], 1);
    mbar_init(&w.stg->bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  w.parity = 0;
}

// HashArgs of matrix m inside batch b.
__device__ __forceinline__ HashArgs matrix_view(const BatchArgs &b, const BatchMatrix &m,
                                                uint32_t chunk) {
  HashArgs v = b.base;
  v.weights = m.weights;
  v.cols = m.cols;
  v.indptr = m.indptr;
  v.out = m.out;
  v.rows = m.rows;
  v.nnz = m.nnz;
  v.chunk = chunk;
  v.nchunks = m.nchunks;
  v.snap = b.plan->snap;
  v.part_t = b.plan->filter;
  v.chunk_row = b.base.chunk_row + m.chunk_base;
  v.part_ln = b.base.part_ln + static_cast<size_t>(2) * m.chunk_base * b.base.s_pad;
  v.part_kt = b.base.part_kt + static_cast<size_t>(2) * m.chunk_base * b.base.s_pad;
  return v;
}

}  // namespace
}  // namespace mhb

#endif  // MHCUDA_B200_HASH_DEVICE_CUH
