// Internal declarations shared by the kernels (*.cu) and the host engine.
// Nothing here is part of the public ABI (include/minhashcuda*.h is).
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

struct MinhashCudaGenerator_;

namespace mhb {

constexpr uint32_t kNone = 0xFFFFFFFFu;

// Device status word bits (written by kernels, read by the host).
constexpr uint32_t kStatusBadColumn = 1u;  // a column index >= dim was seen
constexpr uint32_t kStatusBadIndptr = 2u;  // row offsets decrease or disagree with nnz
constexpr uint32_t kStatusStall = 4u;      // a bounded wait on a staging copy gave up

// Parameter table: one contiguous block of 3 * s_pad floats per column, its
// samples in pairs r r ln_c ln_c beta beta: r of sample s at
//   params[d * 3 * s_pad + (s / 2) * 6 + s % 2]      (param_index)
// and its ln_c and beta 2 and 4 floats further.  s_pad = samples rounded up to
// a multiple of 4, so a lane can fetch 4 consecutive samples as three aligned
// float4, and a single sample's three values lie in 24 bytes.
inline uint32_t padded_samples(uint32_t samples) { return (samples + 3u) & ~3u; }

// Work decomposition of one hash launch.
//
// The CSR's nnz positions [0, nnz) (relative to indptr[0]) are cut into
// `nchunks` chunks of `chunk` positions (a multiple of 32; of 8 in tiny
// launches, whose columns are never packed).  A row belongs to
// the chunk holding its first position (trailing empty rows to the last
// chunk).  A warp hashes one (chunk, sample-tile) item: it finishes every row
// that lies inside the chunk and leaves a partial arg-min for the row that
// runs in from the previous chunk ("head", slot 2c) and for the row that runs
// out past the chunk's end ("tail", slot 2c+1).  A finalize pass merges the
// partials of every row that crosses a chunk boundary, earlier positions
// winning ties exactly as the reference's strict '<' scan does.
struct HashPlan {
  uint32_t chunk;    // positions per chunk, multiple of 32 (of 8 in tiny launches)
  uint32_t nchunks;  // >= 1
  uint32_t spl;      // samples per lane in one item: 1, 2 or 4
  uint32_t minb;     // kernel variant: minimum resident blocks per SM (4; 3 or 2 for spl 4)
  uint32_t ntiles;   // sample tiles of 32*spl samples (filter: of 16*filter)
  uint32_t grid;     // persistent grid (blocks of plan_block_warps warps)
  uint32_t filter;   // 0: the dense kernel; 8, 4, 2: the bound-filtered one
                     // (filter_kernels.cu) with that many lanes per entry
  uint32_t snap;     // HashArgs::snap
  uint32_t keep;     // dense, 4 blocks per SM: t kept per minimum (RowState)
};

constexpr int kHashBlock = 256;
constexpr int kFilterBlock = 128;

// True when tiles of 32 * spl samples are at least three quarters full.
constexpr bool tile_fills(uint32_t s_pad, uint32_t spl) {
  return 4 * s_pad >= 3 * ((s_pad + 32 * spl - 1) / (32 * spl)) * (32 * spl);
}
// Row stride in bytes of the bound table (one byte per sample): whole
// 32-byte sectors.
constexpr uint32_t bound_stride(uint32_t s_pad) { return (s_pad + 31) & ~31u; }
// Sample counts the filter kernels serve: below 32 the dense kernels read no
// more sectors per entry than the bounds would add.
constexpr uint32_t kFilterMinSamples = 32;
// Most lanes the filter kernels give one entry (16 samples each).
constexpr uint32_t filter_lanes(uint32_t s_pad) { return s_pad > 64 ? 8 : s_pad > 32 ? 4 : 2; }
constexpr uint32_t filter_tiles(uint32_t s_pad, uint32_t lanes) {
  return (s_pad + 16 * lanes - 1) / (16 * lanes);
}
// Threshold arithmetic of the filter kernels (filter_kernels.cu): m is a
// sample's threshold and l an entry's ln(weight), both in steps of 1/20 and
// rounded up, clamped to what 16 bits hold.
constexpr int kThrLimit = 8191;
constexpr int kThrBias = 241 + 16384;
// Below -8192: a threshold of -409.6 lets a few entries more pass.  Above 8191:
// finite weights (l >= -2080) all pass there, as they have to; no value of the
// generator's tables is above 400.
constexpr int clamp_min(int q) { return q < -kThrLimit - 1 ? -kThrLimit - 1 : q < kThrLimit ? q : kThrLimit; }
// Below: only weights of 0, which never win.  Above: only infinite weights,
// whose ln_a of -inf wins whatever the threshold: l + m has to pass byte 255 at
// m = -8192 too, hence the 256 more.
constexpr int clamp_weight(int q) {
  return q < -kThrLimit - 1 ? -kThrLimit - 1 : q < kThrLimit + 256 ? q : kThrLimit + 256;
}
// The 16-bit difference whose bit 15 is clear when the entry passes.
constexpr uint32_t filter_diff(uint32_t byte, int m, int l) {
  return 0xC000u + byte - static_cast<uint32_t>(m + kThrBias) - static_cast<uint32_t>(l);
}
// Samples per lane of the dense kernel: one hash launch of a whole batch or a
// large matrix, and one of `nnz` entries.  Launches under 2^26 evaluations with
// fewer 64-entry items than two per resident warp take one sample per lane, for
// more items.
constexpr uint64_t kSmallItems = 9472;
constexpr uint32_t dense_spl(uint32_t s_pad) {
  return tile_fills(s_pad, 4) ? 4 : tile_fills(s_pad, 2) ? 2 : 1;
}
constexpr uint32_t dense_spl(uint32_t s_pad, uint32_t samples, uint64_t nnz) {
  const uint32_t spl = dense_spl(s_pad), tiles = (s_pad + 32 * spl - 1) / (32 * spl);
  return nnz * samples < (1ull << 26) && nnz / 64 * tiles < kSmallItems ? 1 : spl;
}
// Mean rows below which a dense launch keeps t with each minimum (RowState): an
// instruction more per evaluation, against three gathers, a logarithm and a
// division per (row, sample) at the row's end.  4M entries, without / with it on
// uniform columns [on Zipf ones, whose parameters come from L2]:
//  - 128 samples (s_pad compiled in) rows of 20 1.28 / 1.08 ms [0.72 / 0.67], 70
//    1.12 / 1.03 [0.57 / 0.57], 100 1.08 / 1.02 [0.571 / 0.580], 140 and more 3%
//    faster [2-4% slower]; 64 samples rows of 50 10% faster [0.4% slower], 70 9%
//    faster [2% slower], 140 5% faster [4% slower];
//  - other sample counts never lose: 200 samples rows of 100 5% faster [0.5%],
//    of 500 even.
//  - One sample per lane only in tiny launches (one 300-entry row 21.9 -> 17.8 us
//    alone); 400,000 rows of 20 at 32 samples 0.84 -> 0.99 ms.
//  - Not in device batches, whose mean row the host does not know: 128 samples
//    rows of 10 to 60 1.12-1.07 times as fast [1.14-0.97], of 100 and more 1.04-1.0
//    [0.96-0.93]; 64 samples 0.86-0.99 [1.12-1.0].
constexpr uint32_t keep_rows(uint32_t s_pad, uint32_t spl, bool tiny) {
  if (tiny) return 512;
  if (spl == 4 && (s_pad == 128 || s_pad == 256)) return 96;
  if (spl == 2 && s_pad == 64) return 64;
  return spl > 1 ? 512 : 0;
}

// Which launches the filter kernels hash.  They evaluate 11-17 candidates per
// (row, sample) whatever the row's length, the dense ones every entry; and their
// warps wait longer for each step, which small launches do not hide.  On Zipf(1.1)
// columns, whose parameters come from L2, the dense kernels are faster than on
// uniform columns over large tables, where they wait for HBM; the host knows
// neither, so the lines lie where Zipf columns stop losing (by a few percent
// where uniform ones gain a fifth).  The mean row that takes falls as launches
// grow.  Dense / filtered time over 16,767 launches and 4,482 device batches of
// 32 to 512 samples, rows of even length and ragged ones, as geometric means on
// Zipf [uniform] columns for mean rows of 105-120, 150-170 and 215-250 entries:
//  - full dense tiles (128, 256, 384 samples): 134-168M evaluations .71 [.98], .81
//    [1.16], .98 [1.26]; 268-400M .77 [.98], .90 [1.20], 1.01 [1.39]; 800-1200M .93
//    [1.17], 1.11 [1.31], 1.25 [1.54]; above 1800M 1.00 [1.18], 1.19 [1.42], 1.44
//    [1.78]; at 67-134M .92-.99 [1.15-1.33] even in rows of 400;
//  - 64 samples: 268-400M .78 [.84], .88 [.97], 1.04 [1.29]; 800-1200M .80 [.98],
//    .94 [1.18], 1.09 [1.52]; above 1800M .88 [1.0], 1.02 [1.21], 1.29 [1.35];
//  - tiles filled less (96, 100, 200): 168-268M .86 [.98], 1.00 [1.19], 1.18 [1.35];
//    800-1200M 1.07 [1.07], 1.34 [1.31], 1.51 [1.79];
//  - two samples per lane (48, 60, 160): 67-100M .86 [.96], .96 [1.13], 1.17 [1.31];
//    168-268M .95 [.97], 1.10 [1.14], 1.34 [1.26];
//  - one sample per lane (32, 80): 67-100M 1.11 [1.19], 1.11 [1.46], 1.29 [1.48];
//  - small launches of 128 samples, which the dense kernel takes with one sample per
//    lane: 25-38M .86 [.99], .99 [1.09], 1.08 [1.27]; 38-67M .93 [1.18], 1.15 [1.34],
//    1.15 [1.43]; 12-25M rows of 190 .98 [1.1], of 300 1.03-1.09 [1.18-1.29];
//  - long rows, which dense chunks cut into many partials: rows of 12,000 at 70M 1.05;
//  - a device batch of 128 or 256 samples, whose tiles are always the widest: rows of
//    170 and 300 at 268-400M .84 [1.22], 1.01 [1.19], at 400-600M 1.10 [1.23], 1.10
//    [1.38]; rows of 135 at 1200-1800M 1.03 [1.31].
struct FilterRule {
  uint32_t min_row;                // entries of the mean row (filter_row)
  uint64_t min_evals, min_batch;   // evaluations of a launch, of a device batch
};
constexpr FilterRule filter_rule(uint32_t s_pad) {
  const uint32_t spl = dense_spl(s_pad);
  const uint32_t lanes = (s_pad + 32 * spl - 1) / (32 * spl) * (32 * spl);
  if (spl == 1) return {104, 1ull << 26, 1ull << 25};
  if (s_pad == 64) return {288, 1ull << 27, 9ull << 26};
  if (spl == 2) return {120, 9ull << 22, 1ull << 27};
  if (5 * s_pad <= 4 * lanes) return {152, 7ull << 24, 1ull << 27};
  return {168, 1ull << 27, 7ull << 26};
}
// The mean row from which a launch of `evals` evaluations is filtered.  A device
// batch needs those of a launch of half its size.
constexpr uint64_t filter_row(uint64_t row, uint64_t evals) {
  if (row <= 104) return row;
  if (evals < 1ull << 26) row = 2 * row;
  else if (evals < 5ull << 25) row = row * 5 / 4 < 288 ? row * 5 / 4 : 288;
  else if (evals >= 3ull << 30) row = row / 2;
  else if (evals >= 3ull << 29) row = row * 5 / 8;
  else if (evals >= 3ull << 28) row = row * 3 / 4;
  return row > 104 ? row : 104;
}
// Rows (and one per matrix) from which a device batch launches both kernels, one
// of which returns at once: 2 us of a batch that takes 55-80 with 600 rows of 100
// entries.  Fewer rows reach min_batch only with over 4096 entries each.
constexpr uint64_t filter_batch_rows(uint32_t s_pad) {
  const uint64_t rows = filter_rule(s_pad).min_batch / (4096ull * s_pad);
  return rows > 512 ? rows : 512;
}
constexpr bool filter_pays(uint32_t s_pad, uint32_t samples, uint64_t nnz, uint64_t rows) {
  const FilterRule rule = filter_rule(s_pad);
  const uint64_t evals = nnz * s_pad;
  if (evals < 1ull << 23) return false;
  if (nnz >= 12288 * rows) return true;
  if (evals < 1ull << 26 && dense_spl(s_pad, samples, nnz) == 1)
    return nnz >= (evals >= 9ull << 22 ? 120 : evals >= 3ull << 23 ? 144 : 320) * rows;
  return evals >= rule.min_evals && nnz >= filter_row(rule.min_row, evals) * rows;
}

// Whether a parameter table is one the filter kernels were made for.  Their
// guesses and thresholds expect row minima of a generator's distribution; with
// others every entry passes or samples are scanned twice, and the dense kernels
// are up to 17 times faster (128 samples, rows of 1400
// entries: ln_c - 500 4.5 ms against 0.77, ln_c + 6 12.1, ln_c + 1 0.99, all
// entries equal 8.3).  What matters is how many (column, sample) have ln_c - r
// below a value: it is compared at four, over the table and for each sample.
constexpr int kFitCuts = 4;
// In bytes of the bound table (ln_c - r below -8, -6, -4, -2; a byte of 0 counts
// at all of them), and the share of a generator's entries below: ln_c of a
// Gamma(2, 1) variate minus another one, integrated numerically.
constexpr uint32_t fit_byte(int k) { return 80u + 40u * k; }
constexpr double kFitShare[kFitCuts] = {0.0028256, 0.0159236, 0.0811733, 0.3368440};
// counts[s][k]: entries of sample s below cut k, of dim columns.  Beyond six
// standard deviations (and six entries, for expectations near zero) the table
// may be off by a tenth, a shift of ln_c by 0.1, and a sample by half.
inline bool bounds_fit(const uint32_t *counts, uint32_t dim, uint32_t samples) {
  for (int k = 0; k < kFitCuts; ++k) {
    double all = 0.0;
    auto off = [&](double count, double entries, double share) {
      const double e = entries * kFitShare[k];
      return std::abs(count - e) > share * e + 6.0 * std::sqrt(e) + 6.0;
    };
    for (uint32_t s = 0; s < samples; ++s) {
      const double n = counts[s * kFitCuts + k];
      if (off(n, dim, 0.5)) return false;
      all += n;
    }
    if (off(all, static_cast<double>(dim) * samples, 0.1)) return false;
  }
  return true;
}
// Work division of a filtered launch over `total` = entries x sample tiles and
// `warps` resident warps: positions per chunk and the snap distance.  `waves`
// chunks per warp, but none shorter than a mean row as long as that leaves
// `parts` per warp, nor than 128 positions; rows are kept whole up to two such
// parts.  parts: eight, or min_items if that is more (a server that wants short
// items): rows in pieces start their search anew.
struct FilterSplit {
  uint32_t chunk, snap;
};
__host__ __device__ inline FilterSplit filter_split(uint64_t total, uint64_t warps, uint64_t waves,
                                                    uint64_t avg_row, uint32_t min_items = 8) {
  const uint64_t share = total / warps;
  const uint64_t parts = min_items > 8 ? min_items : 8;
  const uint64_t shortest = share / (min_items > waves ? min_items : waves);
  const uint64_t whole = share / parts < avg_row ? share / parts : avg_row;
  uint64_t chunk = shortest > whole ? shortest : whole;
  chunk = chunk < 128 ? 128 : chunk > (1u << 24) ? (1u << 24) : (chunk + 31) & ~31ull;
  uint64_t snap = 2 * share / parts < 8192 ? 2 * share / parts : 8192;
  snap = snap > chunk ? snap : chunk;
  return FilterSplit{static_cast<uint32_t>(chunk), static_cast<uint32_t>(snap)};
}

struct HashArgs {
  const float *params;       // [dim][s_pad / 2][r r c c b b], see param_index
  uint32_t dim;
  uint32_t samples;
  uint32_t s_pad;
  const float *weights;      // CSR values, weights[p] for relative position p
  const uint32_t *cols;      // CSR column indices
  const uint32_t *indptr;    // rows+1 absolute offsets, indptr[0] = base
  uint32_t rows;
  uint32_t nnz;              // indptr[rows] - indptr[0]
  uint32_t chunk;
  uint32_t nchunks;
  uint32_t ntiles;
  uint32_t *chunk_row;       // [nchunks] first row owned by each chunk
  float *part_ln;            // [2*nchunks][s_pad] partial minima
  uint2 *part_kt;            // [2*nchunks][s_pad] partial (position of the minimum, its t or 0)
  uint32_t *out;             // [rows][samples][2]
  uint32_t *status;          // device status word
  uint32_t host_csr;         // weights/cols/indptr/out are mapped host memory
  // Packed columns (col_hi_bits 4 or 8; cols unused): column p is
  // cols_lo[p] | hi(p) << 16, hi(p) the nibble p of cols_hi (4: entry p in
  // byte p/2, low nibble for even p) or its byte p (8).  Device memory, both
  // arrays 16-byte aligned.  col_hi_bits 0: the columns are `cols`.
  const uint16_t *cols_lo;
  const uint8_t *cols_hi;
  uint32_t col_hi_bits;
  // Lower bounds of ln_c - r ([dim][b_stride] bytes, filter_kernels.cu), or
  // nullptr when the generator has none.
  const uint8_t *bounds;
  uint32_t b_stride;
  // Filtered launches: a chunk begins at the next row when that is at most
  // `snap` positions away (chunk_begin); warps take items off *next_item,
  // which the plan kernel sets to 0.  0 and nullptr for dense launches.
  uint32_t snap;
  uint32_t *next_item;
  uint32_t part_t;           // partials carry t (filtered and KEEP launches)
};

// One matrix of a device-resident batch (mhcuda_calc_batch_device).  The
// host fills the CSR pointers, rows and plan_base; batch_setup_kernel fills
// nnz, chunk_base and nchunks on the device.
struct BatchMatrix {
  const float *weights;    // weights[p] for relative position p
  const uint32_t *cols;
  const uint32_t *indptr;  // rows+1 absolute offsets, indptr[0] = offset of weights[0]
  uint32_t *out;           // [rows][samples][2]
  uint32_t rows;
  uint32_t nnz;
  uint32_t chunk_base;     // index of its first chunk in the batch's chunk space
  uint32_t nchunks;        // 0 for a matrix without rows
};

// Work decomposition of a batch, computed on the device.
struct BatchPlan {
  uint32_t chunk;    // positions per chunk, the same for every matrix
  uint32_t nchunks;  // chunks of all matrices
  uint32_t filter;   // the bound-filtered launch does the work, not the dense one
  uint32_t snap;     // its HashArgs::snap
};

struct BatchArgs {
  HashArgs base;          // generator fields, ntiles, status and the batch-wide scratch
                          // (chunk_row, part_ln, part_kt indexed by batch chunk)
  BatchMatrix *mats;      // [count]
  const uint32_t *plan_base;  // [count] first plan thread of each matrix (rows+1 each)
  uint32_t count;
  uint32_t max_chunks;    // chunk slots the scratch holds
  BatchPlan *plan;
  uint32_t *chunk_owner;  // [max_chunks] matrix of each batch chunk
  // [0] the dense kernel, [1] the filtered one:
  uint64_t warps[2];   // resident warps
  uint64_t waves;      // items per resident warp to aim for
  uint32_t ntiles[2];
  // A batch is filtered when its entries reach filter_min_nnz and its mean row
  // has filter_row(filter_min_row, half its evaluations); 0: never (then only
  // the dense kernel is launched), 1: whatever the row.
  uint32_t filter_min_row;
  uint64_t filter_min_nnz;
};

// Launchers (hash_kernels.cu).  All enqueue on `stream` and return the launch
// error, if any.
cudaError_t launch_plan(const HashArgs &a, cudaStream_t stream, bool clear_status = false);
cudaError_t launch_hash(const HashArgs &a, const HashPlan &plan, cudaStream_t stream);
cudaError_t launch_finalize(const HashArgs &a, cudaStream_t stream);
// A whole device-resident batch: setup (per-matrix nnz, chunk size, chunk
// tables), plan, one persistent hash launch over all matrices' chunks and
// finalize.  dense.spl/minb/grid select the dense variant; with
// b.filter_min_row the filtered one (filtered.grid) is launched too and the
// one that setup did not choose returns at once.  plan_threads is the sum of
// rows+1 over the matrices that have rows.
cudaError_t launch_batch(const BatchArgs &b, const HashPlan &dense, const HashPlan &filtered,
                         uint32_t plan_threads, cudaStream_t stream);
// The bound-filtered hash launches behind launch_hash / launch_batch, their
// resident blocks per SM (filter_kernels.cu).
cudaError_t launch_filter(const HashArgs &a, const HashPlan &plan, cudaStream_t stream);
cudaError_t launch_filter_batch(const BatchArgs &b, const HashPlan &plan, cudaStream_t stream);
int filter_blocks_per_sm(uint32_t s_pad, uint32_t lanes);
// Blocks per SM the hash kernel variant launched for (samples per lane,
// register budget, s_pad) reaches, and its registers per thread.
int hash_blocks_per_sm(uint32_t spl, uint32_t minb, uint32_t s_pad);
// The same for the kernel a plan selects.
int plan_blocks_per_sm(const HashPlan &plan, uint32_t s_pad);
// Warps per block of that kernel.
constexpr uint32_t plan_block_warps(const HashPlan &plan) {
  return (plan.filter ? kFilterBlock : kHashBlock) / 32;
}
size_t hash_kernel_registers(uint32_t spl, uint32_t minb, uint32_t s_pad);

// Parameter kernels (param_kernels.cu).
// Blocks of sample rows in [samples][dim] order: the five uniform runs U1..U5
// (draw), or r, ln_c and beta themselves.
struct ParamSources {
  const float *src[5];
};
// Fills samples [s_base, s_base + samples) of every column of the parameter
// table and, if there is one, of the bound table (bound_byte).  parts: bits 0,
// 1, 2 for r, ln_c, beta; the bound table is written when all are.  counts (not
// draw; or nullptr): what bounds_fit compares, added to counts[s_base + s].
cudaError_t launch_pack_params(const ParamSources &in, bool draw, uint32_t parts, uint32_t dim, uint32_t s_base,
                               uint32_t samples, uint32_t s_pad, float *params, uint8_t *bounds,
                               uint32_t *counts, cudaStream_t stream);
// dst[s*dim + d] = r, ln_c or beta (which 0, 1, 2) of column d, sample
// s_base + s, for s < samples.
cudaError_t launch_unpack_params(const float *params, uint32_t which, uint32_t dim,
                                 uint32_t s_base, uint32_t samples, uint32_t s_pad, float *dst,
                                 cudaStream_t stream);
cudaError_t launch_logf(const float *in, float *out, size_t n, cudaStream_t stream);

// memcpy for host staging moves: non-temporal stores for large pieces
// (host_copy.cc).
void stream_copy(void *dst, const void *src, size_t bytes);
// float64 -> float32 (round to nearest) and 64-bit -> uint32 (values outside
// [0, 2^32) become 0xFFFFFFFF), with non-temporal stores for large pieces.
void convert_f64_to_f32(float *dst, const double *src, size_t n);
void convert_i64_to_u32(uint32_t *dst, const uint64_t *src, size_t n);
// Packed columns for the host->device link: lo[i] = low 16 bits of src[i],
// hi = the bits above, as bytes (hi_bits 8: hi[i]) or nibbles (hi_bits 4:
// entry i in byte i/2, the low nibble for even i).  Returns false if some
// column needs more than 16 + hi_bits bits.  A range split across calls must
// be split at even entries.
bool pack_cols(const uint32_t *src, size_t n, uint16_t *lo, uint8_t *hi, int hi_bits);

// Makes `device` current for the calling thread while the guard lives and
// then gives the thread back the state it came with: its previous device, or
// no current context at all when it had none (restoring "device 0" there
// would create a context on device 0 that the caller never asked for).
// Every extern "C" entry point that works on a device holds one.
class DeviceGuard {
 public:
  explicit DeviceGuard(int device);
  ~DeviceGuard();
  DeviceGuard(const DeviceGuard &) = delete;
  DeviceGuard &operator=(const DeviceGuard &) = delete;
  bool ok() const { return ok_; }

 private:
  int prev_ = -1;
  bool had_context_ = true;
  bool changed_ = false;
  bool ok_ = false;
};

// Read-only view of a generator's fields for entry points that live outside
// engine.cu (engine.cu).
struct GeneratorView {
  const float *params;
  const uint8_t *bounds;  // nullptr: no bound table
  uint32_t dim;
  uint32_t samples;
  uint32_t s_pad;
  int device;
  int sm_count;
  int verbosity;
  cudaStream_t stream;
};
bool generator_view(const MinhashCudaGenerator_ *gen, GeneratorView *view);
// The engine's work decomposition for `nnz` entries in `rows` rows, with at
// least `min_items` warp items per resident warp where chunks allow.
// allow_filter: false for a CSR in mapped host memory, which the filtered
// kernels would read twice.
HashPlan plan_for_generator(const MinhashCudaGenerator_ *gen, uint64_t nnz, uint64_t rows,
                            uint32_t min_items = 8, bool allow_filter = true);

}  // namespace mhb
