// Parameter-table kernels for sm_100a.
//
// Replace gamma_cuda / log_cuda (kernel.cu:18-36 of src-d/minhashcuda) and
// the layout the reference keeps its table in.  The reference runs
//   U1->rs, U2->ln_cs, U3->betas, rs=-logf(U2*U1), U4->ln_cs,
//   ln_cs=-logf(U3*U4), U5->betas, ln_cs=logf(ln_cs)        (minhashcuda.cc:186-200)
// as three element-wise kernels on [samples][dim] arrays, each followed by a
// device-wide synchronisation.  Here one pass reads a block of sample rows of
// all five uniform runs (or of the three assigned arrays) in [samples][dim]
// order, applies the same float operations (each rounded to float as in the
// reference: -logf(a*b), then logf of that), and writes columns of the table
// (12 contiguous bytes per sample, in pairs r r c c b b) and of the byte table of bounds through shared-memory tiles, so reads and writes are
// coalesced and neither table is read back.
#include <cstdint>

#include "hash_device.cuh"
#include "wmh_internal.h"

namespace mhb {
namespace {

constexpr int kTile = 32;
constexpr int kRowsPerPass = 8;

// Block of 256: tile of 8 samples x 128 columns.  The sources hold `samples`
// rows of `dim` values, the rows s_base.. of the [samples][dim] streams.
// PARTS: bits 0, 1, 2 for r, ln_c, beta; only their sources are read and only
// they are written (bounds need all three).  Bound by HBM (five floats in,
// three and a byte out): eight samples of a column are 96 contiguous bytes,
// whole sectors, for blocks of any multiple of eight sample rows.
constexpr uint32_t kPackS = 8, kPackD = 128;

template <bool DRAW>
__global__ void __launch_bounds__(256) pack_kernel(const ParamSources in, uint32_t parts,
                                                   uint32_t dim, uint32_t s_base, uint32_t samples,
                                                   uint32_t s_pad, float *__restrict__ params,
                                                   uint32_t b_stride, uint8_t *__restrict__ bounds,
                                                   uint32_t *__restrict__ counts) {
  __shared__ float tile[3][kPackS][kPackD + 1];
  const uint32_t d0 = blockIdx.x * kPackD;
  const uint32_t s0 = blockIdx.y * kPackS;
  // Read [s][d] rows, coalesced along d.
#pragma unroll
  for (uint32_t n = threadIdx.x; n < kPackS * kPackD; n += 256) {
    const uint32_t k = n / kPackD, x = n % kPackD;
    const uint32_t s = s0 + k, d = d0 + x;
    if (s < samples && d < dim) {
      const size_t i = static_cast<size_t>(s) * dim + d;
      if constexpr (DRAW) {
        // kernel.cu:24 with v1 * v2 of the runs (U2, U1) and (U3, U4), then
        // kernel.cu:35 for the second.
        if (parts & 1u) tile[0][k][x] = -logf(in.src[1][i] * in.src[0][i]);
        if (parts & 2u) {
          const float g = -logf(in.src[2][i] * in.src[3][i]);
          tile[1][k][x] = logf(g);
        }
        if (parts & 4u) tile[2][k][x] = in.src[4][i];
      } else {
#pragma unroll
        for (int m = 0; m < 3; ++m)
          if (parts >> m & 1u) tile[m][k][x] = in.src[m][i];
      }
    }
  }
  __syncthreads();
  // Write columns: the tile's 24 floats of a column are contiguous when
  // s_base is even.
#pragma unroll
  for (uint32_t n = threadIdx.x; n < kPackD * 3 * kPackS; n += 256) {
    const uint32_t x = n / (3 * kPackS), f = n % (3 * kPackS);
    const uint32_t s = f / 6 * 2 + (f & 1u), which = f % 6 / 2;
    if (d0 + x < dim && s0 + s < samples && (parts >> which & 1u))
      params[static_cast<size_t>(d0 + x) * 3 * s_pad + param_index(s_base + s0 + s) + 2 * which] =
          tile[which][s][x];
  }
  if (!bounds || parts != 7u) return;
  uint32_t below[kFitCuts] = {};  // of sample threadIdx.x % kPackS, this thread's columns
#pragma unroll
  for (uint32_t n = threadIdx.x; n < kPackD * kPackS; n += 256) {
    const uint32_t x = n / kPackS, s = n % kPackS;
    if (d0 + x < dim && s0 + s < samples) {
      const uint32_t byte = bound_byte(tile[0][s][x], tile[1][s][x], tile[2][s][x]);
      bounds[static_cast<size_t>(d0 + x) * b_stride + s_base + s0 + s] = static_cast<uint8_t>(byte);
      if constexpr (!DRAW) {
#pragma unroll
        for (int k = 0; k < kFitCuts; ++k) below[k] += byte < fit_byte(k);
      }
    }
  }
  if constexpr (!DRAW) {
    if (!counts) return;
    __shared__ uint32_t sums[kPackS][kFitCuts];
    if (threadIdx.x < kPackS * kFitCuts) sums[threadIdx.x / kFitCuts][threadIdx.x % kFitCuts] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFitCuts; ++k)
      if (below[k]) atomicAdd(&sums[threadIdx.x % kPackS][k], below[k]);
    __syncthreads();
    const uint32_t s = threadIdx.x / kFitCuts, k = threadIdx.x % kFitCuts;
    if (s < kPackS && s0 + s < samples && sums[s][k])
      atomicAdd(&counts[static_cast<size_t>(s_base + s0 + s) * kFitCuts + k], sums[s][k]);
  }
}

__global__ void unpack_kernel(const float *__restrict__ params, uint32_t which, uint32_t dim,
                              uint32_t s_base, uint32_t samples, uint32_t s_pad,
                              float *__restrict__ dst) {
  __shared__ float tile[kTile][kTile + 1];
  const uint32_t d0 = blockIdx.x * kTile;
  const uint32_t s0 = blockIdx.y * kTile;
  for (int k = threadIdx.y; k < kTile; k += kRowsPerPass) {
    const uint32_t d = d0 + k, s = s0 + threadIdx.x;
    if (d < dim && s < samples)
      tile[k][threadIdx.x] =
          params[static_cast<size_t>(d) * 3 * s_pad + param_index(s_base + s) + 2 * which];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < kTile; k += kRowsPerPass) {
    const uint32_t s = s0 + k, d = d0 + threadIdx.x;
    if (s < samples && d < dim) dst[static_cast<size_t>(s) * dim + d] = tile[threadIdx.x][k];
  }
}

}  // namespace

cudaError_t launch_pack_params(const ParamSources &in, bool draw, uint32_t parts, uint32_t dim, uint32_t s_base,
                               uint32_t samples, uint32_t s_pad, float *params, uint8_t *bounds,
                               uint32_t *counts, cudaStream_t stream) {
  const dim3 block(256);
  const dim3 grid((dim + kPackD - 1) / kPackD, (samples + kPackS - 1) / kPackS);
  if (grid.x == 0 || grid.y == 0) return cudaSuccess;
  const uint32_t stride = bound_stride(s_pad);
  if (draw) {
    pack_kernel<true><<<grid, block, 0, stream>>>(in, parts, dim, s_base, samples, s_pad, params,
                                                  stride, bounds, nullptr);
  } else {
    pack_kernel<false><<<grid, block, 0, stream>>>(in, parts, dim, s_base, samples, s_pad, params,
                                                   stride, bounds, counts);
  }
  return cudaGetLastError();
}

cudaError_t launch_unpack_params(const float *params, uint32_t which, uint32_t dim,
                                 uint32_t s_base, uint32_t samples, uint32_t s_pad, float *dst,
                                 cudaStream_t stream) {
  const dim3 block(kTile, kRowsPerPass);
  const dim3 grid((dim + kTile - 1) / kTile, (samples + kTile - 1) / kTile);
  if (grid.x == 0 || grid.y == 0) return cudaSuccess;
  unpack_kernel<<<grid, block, 0, stream>>>(params, which, dim, s_base, samples, s_pad, dst);
  return cudaGetLastError();
}

}  // namespace mhb
