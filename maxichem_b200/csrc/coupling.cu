// The GCM step's conversions either side of a call (maxichem/coupling/composition.py:102-183 of the reference): mass
// mixing ratios q [B][ns] to mole fractions x = (q / mw) / sum(q / mw), and back, q = x mw (mass / sum(x mw)). One
// warp per cell streams its row (consecutive lanes, consecutive addresses), so each conversion reads and writes
// [B][ns] once: the FP64 divisions and HBM share the time. Row sums are formed in the warp's order (lane l adds entries
// l, l + 32, ..., then a butterfly). Problems are reported as bits or-ed into one word for the host to explain.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <type_traits>

#include "../../include/maxichem_b200.h"

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int WARPS = 8;  // warps (cells in flight) per block

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

// q -> x. bad bits: 1 a non-finite q, 2 a negative q (unless signed_ok), 4 a cell whose sum of q / mw is not above 0.
// A lane keeps its R = ceil(ns / 32) quotients (species lane, lane + 32, ...) between the sum and the result: the FP64
// divisions, not the memory, were the time, three per value and now two, and the row's loads are under way together.
// R is exact, since a row of padding alone costs its divisions too. Microseconds of 262,144 cells with a quotient
// formed anew for each use, and so: 5 species 58 and 54, 69 species 150 and 105, 128 species 210 and 110, 254 species
// 524 and 247 (with R 2, 3 or 8 only: 83, 106, 251 and 247).
template <int R>
__global__ void __launch_bounds__(32 * WARPS) mass_to_mole_kernel(const double* __restrict__ q,
                                                                  const double* __restrict__ mw, int64_t B, int ns,
                                                                  int signed_ok, double* __restrict__ x,
                                                                  int* __restrict__ bad) {
  const int lane = threadIdx.x & 31;
  int flags = 0;
  double m[R];
#pragma unroll
  for (int p = 0; p < R; p++) m[p] = lane + 32 * p < ns ? __ldg(mw + lane + 32 * p) : 1.0;
  for (int64_t cell = (int64_t)blockIdx.x * WARPS + (threadIdx.x >> 5); cell < B; cell += (int64_t)gridDim.x * WARPS) {
    const double* qc = q + cell * ns;
    double* xc = x + cell * ns;
    double part = 0.0, v[R];
#pragma unroll
    for (int p = 0; p < R; p++) v[p] = lane + 32 * p < ns ? qc[lane + 32 * p] : 0.0;
#pragma unroll
    for (int p = 0; p < R; p++) {
      flags |= isfinite(v[p]) ? 0 : 1;
      flags |= (!signed_ok && v[p] < 0.0) ? 2 : 0;
      v[p] = v[p] / m[p];
      if (lane + 32 * p < ns) part += v[p];
    }
    const double total = warp_sum(part);
    flags |= (!signed_ok && !(total > 0.0)) ? 4 : 0;
#pragma unroll
    for (int p = 0; p < R; p++)
      if (lane + 32 * p < ns) xc[lane + 32 * p] = v[p] / total;
  }
  flags = __reduce_or_sync(FULL, flags);
  if (lane == 0 && flags) atomicOr(bad, flags);
}

// x, mass -> q. bad bits: 1 a non-finite x, 2 a negative x, 4 a cell whose sum of x mw is not above 0, 8 a mass that
// is negative or not finite
template <int R>
__global__ void __launch_bounds__(32 * WARPS) mole_to_mass_kernel(const double* __restrict__ x,
                                                                  const double* __restrict__ mw,
                                                                  const double* __restrict__ mass, int64_t B, int ns,
                                                                  double* __restrict__ q, int* __restrict__ bad) {
  const int lane = threadIdx.x & 31;
  int flags = 0;
  double m[R];
#pragma unroll
  for (int p = 0; p < R; p++) m[p] = lane + 32 * p < ns ? __ldg(mw + lane + 32 * p) : 0.0;
  for (int64_t cell = (int64_t)blockIdx.x * WARPS + (threadIdx.x >> 5); cell < B; cell += (int64_t)gridDim.x * WARPS) {
    const double* xc = x + cell * ns;
    double* qc = q + cell * ns;
    double part = 0.0, v[R];
#pragma unroll
    for (int p = 0; p < R; p++) v[p] = lane + 32 * p < ns ? xc[lane + 32 * p] : 0.0;
    const double total = mass[cell];
#pragma unroll
    for (int p = 0; p < R; p++) {
      flags |= isfinite(v[p]) ? 0 : 1;
      flags |= v[p] < 0.0 ? 2 : 0;
      v[p] = v[p] * m[p];
      if (lane + 32 * p < ns) part += v[p];
    }
    const double weight = warp_sum(part);
    flags |= weight > 0.0 ? 0 : 4;
    flags |= (isfinite(total) && total >= 0.0) ? 0 : 8;
    const double f = total / weight;
#pragma unroll
    for (int p = 0; p < R; p++)
      if (lane + 32 * p < ns) qc[lane + 32 * p] = v[p] * f;
  }
  flags = __reduce_or_sync(FULL, flags);
  if (lane == 0 && flags) atomicOr(bad, flags);
}

int grid_for(int64_t B) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t blocks = (B + WARPS - 1) / WARPS;
  const int64_t most = (int64_t)sms * 8;  // 8 blocks of 256 threads per SM
  return (int)(blocks < most ? (blocks > 0 ? blocks : 1) : most);
}

// f with the row count r (1 .. MAX_ROWS) as a constant
constexpr int MAX_ROWS = (MX_MAX_SPECIES + 31) / 32;
template <int R = 1, class F>
void for_rows(int r, const F& f) {
  if (r == R)
    f(std::integral_constant<int, R>{});
  else if constexpr (R < MAX_ROWS)
    for_rows<R + 1>(r, f);
}

}  // namespace

extern "C" int mx_mass_to_mole(const double* q, const double* mw, int64_t B, int32_t ns, int32_t signed_ok,
                               double* x, int32_t* bad, void* stream) {
  if (B < 0 || ns < 1 || ns > MX_MAX_SPECIES || !mw || !bad || (B > 0 && (!q || !x))) return MX_ERR_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(bad, 0, sizeof(int32_t), st);
  if (e == cudaSuccess && B > 0) {
    for_rows((ns + 31) / 32, [&](auto rows) {
      mass_to_mole_kernel<decltype(rows)::value><<<grid_for(B), 32 * WARPS, 0, st>>>(q, mw, B, ns, signed_ok, x, bad);
    });
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? MX_OK : MX_ERR_CUDA;
}

extern "C" int mx_mole_to_mass(const double* x, const double* mw, const double* mass, int64_t B, int32_t ns,
                               double* q, int32_t* bad, void* stream) {
  if (B < 0 || ns < 1 || ns > MX_MAX_SPECIES || !mw || !bad || (B > 0 && (!x || !mass || !q))) return MX_ERR_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(bad, 0, sizeof(int32_t), st);
  if (e == cudaSuccess && B > 0) {
    for_rows((ns + 31) / 32, [&](auto rows) {
      mole_to_mass_kernel<decltype(rows)::value><<<grid_for(B), 32 * WARPS, 0, st>>>(x, mw, mass, B, ns, q, bad);
    });
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? MX_OK : MX_ERR_CUDA;
}
