// FP64 contractions (sm_103a).
//
// FP64 is the scarce unit here: 1.05 TFLOP/s whether issued as DMMA or FMA,
// 1.7 FMA per clock and SM, so a warp's FMA occupies its sub-partition for
// about 74 clocks.  Loads, index lookups and shuffles between them are free by
// comparison; what counts is how many FMAs a call issues, padding and zeros
// included, and that every SM has its share of them.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "engine.h"

namespace gi {

// ------------------------------------------------------------------ one vector
// The half line strength of one vector has a column of Y per (k, tau) slot,
// most of them half zeros (a symmetry leaves a slot only some functions).  Each
// column is packed to its non-zero values and their places, and a block
// contracts four rows of the dipole with every packed column: exactly the
// non-zero products.  (64-wide GEMM tiles spent 64 columns of products on 21:
// N = 2000, J = 10 took 2360 us, packed 274 us.)

constexpr int kPackSmem = 200 * 1024;  // longest row packed (25,600 functions)

// Row `slot` of Y in place: n values, then their places as int32, count n; or
// left as it is with count -1 when that would not fit the row.
__global__ void __launch_bounds__(256) k_pack_y(double* __restrict__ Y, int N, int Kp, int fits,
                                                int32_t* __restrict__ count) {
  extern __shared__ __align__(16) double row[];
  __shared__ int part[256];
  double* y = Y + (size_t)blockIdx.x * Kp;
  if (!fits) {
    if (threadIdx.x == 0) count[blockIdx.x] = -1;
    return;
  }
  for (int v = threadIdx.x; v < N; v += 256) row[v] = y[v];
  __syncthreads();
  const int per = (N + 255) / 256, a = min((int)threadIdx.x * per, N), b = min(a + per, N);
  int c = 0;
  for (int v = a; v < b; ++v) c += row[v] != 0.0;
  part[threadIdx.x] = c;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {
    const int s = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += s;
    __syncthreads();
  }
  const int n = part[255];
  if (n * 12 > Kp * 8) {
    if (threadIdx.x == 0) count[blockIdx.x] = -1;
    return;
  }
  int32_t* at = reinterpret_cast<int32_t*>(y + n);
  int j = part[threadIdx.x] - c;
  for (int v = a; v < b; ++v)
    if (row[v] != 0.0) {
      y[j] = row[v];
      at[j++] = v;
    }
  if (threadIdx.x == 0) count[blockIdx.x] = n;
}

// Z_c[slot][f] = sum_v mu_c(v, f) Y[slot][v]: block = four rows f of component
// blockIdx.y, staged in shared memory when they fit; a warp takes every fourth
// slot, its lanes the slot's values.
constexpr int kRows = 4;
__global__ void __launch_bounds__(128)
    k_dipole_rows(const double* __restrict__ mu, size_t mstride, int Kp, int rows,
                  const double* __restrict__ Y, const int32_t* __restrict__ count, int nslot,
                  int N, int staged, double* __restrict__ Z, size_t zc, int ldz) {
  extern __shared__ __align__(16) double sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int f0 = blockIdx.x * kRows, nr = min(kRows, rows - f0);
  const double* m = mu + blockIdx.y * mstride + (size_t)f0 * Kp;
  const double* r[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) r[i] = m + (size_t)min(i, nr - 1) * Kp;
  if (staged) {
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const double2* src = reinterpret_cast<const double2*>(r[i]);
      double2* dst = reinterpret_cast<double2*>(sm + (size_t)i * Kp);
      for (int k = threadIdx.x; k < Kp / 2; k += 128) dst[k] = src[k];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kRows; ++i) r[i] = sm + (size_t)i * Kp;
  }
  for (int slot = warp; slot < nslot; slot += 4) {
    const double* y = Y + (size_t)slot * Kp;
    // (bounded: lists that another call is overwriting must not send a read
    // out of the row)
    const int cnt = count[slot], n = cnt < 0 ? N : min(cnt, Kp * 2 / 3);
    const int32_t* at = reinterpret_cast<const int32_t*>(y + n);
    double acc[kRows] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
    for (int j = lane; j < n; j += 32) {
      const double x = y[j];
      const int v = cnt < 0 ? j : (int)min((unsigned)at[j], (unsigned)(N - 1));
#pragma unroll
      for (int i = 0; i < kRows; ++i) acc[i] = fma(r[i][v], x, acc[i]);
    }
    // four sums over 32 lanes in six additions: halves of the warp take two
    // rows each, quarters one
    const bool up = lane & 16;
    double p0 = up ? acc[2] : acc[0], p1 = up ? acc[3] : acc[1];
    p0 += __shfl_xor_sync(0xffffffffu, up ? acc[0] : acc[2], 16);
    p1 += __shfl_xor_sync(0xffffffffu, up ? acc[1] : acc[3], 16);
    const bool odd = lane & 8;
    double s = (odd ? p1 : p0) + __shfl_xor_sync(0xffffffffu, odd ? p0 : p1, 8);
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const int i = (up ? 2 : 0) + (odd ? 1 : 0);
    if ((lane & 7) == 0 && i < nr) Z[blockIdx.y * zc + (size_t)slot * ldz + f0 + i] = s;
  }
}

static cudaError_t attributes() {
  static std::once_flag once;
  static cudaError_t status = cudaSuccess;
  std::call_once(once, [] {
    status = cudaFuncSetAttribute(k_pack_y, cudaFuncAttributeMaxDynamicSharedMemorySize, kPackSmem);
    if (status == cudaSuccess)
      status = cudaFuncSetAttribute(k_dipole_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kPackSmem);
  });
  return status;
}

cudaError_t launch_pack_y(double* Y, int nslot, int N, int Kp, int32_t* count, cudaStream_t s) {
  cudaError_t e = attributes();
  if (e != cudaSuccess || nslot <= 0) return e;
  const size_t row = (size_t)N * sizeof(double);
  const int fits = row <= (size_t)kPackSmem;
  k_pack_y<<<nslot, 256, fits ? row : 0, s>>>(Y, N, Kp, fits, count);
  return cudaGetLastError();
}

cudaError_t launch_dipole_rows(const double* mu, size_t mstride, int Kp, int rows, const double* Y,
                               const int32_t* count, int nslot, int N, double* Z, size_t zc,
                               int ldz, cudaStream_t s) {
  cudaError_t e = attributes();
  if (e != cudaSuccess || nslot <= 0 || rows <= 0) return e;
  // staged: two blocks an SM at least
  const size_t sm = (size_t)kRows * Kp * sizeof(double);
  const int staged = sm <= (size_t)100 * 1024;
  k_dipole_rows<<<dim3((rows + kRows - 1) / kRows, 3), 128, staged ? sm : 0, s>>>(
      mu, mstride, Kp, rows, Y, count, nslot, N, staged, Z, zc, ldz);
  return cudaGetLastError();
}

}  // namespace gi
