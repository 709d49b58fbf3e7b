// FP64 contractions (sm_103a).
//
// FP64 is the scarce unit here: 1.05 TFLOP/s whether issued as DMMA or FMA,
// 1.7 FMA per clock and SM, so a warp's FMA occupies its sub-partition for
// about 74 clocks.  Loads, index lookups and shuffles between them are free by
// comparison; what counts is how many FMAs a call issues, padding and zeros
// included, and that every SM has its share of them.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "engine.h"
#include "once.h"

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

// ------------------------------------------------------------------ GEMMs
// C[coff(row tile) + n ldc + r] = sum_k A[row][vl[k]] B[n][k] for a list of
// problems in one launch (DMMA m8n8k4).  A block is a 32 x 32 tile, a warp 16 x
// 16 of it, operands straight from L1 and L2: a step of 16 k keeps a
// sub-partition's FP64 pipe busy for 9500 clocks, so nothing else shows, and
// small tiles fill the GPU at small sizes and waste little at ragged ones
// (64 x 64 tiles, one launch per final block: 27 tiles of 300 us for a 187 x 561
// problem; C2v N = 200, J <= 2: 4.6 ms of GEMMs, 0.6 ms this way).
struct ParamsF {
  ProbF p[kMaxProbF];
  int nprob;
};
__global__ void __launch_bounds__(128) k_gemm_f64(const __grid_constant__ ParamsF P) {
  int q = 0;
  while (q + 1 < P.nprob && P.p[q + 1].first <= (int)blockIdx.x) ++q;
  const ProbF& pr = P.p[q];
  const int local = blockIdx.x - pr.first;
  // row tiles fastest: the blocks in flight share columns of B
  const int rt = local % pr.nM, n0 = (local / pr.nM) * 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  // rows of the tile: at/rowsrc (128-row tiles, four blocks each) or plain rows
  int tile = 0, r0 = rt * 32, rows = pr.M;
  int64_t coff = 0;
  if (pr.at) {
    const ATile a = pr.at[rt >> 2];
    tile = a.tile * 128;
    r0 = (rt & 3) * 32;
    rows = a.rows;
    coff = a.coff;
  }
  if (r0 >= rows) return;
  const int wr = r0 + (warp >> 1) * 16, wc = n0 + (warp & 1) * 16;
  if (wr >= rows || wc >= pr.Nc) return;
  const double *a[2], *b[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = min(wr + i * 8 + g, rows - 1), n = min(wc + i * 8 + g, pr.Nc - 1);
    a[i] = pr.A + (size_t)(pr.at ? pr.rowsrc[tile + r] : r) * pr.lda;
    b[i] = pr.B + (size_t)n * pr.ldb + t;
  }
  double acc[2][2][2] = {};
  double av[2][4], bv[2][4];
  auto fetch = [&](int k) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const int v = pr.vl ? pr.vl[k + kk * 4 + t] : k + kk * 4 + t;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        av[i][kk] = v >= 0 ? a[i][v] : 0.0;
        bv[i][kk] = b[i][k + kk * 4];
      }
    }
  };
  fetch(0);
  for (int k = 0; k < pr.K; k += 16) {
    double ac[2][4], bc[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        ac[i][kk] = av[i][kk];
        bc[i][kk] = bv[i][kk];
      }
    if (k + 16 < pr.K) fetch(k + 16);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          asm volatile(
              "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
              : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
              : "d"(ac[i][kk]), "d"(bc[j][kk]));
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = wr + i * 8 + g, n = wc + j * 8 + t * 2 + e;
        if (r < rows && n < pr.Nc) pr.C[coff + (long long)n * pr.ldc + r] = acc[i][j][e];
      }
}

cudaError_t launch_gemm_f64(std::vector<ProbF> probs, cudaStream_t s) {
  probs.erase(std::remove_if(probs.begin(), probs.end(),
                             [](const ProbF& p) { return p.nM <= 0 || p.Nc <= 0 || p.K <= 0; }),
              probs.end());
  if (probs.empty()) return cudaSuccess;
  if (probs.size() > (size_t)kMaxProbF) return cudaErrorInvalidValue;
  // longest contractions first
  std::stable_sort(probs.begin(), probs.end(),
                   [](const ProbF& a, const ProbF& b) { return a.K > b.K; });
  ParamsF* P = new ParamsF();
  P->nprob = (int)probs.size();
  long long blocks = 0;
  cudaError_t e = cudaSuccess;
  for (int q = 0; q < P->nprob; q++) {
    if (probs[q].K & 15) e = cudaErrorInvalidValue;
    P->p[q] = probs[q];
    P->p[q].first = (int)blocks;
    blocks += (long long)probs[q].nM * ((probs[q].Nc + 31) / 32);
    if (blocks > 0x7FFF0000ll) e = cudaErrorInvalidValue;
  }
  if (e == cudaSuccess) {
    k_gemm_f64<<<(unsigned)blocks, 128, 0, s>>>(*P);
    e = cudaGetLastError();
  }
  delete P;
  return e;
}

static cudaError_t attributes() {
  static OncePerDevice once;
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  return once.run(device, [] {
    const cudaError_t a =
        cudaFuncSetAttribute(k_pack_y, cudaFuncAttributeMaxDynamicSharedMemorySize, kPackSmem);
    return a != cudaSuccess
               ? a
               : cudaFuncSetAttribute(k_dipole_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kPackSmem);
  });
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
