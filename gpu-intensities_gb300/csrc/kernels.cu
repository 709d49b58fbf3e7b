// Gather/scatter, stencil, epilogue and line order kernels of the line-intensity
// engine (sm_103a).
//
// Factorisation of the reference's half line strength
// (dipole_kernals.cu:162-227).  With keyI = 2kI+tauI, the reference sums
//   h[rF] = sgnF * sum_rI [|kI-kF|<=1] R(keyI,keyF) * mu_c(icontrI, icontrF) * vI[rI]
// where R (sign, L, 3j, 1/sqrt2) and the component c depend only on the two
// keys.  Grouping the initial roots by key gives
//   Y[slotI][v] = sum_{rI: key=slotI, icontrI=v} vI[rI]            (k_build_y)
//   Z_c[slotI][f] = sum_v mu_c(v, f) Y[slotI][v]                    (a GEMM)
//   h[rF] = sum_{terms of keyF} coef * Z_c[slotI][icontrF(rF)]      (k_build_h)
// and the reference's per-final-vector correlate + Ddot (cuda_host.cu:1301-1317)
// becomes a GEMM against H projected back onto the symmetrised basis:
//   H[s] = sum_lambda repres_F[s, idegF, lambda] * h[root(case(s), lambda)].
#include <cuda_runtime.h>

#include <algorithm>

#include "engine.h"
#include "epilogue.cuh"
#include "items.cuh"

namespace gi {

// ------------------------------------------------------------------ Y build
// One thread per (slot, v) element of one column (i, d).  Fuses the
// symmetrised -> primitive transform (dipole_kernals.cu:38-71) with the
// scatter of primitive roots onto their (key, J=0 index) position.
__global__ void k_build_y(const double* __restrict__ vecs, int ld, const int32_t* __restrict__ ivec,
                          int ndeg, const int32_t* __restrict__ yptr,
                          const int32_t* __restrict__ yroot, const int32_t* __restrict__ root_case,
                          const int32_t* __restrict__ root_lam,
                          const int32_t* __restrict__ case_iterm,
                          const int32_t* __restrict__ case_nelem, const double* __restrict__ rep,
                          int Ntot, int degen, int nslot, int N, int Kp, double* __restrict__ Y) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int col = blockIdx.y;  // i * ndeg + d
  const int i = col / ndeg, d = col - i * ndeg;
  if (e >= nslot * Kp) return;
  const int slot = e / Kp, v = e - slot * Kp;
  double acc = 0.0;
  if (v < N) {
    const double* vs = vecs + (size_t)ivec[i] * ld;
    const int q = slot * N + v;
    for (int p = yptr[q]; p < yptr[q + 1]; ++p) {
      const int r = yroot[p];
      const int c = root_case[r], lam = root_lam[r];
      const int it = case_iterm[c], ne = case_nelem[c];
      const double* rr = rep + (size_t)d * Ntot + (size_t)lam * degen * Ntot;
      for (int j = 0; j < ne; ++j) acc = fma(vs[it + j], rr[it + j], acc);
    }
  }
  Y[((size_t)col * nslot + slot) * Kp + v] = acc;
}

cudaError_t launch_build_y(const double* vecs, int ld, const int32_t* ivec, int nI, int ndeg,
                           const Basis& b, int gamma, int degen, int N, int Kp, double* Y,
                           cudaStream_t s, int d0) {
  if (nI == 0) return cudaSuccess;
  dim3 grid((b.nslot * Kp + 255) / 256, nI * ndeg);
  // d0: the first degenerate component (ndeg = 1, d0 = d: component d alone)
  k_build_y<<<grid, 256, 0, s>>>(vecs, ld, ivec, ndeg, b.d_yptr.p, b.d_yroot.p, b.d_root_case.p,
                                 b.d_root_lam.p, b.d_case_iterm[gamma].p,
                                 b.d_case_nelem[gamma].p,
                                 b.d_rep[gamma].p + (size_t)d0 * b.Ntotal[gamma], b.Ntotal[gamma],
                                 degen, b.nslot, N, Kp, Y);
  return cudaGetLastError();
}

// The CSR of k_build_y flattened: one thread per (slot, v), its (symmetrised
// function, coefficients) entries in the same order, zero coefficients left out.
__global__ void k_y_table(const int32_t* __restrict__ yptr, const int32_t* __restrict__ yroot,
                          const int32_t* __restrict__ root_case,
                          const int32_t* __restrict__ root_lam,
                          const int32_t* __restrict__ case_iterm,
                          const int32_t* __restrict__ case_nelem, const double* __restrict__ rep,
                          int Ntot, int degen, long long nsv, int E, int32_t* __restrict__ ys,
                          double* __restrict__ yc) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= nsv) return;
  int n = 0;
  for (int p = yptr[q]; p < yptr[q + 1]; ++p) {
    const int r = yroot[p];
    const int c = root_case[r], lam = root_lam[r];
    for (int j = 0; j < case_nelem[c]; ++j) {
      const int s = case_iterm[c] + j;
      bool any = false;
      for (int d = 0; d < degen; ++d)
        any = any || rep[s + (size_t)d * Ntot + (size_t)lam * degen * Ntot] != 0.0;
      if (!any || n == E) continue;
      ys[n * nsv + q] = s;
      for (int d = 0; d < degen; ++d)
        yc[((long long)d * E + n) * nsv + q] =
            rep[s + (size_t)d * Ntot + (size_t)lam * degen * Ntot];
      ++n;
    }
  }
  for (; n < E; ++n) {
    ys[n * nsv + q] = 0;
    for (int d = 0; d < degen; ++d) yc[((long long)d * E + n) * nsv + q] = 0.0;
  }
}

struct RootMaskArgs {
  const int32_t *iterm[GI_MAX_REP], *nelem[GI_MAX_REP];
  const double* rep[GI_MAX_REP];
  int ntot[GI_MAX_REP], degen[GI_MAX_REP], nrep;
};
__global__ void k_root_masks(const __grid_constant__ RootMaskArgs a,
                             const int32_t* __restrict__ root_case,
                             const int32_t* __restrict__ root_lam, int D,
                             uint8_t* __restrict__ mask, int32_t* __restrict__ ent) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= D) return;
  const int c = root_case[r], lam = root_lam[r];
  unsigned m = 0;
  for (int g = 0; g < a.nrep; ++g) {
    const double* rr = a.rep[g] + a.iterm[g][c] + (size_t)lam * a.degen[g] * a.ntot[g];
    int n = 0;
    for (int j = 0; j < a.nelem[g][c]; ++j) {
      bool any = false;
      for (int d = 0; d < a.degen[g]; ++d) any = any || rr[j + (size_t)d * a.ntot[g]] != 0.0;
      n += any;
    }
    if (n) m |= 1u << g;
    if (n > ent[g]) atomicMax(ent + g, n);
  }
  mask[r] = (uint8_t)m;
}
cudaError_t launch_root_masks(const Basis& b, const std::vector<int32_t>& degen, uint8_t* mask,
                              int32_t* ent, cudaStream_t s) {
  RootMaskArgs a{};
  a.nrep = (int)degen.size();
  for (int g = 0; g < a.nrep; ++g) {
    a.iterm[g] = b.d_case_iterm[g].p;
    a.nelem[g] = b.d_case_nelem[g].p;
    a.rep[g] = b.d_rep[g].p;
    a.ntot[g] = b.Ntotal[g];
    a.degen[g] = degen[g];
  }
  k_root_masks<<<(b.D + 255) / 256, 256, 0, s>>>(a, b.d_root_case.p, b.d_root_lam.p, b.D, mask,
                                                 ent);
  return cudaGetLastError();
}

__global__ void k_root_z(const int32_t* __restrict__ root_v, const int32_t* __restrict__ zpos, int D,
                         int32_t* __restrict__ out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < D) out[r] = zpos[root_v[r]];
}
cudaError_t launch_root_z(const Basis& b, const int32_t* zpos, int32_t* out, cudaStream_t s) {
  k_root_z<<<(b.D + 255) / 256, 256, 0, s>>>(b.d_root_v.p, zpos, b.D, out);
  return cudaGetLastError();
}

cudaError_t launch_y_table(const Basis& b, int gamma, int degen, int N, int E, int32_t* ys,
                           double* yc, cudaStream_t s) {
  const long long nsv = (long long)b.nslot * N;
  if (nsv == 0 || E == 0) return cudaSuccess;
  k_y_table<<<(unsigned)((nsv + 255) / 256), 256, 0, s>>>(
      b.d_yptr.p, b.d_yroot.p, b.d_root_case.p, b.d_root_lam.p, b.d_case_iterm[gamma].p,
      b.d_case_nelem[gamma].p, b.d_rep[gamma].p, b.Ntotal[gamma], degen, nsv, E, ys, yc);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ H build
// One thread per symmetrised final function s of one initial column (i, dI);
// writes H for every final degenerate component dF.
template <int NDEGF>
__device__ __forceinline__ void build_h_col(
    const double* __restrict__ Z, size_t zc, int ldz, int nslotI, int colI,
    const int32_t* __restrict__ s_case, const int32_t* __restrict__ case_ptr,
    const int32_t* __restrict__ case_roots, const int32_t* __restrict__ root_v,
    const int32_t* __restrict__ root_key, const int32_t* __restrict__ root_lam,
    const double* __restrict__ rep, int Ntot, const StencilTerm* __restrict__ st,
    const int32_t* __restrict__ st_n, int st_max, int nsizeF, int ldh, int s,
    double* __restrict__ H, const int32_t* __restrict__ slotcol) {
  double acc[NDEGF];
#pragma unroll
  for (int d = 0; d < NDEGF; ++d) acc[d] = 0.0;
  if (s < nsizeF) {
    const double* zcol = Z + (size_t)colI * (slotcol ? 1 : nslotI) * ldz;
    const int cs = s_case[s];
    for (int p = case_ptr[cs]; p < case_ptr[cs + 1]; ++p) {
      const int r = case_roots[p];
      const int v = root_v[r], key = root_key[r], lam = root_lam[r];
      // a root the symmetrised function has no part in is passed over: its
      // rows of Z may not have been computed
      double w[NDEGF];
      bool any = false;
#pragma unroll
      for (int d = 0; d < NDEGF; ++d) {
        w[d] = rep[s + (size_t)d * Ntot + (size_t)lam * NDEGF * Ntot];
        any = any || w[d] != 0.0;
      }
      if (!any) continue;
      double h = 0.0;
      const int nt = st_n[key];
      for (int t = 0; t < nt; ++t) {
        const StencilTerm term = st[key * st_max + t];
        const size_t col = slotcol ? slotcol[term.slotI] : term.slotI;
        h = fma(term.coef, zcol[(size_t)term.c * zc + col * ldz + v], h);
      }
#pragma unroll
      for (int d = 0; d < NDEGF; ++d) acc[d] = fma(w[d], h, acc[d]);
    }
  }
#pragma unroll
  for (int d = 0; d < NDEGF; ++d) H[((size_t)colI * NDEGF + d) * ldh + s] = acc[d];
}

template <int NDEGF>
__global__ void k_build_h(const double* __restrict__ Z, size_t zc, int ldz, int nslotI, int ndegI,
                          const int32_t* __restrict__ s_case, const int32_t* __restrict__ case_ptr,
                          const int32_t* __restrict__ case_roots,
                          const int32_t* __restrict__ root_v, const int32_t* __restrict__ root_key,
                          const int32_t* __restrict__ root_lam, const double* __restrict__ rep,
                          int Ntot, const StencilTerm* __restrict__ st,
                          const int32_t* __restrict__ st_n, int st_max, int nsizeF, int ldh,
                          double* __restrict__ H, const int32_t* __restrict__ slotcol) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const int colI = blockIdx.y;  // i * ndegI + dI
  if (s >= ldh) return;
  build_h_col<NDEGF>(Z, zc, ldz, nslotI, colI, s_case, case_ptr, case_roots, root_v, root_key,
                     root_lam, rep, Ntot, st, st_n, st_max, nsizeF, ldh, s, H, slotcol);
}

// Every H build of a group of final blocks in one launch: item k covers
// blocks [items[k].blk0, items[k].blk0 + items[k].nblk) of the 1-D grid, each
// block 256 functions s of kHCols initial columns (the item lookup is paid
// once per kHCols columns).
__global__ void __launch_bounds__(256) k_build_h_items(const HItem* __restrict__ items,
                                                        const long long* __restrict__ firsts,
                                                        int nitems) {
  const long long b = blockIdx.x;
  const int lo = find_item(nitems, b, [&](int k) { return firsts[k]; });
  const HItem& it = items[lo];
  const long long rel = b - it.blk0;
  const int nsb = (it.ldh + 255) >> 8;
  const int cb = (int)(rel / nsb);
  const int s = (int)(rel - (long long)cb * nsb) * 256 + threadIdx.x;
  if (s >= it.ldh) return;
  const int c1 = min(it.ncol, (cb + 1) * kHCols);
  for (int colI = cb * kHCols; colI < c1; ++colI) {
    if (it.ndegF == 2)
      build_h_col<2>(it.Z, it.zc, it.ldz, it.nslotI, colI, it.s_case, it.case_ptr, it.case_roots,
                     it.root_v, it.root_key, it.root_lam, it.rep, it.Ntot, it.st, it.st_n,
                     it.st_max, it.nsizeF, it.ldh, s, it.H, it.slotcol);
    else
      build_h_col<1>(it.Z, it.zc, it.ldz, it.nslotI, colI, it.s_case, it.case_ptr, it.case_roots,
                     it.root_v, it.root_key, it.root_lam, it.rep, it.Ntot, it.st, it.st_n,
                     it.st_max, it.nsizeF, it.ldh, s, it.H, it.slotcol);
  }
}

cudaError_t launch_build_h_items(const HItem* items, const long long* firsts, int nitems,
                                 long long nblocks, cudaStream_t st) {
  if (nitems <= 0 || nblocks <= 0) return cudaSuccess;
  if (nblocks > 0x7FFFFFFFll) return cudaErrorInvalidValue;
  k_build_h_items<<<(unsigned)nblocks, 256, 0, st>>>(items, firsts, nitems);
  return cudaGetLastError();
}

// The item of an H build (one per (initial unit, final block) of a group).
HItem make_h_item(const double* Z, size_t zstride_c, int ldz, int nslotI, int ndegI, int nI,
                  const Basis& bF, int gammaF, int degF, int nsizeF, int ldh,
                  const StencilTerm* st, const int32_t* st_n, int st_max, double* H,
                  long long blk0) {
  HItem it{};
  it.Z = Z;
  it.zc = zstride_c;
  it.ldz = ldz;
  it.nslotI = nslotI;
  it.ndegF = degF;
  it.nsizeF = nsizeF;
  it.ldh = ldh;
  it.Ntot = bF.Ntotal[gammaF];
  it.st_max = st_max;
  it.s_case = bF.d_s_case[gammaF].p;
  it.case_ptr = bF.d_case_ptr.p;
  it.case_roots = bF.d_case_roots.p;
  it.root_v = bF.d_root_v.p;
  it.root_key = bF.d_root_key.p;
  it.root_lam = bF.d_root_lam.p;
  it.rep = bF.d_rep[gammaF].p;
  it.st = st;
  it.st_n = st_n;
  it.H = H;
  it.blk0 = blk0;
  it.ncol = nI * ndegI;
  it.nblk = (long long)((it.ncol + kHCols - 1) / kHCols) * ((ldh + 255) / 256);
  return it;
}

cudaError_t launch_build_h(const double* Z, size_t zstride_c, int ldz, int nslotI, int ndegI,
                           int nI, const Basis& bF, int gammaF, int degF, int nsizeF, int ldh,
                           const StencilTerm* st, const int32_t* st_n, int st_max, double* H,
                           cudaStream_t s, const int32_t* root_z, const int32_t* slotcol) {
  if (nI == 0) return cudaSuccess;
  const int32_t* root_v = root_z ? root_z : bF.d_root_v.p;
  dim3 grid((ldh + 255) / 256, nI * ndegI);
  if (degF == 1)
    k_build_h<1><<<grid, 256, 0, s>>>(Z, zstride_c, ldz, nslotI, ndegI, bF.d_s_case[gammaF].p,
                                      bF.d_case_ptr.p, bF.d_case_roots.p, root_v,
                                      bF.d_root_key.p, bF.d_root_lam.p, bF.d_rep[gammaF].p,
                                      bF.Ntotal[gammaF], st, st_n, st_max, nsizeF, ldh, H,
                                      slotcol);
  else if (degF == 2)
    k_build_h<2><<<grid, 256, 0, s>>>(Z, zstride_c, ldz, nslotI, ndegI, bF.d_s_case[gammaF].p,
                                      bF.d_case_ptr.p, bF.d_case_roots.p, root_v,
                                      bF.d_root_key.p, bF.d_root_lam.p, bF.d_rep[gammaF].p,
                                      bF.Ntotal[gammaF], st, st_n, st_max, nsizeF, ldh, H,
                                      slotcol);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

// Primitive-space half line strength of one column (the reference's half_ls
// buffer, dipole_kernals.cu:223-224).
__global__ void k_half_ls_prim(const double* __restrict__ Z, size_t zc, int ldz,
                               const int32_t* __restrict__ root_v,
                               const int32_t* __restrict__ root_key,
                               const StencilTerm* __restrict__ st, const int32_t* __restrict__ st_n,
                               int st_max, int D, double* __restrict__ h) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= D) return;
  const int v = root_v[r], key = root_key[r];
  double acc = 0.0;
  for (int t = 0; t < st_n[key]; ++t) {
    const StencilTerm term = st[key * st_max + t];
    acc = fma(term.coef, Z[(size_t)term.c * zc + (size_t)term.slotI * ldz + v], acc);
  }
  h[r] = acc;
}

cudaError_t launch_half_ls_prim(const double* Z, size_t zstride_c, int ldz, const Basis& bF,
                                const StencilTerm* st, const int32_t* st_n, int st_max,
                                double* h, cudaStream_t s) {
  k_half_ls_prim<<<(bF.D + 255) / 256, 256, 0, s>>>(Z, zstride_c, ldz, bF.d_root_v.p,
                                                    bF.d_root_key.p, st, st_n, st_max, bF.D, h);
  return cudaGetLastError();
}

// The same from a Z split into K parts (the narrow split-precision GEMM):
// Z_c[col][v] = sum_p Zp[p][col][c * cstride + v], col = colbase + slot.
__global__ void k_half_ls_prim_parts(const double* __restrict__ Zp, int nparts, size_t pstride,
                                     int ldz, int cstride, const int32_t* __restrict__ root_v,
                                     const int32_t* __restrict__ root_key,
                                     const StencilTerm* __restrict__ st,
                                     const int32_t* __restrict__ st_n, int st_max, int D,
                                     double* __restrict__ h,
                                     const int32_t* __restrict__ slotcol) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= D) return;
  const int v = root_v[r], key = root_key[r];
  double acc = 0.0;
  for (int t = 0; t < st_n[key]; ++t) {
    const StencilTerm term = st[key * st_max + t];
    const int col = slotcol ? slotcol[term.slotI] : term.slotI;
    const double* z = Zp + (size_t)col * ldz + (size_t)term.c * cstride + v;
    double zs = z[0];
    for (int p = 1; p < nparts; ++p) zs += z[(size_t)p * pstride];
    acc = fma(term.coef, zs, acc);
  }
  h[r] = acc;
}

cudaError_t launch_half_ls_prim_parts(const double* Zp, int nparts, size_t pstride, int ldz,
                                      int cstride, const Basis& bF, const StencilTerm* st,
                                      const int32_t* st_n, int st_max, double* h,
                                      cudaStream_t s, const int32_t* root_z,
                                      const int32_t* slotcol) {
  k_half_ls_prim_parts<<<(bF.D + 255) / 256, 256, 0, s>>>(
      Zp, nparts, pstride, ldz, cstride, root_z ? root_z : bF.d_root_v.p, bF.d_root_key.p, st, st_n,
      st_max, bF.D, h, slotcol);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ epilogue
// One thread per (initial level i, final level f) of a part: the per-line
// epilogue of epilogue.cuh on the moments of T.
__device__ __forceinline__ void epilogue_block(
    int fb, int i, const double* __restrict__ T, int ldt, int nF,
    const int32_t* __restrict__ levelI, const double* __restrict__ EI,
    const int32_t* __restrict__ levelF, const double* __restrict__ EF,
    const uint8_t* __restrict__ upper_ok, const double* __restrict__ hn, const EpiParams& p,
    gi_line* __restrict__ out, unsigned long long* counter, long long cap,
    RefineRec* __restrict__ rec, long long rec_cap) {
  const int f = fb * 128 + threadIdx.x;
  // the initial level's Boltzmann factor, once per block (FP64 exp is scarce)
  __shared__ double boltz_i;
  if (threadIdx.x == 0) boltz_i = exp(-(EI[i] - p.zpe) * p.beta);
  __syncthreads();
  double t[4] = {0.0, 0.0, 0.0, 0.0}, hnq[4] = {0.0, 0.0, 0.0, 0.0};
  const bool ok_f = f < nF && upper_ok[f];
  if (ok_f)
    for (int dF = 0; dF < p.ndegF; ++dF)
      for (int dI = 0; dI < p.ndegI; ++dI)
        if (p.combo_mask & (1 << (dI + 2 * dF))) {
          const int col = (i * p.ndegI + dI) * p.ndegF + dF;
          t[dI + 2 * dF] = T[(size_t)col * ldt + f];
          hnq[dI + 2 * dF] = hn[col];
        }
  LineEval r;
  eval_line(p, t, hnq, EI[i], ok_f ? EF[f] : 0.0, boltz_i, ok_f, levelI[i],
            ok_f ? levelF[f] : -1, r);
  append_line(r, p.part, i, f, out, counter, cap, rec, rec_cap);
}

__global__ void __launch_bounds__(128)
    k_epilogue(const double* __restrict__ T, int ldt, int nF, const int32_t* __restrict__ levelI,
               const double* __restrict__ EI, const int32_t* __restrict__ levelF,
               const double* __restrict__ EF, const uint8_t* __restrict__ upper_ok,
               const double* __restrict__ hn, EpiParams p, gi_line* __restrict__ out,
               unsigned long long* counter, long long cap, RefineRec* __restrict__ rec,
               long long rec_cap) {
  epilogue_block(blockIdx.x, blockIdx.y, T, ldt, nF, levelI, EI, levelF, EF, upper_ok, hn, p, out,
                 counter, cap, rec, rec_cap);
}
// Every part of a group of final blocks in one launch.
__global__ void __launch_bounds__(128)
    k_epilogue_items(const EpiItem* __restrict__ items, int nitems, gi_line* __restrict__ out,
                     unsigned long long* counter, long long cap, RefineRec* __restrict__ rec,
                     long long rec_cap) {
  const long long b = blockIdx.x;
  const EpiItem& it = items[find_item(nitems, b, [&](int k) { return items[k].blk0; })];
  const int nfb = (it.nF + 127) >> 7, rel = (int)(b - it.blk0);
  epilogue_block(rel % nfb, rel / nfb, it.T, it.ldt, it.nF, it.lvI, it.EI, it.lvF, it.EF, it.upper,
                 it.hn, it.ep, out, counter, cap, rec, rec_cap);
}
cudaError_t launch_epilogue_items(const EpiItem* items, int nitems, long long blocks, gi_line* out,
                                  unsigned long long* counter, long long cap, RefineRec* rec,
                                  long long rec_cap, cudaStream_t s) {
  if (nitems <= 0 || blocks <= 0) return cudaSuccess;
  if (blocks > 0x7FFFFFFFll) return cudaErrorInvalidValue;
  k_epilogue_items<<<(unsigned)blocks, 128, 0, s>>>(items, nitems, out, counter, cap, rec, rec_cap);
  return cudaGetLastError();
}

__global__ void k_boltz(const double* __restrict__ E, int n, double zpe, double beta,
                        double* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) out[k] = exp(-(E[k] - zpe) * beta);
}

// Full line records -> compact ones (the read-back of GI_RUN_COMPACT_LINES).
__global__ void k_pack_lines(const gi_line* __restrict__ in, gi_line_compact* __restrict__ out,
                             long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const gi_line& L = in[i];
    gi_line_compact o;
    o.level_i = L.level_i;
    o.level_f = L.level_f;
    o.nu = L.nu;
    o.S = L.S;
    o.A = L.A;
    o.I = L.I;
    out[i] = o;
  }
}

cudaError_t launch_pack_lines(const gi_line* in, gi_line_compact* out, long long n,
                              cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const long long blocks = std::min<long long>((n + 255) / 256, 152 * 16);
  k_pack_lines<<<(unsigned)blocks, 256, 0, st>>>(in, out, n);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ line order
// Lines ordered by (level_i, level_f).  A pair of levels has at most one line,
// so within one initial level a line's place is the number of smaller final
// levels present: counted directly for short lists, else from a bitmap of the
// final levels.  Three passes over 4-8 B per line and one over the records:
// bound by the records' 80 B read and written.
__global__ void k_sort_count(const gi_line* __restrict__ in, long long n, int32_t* __restrict__ cnt) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x)
    atomicAdd(cnt + in[k].level_i, 1);
}
// first[i] = lines of levels below i (first[nlev] = all), cur = a copy (over cnt).
__global__ void __launch_bounds__(1024) k_sort_scan(int32_t* __restrict__ cur,
                                                    int32_t* __restrict__ first, int nlev) {
  __shared__ int part[1024];
  const int per = (nlev + 1023) / 1024, a = threadIdx.x * per, b = min(a + per, nlev);
  int s = 0;
  for (int i = a; i < b; ++i) s += cur[i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const int v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  s = threadIdx.x ? part[threadIdx.x - 1] : 0;
  for (int i = a; i < b; ++i) {
    const int c = cur[i];
    first[i] = s;
    cur[i] = s;
    s += c;
  }
  if (threadIdx.x == 1023) first[nlev] = part[1023];
}
__global__ void k_sort_deal(const gi_line* __restrict__ in, long long n, int32_t* __restrict__ cur,
                            int2* __restrict__ lst) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x) {
    const int2 l = *reinterpret_cast<const int2*>(in + k);  // level_i, level_f
    lst[atomicAdd(cur + l.x, 1)] = make_int2(l.y, (int)k);
  }
}
constexpr int kSortDirect = 512;
__global__ void __launch_bounds__(256) k_sort_place(const gi_line* __restrict__ in,
                                                    const int2* __restrict__ lst,
                                                    const int32_t* __restrict__ first, int nlev,
                                                    gi_line* __restrict__ out) {
  extern __shared__ unsigned sm[];  // bitmap of the final levels, then its prefix counts
  const int f0 = first[blockIdx.x], n = first[blockIdx.x + 1] - f0;
  if (n == 0) return;
  auto copy = [&](int k, int rank) {
    const uint4* src = reinterpret_cast<const uint4*>(in + lst[f0 + k].y);
    uint4* dst = reinterpret_cast<uint4*>(out + f0 + rank);
#pragma unroll
    for (int q = 0; q < 5; ++q) dst[q] = src[q];
  };
  static_assert(sizeof(gi_line) == 80, "five 16-byte words");
  if (n <= kSortDirect) {
    for (int k = threadIdx.x; k < n; k += 256) sm[k] = (unsigned)lst[f0 + k].x;
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += 256) {
      const unsigned f = sm[k];
      int rank = 0;
      for (int j = 0; j < n; ++j) rank += sm[j] < f;
      copy(k, rank);
    }
    return;
  }
  const int nw = (nlev + 31) >> 5;
  unsigned* pre = sm + nw;
  for (int w = threadIdx.x; w < nw; w += 256) sm[w] = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += 256) {
    const int f = lst[f0 + k].x;
    atomicOr(sm + (f >> 5), 1u << (f & 31));
  }
  __syncthreads();
  __shared__ unsigned part[256];
  const int per = (nw + 255) / 256, a = min((int)threadIdx.x * per, nw), b = min(a + per, nw);
  unsigned s = 0;
  for (int w = a; w < b; ++w) s += __popc(sm[w]);
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {
    const unsigned v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  s = threadIdx.x ? part[threadIdx.x - 1] : 0;
  for (int w = a; w < b; ++w) {
    pre[w] = s;
    s += __popc(sm[w]);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += 256) {
    const int f = lst[f0 + k].x;
    copy(k, (int)(pre[f >> 5] + __popc(sm[f >> 5] & ((1u << (f & 31)) - 1u))));
  }
}

cudaError_t launch_sort_lines(const gi_line* in, gi_line* out, long long n, int nlev, int32_t* ws,
                              cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (nlev <= 0 || nlev > kSortMaxLevels || n > 0x7FFFFFFFll) return cudaErrorInvalidValue;
  const size_t sm = std::max<size_t>(8 * (size_t)((nlev + 31) / 32), 4 * kSortDirect);
  cudaError_t e = cudaSuccess;
  if (sm > 48 * 1024)
    e = cudaFuncSetAttribute(k_sort_place, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  // lists first: 8-byte aligned; then the cursors and the offsets
  int2* lst = reinterpret_cast<int2*>(ws);
  int32_t* cur = ws + 2 * n;
  int32_t* first = cur + nlev;
  if (e == cudaSuccess) e = cudaMemsetAsync(cur, 0, sizeof(int32_t) * nlev, st);
  if (e != cudaSuccess) return e;
  const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 152 * 16);
  k_sort_count<<<blocks, 256, 0, st>>>(in, n, cur);
  k_sort_scan<<<1, 1024, 0, st>>>(cur, first, nlev);
  k_sort_deal<<<blocks, 256, 0, st>>>(in, n, cur, lst);
  k_sort_place<<<nlev, 256, sm, st>>>(in, lst, first, nlev, out);
  return cudaGetLastError();
}

cudaError_t launch_boltz(const double* E, int n, double zpe, double beta, double* out,
                         cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_boltz<<<(n + 255) / 256, 256, 0, s>>>(E, n, zpe, beta, out);
  return cudaGetLastError();
}

// Euclidean norm of each H column (the scale of its transition moments' error).
__global__ void k_col_norms(const double* __restrict__ H, int ldh, int n, double* __restrict__ out) {
  const double* h = H + (size_t)blockIdx.x * ldh;
  double acc = 0.0;
  for (int s = threadIdx.x; s < n; s += blockDim.x) acc = fma(h[s], h[s], acc);
  __shared__ double part[32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    acc = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (threadIdx.x == 0) out[blockIdx.x] = sqrt(acc);
  }
}

// The columns of every H of a group in one launch (item k: columns
// [items[k].col0, items[k+1].col0) of the grid).
__global__ void k_col_norms_items(const NormItem* __restrict__ items, int nitems) {
  const long long b = blockIdx.x;
  const int lo = find_item(nitems, b, [&](int k) { return items[k].col0; });
  const NormItem& it = items[lo];
  const double* h = it.H + (size_t)(b - it.col0) * it.ldh;
  double acc = 0.0;
  for (int s = threadIdx.x; s < it.n; s += blockDim.x) acc = fma(h[s], h[s], acc);
  __shared__ double part[32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    acc = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (threadIdx.x == 0) it.out[b - it.col0] = sqrt(acc);
  }
}

cudaError_t launch_col_norms_items(const NormItem* items, int nitems, long long ncol,
                                   cudaStream_t s) {
  if (nitems <= 0 || ncol <= 0) return cudaSuccess;
  if (ncol > 0x7FFFFFFFll) return cudaErrorInvalidValue;
  k_col_norms_items<<<(unsigned)ncol, 256, 0, s>>>(items, nitems);
  return cudaGetLastError();
}

cudaError_t launch_col_norms(const double* H, int ldh, int n, int ncol, double* out,
                             cudaStream_t s) {
  if (ncol <= 0) return cudaSuccess;
  k_col_norms<<<ncol, 256, 0, s>>>(H, ldh, n, out);
  return cudaGetLastError();
}

cudaError_t launch_epilogue(const double* T, int ldt, int nI, int nF, const int32_t* levelI,
                            const double* EI, const int32_t* levelF, const double* EF,
                            const uint8_t* upper_ok, const double* hn, const EpiParams& p,
                            gi_line* out, unsigned long long* counter, long long cap,
                            RefineRec* rec, long long rec_cap, cudaStream_t s) {
  if (nI == 0 || nF == 0) return cudaSuccess;
  dim3 grid((nF + 127) / 128, nI);
  k_epilogue<<<grid, 128, 0, s>>>(T, ldt, nF, levelI, EI, levelF, EF, upper_ok, hn, p, out, counter,
                                  cap, rec, rec_cap);
  return cudaGetLastError();
}

}  // namespace gi
