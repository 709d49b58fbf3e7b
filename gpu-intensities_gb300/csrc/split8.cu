// Split-precision GEMMs on the fp8 tensor pipe (sm_103a): the default scheme.
//
// C[n*ldc + m] = sum_k A[m][k] B[n][k] in FP64 accuracy from e4m3 products.
// Each row is scaled by its own power of two so |x| < 1/2 and cut into eleven
// balanced base-32 digits,
//   x = sum_p a_p 2^(-5(p+1)) + tail,  a_p in [-16, 16],  |tail| <= 2^-56,
// every digit an exact e4m3 integer.  Products a_p b_q with p + q = d <= 10
// share the weight 2^(-5d) and one fp32 accumulator, which stays an exact
// integer while it is at most 2^24: a product is at most 2^8 and diagonal d
// has d + 1 of them per k, so every diagonal is exact for any operands up to
// K = 5952 (11 * 5952 * 2^8 < 2^24; the tensor pipe's fp32 sums of e4m3
// products were checked bit for bit up to there).  Longer K runs in segments
// whose FP64 results are added.
//
// Why e4m3: 66 digit products of the fp8 pipe replace 45 of the bf16 pipe
// (nine base-64 digits) at twice the rate, and an element is 11 bytes instead
// of 18, everywhere it is stored or moved.
//
// Why stacked: an MMA costs max(N/2, 32 + N/4) cycles for M = 128 (measured,
// N = 32..256: below N = 128 it waits for its operands, 128 B/clk of shared
// memory).  The digit planes of B lie one after the other in shared memory
// (40 rows each), and so do the accumulators of the diagonals in tensor
// memory, so plane p of A times planes 0..10-p of B is ONE product of width
// 40 (11 - p) onto diagonals p..10: 16 MMAs of up to 224 columns per K slice,
// 1376 cycles against 66 x 42 for one MMA per digit pair.
//
// Why blocked operands: the cuts write the digits where the MMA's
// shared-memory image wants them (32-byte rows, 32-byte swizzle), one K slice
// of a tile contiguous in memory, so a stage is two bulk copies (45,056 and
// 14,080 bytes) with no tensor maps.
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "epilogue.cuh"
#include "items.cuh"
#include "once.h"
#include "split8.h"
#include "tc.cuh"

namespace gi {
namespace {

constexpr int kS = kDigits8, kW = 5, kBN = kCols8, kBM = 128;
constexpr uint32_t kAP = kBM * 32, kBP = kBN * 32;  // bytes of a plane's K slice
constexpr uint32_t kAS = kS * kAP, kBS = kS * kBP, kStage = kAS + kBS;
constexpr int kST = 3;            // stages
constexpr int kSegSlices = 186;   // K = 5952 per exact segment
constexpr int kHi = 6;            // diagonals 0..5 in the high word of an exact sum
// Planes summed over a segment's slices up to which its sums stay within 2^22: a slice of
// np planes adds np products per k to diagonal 10, fewer to the others.
constexpr int kSmallPlanes = (1 << 22) / (32 * 256);
constexpr int kAhead = 8;         // B slices fetched into L2 ahead of their copies
constexpr int kRing = 4;          // work items in flight between the roles
constexpr int kThreads = 320;     // warp 0 copies, warp 1 MMA, warps 2..9 epilogue
// the earlier segments' sums of a tile, or its moments (20 per epilogue thread), after the
// stages (256 bytes the junk columns read) and the barriers
constexpr size_t kSumOff = (size_t)kST * kStage + 256 + 512;
constexpr size_t kListOff = kSumOff + sizeof(double) * 20 * 256;  // 640 lines per warp
constexpr size_t kSmem = kListOff + sizeof(uint16_t) * 640 * 8 + 1024;
static_assert(kSmem <= 227 * 1024, "shared memory");
static_assert(kStage % 256 == 0 && kAS % 256 == 0, "swizzle periods");
static_assert((size_t)kS * kSegSlices * 32 * 256 <= (1u << 24), "exact diagonal sums");
static_assert(kS * kBN + 8 <= 512, "tensor memory columns");

struct Params8 {
  Prob8 p[kMaxProb8];
  int nprob, nitems, fused;
  int* ctr;  // [0] next item, [1] finished CTAs; both back to 0 at the end
  gi_line* out;
  unsigned long long* counter;
  long long cap;
  RefineRec* rec;
  long long rec_cap;
};
static_assert(sizeof(Params8) <= 32764, "kernel parameter limit");

__device__ __forceinline__ void mma_e4m3(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
// kind::f8f6f4, e4m3 x e4m3 -> f32, K-major, M = 128.
__host__ __device__ constexpr uint32_t idesc_e4m3(int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::
          "r"(sptr(dst)),
      "l"(src), "r"(bytes), "r"(sptr(bar))
      : "memory");
}
// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void prefetch_l2(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(sptr(b)) : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

// Plane p = 11 - J of A of one K slice (a0, b0: shared-memory addresses / 16 of
// its A and B) with planes 0..J-1 of B: a window of 40 J columns, rounded up to
// a multiple of 16 (the extra 8 fall on columns 440..447, which nothing reads).
// Windows past 256 columns take two MMAs.
template <int J>
__device__ __forceinline__ void mma_window(uint32_t tmem, uint32_t a0, uint32_t b0, uint32_t acc) {
  constexpr int N = (kBN * J + 15) / 16 * 16;
  constexpr int N1 = N > 256 ? (N / 2 + 15) / 16 * 16 : N;
  // sdesc_sw32 without the address: 32-byte rows, 8-row groups 256 bytes apart
  constexpr uint64_t kDesc = (uint64_t)1 << 16 | (uint64_t)(256 >> 4) << 32 | (uint64_t)1 << 46 |
                             (uint64_t)6 << 61;
  const uint32_t d = tmem + (uint32_t)(kS - J) * kBN;
  const uint64_t a = kDesc | (a0 + (uint32_t)((kS - J) * kAP >> 4));
  mma_e4m3(d, a, kDesc | b0, idesc_e4m3(N1), acc);
  if constexpr (N > 256)
    mma_e4m3(d + N1, a, kDesc | (b0 + (uint32_t)(N1 * 32 >> 4)), idesc_e4m3(N - N1), acc);
}

// The exact sums of 20 columns, hi = diagonals 0..5 and lo = 6..10 (below 2^53
// each).  The tensor memory is held meanwhile, 20 x 11 conversions a thread at 8
// clocks a warp; a sum within 2^22 is instead read off the bits of itself plus
// 1.5 2^23, one addition (SMALL: the segments of up to about 46 slices, where
// this time is the larger part: 2200 clocks a tile instead of 4000; a C3v J = 20, 21
// batch at N = 3000 took 18.15 ms instead of 18.65, a C2v one at N = 2000 3.37 instead
// of 3.44).
template <bool SMALL>
__device__ __forceinline__ void fold_sums(uint32_t t0, long long* hi, long long* lo) {
  auto whole = [](uint32_t f) {
    const float x = __uint_as_float(f);
    return SMALL ? __float_as_int(x + 12582912.0f) - 0x4B400000 : __float2int_rn(x);
  };
#pragma unroll
  for (int ch = 0; ch < 5; ++ch) {
    uint32_t f[kS][4];
#pragma unroll
    for (int d = 0; d < kS; ++d) tmem_ld4(t0 + d * kBN + ch * 4, f[d]);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      // pairs of diagonals fit 32 bits (|sum| <= 2^24): 2^29 + 2^24
      auto pair = [&](int d) { return whole(f[d][j]) * 32 + whole(f[d + 1][j]); };
      hi[ch * 4 + j] = pair(0) * 1048576ll + (pair(2) * 1024ll + pair(4));
      lo[ch * 4 + j] = pair(6) * 32768ll + (pair(8) * 32ll + whole(f[10][j]));
    }
  }
}

// The lines of a warp's 20 columns of 32 final levels (m0.. + lane; sum: this
// thread's moments).  Groups of G = ndegI * ndegF consecutive columns are the
// moments of one initial level.  A line costs about a hundred FP64 instructions,
// 150,000 clocks a tile if every line took them, while most lines end below the
// threshold: those are told by line_below; the rest are listed (moments and
// list in shared memory) and evaluated with full warps.
template <int G>
__device__ __forceinline__ void lines_of(const Params8& P, const Prob8& pr, int n0, int m0,
                                         int lane, int rows_left, const double* sum, double* mom,
                                         uint16_t* lst) {
  constexpr int kGroups = 20 / G;
  const int m = m0 + lane;
  const bool ok_f = lane < rows_left && pr.upper[m];
  const double ef = ok_f ? pr.EF[m] : 0.0;
#pragma unroll
  for (int j = 0; j < 20; ++j) mom[j * 256 + lane] = sum[j];
  auto part_of = [&](int n) {
    int q = 0;
    while (q + 1 < pr.nparts && pr.parts[q + 1].c0 <= n) ++q;
    return q;
  };
  int cnt = 0, npass = 0;
#pragma unroll
  for (int g = 0; g < kGroups; ++g) {
    const int n = n0 + g * G;
    if (n >= pr.Nc) break;  // the same for every lane
    const EpiPart& pt = pr.parts[part_of(n)];
    const int i = (n - pt.c0) / G;
    const double nu = ef - pt.EI[i];
    const bool pass = ok_f && nu >= pt.ep.fw0 && nu <= pt.ep.fw1;
    const bool live = pass && !line_below<G>(pt, sum + g * G, pt.hn + i * G, nu, pt.BI[i]);
    npass += __popc(__ballot_sync(0xffffffffu, pass));
    const unsigned mask = __ballot_sync(0xffffffffu, live);
    if (live) lst[cnt + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)(g * 32 + lane);
    cnt += __popc(mask);
  }
  if (npass && lane == 0) atomicAdd(P.counter + 1, (unsigned long long)npass);
  __syncwarp();
  for (int k0 = 0; k0 < cnt; k0 += 32) {
    const bool on = k0 + lane < cnt;
    const int code = on ? lst[k0 + lane] : 0;
    const int g = code >> 5, src = code & 31;
    const int n = n0 + g * G;
    const EpiPart& pt = pr.parts[part_of(n)];
    const EpiParams& ep = pt.ep;
    const int i = (n - pt.c0) / G, mm = m0 + src;
    double t[4] = {0.0, 0.0, 0.0, 0.0}, hnq[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int o = 0; o < G; ++o) {
      const int q = moment_of<G>(o, ep.ndegF);
      if (ep.combo_mask & (1 << q)) {
        t[q] = mom[(g * G + o) * 256 + src];
        hnq[q] = pt.hn[i * G + o];
      }
    }
    LineEval r;
    eval_line(ep, t, hnq, pt.EI[i], on ? pr.EF[mm] : 0.0, pt.BI[i], on, pt.lvI[i],
              on ? pr.lvF[mm] : -1, r);
    r.pass = false;  // counted above
    append_line(r, ep.part, i, mm, P.out, P.counter, P.cap, P.rec, P.rec_cap);
  }
  __syncwarp();
}

// One persistent CTA per SM; work items are 128 x 40 tiles of the launch's
// problems, dealt out by an atomic counter (tiles differ in K).  Bound: the
// tensor pipe; a tile's epilogue holds the tensor memory only while it folds
// the diagonals into exact integers, the conversion to FP64 and the stores (or
// the lines) overlap the next tile's MMAs.
__global__ void __launch_bounds__(kThreads, 1)
    k_split8(const __grid_constant__ Params8 P, int* err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)kST * kStage + 256);
  uint64_t* empty = full + kST;
  uint64_t* itemf = empty + kST;   // a work item has been published
  uint64_t* iteme = itemf + kRing; // ... and taken by every epilogue warp
  uint64_t* accf = iteme + kRing;  // a segment's sums are final
  uint64_t* tfree = accf + 1;      // ... and have been read
  uint64_t* drain = tfree + 1;
  int* items = reinterpret_cast<int*>(drain + 1);
  int* meta = items + kRing;       // per stage: bit 0 first, 1 last of a segment, 2 of a tile,
                                   // 3 quit, 4..7 planes np (windows up to np), 8 small sums
  int* seg_last = meta + kST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(seg_last + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kST; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&itemf[i], 1);
      mbar_init(&iteme[i], 8);
    }
    mbar_init(accf, 2);  // the MMAs' commit and the issuer's own arrival
    mbar_init(tfree, 8);
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(
                     sptr(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  // item -> problem, row tile, column tile (GA row tiles stay in L2 while the
  // column tiles stream past them)
  auto decode = [&](int item, int& pi, int& ai, int& ct) {
    pi = 0;
    while (pi + 1 < P.nprob && P.p[pi + 1].first <= item) ++pi;
    const Prob8& pr = P.p[pi];
    const int local = item - pr.first;
    const int grp = local / (pr.GA * pr.nB);
    const int r = local - grp * pr.GA * pr.nB;
    const int gsz = min(pr.GA, pr.nA - grp * pr.GA);
    ai = grp * pr.GA + r % gsz;
    ct = r / gsz;
  };

  if (warp == 0) {
    // scheduler and copies: the warp reads the slice lists, lane 0 copies
    int it = 0, ic = 0;
    bool ok = true;
    int item = lane == 0 ? atomicAdd(P.ctr, 1) : 0;
    item = __shfl_sync(0xffffffffu, item, 0);
    for (; ok; ++ic) {
      const int slot = ic % kRing;
      if (ic >= kRing)
        ok = __all_sync(0xffffffffu, mbar_wait(&iteme[slot], ((ic / kRing) - 1) & 1, abort_flag,
                                               err, 41));
      if (!ok) break;
      const bool quit = item >= P.nitems;
      if (lane == 0) {
        items[slot] = quit ? -1 : item;
        mbar_arrive(&itemf[slot]);
      }
      if (quit) break;
      int next = lane == 0 ? atomicAdd(P.ctr, 1) : 0;  // used after this tile's copies
      int pi, ai, ct;
      decode(item, pi, ai, ct);
      const Prob8& pr = P.p[pi];
      const int tile = pr.at ? pr.at[ai].tile : ai;
      const uint8_t* Ab = pr.A + (size_t)tile * pr.nkA * kAS;
      const uint8_t* Bb = pr.B + (size_t)ct * pr.nkB * kBS;
      const int32_t* za = pr.za ? pr.za + (size_t)tile * pr.nkA : nullptr;
      // the slices with a digit in A, and the first of those with the fewest zero
      // planes: it starts the sums (and must cover every diagonal)
      int total = pr.nk, kfirst = 0;
      if (za) {
        total = 0;
        unsigned best = ~0u;
        for (int base = 0; base < pr.nk; base += 32) {
          const int k = base + lane;
          const int z = k < pr.nk ? za[pr.kl ? pr.kl[k] : k] : kS;
          total += __popc(__ballot_sync(0xffffffffu, z < kS));
          best = min(best, ((unsigned)min(z, kS) << 24) | (unsigned)min(k, pr.nk - 1));
        }
        best = __reduce_min_sync(0xffffffffu, best);
        kfirst = (int)(best & 0xFFFFFFu);
        total = max(total, 1);  // nothing but zeros: one slice, which writes them
      }
      int done = 0, planes = 0;
      auto slice = [&](int k, int ks, int z) {  // (warp-uniform arguments)
        const int st = it % kST, in_seg = done % kSegSlices;
        const bool last = done + 1 == total;
        const uint32_t np = kS - (in_seg == 0 ? 0 : z);  // planes of A and of B
        planes = (in_seg == 0 ? 0 : planes) + (int)np;
        if (lane == 0) {
          if (it >= kST) ok = mbar_wait(&empty[st], ((it / kST) - 1) & 1, abort_flag, err, 42);
          if (ok) {
            unsigned char* sa = smem + (size_t)st * kStage;
            meta[st] = (in_seg == 0 ? 1 : 0) | ((last || in_seg == kSegSlices - 1) ? 2 : 0) |
                       (last ? 4 : 0) | (int)(np << 4) | (planes <= kSmallPlanes ? 256 : 0);
            mbar_expect_tx(&full[st], np * (kAP + kBP));
            bulk_load(sa + (kS - np) * kAP, Ab + (size_t)ks * kAS + (kS - np) * kAP, np * kAP,
                      &full[st]);
            bulk_load(sa + kAS, Bb + (size_t)k * kBS, np * kBP, &full[st]);
          }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) return;
        ++it;
        ++done;
        if (done == 2) {  // the next tile's first B slices on their way to L2
          const int nx = __shfl_sync(0xffffffffu, next, 0);
          if (nx < P.nitems) {
            int pj, aj, cj;
            decode(nx, pj, aj, cj);
            const Prob8& pn = P.p[pj];
            if (lane < min(kAhead, pn.nk))
              prefetch_l2(pn.B + ((size_t)cj * pn.nkB + lane) * kBS, kBS);
          }
        }
      };
      if (za) slice(kfirst, pr.kl ? pr.kl[kfirst] : kfirst, 0);
      for (int base = 0; base < pr.nk && ok; base += 32) {
        const int k = base + lane;
        const int ks = k < pr.nk ? (pr.kl ? pr.kl[k] : k) : 0;
        const int z = k < pr.nk ? (za ? za[ks] : 0) : kS;
        unsigned mask = __ballot_sync(0xffffffffu, z < kS && !(za && k == kfirst));
        // the B slices of this stretch: no tile in flight may have touched them
        if (mask >> lane & 1) prefetch_l2(Bb + (size_t)k * kBS, (kS - z) * kBP);
        while (mask && ok) {
          const int b = __ffs(mask) - 1;
          mask &= mask - 1;
          slice(base + b, __shfl_sync(0xffffffffu, ks, b), __shfl_sync(0xffffffffu, z, b));
        }
      }
      item = __shfl_sync(0xffffffffu, next, 0);
    }
    if (lane == 0) {
      if (ok) {  // the MMA issuer leaves on a stage without copies
        const int st = it % kST;
        if (it < kST || mbar_wait(&empty[st], ((it / kST) - 1) & 1, abort_flag, err, 43)) {
          meta[st] = 8;
          mbar_arrive(&full[st]);
        }
      }
      if (*abort_flag) {  // copies in flight land before the shared memory goes away
        for (int j = (it > kST ? it - kST : 0); j < it; ++j) {
          const uint64_t t0 = gtimer();
          while (!mbar_try(&full[j % kST], (j / kST) & 1) && gtimer() - t0 < 1000000000ull) {
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // MMA issuer.  About four MMAs queue behind the one running, so whatever
    // the issuer does between MMAs has to fit their time: the whole warp runs the
    // loop (its control and addresses stay in uniform registers) and one lane
    // issues; the wait for the next slice comes before the three widest of the
    // narrow windows.  1667 cycles a slice with one lane looping and the wait
    // between slices, 1522 this way (1376 of MMAs).
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t sbase = __shfl_sync(0xffffffffu, sptr(smem), 0);
    int st = 0, seg = 0;
    uint32_t parity = 0;
    bool ok = __all_sync(0xffffffffu, mbar_wait(&full[0], 0, abort_flag, err, 44));
    int mt = ok ? __shfl_sync(0xffffffffu, meta[0], 0) : 8;
    while (!(mt & 8)) {
      if ((mt & 1) && seg > 0) {  // the epilogue has read the previous segment
        if (!__all_sync(0xffffffffu, mbar_wait(tfree, (seg - 1) & 1, abort_flag, err, 45))) break;
      }
      if (mt & 1) asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t a0 = (sbase + (uint32_t)st * kStage) >> 4, b0 = a0 + (kAS >> 4);
      const int np = mt >> 4 & 15;  // planes 11 - np.. of A have digits
      auto finish = [&] {
        if (np >= 8) mma_window<8>(tm, a0, b0, 1u);
        if (np >= 9) mma_window<9>(tm, a0, b0, 1u);
        if (np >= 10) mma_window<10>(tm, a0, b0, 1u);
        mma_commit(&empty[st]);
        if (mt & 2) {
          *seg_last = mt;
          mma_commit(accf);
          mbar_arrive(accf);
        }
      };
      // A slice without the wide windows is given back before the wait (after it, two
      // slices instead of three are in flight), and so is the last of a segment,
      // whose sums the epilogue waits for: both GEMMs of a C3v N = 3000 batch 13.25 -> 12.96 ms,
      // of a C2v N = 5000 one without zero planes 3.84 -> 3.73 ms.
      const bool early = np < 8 || (mt & 2);
      if (elect_one()) {
        if (np == 11) mma_window<11>(tm, a0, b0, (mt & 1) ? 0u : 1u);
        mma_window<1>(tm, a0, b0, 1u);
        if (np >= 2) mma_window<2>(tm, a0, b0, 1u);
        if (np >= 3) mma_window<3>(tm, a0, b0, 1u);
        if (np >= 4) mma_window<4>(tm, a0, b0, 1u);
        if (np >= 5) mma_window<5>(tm, a0, b0, 1u);
        if (np >= 6) mma_window<6>(tm, a0, b0, 1u);
        if (np >= 7) mma_window<7>(tm, a0, b0, 1u);
        if (early) finish();
      }
      __syncwarp();
      const int nst = st + 1 == kST ? 0 : st + 1;
      if (nst == 0) parity ^= 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&full[nst], parity, abort_flag, err, 44));
      const int next = ok ? __shfl_sync(0xffffffffu, meta[nst], 0) : 8;
      if (!early && elect_one()) finish();
      __syncwarp();
      if (mt & 2) ++seg;
      st = nst;
      mt = next;
    }
    // every MMA issued has completed before the tensor memory is freed
    if (elect_one()) mma_commit(drain);
    const uint64_t t0 = gtimer();
    while (!mbar_try(drain, 0) && gtimer() - t0 < 1000000000ull) {
    }
    __syncwarp();
  } else {
    // warps 2..9: tensor-memory lane quadrant (warp % 4), 20 of the 40 columns
    const int q4 = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lanes = (uint32_t)(q4 * 32) << 16;
    const int r = q4 * 32 + lane;  // row within the tile
    double* prev = reinterpret_cast<double*>(smem + kSumOff) + (threadIdx.x - 64);
    int seg = 0;
    bool ok = true;
    for (int ic = 0; ok; ++ic) {
      const int slot = ic % kRing;
      ok = mbar_wait(&itemf[slot], (ic / kRing) & 1, abort_flag, err, 46, 64);
      if (!ok) break;
      const int item = items[slot];
      __syncwarp();
      if (lane == 0) mbar_arrive(&iteme[slot]);
      if (item < 0) break;
      int pi, ai, ct;
      decode(item, pi, ai, ct);
      const Prob8& pr = P.p[pi];
      ATile at;
      if (pr.at) {
        at = pr.at[ai];
      } else {
        at.tile = ai;
        at.rows = min(kBM, pr.M - ai * kBM);
        at.coff = (int64_t)ai * kBM;
      }
      const bool row_ok = r < at.rows;
      const int er = pr.ea[at.tile * kBM + r] - 2 * kW;
      const int n0 = ct * kBN + half * 20;
      double sum[20];
      for (bool last = false, first = true; !last; first = false, ++seg) {
        ok = mbar_wait(accf, seg & 1, abort_flag, err, 47, 128);
        if (!ok) break;
        const int flags = *seg_last;
        last = (flags & 4) != 0;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // exact sums, hi = diagonals 0..5 and lo = 6..10 (below 2^53 each)
        long long hi[20], lo[20];
        const uint32_t t0 = tmem + lanes + half * 20;
        if (flags & 256)
          fold_sums<true>(t0, hi, lo);
        else
          fold_sums<false>(t0, hi, lo);
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(tfree);
        const int32_t* eb = pr.eb + n0;
#pragma unroll
        for (int j = 0; j < 20; j += 2) {
          const int e0 = er + eb[j], e1 = er + eb[j + 1];
          const double2 o =
              scaled_pair2(hi[j], e0 - kW * (kHi - 1), lo[j], e0 - kW * (kS - 1), hi[j + 1],
                           e1 - kW * (kHi - 1), lo[j + 1], e1 - kW * (kS - 1));
          sum[j] = o.x;
          sum[j + 1] = o.y;
        }
        if (!first) {
#pragma unroll
          for (int j = 0; j < 20; ++j) sum[j] += prev[j * 256];
        }
        if (!last) {
#pragma unroll
          for (int j = 0; j < 20; ++j) prev[j * 256] = sum[j];
        }
      }
      if (!ok) break;
      if (P.fused) {
        const int G = pr.parts[0].grp, m0 = ai * kBM + q4 * 32, left = at.rows - q4 * 32;
        double* mom = reinterpret_cast<double*>(smem + kSumOff) + (warp - 2) * 32;
        uint16_t* lst = reinterpret_cast<uint16_t*>(smem + kListOff) + (warp - 2) * 640;
        if (G == 4)
          lines_of<4>(P, pr, n0, m0, lane, left, sum, mom, lst);
        else if (G == 2)
          lines_of<2>(P, pr, n0, m0, lane, left, sum, mom, lst);
        else
          lines_of<1>(P, pr, n0, m0, lane, left, sum, mom, lst);
      } else if (row_ok) {
        double* dst = pr.C + at.coff + r;
#pragma unroll
        for (int j = 0; j < 20; ++j)
          if (n0 + j < pr.Nc) dst[(long long)(n0 + j) * pr.ldc] = sum[j];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(P.ctr + 1, 1) == (int)gridDim.x - 1) {  // the last CTA: ready for the next launch
      P.ctr[0] = 0;
      P.ctr[1] = 0;
    }
  }
}

// ------------------------------------------------------------------ digits
// X = round(x 2^(55 - e)), |X| <= 2^54; adding 16 in every base-32 place makes
// the balanced digits plain 5-bit fields (minus 16), with no carry chain.  The
// top field is not masked: it reaches 32 (the digit 16).
constexpr unsigned long long bias_of(int n) {
  return n == 0 ? 0ull : bias_of(n - 1) | (16ull << (kW * (n - 1)));
}
constexpr unsigned long long kBias = bias_of(kS);
// e4m3 of two digits u - 16, u = 0..32: 0x6400 | u is the half 1024 + u.
__device__ __forceinline__ uint32_t e4m3x2(uint32_t u0, uint32_t u1) {
  const uint32_t h = (u0 | 0x6400u) | ((u1 | 0x6400u) << 16);
  const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&h), __float2half2_rn(1040.0f));
  return (uint32_t)__nv_cvt_halfraw2_to_fp8x2(static_cast<__half2_raw>(d), __NV_SATFINITE,
                                              __NV_E4M3);
}
// The digits of four consecutive elements k..k+3 of a row: one word per plane,
// planes `ps` bytes apart.  Returns the first plane with a digit (kS: none).
__device__ __forceinline__ int cut4(const double* x, int e, uint8_t* dst, uint32_t ps) {
  unsigned long long b[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) b[i] = (unsigned long long)fixed_point(x[i], e, kW * kS) + kBias;
  int z = kS;
#pragma unroll
  for (int p = kS - 1; p >= 0; --p) {
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      u[i] = (uint32_t)(b[i] >> (kW * (kS - 1 - p)));
      if (p > 0) u[i] &= 31u;
    }
    const uint32_t w = e4m3x2(u[0], u[1]) | (e4m3x2(u[2], u[3]) << 16);
    if (w) z = p;
    *reinterpret_cast<uint32_t*>(dst + p * ps) = w;
  }
  return z;
}
// Byte of element k (a multiple of 4) of row r within a tile's slices of
// `ss` bytes: 32-byte rows, 16-byte halves swapped in every other group of
// four rows (the 32-byte swizzle).
__device__ __forceinline__ size_t row_byte(int r, int k, uint32_t ss) {
  return (size_t)(k >> 5) * ss + r * 32 + ((((k >> 4) ^ (r >> 2)) & 1) << 4) + (k & 15);
}

__device__ __forceinline__ int block_exponent(unsigned long long mx) {
  __shared__ unsigned long long wmax[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = wmax[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) mx = max(mx, wmax[i]);
  return row_exponent(mx) + 1;  // |x| < 2^(e-1): every digit within 16
}
__device__ __forceinline__ unsigned long long magnitude(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
}

// One row of K = 4 K4 doubles (null: zeros) into row r of a tile; vk gathers
// its elements (-1: zero).  Memory bound: 8 B read (twice, the second time
// from L2) and 11 B written per element.  za (or null): the first plane with a
// digit of each slice, taken to the least of the tile's rows.
__device__ __forceinline__ void cut_row(const double* __restrict__ x, const int32_t* __restrict__ vk,
                                        int K, uint8_t* tile, uint32_t ps, uint32_t ss, int r,
                                        int32_t* e_out, int32_t* za = nullptr) {
  auto get = [&](int k, double* v) {
    if (!x) {
      v[0] = v[1] = v[2] = v[3] = 0.0;
    } else if (vk) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int s = vk[k + i];
        v[i] = s >= 0 ? x[s] : 0.0;
      }
    } else {
      const double2 a = *reinterpret_cast<const double2*>(x + k);
      const double2 b = *reinterpret_cast<const double2*>(x + k + 2);
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
  };
  unsigned long long mx = 0;
  for (int k = threadIdx.x * 4; k < K; k += 1024) {
    double v[4];
    get(k, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) mx = max(mx, magnitude(v[i]));
  }
  const int e = block_exponent(mx);
  if (threadIdx.x == 0) *e_out = e;
  for (int k = threadIdx.x * 4; k < K; k += 1024) {
    double v[4];
    get(k, v);
    int z = cut4(v, e, tile + row_byte(r, k, ss), ps);
    if (za) {  // K is a multiple of 32: the eight threads of a slice are all here
      const unsigned eight = 0xffu << (threadIdx.x & 24);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) z = min(z, __shfl_xor_sync(eight, z, o));
      if ((threadIdx.x & 7) == 0 && z < za[k >> 5]) atomicMin(za + (k >> 5), z);
    }
  }
}

// Rows of an A operand: block b is row b % 128 of tile b / 128.  rowsrc: source
// row of each (-1: zeros); null: row b of `rows`.  za[tile][slice] (or null; at
// least kS before): the planes from the top that are zero in all 128 rows (a
// dipole's elements fall off away from the diagonal, and a slice of elements
// 2^-5z of their rows' largest has nothing in its first z planes).  Taken here,
// where the digits are at hand; reading them back took 27 us at N = 2000.
__global__ void __launch_bounds__(256) k_cut8_a(const double* __restrict__ X, size_t ldx, int rows,
                                                int K, const int32_t* __restrict__ rowsrc,
                                                const int32_t* __restrict__ vk,
                                                uint8_t* __restrict__ out,
                                                int32_t* __restrict__ e_out, int32_t* za) {
  const int b = blockIdx.x, src = rowsrc ? rowsrc[b] : (b < rows ? b : -1);
  cut_row(src >= 0 ? X + (size_t)src * ldx : nullptr, vk, K,
          out + (size_t)(b >> 7) * (K >> 5) * kAS, kAP, kAS, b & 127, e_out + b, za ? za + (size_t)(b >> 7) * (K >> 5) : nullptr);
}

constexpr int kMaxOps8 = kMaxProb8;
struct CutOps8 {
  int n;
  int row0[kMaxOps8 + 1];
  int K[kMaxOps8];
  int ldx[kMaxOps8];
  const double* X[kMaxOps8];
  uint8_t* out[kMaxOps8];
  int32_t* e[kMaxOps8];
};
__global__ void __launch_bounds__(256) k_cut8_b(const __grid_constant__ CutOps8 ops) {
  const int b = blockIdx.x;
  int j = 0;
  while (j + 1 < ops.n && ops.row0[j + 1] <= b) ++j;
  const int n = b - ops.row0[j], t = n / kBN;
  cut_row(ops.X[j] + (size_t)n * ops.ldx[j], nullptr, ops.K[j],
          ops.out[j] + (size_t)t * (ops.K[j] >> 5) * kBS, kBP, kBS, n - t * kBN, ops.e[j] + n);
}

// Columns of Y straight into digits: block = one column (i, d) of a (unit,
// slot) group.  The value at each K position is the symmetrised -> primitive
// transform of the roots of that (slot, function) (k_build_y's arithmetic, from
// the basis's table), held in shared memory between the exponent and the cut
// (recomputed when the row does not fit).
template <bool DIGITS>
__global__ void __launch_bounds__(256) k_build_y8(const YItem8* __restrict__ items,
                                                  const int32_t* __restrict__ tile_item, int n,
                                                  int cached) {
  extern __shared__ __align__(16) double ys[];
  const long long b = blockIdx.x;
  int q = tile_item ? tile_item[b >> 6] : 0;
  while (q + 1 < n && items[q + 1].blk0 <= b) ++q;
  const YItem8& it = items[q];
  const int j = (int)(b - (tile_item ? it.blk0 : 0));  // i * ndeg + d
  const int i = j / it.ndeg, d = j - i * it.ndeg;
  const int K = it.nk * 32;
  const double* vs = it.vecs + (size_t)it.ivec[i] * it.ld;
  const double* yc = it.yc + (size_t)d * it.nent * it.nsv;
  // four consecutive positions: their loads are independent (a position's are
  // a chain of three)
  auto values = [&](int k, double* x) {
    const int4 v4 = *reinterpret_cast<const int4*>(it.vlist + k);
    const int v[4] = {v4.x, v4.y, v4.z, v4.w};
    x[0] = x[1] = x[2] = x[3] = 0.0;
    for (int n = 0; n < it.nent; ++n) {
      int s[4];
      double c[4];
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        s[q4] = v[q4] >= 0 ? it.ys[n * it.nsv + v[q4]] : 0;
        c[q4] = v[q4] >= 0 ? yc[n * it.nsv + v[q4]] : 0.0;
      }
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)
        if (c[q4] != 0.0) x[q4] = fma(vs[s[q4]], c[q4], x[q4]);
    }
  };
  if constexpr (!DIGITS) {
    double* y = reinterpret_cast<double*>(it.out) + (size_t)(it.col0 + j) * K;
    for (int k = threadIdx.x * 4; k < K; k += 1024) {
      double x[4];
      values(k, x);
      *reinterpret_cast<double2*>(y + k) = make_double2(x[0], x[1]);
      *reinterpret_cast<double2*>(y + k + 2) = make_double2(x[2], x[3]);
    }
    return;
  }
  unsigned long long mx = 0;
  for (int k = threadIdx.x * 4; k < K; k += 1024) {
    double x[4];
    values(k, x);
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4) mx = max(mx, magnitude(x[q4]));
    if (cached) {
      *reinterpret_cast<double2*>(ys + k) = make_double2(x[0], x[1]);
      *reinterpret_cast<double2*>(ys + k + 2) = make_double2(x[2], x[3]);
    }
  }
  const int e = block_exponent(mx);  // its barrier: every value of the row is in shared memory
  const int col = it.col0 + j, t = col / kBN, r = col - t * kBN;
  if (threadIdx.x == 0) it.e_out[col] = e;
  uint8_t* tile = it.out + (size_t)t * it.nk * kBS;
  for (int k = threadIdx.x * 4; k < K; k += 1024) {
    double v[4];
    if (cached) {
      const double2 a = *reinterpret_cast<const double2*>(ys + k);
      const double2 c = *reinterpret_cast<const double2*>(ys + k + 2);
      v[0] = a.x; v[1] = a.y; v[2] = c.x; v[3] = c.y;
    } else {
      values(k, v);
    }
    cut4(v, e, tile + row_byte(r, k, kBS), kBP);
  }
}
constexpr int kYSmem = 200 * 1024;  // longest cached row: 25,600 functions

cudaError_t attributes8() {
  static OncePerDevice once;
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  return once.run(device, [] {
    const cudaError_t a =
        cudaFuncSetAttribute(k_split8, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    return a != cudaSuccess
               ? a
               : cudaFuncSetAttribute(k_build_y8<true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, kYSmem);
  });
}

}  // namespace

// ------------------------------------------------------------------ host
struct Split8 {
  bool on = false;
  std::unique_ptr<VibPlan> plan;    // (null in a serving worker)
  // device tables of the plan `order_uid` for panels of `panel` rows: rowsrc, vk
  // and zpos in one allocation
  uint64_t order_uid = 0;
  int panel = 0;
  DevArray<int32_t> tables;
  const int32_t *rowsrc = nullptr, *vk = nullptr, *zpos = nullptr;
  std::vector<size_t> panel_tile;   // first row-source tile of each panel, and the end
  size_t most_tiles = 0;            // of a panel
  // the dipole's digits in that order
  bool mu_valid = false;
  DevArray<uint8_t> mu;
  DevArray<int32_t> mu_exp;
  DevArray<int32_t> za;             // zero planes of every slice of it
  std::vector<double> products;     // split8_products
  DevArray<uint8_t> b;              // B operand workspace
  DevArray<int32_t> b_exp;
  DevArray<int> ctr, err;
  bool err_clean = false;           // the error word is 0
};

static Split8* st8(Ctx* c) {
  if (!c->split8) c->split8 = new Split8();
  return c->split8;
}
static gi_status check8(Ctx* c, cudaError_t e, const char* what) {
  if (e == cudaSuccess) return GI_OK;
  c->err = std::string("split precision: ") + what + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? GI_ERR_NOMEM : GI_ERR_CUDA;
}

bool split8_selected(const Ctx* c) {
  if (c->params.split_slices > 0 || getenv("GI_SPLIT_FORCE")) return false;
  const char* l = getenv("GI_SPLIT_LAYOUT");
  return !(l && std::strcmp(l, "plain") == 0);
}
bool split8_active(const Ctx* c) { return c->split8 && c->split8->on; }

const VibPlan* vib_plan(Ctx* c, gi_status* st) {
  *st = GI_OK;
  Ctx* o = c->parent ? c->parent : c;
  Split8* S = st8(o);
  uint64_t key = 14695981039346656037ull ^ (uint64_t)o->N;
  for (auto& kv : o->bases) key = (key ^ kv.second->uid) * 1099511628211ull;
  if (S->plan && S->plan->key == key) return S->plan.get();
  if (c->parent) {  // bases cannot change while serving
    *st = fail(c, GI_ERR_STATE, "split precision: the serving context is not prepared");
    return nullptr;
  }
  auto vp = std::make_unique<VibPlan>();
  const int N = o->N;
  vp->key = key;
  vp->N = N;
  // classes (-1: used by no basis): the common refinement of the bases' kinds
  std::vector<int> cls(N, 0);
  std::vector<uint8_t> used(N, 0);
  vp->ncls = 1;
  for (auto& kv : o->bases) {
    const Basis& b = *kv.second;
    std::vector<int> id((size_t)vp->ncls * (b.nkind + 1), -1);
    int n = 0;
    for (int v = 0; v < N; v++) {
      const int kind = v < (int)b.v_kind.size() ? b.v_kind[v] : -1;
      used[v] |= kind >= 0;
      int& x = id[(size_t)cls[v] * (b.nkind + 1) + kind + 1];
      if (x < 0) x = n++;
      cls[v] = x;
    }
    vp->ncls = n;
    if (n > 1024) break;  // far too many to tell apart below
  }
  {  // without the unused ones, in order of appearance
    std::map<int, int> id;
    for (int v = 0; v < N; v++)
      cls[v] = used[v] ? id.emplace(cls[v], (int)id.size()).first->second : -1;
    vp->ncls = std::max<int>(1, (int)id.size());
  }
  const bool one = vp->ncls > 32;  // masks of classes are 32 bits: too many kinds, one class
  if (one) {
    vp->ncls = 1;
    for (auto& kv : o->bases)
      for (size_t v = 0; v < std::min<size_t>(N, kv.second->v_kind.size()); v++)
        used[v] |= kv.second->v_kind[v] >= 0;
    for (int v = 0; v < N; v++) cls[v] = used[v] ? 0 : -1;
  }
  vp->members.assign(vp->ncls, {});
  for (int v = 0; v < N; v++)
    if (cls[v] >= 0) vp->members[cls[v]].push_back(v);
  vp->zpos.assign(N, -1);
  int z = 0, s = 0;
  for (int k = 0; k < vp->ncls; k++) {
    const int n = (int)vp->members[k].size();
    vp->z0.push_back(z);
    vp->s0.push_back(s);
    for (int i = 0; i < n; i++) vp->zpos[vp->members[k][i]] = z + i;
    vp->vk.insert(vp->vk.end(), vp->members[k].begin(), vp->members[k].end());
    vp->vk.resize((size_t)round_up((int)vp->vk.size(), 32), -1);
    z += round_up(n, 16);
    s = (int)(vp->vk.size() / 32);
  }
  vp->s0.push_back(s);
  vp->nk = s;
  vp->ldz = std::max(round_up(z, 64), 64);
  for (auto& kv : o->bases) {
    const Basis& b = *kv.second;
    auto& sup = vp->support[b.uid];
    sup.assign((size_t)o->nrep * b.nslot, 0);
    for (int k = 0; k < vp->ncls; k++) {
      if (vp->members[k].empty()) continue;
      // a class is of one kind; with all functions in one class, every kind
      const size_t v = vp->members[k][0];
      const int kind = v < b.v_kind.size() ? b.v_kind[v] : -1;
      for (int q = one ? 0 : kind; q >= 0 && q < (one ? b.nkind : kind + 1); q++)
        for (int slot = 0; slot < b.nslot; slot++)
          for (unsigned m = b.kind_mask[(size_t)q * b.nslot + slot]; m; m &= m - 1)
            sup[(size_t)__builtin_ctz(m) * b.nslot + slot] |= 1u << k;
    }
  }
  S->plan = std::move(vp);
  return S->plan.get();
}

std::vector<VibTile> split8_tiles(const VibPlan& vp, int f0, int rows) {
  std::vector<VibTile> t;
  for (int comp = 0; comp < 3; comp++)
    for (int k = 0; k < vp.ncls; k++) {
      const auto& m = vp.members[k];
      const int a = (int)(std::lower_bound(m.begin(), m.end(), f0) - m.begin());
      const int b = (int)(std::lower_bound(m.begin(), m.end(), f0 + rows) - m.begin());
      for (int i = a; i < b; i += kBM) t.push_back(VibTile{comp, k, i, std::min(kBM, b - i)});
    }
  return t;
}

gi_status ensure_root_z(Ctx* c, Basis& b, const VibPlan& vp, bool* pending) {
  if (b.z_uid == vp.uid) return GI_OK;
  const Split8* S = (c->parent ? c->parent : c)->split8;
  GI_CUDA(c, b.d_root_z.reserve(std::max(b.D, 1)));
  GI_CUDA(c, launch_root_z(b, S->zpos, b.d_root_z.p, cudaStreamLegacy));
  if (pending)
    *pending = true;
  else
    GI_CUDA(c, cudaStreamSynchronize(cudaStreamLegacy));
  b.z_uid = vp.uid;
  return GI_OK;
}

uint32_t vib_support(const VibPlan& vp, const Basis& b, int gamma, int slot) {
  auto it = vp.support.find(b.uid);
  return it == vp.support.end() ? vp.all() : it->second[(size_t)gamma * b.nslot + slot];
}

void vib_rows_needed(const Ctx* c, const VibPlan& vp, const Basis& bI, int gF, int slot,
                     uint32_t rset[3]) {
  const Ctx* o = c->parent ? c->parent : c;
  int key = 0;
  while (bI.slot_of_key[key] != slot) key++;
  const int kI = key >> 1, tauI = key & 1;
  for (int jF = bI.J - 1; jF <= bI.J + 1; jF++) {
    auto it = o->bases.find(jF);
    if (it == o->bases.end()) continue;
    const Basis& bF = *it->second;
    for (int kF = std::max(kI - 1, 0); kF <= std::min(kI + 1, jF); kF++)
      for (int tauF = 0; tauF < 2; tauF++) {
        const int sF = bF.slot_of_key[2 * kF + tauF];
        if (sF < 0 || (kF == kI && tauF == tauI)) continue;
        // the component of the two keys (stencil_fill)
        rset[kF == kI ? 2 : tauF != tauI ? 0 : 1] |= vib_support(vp, bF, gF, sF);
      }
  }
}

static cudaError_t cut_dipole(Ctx* c, Split8* S, const VibPlan& vp, const double* mu, int p) {
  const size_t t0 = S->panel_tile[p], nt = S->panel_tile[p + 1] - t0;
  if (nt == 0) return cudaSuccess;
  // every byte kS: above kS as a word, the start of the minimum
  const cudaError_t e = cudaMemsetAsync(S->za.p, kS, nt * vp.nk * sizeof(int32_t), c->stream);
  if (e != cudaSuccess) return e;
  k_cut8_a<<<(unsigned)(nt * kBM), 256, 0, c->stream>>>(mu, (size_t)c->Kp, 0, vp.nk * 32,
                                                        S->rowsrc + t0 * kBM, S->vk, S->mu.p,
                                                        S->mu_exp.p, S->za.p);
  return cudaGetLastError();
}

gi_status vib_prepare(Ctx* c, const VibPlan** out) {
  gi_status g;
  const VibPlan* vp = vib_plan(c, &g);
  *out = vp;
  if (!vp) return g;
  if (c->parent) {
    const Split8* P = c->parent->split8;
    if (!P || P->order_uid != vp->uid)
      return fail(c, GI_ERR_STATE, "the serving context's dipole order is not prepared");
    return GI_OK;
  }
  Split8* S = st8(c);
  const int P = dipole_panel_rows(c);  // 0: the dipole is resident
  if (S->order_uid == vp->uid && S->panel == P) return GI_OK;
  S->order_uid = 0;
  S->mu_valid = false;
  const int N = c->N, step = P ? P : N;
  std::vector<int32_t> src;
  S->panel_tile.assign(1, 0);
  S->most_tiles = 0;
  for (int f0 = 0; f0 < N; f0 += step) {
    const auto tiles = split8_tiles(*vp, f0, std::min(step, N - f0));
    for (const VibTile& t : tiles)
      for (int r = 0; r < kBM; r++)
        src.push_back(r < t.rows ? t.comp * step + vp->members[t.cls][t.i0 + r] - f0 : -1);
    S->panel_tile.push_back(S->panel_tile.back() + tiles.size());
    S->most_tiles = std::max(S->most_tiles, tiles.size());
  }
  const size_t nsrc = src.size(), nvk = vp->vk.size();
  src.insert(src.end(), vp->vk.begin(), vp->vk.end());
  src.insert(src.end(), vp->zpos.begin(), vp->zpos.end());
  if ((g = check8(c, S->tables.assign(src), "dipole order")) != GI_OK) return g;
  S->rowsrc = S->tables.p;
  S->vk = S->rowsrc + nsrc;
  S->zpos = S->vk + nvk;
  S->panel = P;
  S->order_uid = vp->uid;
  return GI_OK;
}

const int32_t* vib_rowsrc(const Ctx* c, int panel) {
  const Split8* S = (c->parent ? c->parent : c)->split8;
  return S->rowsrc + S->panel_tile[panel] * kBM;
}

gi_status split8_prepare(Ctx* c) {
  Split8* S = st8(c);
  S->on = true;
  const VibPlan* vp;
  gi_status g = vib_prepare(c, &vp);
  if (g != GI_OK) return g;
  if (!S->err.p) {
    if ((g = check8(c, S->err.reserve(1), "error word")) != GI_OK) return g;
    if ((g = check8(c, S->ctr.reserve(2), "work counter")) != GI_OK) return g;
    if ((g = check8(c, cudaMemsetAsync(S->ctr.p, 0, 2 * sizeof(int), c->stream), "work counter")) !=
        GI_OK)
      return g;
  }
  if (!S->err_clean) {
    if ((g = check8(c, cudaMemsetAsync(S->err.p, 0, sizeof(int), c->stream), "error word")) !=
        GI_OK)
      return g;
    S->err_clean = true;
  }
  if ((g = check8(c, attributes8(), "kernel attributes")) != GI_OK) return g;
  if (c->parent) {
    const Split8* P = c->parent->split8;
    if (!P->mu_valid)
      return fail(c, GI_ERR_STATE,
                  "split precision: the dipole digits of the serving context are not prepared");
    return GI_OK;
  }
  if (S->mu_valid) return GI_OK;
  if ((g = check8(c, S->mu.reserve(a_bytes8(S->most_tiles, vp->nk)), "dipole digits")) != GI_OK)
    return g;
  if ((g = check8(c, S->mu_exp.reserve(S->most_tiles * kBM), "dipole exponents")) != GI_OK) return g;
  const size_t nza = S->most_tiles * vp->nk;
  if ((g = check8(c, S->za.reserve(std::max<size_t>(nza, 1)), "zero planes")) != GI_OK) return g;
  std::vector<int32_t> h_za(S->panel ? 0 : nza);
  if (!S->panel) {
    if ((g = check8(c, cut_dipole(c, S, *vp, c->d_mu.p, 0), "dipole digits")) != GI_OK) return g;
    if (nza)
      g = check8(c, cudaMemcpyAsync(h_za.data(), S->za.p, nza * sizeof(int32_t), cudaMemcpyDeviceToHost, c->stream),
                 "zero planes");
    if (g != GI_OK) return g;
    if ((g = check8(c, cudaStreamSynchronize(c->stream), "dipole digits")) != GI_OK) return g;
  }
  const size_t ntile = split8_tiles(*vp, 0, c->N).size();
  S->products.assign(ntile * vp->ncls, 0.0);
  for (size_t t = 0; t < ntile; t++)
    for (int k = 0; k < vp->ncls; k++) {
      int left = (int)vp->members[k].size();
      for (int q = vp->s0[k]; q < vp->s0[k + 1]; q++, left -= 32) {
        const int np = kS - (h_za.empty() ? 0 : std::min(h_za[t * vp->nk + q], kS));
        S->products[t * vp->ncls + k] += 0.5 * np * (np + 1) * std::min(left, 32);
      }
    }
  S->mu_valid = true;
  return GI_OK;
}

// A final block's digits, cut once and kept with the block until its vectors
// change (serving workers share blocks: the cut happens under the model lock
// and the others wait on its event).
static gi_status block_digits8(Ctx* c, Block& fb, bool wait) {
  const int vpad = round_up(fb.nvec, kBM);
  gi_status g;
  std::lock_guard<std::mutex> lk(c->mmu());
  if (fb.digits_s != kS || fb.digits_w != kW || fb.digits_layout != 2) {
    const size_t nd = a_bytes8(vpad / kBM, fb.ld / 32) / sizeof(uint16_t);
    if (fb.d_digits.n != std::max<size_t>(nd, 1)) {
      g = check8(c, fb.d_digits.alloc(nd), "V digits");
      if (g != GI_OK) return g;
    }
    if (fb.d_digit_exp.n != (size_t)std::max(vpad, 1)) {
      g = check8(c, fb.d_digit_exp.alloc(vpad), "V exponents");
      if (g != GI_OK) return g;
    }
    if (vpad) {
      g = check8(c, timed(c, GI_PHASE_SLICE, [&] {
                   k_cut8_a<<<vpad, 256, 0, c->stream>>>(
                       fb.d_vecs.p, (size_t)fb.ld, fb.nvec, fb.ld, nullptr, nullptr,
                       reinterpret_cast<uint8_t*>(fb.d_digits.p), fb.d_digit_exp.p,
                       nullptr);
                   return cudaGetLastError();
                 }),
                 "V digits");
      if (g != GI_OK) return g;
    }
    if (!fb.digits_ev) {
      g = check8(c, cudaEventCreateWithFlags(&fb.digits_ev, cudaEventDisableTiming), "event");
      if (g != GI_OK) return g;
    }
    g = check8(c, cudaEventRecord(fb.digits_ev, c->stream), "event");
    if (g != GI_OK) return g;
    fb.digits_s = kS;
    fb.digits_w = kW;
    fb.digits_layout = 2;
  }
  if (wait && fb.digits_ev) {
    // inside a graph capture the cut precedes the capture on this stream
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    g = check8(c, cudaStreamIsCapturing(c->stream, &cs), "capture status");
    if (g != GI_OK) return g;
    if (cs == cudaStreamCaptureStatusNone) {
      g = check8(c, cudaStreamWaitEvent(c->stream, fb.digits_ev, 0), "event wait");
      if (g != GI_OK) return g;
    }
  }
  return GI_OK;
}

gi_status split8_reserve(Ctx* c, size_t b_bytes, size_t cols, const std::vector<Block*>& finals) {
  Split8* S = st8(c);
  gi_status g = check8(c, S->b.reserve(std::max<size_t>(b_bytes, 1)), "B digits");
  if (g != GI_OK) return g;
  // a tile's epilogue reads the exponents of all its columns
  g = check8(c, S->b_exp.reserve(cols + kCols8), "B exponents");
  if (g != GI_OK) return g;
  for (Block* b : finals) {
    g = block_digits8(c, *b, false);
    if (g != GI_OK) return g;
  }
  return GI_OK;
}
void split8_dipole_operand(Ctx* c, Prob8* p) {
  const Split8* D = (c->parent ? c->parent : c)->split8;
  p->A = D->mu.p;
  p->ea = D->mu_exp.p;
  p->za = D->za.p;
  p->nkA = D->plan->nk;
}
const std::vector<double>& split8_products(const Ctx* c) {
  return (c->parent ? c->parent : c)->split8->products;
}
uint8_t* split8_b(Ctx* c) { return st8(c)->b.p; }
int32_t* split8_b_exp(Ctx* c) { return st8(c)->b_exp.p; }

gi_status split8_build_y(Ctx* c, const YItem8* items, const int32_t* tile_item, int n,
                         long long blocks, bool digits) {
  if (n <= 0 || blocks <= 0) return GI_OK;
  if (blocks > 0x7FFFFFFFll) return check8(c, cudaErrorInvalidValue, "Y digits");
  gi_status g;
  const VibPlan* vp = vib_plan(c, &g);
  if (!vp) return g;
  const size_t row = (size_t)vp->nk * 32 * sizeof(double);
  const int cached = row <= (size_t)kYSmem;
  return check8(c, timed(c, GI_PHASE_CORRELATE, [&] {
                  if (digits)
                    k_build_y8<true><<<(unsigned)blocks, 256, cached ? row : 0, c->stream>>>(
                        items, tile_item, n, cached);
                  else
                    k_build_y8<false><<<(unsigned)blocks, 256, 0, c->stream>>>(items, tile_item, n,
                                                                              0);
                  return cudaGetLastError();
                }),
                "Y digits");
}

// Launches the problems as one work list, longest contractions first.  tune:
// the launch only stores C, so the autotuner may repeat it.
gi_status split8_launch(Ctx* c, int phase, std::vector<Prob8>& probs, const FusedLines* lines,
                        bool tune) {
  Split8* S = st8(c);
  std::vector<Prob8> live;
  for (const Prob8& p : probs)
    if (p.nA > 0 && p.Nc > 0 && p.nk > 0) live.push_back(p);
  if (live.empty()) return GI_OK;
  if (live.size() > (size_t)kMaxProb8) return check8(c, cudaErrorInvalidValue, "problem count");
  std::stable_sort(live.begin(), live.end(),
                   [](const Prob8& a, const Prob8& b) { return a.nk > b.nk; });
  Params8* P = new Params8();  // 16 KB: not on the host stack
  P->nprob = (int)live.size();
  P->fused = lines ? 1 : 0;
  P->ctr = S->ctr.p;
  if (lines) {
    P->out = lines->out;
    P->counter = lines->counter;
    P->cap = lines->cap;
    P->rec = lines->rec;
    P->rec_cap = lines->rec_cap;
  }
  long long total_a = 0, total_n = 0, max_k = 0;
  for (const Prob8& p : live) {
    total_a = std::max<long long>(total_a, p.nA);
    total_n += p.Nc;
    max_k = std::max<long long>(max_k, p.nk);
  }
  auto run = [&](const GemmConfig& cfg) -> cudaError_t {
    long long items = 0;
    for (int q = 0; q < P->nprob; q++) {
      Prob8& p = P->p[q];
      p = live[q];
      p.nB = (p.Nc + kBN - 1) / kBN;
      // row tiles whose digits share ga_mb MB of L2
      p.GA = (int)std::max<size_t>(1, std::min<size_t>(p.nA, ((size_t)cfg.ga_mb << 20) /
                                                                 ((size_t)p.nk * kAS)));
      p.first = (int)items;
      items += (long long)p.nA * p.nB;
    }
    if (items > 0x7FFF0000ll) return cudaErrorInvalidValue;
    P->nitems = (int)items;
    const int grid = (int)std::min<long long>(items, std::max(c->nsm, 1));
    k_split8<<<grid, kThreads, kSmem, c->stream>>>(*P, S->err.p);
    return cudaGetLastError();
  };
  gi_status g = GI_OK;
  timed(c, phase, [&] {
    if (tune)
      g = split_tuned(c, kS, (int)total_a, (int)total_n, (int)(max_k * 32), 2, run);
    else
      g = check8(c, run(GemmConfig{6, 64}), "GEMM launch");
    return cudaSuccess;
  });
  delete P;
  return g;
}

gi_status split8_gemm_dipole(Ctx* c, const std::vector<Band8>& bands, double* Z, int ldz) {
  Split8* S = st8(c);
  gi_status g;
  const VibPlan* vp = vib_plan(c, &g);
  if (!vp) return g;
  auto launch = [&](int panel) {
    std::vector<Prob8> probs;
    for (const Band8& b : bands) {
      Prob8 p{};
      split8_dipole_operand(c, &p);
      p.B = S->b.p + b.boff;
      p.eb = S->b_exp.p + b.col0;
      p.C = Z + b.col0 * (size_t)ldz;
      p.ldc = ldz;
      p.at = b.at[panel];
      p.nA = b.nA[panel];
      p.kl = b.kl;
      p.nkB = p.nk = b.nk;
      p.Nc = (int)b.ncol;
      probs.push_back(p);
    }
    return split8_launch(c, GI_PHASE_HALFLS_GEMM, probs, nullptr, true);
  };
  if (!S->panel || c->parent) return launch(0);
  int p = 0;
  return for_each_dipole_panel(c, c->stream, [&](const double* mu, size_t, int, int) -> gi_status {
    gi_status q = check8(c, timed(c, GI_PHASE_SLICE, [&] { return cut_dipole(c, S, *vp, mu, p); }),
                         "dipole panel digits");
    return q != GI_OK ? q : launch(p++);
  });
}

gi_status split8_gemm_final(Ctx* c, const std::vector<FinalJob>& jobs, const FusedLines* lines) {
  Split8* S = st8(c);
  if (jobs.empty() || (int)jobs.size() > kMaxOps8)
    return fail(c, GI_ERR_STATE, "split precision: final GEMM problem count");
  gi_status g;
  const char* bs_env = getenv("GI_BATCH_SMALL");
  const bool batch = !(bs_env && bs_env[0] == '0');  // off: one cut per problem
  std::vector<Prob8> probs;
  CutOps8* ops = new CutOps8();
  size_t boff = 0, eoff = 0;
  g = GI_OK;
  auto cut = [&] {
    if (ops->n == 0) return GI_OK;
    const gi_status q = check8(c, timed(c, GI_PHASE_SLICE, [&] {
                                 k_cut8_b<<<ops->row0[ops->n], 256, 0, c->stream>>>(*ops);
                                 return cudaGetLastError();
                               }),
                               "H digits");
    ops->n = 0;
    return q;
  };
  for (const FinalJob& j : jobs) {
    Block& fb = *j.fb;
    if ((g = block_digits8(c, fb, /*wait=*/true)) != GI_OK) break;
    if (j.ncol <= 0) continue;
    Prob8 p{};
    p.A = reinterpret_cast<const uint8_t*>(fb.d_digits.p);
    p.ea = fb.d_digit_exp.p;
    p.B = S->b.p + boff;
    p.eb = S->b_exp.p + eoff;
    p.C = j.T;
    p.ldc = j.ldt;
    p.nkA = p.nkB = p.nk = j.ldh / 32;
    p.M = fb.nvec;
    p.nA = (fb.nvec + kBM - 1) / kBM;
    p.Nc = j.ncol;
    p.parts = j.parts;
    p.nparts = j.nparts;
    p.EF = j.EF;
    p.upper = j.upper;
    p.lvF = j.lvF;
    if (boff + b_bytes8(j.ncol, p.nk) > S->b.n || eoff + j.ncol + kCols8 > S->b_exp.n ||
        (lines && (!j.parts || j.nparts <= 0))) {
      g = fail(c, GI_ERR_STATE, "split precision: final GEMM workspace not prepared");
      break;
    }
    probs.push_back(p);
    const int o = ops->n++;
    if (o == 0) ops->row0[0] = 0;
    ops->K[o] = j.ldh;
    ops->ldx[o] = j.ldh;
    ops->X[o] = j.H;
    ops->out[o] = S->b.p + boff;
    ops->e[o] = S->b_exp.p + eoff;
    ops->row0[o + 1] = ops->row0[o] + j.ncol;
    boff += b_bytes8(j.ncol, p.nk);
    eoff += round_up(j.ncol, kCols8);  // whole tiles: aligned exponents
    c->stats.flops_tensor +=
        (double)kS * (kS + 1) / 2 * 2.0 * fb.nvec * (double)j.ncol * fb.nsize;
    if (!batch && (g = cut()) != GI_OK) break;
  }
  if (g == GI_OK) g = cut();
  delete ops;
  if (g != GI_OK) return g;
  return split8_launch(c, GI_PHASE_FINAL_GEMM, probs, lines, !lines && jobs.size() == 1);
}

uint64_t split8_identity(Ctx* c) {
  Split8* S = st8(c);
  const Split8* D = c->parent ? c->parent->split8 : S;
  uint64_t h = 14695981039346656037ull;
  for (uint64_t v : {(uint64_t)(uintptr_t)S->b.p, (uint64_t)(uintptr_t)S->b_exp.p,
                     (uint64_t)(uintptr_t)S->ctr.p, (uint64_t)(uintptr_t)S->err.p,
                     (uint64_t)(uintptr_t)D->mu.p, (uint64_t)(uintptr_t)D->mu_exp.p, (uint64_t)(uintptr_t)D->za.p,
                     D->order_uid,
                     split_tuner_version()})
    h = (h ^ v) * 1099511628211ull;
  return h;
}
void split8_error_seen(Ctx* c) {
  if (c->split8) c->split8->err_clean = false;
}
const int* split8_error_word(const Ctx* c) { return c->split8 ? c->split8->err.p : nullptr; }
void split8_deactivate(Ctx* c) { c->split8->on = false; }
void split8_invalidate(Ctx* c) {
  if (c->split8) c->split8->mu_valid = false;
}
void split8_release(Ctx* c) {
  delete c->split8;
  c->split8 = nullptr;
}

gi_status split8_probe(Ctx* c, int M, int N, int K, const double* dA, const double* dB, int ld,
                       double* dC) {
  Split8* S = st8(c);
  S->on = true;
  const int vpad = round_up(M, kBM), nk = ld / 32;
  DevArray<uint8_t> a, b;
  DevArray<int32_t> ea, eb;
  gi_status g = check8(c, S->err.reserve(1), "error word");
  if (g == GI_OK) g = check8(c, S->ctr.reserve(2), "work counter");
  if (g == GI_OK) g = check8(c, cudaMemset(S->err.p, 0, sizeof(int)), "error word");
  if (g == GI_OK) g = check8(c, cudaMemset(S->ctr.p, 0, 2 * sizeof(int)), "work counter");
  if (g == GI_OK) g = check8(c, attributes8(), "kernel attributes");
  if (g == GI_OK) g = check8(c, a.alloc(a_bytes8(vpad / kBM, nk)), "A digits");
  if (g == GI_OK) g = check8(c, b.alloc(b_bytes8(N, nk)), "B digits");
  if (g == GI_OK) g = check8(c, ea.alloc(vpad), "A exponents");
  if (g == GI_OK) g = check8(c, eb.alloc(N + kCols8), "B exponents");
  if (g == GI_OK) g = check8(c, cudaDeviceSynchronize(), "operands");
  if (g != GI_OK) return g;
  k_cut8_a<<<vpad, 256, 0, c->stream>>>(dA, (size_t)ld, M, ld, nullptr, nullptr, a.p, ea.p,
                                        nullptr);
  if ((g = check8(c, cudaGetLastError(), "A digits")) != GI_OK) return g;
  CutOps8* ops = new CutOps8();
  ops->n = 1;
  ops->row0[0] = 0;
  ops->row0[1] = N;
  ops->K[0] = ops->ldx[0] = ld;
  ops->X[0] = dB;
  ops->out[0] = b.p;
  ops->e[0] = eb.p;
  k_cut8_b<<<N, 256, 0, c->stream>>>(*ops);
  delete ops;
  if ((g = check8(c, cudaGetLastError(), "B digits")) != GI_OK) return g;
  Prob8 p{};
  p.A = a.p;
  p.ea = ea.p;
  p.B = b.p;
  p.eb = eb.p;
  p.C = dC;
  p.ldc = M;
  p.nkA = p.nkB = p.nk = nk;
  p.M = M;
  p.nA = vpad / kBM;
  p.Nc = N;
  std::vector<Prob8> probs{p};
  g = split8_launch(c, GI_PHASE_FINAL_GEMM, probs, nullptr, true);
  if (g == GI_OK) g = check8(c, cudaStreamSynchronize(c->stream), "probe");
  return g;
}

}  // namespace gi
