/*
 * CSR step on the device: CSRCSBEND (track_through_csbendCSR, csbend.c:1899-3044)
 * and CSRDRIFT mode 0 (track_through_driftCSR, csbend.c:3176-3533).
 * See b2e_csr.h for the kernel pipeline.  Every floating-point expression
 * keeps the reference's operation order; histogram counts are integers and
 * min/max are exact, so the pipeline reproduces the CPU oracle bit for bit
 * regardless of thread scheduling.
 */
#include <math.h>
#include <string.h>
#include <stdio.h>
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <utility>
#include "b2e_csr.h"
#include "b2e_roots.h"
#include "b2e_fft.h"
#include "b2e_fast.cuh"
#include "b2e_kernels.h"
#include "b2e_sg.h"
#include "b2e_wakenet.h"

namespace b2e {

static const double kPI = 3.141592653589793238462643383279502884;
static const double kC = 2.99792458e8;
static const double kE = 1.602176634e-19;
static const double kME = 9.1093837015e-31;

struct CsrDevState {
  unsigned long long ct_min_key, ct_max_key; /* order-preserving keys of min/max c*t */
  double ctLower, ctUpper, dct;              /* binning of the current kick */
  double s0, dctBin;                         /* csrWake.s0, csrWake.dctBin */
  long long nBinned;
  double dGamma[B2E_CSR_MAX_BINS];           /* csrWake.dGamma: last dipole wake */
  double phi_last;                           /* SolveForPhiStupakov's start value */
};

/* Per-bunch view for the CSR kernels.  Bunches are contiguous particle ranges
 * [offs[b], offs[b+1]); each has its own binning and wake state, its own
 * CSRConstant (zero when the bunch has at most one particle at the element
 * entrance) and, in CSRDRIFT, its own choice between wake kicks and the exact
 * drift.  A single bunch is n = 1 (offs is then not read). */
struct CsrBunches {
  const int64_t *offs;
  int n;
  CsrDevState *st;
  const double *csr_const; /* [3][n]: CSRConstant, the IGF wake factor, GSConstant */
  const unsigned char *active; /* more than one particle alive at the element entrance */
  const unsigned char *mode;   /* CSRDRIFT: 1 = wake kicks, 0 = exact drift */
};

__device__ __forceinline__ int bunch_of(int64_t i, const CsrBunches &B) {
  if (B.n <= 1)
    return 0;
  int lo = 0, hi = B.n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (B.offs[mid] <= i)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ unsigned long long key_of(double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double value_of(unsigned long long k) {
  unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}

/* binParticleCoordinate's range expansion (csbend.c:3079-3094) */
__device__ __forceinline__ void expand_range(double *lower, double *upper, double factor) {
  if (factor > 1) {
    double center = (*lower + *upper) / 2, range = (*upper - *lower) * factor;
    *lower = center - range / 2;
    *upper = center + range / 2;
  }
}

/* Range of c*t per bunch, for kernels whose threads take particles of rising
 * index: each thread keeps the range of the warp's current bunch in registers,
 * and a warp sends its two atomics when the bunch changes and at the end.  A pair
 * for every 32 particles would be 62,500 atomics on two words for a bunch of a
 * million. */
struct BunchRange {
  unsigned long long kmin = ~0ull, kmax = 0ull;
  int cur;
  __device__ explicit BunchRange(int bunch) : cur(bunch) {}
  /* all lanes of the warp */
  __device__ void flush(const CsrBunches &B) {
    for (int off = 16; off > 0; off >>= 1) {
      kmin = min(kmin, __shfl_down_sync(0xffffffffu, kmin, off));
      kmax = max(kmax, __shfl_down_sync(0xffffffffu, kmax, off));
    }
    if ((threadIdx.x & 31) == 0 && kmax != 0ull) {
      atomicMin(&B.st[cur].ct_min_key, kmin);
      atomicMax(&B.st[cur].ct_max_key, kmax);
    }
    kmin = ~0ull;
    kmax = 0ull;
  }
  /* all lanes of the warp: a particle of bunch b, if valid */
  __device__ void add(double v, bool valid, int b, const CsrBunches &B) {
    const int b0 = __shfl_sync(0xffffffffu, b, 0);
    if (__all_sync(0xffffffffu, b == b0)) {
      if (b0 != cur) {
        flush(B);
        cur = b0;
      }
      if (valid) {
        kmin = min(kmin, key_of(v));
        kmax = max(kmax, key_of(v));
      }
    } else if (valid) {
      /* the warp straddles bunches */
      atomicMin(&B.st[b].ct_min_key, key_of(v));
      atomicMax(&B.st[b].ct_max_key, key_of(v));
    }
  }
};

/* CSR energy kick from the previous kick's wake (csbend.c:2692-2711) */
__device__ __forceinline__ double csr_kick(double CT, double X, double DP, const CsrDevState *st, int nBins,
                                           double Po, double rho0) {
  double f = (CT - st->ctLower) / st->dct;
  long long iBin = (long long)f;
  f -= iBin;
  if (iBin >= 0 && iBin < nBins - 1)
    DP += ((1 - f) * st->dGamma[iBin] + f * st->dGamma[iBin + 1]) / Po * (1 + X / rho0);
  return DP;
}

/* Programmatic dependent launch (sm_90 and later, PTX griddepcontrol): a
 * kernel of the kick chain launched with the programmatic-serialization
 * attribute may be scheduled while its predecessor's last CTAs still run.
 * Each such kernel first lets its own successor be scheduled (once all of its
 * CTAs have started), then waits until the predecessor grid has completed
 * and its memory is visible, before touching any memory.  In a kernel
 * launched without the attribute both instructions return at once. */
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_enter() {
  chain_release();
  chain_wait();
}

/* entrance: offsets, tilt, c*t = s/beta, entrance edge (csbend.c:2286-2377) */
__global__ void csr_entry_kernel(DevParticles P, int64_t n, double *beta0, const DevElem *ep, BendExtra bx,
                                 double Po) {
  chain_enter();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || P.lost_pass[i] >= 0)
    return;
  const DevElem &e = *ep;
  const double *c = e.c;
  const double ct = c[CB_COS_TT], st = c[CB_SIN_TT];
  double x = P.x[i], xp = P.xp[i], y = P.y[i], yp = P.yp[i], s = P.s[i], dp = P.dp[i];
  double X, Y, XP, YP, p0, b0, rho;
  s = s + c[CB_DZI] * sqrt((1 + xp * xp) + yp * yp);
  x = (x + c[CB_DXI]) + c[CB_DZI] * xp;
  y = (y + c[CB_DYI]) + c[CB_DZI] * yp;
  X = x * ct + y * st;
  Y = -x * st + y * ct;
  XP = xp * ct + yp * st;
  YP = -xp * st + yp * ct;
  p0 = Po * (1 + dp);
  b0 = p0 / sqrt(p0 * p0 + 1);
  s = s / b0;
  if (e.flags & EF_EDGE1) {
    rho = (1 + dp) * c[CB_RHO_ACTUAL];
    if (e.flags & EF_EDGE_ORDER2) {
      bend_edge_order2(X, XP, Y, YP, rho, c[CB_PSI1] * (1 + dp), c[CB_TAN_E1], c[CB_E1], bx.c[BX_SEC2_E1],
                       bx.c[BX_EDGE_N], -1);
    } else {
      XP = XP + (c[CB_TAN_E1] / rho) * X;
      YP = YP - (b2e_tan(c[CB_E1] - c[CB_PSI1] / (1 + dp)) / rho) * Y;
    }
  }
  P.x[i] = X;
  P.xp[i] = XP;
  P.y[i] = Y;
  P.yp[i] = YP;
  P.s[i] = s;
  beta0[i] = b0;
}

/* one particle's kick: coordinates, c*t and the entrance velocity */
struct SlicePart {
  double X, XP, Y, YP, CT, DP, beta0;
};

/* a bunch's wake as the kick reads it */
struct SliceWake {
  const double *dGamma;
  double lower, dct;
  int nBins, apply;
};

/* Optional wake kick of the previous kick, one integrator slice, c*t update
 * (csbend.c:2385-2450), in the general form */
__device__ __forceinline__ int csr_slice_general(SlicePart *p, const DevElem &e, const CsrDevState *st, int nBins,
                                                 int apply, double Po) {
  const double *c = e.c;
  double f, Q1, Q3, Q4;
  if (apply)
    p->DP = csr_kick(p->CT, p->X, p->DP, st, nBins, Po, c[CB_RHO0]);
  f = (1 + p->DP) / sqrt((1 + p->XP * p->XP) + p->YP * p->YP);
  Q1 = p->XP * f;
  Q3 = p->YP * f;
  const RadSite no_rad = {0, 0, 0, 0, 0, nullptr};
  const int lost =
    csbend_integrate<false>(p->X, Q1, p->Y, Q3, Q4, p->DP, c, 1, (int)c[CB_NSUB], false, nullptr, e, no_rad);
  f = 1 / sqrt(((1 + p->DP) * (1 + p->DP) - Q1 * Q1) - Q3 * Q3);
  p->XP = Q1 * f;
  p->YP = Q3 * f;
  if (!lost)
    p->CT = p->CT + Q4 / p->beta0;
  return lost;
}

/* out of line, for particles near a limit of the straight-line form */
static __device__ __noinline__ int csr_slice_outlier(SlicePart *p, const DevElem *e, const CsrDevState *st, int nBins,
                                                     int apply, double Po) {
  return csr_slice_general(p, *e, st, nBins, apply, Po);
}

static __device__ __noinline__ double divide_ieee(double a, double b) { return a / b; }

/* The same in the straight-line form of b2e_fast.cuh (four substeps).  Returns
 * false where that does not apply; the caller then reads the particle again.
 * ct0 and beta0 are read where they are used, from shared memory. */
__device__ __forceinline__ bool csr_slice_fast(SlicePart &p, const DevElem &e, const SliceWake &w, const double *ct0,
                                               const double *beta0, double Po, double inv_Po) {
  const double *c = e.c;
  double r, ir, f, dist;
  if (w.apply) {
    f = fp_quot(*ct0 - w.lower, w.dct, fp_recip(w.dct));
    const long long iBin = (long long)f;
    f -= iBin;
    if (iBin >= 0 && iBin < w.nBins - 1) {
      const double g = (1 - f) * w.dGamma[iBin] + f * w.dGamma[iBin + 1];
      const double h = fp_plain(g, FP_HI_2P100) ? fp_quot(g, Po, inv_Po) : divide_ieee(g, Po);
      p.DP += h * (1 + fp_quot(p.X, c[CB_RHO0], c[CB_INV_RHO0]));
    }
  }
  double A = 1 + p.DP;
  r = fp_sqrt_recip((1 + p.XP * p.XP) + p.YP * p.YP, ir);
  bool ok = fp_abs_hi(p.X) < FP_HI_2P100 && fp_plain(p.XP, FP_HI_2) && fp_plain(p.YP, FP_HI_2) &&
            fp_within(A, FP_HI_2M4, FP_HI_2P4);
  f = fp_quot(A, r, ir);
  p.XP = p.XP * f;
  p.YP = p.YP * f;
  /* a kick adds a zero to QY, which a negative zero would not survive */
  ok = ok && fp_hi(p.YP) != 0x80000000u;
  ok = bend_slices_fast<TRIP_NONE>(p.X, p.XP, p.Y, p.YP, dist, A, 0.0, c, 1, 4, nullptr, e) && ok;
  const double d = (A * A - p.XP * p.XP) - p.YP * p.YP;
  r = fp_sqrt_recip(d, ir);
  ok = ok && fp_within(d, FP_HI_2M10, FP_HI_2P10) && fp_plain(dist, FP_HI_2P100);
  f = fp_quot(1.0, r, ir);
  p.XP = p.XP * f;
  p.YP = p.YP * f;
  const double b0 = *beta0;
  p.CT = *ct0 + fp_quot(dist, b0, fp_recip(b0));
  return ok && fp_within(b0, FP_HI_2M10, FP_HI_2);
}

constexpr int SLICE_THREADS = 128, SLICE_COLS = 7, SLICE_BLOCKS_PER_SM = 6;

__device__ __forceinline__ void copy8_async(void *smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void copy4_async(void *smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}

/* One kick of every particle, and min/max of c*t per bunch (csbend.c:3066-3076).
 * Each block takes a run of 128-particle tiles; a thread copies its particle of
 * the next tile into shared memory (its own words only, so no barrier) while it
 * integrates the current one.  Bound by the FP64 pipe and its register ports:
 * of about 920 warp instructions per 32 particles 430 are FP64, and an fma of
 * three different registers issues every third cycle, not every second.  20 to
 * 32 warps per SM, and two particles per thread, all measured within 2 %.  48.6 us
 * for 1e6 particles under ncu; 59.3 us with a block per 256 particles that waits
 * for the loss word, then for the coordinates, then for the velocity, and two
 * atomics per warp. */
template <bool STRAIGHT>
__global__ void __launch_bounds__(SLICE_THREADS, SLICE_BLOCKS_PER_SM)
    csr_slice_kernel(DevParticles P, int64_t n, int64_t tiles_per_block, const double *beta0,
                     const __grid_constant__ DevElem e, CsrBunches B, int after_first_kick, int nBins, double Po,
                     double inv_Po, int pass, int elem_index) {
  __shared__ double col[2][SLICE_COLS][SLICE_THREADS];
  __shared__ int32_t lost_word[2][SLICE_THREADS];
  chain_enter();
  const int t = threadIdx.x;
  const int64_t begin = blockIdx.x * tiles_per_block * SLICE_THREADS + t;
  const int64_t end = min(n, (blockIdx.x + 1) * tiles_per_block * SLICE_THREADS);
  const bool usual_Po = fp_within(Po, FP_HI_2M10, FP_HI_2P100);
  auto fetch = [&](int64_t i, int slot) {
    if (i < end) {
      copy8_async(&col[slot][0][t], P.x + i);
      copy8_async(&col[slot][1][t], P.xp + i);
      copy8_async(&col[slot][2][t], P.y + i);
      copy8_async(&col[slot][3][t], P.yp + i);
      copy8_async(&col[slot][4][t], P.s + i);
      copy8_async(&col[slot][5][t], P.dp + i);
      copy8_async(&col[slot][6][t], beta0 + i);
      copy4_async(&lost_word[slot][t], P.lost_pass + i);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int bunch = begin - t < n ? bunch_of(begin - t, B) : 0;
  int64_t bunch_end = B.n <= 1 ? n : B.offs[bunch + 1];
  BunchRange range(bunch);
  fetch(begin, 0);
  int slot = 0;
  /* the loop's bounds are the same for all threads of the block */
  for (int64_t i = begin; i - t < end; i += SLICE_THREADS, slot ^= 1) {
    fetch(i + SLICE_THREADS, slot ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    while (i < end && i >= bunch_end && bunch < B.n - 1) {
      bunch++;
      bunch_end = B.offs[bunch + 1];
    }
    const CsrDevState *st = B.st + bunch;
    bool alive = i < end && lost_word[slot][t] < 0;
    SlicePart p;
    if (alive) {
      const double(*v)[SLICE_THREADS] = col[slot];
      const SliceWake w = {st->dGamma, st->ctLower, st->dct, nBins, after_first_kick && B.csr_const[bunch] != 0};
      int lost = 0;
      if constexpr (STRAIGHT) {
        p.X = v[0][t];
        p.XP = v[1][t];
        p.Y = v[2][t];
        p.YP = v[3][t];
        p.DP = v[5][t];
        if (!(usual_Po && (!w.apply || fp_within(w.dct, FP_HI_2M250, FP_HI_2P100)) &&
              csr_slice_fast(p, e, w, &v[4][t], &v[6][t], Po, inv_Po))) {
          SlicePart q = {v[0][t], v[1][t], v[2][t], v[3][t], v[4][t], v[5][t], v[6][t]};
          lost = csr_slice_outlier(&q, &e, st, nBins, w.apply, Po);
          p = q;
        }
      } else {
        p = {v[0][t], v[1][t], v[2][t], v[3][t], v[4][t], v[5][t], v[6][t]};
        lost = csr_slice_general(&p, e, st, nBins, w.apply, Po);
      }
      P.x[i] = p.X;
      P.xp[i] = p.XP;
      P.y[i] = p.Y;
      P.yp[i] = p.YP;
      P.dp[i] = p.DP;
      if (lost) {
        P.lost_pass[i] = pass;
        P.lost_elem[i] = elem_index;
        alive = false;
      } else {
        P.s[i] = p.CT;
      }
    }
    __syncwarp();
    range.add(p.CT, alive, bunch, B);
  }
  range.flush(B);
}

/* The straight-line form holds four substeps (INTEGRATION_ORDER 4) and takes
 * elements of EF_FAST.  The others have a kernel of their own: 1e6 particles
 * through 10 kicks per dipole at INTEGRATION_ORDER 6 took 5.89 ms with the
 * general form called out of line from one kernel for all, 5.48 ms with it in
 * line; 3.12 and 2.86 ms at order 2. */
static auto slice_kernel(const DevElem &e) {
  return (e.flags & EF_FAST) && e.c[CB_NSUB] == 4 ? csr_slice_kernel<true> : csr_slice_kernel<false>;
}

/* grid and tiles per block: as many blocks as the SMs hold at once, each with
 * an equal run of tiles */
static inline int slice_grid(int64_t n, int64_t *tiles_per_block) {
  const int64_t tiles = std::max<int64_t>(1, (n + SLICE_THREADS - 1) / SLICE_THREADS);
  const int64_t slots = 148 * SLICE_BLOCKS_PER_SM;
  *tiles_per_block = (tiles + slots - 1) / slots;
  return (int)((tiles + *tiles_per_block - 1) / *tiles_per_block);
}

/* histogram of c*t with the range of binParticleCoordinate (csbend.c:3047-3113):
 * shared-memory integer counts, then added to global counts. */
static const int kHistUnroll = 4;

/* Copies of the shared-memory counts per histogram CTA: warp w adds into
 * copy w % copies, so warps of a CTA do not queue on the central bins' counters
 * (integer counts: the sum over copies is the same in any order).  As many
 * as fit 48 KB, at most B2E_HIST_COPIES.  One by default: on the 1e6-particle
 * chicane (600 bins) 1, 4 and 8 copies measured 94.1, 94.2 and 94.5 us per
 * kick (the zeroing and the final sum over copies cost what the spread
 * saves); a compile-time option for beams with sharper peaks. */
#ifndef B2E_HIST_COPIES
#define B2E_HIST_COPIES 1
#endif
static inline size_t hist_smem(int nBins) {
  const size_t one = sizeof(unsigned int) * (size_t)nBins;
  size_t copies = (48 * 1024) / one;
  copies = copies < 1 ? 1 : (copies > B2E_HIST_COPIES ? B2E_HIST_COPIES : copies);
  return copies * one;
}

/* histogram CTAs (1024 threads) per bunch: one per 1024 particles, at most one
 * per SM over all bunches (two take 1.2 us more per kick at 1e6 particles, for
 * the atomics with which each adds its counts to the bunch's) */
static inline int hist_blocks(int64_t per_bunch, int nbunch) {
  return (int)std::min<int64_t>(std::max<int64_t>(1, 148 / std::max(nbunch, 1)),
                                std::max<int64_t>(1, (per_bunch + 1023) / 1024));
}

/* launch with programmatic stream serialization (the kernel begins with
 * chain_enter) */
template <typename... KArgs, typename... Args>
static cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                  Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

__global__ void csr_hist_kernel(DevParticles P, int64_t n, CsrBunches B, unsigned int *counts_all, int nBins,
                                double factor) {
  extern __shared__ unsigned int scount[];
  chain_release();
  /* the launch gives copies x nBins counters (hist_smem) */
  unsigned int smem_bytes;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(smem_bytes));
  const int copies = (int)(smem_bytes / (sizeof(unsigned int) * nBins));
  unsigned int *mycount = scount + (size_t)((threadIdx.x >> 5) % copies) * nBins;
  for (int b = threadIdx.x; b < copies * nBins; b += blockDim.x)
    scount[b] = 0;
  __syncthreads();
  chain_wait(); /* so far only this block's shared memory */
  const int bunch = blockIdx.y;
  if (!B.active[bunch])
    return;
  CsrDevState *st = B.st + bunch;
  unsigned int *counts = counts_all + (size_t)bunch * nBins;
  const int64_t first = B.n <= 1 ? 0 : B.offs[bunch], end = B.n <= 1 ? n : B.offs[bunch + 1];
  double lower = value_of(st->ct_min_key), upper = value_of(st->ct_max_key), dct;
  expand_range(&lower, &upper, factor);
  dct = (upper - lower) / nBins;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->ctLower = lower;
    st->ctUpper = upper;
    st->dct = dct;
  }
  /* kHistUnroll particles per thread and sweep, their loads issued together
   * (the loss word and c*t are read unconditionally within the range, so
   * neither waits on the other); the loop bounds are uniform over the block */
  /* (c*t - lower)/dct through the reciprocal, rounded as the division */
  const double inv_dct = fp_recip(dct);
  const bool recip_ok = fp_within(dct, FP_HI_2M250, FP_HI_2P100);
  /* chunks of blockDim.x particles, chunk c to CTA c mod gridDim.x */
  const int64_t G = gridDim.x, D = blockDim.x;
  for (int64_t c0 = blockIdx.x; first + c0 * D < end; c0 += G * kHistUnroll) {
    int32_t lp[kHistUnroll];
    double ct[kHistUnroll];
#pragma unroll
    for (int u = 0; u < kHistUnroll; u++) {
      const int64_t i = first + (c0 + u * G) * D + threadIdx.x;
      lp[u] = i < end ? P.lost_pass[i] : 0;
      ct[u] = i < end ? P.s[i] : 0.0;
    }
    int bin[kHistUnroll];
#pragma unroll
    for (int u = 0; u < kHistUnroll; u++) {
      const double a = ct[u] - lower, q = recip_ok ? fp_quot(a, dct, inv_dct) : a / dct;
      /* the truncated quotient in [0, nBins); out of it for NaN */
      bin[u] = lp[u] < 0 && q > -1 && q < nBins ? (int)q : -1;
    }
    /* one shared-memory atomic per particle, unless neighbouring lanes share a
     * bin (a beam stored in c*t order, where a warp's particles would queue on
     * one counter; looked for in the sweep's first particles): then one atomic
     * per distinct bin */
    const int lane = threadIdx.x & 31, prev = __shfl_up_sync(0xffffffffu, bin[0], 1);
    const bool shared_bins = __any_sync(0xffffffffu, lane > 0 && bin[0] >= 0 && bin[0] == prev);
#pragma unroll
    for (int u = 0; u < kHistUnroll; u++) {
      if (shared_bins) {
        const unsigned int peers = __match_any_sync(0xffffffffu, bin[u]);
        if (bin[u] >= 0 && lane == __ffs(peers) - 1)
          atomicAdd(&mycount[bin[u]], (unsigned int)__popc(peers));
      } else if (bin[u] >= 0) {
        atomicAdd(&mycount[bin[u]], 1u);
      }
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nBins; b += blockDim.x) {
    unsigned int c = 0;
    for (int k = 0; k < copies; k++)
      c += scount[(size_t)k * nBins + b];
    if (c)
      atomicAdd(&counts[b], c);
  }
}

struct WakeArgs {
  int nBins, sgHalf, sgdHalf, trapz, steady;
  /* Savitzky-Golay weights of smoothing and derivative (sg_table) */
  const double *sg_w, *sgd_w;
  double slippage, slippage13, c1, c2, csr_constant;
  double length, nSlices;   /* element length and kicks: c1 and c2 of each bunch */
  double *wakelog;          /* nBins values per bunch for this kick, or null */
  /* page record (CSRCSBEND OUTPUT_FILE): B2E_CSR_PAGE_HEADER + 4 nBins values
   * per bunch for this kick, or null; the header's host-known fields */
  double *pagelog;
  double page_element, page_kick, page_angle, page_ds_kick, page_p_central, page_range_factor;
  /* integrated Green's function (csbend.c:2593-2621, :2676-2680) */
  int igf;
  double gamma2, gamma3, rho0, const1, q4pe, igf_factor;
  /* low/high-pass filters of the histogram (applyLHPassFilters): on when
   * HIGH_FREQUENCY_CUTOFF0 > 0 or LOW_FREQUENCY_CUTOFF0 >= 0 */
  int lh, clip;
  double startHP, endHP, startLP, endLP;
};

/* applyLHPassFilters (csbend.c:4611-4703) on hist[0..nb) in one CTA with the
 * transform of b2e_fft.h; scratch: ri = sm + nb (nb + 2 values), twiddles at
 * sm + 2 nb + 2 and sm + 3 nb + 2 (the filters' arrays are not yet in use) */
__device__ void lh_pass_filters(const WakeArgs &a, double *sm) {
  const int nb = a.nBins, freq = nb / 2 + 1;
  double *hist = sm, *ri = sm + nb, *tc = sm + 2 * nb + 2, *ts = sm + 3 * nb + 2;
  __shared__ double orig_sum;
  for (int t = threadIdx.x; t < nb; t += blockDim.x)
    b2e_dft_twiddle(nb, t, &tc[t], &ts[t]);
  __syncthreads();
  for (int k = threadIdx.x; k < freq; k += blockDim.x)
    b2e_rdft_pair(hist, nb, k, tc, ts, &ri[2 * k], &ri[2 * k + 1]);
  __syncthreads();
  if (threadIdx.x == 0) {
    b2e_lh_ramps(ri, freq, a.startHP, a.endHP, a.startLP, a.endLP);
    double sum = 0;
    for (int b = 0; b < nb; b++)
      sum += hist[b];
    orig_sum = sum;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < nb; j += blockDim.x)
    hist[j] = b2e_rdft_sample(ri, nb, j, tc, ts);
  __syncthreads();
  if (a.clip) {
    /* correctDistribution (csbend.c:4705-4721) to the unfiltered sum */
    __shared__ double factor;
    __shared__ int skip;
    if (threadIdx.x == 0) {
      double sum = 0;
      for (int b = 0; b < nb; b++) {
        if (hist[b] < 0)
          hist[b] = 0;
        sum += hist[b];
      }
      skip = !sum;
      factor = skip ? 1 : orig_sum / sum;
    }
    __syncthreads();
    if (!skip)
      for (int b = threadIdx.x; b < nb; b += blockDim.x)
        hist[b] = hist[b] * factor;
    __syncthreads();
  }
}

/* Savitzky-Golay weights of a filter over nb bins.  The window of bin b is
 * width = min(2 half + 1, nb) bins from start = clamp(b - half, 0, nb - width)
 * (b2e_sg_window), and its weights depend on b - start only: [row][width], row =
 * b - start, width rows. */
B2E_SG_FN int sg_width(int half, int nb) { return half <= 0 ? 1 : (2 * half + 1 < nb ? 2 * half + 1 : nb); }
B2E_SG_FN void sg_row(int half, int order, int deriv, int nb, int row, double *w) {
  const long width = sg_width(half, nb), ord = order < width - 1 ? order : width - 1;
  double t[B2E_SG_MAX_WIDTH];
  /* no window: the bin itself; the derivative of a constant fit is zero */
  if (half <= 0 && deriv == 0)
    w[0] = 1;
  else if (deriv > ord || b2e_sg_weights(t, width, -(long)row, ord, deriv))
    for (int k = 0; k < width; k++)
      w[k] = 0;
  else
    for (int k = 0; k < width; k++)
      w[k] = t[k];
}

template <bool CLIP = false>
__device__ __forceinline__ void sg_apply(const double *in, double *out, int nb, int half, const double *w) {
  const int width = sg_width(half, nb);
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const int start = half <= 0 ? b : min(max(b - half, 0), nb - width);
    const double *wb = w + (b - start) * width;
    double s = 0;
    for (int k0 = 0; k0 < width; k0 += 8) {
      double term[8];
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (k0 + k < width)
          term[k] = wb[k0 + k] * in[start + k0 + k];
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (k0 + k < width)
          s += term[k];
    }
    out[b] = CLIP && s < 0 ? 0 : s;
  }
}

/* ((v[0] + v[1]) + v[2]) + ... in index order, as a serial loop forms it, eight
 * values loading while eight are added: 10.6 cycles a value measured (600 bins),
 * 8.4 being the latency of a dependent addition */
__device__ __forceinline__ double ordered_sum(const double *v, int n) {
  double s = 0, r[8], q[8];
  auto load = [&](double(&to)[8], int from) {
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (from + k < n)
        to[k] = v[from + k];
  };
  auto add = [&](const double(&of)[8]) {
#pragma unroll
    for (int k = 0; k < 8; k++)
      s += of[k];
  };
  int b = 0;
  load(r, 0);
  for (; b + 24 <= n; b += 16) {
#pragma unroll
    for (int k = 0; k < 8; k++)
      q[k] = v[b + 8 + k];
    add(r);
#pragma unroll
    for (int k = 0; k < 8; k++)
      r[k] = v[b + 16 + k];
    add(q);
  }
  /* r holds v[b...b + 7] as far as they go; at most 23 are left */
  for (; b < n; b += 8) {
    load(q, b + 8);
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (b + k < n)
        s += r[k];
#pragma unroll
    for (int k = 0; k < 8; k++)
      r[k] = q[k];
  }
  return s;
}

/* weights up to this many per table are staged in shared memory (windows of 17) */
constexpr int SG_STAGE = 17 * 17;

/* both tables into stage, which a then points to; wider ones stay where they
 * are.  The tables are older than any kernel in flight: a chained kernel stages
 * them before it waits for its predecessor. */
__device__ __forceinline__ void stage_weights(WakeArgs &a, double (&stage)[2][SG_STAGE]) {
  const int w0 = sg_width(a.sgHalf, a.nBins), w1 = sg_width(a.sgdHalf, a.nBins);
  if (w0 * w0 > SG_STAGE || w1 * w1 > SG_STAGE)
    return;
  for (int k = threadIdx.x; k < w0 * w0; k += blockDim.x)
    stage[0][k] = a.sg_w[k];
  for (int k = threadIdx.x; k < w1 * w1; k += blockDim.x)
    stage[1][k] = a.sgd_w[k];
  a.sg_w = stage[0];
  a.sgd_w = stage[1];
}

/* Filters of one kick's wake (csbend.c:2566-2591) on one CTA: Savitzky-Golay
 * smoothing of the counts, correctDistribution, density per unit ct, its
 * derivative filter and the (dct*b)^(1/3) denominators.  Leaves hist = sm,
 * deriv = sm + nBins, denom = sm + 2 nBins (tmp = sm + 3 nBins is scratch) and,
 * with INVERSE, 1/denom at sm + 4 nBins + 8; returns whether the quotients
 * deriv/denom may be formed with them (fp_quot): every value plain.  `first` is
 * this thread's first count, loaded ahead. */
template <typename CountT, typename SumT, bool INVERSE = false>
__device__ bool wake_filters(const CountT *counts, CountT first, const WakeArgs &a, const double dct, double *sm,
                             SumT *nbinned_out) {
  constexpr bool EXACT = std::is_integral<SumT>::value;
  const int nb = a.nBins, warps = blockDim.x >> 5;
  double *inv = sm + 4 * nb + 8;
  double *hist = sm, *deriv = sm + nb, *denom = sm + 2 * nb, *tmp = sm + 3 * nb;
  __shared__ double nBinnedD, smoothed_sum;
  __shared__ SumT warp_sums[32];
  const bool plain_dct = fp_within(dct, FP_HI_2M250, FP_HI_2P100);
  const double inv_dct = fp_recip(dct);
  /* the total of the counts: integers in any order (per thread, warp shuffles,
   * then the last warp), real values in bin order as the reference's loop; it is
   * needed from the second barrier on, so it forms beside the work in between */
  SumT part = 0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const CountT v = b == threadIdx.x ? first : counts[b];
    hist[b] = (double)v;
    if (EXACT)
      part += v;
  }
  if (EXACT) {
    for (int o = 16; o > 0; o >>= 1)
      part += __shfl_down_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0)
      warp_sums[threadIdx.x >> 5] = part;
  }
  __syncthreads();
  if (EXACT) {
    if ((int)(threadIdx.x >> 5) == warps - 1) {
      const int lane = threadIdx.x & 31;
      SumT total = lane < warps ? warp_sums[lane] : 0;
      for (int o = 16; o > 0; o >>= 1)
        total += __shfl_down_sync(0xffffffffu, total, o);
      if (lane == 0) {
        nBinnedD = 1.0 * total;
        if (nbinned_out)
          *nbinned_out = total;
      }
    }
  } else if (a.lh) {
    if (threadIdx.x == 0)
      nBinnedD = ordered_sum(hist, nb);
    __syncthreads();
  }
  if (a.lh)
    lh_pass_filters(a, sm);
  if (a.sgHalf > 0) {
    /* correctDistribution (csbend.c:4705-4721): negative bins clipped as the
     * smoothing writes them, then the sum in bin order, as the reference forms
     * it */
    sg_apply<true>(hist, tmp, nb, a.sgHalf, a.sg_w);
    __syncthreads();
    /* thread 0 runs the serial sum, for real counts thread 32 that of the
     * counts, and other warps form the denominators: not those of the first
     * sub-partition (every fourth), whose FP64 pipe the sum waits for, 11.7
     * cycles an addition with them there */
    const int warp = threadIdx.x >> 5;
    const bool helps = EXACT ? (warp & 3) != 0 : warp >= 2;
    const int rank = EXACT ? warp - (warp >> 2) - 1 : warp - 2, helpers = EXACT ? warps - (warps + 3) / 4 : warps - 2;
    if (threadIdx.x == 0)
      smoothed_sum = ordered_sum(tmp, nb);
    else if (!EXACT && !a.lh && threadIdx.x == 32)
      nBinnedD = ordered_sum(hist, nb);
    else if (helps)
      for (int b = rank * 32 + (threadIdx.x & 31); b < nb; b += helpers * 32) {
        const double v = b2e_pow13(dct * b);
        denom[b] = v;
        if (INVERSE)
          inv[b] = fp_recip(v);
      }
    __syncthreads();
  }
  const double sum = a.sgHalf > 0 ? smoothed_sum : 0, factor = a.sgHalf > 0 ? nBinnedD / sum : 0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    if (a.sgHalf <= 0) {
      denom[b] = b2e_pow13(dct * b);
      if (INVERSE)
        inv[b] = fp_recip(denom[b]);
    }
    const double h = a.sgHalf > 0 ? (sum == 0 ? tmp[b] : tmp[b] * factor) : hist[b];
    hist[b] = plain_dct && fp_plain(h, FP_HI_2P700) ? fp_quot(h, dct, inv_dct) : divide_ieee(h, dct);
  }
  __syncthreads();
  sg_apply(hist, deriv, nb, a.sgdHalf, a.sgd_w);
  if (!INVERSE) {
    __syncthreads();
    return false;
  }
  /* each thread checks the values it wrote */
  bool plain = fp_within(dct, FP_HI_2M250, FP_HI_2P100);
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    plain = plain && fp_plain(deriv[b], FP_HI_2P700);
  return __syncthreads_and(plain);
}

/* bins of slippage; clamped to [0, nb] so indexing stays in bounds for a
 * degenerate bin size (the comparisons below give the same result) */
__device__ __forceinline__ void slippage_bins(const WakeArgs &a, double dct, long long *diS, long long *diS4) {
  long long d = (long long)(a.slippage / dct), d4 = (long long)(4 * a.slippage / dct);
  *diS = d < 0 ? 0 : (d > a.nBins ? a.nBins : d);
  *diS4 = d4 < 0 ? 0 : (d4 > a.nBins ? a.nBins : d4);
}

/* T1 (integral) and T2 (slippage boundary) of bin ib before the c1/c2 factors
 * (csbend.c:2623-2662) */
__device__ __forceinline__ void wake_terms(int ib, const WakeArgs &a, const double dct, const double *hist,
                                           const double *deriv, const double *denom, long long diS, long long diS4,
                                           double *T1out, double *T2out) {
  const int nb = a.nBins;
  double T1 = 0, T2 = 0, term1 = 0, term2 = 0;
  long long count, j;
  if (a.steady) {
    if (!a.trapz) {
      for (j = ib + 1; j < nb; j++)
        T1 += deriv[j] / denom[j - ib];
    } else {
      if ((j = ib + 1) < nb)
        term1 = deriv[j] / denom[j - ib];
      for (count = 0, j = ib + 1; j < nb; j++, count++)
        T1 += (term2 = deriv[j] / denom[j - ib]);
      if ((ib + 1) < nb)
        T1 += 0.3 * (denom[1] * denom[1]) * (2 * deriv[ib + 1] + 3 * deriv[ib]) / dct;
      if (count > 1)
        T1 -= (term1 + term2) / 2;
    }
  } else {
    if (!a.trapz) {
      for (j = ib + 1; j <= (ib + diS) && j < nb; j++)
        T1 += deriv[j] / denom[j - ib];
    } else {
      if ((j = ib + 1) < nb && j <= (ib + diS))
        term1 = deriv[j] / denom[j - ib] / 2;
      for (count = 0, j = ib + 1; j <= (ib + diS) && j < nb; count++, j++)
        T1 += (term2 = deriv[j] / denom[j - ib]);
      if (diS > 0 && (ib + 1) < nb)
        T1 += 0.3 * (denom[1] * denom[1]) * (2 * deriv[ib + 1] + 3 * deriv[ib]) / dct;
      if (count > 1)
        T1 -= (term1 + term2) / 2;
    }
    if ((ib + diS) < nb)
      T2 += hist[ib + diS];
    if ((ib + diS4) < nb)
      T2 -= hist[ib + diS4];
  }
  *T1out = T1;
  *T2out = T2;
}

/* The same for the bins ib = first + m*stride, m < NI, of one thread, with the
 * quotients deriv/denom through the stored reciprocals (three operations each)
 * and each (denom, 1/denom) pair read once for all NI bins.  Every sum is in
 * wake_terms' order; the steady and the transient integral differ in the
 * length of the sum and in the halved first term. */
template <int NI>
__device__ void wake_terms_inverse(int first, int stride, const WakeArgs &a, const double dct, const double *hist,
                                   const double *deriv, const double *denom, const double *inv, long long diS,
                                   long long diS4, double *T1, double *T2) {
  const int nb = a.nBins;
  int len[NI]; /* terms of each sum; nonincreasing in m */
  double last[NI];
#pragma unroll
  for (int m = 0; m < NI; m++) {
    const int ib = first + m * stride;
    const long long room = nb - 1 - ib;
    len[m] = ib < nb ? (int)(a.steady || room < diS ? room : diS) : 0;
    T1[m] = T2[m] = last[m] = 0;
  }
  int k = 1;
#pragma unroll
  for (int live = NI; live > 0; live--)
    for (; k <= len[live - 1]; k++) {
      const double b = denom[k], y = inv[k];
#pragma unroll
      for (int m = 0; m < live; m++) {
        last[m] = fp_quot(deriv[first + m * stride + k], b, y);
        T1[m] += last[m];
      }
    }
#pragma unroll
  for (int m = 0; m < NI; m++) {
    const int ib = first + m * stride;
    if (ib >= nb)
      continue;
    if (a.trapz) {
      if ((a.steady || diS > 0) && ib + 1 < nb)
        T1[m] += 0.3 * (denom[1] * denom[1]) * (2 * deriv[ib + 1] + 3 * deriv[ib]) / dct;
      if (len[m] > 1) {
        const double t = fp_quot(deriv[ib + 1], denom[1], inv[1]);
        T1[m] -= ((a.steady ? t : t / 2) + last[m]) / 2;
      }
    }
    if (!a.steady) {
      if (ib + diS < nb)
        T2[m] += hist[ib + diS];
      if (ib + diS4 < nb)
        T2[m] -= hist[ib + diS4];
    }
  }
}

/* Steady-state wake by the integrated Green's function (csbend.c:2593-2621,
 * :2676-2680, convolveArrays1 :5484-5491): chi(z) per bin, its second
 * difference, the one-sided convolution with the density (per-bin serial
 * sums in the reference's order), times -q_macro/(m c^2) L/N_KICKS.  chik and
 * grnk are nBins scratch arrays in shared memory. */
__device__ void igf_wake(const WakeArgs &a, const double dct, const double *hist, double *chik, double *grnk,
                         double *dgamma) {
  const int nb = a.nBins;
  const double frac = 9.0 / 16.0;
  for (int ib = threadIdx.x; ib < nb; ib += blockDim.x) {
    const double z = ib * dct;
    const double xmu = 3.0 * a.gamma3 * z / (2.0 * a.rho0);
    const double aa = sqrt(xmu * xmu + 1.0);
    const double b = aa + xmu;
    double chi;
    if (xmu < 1e-3) {
      const double x2 = xmu * xmu, x3 = xmu * xmu * xmu;
      chi = frac * a.const1 + 0.50 * x2 - (7.0 / 54.0) * (x2 * x2) + (140.0 / 2187.0) * (x3 * x3);
    } else {
      const double b13 = b2e_pow13(b), b23 = b2e_pow23(b), b43 = b2e_pow43(b);
      const double q = (1 - b23) / xmu;
      chi = frac * (3.0 * (-2.0 * xmu * b13 + b23 + b43) + b2e_log((q * q) / (1 + b23 + b43)));
    }
    chik[ib] = chi;
  }
  __syncthreads();
  const double const2 = (16.0 / 27.0) * a.q4pe / (a.gamma2 * dct);
  for (int ib = threadIdx.x; ib < nb; ib += blockDim.x) {
    double g;
    if (ib == 0)
      g = const2 * (chik[1] - chik[0]);
    else if (ib < nb - 1)
      g = const2 * (chik[ib + 1] - 2.0 * chik[ib] + chik[ib - 1]);
    else
      g = 0;
    grnk[ib] = g;
  }
  __syncthreads();
  for (int ib = threadIdx.x; ib < nb; ib += blockDim.x) {
    double out = 0;
    for (int ib1 = ib; ib1 < nb; ib1++)
      out += hist[ib1] * grnk[ib1 - ib];
    const double dg = out * a.igf_factor;
    dgamma[ib] = dg;
    if (a.wakelog)
      a.wakelog[ib] = dg;
  }
}

/* Wake of one kick (csbend.c:2566-2673) on one CTA, from a histogram of
 * counts (unsigned counts in tracking, real-valued counts for batched
 * profiles).  sm holds 5*nBins + 8 doubles.  NI: bins a thread takes at a time.  Writes dgamma[nBins], the wake log
 * when a.wakelog is set, the binned total when nbinned_out is set, and the
 * smoothed density (per unit ct) and its derivative when hist_out/deriv_out
 * are set. */
template <typename CountT, typename SumT, int NI>
__device__ void wake_body(const CountT *counts, CountT first, const WakeArgs &a, const double dct, double *sm,
                          double *dgamma, SumT *nbinned_out, double *hist_out, double *deriv_out,
                          double *page = nullptr) {
  const int nb = a.nBins;
  const bool inverse = wake_filters<CountT, SumT, true>(counts, first, a, dct, sm, nbinned_out);
  const double *hist = sm, *deriv = sm + nb, *denom = sm + 2 * nb, *inv = sm + 4 * nb + 8;
  double *page_t1 = page ? page + 2 * nb : nullptr, *page_t2 = page ? page + 3 * nb : nullptr;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    if (hist_out)
      hist_out[b] = hist[b];
    if (deriv_out)
      deriv_out[b] = deriv[b];
    if (page) {
      page[b] = hist[b];
      page[nb + b] = deriv[b];
      page_t1[b] = 0; /* the IGF path and an empty range leave T1 and T2 at zero */
      page_t2[b] = 0;
    }
  }
  long long diS, diS4;
  slippage_bins(a, dct, &diS, &diS4);
  if (!(dct > 0)) {
    for (int ib = threadIdx.x; ib < nb; ib += blockDim.x) {
      dgamma[ib] = 0;
      if (a.wakelog)
        a.wakelog[ib] = 0;
    }
    return;
  }
  if (a.igf) {
    igf_wake(a, dct, hist, sm + 3 * nb, sm + 2 * nb, dgamma);
    return;
  }
  for (int i0 = threadIdx.x; i0 < nb; i0 += NI * blockDim.x) {
    double T1[NI], T2[NI];
    if (inverse && a.csr_constant)
      wake_terms_inverse<NI>(i0, blockDim.x, a, dct, hist, deriv, denom, inv, diS, diS4, T1, T2);
#pragma unroll
    for (int m = 0; m < NI; m++) {
      const int ib = i0 + m * blockDim.x;
      if (ib >= nb)
        break;
      if (!a.csr_constant)
        T1[m] = T2[m] = 0;
      else {
        if (!inverse)
          wake_terms(ib, a, dct, hist, deriv, denom, diS, diS4, &T1[m], &T2[m]);
        T1[m] *= a.c1;
        T2[m] *= a.c2;
      }
      const double dg = T1[m] + T2[m];
      dgamma[ib] = dg;
      if (a.wakelog)
        a.wakelog[ib] = dg;
      if (page) {
        page_t1[ib] = T1[m];
        page_t2[ib] = T2[m];
      }
    }
  }
}

/* threads of a wake CTA: one per bin in the warps that form the denominators
 * beside the serial sum, three of four */
static inline int wake_threads(int bins) {
  const int need = std::max(1, (bins + 31) / 32);
  return std::min(1024, 32 * (need + (need + 2) / 3));
}

/* wake of one kick, one CTA per bunch; c1 and c2 from the bunch's CSRConstant
 * in the host expression's order (csbend.c:2664-2667).  With recycle set the
 * CTA also readies its bunch for the next binning pass once this one's inputs
 * are consumed: empty c*t range keys (the histogram kernel, the only reader,
 * has finished) and zero counts (after they are read into shared memory). */
__global__ void __launch_bounds__(1024, 1) csr_wake_kernel(CsrBunches B, unsigned int *counts_all, WakeArgs a,
                                                           int recycle) {
  extern __shared__ double sm[];
  __shared__ double stage[2][SG_STAGE];
  chain_release();
  stage_weights(a, stage);
  chain_wait();
  const int bunch = blockIdx.x;
  /* the bunch's scalars and the first counts load together with its active
   * flag (all in bounds) */
  const int active = B.active[bunch];
  unsigned int *counts = counts_all + (size_t)bunch * a.nBins;
  const unsigned int first = threadIdx.x < a.nBins ? counts[threadIdx.x] : 0;
  const double csr_constant = B.csr_const[bunch], igf_factor = B.csr_const[B.n + bunch];
  CsrDevState *st = B.st + bunch;
  const double dct = st->dct;
  double *page = nullptr;
  if (a.pagelog) {
    page = a.pagelog + (size_t)bunch * (B2E_CSR_PAGE_HEADER + 4 * a.nBins);
    if (threadIdx.x == 0) {
      /* the binning's range, as the histogram kernel formed it; a bunch
       * without CSR on this kick gets element index -1 and no arrays */
      double lower = value_of(st->ct_min_key), upper = value_of(st->ct_max_key);
      expand_range(&lower, &upper, a.page_range_factor);
      page[0] = active ? a.page_element : -1.0;
      page[1] = a.page_kick;
      page[2] = bunch;
      page[3] = a.nBins;
      page[4] = lower;
      page[5] = upper;
      page[6] = dct;
      page[7] = a.slippage;
      page[8] = a.page_angle;
      page[9] = a.page_ds_kick;
      page[10] = a.page_p_central;
      page[11] = B.csr_const[3 * B.n + bunch];
    }
    __syncthreads(); /* the keys are read before they are emptied below */
    page += B2E_CSR_PAGE_HEADER;
  }
  if (recycle && threadIdx.x == 0) {
    st->ct_min_key = ~0ull;
    st->ct_max_key = 0ull;
  }
  if (!active) {
    /* a bunch of a train without a wake on this kick: zeros in the log */
    if (a.wakelog)
      for (int b = threadIdx.x; b < a.nBins; b += blockDim.x)
        a.wakelog[(size_t)bunch * a.nBins + b] = 0;
    return;
  }
  WakeArgs w = a;
  w.csr_constant = csr_constant;
  w.c1 = csr_constant * a.length / a.nSlices;
  w.c2 = -csr_constant * a.length / a.nSlices / a.slippage13;
  w.igf_factor = igf_factor;
  w.wakelog = a.wakelog ? a.wakelog + (size_t)bunch * a.nBins : nullptr;
  wake_body<unsigned int, long long, 1>(counts, first, w, dct, sm, st->dGamma, &st->nBinned, nullptr, nullptr, page);
  if (recycle) /* the counts were copied to shared memory before the first barrier */
    for (int b = threadIdx.x; b < a.nBins; b += blockDim.x)
      counts[b] = 0;
}

/* deterministic sum over the CTA (blockDim.x a power of two, red >= blockDim.x doubles) */
__device__ double block_sum(double v, double *red) {
  red[threadIdx.x] = v;
  __syncthreads();
  for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s)
      red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  const double r = red[0];
  __syncthreads();
  return r;
}

/* Learned wake, step 1 (one CTA per bunch): the kick's filters, then the
 * network inputs in bin units -- density and derivative normalised to unit
 * sum and by k = 1/rms(derivative) over the network's L bins, the slippage
 * code log2(diS)/log2(L), and the density at bin i + diS -- padded with zeros
 * to L bins.  The tables (density, derivative, denominators) and the
 * per-bunch scalars (sum, k, dct) are kept for step 3. */
__global__ void __launch_bounds__(1024, 1) csr_sur_filter_kernel(CsrBunches B, const unsigned int *counts_all, WakeArgs a, int L, float sc_dens,
                                      float sc_deriv, double *tab, double *scal, float *inputs) {
  extern __shared__ double sm[];
  __shared__ double stage[2][SG_STAGE];
  stage_weights(a, stage);
  const int b = blockIdx.x, nb = a.nBins;
  float *in = inputs + (size_t)b * 4 * L;
  if (!B.active[b]) {
    for (int i = threadIdx.x; i < 4 * L; i += blockDim.x)
      in[i] = 0.f;
    return;
  }
  CsrDevState *st = B.st + b;
  const double dct = st->dct;
  const unsigned int *counts = counts_all + (size_t)b * nb;
  wake_filters<unsigned int, long long>(counts, threadIdx.x < nb ? counts[threadIdx.x] : 0, a, dct, sm, &st->nBinned);
  const double *hist = sm, *deriv = sm + nb, *denom = sm + 2 * nb;
  double *red = sm + 3 * nb;
  double *t = tab + (size_t)b * 3 * B2E_CSR_MAX_BINS;
  double part = 0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    t[i] = hist[i];
    t[B2E_CSR_MAX_BINS + i] = deriv[i];
    t[2 * B2E_CSR_MAX_BINS + i] = denom[i];
    part += hist[i] * dct;
  }
  const double total = block_sum(part, red);
  part = 0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    const double d = deriv[i] * dct / total;
    part += d * d;
  }
  const double k = 1.0 / sqrt(block_sum(part, red) / L);
  long long diS, diS4;
  slippage_bins(a, dct, &diS, &diS4);
  const float code = (float)(log2((double)(diS < 1 ? 1 : (diS > L ? L : diS))) / log2((double)L));
  const double fd = k / total * sc_dens, fg = k / total * sc_deriv;
  const int dsh = (int)(diS < 1 ? 1 : diS);
  for (int i = threadIdx.x; i < L; i += blockDim.x) {
    in[i] = i < nb ? (float)(hist[i] * dct * fd) : 0.f;
    in[L + i] = i < nb ? (float)(deriv[i] * dct * fg) : 0.f;
    in[2 * L + i] = code;
    in[3 * L + i] = i + dsh < nb ? (float)(hist[i + dsh] * dct * fd) : 0.f;
  }
  if (threadIdx.x == 0) {
    scal[b * 4 + 0] = total;
    scal[b * 4 + 1] = k;
    scal[b * 4 + 2] = dct;
  }
}

/* Learned wake, step 3 (one CTA per bunch): the network's T1 (bin units) to
 * the kick's T1 (times dct^(-4/3)), the gate -- the plain T1 and T2 at every
 * stride-th bin from `start`, relative rms error of the wake c1 T1 + c2 T2
 * there -- and the kick's dGamma: the learned T1 with the exact T2, or, when
 * the error exceeds tol, the plain wake exactly as csr_wake_kernel forms it. */
__global__ void __launch_bounds__(1024, 1) csr_sur_combine_kernel(CsrBunches B, WakeArgs a, const double *tab, const double *scal, const float *y,
                                       int L, float sc_target, double tol, int stride, int start, double *gate_log,
                                       unsigned long long *counters) {
  extern __shared__ double sm[];
  const int b = blockIdx.x, nb = a.nBins;
  if (!B.active[b]) {
    if (a.wakelog)
      for (int i = threadIdx.x; i < nb; i += blockDim.x)
        a.wakelog[(size_t)b * nb + i] = 0;
    if (threadIdx.x == 0)
      gate_log[b] = 0;
    return;
  }
  CsrDevState *st = B.st + b;
  double *hist = sm, *deriv = sm + nb, *denom = sm + 2 * nb, *red = sm + 3 * nb;
  const double *t = tab + (size_t)b * 3 * B2E_CSR_MAX_BINS;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    hist[i] = t[i];
    deriv[i] = t[B2E_CSR_MAX_BINS + i];
    denom[i] = t[2 * B2E_CSR_MAX_BINS + i];
  }
  __syncthreads();
  const double csr_constant = B.csr_const[b];
  const double c1 = csr_constant * a.length / a.nSlices;
  const double c2 = -csr_constant * a.length / a.nSlices / a.slippage13;
  const double total = scal[b * 4 + 0], k = scal[b * 4 + 1], dct = scal[b * 4 + 2];
  double *wl = a.wakelog ? a.wakelog + (size_t)b * nb : nullptr;
  if (!(dct > 0) || !csr_constant) {
    for (int ib = threadIdx.x; ib < nb; ib += blockDim.x) {
      st->dGamma[ib] = 0;
      if (wl)
        wl[ib] = 0;
    }
    if (threadIdx.x == 0)
      gate_log[b] = 0;
    return;
  }
  long long diS, diS4;
  slippage_bins(a, dct, &diS, &diS4);
  const double unit = 1.0 / dct / b2e_pow13(dct); /* dct^(-4/3) */
  const float *yb = y + (size_t)b * L;
  /* gate */
  double e2 = 0, w2 = 0;
  if (diS > 0)
    for (int ib = start + threadIdx.x * stride; ib < nb; ib += blockDim.x * stride) {
      double T1p, T2;
      wake_terms(ib, a, dct, hist, deriv, denom, diS, diS4, &T1p, &T2);
      const double T1s = (double)yb[ib] / sc_target / k * total * unit;
      const double d = (T1s - T1p) * c1, wp = T1p * c1 + T2 * c2;
      e2 += d * d;
      w2 += wp * wp;
    }
  e2 = block_sum(e2, red);
  w2 = block_sum(w2, red);
  const double err = diS > 0 ? (w2 > 0 ? sqrt(e2 / w2) : (e2 > 0 ? INFINITY : 0.0)) : 0.0;
  const bool plain = !(err <= tol);
  for (int ib = threadIdx.x; ib < nb; ib += blockDim.x) {
    double T1, T2;
    if (plain) {
      wake_terms(ib, a, dct, hist, deriv, denom, diS, diS4, &T1, &T2);
    } else {
      T1 = diS > 0 ? (double)yb[ib] / sc_target / k * total * unit : 0.0;
      T2 = 0;
      if ((ib + diS) < nb)
        T2 += hist[ib + diS];
      if ((ib + diS4) < nb)
        T2 -= hist[ib + diS4];
    }
    T1 *= c1;
    T2 *= c2;
    const double dg = T1 + T2;
    st->dGamma[ib] = dg;
    if (wl)
      wl[ib] = dg;
  }
  if (threadIdx.x == 0) {
    gate_log[b] = err;
    atomicAdd(&counters[0], 1ull);
    if (plain)
      atomicAdd(&counters[1], 1ull);
  }
}

/* Batched wake integral of many profiles in bin units (dct = 1), one CTA per
 * profile: out = T1 (c1 = 1, no T2 term) for the profile's slippage in bins;
 * hist_out/deriv_out receive the smoothed density and its derivative.  The
 * filters' weights come as an argument (windows up to 17 bins: no table to
 * allocate and fill per call) or, for wider windows, from a.sg_w.
 * 256 threads with four bins each: the integral's 0.3 million terms per
 * 1,024-bin profile are bound by the FP64 pipe (four operations a term), with
 * 2.5 shared-memory words read per term instead of two per division. */
constexpr int BATCH_THREADS = 256, BATCH_BINS = 4;
struct SgTables {
  double w[2][SG_STAGE];
};
__global__ void __launch_bounds__(BATCH_THREADS, 3)
    wake_batch_kernel(const double *counts, const double *slippage_bins, WakeArgs a, const __grid_constant__ SgTables sg,
                      double *t1_out, double *hist_out, double *deriv_out) {
  extern __shared__ double sm[];
  const size_t off = (size_t)blockIdx.x * a.nBins;
  WakeArgs w = a;
  if (!w.sg_w) {
    w.sg_w = sg.w[0];
    w.sgd_w = sg.w[1];
  }
  __shared__ double stage[2][SG_STAGE];
  stage_weights(w, stage);
  w.slippage = slippage_bins[blockIdx.x];
  w.slippage13 = 1;
  w.c1 = 1;
  w.c2 = 0;
  w.csr_constant = 1;
  w.wakelog = nullptr;
  wake_body<double, double, BATCH_BINS>(counts + off, threadIdx.x < a.nBins ? counts[off + threadIdx.x] : 0, w, 1.0, sm,
                                        t1_out + off, (double *)nullptr, hist_out + off, deriv_out + off);
}

/* Blocks of the kernels that collect ranges, and the run of particles each
 * takes: an equal share of the whole 256-particle tiles, one tile per block
 * while eight blocks per SM hold them all.  A million particles send 15,632
 * atomics to the bunch's two words instead of the 62,500 of one tile per block:
 * chicane of 1e6 particles 5.80 ms against 5.87, a train of five bunches 17.72
 * against 17.99 ms. */
struct Sweep {
  int grid;
  int64_t share;
};
static Sweep sweep_of(int64_t n) {
  const int64_t tiles = std::max<int64_t>(1, (n + 255) / 256);
  Sweep w;
  w.share = (tiles + 148 * 8 - 1) / (148 * 8) * 256;
  w.grid = (int)((n + w.share - 1) / w.share);
  if (w.grid < 1)
    w.grid = 1;
  return w;
}

/* after the last kick: its wake kick and the min/max for the exit binning */
__global__ void csr_last_kick_kernel(DevParticles P, int64_t n, int64_t share, CsrBunches B, int nBins, double Po,
                                     double rho0) {
  chain_enter();
  const int64_t first = blockIdx.x * share, end = min(n, first + share);
  BunchRange range(first < n ? bunch_of(first, B) : 0);
  for (int64_t i = first + threadIdx.x; i - threadIdx.x < end; i += blockDim.x) {
    const bool alive = i < n && P.lost_pass[i] < 0;
    const int b = i < n ? bunch_of(i, B) : B.n - 1;
    double CT = 0;
    if (alive) {
      CT = P.s[i];
      if (B.active[b] && B.csr_const[b] != 0)
        P.dp[i] = csr_kick(CT, P.x[i], P.dp[i], B.st + b, nBins, Po, rho0);
    }
    range.add(CT, alive, b, B);
  }
  range.flush(B);
}

/* exit: c*t -> s at the final velocity, exit edge, back to the lab frame
 * (csbend.c:2810-2955); csrWake.s0 from the exit binning's lower edge. */
__global__ void csr_exit_kernel(DevParticles P, int64_t n, const DevElem *ep, BendExtra bx, CsrBunches B, double factor,
                                double Po,
                                int pass, int elem_index) {
  chain_enter();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const DevElem &e = *ep;
  const double *c = e.c;
  if (blockIdx.x == 0)
    for (int b = threadIdx.x; b < B.n; b += blockDim.x) {
      CsrDevState *st = B.st + b;
      const int do_bin = B.active[b];
      double lower = 0, upper = 0;
      st->dctBin = do_bin ? st->dct : 0;
      if (do_bin) {
        lower = value_of(st->ct_min_key);
        upper = value_of(st->ct_max_key);
        expand_range(&lower, &upper, factor);
      }
      st->s0 = lower + c[CB_DZF];
    }
  if (i >= n || P.lost_pass[i] >= 0)
    return;
  const double ct = c[CB_COS_TT], sn = c[CB_SIN_TT];
  double X = P.x[i], XP = P.xp[i], Y = P.y[i], YP = P.yp[i], CT = P.s[i], DP = P.dp[i];
  double p1 = Po * (1 + DP), beta1 = p1 / sqrt(p1 * p1 + 1), s, x, y, xp, yp, rho;
  s = CT * beta1;
  if (p1 <= 0) {
    P.lost_pass[i] = pass;
    P.lost_elem[i] = elem_index;
    return;
  }
  if (e.flags & EF_EDGE2) {
    rho = (1 + DP) * c[CB_RHO_ACTUAL];
    if (e.flags & EF_EDGE_ORDER2) {
      bend_edge_order2(X, XP, Y, YP, rho, c[CB_PSI2] * (1 + DP), c[CB_TAN_E2], c[CB_E2], bx.c[BX_SEC2_E2],
                       bx.c[BX_EDGE_N], 1);
    } else {
      XP = XP + (c[CB_TAN_E2] / rho) * X;
      YP = YP - (b2e_tan(c[CB_E2] - c[CB_PSI2] / (1 + DP)) / rho) * Y;
    }
  }
  /* the ETILT offsets are zero without ETILT */
  x = (X * ct - Y * sn) + bx.c[BX_ETILT0];
  y = (X * sn + Y * ct) + bx.c[BX_ETILT0 + 2];
  xp = (XP * ct - YP * sn) + bx.c[BX_ETILT0 + 1];
  yp = (XP * sn + YP * ct) + bx.c[BX_ETILT0 + 3];
  x = x + (c[CB_DXF] + c[CB_DZF] * xp);
  y = y + (c[CB_DYF] + c[CB_DZF] * yp);
  s = s + (c[CB_DZF] * sqrt((1 + xp * xp) + yp * yp) + bx.c[BX_ETILT0 + 4]);
  P.x[i] = x;
  P.xp[i] = xp;
  P.y[i] = y;
  P.yp[i] = yp;
  P.s[i] = s;
}

/* exact drift of particle i */
__device__ __forceinline__ void exact_drift(const DevParticles &P, int64_t i, double L) {
  const double xp = P.xp[i], yp = P.yp[i];
  P.x[i] = P.x[i] + xp * L;
  P.y[i] = P.y[i] + yp * L;
  P.s[i] = P.s[i] + L * sqrt((1 + xp * xp) + yp * yp);
}

/* The particles of a CSRDRIFT's bunches without a wake (csbend.c:3196-3212):
 * its first kick kernel takes them through the whole length, so that no pass of
 * its own asks every particle for its bunch's mode */
struct PlainDrift {
  double length;
  int now; /* the first kick */
};

/* CSRDRIFT mode 0, one kick (csbend.c:3415-3502) */
__global__ void csr_drift_kick_kernel(DevParticles P, int64_t n, CsrBunches B, PlainDrift plain, double dz,
                                      double s0_incr, double factor, int apply, int nBins, double Po) {
  chain_enter();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || P.lost_pass[i] >= 0)
    return;
  const int b = bunch_of(i, B);
  if (!B.mode[b]) {
    if (plain.now)
      exact_drift(P, i, plain.length);
    return;
  }
  const CsrDevState *st = B.st + b;
  double x = P.x[i], xp = P.xp[i], y = P.y[i], yp = P.yp[i], s = P.s[i], dp = P.dp[i], p, beta;
  x = x + xp * dz;
  y = y + yp * dz;
  p = Po * (1 + dp);
  beta = p / sqrt(p * p + 1);
  s = (s + dz * sqrt((1 + xp * xp) + yp * yp)) / beta;
  if (apply) {
    const double ct0 = st->s0 + s0_incr;
    double f = (s - ct0) / st->dctBin;
    long long iBin = (long long)f;
    f -= iBin;
    if (iBin >= 0 && iBin < nBins - 1)
      dp = dp + ((1 - f) * st->dGamma[iBin] + f * st->dGamma[iBin + 1]) / Po * factor;
  }
  p = (1 + dp) * Po;
  beta = p / sqrt(p * p + 1);
  P.x[i] = x;
  P.y[i] = y;
  P.s[i] = beta * s;
  P.dp[i] = dp;
}

/* ---- CSRDRIFT, Stupakov mode (csbend.c:3803-4159) ---------------------- */

/* phi_last starts at -1, the value SolveForPhiStupakov's static holds before
 * its first call (csbend.c:4177) */
__global__ void csr_init_state_kernel(CsrDevState *st, int n) {
  for (int b = threadIdx.x; b < n; b += blockDim.x)
    st[b].phi_last = -1;
}

/* one kick's drift: the particles move back by dz_back first (only on the
 * first kick when the drift does not start where the last CSR element ended,
 * csbend.c:3835-3848), then forward by dz; c*t = s/beta; min/max of c*t per
 * bunch (csbend.c:3876-3893) */
__global__ void stupakov_drift_kernel(DevParticles P, int64_t n, int64_t share, CsrBunches B, PlainDrift plain,
                                      double dz_back, double dz, double Po) {
  chain_enter();
  const int64_t first = blockIdx.x * share, end = min(n, first + share);
  BunchRange range(first < n ? bunch_of(first, B) : 0);
  for (int64_t i = first + threadIdx.x; i - threadIdx.x < end; i += blockDim.x) {
    const int b = i < n ? bunch_of(i, B) : B.n - 1;
    const bool alive = i < n && P.lost_pass[i] < 0, mine = alive && B.mode[b];
    double ct = 0;
    if (alive && !mine && plain.now)
      exact_drift(P, i, plain.length);
    if (mine) {
      double x = P.x[i], xp = P.xp[i], y = P.y[i], yp = P.yp[i], s = P.s[i];
      if (dz_back != 0) {
        x = x - dz_back * xp;
        y = y - dz_back * yp;
        s = s - dz_back * sqrt((1 + xp * xp) + yp * yp);
      }
      x = x + xp * dz;
      y = y + yp * dz;
      const double p = Po * (1 + P.dp[i]), beta = p / sqrt(p * p + 1);
      ct = (s + dz * sqrt((1 + xp * xp) + yp * yp)) / beta;
      P.x[i] = x;
      P.y[i] = y;
      P.s[i] = ct;
    }
    range.add(ct, mine, b, B);
  }
  range.flush(B);
}

/* fn of SolveForPhiStupakov (csbend.c:4163-4165) */
struct StupakovFn {
  double x, x4;
  __device__ double operator()(double phi) const { return phi * phi * phi * (phi + x4) / (phi + x); }
};

/* The grid of b2e_zero_interp's scan for SolveForPhiStupakov and the function
 * on it: neither depends on the distance, so a kick's solutions share them.
 * The scan takes steps of phim/100 from 0 and ends beyond 1.01 phim. */
#define PHI_SCAN 128
struct PhiScan {
  double x[PHI_SCAN + 1], f[PHI_SCAN + 1];
};

__device__ __forceinline__ void phi_scan_fill(PhiScan &scan, const StupakovFn &fn, double phim) {
  const double dx = phim / 100;
  for (int k = threadIdx.x; k <= PHI_SCAN; k += blockDim.x) {
    double x = 0;
    for (int j = 0; j < k; j++) /* the scan's own sums */
      x = x + dx;
    scan.x[k] = x;
    scan.f[k] = fn(x);
  }
}

/* b2e_zero_interp(fn, value, 0, phim * 1.01, phim / 100, tol) by one warp: the
 * scan for a hit or a change of sign 32 steps at a time, the refinement in
 * every lane alike */
__device__ double phi_interp(const PhiScan &scan, const StupakovFn &fn, double value, double phim, double tol) {
  const double x_f = phim * 1.01, dx = phim / 100;
  if (!(dx > 0) || !(scan.x[PHI_SCAN] > x_f))
    return b2e_zero_interp(fn, value, 0, x_f, dx, tol);
  if (fabs(scan.f[0] - value) < tol)
    return 0;
  int found = 0;
  for (int base = 1; base <= PHI_SCAN && found == 0; base += 32) {
    const int k = base + (threadIdx.x & 31);
    const double ga = scan.f[k - 1] - value, gb = scan.f[k] - value;
    const bool here =
        scan.x[k] > x_f || fabs(gb) < tol || (ga == ga && gb == gb && (ga < 0) != (gb < 0));
    const unsigned any = __ballot_sync(0xffffffffu, here);
    if (any)
      found = base + __ffs(any) - 1;
  }
  double xa = scan.x[found - 1], xb = scan.x[found], xm = xa;
  double ga = scan.f[found - 1] - value, gb = scan.f[found] - value;
  if (xb > x_f)
    return x_f + dx;
  if (fabs(gb) < tol)
    return xb;
  for (int k = 0, side = 0; k < B2E_ROOT_MAX_REFINE; k++) {
    xm = xa - ga * (xb - xa) / (gb - ga);
    const double gm = fn(xm) - value;
    if (fabs(gm) < tol)
      return xm;
    if ((gm < 0) == (ga < 0)) {
      xa = xm;
      ga = gm;
      if (side == -1)
        gb = gb / 2;
      side = -1;
    } else {
      xb = xm;
      gb = gm;
      if (side == 1)
        ga = ga / 2;
      side = 1;
    }
  }
  return xm;
}

/* The solving part of SolveForPhiStupakov (csbend.c:4169-4202) by one warp:
 * phi for the scaled distance ds (> 0) from the previous solution phi_last.
 * b2e_zero_newton's passes with the two values of a pass formed by even and
 * odd lanes; a pass that ends within the tolerance has made the check of its
 * answer. */
__device__ double stupakov_phi(const PhiScan &scan, const StupakovFn &fn, double ds, double tol, double phim,
                               double *phi_last) {
  const double dx = phim / 1000;
  double phi = *phi_last, x_diff = phi;
  bool fits;
#pragma unroll 1
  for (int pass = 0;; pass++) {
    const double next = phi + dx, g_lane = fn(threadIdx.x & 1 ? next : phi) - ds;
    const double g = __shfl_sync(0xffffffffu, g_lane, 0), g_diff = __shfl_sync(0xffffffffu, g_lane, 1);
    fits = fabs(g) < tol;
    if (fits)
      break;
    if (pass == 2) {
      phi = (phi + x_diff) / 2;
      break;
    }
    x_diff = next;
    phi = phi - g / ((g_diff - g) / dx);
  }
  if (phi < 0 || phi > phim || (!fits && fabs(ds - fn(phi)) > tol))
    phi = phi_interp(scan, fn, ds, phim, tol);
  if (phi < 0 || phi > phim)
    return -1;
  *phi_last = phi;
  return phi;
}

/* per-kick scalars, formed on the host as the reference writes them */
struct StupakovArgs {
  double x;      /* zTravel / rho */
  double dsMax;  /* rho/24 theta^3 (theta + 4x)/(theta + x) */
  double dsC;    /* rho/6 theta^2 (theta + 3x), case C */
  double theta, rho, dz0;
  int trapz;
};

/* bins of a distance, clamped to [0, nb] (the comparisons against nb give
 * the reference's result; a negative distance does not occur behind a dipole) */
__device__ __forceinline__ long long clamp_bins(double d, int nb) {
  if (!(d > 0))
    return 0;
  return d >= (double)nb ? nb : (long long)d;
}

/* marks in place of a solution's tolerance */
#define PHI_KNOWN (-1.0)
#define PHI_MAX (-2.0)
#define PHI_END (-3.0)

/* wake of one Stupakov kick, one CTA per bunch (csbend.c:3950-4054): the
 * histogram filters of the last dipole, phi solutions (one warp, each starting
 * from the previous one: the latency of that chain bounds the kernel, about 16 us
 * (30,000 cycles) for 300 bins with the scan tabulated, the values of a Newton
 * pass side by side and all that is no part of the chain formed by the whole
 * block; 64 us on one thread), then per bin case C, case D's
 * boundary term and its integral in the reference's order, times -4/rho
 * GSConstant dz0.  Shared memory: 4 nBins + 8 doubles for the filters, nBins
 * for phi. */
__global__ void __launch_bounds__(1024, 1)
    stupakov_wake_kernel(CsrBunches B, const unsigned int *counts_all, WakeArgs a, StupakovArgs sa) {
  extern __shared__ double sm[];
  __shared__ double stage[2][SG_STAGE];
  __shared__ PhiScan scan;
  chain_release();
  stage_weights(a, stage);
  chain_wait();
  const int bunch = blockIdx.x;
  if (!B.mode[bunch])
    return;
  CsrDevState *st = B.st + bunch;
  const int nb = a.nBins;
  const double dct = st->dct;
  const unsigned int *counts = counts_all + (size_t)bunch * nb;
  wake_filters<unsigned int, unsigned long long>(counts, threadIdx.x < nb ? counts[threadIdx.x] : 0, a, dct, sm,
                                                 nullptr);
  const double *hist = sm, *deriv = sm + nb;
  double *phi = sm + 4 * nb + 8;
  if (!(dct > 0)) {
    for (int ib = threadIdx.x; ib < nb; ib += blockDim.x)
      st->dGamma[ib] = 0;
    return;
  }
  /* what a solution does not need the previous one for; the tolerance is below
   * zero where there is nothing to solve */
  const StupakovFn fn = {sa.x, 4 * sa.x};
  double *scaled = sm + 2 * nb, *tol = sm + 3 * nb;
  phi_scan_fill(scan, fn, sa.theta);
  const double at_phim = fn(sa.theta);
  for (int ib = threadIdx.x; ib < nb; ib += blockDim.x) {
    double ds = ib * dct / sa.rho, t = PHI_KNOWN, p = -1;
    if (ib * dct > sa.dsMax)
      t = PHI_END;
    else if (ds == 0)
      p = 0;
    else if (!(ds < 0)) {
      ds *= 24;
      t = ds / 1e4;
      if (fabs(ds - at_phim) < t) {
        t = PHI_MAX;
        p = sa.theta;
      }
    }
    scaled[ib] = ds;
    tol[ib] = t;
    phi[ib] = p;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double last = st->phi_last;
    for (int ib = 0; ib < nb; ib++) {
      const double t = tol[ib];
      if (t == PHI_END)
        break;
      if (t == PHI_KNOWN)
        continue;
      if (last == -1)
        last = sa.theta / 2;
      if (t == PHI_MAX) {
        last = sa.theta;
        continue;
      }
      const double p = stupakov_phi(scan, fn, scaled[ib], t, sa.theta, &last);
      if (threadIdx.x == 0)
        phi[ib] = p;
    }
    if (threadIdx.x == 0)
      st->phi_last = last;
  }
  __syncthreads();
  const long long diC = clamp_bins(sa.dsC / dct, nb), diD = clamp_bins(sa.dsMax / dct, nb);
  const double fC = -1 / (sa.theta + 2 * sa.x), factor = -4 / sa.rho * B.csr_const[2 * B.n + bunch] * sa.dz0;
  for (int ib = threadIdx.x; ib < nb; ib += blockDim.x) {
    double g = ib + diC < nb ? fC * hist[ib + diC] : 0, term1 = 0, term2 = 0;
    if (ib + diD < nb)
      g = g + hist[ib + diD] / (sa.theta + 2 * sa.x);
    int count = 0;
    for (int j = ib; j < nb; j++) {
      const double p = phi[j - ib];
      if (!(p >= 0))
        break;
      if (p > 0) {
        term2 = deriv[j] / (p + 2 * sa.x);
        g = g - term2;
        if (count == 0)
          term1 = term2;
        count++;
      }
    }
    if (count > 1 && sa.trapz)
      g = g + (term1 + term2) / 2;
    st->dGamma[ib] = g * factor;
  }
}

/* kick from the wake and c*t back to s at the new velocity (csbend.c:4078-4096) */
__global__ void stupakov_kick_kernel(DevParticles P, int64_t n, CsrBunches B, int nBins, double Po) {
  chain_enter();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || P.lost_pass[i] >= 0)
    return;
  const int b = bunch_of(i, B);
  if (!B.mode[b])
    return;
  const CsrDevState *st = B.st + b;
  const double ct = P.s[i];
  double dp = P.dp[i], f = (ct - st->ctLower) / st->dct;
  const long long iBin = (long long)f;
  f -= iBin;
  if (iBin >= 0 && iBin < nBins - 1)
    dp = dp + ((1 - f) * st->dGamma[iBin] + f * st->dGamma[iBin + 1]) / Po;
  const double p = (1 + dp) * Po, beta = p / sqrt(p * p + 1);
  P.dp[i] = dp;
  P.s[i] = beta * ct;
}

/* empty min/max keys of every bunch before a binning pass */
__global__ void csr_reset_keys_kernel(CsrBunches B) {
  for (int b = threadIdx.x; b < B.n; b += blockDim.x) {
    B.st[b].ct_min_key = ~0ull;
    B.st[b].ct_max_key = 0ull;
  }
}

/* min/max keys of every bunch to a contiguous [2][n] buffer and back, around
 * an all-rank reduction */
__global__ void csr_keys_gather_kernel(CsrBunches B, unsigned long long *keys) {
  for (int b = threadIdx.x; b < B.n; b += blockDim.x) {
    keys[b] = B.st[b].ct_min_key;
    keys[B.n + b] = B.st[b].ct_max_key;
  }
}
__global__ void csr_keys_scatter_kernel(CsrBunches B, const unsigned long long *keys) {
  for (int b = threadIdx.x; b < B.n; b += blockDim.x) {
    B.st[b].ct_min_key = keys[b];
    B.st[b].ct_max_key = keys[B.n + b];
  }
}

__global__ void csr_s0_add_kernel(CsrBunches B, double incr) {
  chain_enter();
  for (int b = threadIdx.x; b < B.n; b += blockDim.x)
    if (B.mode[b])
      B.st[b].s0 = B.st[b].s0 + incr;
}

/* do_tracking's sweeps after a collective element (do_tracking.c:2455-2475,
 * :2629): MAXAMP aperture if one is active, then inf/NaN in x or y. */
__global__ void post_element_sweep_kernel(DevParticles P, int64_t n, const DevAperture *ap, int pass, int elem_index) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || P.lost_pass[i] >= 0)
    return;
  Part p;
  p.x = P.x[i];
  p.y = P.y[i];
  bool lost = false;
  if (ap && ap->mode) {
    p.xp = P.xp[i];
    p.yp = P.yp[i];
    lost = !maxamp_ok(p, *ap);
  }
  if (!lost && !finite_xy(p))
    lost = true;
  if (lost) {
    P.lost_pass[i] = pass;
    P.lost_elem[i] = elem_index;
  }
}

cudaError_t launch_post_element_sweep(const DevParticles &P, int64_t n, const DevAperture *ap, int pass, int elem,
                                      cudaStream_t stream) {
  const int grid = (int)std::max<int64_t>(1, (n + 255) / 256);
  post_element_sweep_kernel<<<grid, 256, 0, stream>>>(P, n, ap, pass, elem);
  return cudaGetLastError();
}

/* exact drift of the particles of the bunches whose CSRDRIFT mode is `mode`
 * (every particle when the mode table is null) */
__global__ void edrift_kernel(DevParticles P, int64_t n, double L, CsrBunches B, int mode) {
  chain_enter();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || P.lost_pass[i] >= 0)
    return;
  if (B.mode && B.mode[bunch_of(i, B)] != mode)
    return;
  exact_drift(P, i, L);
}

/* ------------------------------------------------------------------ host -- */

static int grid_for(int64_t n) { return (int)std::max<int64_t>(1, (n + 255) / 256); }

int csr_configure(CsrState &st, const b2e_element *el, int n, const CompiledLattice &lat, const b2e_run_options &opt,
                  std::string &err) {
  csr_release(st);
  st.elems.clear();
  st.p_central = opt.p_central;
  st.enabled = !lat.csr_elements.empty();
  if (!st.enabled)
    return B2E_OK;
  std::vector<double> sgw;
  st.sg_offset.clear();
  for (int idx : lat.csr_elements) {
    const b2e_element &e = el[idx];
    const DevElem &d = lat.elems[idx];
    CsrElem ce;
    ce.index = idx;
    ce.kind = d.kind;
    if (d.kind == K_CSRCSBEND) {
      const double *p = e.p;
      ce.bins = (int)p[B2E_BEND_BINS];
      if (ce.bins < 2) {
        err = "Less than 2 bins for CSR!";
        return B2E_ERR_LATTICE;
      }
      if (ce.bins > B2E_CSR_MAX_BINS) {
        err = "CSRCSBEND BINS above the engine maximum (4096)";
        return B2E_ERR_LATTICE;
      }
      ce.nSlices = (int)d.c[CB_NSLICES];
      ce.nSub = (int)d.c[CB_NSUB];
      ce.sgHalf = (int)p[B2E_BEND_SG_HALFWIDTH];
      ce.sgOrder = (int)p[B2E_BEND_SG_ORDER];
      ce.sgdHalf = (int)p[B2E_BEND_SGDERIV_HALFWIDTH];
      ce.sgdOrder = (int)p[B2E_BEND_SGDERIV_ORDER];
      /* csbend.c:2042-2050 */
      if (ce.sgdHalf <= 0)
        ce.sgdHalf = ce.sgHalf;
      if (ce.sgdHalf <= 0)
        ce.sgdHalf = 1;
      if (ce.sgdOrder <= 0)
        ce.sgdOrder = ce.sgOrder;
      if (ce.sgdOrder <= 0)
        ce.sgdOrder = 1;
      if (2 * std::max(ce.sgHalf, ce.sgdHalf) + 1 > B2E_SG_MAX_WIDTH) {
        err = "Savitzky-Golay half-width too large";
        return B2E_ERR_LATTICE;
      }
      ce.trapz = p[B2E_BEND_TRAPAZOID_INTEGRATION] != 0;
      ce.steady = p[B2E_BEND_STEADY_STATE] != 0;
      ce.igf = p[B2E_BEND_IGF] != 0;
      if (ce.igf && !ce.steady) {
        err = "Must have STEADY_STATE=1 when IGF=1"; /* csbend.c:2598 */
        return B2E_ERR_LATTICE;
      }
      ce.csr = p[B2E_BEND_CSR] != 0;
      ce.lowCut0 = p[B2E_BEND_LOW_FREQUENCY_CUTOFF0];
      ce.lowCut1 = p[B2E_BEND_LOW_FREQUENCY_CUTOFF1];
      ce.highCut0 = p[B2E_BEND_HIGH_FREQUENCY_CUTOFF0];
      ce.highCut1 = p[B2E_BEND_HIGH_FREQUENCY_CUTOFF1];
      ce.lh = ce.highCut0 > 0 || ce.lowCut0 >= 0;
      ce.clip = p[B2E_BEND_CLIP_NEGATIVE_BINS] != 0;
      ce.angle = fabs(p[B2E_BEND_ANGLE]);
      ce.length = p[B2E_BEND_L];
      ce.rho0 = d.c[CB_RHO0];
      ce.binRangeFactor = p[B2E_BEND_BIN_RANGE_FACTOR] < 1.1 ? 1.1 : p[B2E_BEND_BIN_RANGE_FACTOR];
      ce.dzf = d.c[CB_DZF];
      memcpy(ce.bx.c, lat.rads[idx].c + RB_EXTRA0, sizeof(ce.bx.c));
      ce.z_end = d.z_end;
      /* SAME_BEND_PRECEDES of determine_bend_flags (bend_matrix.c:1342-1363):
       * MARKs in between are transparent */
      ce.same_bend_precedes = 0;
      for (int j = idx - 1; j >= 0; j--) {
        if (el[j].type == B2E_CSRCSBEND && strncmp(el[j].name, e.name, sizeof(e.name)) == 0) {
          ce.same_bend_precedes = 1;
          break;
        }
        if (el[j].type != B2E_MARK)
          break;
      }
      /* Savitzky-Golay weights for smoothing (order sgOrder, derivative 0)
       * and for the derivative (order sgdOrder, derivative 1) */
      st.sg_offset.push_back(sgw.size());
      for (int pass = 0; pass < 2; pass++) {
        const int half = pass == 0 ? ce.sgHalf : ce.sgdHalf, order = pass == 0 ? ce.sgOrder : ce.sgdOrder;
        const int width = sg_width(half, ce.bins);
        for (int row = 0; row < width; row++) {
          sgw.resize(sgw.size() + width);
          sg_row(half, order, pass, ce.bins, row, sgw.data() + sgw.size() - width);
        }
      }
    } else {
      const double *p = e.p;
      ce.stupakov = p[B2E_CSRDRIFT_USE_STUPAKOV] != 0;
      ce.drift_length = p[B2E_CSRDRIFT_L];
      ce.drift_dz = p[B2E_CSRDRIFT_DZ];
      ce.drift_kicks = (int)p[B2E_CSRDRIFT_N_KICKS];
      ce.drift_csr = p[B2E_CSRDRIFT_CSR] != 0;
      ce.z_start = d.z_start;
      st.sg_offset.push_back(sgw.size());
    }
    st.elems.push_back(ce);
  }
  /* one CSRDRIFT mode behind each dipole (csbend.c:3259-3263 stops the run
   * otherwise); the line is read cyclically, as drifts ahead of the first
   * dipole follow the last one on the next pass */
  {
    const int ne = (int)st.elems.size();
    int mode = -1;
    for (int k = 0; k < 2 * ne; k++) {
      const CsrElem &c = st.elems[k % ne];
      if (c.kind == K_CSRCSBEND)
        mode = -1;
      else if (c.drift_csr) {
        if (mode >= 0 && mode != c.stupakov) {
          err = "CSRDRIFT mode changed between dipoles. Pick one mode following each dipole.";
          return B2E_ERR_LATTICE;
        }
        mode = c.stupakov;
      }
    }
  }
  st.revolution_length = lat.total_length;
  st.last_bend = -1;
  if (csr_set_bunches(st, 1, nullptr, err))
    return B2E_ERR_NOMEM;
  if (!sgw.empty()) {
    if (cudaMalloc(&st.d_sg, sizeof(double) * sgw.size()) != cudaSuccess) {
      err = "CSR weight allocation failed";
      return B2E_ERR_NOMEM;
    }
    cudaMemcpy(st.d_sg, sgw.data(), sizeof(double) * sgw.size(), cudaMemcpyHostToDevice);
  }
  return B2E_OK;
}

int csr_set_bunches(CsrState &st, int n_bunches, const int64_t *d_offsets, std::string &err) {
  if (n_bunches < 1 || (n_bunches > 1 && !d_offsets)) {
    err = "CSR: bad bunch layout";
    return B2E_ERR_ARG;
  }
  if (st.d_state)
    cudaFree(st.d_state);
  if (st.d_counts)
    cudaFree(st.d_counts);
  if (st.d_csr_const)
    cudaFree(st.d_csr_const);
  if (st.d_flags)
    cudaFree(st.d_flags);
  if (st.d_alive)
    cudaFree(st.d_alive);
  if (st.h_alive)
    cudaFreeHost(st.h_alive);
  st.h_alive = nullptr;
  if (st.d_keys)
    cudaFree(st.d_keys);
  st.d_keys = nullptr;
  st.d_state = nullptr;
  st.d_counts = nullptr;
  st.d_csr_const = nullptr;
  st.d_flags = nullptr;
  st.d_alive = nullptr;
  st.n_bunches = n_bunches;
  st.d_offsets = d_offsets;
  st.wake_valid.assign(n_bunches, 0);
  st.macro_charge.assign(n_bunches, 0.0);
  if (cudaMalloc(&st.d_state, sizeof(CsrDevState) * n_bunches) != cudaSuccess ||
      cudaMalloc(&st.d_counts, sizeof(unsigned int) * B2E_CSR_MAX_BINS * n_bunches) != cudaSuccess ||
      cudaMalloc(&st.d_csr_const, 4 * sizeof(double) * n_bunches) != cudaSuccess ||
      cudaMalloc(&st.d_flags, 2 * n_bunches) != cudaSuccess ||
      cudaMalloc(&st.d_alive, sizeof(unsigned long long) * n_bunches) != cudaSuccess ||
      cudaMalloc(&st.d_keys, 2 * sizeof(unsigned long long) * n_bunches) != cudaSuccess ||
      cudaMallocHost(&st.h_alive, sizeof(unsigned long long) * n_bunches) != cudaSuccess ||
      (!st.alive_known && cudaEventCreateWithFlags(&st.alive_known, cudaEventDisableTiming) != cudaSuccess)) {
    err = "CSR state allocation failed";
    return B2E_ERR_NOMEM;
  }
  cudaMemset(st.d_state, 0, sizeof(CsrDevState) * n_bunches);
  cudaMemset(st.d_csr_const, 0, 4 * sizeof(double) * n_bunches);
  cudaMemset(st.d_flags, 0, 2 * n_bunches);
  csr_init_state_kernel<<<1, 256>>>((CsrDevState *)st.d_state, n_bunches);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    err = "CSR state initialisation failed";
    return B2E_ERR_CUDA;
  }
  return B2E_OK;
}

/* alive particles per bunch: blockIdx.y is the bunch */
__global__ void alive_per_bunch_kernel(const int32_t *lost_pass, int64_t n, const int64_t *offs, int nb,
                                       unsigned long long *alive) {
  const int b = blockIdx.y;
  const int64_t first = nb <= 1 ? 0 : offs[b], end = nb <= 1 ? n : offs[b + 1];
  unsigned long long c = 0;
  for (int64_t i = first + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < end;
       i += (int64_t)gridDim.x * blockDim.x)
    c += lost_pass[i] < 0;
  for (int off = 16; off > 0; off >>= 1)
    c += __shfl_down_sync(0xffffffffu, c, off);
  if ((threadIdx.x & 31) == 0 && c)
    atomicAdd(&alive[b], c);
}

/* What an element's kernels do per bunch, from the particles alive at its
 * entrance (n_part > 1 decides whether CSR is computed, csbend.c:1987,
 * :3196-3212): a bend's active flags with the constants of the others at zero
 * and empty range keys and counts (one block per bunch), or a drift's mode
 * flags out of the candidates that the host has copied there.  The counts go
 * to the host's memory as well. */
__global__ void csr_begin_kernel(CsrBunches B, const unsigned long long *alive, int drift, double *csr_const,
                                 unsigned int *counts, int nBins, unsigned long long *host_alive) {
  const int b = blockIdx.x;
  const bool some = alive[b] > 1;
  if (threadIdx.x == 0) {
    unsigned char *active = const_cast<unsigned char *>(B.active), *mode = const_cast<unsigned char *>(B.mode);
    host_alive[b] = alive[b];
    active[b] = !drift && some;
    mode[b] = drift && some && mode[b];
    if (!drift) {
      if (!some)
        csr_const[b] = csr_const[2 * B.n + b] = 0;
      B.st[b].ct_min_key = ~0ull;
      B.st[b].ct_max_key = 0ull;
    }
  }
  if (!drift)
    for (int k = threadIdx.x; k < nBins; k += blockDim.x)
      counts[(size_t)b * nBins + k] = 0;
}

static int count_alive(CsrState &st, const int32_t *lost_pass, int64_t n, cudaStream_t stream, std::string &err) {
  const int nb = st.n_bunches;
  if (cudaMemsetAsync(st.d_alive, 0, sizeof(unsigned long long) * nb, stream) != cudaSuccess) {
    err = "CSR: alive count failed";
    return B2E_ERR_CUDA;
  }
  const int gx = (int)std::min<int64_t>(std::max(1, 148 * 4 / nb), std::max<int64_t>(1, (n / nb + 255) / 256));
  alive_per_bunch_kernel<<<dim3(gx, nb), 256, 0, stream>>>(lost_pass, n, st.d_offsets, nb, st.d_alive);
  if (st.reducer && st.reducer(st.reducer_user, B2E_REDUCE_SUM_U64, st.d_alive, nb, stream)) {
    err = "CSR: the all-rank reduction of alive counts failed";
    return B2E_ERR_CUDA;
  }
  if (cudaGetLastError() != cudaSuccess) {
    err = "CSR: alive count failed";
    return B2E_ERR_CUDA;
  }
  return B2E_OK;
}

/* launches csr_begin_kernel and marks the place from which h_alive holds the
 * counts (await_alive) */
static int begin_element(CsrState &st, const CsrBunches &B, int drift, int bins, cudaStream_t stream,
                         std::string &err, int64_t *launches) {
  csr_begin_kernel<<<B.n, 256, 0, stream>>>(B, st.d_alive, drift, st.d_csr_const, st.d_counts, bins, st.h_alive);
  (*launches)++;
  if (cudaGetLastError() != cudaSuccess || cudaEventRecord(st.alive_known, stream) != cudaSuccess) {
    err = "CSR: alive count failed";
    return B2E_ERR_CUDA;
  }
  return B2E_OK;
}

static int await_alive(CsrState &st, std::string &err) {
  if (cudaEventSynchronize(st.alive_known) != cudaSuccess) {
    err = "CSR: alive count failed";
    return B2E_ERR_CUDA;
  }
  return B2E_OK;
}

int csr_reduce_counts(CsrState &st, std::vector<int64_t> &counts, cudaStream_t stream, std::string &err) {
  if (!st.reducer)
    return B2E_OK;
  const int nb = (int)counts.size();
  std::vector<unsigned long long> h(counts.begin(), counts.end());
  if (nb > st.n_bunches || cudaMemcpyAsync(st.d_alive, h.data(), sizeof(unsigned long long) * nb,
                                           cudaMemcpyHostToDevice, stream) != cudaSuccess ||
      st.reducer(st.reducer_user, B2E_REDUCE_SUM_U64, st.d_alive, nb, stream) ||
      cudaMemcpyAsync(h.data(), st.d_alive, sizeof(unsigned long long) * nb, cudaMemcpyDeviceToHost, stream) !=
          cudaSuccess ||
      cudaStreamSynchronize(stream) != cudaSuccess) {
    err = "CSR: the all-rank reduction of bunch sizes failed";
    return B2E_ERR_CUDA;
  }
  counts.assign(h.begin(), h.end());
  return B2E_OK;
}

/* all-rank min/max of every bunch's c*t keys (no-op without a reducer) */
static int reduce_keys(CsrState &st, const CsrBunches &B, cudaStream_t stream, std::string &err, int64_t *launches) {
  if (!st.reducer)
    return B2E_OK;
  csr_keys_gather_kernel<<<1, 32, 0, stream>>>(B, st.d_keys);
  if (st.reducer(st.reducer_user, B2E_REDUCE_MIN_U64, st.d_keys, B.n, stream) ||
      st.reducer(st.reducer_user, B2E_REDUCE_MAX_U64, st.d_keys + B.n, B.n, stream)) {
    err = "CSR: the all-rank reduction of the c*t range failed";
    return B2E_ERR_CUDA;
  }
  csr_keys_scatter_kernel<<<1, 32, 0, stream>>>(B, st.d_keys);
  (*launches) += 2;
  return cudaGetLastError() == cudaSuccess ? B2E_OK : B2E_ERR_CUDA;
}

void csr_reset(CsrState &st) {
  st.wakes_host.clear();
  st.wake_values = 0;
  st.page_values = 0;
  st.timed_kicks = st.timed_learned = 0;
  st.gate_values = 0;
  if (st.d_sur_counts)
    cudaMemset(st.d_sur_counts, 0, 2 * sizeof(unsigned long long));
  st.accumulated_angle = 0;
  st.wake_valid.assign(st.n_bunches, 0);
  st.last_bend = -1;
}

static int ensure_pagelog(CsrState &st, int64_t values, cudaStream_t stream) {
  if (values <= st.pagelog_cap)
    return B2E_OK;
  double *p = nullptr;
  if (cudaMalloc(&p, sizeof(double) * values) != cudaSuccess)
    return B2E_ERR_NOMEM;
  if (st.d_pagelog) {
    /* behind the kernels that still write the old log */
    if ((st.page_values && cudaMemcpyAsync(p, st.d_pagelog, sizeof(double) * st.page_values, cudaMemcpyDeviceToDevice,
                                           stream) != cudaSuccess) ||
        cudaStreamSynchronize(stream) != cudaSuccess) {
      cudaFree(p);
      return B2E_ERR_NOMEM;
    }
    cudaFree(st.d_pagelog);
  }
  st.d_pagelog = p;
  st.pagelog_cap = values;
  return B2E_OK;
}

static int ensure_wakelog(CsrState &st, int64_t values, cudaStream_t stream) {
  if (values <= st.wakelog_cap)
    return B2E_OK;
  double *p = nullptr;
  if (cudaMalloc(&p, sizeof(double) * values) != cudaSuccess)
    return B2E_ERR_NOMEM;
  if (st.d_wakelog) {
    /* behind the kernels that still write the old log */
    if ((st.wake_values && cudaMemcpyAsync(p, st.d_wakelog, sizeof(double) * st.wake_values, cudaMemcpyDeviceToDevice,
                                           stream) != cudaSuccess) ||
        cudaStreamSynchronize(stream) != cudaSuccess) {
      cudaFree(p);
      return B2E_ERR_NOMEM;
    }
    cudaFree(st.d_wakelog);
  }
  st.d_wakelog = p;
  st.wakelog_cap = values;
  return B2E_OK;
}

#define CSR_CUDA(call)                                                                                           \
  do {                                                                                                           \
    cudaError_t e_ = (call);                                                                                     \
    if (e_ != cudaSuccess) {                                                                                     \
      err = std::string(#call) + ": " + cudaGetErrorString(e_);                                                  \
      return B2E_ERR_CUDA;                                                                                       \
    }                                                                                                            \
  } while (0)

static int ensure_surrogate_buffers(CsrState &st, int64_t gate_values, std::string &err) {
  const int nb = st.n_bunches, L = wakenet_bins(st.net);
  if (st.sur_cap_bunches < nb) {
    cudaFree(st.d_sur_in);
    cudaFree(st.d_sur_out);
    cudaFree(st.d_sur_tab);
    cudaFree(st.d_sur_scal);
    st.d_sur_in = st.d_sur_out = nullptr;
    st.d_sur_tab = st.d_sur_scal = nullptr;
    st.sur_cap_bunches = 0;
    if (cudaMalloc(&st.d_sur_in, sizeof(float) * 4 * L * nb) != cudaSuccess ||
        cudaMalloc(&st.d_sur_out, sizeof(float) * L * nb) != cudaSuccess ||
        cudaMalloc(&st.d_sur_tab, sizeof(double) * 3 * B2E_CSR_MAX_BINS * nb) != cudaSuccess ||
        cudaMalloc(&st.d_sur_scal, sizeof(double) * 4 * nb) != cudaSuccess) {
      err = "CSR: wake network buffers";
      return B2E_ERR_NOMEM;
    }
    st.sur_cap_bunches = nb;
  }
  if (!st.d_sur_counts) {
    if (cudaMalloc(&st.d_sur_counts, 2 * sizeof(unsigned long long)) != cudaSuccess) {
      err = "CSR: wake network buffers";
      return B2E_ERR_NOMEM;
    }
    cudaMemset(st.d_sur_counts, 0, 2 * sizeof(unsigned long long));
  }
  if (st.gate_values + gate_values > st.gate_cap) {
    const int64_t cap = std::max<int64_t>(2 * st.gate_cap, st.gate_values + gate_values);
    double *p = nullptr;
    if (cudaMalloc(&p, sizeof(double) * cap) != cudaSuccess) {
      err = "CSR: gate log";
      return B2E_ERR_NOMEM;
    }
    if (st.d_gate_log) {
      if (st.gate_values)
        cudaMemcpy(p, st.d_gate_log, sizeof(double) * st.gate_values, cudaMemcpyDeviceToDevice);
      cudaFree(st.d_gate_log);
    }
    st.d_gate_log = p;
    st.gate_cap = cap;
  }
  return B2E_OK;
}

/* the filter arguments of applyLHPassFilters as the dipole passes them: the
 * low-frequency cutoffs are the high-pass ramp, the high-frequency cutoffs
 * the low-pass ramp (csbend.c:2559-2562) */
static void set_filter_args(WakeArgs &a, int lh, int clip, double lowCut0, double lowCut1, double highCut0,
                            double highCut1) {
  a.lh = lh;
  a.clip = clip;
  a.startHP = lowCut0;
  a.endHP = lowCut1;
  a.startLP = highCut0;
  a.endLP = highCut1;
}

/* Whether the wake kicks of a CSRDRIFT go on: some candidate bunch has the two
 * particles that a wake takes.  Where none has, the first kick's kernel has done
 * the whole drift.  Asked between kicks without waiting for the device, which
 * has the dipole's kernels ahead of it: a wait here drained them and took 8 % of
 * a run of 100 kicks per drift (1,726 -> 1,865 us, 20,011 particles).  Ranks that
 * share bunches have to agree on the number of kicks, so with a reducer the
 * host waits. */
struct DriftKicks {
  bool on = true, known = false;
};
static int drift_goes_on(CsrState &st, const std::vector<unsigned char> &flags, bool wait, DriftKicks &k,
                         std::string &err) {
  if (k.known)
    return B2E_OK;
  const cudaError_t e = wait ? cudaEventSynchronize(st.alive_known) : cudaEventQuery(st.alive_known);
  if (e == cudaErrorNotReady) {
    cudaGetLastError();
    return B2E_OK;
  }
  if (e != cudaSuccess) {
    err = "CSR: alive count failed";
    return B2E_ERR_CUDA;
  }
  k.known = true;
  k.on = false;
  for (int b = 0; b < st.n_bunches; b++)
    k.on = k.on || (flags[st.n_bunches + b] && st.h_alive[b] > 1);
  return B2E_OK;
}

/* CSRDRIFT with USE_STUPAKOV=1 (track_through_driftCSR_Stupakov,
 * csbend.c:3803-4159) for the bunches whose mode flag is set; the others get
 * their exact drift in the first kick's drift kernel.  Per kick: drift and c*t
 * with the min/max keys, the histogram of the last dipole's bin count and range
 * factor, the wake (one CTA per bunch), the kick; then the closing half drift. */
static int stupakov_drift(CsrState &st, const CsrElem &ce, const CsrBunches &B,
                          const std::vector<unsigned char> &flags, const DevParticles &P, int64_t n, double zStart,
                          cudaStream_t stream, std::string &err, int64_t *launches) {
  if (st.last_bend < 0) {
    err = "CSRDRIFT: no dipole wake to follow";
    return B2E_ERR_STATE;
  }
  const CsrElem &bend = st.elems[st.last_bend];
  const int nb = bend.bins, nbunch = B.n, g = grid_for(n);
  const Sweep sweep = sweep_of(n);
  const double Po = st.p_central, rho = st.last_rho, theta = st.last_theta;
  double length = ce.drift_length, dz_back = 0;
  if (zStart != st.zLast) {
    length += (dz_back = zStart - st.zLast);
    zStart = st.zLast;
  }
  long nKicks;
  if (ce.drift_dz > 0) {
    if ((nKicks = (long)(length / ce.drift_dz + 0.5)) < 1)
      nKicks = 1;
  } else
    nKicks = ce.drift_kicks;
  if (nKicks <= 0) {
    err = "nKicks=0 in CSR drift.";
    return B2E_ERR_LATTICE;
  }
  const double dz0 = length / nKicks;
  double dz = dz0 / 2, zTravel = zStart - st.z0;
  const double *sgw = st.d_sg + st.sg_offset[st.last_bend];
  WakeArgs a = {};
  a.nBins = nb;
  a.sgHalf = bend.sgHalf;
  a.sgdHalf = bend.sgdHalf;
  a.trapz = bend.trapz;
  a.sg_w = sgw;
  a.sgd_w = sgw + sg_width(bend.sgHalf, nb) * sg_width(bend.sgHalf, nb);
  set_filter_args(a, bend.lh, bend.clip, bend.lowCut0, bend.lowCut1, bend.highCut0, bend.highCut1);
  const size_t smem = sizeof(double) * (5 * nb + 8);
  CSR_CUDA(cudaFuncSetAttribute(stupakov_wake_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  CsrBunches H = B; /* the histogram bins the bunches in this mode */
  H.active = B.mode;
  DriftKicks kicks;
  for (long iKick = 0; iKick < nKicks; iKick++) {
    if (iKick == 1)
      dz = dz0;
    zTravel += dz;
    StupakovArgs sa;
    sa.x = zTravel / rho;
    sa.dsMax = rho / 24 * b2e_pow(theta, 3) * (theta + 4 * sa.x) / (theta + sa.x);
    sa.dsC = rho / 6 * (theta * theta) * (theta + 3 * sa.x);
    sa.theta = theta;
    sa.rho = rho;
    sa.dz0 = dz0;
    sa.trapz = bend.trapz;
    csr_reset_keys_kernel<<<1, 32, 0, stream>>>(B);
    CSR_CUDA(launch_chained(stupakov_drift_kernel, dim3(sweep.grid), dim3(256), 0, stream, P, n, sweep.share, B,
                            PlainDrift{ce.drift_length, iKick == 0}, iKick == 0 ? dz_back : 0.0, dz, Po));
    (*launches) += 2;
    CSR_CUDA(cudaGetLastError());
    /* a reducer is called only for wakes that are formed */
    if (iKick > 0 || st.reducer)
      if (int rc = drift_goes_on(st, flags, st.reducer, kicks, err))
        return rc;
    if (!kicks.on)
      return B2E_OK;
    int rrc = reduce_keys(st, B, stream, err, launches);
    if (rrc)
      return rrc;
    CSR_CUDA(cudaMemsetAsync(st.d_counts, 0, sizeof(unsigned int) * nb * nbunch, stream));
    const int64_t per = (n + nbunch - 1) / nbunch;
    const int hb = hist_blocks(per, nbunch);
    CSR_CUDA(launch_chained(csr_hist_kernel, dim3(hb, nbunch), dim3(1024), hist_smem(nb), stream, P, n, H,
                            st.d_counts, nb, bend.binRangeFactor));
    (*launches)++;
    CSR_CUDA(cudaGetLastError());
    if (st.reducer && st.reducer(st.reducer_user, B2E_REDUCE_SUM_U32, st.d_counts, (int64_t)nb * nbunch, stream)) {
      err = "CSR: the all-rank reduction of the histogram failed";
      return B2E_ERR_CUDA;
    }
    CSR_CUDA(launch_chained(stupakov_wake_kernel, dim3(nbunch), dim3(wake_threads(nb)), smem, stream, B,
                            (const unsigned int *)st.d_counts, a, sa));
    CSR_CUDA(launch_chained(stupakov_kick_kernel, dim3(g), dim3(256), 0, stream, P, n, B, nb, Po));
    (*launches) += 2;
    CSR_CUDA(cudaGetLastError());
  }
  CSR_CUDA(launch_chained(edrift_kernel, dim3(g), dim3(256), 0, stream, P, n, dz0 / 2, B, 1));
  (*launches)++;
  CSR_CUDA(cudaGetLastError());
  st.zLast = zStart + length;
  return B2E_OK;
}

int csr_track_element(CsrState &st, const DevElem *d_elems, const DevElem &h_elem, const DevParticles &P, int64_t n,
                      int elem, int pass, cudaStream_t stream, std::string &err, int64_t *launches) {
  const int count_rc = count_alive(st, P.lost_pass, n, stream, err);
  if (count_rc)
    return count_rc;
  (*launches)++;
  size_t k = 0;
  while (k < st.elems.size() && st.elems[k].index != elem)
    k++;
  if (k == st.elems.size()) {
    err = "CSR element not configured";
    return B2E_ERR_STATE;
  }
  const CsrElem &ce = st.elems[k];
  const int nbunch = st.n_bunches;
  CsrBunches B;
  B.offs = st.d_offsets;
  B.n = nbunch;
  B.st = (CsrDevState *)st.d_state;
  B.csr_const = st.d_csr_const;
  B.active = st.d_flags;
  B.mode = st.d_flags + nbunch;
  const double Po = st.p_central;
  const int g = grid_for(n);
  std::vector<unsigned char> flags(2 * nbunch, 0);
  if (ce.kind == K_CSRDRIFT) {
    /* track_through_driftCSR (csbend.c:3176-3533), mode 0: bunches with a
     * valid dipole wake and more than one particle get wake kicks, the others
     * an exact drift (csbend.c:3196-3212) */
    bool any = false;
    for (int b = 0; b < nbunch; b++) {
      flags[nbunch + b] = st.wake_valid[b] && ce.drift_csr;
      any = any || flags[nbunch + b];
    }
    /* the flags are settled on the device; what the host needs of them is
     * whether an invalid number of kicks is an error */
    if (any) {
      CSR_CUDA(cudaMemcpyAsync(st.d_flags, flags.data(), flags.size(), cudaMemcpyHostToDevice, stream));
      const int rc = begin_element(st, B, 1, 0, stream, err, launches);
      if (rc)
        return rc;
      if (!(ce.drift_dz > 0) && ce.drift_kicks <= 0) {
        DriftKicks kicks;
        if (int rc2 = drift_goes_on(st, flags, true, kicks, err))
          return rc2;
        any = kicks.on;
      }
    }
    if (!any) {
      CsrBunches all = B;
      all.mode = nullptr;
      edrift_kernel<<<g, 256, 0, stream>>>(P, n, ce.drift_length, all, 0);
      (*launches)++;
      CSR_CUDA(cudaGetLastError());
      return B2E_OK;
    }
    double zStart = ce.z_start;
    /* a drift behind the previous pass's dipole (csbend.c:3251-3255) */
    for (int guard = 0; zStart + 1e-12 < st.zLast && st.revolution_length > 0 && guard < (1 << 20); guard++)
      zStart += st.revolution_length;
    if (ce.stupakov)
      return stupakov_drift(st, ce, B, flags, P, n, zStart, stream, err, launches);
    int nKicks;
    if (ce.drift_dz > 0) {
      if ((nKicks = (int)(ce.drift_length / ce.drift_dz)) < 1)
        nKicks = 1;
    } else
      nKicks = ce.drift_kicks;
    if (nKicks <= 0) {
      err = "nKicks=0 in CSR drift.";
      return B2E_ERR_LATTICE;
    }
    double dz0 = ce.drift_length / nKicks, dz = dz0 / 2;
    double dzFirst = zStart - st.zLast;
    /* csrWake.bins: bins of the last CSRCSBEND tracked (on a later pass,
     * possibly one further down the line) */
    const int lastBins = st.last_bend >= 0 ? st.elems[st.last_bend].bins : 0;
    DriftKicks kicks;
    for (int iKick = 0; iKick < nKicks; iKick++) {
      if (iKick == 1)
        dz = dz0;
      double incr = dz + dzFirst;
      double factor = (dz0 + dzFirst) / st.ds0;
      CSR_CUDA(launch_chained(csr_drift_kick_kernel, dim3(g), dim3(256), 0, stream, P, n, B,
                              PlainDrift{ce.drift_length, iKick == 0}, dz, incr, factor, 1, lastBins, Po));
      CSR_CUDA(launch_chained(csr_s0_add_kernel, dim3(1), dim3(32), 0, stream, B, incr));
      (*launches) += 2;
      CSR_CUDA(cudaGetLastError());
      if (int rc = drift_goes_on(st, flags, false, kicks, err))
        return rc;
      if (!kicks.on)
        return B2E_OK;
      dzFirst = 0;
    }
    dz = dz0 / 2;
    CSR_CUDA(launch_chained(edrift_kernel, dim3(g), dim3(256), 0, stream, P, n, dz, B, 1));
    CSR_CUDA(launch_chained(csr_s0_add_kernel, dim3(1), dim3(32), 0, stream, B, dz));
    (*launches) += 2;
    CSR_CUDA(cudaGetLastError());
    st.zLast = zStart + ce.drift_length;
    return B2E_OK;
  }

  /* ---- CSRCSBEND ---- */
  const DevElem *d_e = d_elems + elem;
  if (!ce.same_bend_precedes)
    st.accumulated_angle = 0;
  st.wake_valid.assign(nbunch, 0);
  if (st.beta0_cap < n) {
    if (st.d_beta0)
      cudaFree(st.d_beta0);
    if (cudaMalloc(&st.d_beta0, sizeof(double) * std::max<int64_t>(n, 1)) != cudaSuccess) {
      err = "CSR beta0 allocation failed";
      return B2E_ERR_NOMEM;
    }
    st.beta0_cap = n;
  }
  if (ensure_wakelog(st, st.wake_values + (int64_t)ce.nSlices * ce.bins * nbunch, stream)) {
    err = "CSR wake log allocation failed";
    return B2E_ERR_NOMEM;
  }
  const int64_t page_stride = B2E_CSR_PAGE_HEADER + 4 * (int64_t)ce.bins;
  if (st.record_pages && ensure_pagelog(st, st.page_values + (int64_t)ce.nSlices * nbunch * page_stride, stream)) {
    err = "CSR page record allocation failed";
    return B2E_ERR_NOMEM;
  }
  st.ds0 = ce.length / ce.nSlices;
  st.zLast = st.z0 = ce.z_end;
  /* CSRConstant (csbend.c:2378-2381), per bunch */
  const double eps0 = 1 / ((4 * kPI * 1e-7) * kC * kC);
  std::vector<double> csr_constant(4 * nbunch, 0.0);
  for (int b = 0; b < nbunch; b++) {
    if (ce.csr) /* zeroed by csr_begin_kernel where one particle or none is alive */
      csr_constant[b] = 2 * st.macro_charge[b] * kE / b2e_pow(3 * ce.rho0 * ce.rho0, 1. / 3.) /
                        (4 * kPI * eps0 * kME * (kC * kC));
    /* the IGF wake's factor (csbend.c:2678-2679) */
    csr_constant[nbunch + b] = -st.macro_charge[b] / (kME * (kC * kC)) * ce.length / ce.nSlices;
    /* GSConstant for a Stupakov CSRDRIFT (csbend.c:2999) */
    csr_constant[2 * nbunch + b] = csr_constant[b] * b2e_pow(3 * ce.rho0 * ce.rho0, 1. / 3.) / 2;
    /* the macro-particle charge, for the page record */
    csr_constant[3 * nbunch + b] = st.macro_charge[b];
  }
  CSR_CUDA(cudaMemcpyAsync(st.d_csr_const, csr_constant.data(), 4 * sizeof(double) * nbunch, cudaMemcpyHostToDevice,
                           stream));
  if (int rc = begin_element(st, B, 0, ce.bins, stream, err, launches))
    return rc;
  const double *sgw = st.d_sg + st.sg_offset[k];
  const size_t wake_smem = sizeof(double) * (5 * ce.bins + 8);
  CSR_CUDA(cudaFuncSetAttribute(csr_wake_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wake_smem));
  /* the host learns which bunches are active once the entry and the first
   * slice are on their way: the device works on while it waits */
  bool any_active = false, use_net = false, recycle = false;
  const size_t sur_smem = sizeof(double) * (3 * ce.bins + 1024);
  auto settle = [&]() -> int {
    if (await_alive(st, err))
      return B2E_ERR_CUDA;
    for (int b = 0; b < nbunch; b++) {
      flags[b] = st.h_alive[b] > 1; /* csbend.c:1987 */
      any_active = any_active || flags[b];
    }
    /* learned wake: trained on the transient integral with trapezoid rule (the
     * CSRCSBEND defaults); other settings, or a bunch train larger than the
     * network's batch, use the plain integral */
    use_net = st.net && any_active && !ce.steady && ce.trapz && !ce.lh && ce.bins <= wakenet_bins(st.net) &&
              nbunch <= wakenet_max_batch(st.net);
    if (use_net) {
      int rc = ensure_surrogate_buffers(st, (int64_t)ce.nSlices * nbunch, err);
      if (rc)
        return rc;
      CSR_CUDA(cudaFuncSetAttribute(csr_sur_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)std::max(sur_smem, sizeof(double) * (4 * ce.bins + 1024))));
      CSR_CUDA(cudaFuncSetAttribute(csr_sur_combine_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sur_smem));
    }
    /* on the plain-integral path the wake kernel empties the range keys and the
     * counts for the next kick; otherwise both are reset before every kick */
    recycle = any_active && !use_net;
    return B2E_OK;
  };
  CSR_CUDA(launch_chained(csr_entry_kernel, dim3(g), dim3(256), 0, stream, P, n, st.d_beta0, d_e, ce.bx, Po));
  (*launches)++;
  CSR_CUDA(cudaGetLastError());
  double phiBend = st.accumulated_angle;
  for (int kick = 0; kick < ce.nSlices; kick++) {
    if (!recycle && kick > 0) {
      csr_reset_keys_kernel<<<1, 32, 0, stream>>>(B);
      (*launches)++;
    }
    int64_t per_block;
    const int slice_blocks = slice_grid(n, &per_block);
    CSR_CUDA(launch_chained(slice_kernel(h_elem), dim3(slice_blocks), dim3(SLICE_THREADS), 0, stream, P, n, per_block,
                            (const double *)st.d_beta0, h_elem, B, (int)(kick > 0), ce.bins, Po, 1 / Po, pass, elem));
    (*launches)++;
    CSR_CUDA(cudaGetLastError());
    if (kick == 0)
      if (int rc = settle())
        return rc;
    if (!any_active)
      continue;
    int rrc = reduce_keys(st, B, stream, err, launches);
    if (rrc)
      return rrc;
    if (!recycle && kick > 0)
      CSR_CUDA(cudaMemsetAsync(st.d_counts, 0, sizeof(unsigned int) * ce.bins * nbunch, stream));
    int64_t per = (n + nbunch - 1) / nbunch;
    int hb = hist_blocks(per, nbunch);
    CSR_CUDA(launch_chained(csr_hist_kernel, dim3(hb, nbunch), dim3(1024), hist_smem(ce.bins), stream, P,
                            n, B, st.d_counts, ce.bins, ce.binRangeFactor));
    (*launches)++;
    CSR_CUDA(cudaGetLastError());
    if (st.reducer && st.reducer(st.reducer_user, B2E_REDUCE_SUM_U32, st.d_counts, (int64_t)ce.bins * nbunch, stream)) {
      err = "CSR: the all-rank reduction of the histogram failed";
      return B2E_ERR_CUDA;
    }
    phiBend += ce.angle / ce.nSlices;
    double slippage = fabs(ce.rho0 * (phiBend * phiBend * phiBend) / 24.0);
    WakeArgs a = {};
    a.nBins = ce.bins;
    a.sgHalf = ce.sgHalf;
    a.sgdHalf = ce.sgdHalf;
    a.trapz = ce.trapz;
    a.steady = ce.steady;
    a.sg_w = sgw;
    a.sgd_w = sgw + sg_width(ce.sgHalf, ce.bins) * sg_width(ce.sgHalf, ce.bins);
    a.slippage = slippage;
    a.slippage13 = b2e_pow(slippage, 1. / 3.);
    a.length = ce.length;
    a.nSlices = ce.nSlices;
    a.c1 = a.c2 = a.csr_constant = 0; /* per bunch in the kernel */
    a.wakelog = st.d_wakelog + st.wake_values;
    /* pages of the plain-integral kicks only (the learned wake writes none) */
    a.pagelog = st.record_pages && !use_net ? st.d_pagelog + st.page_values : nullptr;
    a.page_element = elem;
    a.page_kick = kick;
    a.page_angle = phiBend;
    a.page_ds_kick = ce.length / ce.nSlices;
    a.page_p_central = Po;
    a.page_range_factor = ce.binRangeFactor;
    a.igf = ce.igf;
    set_filter_args(a, ce.lh, ce.clip, ce.lowCut0, ce.lowCut1, ce.highCut0, ce.highCut1);
    {
      /* gamma^2, gamma^3 and the IGF constants as the reference forms them
       * (csbend.c:1981-1982, :2604, :2617) */
      const double gamma2 = Po * Po + 1;
      a.gamma2 = gamma2;
      a.gamma3 = b2e_pow(gamma2, 3. / 2);
      a.rho0 = ce.rho0;
      a.const1 = 6.0 - b2e_log(27.0 / 4.0);
      a.q4pe = kE / (4 * kPI * eps0);
      a.igf_factor = 0;
    }
    cudaEvent_t ev_end = nullptr;
    if (st.time_wake) {
      while ((int64_t)st.wake_events.size() < 2 * (st.timed_kicks + 1)) {
        cudaEvent_t e;
        CSR_CUDA(cudaEventCreate(&e));
        st.wake_events.push_back(e);
      }
      CSR_CUDA(cudaEventRecord(st.wake_events[2 * st.timed_kicks], stream));
      ev_end = st.wake_events[2 * st.timed_kicks + 1];
    }
    if (use_net) {
      const int L = wakenet_bins(st.net);
      csr_sur_filter_kernel<<<nbunch, 1024, std::max(sur_smem, sizeof(double) * 4 * ce.bins), stream>>>(B, st.d_counts, a, L, st.sc_dens, st.sc_deriv,
                                                                st.d_sur_tab, st.d_sur_scal, st.d_sur_in);
      CSR_CUDA(cudaGetLastError());
      int rc = wakenet_infer(st.net, st.d_sur_in, nbunch, st.d_sur_out, stream);
      if (rc) {
        err = "CSR: wake network inference failed";
        return rc;
      }
      csr_sur_combine_kernel<<<nbunch, 1024, sur_smem, stream>>>(B, a, st.d_sur_tab, st.d_sur_scal, st.d_sur_out, L,
                                                                 st.sc_target, st.gate_tol, st.gate_stride,
                                                                 kick % st.gate_stride, st.d_gate_log + st.gate_values,
                                                                 st.d_sur_counts);
      CSR_CUDA(cudaGetLastError());
      st.gate_values += nbunch;
      (*launches) += 3 + 7; /* filter, pack + 6 convolutions, combine */
    } else {
      CSR_CUDA(launch_chained(csr_wake_kernel, dim3(nbunch), dim3(wake_threads(ce.bins)), wake_smem, stream, B, st.d_counts, a,
                              recycle ? 1 : 0));
      (*launches)++;
      CSR_CUDA(cudaGetLastError());
    }
    if (ev_end) {
      CSR_CUDA(cudaEventRecord(ev_end, stream));
      st.timed_kicks++;
      st.timed_learned += use_net;
    }
    st.wake_values += (int64_t)ce.bins * nbunch;
    if (a.pagelog)
      st.page_values += nbunch * page_stride;
  }
  if (ce.nSlices <= 0)
    if (int rc = settle())
      return rc;
  if (!recycle || ce.nSlices <= 0) {
    csr_reset_keys_kernel<<<1, 32, 0, stream>>>(B);
    (*launches)++;
  }
  const Sweep sweep = sweep_of(n);
  CSR_CUDA(launch_chained(csr_last_kick_kernel, dim3(sweep.grid), dim3(256), 0, stream, P, n, sweep.share, B, ce.bins, Po,
                          ce.rho0));
  CSR_CUDA(cudaGetLastError());
  if (any_active) {
    int rrc = reduce_keys(st, B, stream, err, launches);
    if (rrc)
      return rrc;
  }
  CSR_CUDA(launch_chained(csr_exit_kernel, dim3(g), dim3(256), 0, stream, P, n, d_e, ce.bx, B, ce.binRangeFactor, Po, pass,
                          elem));
  (*launches) += 2;
  CSR_CUDA(cudaGetLastError());
  for (int b = 0; b < nbunch; b++)
    st.wake_valid[b] = flags[b];
  /* csrWake.rho, csrWake.bendingAngle (csbend.c:2992-2993) */
  st.last_bend = (int)k;
  st.last_rho = h_elem.c[CB_RHO_ACTUAL];
  st.last_theta = ce.same_bend_precedes ? fabs(phiBend) : ce.angle;
  st.accumulated_angle += ce.angle;
  if (use_net && wakenet_take_status(st.net, stream)) {
    err = "CSR: a bounded wait in the wake network gave up";
    return B2E_ERR_TIMEOUT;
  }
  return B2E_OK;
}

int csr_wake_timing(CsrState &st, double *ms, int64_t *kicks, int64_t *learned, std::string &err) {
  double total = 0;
  for (int64_t k = 0; k < st.timed_kicks; k++) {
    float t = 0;
    cudaError_t e = cudaEventSynchronize(st.wake_events[2 * k + 1]);
    if (e == cudaSuccess)
      e = cudaEventElapsedTime(&t, st.wake_events[2 * k], st.wake_events[2 * k + 1]);
    if (e != cudaSuccess) {
      err = cudaGetErrorString(e);
      return B2E_ERR_CUDA;
    }
    total += t;
  }
  *ms = total;
  *kicks = st.timed_kicks;
  *learned = st.timed_learned;
  return B2E_OK;
}

int csr_copy_pages(CsrState &st, double *pages, int64_t capacity, int64_t *written, std::string &err) {
  int64_t n = std::min<int64_t>(st.page_values, capacity);
  if (n > 0 && pages) {
    cudaError_t e = cudaMemcpy(pages, st.d_pagelog, sizeof(double) * n, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
      err = cudaGetErrorString(e);
      return B2E_ERR_CUDA;
    }
  }
  *written = pages ? n : st.page_values;
  return B2E_OK;
}

int csr_copy_wakes(CsrState &st, double *wakes, int64_t capacity, int64_t *written, std::string &err) {
  int64_t n = std::min<int64_t>(st.wake_values, capacity);
  if (n > 0 && wakes) {
    cudaError_t e = cudaMemcpy(wakes, st.d_wakelog, sizeof(double) * n, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
      err = cudaGetErrorString(e);
      return B2E_ERR_CUDA;
    }
  }
  *written = wakes ? n : st.wake_values;
  return B2E_OK;
}

void csr_release(CsrState &st) {
  if (st.d_beta0)
    cudaFree(st.d_beta0);
  if (st.d_state)
    cudaFree(st.d_state);
  if (st.d_counts)
    cudaFree(st.d_counts);
  if (st.d_csr_const)
    cudaFree(st.d_csr_const);
  if (st.d_flags)
    cudaFree(st.d_flags);
  if (st.d_alive)
    cudaFree(st.d_alive);
  if (st.h_alive)
    cudaFreeHost(st.h_alive);
  st.h_alive = nullptr;
  if (st.alive_known)
    cudaEventDestroy(st.alive_known);
  st.alive_known = nullptr;
  if (st.d_keys)
    cudaFree(st.d_keys);
  st.d_keys = nullptr;
  st.d_csr_const = nullptr;
  st.d_flags = nullptr;
  st.d_alive = nullptr;
  void *sur[] = {st.d_sur_in, st.d_sur_out, st.d_sur_tab, st.d_sur_scal, st.d_gate_log, st.d_sur_counts};
  for (void *q : sur)
    if (q)
      cudaFree(q);
  st.d_sur_in = st.d_sur_out = nullptr;
  st.d_sur_tab = st.d_sur_scal = st.d_gate_log = nullptr;
  st.d_sur_counts = nullptr;
  st.sur_cap_bunches = st.gate_cap = st.gate_values = 0;
  if (st.d_sg)
    cudaFree(st.d_sg);
  if (st.d_wakelog)
    cudaFree(st.d_wakelog);
  if (st.d_pagelog)
    cudaFree(st.d_pagelog);
  for (cudaEvent_t e : st.wake_events)
    cudaEventDestroy(e);
  st.wake_events.clear();
  st.timed_kicks = st.timed_learned = 0;
  st.d_pagelog = nullptr;
  st.pagelog_cap = 0;
  st.page_values = 0;
  st.d_beta0 = nullptr;
  st.d_state = nullptr;
  st.d_counts = nullptr;
  st.d_sg = nullptr;
  st.d_wakelog = nullptr;
  st.beta0_cap = 0;
  st.wakelog_cap = 0;
  st.wake_values = 0;
}

} // namespace b2e

/* ==========================================================================
 * Allocation-free CSR dipole: b2e_csr_bend_static (include/elegant_b200.h).
 *
 * Some callers cannot allocate device memory at the moment they need this
 * computation: a host program that has handed the whole card to its own
 * memory pool, code that runs where cudaMalloc is not permitted, or an
 * embedding that must never fail for lack of memory halfway through a run.
 * For them, this path keeps all of its working memory in one file-scope
 * device array that is part of the loaded library image, so a call needs only
 * the caller's own particle and output buffers.
 *
 * The array holds per-particle entrance velocities (up to
 * B2E_STATIC_MAX_PARTICLES), the CSR binning/wake state, the histogram, the
 * Savitzky-Golay weight tables (of the widest windows) and the
 * element record: about 8.5 MB.  Under lazy module loading (CUDA's default)
 * a device gives it memory when this module is first used there -- the
 * set-up in static_scratch() -- and keeps it until the process exits.  The
 * call only enqueues work: the alive count that decides whether CSR is
 * computed becomes the bunch's flags on the device, so the host never waits
 * for the GPU.  All calls share the array and it keeps the previous
 * call's contents; everything that must start at zero is cleared by each
 * call.  Two calls whose work overlaps on the GPU (different streams, or
 * different host threads) race on this memory: callers must serialise them.
 * ======================================================================== */

/* B2E_STATIC_MAX_PARTICLES and B2E_STATIC_MAX_BINS come from elegant_b200.h */
namespace b2e {

struct StaticCsrScratch {
  double beta0[B2E_STATIC_MAX_PARTICLES];
  CsrDevState state;
  unsigned int counts[B2E_STATIC_MAX_BINS];
  double sg_w[2 * B2E_SG_MAX_WIDTH * B2E_SG_MAX_WIDTH];
  DevElem elem;
  unsigned long long counters[2];
  double csr_const[2];    /* the one bunch's CSRConstant and IGF wake factor */
  unsigned char flags[2]; /* active, CSRDRIFT mode */
};

static __device__ __align__(256) unsigned char g_static_csr_scratch[sizeof(StaticCsrScratch)];

/* Device addresses of g_static_csr_scratch, one per device, looked up by the
 * first call made with that device current (the set-up step).  That lookup is
 * also what makes CUDA load this module on the device under lazy module
 * loading (the default), so the array and the kernels' code take their device
 * memory at that first call, not when the library is loaded.  The cached
 * address belongs to the device's primary context: the library must not be
 * used on a device after cudaDeviceReset. */
#define B2E_STATIC_MAX_DEVICES 64
static void *g_static_addr[B2E_STATIC_MAX_DEVICES];
static std::mutex g_static_mutex;

static StaticCsrScratch *static_scratch(char *err, int64_t errlen) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= B2E_STATIC_MAX_DEVICES) {
    snprintf(err, errlen, "b2e_csr_bend_static: no usable current device (%s)", cudaGetErrorString(e));
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (!g_static_addr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_csr_scratch);
    if (e != cudaSuccess || !p) {
      snprintf(err, errlen, "b2e_csr_bend_static: cudaGetSymbolAddress failed on device %d (%s)", dev,
               cudaGetErrorString(e));
      return nullptr;
    }
    g_static_addr[dev] = p;
  }
  return (StaticCsrScratch *)g_static_addr[dev];
}

__global__ void static_set_elem_kernel(DevElem e, DevElem *dst) { *dst = e; }

/* The bunch's flags from the entrance count (S->counters[1] = particles alive
 * at the entrance; CSR only for more than one, csbend.c:1987), formed on the
 * device so that the host never waits for the count. */
__global__ void static_set_bunch_kernel(StaticCsrScratch *S, double csr_constant, double igf_factor) {
  const int more_than_one = S->counters[1] > 1;
  S->csr_const[0] = more_than_one ? csr_constant : 0.0;
  S->csr_const[1] = igf_factor;
  S->flags[0] = (unsigned char)more_than_one;
  S->flags[1] = 0;
}

/* Savitzky-Golay weights for one element, on the device, with the same helpers
 * and layout as csr_configure: smoothing rows, then derivative rows. */
__global__ void static_sg_weights_kernel(int bins, int sgHalf, int sgOrder, int sgdHalf, int sgdOrder, double *w) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int w0 = sg_width(sgHalf, bins), w1 = sg_width(sgdHalf, bins);
  if (t < w0)
    sg_row(sgHalf, sgOrder, 0, bins, t, w + t * w0);
  else if (t < w0 + w1)
    sg_row(sgdHalf, sgdOrder, 1, bins, t - w0, w + w0 * w0 + (t - w0) * w1);
}

#define STATIC_TRY(call)                                                                                          \
  do {                                                                                                            \
    cudaError_t e_ = (call);                                                                                      \
    if (e_ != cudaSuccess) {                                                                                      \
      snprintf(err, errlen, "b2e_csr_bend_static: %s: %s", #call, cudaGetErrorString(e_));                       \
      return B2E_ERR_CUDA;                                                                                        \
    }                                                                                                             \
  } while (0)

} // namespace b2e

extern "C" int b2e_csr_bend_static(double *const dev_columns[6], int32_t *dev_lost_pass, int32_t *dev_lost_element,
                                   int64_t n, const b2e_element *bend, double p_central, double macro_particle_charge,
                                   double *dev_wakes, int64_t wake_capacity, void *stream, char *errbuf,
                                   int64_t errlen) {
  using namespace b2e;
  char local_err[256];
  char *err = errbuf && errlen > 0 ? errbuf : local_err;
  if (!(errbuf && errlen > 0))
    errlen = sizeof(local_err);
  err[0] = 0;
  /* n = 0 (the set-up call) touches no particle buffer: they may be NULL */
  if (!bend || n < 0 || p_central <= 0 || (n > 0 && (!dev_columns || !dev_lost_pass || !dev_lost_element))) {
    snprintf(err, errlen, "b2e_csr_bend_static: null pointer, negative count or nonpositive p_central");
    return B2E_ERR_ARG;
  }
  for (int c = 0; c < 6 && n > 0; c++)
    if (!dev_columns[c]) {
      snprintf(err, errlen, "b2e_csr_bend_static: column %d is null", c);
      return B2E_ERR_ARG;
    }
  if (n > B2E_STATIC_MAX_PARTICLES) {
    snprintf(err, errlen, "b2e_csr_bend_static: %lld particles exceed the static limit of %d", (long long)n,
             B2E_STATIC_MAX_PARTICLES);
    return B2E_ERR_ARG;
  }
  DevElem d;
  BendExtra bx;
  const char *msg = compile_single_csr_bend(*bend, d, bx);
  if (msg) {
    snprintf(err, errlen, "b2e_csr_bend_static: %s", msg);
    return B2E_ERR_LATTICE;
  }
  const double *p = bend->p;
  const int bins = (int)p[B2E_BEND_BINS], nSlices = (int)d.c[CB_NSLICES];
  if (bins < 2 || bins > B2E_STATIC_MAX_BINS) {
    snprintf(err, errlen, "b2e_csr_bend_static: BINS=%d outside [2, %d]", bins, B2E_STATIC_MAX_BINS);
    return B2E_ERR_ARG;
  }
  int sgHalf = (int)p[B2E_BEND_SG_HALFWIDTH], sgOrder = (int)p[B2E_BEND_SG_ORDER];
  int sgdHalf = (int)p[B2E_BEND_SGDERIV_HALFWIDTH], sgdOrder = (int)p[B2E_BEND_SGDERIV_ORDER];
  if (sgdHalf <= 0)
    sgdHalf = sgHalf;
  if (sgdHalf <= 0)
    sgdHalf = 1;
  if (sgdOrder <= 0)
    sgdOrder = sgOrder;
  if (sgdOrder <= 0)
    sgdOrder = 1;
  if (2 * (sgHalf > sgdHalf ? sgHalf : sgdHalf) + 1 > B2E_SG_MAX_WIDTH) {
    snprintf(err, errlen, "b2e_csr_bend_static: Savitzky-Golay half-width too large");
    return B2E_ERR_ARG;
  }
  if (p[B2E_BEND_IGF] != 0 && p[B2E_BEND_STEADY_STATE] == 0) {
    snprintf(err, errlen, "b2e_csr_bend_static: Must have STEADY_STATE=1 when IGF=1");
    return B2E_ERR_LATTICE;
  }
  if (dev_wakes && wake_capacity < (int64_t)nSlices * bins) {
    snprintf(err, errlen, "b2e_csr_bend_static: wake buffer holds %lld values, %lld needed",
             (long long)wake_capacity, (long long)nSlices * bins);
    return B2E_ERR_ARG;
  }
  StaticCsrScratch *S = static_scratch(err, errlen);
  if (!S)
    return B2E_ERR_CUDA;
  cudaStream_t s = (cudaStream_t)stream;
  DevParticles P;
  P.x = n > 0 ? dev_columns[0] : nullptr;
  P.xp = n > 0 ? dev_columns[1] : nullptr;
  P.y = n > 0 ? dev_columns[2] : nullptr;
  P.yp = n > 0 ? dev_columns[3] : nullptr;
  P.s = n > 0 ? dev_columns[4] : nullptr;
  P.dp = n > 0 ? dev_columns[5] : nullptr;
  P.lost_pass = dev_lost_pass;
  P.lost_elem = dev_lost_element;

  static_set_elem_kernel<<<1, 1, 0, s>>>(d, &S->elem);
  static_sg_weights_kernel<<<1, 2 * B2E_SG_MAX_WIDTH, 0, s>>>(bins, sgHalf, sgOrder, sgdHalf, sgdOrder, S->sg_w);
  STATIC_TRY(cudaGetLastError());
  /* particles alive at the entrance decide whether CSR is computed
   * (csbend.c:1987): counted and turned into the bunch's flags on the device;
   * the histogram and wake kernels do nothing for an inactive bunch */
  STATIC_TRY(cudaMemsetAsync(S->counters, 0, sizeof(S->counters), s));
  STATIC_TRY(launch_effort(dev_lost_pass, n, 0, 0, &S->counters[0], &S->counters[1], s));

  const double Po = p_central;
  const double angle = fabs(p[B2E_BEND_ANGLE]), length = p[B2E_BEND_L], rho0 = d.c[CB_RHO0];
  const double brf = p[B2E_BEND_BIN_RANGE_FACTOR] < 1.1 ? 1.1 : p[B2E_BEND_BIN_RANGE_FACTOR];
  const double eps0 = 1 / ((4 * kPI * 1e-7) * kC * kC);
  double csr_constant = 0;
  if (p[B2E_BEND_CSR] != 0)
    csr_constant = 2 * macro_particle_charge * kE / b2e_pow(3 * rho0 * rho0, 1. / 3.) / (4 * kPI * eps0 * kME * (kC * kC));
  const int g = (int)std::max<int64_t>(1, (n + 255) / 256);
  CsrDevState *dst = &S->state;
  static_set_bunch_kernel<<<1, 1, 0, s>>>(S, csr_constant,
                                          -macro_particle_charge / (kME * (kC * kC)) * length / nSlices);
  CsrBunches B;
  B.offs = nullptr;
  B.n = 1;
  B.st = dst;
  B.csr_const = S->csr_const;
  B.active = &S->flags[0];
  B.mode = &S->flags[1];

  /* the wake kernel's shared-memory limit is a per-function setting that the
   * context path also changes: set it for this call's bin count */
  const size_t wake_smem = sizeof(double) * (5 * bins + 8);
  STATIC_TRY(cudaFuncSetAttribute(csr_wake_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wake_smem));
  csr_entry_kernel<<<g, 256, 0, s>>>(P, n, S->beta0, &S->elem, bx, Po);
  STATIC_TRY(cudaGetLastError());
  double phiBend = 0;
  for (int kick = 0; kick < nSlices; kick++) {
    csr_reset_keys_kernel<<<1, 32, 0, s>>>(B);
    int64_t per_block;
    const int slice_blocks = slice_grid(n, &per_block);
    slice_kernel(d)<<<slice_blocks, SLICE_THREADS, 0, s>>>(P, n, per_block, S->beta0, d, B, kick > 0, bins, Po,
                                                               1 / Po, 0, 0);
    STATIC_TRY(cudaGetLastError());
    STATIC_TRY(cudaMemsetAsync(S->counts, 0, sizeof(unsigned int) * bins, s));
    int hb = hist_blocks(n, 1);
    csr_hist_kernel<<<dim3(hb, 1), 1024, sizeof(unsigned int) * bins, s>>>(P, n, B, S->counts, bins, brf);
    STATIC_TRY(cudaGetLastError());
    phiBend += angle / nSlices;
    double slippage = fabs(rho0 * (phiBend * phiBend * phiBend) / 24.0);
    WakeArgs a = {};
    a.nBins = bins;
    a.sgHalf = sgHalf;
    a.sgdHalf = sgdHalf;
    a.trapz = p[B2E_BEND_TRAPAZOID_INTEGRATION] != 0;
    a.steady = p[B2E_BEND_STEADY_STATE] != 0;
    a.sg_w = S->sg_w;
    a.sgd_w = S->sg_w + sg_width(sgHalf, bins) * sg_width(sgHalf, bins);
    a.slippage = slippage;
    a.slippage13 = b2e_pow(slippage, 1. / 3.);
    a.length = length;
    a.nSlices = nSlices;
    a.c1 = a.c2 = a.csr_constant = 0; /* formed in the kernel from B.csr_const */
    a.wakelog = dev_wakes ? dev_wakes + (size_t)kick * bins : nullptr;
    a.igf = p[B2E_BEND_IGF] != 0;
    set_filter_args(a, p[B2E_BEND_HIGH_FREQUENCY_CUTOFF0] > 0 || p[B2E_BEND_LOW_FREQUENCY_CUTOFF0] >= 0,
                    p[B2E_BEND_CLIP_NEGATIVE_BINS] != 0, p[B2E_BEND_LOW_FREQUENCY_CUTOFF0],
                    p[B2E_BEND_LOW_FREQUENCY_CUTOFF1], p[B2E_BEND_HIGH_FREQUENCY_CUTOFF0],
                    p[B2E_BEND_HIGH_FREQUENCY_CUTOFF1]);
    a.gamma2 = Po * Po + 1;
    a.gamma3 = b2e_pow(a.gamma2, 3. / 2);
    a.rho0 = rho0;
    a.const1 = 6.0 - b2e_log(27.0 / 4.0);
    a.q4pe = kE / (4 * kPI * eps0);
    a.igf_factor = 0;
    csr_wake_kernel<<<1, wake_threads(bins), wake_smem, s>>>(B, S->counts, a, 0);
    STATIC_TRY(cudaGetLastError());
  }
  csr_reset_keys_kernel<<<1, 32, 0, s>>>(B);
  const Sweep sweep = sweep_of(n);
  csr_last_kick_kernel<<<sweep.grid, 256, 0, s>>>(P, n, sweep.share, B, bins, Po, rho0);
  csr_exit_kernel<<<g, 256, 0, s>>>(P, n, &S->elem, bx, B, brf, Po, 0, 0);
  STATIC_TRY(cudaGetLastError());
  STATIC_TRY(launch_post_element_sweep(P, n, nullptr, 0, 0, s));
  return B2E_OK;
}

/* Network inputs of batched profiles (b2e_wake_features), one CTA per
 * profile: the tracking path's feature step (csr_sur_filter_kernel) on
 * bin-unit density and derivative. */
namespace b2e {
__global__ void wake_features_kernel(const double *dens, const double *deriv, const double *slip, int nb,
                                     double sc_dens, double sc_deriv, int shift, float *inputs, double *scales) {
  __shared__ double red[1024];
  const int p = blockIdx.x;
  const double *h = dens + (size_t)p * nb, *d = deriv + (size_t)p * nb;
  float *in = inputs + (size_t)p * 4 * nb;
  double part = 0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    part += h[i];
  double total = block_sum(part, red);
  total = total > 1e-300 ? total : 1e-300;
  part = 0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    const double g = d[i] / total;
    part += g * g;
  }
  const double ms = block_sum(part, red) / nb;
  double k = sqrt(ms);
  k = 1.0 / (k > 1e-300 ? k : 1e-300);
  const double sv = slip[p];
  long long dis = (long long)floor(sv);
  dis = dis < 1 ? 1 : (dis > nb ? nb : dis);
  const float code = (float)(log2((double)dis) / log2((double)nb));
  const double fd = k / total * sc_dens, fg = k / total * sc_deriv;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    in[i] = (float)(h[i] * fd);
    in[nb + i] = (float)(d[i] * fg);
    in[2 * nb + i] = code;
    in[3 * nb + i] = shift && i + dis < nb ? (float)(h[i + dis] * fd) : 0.f;
  }
  if (threadIdx.x == 0) {
    scales[2 * p] = total;
    scales[2 * p + 1] = k;
  }
}

__global__ void wake_t1_kernel(const float *y, const double *scales, const double *slip, int nb, double sc_target,
                               double *t1) {
  const int p = blockIdx.x;
  const double total = scales[2 * p], k = scales[2 * p + 1];
  const bool empty = slip[p] < 1; /* diS = 0: the integral is empty */
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    t1[(size_t)p * nb + i] = empty ? 0.0 : (double)y[(size_t)p * nb + i] / sc_target / k * total;
}
} // namespace b2e

extern "C" int b2e_wake_features(const double *dev_density, const double *dev_derivative,
                                 const double *dev_slippage_bins, int32_t n_profiles, int32_t bins,
                                 double density_scale, double derivative_scale, int32_t shift, float *dev_inputs,
                                 double *dev_scales, void *stream) {
  if (!dev_density || !dev_derivative || !dev_slippage_bins || !dev_inputs || !dev_scales || n_profiles < 0 ||
      bins < 2)
    return B2E_ERR_ARG;
  if (n_profiles == 0)
    return B2E_OK;
  b2e::wake_features_kernel<<<n_profiles, 1024, 0, (cudaStream_t)stream>>>(
      dev_density, dev_derivative, dev_slippage_bins, bins, density_scale, derivative_scale, shift, dev_inputs,
      dev_scales);
  return cudaGetLastError() == cudaSuccess ? B2E_OK : B2E_ERR_CUDA;
}

extern "C" int b2e_wake_t1_from_output(const float *dev_y, const double *dev_scales, const double *dev_slippage_bins,
                                       int32_t n_profiles, int32_t bins, double target_scale, double *dev_t1,
                                       void *stream) {
  if (!dev_y || !dev_scales || !dev_slippage_bins || !dev_t1 || n_profiles < 0 || bins < 2)
    return B2E_ERR_ARG;
  if (n_profiles == 0)
    return B2E_OK;
  b2e::wake_t1_kernel<<<n_profiles, 256, 0, (cudaStream_t)stream>>>(dev_y, dev_scales, dev_slippage_bins, bins,
                                                                   target_scale, dev_t1);
  return cudaGetLastError() == cudaSuccess ? B2E_OK : B2E_ERR_CUDA;
}

/* Batched wake integral for the wake-network data set: n_profiles histograms
 * of `bins` real-valued counts, each with its own slippage in bins. */
using b2e::WakeArgs;
using b2e::BATCH_THREADS;
using b2e::sg_row;
using b2e::sg_width;
using b2e::SG_STAGE;
using b2e::SgTables;
using b2e::static_sg_weights_kernel;
using b2e::wake_batch_kernel;
extern "C" int b2e_csr_wake_batch(const double *dev_counts, const double *dev_slippage_bins, int32_t n_profiles,
                                  int32_t bins, int32_t sg_halfwidth, int32_t sg_order, int32_t sgd_halfwidth,
                                  int32_t sgd_order, int32_t trapezoid, int32_t steady, double *dev_t1,
                                  double *dev_density, double *dev_derivative, void *stream) {
  if (!dev_counts || !dev_slippage_bins || !dev_t1 || !dev_density || !dev_derivative || n_profiles < 0 ||
      bins < 2 || bins > B2E_CSR_MAX_BINS)
    return B2E_ERR_ARG;
  if (sgd_halfwidth <= 0)
    sgd_halfwidth = sg_halfwidth;
  if (sgd_halfwidth <= 0)
    sgd_halfwidth = 1;
  if (sgd_order <= 0)
    sgd_order = sg_order;
  if (sgd_order <= 0)
    sgd_order = 1;
  if (2 * std::max(sg_halfwidth, sgd_halfwidth) + 1 > B2E_SG_MAX_WIDTH)
    return B2E_ERR_ARG;
  if (n_profiles == 0)
    return B2E_OK;
  cudaStream_t s = (cudaStream_t)stream;
  /* windows up to 17 bins: the weights travel as a kernel argument; wider
   * ones through a table in device memory */
  const int w0 = sg_width(sg_halfwidth, bins), w1 = sg_width(sgd_halfwidth, bins);
  SgTables tables = {};
  double *w = nullptr;
  if (w0 * w0 <= SG_STAGE && w1 * w1 <= SG_STAGE) {
    for (int row = 0; row < w0; row++)
      sg_row(sg_halfwidth, sg_order, 0, bins, row, tables.w[0] + row * w0);
    for (int row = 0; row < w1; row++)
      sg_row(sgd_halfwidth, sgd_order, 1, bins, row, tables.w[1] + row * w1);
  } else {
    if (cudaMallocAsync((void **)&w, sizeof(double) * (w0 * w0 + w1 * w1), s) != cudaSuccess)
      return B2E_ERR_NOMEM;
    static_sg_weights_kernel<<<1, 2 * B2E_SG_MAX_WIDTH, 0, s>>>(bins, sg_halfwidth, sg_order, sgd_halfwidth, sgd_order,
                                                                w);
  }
  WakeArgs a = {};
  a.nBins = bins;
  a.sgHalf = sg_halfwidth;
  a.sgdHalf = sgd_halfwidth;
  a.trapz = trapezoid != 0;
  a.steady = steady != 0;
  a.sg_w = w;
  a.sgd_w = w ? w + w0 * w0 : nullptr;
  a.slippage = 0;
  a.slippage13 = 1;
  a.c1 = 1;
  a.c2 = 0;
  a.csr_constant = 1;
  a.wakelog = nullptr;
  a.length = a.nSlices = 1;
  a.igf = 0;
  a.gamma2 = a.gamma3 = a.rho0 = a.const1 = a.q4pe = a.igf_factor = 0;
  const size_t smem = sizeof(double) * (5 * bins + 8);
  cudaError_t e = cudaFuncSetAttribute(wake_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) {
    wake_batch_kernel<<<n_profiles, BATCH_THREADS, smem, s>>>(dev_counts, dev_slippage_bins, a, tables, dev_t1,
                                                              dev_density, dev_derivative);
    e = cudaGetLastError();
  }
  if (w)
    cudaFreeAsync(w, s);
  return e == cudaSuccess ? B2E_OK : B2E_ERR_CUDA;
}
