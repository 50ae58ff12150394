/*
 * Fused multi-pass tracking kernel for the non-collective element subset
 * (DRIF, EDRIFT, KQUAD, KSEXT, CSBEND, RFCA, MAXAMP, MARK, CHARGE).
 *
 * One thread owns one particle for the whole launch: the six coordinates stay
 * in registers across every element of every pass in the launch, so HBM
 * traffic is one 48-byte load and one 48-byte store per particle per launch
 * and the kernel is bound by the FP64 pipe.  This is the B200 replacement for
 * gpuElegant's one-launch-per-element functor kernels
 * (gpu_particle_template_function.hcu:64-86), which re-read and re-write every
 * particle for every element.
 *
 * A thread block tracks one tile (a contiguous run of particles of a single
 * lattice instance), so batched ensembles with uneven particle counts share
 * one launch without mixing instances inside a block.  The instance's
 * compiled elements and apertures are staged in shared memory at block start.
 *
 * Losses: a lost particle records (pass, element) in its loss columns and
 * stops; it keeps its slot (elegant instead swaps lost rows to the tail of the
 * array, do_tracking.c:4584 -- the order of rows is not part of the result,
 * IDs are).
 */
#include <cuda_runtime.h>
#include "b2e_fast.cuh"
#include "b2e_kernels.h"

namespace b2e {



/* Per-pass beam moments of one tile, for the ensemble history: count, means
 * of x, xp, y, yp, then sums of squared deviations (x, xp, xx', y, yp, yy')
 * about the tile means -- two reductions over the tile's four warps in a
 * fixed order, so the result does not depend on scheduling.  Every thread of
 * the block calls it; the 128-thread group g of the block reduces its own
 * tile and writes it to out (when out is not null). */
__device__ __forceinline__ void tile_moments(const Part &p, bool alive, double *out) {
  __shared__ double red_all[8][4][12];
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 3;
  double(*red)[12] = red_all[threadIdx.x >> 7];
  double v[5] = {alive ? 1.0 : 0.0, alive ? p.x : 0.0, alive ? p.xp : 0.0, alive ? p.y : 0.0, alive ? p.yp : 0.0};
  for (int k = 0; k < 5; k++)
    for (int off = 16; off > 0; off >>= 1)
      v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
  if (lane == 0)
    for (int k = 0; k < 5; k++)
      red[warp][k] = v[k];
  __syncthreads();
  double tot[5];
  for (int k = 0; k < 5; k++)
    tot[k] = ((red[0][k] + red[1][k]) + red[2][k]) + red[3][k];
  const double n = tot[0];
  double m[4];
  for (int k = 0; k < 4; k++)
    m[k] = n > 0 ? tot[k + 1] / n : 0.0;
  const double dx = p.x - m[0], dxp = p.xp - m[1], dy = p.y - m[2], dyp = p.yp - m[3];
  double q[6] = {alive ? dx * dx : 0.0,  alive ? dxp * dxp : 0.0, alive ? dx * dxp : 0.0,
                 alive ? dy * dy : 0.0,  alive ? dyp * dyp : 0.0, alive ? dy * dyp : 0.0};
  for (int k = 0; k < 6; k++)
    for (int off = 16; off > 0; off >>= 1)
      q[k] += __shfl_down_sync(0xffffffffu, q[k], off);
  if (lane == 0)
    for (int k = 0; k < 6; k++)
      red[warp][5 + k] = q[k];
  __syncthreads();
  if ((threadIdx.x & 127) == 0 && out) {
    out[0] = n;
    for (int k = 0; k < 4; k++)
      out[1 + k] = m[k];
    for (int k = 0; k < 6; k++)
      out[5 + k] = ((red[0][5 + k] + red[1][5 + k]) + red[2][5 + k]) + red[3][5 + k];
  }
  __syncthreads();
}

/* MINB is the occupancy target (blocks of 128 threads per SM) handed to the
 * register allocator: 4 keeps every value in registers (~118 registers),
 * 5/6/8 trade a few spills to L1 for more resident warps to hide FP64
 * latency.  SYNC sets how often the four warps of a block are brought back
 * in step: 0 never, 1 after every pass, 2 after every element; warps that
 * stay on the same element share its instruction stream and its shared-
 * memory record.  The arithmetic is identical in every variant.  HIST records
 * the per-pass tile moments (it needs SYNC >= 1); when SYNC >= 1 every thread
 * stays in the pass loop until the whole tile is lost.  FAST: magnets of EF_FAST
 * take the straight-line maps and the general ones are called out of line;
 * without it the general maps are in line. */
template <bool STAGED, int MINB, int SYNC, bool HIST, int TPB, bool RAD = false, bool FAST = true>
__global__ void __launch_bounds__(128 * TPB, MINB) ring_kernel(RingLaunch L) {
  static_assert(!HIST || SYNC >= 1, "history needs the per-pass barrier");
  static_assert(TPB == 1 || ((TPB == 2 || TPB == 4 || TPB == 8) && SYNC >= 1), "tiles of a block run in step");
  extern __shared__ __align__(16) unsigned char smem[];
  /* TPB tiles per block, 128 threads each; a missing second tile (odd tile
   * count) leaves its threads idle but inside the barriers */
  const int group = TPB == 1 ? 0 : (int)(threadIdx.x >> 7), lt = threadIdx.x & 127;
  (void)group;
  const int tidx = blockIdx.x * TPB + group;
  DevTile tile = {0, 0, 0};
  if (tidx < L.n_tiles)
    tile = L.tiles[tidx];
  const DevElem *elems = L.elems + (size_t)tile.inst * L.n_elems;
  const DevAperture *aps = L.aps + (size_t)tile.inst * L.n_aps;
  const DevRfState *rf = L.rf + (size_t)tile.inst * L.n_rf;

  if (STAGED) {
    /* stage this tile's instance's element and aperture records in shared memory */
    const size_t stage = sizeof(DevElem) * L.n_elems + sizeof(DevAperture) * L.n_aps;
    DevElem *se = reinterpret_cast<DevElem *>(smem + group * stage);
    DevAperture *sa = reinterpret_cast<DevAperture *>(smem + group * stage + sizeof(DevElem) * L.n_elems);
    const int nw_e = (int)(sizeof(DevElem) * L.n_elems / 8), nw_a = (int)(sizeof(DevAperture) * L.n_aps / 8);
    const double *src_e = reinterpret_cast<const double *>(elems);
    const double *src_a = reinterpret_cast<const double *>(aps);
    double *dst_e = reinterpret_cast<double *>(se), *dst_a = reinterpret_cast<double *>(sa);
    for (int i = lt; i < nw_e; i += 128)
      dst_e[i] = src_e[i];
    for (int i = lt; i < nw_a; i += 128)
      dst_a[i] = src_a[i];
    __syncthreads();
    elems = se;
    aps = sa;
  }

  const int64_t ip = tile.start + lt;
  const bool tracked = lt < tile.count && L.P.lost_pass[ip] < 0;
  if (SYNC == 0 && !tracked)
    return;

  Part p = {0, 0, 0, 0, 0, 0};
  if (tracked) {
    p.x = L.P.x[ip];
    p.xp = L.P.xp[ip];
    p.y = L.P.y[ip];
    p.yp = L.P.yp[ip];
    p.s = L.P.s[ip];
    p.dp = L.P.dp[ip];
  }

  int lost = LOSS_NONE, lost_pass = -1, lost_elem = -1;
  bool active = tracked;
  RadSite rs = {0, 0, 0, 0, 0, nullptr};
  const DevRad *rads = RAD ? L.rads + (size_t)tile.inst * L.n_elems : nullptr;
  if (RAD) {
    rs.id = tracked ? (L.ids ? L.ids[ip] : ip + 1) : 0;
    rs.seed = L.isr_seed;
    rs.limit = L.sr_limit;
  }
  for (int pass = L.pass_begin; pass <= L.pass_end; pass++) {
    if (SYNC == 0) {
      if (!active)
        break;
    } else if (!__syncthreads_or(active)) {
      break; /* the whole tile is lost (history slots stay zero: no survivors) */
    }
    const int e0 = pass == L.pass_begin ? L.elem_begin : 0;
    const int e1 = pass == L.pass_end ? L.elem_end : L.n_elems;
    for (int ie = e0; ie < e1; ie++) {
      if (SYNC == 2)
        __syncthreads();
      if (!active) {
        if (SYNC == 2)
          continue;
        break;
      }
      const DevElem &e = elems[ie];
      const int iap = pass == 0 ? e.ap_pass0 : e.ap_later;
      const DevAperture *ap = iap >= 0 ? &aps[iap] : nullptr;
      switch (e.kind) {
      case K_DRIF_O2:
        drif_o2(p, e);
        break;
      case K_DRIF_O1:
        drif_o1(p, e);
        break;
      case K_EDRIFT:
        edrift(p, e.c[DR_L]);
        break;
      case K_KMULT:
        if (RAD) {
          rs.pass = pass;
          rs.elem = ie;
          rs.rc = rads[ie].c;
        }
        if constexpr (!FAST)
          lost = kmult<RAD>(p, e, ap, L.g, rs);
        else if (!((e.flags & EF_FAST) && (RAD && (e.flags & EF_SR) ? kmult_fast<true>(p, e, ap, L.g, rs.rc)
                                                                    : kmult_fast<false>(p, e, ap, L.g, nullptr))))
          lost = kmult_general<RAD>(p, e, ap, L.g, rs);
        break;
      case K_CSBEND:
        if (RAD) {
          rs.pass = pass;
          rs.elem = ie;
          rs.rc = rads[ie].c;
        }
        if constexpr (!FAST)
          lost = csbend<RAD>(p, e, ap, L.g, rs);
        else if (!((e.flags & EF_FAST) && (RAD && (e.flags & EF_SR) ? csbend_fast<true>(p, e, ap, L.g, rs.rc)
                                                                    : csbend_fast<false>(p, e, ap, L.g, nullptr))))
          lost = csbend_general<RAD>(p, e, ap, L.g, rs);
        break;
      case K_MALIGN: {
        const double *mc = e.c;
        const int on_pass = (int)mc[MA_ON_PASS];
        if (on_pass == -1 || on_pass == pass) {
          bool hit = true;
          if (mc[MA_START_PID] >= 0) {
            const double id = (double)(L.ids ? L.ids[ip] : ip + 1);
            hit = !(id < mc[MA_START_PID] || id > mc[MA_END_PID]);
          }
          if (hit)
            malign(p, mc, L.g.p_central);
        }
        break;
      }
      case K_RFCA: {
        const DevRfState rs = rf[(int)e.c[RF_SLOT]];
        if (!rs.set) {
          /* the host runs the fiducial pass before any launch that needs it */
          atomicOr(L.error_flag, 1u);
          lost = LOSS_ENERGY;
        } else
          lost = rfca(p, e, rs, L.g);
        break;
      }
      default: /* MARK, CHARGE, WATCH (recorded between launches) */
        break;
      }
      if (!lost && !(ap && ap_surely_inside(p.x, p.y, ap))) {
        if (!(e.flags & EF_NO_APERTURE) && ap && !maxamp_ok(p, *ap))
          lost = LOSS_APERTURE;
        else if (!finite_xy(p))
          lost = LOSS_NAN;
      }
      if (lost) {
        lost_pass = pass;
        lost_elem = ie;
        active = false;
      }
    }
    if (L.tbt && active && e1 == L.n_elems) {
      const int r = pass - L.tbt_pass0 + 1;
      if (r >= 1 && r < L.tbt_records) {
        double *o = L.tbt + (size_t)r * 4 * L.tbt_rows + ip;
        o[0] = p.x;
        o[L.tbt_rows] = p.xp;
        o[2 * L.tbt_rows] = p.y;
        o[3 * L.tbt_rows] = p.yp;
      }
    }
    if (HIST && e1 == L.n_elems && pass >= L.hist_pass0)
      tile_moments(p, active,
                   tidx < L.n_tiles ? L.hist + ((size_t)tidx * L.hist_passes + (pass - L.hist_pass0)) * 11 : nullptr);
  }

  if (!tracked)
    return;
  L.P.x[ip] = p.x;
  L.P.xp[ip] = p.xp;
  L.P.y[ip] = p.y;
  L.P.yp[ip] = p.yp;
  L.P.s[ip] = p.s;
  L.P.dp[ip] = p.dp;
  if (lost) {
    L.P.lost_pass[ip] = lost_pass;
    L.P.lost_elem[ip] = lost_elem;
  }
}

/* Ensemble history: merge the tiles of each instance, pass by pass, in tile
 * order with the pairwise update of Chan, Golub & LeVeque (1979) for means
 * and co-moments; rms emittance as rms_emittance (final_props.c:844-880):
 * sqrt(Sxx Sx'x' - Sxx'^2)/n.  out[inst][pass][5] = survivors, <x>, <y>,
 * emittance x, emittance y. */
__global__ void history_merge_kernel(const double *partials, int hist_passes, const int *tile_first, int n_inst,
                                     double *out) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_inst * hist_passes)
    return;
  const int inst = idx / hist_passes, j = idx - inst * hist_passes;
  double n = 0, m[4] = {0, 0, 0, 0}, S[6] = {0, 0, 0, 0, 0, 0};
  for (int t = tile_first[inst]; t < tile_first[inst + 1]; t++) {
    const double *b = partials + ((size_t)t * hist_passes + j) * 11;
    const double nb = b[0];
    if (nb == 0)
      continue;
    if (n == 0) {
      n = nb;
      for (int k = 0; k < 4; k++)
        m[k] = b[1 + k];
      for (int k = 0; k < 6; k++)
        S[k] = b[5 + k];
      continue;
    }
    const double N = n + nb, w = n * nb / N;
    double d[4];
    for (int k = 0; k < 4; k++)
      d[k] = b[1 + k] - m[k];
    S[0] += b[5] + d[0] * d[0] * w;
    S[1] += b[6] + d[1] * d[1] * w;
    S[2] += b[7] + d[0] * d[1] * w;
    S[3] += b[8] + d[2] * d[2] * w;
    S[4] += b[9] + d[3] * d[3] * w;
    S[5] += b[10] + d[2] * d[3] * w;
    for (int k = 0; k < 4; k++)
      m[k] += d[k] * nb / N;
    n = N;
  }
  double *o = out + (size_t)idx * 5;
  o[0] = n;
  o[1] = m[0];
  o[2] = m[2];
  double ex = S[0] * S[1] - S[2] * S[2], ey = S[3] * S[4] - S[5] * S[5];
  o[3] = n > 0 ? (ex > 0 ? sqrt(ex) : 0) / n : 0;
  o[4] = n > 0 ? (ey > 0 ? sqrt(ey) : 0) / n : 0;
}

cudaError_t launch_history_merge(const double *partials, int hist_passes, const int *tile_first, int n_inst,
                                 double *out, cudaStream_t stream) {
  const int total = n_inst * hist_passes;
  if (total <= 0)
    return cudaSuccess;
  history_merge_kernel<<<(total + 127) / 128, 128, 0, stream>>>(partials, hist_passes, tile_first, n_inst, out);
  return cudaGetLastError();
}

/* RFCA fiducial time (findFiducialTime, simple_rfca.c:62-257).  TMEAN:
 * Kahan-compensated mean of (s + sOffset)/(c*beta) over the particles that
 * reach the cavity on the first pass, in particle order (the reference's
 * serial sum, bit for bit, when no particle was lost upstream on that pass;
 * elegant's swap-to-tail would otherwise reorder the survivors).  LIGHT:
 * (zEnd - L + sOffset)/c (:97-100).  PMAXIMUM (:126-147): the arrival time of
 * the particle with the highest delta, found as the reference's loop does: the
 * first particle's delta is the starting best and only a later, strictly
 * higher one is taken, so a beam whose first particle is highest has no
 * fiducial particle (the reference stops there; here bit 2 of the error flag
 * is set and the cavity stays unset).
 *
 * The Kahan sum in parallel.  Let all n terms be positive and of one binade,
 * integers m_i q with q their common ulp.  Each step forms Y = b + error, sum =
 * RN(tsum + Y) and error = tsum + Y - sum exactly (Fast2Sum: tsum has at least
 * Y's exponent).  |error| is at most half an ulp of the sum, no more than n q,
 * so while m_i <= 2^53 - 2n, Y too is an exact integer multiple of q below
 * 2^53 q.  Nothing is then rounded away, sum + error is the exact sum of the
 * terms so far, and sum is that sum rounded to nearest even: the result is
 * RN(q sum m_i), an integer sum that any order gives.  Arrival times of a bunch
 * behind the first metres of a line nearly always qualify; where they do not,
 * one thread runs the reference's loop on tiles of terms formed by the block.
 * 11 us for 10,000 particles; 28 ns a particle in the loop, 400 ns with the two
 * divisions and the square root of each term inside it. */
struct FidAcc {
  unsigned long long lo, hi; /* sums of the significands' low 32 bits and of the rest */
  unsigned long long n, done, m_max;
  unsigned int e_max, e_min_c; /* largest exponent field; 2047 less the smallest */
};

__device__ __forceinline__ double arrival_time(const DevParticles &P, int64_t ip, double sOffset, double p_central) {
  const double pp = p_central * (1 + P.dp[ip]);
  const double beta = pp / sqrt(pp * pp + 1); /* beta_from_delta, do_tracking.c:95 */
  return (P.s[ip] + sOffset) / (B2E_C_MKS * beta);
}

/* v 2^scale rounded to nearest even */
__device__ double round_u128(unsigned __int128 v, int scale) {
  int bits = 0;
  for (unsigned __int128 t = v; t; t >>= 1)
    bits++;
  if (bits > 53) {
    const int sh = bits - 53;
    const unsigned __int128 rest = v & (((unsigned __int128)1 << sh) - 1), half = (unsigned __int128)1 << (sh - 1);
    v >>= sh;
    if (rest > half || (rest == half && (v & 1)))
      v++;
    scale += sh;
  }
  return ldexp((double)(unsigned long long)v, scale);
}

__device__ void fiducial_set(DevRfState &rs, const DevElem &e, double tsum, int64_t nsum) {
  if (nsum > 0) {
    const double omega = e.c[RF_OMEGA];
    const double t0 = tsum / nsum, phase_fiducial = -omega * t0;
    rs.phase_fiducial = phase_fiducial;
    rs.phase = phase_fiducial + e.c[RF_PHASE_DEG_RAD];
    rs.set = 1;
  } else {
    rs.set = 0;
  }
}

/* cavities that need no sum: a group's later members, an explicit T_REFERENCE,
 * LIGHT and PMAXIMUM */
__device__ void fiducial_without_sum(const DevParticles &P, int64_t first, int64_t end, const DevElem &e, int mode,
                                     DevRfState *rf, DevRfState &rs, double p_central, unsigned int *error_flag) {
  const int leader = (int)e.c[RF_LEADER];
  if (leader >= 0) {
    /* a later cavity of a PHASE_REFERENCE group: the group's phase
     * (REF_PHASE_RETURNED, simple_rfca.c:419-421) plus its own PHASE */
    rs.phase_fiducial = rf[leader].phase_fiducial;
    rs.phase = rf[leader].phase_fiducial + e.c[RF_PHASE_DEG_RAD];
    rs.set = rf[leader].set;
    return;
  }
  double tsum = 0;
  int64_t nsum = 0;
  if (e.c[RF_T_REFERENCE] != -1) {
    /* explicit T_REFERENCE replaces the fiducial search */
    tsum = e.c[RF_T_REFERENCE];
    nsum = 1;
  } else if (mode == B2E_FIDUCIAL_LIGHT) {
    tsum = ((e.z_end - e.c[RF_L_TOTAL]) + e.c[RF_SOFFSET]) / B2E_C_MKS;
    nsum = 1;
  } else {
    double best = 0;
    int64_t ibest = -1;
    bool seen = false;
    for (int64_t ip = first; ip < end; ip++) {
      if (P.lost_pass[ip] >= 0)
        continue;
      if (!seen) {
        best = P.dp[ip];
        seen = true;
      } else if (best < P.dp[ip]) {
        best = P.dp[ip];
        ibest = ip;
      }
    }
    if (ibest >= 0) {
      tsum = arrival_time(P, ibest, e.c[RF_SOFFSET], p_central);
      nsum = 1;
    } else if (seen) {
      atomicOr(error_flag, 2u);
    }
  }
  fiducial_set(rs, e, tsum, nsum);
}

/* gx blocks per instance; the last one to finish its share forms the result.
 * acc: one zeroed record per instance.  A block of one warp takes a whole
 * instance (gx = 1) and needs none. */
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
    rf_fiducial_kernel(DevParticles P, const int64_t *inst_offsets, int gx, const DevElem *elems, int n_elems,
                       int elem_index, DevRfState *rf, int n_rf, double p_central, int64_t max_rows, FidAcc *acc_all,
                       unsigned int *error_flag) {
  constexpr int TILE = 4 * THREADS;
  __shared__ double tile[TILE];
  const int inst = blockIdx.x / gx, part = blockIdx.x - inst * gx;
  const DevElem &e = elems[(size_t)inst * n_elems + elem_index];
  DevRfState *rf_inst = rf + (size_t)inst * n_rf;
  DevRfState &rs = rf_inst[(int)e.c[RF_SLOT]];
  const int64_t first = inst_offsets[inst];
  int64_t end = inst_offsets[inst + 1];
  if (max_rows > 0 && end - first > max_rows)
    end = first + max_rows;
  const int mode = (int)e.c[RF_FID_MODE];
  if (e.c[RF_LEADER] >= 0 || e.c[RF_T_REFERENCE] != -1 || mode == B2E_FIDUCIAL_LIGHT ||
      mode == B2E_FIDUCIAL_PMAXIMUM) {
    if (part == 0 && threadIdx.x == 0)
      fiducial_without_sum(P, first, end, e, mode, rf_inst, rs, p_central, error_flag);
    return;
  }
  const double sOffset = e.c[RF_SOFFSET];
  FidAcc a = {0, 0, 0, 0, 0, 0, 0};
  for (int64_t ip = first + part * THREADS + threadIdx.x; ip < end; ip += (int64_t)gx * THREADS) {
    if (P.lost_pass[ip] >= 0)
      continue;
    const unsigned long long bits = (unsigned long long)__double_as_longlong(arrival_time(P, ip, sOffset, p_central));
    const unsigned long long m = (bits & 0xfffffffffffffull) | 0x10000000000000ull;
    const unsigned int ex = (unsigned int)(bits >> 52); /* with the sign: beyond 2047 for a negative term */
    a.lo += m & 0xffffffffull;
    a.hi += m >> 32;
    a.n++;
    a.m_max = max(a.m_max, m);
    a.e_max = max(a.e_max, ex);
    a.e_min_c = max(a.e_min_c, 2047u - min(ex, 2047u));
  }
  for (int off = 16; off > 0; off >>= 1) {
    a.lo += __shfl_down_sync(0xffffffffu, a.lo, off);
    a.hi += __shfl_down_sync(0xffffffffu, a.hi, off);
    a.n += __shfl_down_sync(0xffffffffu, a.n, off);
    a.m_max = max(a.m_max, __shfl_down_sync(0xffffffffu, a.m_max, off));
    a.e_max = max(a.e_max, __shfl_down_sync(0xffffffffu, a.e_max, off));
    a.e_min_c = max(a.e_min_c, __shfl_down_sync(0xffffffffu, a.e_min_c, off));
  }
  if constexpr (THREADS > 32) {
    __shared__ int last;
    FidAcc *acc = acc_all + inst;
    if ((threadIdx.x & 31) == 0 && a.n) {
      atomicAdd(&acc->lo, a.lo);
      atomicAdd(&acc->hi, a.hi);
      atomicAdd(&acc->n, a.n);
      atomicMax(&acc->m_max, a.m_max);
      atomicMax(&acc->e_max, a.e_max);
      atomicMax(&acc->e_min_c, a.e_min_c);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
      last = atomicAdd(&acc->done, 1ull) == (unsigned long long)(gx - 1);
    __syncthreads();
    if (!last)
      return;
    __threadfence();
    a.lo = __ldcg(&acc->lo);
    a.hi = __ldcg(&acc->hi);
    a.n = __ldcg(&acc->n);
    a.m_max = __ldcg(&acc->m_max);
    a.e_max = __ldcg(&acc->e_max);
    a.e_min_c = __ldcg(&acc->e_min_c);
  }
  /* one warp has its sums in lane 0; otherwise every thread has them */
  const unsigned long long n = THREADS > 32 ? a.n : __shfl_sync(0xffffffffu, a.n, 0);
  const bool exact = n && n < (1ull << 31) && a.e_max + a.e_min_c == 2047u && a.e_max > 100 && a.e_max < 1900 &&
                     a.m_max <= (1ull << 53) - 2 * n;
  if (THREADS > 32 ? exact : __shfl_sync(0xffffffffu, exact, 0)) {
    if (threadIdx.x == 0)
      fiducial_set(rs, e, round_u128(((unsigned __int128)a.hi << 32) + a.lo, (int)a.e_max - 1075), (int64_t)n);
    return;
  }
  double tsum = 0, error = 0;
  for (int64_t t0 = first; t0 < end; t0 += TILE) {
    const int len = (int)min((int64_t)TILE, end - t0);
    for (int k = threadIdx.x; k < len; k += THREADS)
      tile[k] = P.lost_pass[t0 + k] < 0 ? arrival_time(P, t0 + k, sOffset, p_central) : 0.0;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int k = 0; k < len; k++) {
        if (P.lost_pass[t0 + k] >= 0)
          continue;
        /* KahanPlus (kahan.c:28-35) */
        const double Y = tile[k] + error, sum = tsum + Y;
        error = Y - (sum - tsum);
        tsum = sum;
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    fiducial_set(rs, e, tsum, (int64_t)n);
}

/* Effort (particle-passes) and survivor count from the loss columns. */
__global__ void effort_kernel(const int32_t *lost_pass, int64_t n, int pass_begin, int pass_end, unsigned long long *effort,
                              unsigned long long *survivors) {
  unsigned long long e = 0, s = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int lp = lost_pass[i];
    int alive = lp < 0 ? pass_end - pass_begin : lp - pass_begin;
    e += (unsigned long long)(alive < 0 ? 0 : (alive > pass_end - pass_begin ? pass_end - pass_begin : alive));
    s += lp < 0;
  }
  for (int off = 16; off > 0; off >>= 1) {
    e += __shfl_down_sync(0xffffffffu, e, off);
    s += __shfl_down_sync(0xffffffffu, s, off);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(effort, e);
    atomicAdd(survivors, s);
  }
}

template <int MINB, int SYNC, bool HIST, int TPB, bool RAD = false, bool FAST = true>
static cudaError_t launch_ring_v(const RingLaunch &L, int n_tiles, bool staged, size_t smem_bytes,
                                 cudaStream_t stream) {
  const int grid = (n_tiles + TPB - 1) / TPB;
  if (staged && smem_bytes * TPB > 200 * 1024)
    staged = false; /* two instances' records do not fit: read them from global memory */
  if (staged) {
    const size_t bytes = smem_bytes * TPB;
    cudaError_t err = cudaFuncSetAttribute(ring_kernel<true, MINB, SYNC, HIST, TPB, RAD, FAST>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (err != cudaSuccess)
      return err;
    ring_kernel<true, MINB, SYNC, HIST, TPB, RAD, FAST><<<grid, 128 * TPB, bytes, stream>>>(L);
  } else {
    ring_kernel<false, MINB, SYNC, HIST, TPB, RAD, FAST><<<grid, 128 * TPB, 0, stream>>>(L);
  }
  return cudaGetLastError();
}

template <int SYNC, bool HIST>
static cudaError_t launch_ring_s(const RingLaunch &L, int n_tiles, bool staged, size_t smem_bytes,
                                 cudaStream_t stream, int minb_index) {
  switch (minb_index) {
  case 1:
    return launch_ring_v<5, SYNC, HIST, 1>(L, n_tiles, staged, smem_bytes, stream);
  case 2:
    return launch_ring_v<6, SYNC, HIST, 1>(L, n_tiles, staged, smem_bytes, stream);
  case 3:
    return launch_ring_v<8, SYNC, HIST, 1>(L, n_tiles, staged, smem_bytes, stream);
  default:
    return launch_ring_v<4, SYNC, HIST, 1>(L, n_tiles, staged, smem_bytes, stream);
  }
}

template <bool HIST>
static cudaError_t launch_ring_group(const RingLaunch &L, int n_tiles, bool staged, size_t smem_bytes,
                                     cudaStream_t stream, int index) {
  switch (index) {
  case 1:
    return launch_ring_v<3, 2, HIST, 2>(L, n_tiles, staged, smem_bytes, stream);
  case 2:
    return launch_ring_v<4, 2, HIST, 2>(L, n_tiles, staged, smem_bytes, stream);
  case 3:
    return launch_ring_v<2, 2, HIST, 4>(L, n_tiles, staged, smem_bytes, stream);
  case 4:
    return launch_ring_v<1, 2, HIST, 8>(L, n_tiles, staged, smem_bytes, stream);
  default:
    return launch_ring_v<2, 2, HIST, 2>(L, n_tiles, staged, smem_bytes, stream);
  }
}

/* variant 1..12: one 128-particle tile per block, occupancy target MINB =
 * {4, 5, 6, 8}[(variant-1) % 4] blocks per SM, barrier level SYNC =
 * (variant-1) / 4 (with history at least 1).  Variants 13..17 keep several
 * tiles of a block in step with a barrier after every element: two tiles per
 * 256-thread block at {2, 3, 4} blocks per SM, four tiles per 512-thread
 * block at 2, eight tiles per 1024-thread block at 1. */
cudaError_t launch_ring(const RingLaunch &L, int n_tiles, bool staged, size_t smem_bytes, cudaStream_t stream,
                        int variant) {
  if (n_tiles <= 0)
    return cudaSuccess;
  if (L.rad) { /* radiating lattices: one configuration (two tiles per block, a barrier per element) */
    /* Without a single straight-line magnet the general maps are in line: out
     * of line they keep the particle and the constants' addresses in memory,
     * 4 to 6 % of a turn.  Quantum excitation everywhere, 10 turns of 200
     * particles 16.1 -> 15.2 ms, an ensemble of 256 instances 56.2 -> 51.0 ms for
     * 3 turns; field terms and steering 3.54 -> 3.26 ms.  One magnet in twenty of
     * the other kind makes up for it: a straight-line map takes less than half of
     * the time. */
    if (!L.fast)
      return L.hist ? launch_ring_v<2, 2, true, 2, true, false>(L, n_tiles, staged, smem_bytes, stream)
                    : launch_ring_v<2, 2, false, 2, true, false>(L, n_tiles, staged, smem_bytes, stream);
    return L.hist ? launch_ring_v<2, 2, true, 2, true>(L, n_tiles, staged, smem_bytes, stream)
                  : launch_ring_v<2, 2, false, 2, true>(L, n_tiles, staged, smem_bytes, stream);
  }
  if (variant < 1 || variant > B2E_RING_VARIANTS)
    variant = 1;
  if (variant > 12)
    return L.hist ? launch_ring_group<true>(L, n_tiles, staged, smem_bytes, stream, variant - 13)
                  : launch_ring_group<false>(L, n_tiles, staged, smem_bytes, stream, variant - 13);
  const int minb_index = (variant - 1) % 4, sync = (variant - 1) / 4;
  if (L.hist)
    return sync == 2 ? launch_ring_s<2, true>(L, n_tiles, staged, smem_bytes, stream, minb_index)
                     : launch_ring_s<1, true>(L, n_tiles, staged, smem_bytes, stream, minb_index);
  switch (sync) {
  case 1:
    return launch_ring_s<1, false>(L, n_tiles, staged, smem_bytes, stream, minb_index);
  case 2:
    return launch_ring_s<2, false>(L, n_tiles, staged, smem_bytes, stream, minb_index);
  default:
    return launch_ring_s<0, false>(L, n_tiles, staged, smem_bytes, stream, minb_index);
  }
}

/* Stable partition of every instance's particles: survivors first, in their
 * order, lost particles after them (last to first).  One block per instance
 * walks its range in chunks of blockDim particles; a warp ballot gives each
 * particle its rank among its warp's survivors (or losses) and a scan over
 * the block's warp totals the chunk offsets (lost-particle compaction with
 * warp ballots and prefix sums). */
__global__ void compact_kernel(DevParticles src, const int64_t *ids_src, DevParticles dst, int64_t *ids_dst,
                               const int64_t *offs, int *alive_out) {
  __shared__ int warp_alive[32], warp_dead[32];
  __shared__ int base_alive, base_dead;
  const int inst = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int64_t first = offs[inst], end = offs[inst + 1];
  if (threadIdx.x == 0) {
    base_alive = 0;
    base_dead = 0;
  }
  __syncthreads();
  const unsigned below = (1u << lane) - 1u;
  for (int64_t c = first; c < end; c += blockDim.x) {
    const int64_t i = c + threadIdx.x;
    const bool valid = i < end;
    const bool alive = valid && src.lost_pass[i] < 0;
    const unsigned ba = __ballot_sync(0xffffffffu, alive), bd = __ballot_sync(0xffffffffu, valid && !alive);
    if (lane == 0) {
      warp_alive[warp] = __popc(ba);
      warp_dead[warp] = __popc(bd);
    }
    __syncthreads();
    int pa = 0, pd = 0, ta = 0, td = 0;
    for (int w = 0; w < nw; w++) {
      if (w < warp) {
        pa += warp_alive[w];
        pd += warp_dead[w];
      }
      ta += warp_alive[w];
      td += warp_dead[w];
    }
    if (valid) {
      const int64_t d = alive ? first + base_alive + pa + __popc(ba & below)
                              : end - 1 - (base_dead + pd + __popc(bd & below));
      dst.x[d] = src.x[i];
      dst.xp[d] = src.xp[i];
      dst.y[d] = src.y[i];
      dst.yp[d] = src.yp[i];
      dst.s[d] = src.s[i];
      dst.dp[d] = src.dp[i];
      dst.lost_pass[d] = src.lost_pass[i];
      dst.lost_elem[d] = src.lost_elem[i];
      ids_dst[d] = ids_src[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      base_alive += ta;
      base_dead += td;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    alive_out[inst] = base_alive;
}

cudaError_t launch_compact(DevParticles src, const int64_t *ids_src, DevParticles dst, int64_t *ids_dst,
                           const int64_t *offs, int n_inst, int *alive_out, cudaStream_t stream) {
  if (n_inst <= 0)
    return cudaSuccess;
  compact_kernel<<<n_inst, 1024, 0, stream>>>(src, ids_src, dst, ids_dst, offs, alive_out);
  return cudaGetLastError();
}

size_t fiducial_scratch_bytes(int n_inst) { return sizeof(FidAcc) * (size_t)n_inst; }

cudaError_t launch_fiducial(DevParticles P, const int64_t *inst_offsets, int n_inst, int64_t n, const DevElem *elems,
                            int n_elems, int elem_index, DevRfState *rf, int n_rf, double p_central,
                            int64_t max_rows, void *scratch, unsigned int *error_flag, cudaStream_t stream) {
  if (n_inst <= 0)
    return cudaSuccess;
  /* blocks per instance: one per 1,024 rows of an average instance, at most
   * four per SM over all instances */
  int64_t rows = n / n_inst;
  if (max_rows > 0 && rows > max_rows)
    rows = max_rows;
  int64_t gx = (rows + 1023) / 1024, cap = 148 * 4 / n_inst;
  gx = gx > cap ? cap : gx;
  gx = gx < 1 ? 1 : gx;
  /* instances of a few particles: a warp each, without the zeroed records and
   * their atomics.  Whole calls of 20,000 instances of three: 316 us with blocks
   * of 256 threads, 216 so; 3,000 of 64: 119 and 99 us. */
  if (rows <= 64) {
    rf_fiducial_kernel<32><<<(unsigned)n_inst, 32, 0, stream>>>(P, inst_offsets, 1, elems, n_elems, elem_index, rf,
                                                                n_rf, p_central, max_rows, nullptr, error_flag);
    return cudaGetLastError();
  }
  cudaError_t err = cudaMemsetAsync(scratch, 0, fiducial_scratch_bytes(n_inst), stream);
  if (err != cudaSuccess)
    return err;
  rf_fiducial_kernel<256><<<(unsigned)(gx * n_inst), 256, 0, stream>>>(P, inst_offsets, (int)gx, elems, n_elems,
                                                                       elem_index, rf, n_rf, p_central, max_rows,
                                                                       (FidAcc *)scratch, error_flag);
  return cudaGetLastError();
}

__global__ void tbt_start_kernel(DevParticles P, int64_t n, double *tbt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const bool live = P.lost_pass[i] < 0;
  tbt[i] = live ? P.x[i] : NAN;
  tbt[n + i] = live ? P.xp[i] : NAN;
  tbt[2 * n + i] = live ? P.y[i] : NAN;
  tbt[3 * n + i] = live ? P.yp[i] : NAN;
}

/* WATCH record of the particles alive at a WATCH element (the ring launches
 * stop there on its passes): x..delta and the ID as a double, NaN (left from
 * the fill) in the rows of lost particles. */
__global__ void watch_copy_kernel(DevParticles P, const int64_t *ids, int64_t n, double *out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || P.lost_pass[i] >= 0)
    return;
  out[i] = P.x[i];
  out[n + i] = P.xp[i];
  out[2 * n + i] = P.y[i];
  out[3 * n + i] = P.yp[i];
  out[4 * n + i] = P.s[i];
  out[5 * n + i] = P.dp[i];
  out[6 * n + i] = (double)(ids ? ids[i] : i + 1);
}

cudaError_t launch_watch_copy(DevParticles P, const int64_t *ids, int64_t n, double *out, cudaStream_t stream) {
  if (n <= 0)
    return cudaSuccess;
  watch_copy_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(P, ids, n, out);
  return cudaGetLastError();
}

cudaError_t launch_tbt_start(DevParticles P, int64_t n, double *tbt, cudaStream_t stream) {
  if (n > 0)
    tbt_start_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(P, n, tbt);
  return cudaGetLastError();
}

cudaError_t launch_effort(const int32_t *lost_pass, int64_t n, int pass_begin, int pass_end, unsigned long long *effort,
                          unsigned long long *survivors, cudaStream_t stream) {
  int nb = (int)((n + 255) / 256);
  if (nb > 148 * 8)
    nb = 148 * 8;
  if (nb < 1)
    nb = 1;
  effort_kernel<<<nb, 256, 0, stream>>>(lost_pass, n, pass_begin, pass_end, effort, survivors);
  return cudaGetLastError();
}

} // namespace b2e

/* ---- division self-test (b2e_selftest_division) ------------------------- */
namespace b2e {

__global__ void division_selftest_kernel(const double *b, int nb, int64_t samples, uint64_t seed,
                                         unsigned long long *mismatches) {
  const int ib = blockIdx.y;
  const double bv = b[ib], y = 1 / bv;
  unsigned long long bad = 0;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < samples; k += (int64_t)gridDim.x * blockDim.x) {
    /* SplitMix64 of (seed, divisor, sample) -> sign, exponent, mantissa */
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(k * nb + ib + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const int ex = (int)((z >> 52) % 81) - 40;
    const double m = 1.0 + (double)(z & ((1ull << 52) - 1)) * 0x1p-52;
    const double a = ldexp((z >> 63) ? -m : m, ex);
    const double q1 = a / bv, q2 = div_rn_recip(a, bv, y);
    bad += __double_as_longlong(q1) != __double_as_longlong(q2);
  }
  for (int off = 16; off > 0; off >>= 1)
    bad += __shfl_down_sync(0xffffffffu, bad, off);
  if ((threadIdx.x & 31) == 0 && bad)
    atomicAdd(mismatches, bad);
}

} // namespace b2e

extern "C" int b2e_selftest_division(const double *host_b, int32_t n_b, int64_t samples, uint64_t seed,
                                     int64_t *mismatches) {
  using namespace b2e;
  if (!host_b || n_b < 1 || n_b > 65535 || samples < 1 || !mismatches)
    return B2E_ERR_ARG;
  double *db = nullptr;
  unsigned long long *dm = nullptr, hm = 0;
  if (cudaMalloc(&db, sizeof(double) * n_b) != cudaSuccess)
    return B2E_ERR_NOMEM;
  if (cudaMalloc(&dm, sizeof(unsigned long long)) != cudaSuccess) {
    cudaFree(db);
    return B2E_ERR_NOMEM;
  }
  cudaMemcpy(db, host_b, sizeof(double) * n_b, cudaMemcpyHostToDevice);
  cudaMemset(dm, 0, sizeof(unsigned long long));
  division_selftest_kernel<<<dim3(148 * 4, n_b), 256>>>(db, n_b, samples, seed, dm);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpy(&hm, dm, sizeof(hm), cudaMemcpyDeviceToHost);
  cudaFree(db);
  cudaFree(dm);
  if (e != cudaSuccess)
    return B2E_ERR_CUDA;
  *mismatches = (int64_t)hm;
  return B2E_OK;
}

/* ---- rounding self-test (b2e_selftest_rounding) ------------------------- */
namespace b2e {

__device__ __forceinline__ uint64_t rounding_hash(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; /* SplitMix64 */
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

/* an operand of one of four kinds: any significand over 60 binades, up to 2^40
 * ulp either side of 1, the same around a power of two, and a short
 * significand (exact quotients and squares) */
__device__ __forceinline__ double rounding_operand(uint64_t z, int kind) {
  const double m = __longlong_as_double((long long)(0x3ff0000000000000ull | (z >> 12)));
  const int ex = (int)(z % 61) - 30;
  const long long k = (long long)((z >> 20) >> (z % 41)); /* log-uniform below 2^44 */
  switch (kind) {
  case 0:
    return ldexp(m, ex);
  case 1:
    return __longlong_as_double(0x3ff0000000000000ll + ((z & 64) ? k >> 4 : -(k >> 4)));
  case 2:
    return ldexp(__longlong_as_double(0x3ff0000000000000ll + ((z & 64) ? k >> 4 : -(k >> 4))), ex);
  default:
    return ldexp((double)(1 + (z >> 44)), ex - 20);
  }
}

/* counts[0]: quotients through fp_recip, [1]: square roots, [2]: quotients
 * through a root's reciprocal, [3]: polished reciprocals, fp_polish(fp_recip)
 * against 1/b.  Every
 * second numerator is placed next to the midpoint of two quotients, every
 * second radicand next to the square of a midpoint. */
__global__ void rounding_selftest_kernel(int64_t samples, uint64_t seed, unsigned long long *counts) {
  unsigned long long bad[4] = {0, 0, 0, 0};
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < samples; k += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t z0 = rounding_hash(seed + 0x9E3779B97F4A7C15ull * (uint64_t)(2 * k + 1));
    const uint64_t z1 = rounding_hash(seed + 0x9E3779B97F4A7C15ull * (uint64_t)(2 * k + 2));
    const int kb = (int)(k & 3), ka = (int)((k >> 2) & 3);
    const double b = rounding_operand(z0, kb), a0 = rounding_operand(z1, ka);
    /* b times the midpoint above a0: the quotient lies next to that midpoint */
    const double half_ulp = __longlong_as_double(((__double_as_longlong(a0) >> 52) - 53) << 52);
    const double a = (k & 16) ? fma(a0, b, half_ulp * b) : (k & 32 ? -a0 : a0);
    const double yb = fp_recip(b);
    bad[0] += __double_as_longlong(fp_quot(a, b, yb)) != __double_as_longlong(a / b);
    bad[3] += __double_as_longlong(fp_polish(b, yb)) != __double_as_longlong(1.0 / b);
    const double d = (k & 16) ? fma(b, b, 2 * b * __longlong_as_double(((__double_as_longlong(b) >> 52) - 53) << 52)) : b;
    double y;
    const double s = fp_sqrt_recip(d, y);
    bad[1] += __double_as_longlong(s) != __double_as_longlong(sqrt(d));
    bad[2] += __double_as_longlong(fp_quot(a, s, y)) != __double_as_longlong(a / sqrt(d));
  }
  for (int c = 0; c < 4; c++) {
    for (int off = 16; off > 0; off >>= 1)
      bad[c] += __shfl_down_sync(0xffffffffu, bad[c], off);
    if ((threadIdx.x & 31) == 0 && bad[c])
      atomicAdd(counts + c, bad[c]);
  }
}

} // namespace b2e

extern "C" int b2e_selftest_rounding(int64_t samples, uint64_t seed, int64_t mismatches[4]) {
  using namespace b2e;
  if (samples < 1 || !mismatches)
    return B2E_ERR_ARG;
  unsigned long long *dm = nullptr, hm[4] = {0, 0, 0, 0};
  if (cudaMalloc(&dm, sizeof(hm)) != cudaSuccess)
    return B2E_ERR_NOMEM;
  cudaMemset(dm, 0, sizeof(hm));
  rounding_selftest_kernel<<<148 * 8, 256>>>(samples, seed, dm);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpy(hm, dm, sizeof(hm), cudaMemcpyDeviceToHost);
  cudaFree(dm);
  if (e != cudaSuccess)
    return B2E_ERR_CUDA;
  for (int c = 0; c < 4; c++)
    mismatches[c] = (int64_t)hm[c];
  return B2E_OK;
}

/* ---- quotients next to midpoints (b2e_selftest_quotient) ---------------- */
namespace b2e {

/* whether fp_quot(a, b, y) rounds every a of [1, 2) right whose quotient by b =
 * B 2^-52 lies next to a midpoint: A 2^s - M B = k with |k| up to 3, s = 53 for a >=
 * b (midpoints M 2^-53) and 54 for a < b (M 2^-54), M odd in [2^53, 2^54) */
__device__ __forceinline__ bool hardest_quotients_right(uint64_t B, double y) {
  const double b = __longlong_as_double((long long)((B & 0xfffffffffffffull) | 0x3ff0000000000000ull));
  const int v = B & 1 ? 0 : 1;
  if (v && !(B & 2)) /* multiples of 4: so is k */
    return true;
  uint64_t inv = B >> v; /* of B / 2^v modulo 2^64: Newton doubles the right bits, 3 to begin with */
  for (int i = 0; i < 5; i++)
    inv *= 2 - (B >> v) * inv;
  bool right = true;
#pragma unroll 1
  for (int k = -3; k <= 3; k++) {
    if (k == 0 || (v ? k != 2 && k != -2 : (k & 1) == 0))
      continue;
    for (int s = 53; s <= 54; s++) {
      const uint64_t step = 1ull << (s - v);
      for (uint64_t M = (0 - (uint64_t)(int64_t)(v ? k / 2 : k) * inv) & (step - 1); M < 1ull << 54; M += step) {
        const __int128 n = (__int128)((unsigned __int128)M * B) + k; /* A 2^s */
        const uint64_t A = (uint64_t)(n >> s);
        if (M >> 53 != 1 || A >> 52 != 1)
          continue;
        const double a = __longlong_as_double((long long)((A & 0xfffffffffffffull) | 0x3ff0000000000000ull));
        right = right && __double_as_longlong(fp_quot(a, b, y)) == __double_as_longlong(a / b);
      }
    }
  }
  return right;
}

__global__ void quotient_selftest_kernel(int64_t samples, uint64_t seed, unsigned long long *counts) {
  unsigned long long n[5] = {0, 0, 0, 0, 0};
  const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  /* seeds: they follow from the high word, so both ends of its low words bound
   * the error (and every exponent gives the same significand) */
  for (int64_t k = first; k < (1 << 21); k += stride) {
    const uint64_t bits = 0x3ff0000000000000ull | (uint64_t)(k >> 1) << 32 | (k & 1 ? 0xffffffffull : 0);
    const double b = __longlong_as_double((long long)bits), y0 = fp_rcp_seed(b);
    const int ex = (int)(rounding_hash(seed ^ bits) % 401) - 200;
    n[0] += !(fabs(fma(-b, y0, 1.0)) <= 0x1p-19) || fp_rcp_seed(ldexp(b, ex)) != ldexp(y0, -ex) ||
            y0 != fp_rcp_seed(__longlong_as_double((long long)(bits & ~0xffffffffull)));
  }
  /* every significand of the last 2^-18 below 2 */
  for (int64_t k = first; k < (1ll << 34); k += stride) {
    const uint64_t B = (1ull << 53) - 1 - (uint64_t)k;
    const double b = __longlong_as_double((long long)((B & 0xfffffffffffffull) | 0x3ff0000000000000ull));
    const double y = fp_recip(b);
    n[1] += __double_as_longlong(y) != __double_as_longlong(1.0 / b);
    n[2] += !hardest_quotients_right(B, y);
  }
  for (int64_t k = first; k < samples; k += stride) {
    const uint64_t B = (rounding_hash(seed + 0x9E3779B97F4A7C15ull * (uint64_t)(k + 1)) >> 11) | (1ull << 52);
    const double b = __longlong_as_double((long long)((B & 0xfffffffffffffull) | 0x3ff0000000000000ull));
    const double y = fp_recip(b);
    n[3] += __double_as_longlong(y) != __double_as_longlong(1.0 / b);
    n[4] += !hardest_quotients_right(B, y);
  }
  for (int c = 0; c < 5; c++) {
    for (int off = 16; off > 0; off >>= 1)
      n[c] += __shfl_down_sync(0xffffffffu, n[c], off);
    if ((threadIdx.x & 31) == 0 && n[c])
      atomicAdd(counts + c, n[c]);
  }
}

} // namespace b2e

extern "C" int b2e_selftest_quotient(int64_t samples, uint64_t seed, int64_t counts[5]) {
  using namespace b2e;
  if (samples < 1 || !counts)
    return B2E_ERR_ARG;
  unsigned long long *dm = nullptr, hm[5] = {0, 0, 0, 0, 0};
  if (cudaMalloc(&dm, sizeof(hm)) != cudaSuccess)
    return B2E_ERR_NOMEM;
  cudaMemset(dm, 0, sizeof(hm));
  quotient_selftest_kernel<<<148 * 8, 256>>>(samples, seed, dm);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpy(hm, dm, sizeof(hm), cudaMemcpyDeviceToHost);
  cudaFree(dm);
  if (e != cudaSuccess)
    return B2E_ERR_CUDA;
  for (int c = 0; c < 5; c++)
    counts[c] = (int64_t)hm[c];
  return B2E_OK;
}
