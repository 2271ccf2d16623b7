// Repose (MiniSlope) relaxation kernels.
//
// Arrays are generic 2-D fields whose axis 0 (rows) uses spacing s0 and axis 1
// (columns) spacing s1, the convention of the reference's
// ``relax_critical_slope(height, grid_spacing)`` (slope_model.py:273-343).
// Direction order and parity rule follow ``_neighbor_pairs`` (:744-750): for
// (d0, d1) in ((1,0,s0), (0,1,s1), (1,1,hyp), (1,-1,hyp)), parity on the
// axis-0 coordinate of endpoint a when d0 != 0, else on its axis-1 coordinate.
//
// Full-domain sweeps (relax_critical_slope itself) are in sb_sweep.cuh.
//
// relax_reached_kernel   -- one reached-gated iteration per launch, temporally
//                           blocked: a (T+2*8)^2 halo box in shared memory runs
//                           all eight sub-phases (the exact region shrinks by
//                           one cell per sub-phase), the T^2 interior is
//                           written back.
#pragma once

#include <climits>

#include "sb_common.cuh"
#include "sb_fv.cuh"

namespace sb {

constexpr int kRelaxTile = 32;
constexpr int kRelaxHalo = 8;
constexpr int kRelaxBox = kRelaxTile + 2 * kRelaxHalo;  // 48

struct RelaxConst {
  int n0, n1, pitch, tiles1, ntiles;
  double s0, s1;
  double crit[4];       // tan(angle) * L per direction
  double crit_q[4];     // FX: crit / Q
  double tol, tol_q;
  int max_iterations;
  int weighted;         // frontier: Triangle-A-C vertex weights (else uniform)
  int ftile;            // frontier tile size
  double f;             // weight unit s0*s1/6
};

struct RelaxControl {
  int iterations;
  int done;
  int converged;
  int status;
  unsigned long long max_excess_bits;  // double bits of this iteration's max excess
  unsigned int arrive;
  int parity;        // buffer holding the current field (full relax)
  int n_active;      // frontier: active tiles at the start of the last round
  int rounds;
  int moved_edges;
  int confirm;       // reached-gated sweep: 1 while the confirming scan is pending
  int bb[4];         // reached-gated sweep: bounding box of reached cells (min0, max0, min1, max1)
};

__device__ __forceinline__ void dir_of(int d, int& d0, int& d1) {
  d0 = d == 1 ? 0 : 1;
  d1 = d == 0 ? 0 : (d == 3 ? -1 : 1);
}

// ------------------------------------------------------------------------
// Reached-gated full-domain iteration: the event-driven reached-bbox
// MiniSlope backend (EventDrivenMinimumSlopeAdapter._relax_dynamic_frontier,
// solvers/event_driven_slope.py:166-302).
//
// A 48^2 TMA box, 8 sub-phases in shared memory, the 32^2 interior written
// back, and the reached mask staged
// in a second TMA box: a pair moves only if one endpoint is reached, both
// endpoints of a moved pair become reached (the mask can spread one cell per
// sub-phase, so the 8-cell halo stays exact), and the iteration maximum takes
// only reachable pairs.  A box that holds no reached cell when its CTA starts
// cannot change its interior within one iteration, so CTAs whose box misses
// the reached bounding box (grown with atomics, never shrunk) skip the
// iteration; both ping-pong buffers hold the same values for such tiles
// (begin kernel), so nothing needs writing.  An iteration whose maximum is
// <= tolerance is followed by a confirming scan of all reachable pairs on the
// post-iteration state (no update, not counted); the solve ends when that
// scan is <= tolerance too, otherwise the iterations continue.
// ------------------------------------------------------------------------
template <bool FX>
__global__ void __launch_bounds__(kThreads)
    relax_reached_kernel(const RelaxConst c, const __grid_constant__ CUtensorMap tm0,
                         const __grid_constant__ CUtensorMap tm1,
                         const __grid_constant__ CUtensorMap tr0,
                         const __grid_constant__ CUtensorMap tr1,
                         typename FvTypes<FX>::H* __restrict__ f0,
                         typename FvTypes<FX>::H* __restrict__ f1, int* __restrict__ r0,
                         int* __restrict__ r1, RelaxControl* ctl,
                         cudaGraphConditionalHandle handle, int use_handle) {
  using H = typename FvTypes<FX>::H;
  __shared__ alignas(128) H s[kRelaxBox * kRelaxBox];
  __shared__ alignas(128) int rs[kRelaxBox * kRelaxBox];
  __shared__ alignas(8) uint64_t bar;
  __shared__ double red[kThreads / 32];
  __shared__ int bbs[4];
  __shared__ int last;
  if (*(volatile int*)&ctl->done) return;
  const int parity_buf = ctl->parity;
  const int confirm = ctl->confirm;
  const int t1 = blockIdx.x % c.tiles1, t0 = blockIdx.x / c.tiles1;
  const int g0 = t0 * kRelaxTile - kRelaxHalo, g1 = t1 * kRelaxTile - kRelaxHalo;
  const volatile int* vb = ctl->bb;
  const int bmin0 = vb[0], bmax0 = vb[1], bmin1 = vb[2], bmax1 = vb[3];
  const bool work = bmin0 <= bmax0 && bmax0 >= g0 && bmin0 < g0 + kRelaxBox && bmax1 >= g1 &&
                    bmin1 < g1 + kRelaxBox;  // block-uniform
  double worst = 0.0;
  bool loaded = true;
  if (work) {
    if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      bbs[0] = INT_MAX;
      bbs[1] = INT_MIN;
      bbs[2] = INT_MAX;
      bbs[3] = INT_MIN;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      mbar_expect_tx(&bar, kRelaxBox * kRelaxBox * (unsigned)(sizeof(H) + sizeof(int)));
      tma_load_2d(s, parity_buf ? &tm1 : &tm0, g1, g0, &bar);
      tma_load_2d(rs, parity_buf ? &tr1 : &tr0, g1, g0, &bar);
    }
    loaded = mbar_wait(&bar, 0);
    if (confirm) {
      // all reachable pairs owned by the interior, every direction, no update
      for (int d = 0; d < 4 && loaded; ++d) {
        int d0, d1;
        dir_of(d, d0, d1);
        for (int k = threadIdx.x; k < kRelaxTile * kRelaxTile; k += kThreads) {
          const int la0 = kRelaxHalo + k / kRelaxTile, la1 = kRelaxHalo + k % kRelaxTile;
          const int a0 = g0 + la0, a1 = g1 + la1, b0 = a0 + d0, b1 = a1 + d1;
          if (a0 >= c.n0 || a1 >= c.n1 || b0 >= c.n0 || b1 < 0 || b1 >= c.n1) continue;
          const int ia = la0 * kRelaxBox + la1, ib = (la0 + d0) * kRelaxBox + la1 + d1;
          if (!(rs[ia] | rs[ib])) continue;
          double ex;
          if constexpr (FX) {
            const long long df = (long long)s[ia] - (long long)s[ib];
            ex = (double)(df < 0 ? -df : df) - c.crit_q[d];
          } else {
            ex = fabs(s[ia] - s[ib]) - c.crit[d];
          }
          worst = fmax(worst, ex);
        }
      }
    } else {
      for (int d = 0; d < 4; ++d) {
        int d0, d1;
        dir_of(d, d0, d1);
        for (int par = 0; par < 2; ++par) {
          // (1) reachable inactive-parity pairs owned by the interior, before
          // this sub-phase's update
          constexpr int kHalfTile = kRelaxTile / 2;
          const int ifirst = d0 ? ((1 - par - g0) & 1) : ((1 - par - g1) & 1);
          for (int k = threadIdx.x; k < kHalfTile * kRelaxTile; k += kThreads) {
            const int la0 = kRelaxHalo + (d0 ? ifirst + 2 * (k / kRelaxTile) : k / kHalfTile);
            const int la1 = kRelaxHalo + (d0 ? k % kRelaxTile : ifirst + 2 * (k % kHalfTile));
            const int a0 = g0 + la0, a1 = g1 + la1, b0 = a0 + d0, b1 = a1 + d1;
            if (a0 >= c.n0 || a1 >= c.n1 || b0 >= c.n0 || b1 < 0 || b1 >= c.n1) continue;
            const int ia = la0 * kRelaxBox + la1, ib = (la0 + d0) * kRelaxBox + la1 + d1;
            if (!(rs[ia] | rs[ib])) continue;
            double ex;
            if constexpr (FX) {
              const long long df = (long long)s[ia] - (long long)s[ib];
              ex = (double)(df < 0 ? -df : df) - c.crit_q[d];
            } else {
              ex = fmax(fabs(s[ia] - s[ib]) - c.crit[d], 0.0);
            }
            worst = fmax(worst, ex);
          }
          __syncthreads();
          // (2) gated Jacobi update of the active-parity pairs inside the box
          if (loaded) {
            constexpr int kHalf = kRelaxBox / 2;
            const int first = d0 ? ((par - g0) & 1) : ((par - g1) & 1);
            for (int k = threadIdx.x; k < kHalf * kRelaxBox; k += kThreads) {
              int la0, la1;
              if (d0) {
                la0 = first + 2 * (k / kRelaxBox);
                la1 = k % kRelaxBox;
              } else {
                la0 = k / kHalf;
                la1 = first + 2 * (k % kHalf);
              }
              const int lb0 = la0 + d0, lb1 = la1 + d1;
              if (lb0 >= kRelaxBox || lb1 < 0 || lb1 >= kRelaxBox) continue;
              const int a0 = g0 + la0, a1 = g1 + la1, b0 = a0 + d0, b1 = a1 + d1;
              if (a0 < 0 || a1 < 0 || a0 >= c.n0 || a1 >= c.n1) continue;
              if (b0 >= c.n0 || b1 < 0 || b1 >= c.n1) continue;
              const int ia = la0 * kRelaxBox + la1, ib = lb0 * kRelaxBox + lb1;
              if (!(rs[ia] | rs[ib])) continue;
              const bool owned = la0 >= kRelaxHalo && la0 < kRelaxHalo + kRelaxTile &&
                                 la1 >= kRelaxHalo && la1 < kRelaxHalo + kRelaxTile;
              if constexpr (FX) {
                const long long df = (long long)s[ia] - (long long)s[ib];
                const double ex = (double)(df < 0 ? -df : df) - c.crit_q[d];
                if (owned) worst = fmax(worst, ex);
                if (ex > 0.0) {
                  const long long t = (long long)ceil(ex * 0.5);
                  const long long st = df < 0 ? -t : t;
                  s[ia] = (H)(s[ia] - st);
                  s[ib] = (H)(s[ib] + st);
                  rs[ia] = 1;
                  rs[ib] = 1;
                }
              } else {
                const double diff = s[ia] - s[ib];
                const double ex = fmax(fabs(diff) - c.crit[d], 0.0);
                if (owned) worst = fmax(worst, ex);
                if (ex > 0.0) {
                  const double sg = diff > 0.0 ? 1.0 : (diff < 0.0 ? -1.0 : 0.0);
                  const double t = 0.5 * ex * sg;
                  s[ia] = s[ia] - t;
                  s[ib] = s[ib] + t;
                  rs[ia] = 1;
                  rs[ib] = 1;
                }
              }
            }
          }
          __syncthreads();
        }
      }
      // write back the interior (heights and reached) into the other buffers,
      // and grow the reached bounding box by the interior's reached cells
      H* dst = parity_buf ? f0 : f1;
      int* rdst = parity_buf ? r0 : r1;
      int lo0 = INT_MAX, hi0 = INT_MIN, lo1 = INT_MAX, hi1 = INT_MIN;
      for (int k = threadIdx.x; k < kRelaxTile * kRelaxTile; k += kThreads) {
        const int la0 = kRelaxHalo + k / kRelaxTile, la1 = kRelaxHalo + k % kRelaxTile;
        const int a0 = g0 + la0, a1 = g1 + la1;
        if (a0 < c.n0 && a1 < c.n1 && loaded) {
          const int li = la0 * kRelaxBox + la1;
          dst[(size_t)a0 * c.pitch + a1] = s[li];
          rdst[(size_t)a0 * c.pitch + a1] = rs[li];
          if (rs[li]) {
            lo0 = min(lo0, a0);
            hi0 = max(hi0, a0);
            lo1 = min(lo1, a1);
            hi1 = max(hi1, a1);
          }
        }
      }
      if (lo0 <= hi0) {
        atomicMin(&bbs[0], lo0);
        atomicMax(&bbs[1], hi0);
        atomicMin(&bbs[2], lo1);
        atomicMax(&bbs[3], hi1);
      }
      __syncthreads();
      if (threadIdx.x == 0 && bbs[0] <= bbs[1]) {
        atomicMin(&ctl->bb[0], bbs[0]);
        atomicMax(&ctl->bb[1], bbs[1]);
        atomicMin(&ctl->bb[2], bbs[2]);
        atomicMax(&ctl->bb[3], bbs[3]);
      }
    }
  }
  worst = warp_max(worst);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = worst;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) m = fmax(m, red[w]);
    if (!loaded) atomicExch(&ctl->status, 6);
    atomicMax(&ctl->max_excess_bits, (unsigned long long)__double_as_longlong(m));
    __threadfence();
    last = atomicAdd(&ctl->arrive, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  const double m = __longlong_as_double((long long)ctl->max_excess_bits);
  const double tol = FX ? c.tol_q : c.tol;
  ctl->arrive = 0;
  ctl->max_excess_bits = 0;
  if (ctl->status) {
    ctl->done = 1;
  } else if (confirm) {
    if (m <= tol) {
      ctl->converged = 1;
      ctl->done = 1;
    }
    ctl->confirm = 0;
  } else {
    ctl->iterations += 1;
    ctl->parity = parity_buf ^ 1;
    if (m <= tol) ctl->confirm = 1;
  }
  // the safety cap: a next iteration beyond max_iterations is an error
  if (!ctl->done && !ctl->confirm && ctl->iterations >= c.max_iterations) {
    ctl->status = 4;  // SB_ERR_NONCONVERGENCE
    ctl->done = 1;
  }
  __threadfence();
  if (use_handle) cudaGraphSetConditional(handle, ctl->done ? 0u : 1u);
}

// Start of a reached-gated solve: loop control reset, both ping-pong buffers
// made equal (heights and reached) and the reached bounding box from the seeds.
template <bool FX>
__global__ void __launch_bounds__(kThreads)
    relax_reached_begin_kernel(const RelaxConst c, const typename FvTypes<FX>::H* __restrict__ f0,
                               typename FvTypes<FX>::H* __restrict__ f1,
                               const int* __restrict__ r0, int* __restrict__ r1,
                               RelaxControl* ctl) {
  __shared__ int bbs[4];
  if (threadIdx.x == 0) {
    bbs[0] = INT_MAX;
    bbs[1] = INT_MIN;
    bbs[2] = INT_MAX;
    bbs[3] = INT_MIN;
  }
  __syncthreads();
  int lo0 = INT_MAX, hi0 = INT_MIN, lo1 = INT_MAX, hi1 = INT_MIN;
  const long long n = (long long)c.n0 * c.n1;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int a0 = (int)(i / c.n1), a1 = (int)(i % c.n1);
    const size_t gi = (size_t)a0 * c.pitch + a1;
    f1[gi] = f0[gi];
    const int r = r0[gi] != 0;
    r1[gi] = r;
    if (r) {
      lo0 = min(lo0, a0);
      hi0 = max(hi0, a0);
      lo1 = min(lo1, a1);
      hi1 = max(hi1, a1);
    }
  }
  if (lo0 <= hi0) {
    atomicMin(&bbs[0], lo0);
    atomicMax(&bbs[1], hi0);
    atomicMin(&bbs[2], lo1);
    atomicMax(&bbs[3], hi1);
  }
  __syncthreads();
  if (threadIdx.x == 0 && bbs[0] <= bbs[1]) {
    atomicMin(&ctl->bb[0], bbs[0]);
    atomicMax(&ctl->bb[1], bbs[1]);
    atomicMin(&ctl->bb[2], bbs[2]);
    atomicMax(&ctl->bb[3], bbs[3]);
  }
}

// Triangle-A-C weights of the compact frontier (sb_frontier.cuh).
__device__ __forceinline__ double vertex_weight_fp64(int r, int col, int n0, int n1, double f) {
  double w = 0.0;
  if (r < n0 - 1 && col < n1 - 1) w += 2.0 * f;
  if (r < n0 - 1 && col > 0) w += f;
  if (r > 0 && col > 0) w += 2.0 * f;
  if (r > 0 && col < n1 - 1) w += f;
  return w;
}

__device__ __forceinline__ long long gcd_ll(long long a, long long b) {
  while (b) {
    const long long t = a % b;
    a = b;
    b = t;
  }
  return a;
}

// sum, min and max 8-neighbour slope of a support field (RelaxationStats:
// volume_before/after and max_slope = slope_model.max_neighbor_slope :261-270).
template <bool FX>
__global__ void __launch_bounds__(kThreads)
    field_stats_kernel(int n0, int n1, int pitch, double s0, double s1, double Q, double datum,
                       const typename FvTypes<FX>::H* __restrict__ f, double* __restrict__ partials,
                       long long* __restrict__ ipartials, unsigned int* arrive, double* out) {
  const double diag = hypot(s0, s1);
  double sum = 0.0, mx = 0.0, mn = 1.0e300;
  long long isum = 0;
  const long long n = (long long)n0 * n1;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int a0 = (int)(i / n1), a1 = (int)(i % n1);
    const size_t ia = (size_t)a0 * pitch + a1;
    double va;
    if constexpr (FX) {
      isum += f[ia];
      va = (double)f[ia] * Q + datum;
    } else {
      va = f[ia];
      sum += va;
    }
    mn = fmin(mn, va);
    for (int d = 0; d < 4; ++d) {
      int d0, d1;
      dir_of(d, d0, d1);
      const int b0 = a0 + d0, b1 = a1 + d1;
      if (b0 >= n0 || b1 < 0 || b1 >= n1) continue;
      const size_t ib = (size_t)b0 * pitch + b1;
      const double dist = d == 0 ? s0 : (d == 1 ? s1 : diag);
      double diff;
      if constexpr (FX) diff = (double)((long long)f[ia] - (long long)f[ib]) * Q;
      else diff = f[ia] - f[ib];
      mx = fmax(mx, fabs(diff) / dist);
    }
  }
  sum = warp_sum(sum);
  isum = (long long)warp_sum_u64((unsigned long long)isum);
  mx = warp_max(mx);
  mn = warp_min(mn);
  __shared__ double r[kThreads / 32][3];
  __shared__ long long ri[kThreads / 32];
  __shared__ int last;
  if ((threadIdx.x & 31) == 0) {
    r[threadIdx.x >> 5][0] = sum;
    r[threadIdx.x >> 5][1] = mx;
    r[threadIdx.x >> 5][2] = mn;
    ri[threadIdx.x >> 5] = isum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0, cmin = 1.0e300;
    long long ia = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      a += r[w][0];
      b = fmax(b, r[w][1]);
      cmin = fmin(cmin, r[w][2]);
      ia += ri[w];
    }
    partials[blockIdx.x * 3 + 0] = a;
    partials[blockIdx.x * 3 + 1] = b;
    partials[blockIdx.x * 3 + 2] = cmin;
    ipartials[blockIdx.x] = ia;
    __threadfence();
    last = atomicAdd(arrive, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  double a = 0.0, b = 0.0, cmin = 1.0e300;
  long long ia = 0;
  for (unsigned k = 0; k < gridDim.x; ++k) {
    a += __ldcg(partials + k * 3);
    b = fmax(b, __ldcg(partials + k * 3 + 1));
    cmin = fmin(cmin, __ldcg(partials + k * 3 + 2));
    ia += __ldcg(ipartials + k);
  }
  *arrive = 0;
  out[0] = FX ? (double)ia * Q + datum * (double)n : a;
  out[1] = b;
  out[2] = cmin;
  out[3] = (double)ia;
}

// The ping-pong relaxation may end in the alternate buffer: copy it back
// (every block reads the same flag), then clear the flag in a second launch.
template <bool FX>
__global__ void relax_copyback_kernel(const typename FvTypes<FX>::B* __restrict__ src,
                                      typename FvTypes<FX>::B* __restrict__ dst, long long count,
                                      const RelaxControl* ctl) {
  if (!ctl->parity) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

// reached mask back into the caller-visible field after a reached-gated solve
__global__ void reached_copyback_kernel(const int* __restrict__ src, int* __restrict__ dst,
                                        long long count, const RelaxControl* ctl) {
  if (!ctl->parity) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

__global__ void relax_parity_clear_kernel(RelaxControl* ctl) {
  if (threadIdx.x == 0 && blockIdx.x == 0) ctl->parity = 0;
}

}  // namespace sb
