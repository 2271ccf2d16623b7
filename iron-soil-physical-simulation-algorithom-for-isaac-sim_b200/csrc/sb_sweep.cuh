// Full-domain repose sweeps (reference slope_model.py:273-343,
// relax_critical_slope): all iterations of a relaxation in one cooperative
// launch.
//
// Direction order, parities and transfers are those of the reference's
// _neighbor_pairs (:744-750): for (d0, d1) in ((1,0), (0,1), (1,1), (1,-1)) and
// parity 0, 1 of endpoint a's axis-0 coordinate (axis 1 for (0,1)), half the
// excess over the critical difference moves from the higher to the lower cell
// (FX: rounded up to whole quanta).  The iteration's largest excess, taken over
// all pairs of a direction before each of its two updates, decides convergence.
//
// A warp owns a box of R rows x 64 columns in registers (lane l: columns 2l and
// 2l + 1), runs the eight sub-phases there and writes the interior R - 16 x 48
// cells back; the exact region shrinks by one cell per sub-phase (halo 8, row
// ranges shrink with it).  Pairs inside a lane are register arithmetic, pairs
// across lanes cost two shuffles; there is no shared memory and no block
// barrier, and parities are compile-time because box origins are even.
//
// What bounds it: integer issue and instruction fetch (straight-line code; ncu
// with 48 rows in a box: 2.8 of 6.9 cycles per instruction wait for them).  A
// pair is 8 integer operations (difference, clamp to +-C, excess, half of it
// towards zero, the two new heights, the two running extremes); the
// shared-memory kernel it replaces spent about 40 on index arithmetic, 64-bit
// differences and double conversions, plus 16 block barriers per iteration.
// FX, every tile moving, 24 rows: 7.8 us per sweep at 701^2, 32 at 2048^2; a cut
// pile settling: 4.9 at 701^2 (24 before), 9.2 at 2048^2 (135 before), 19 at
// 4096^2.  On small grids a sweep is latency: flags and box from L2, one warp's
// instructions, the barrier.  A strip streamed through an 11-row register
// window (no row halo, small code) was slower at every size: its chain of
// sub-phases needs more instructions per cell than a box's shrinking rows.
//
// Tiles at rest are skipped: a box without any transfer in an iteration is the
// same before the next one, so its tile runs again only after a tile of its
// 3x3 neighbourhood changed (the halo reaches no further).  Both ping-pong
// buffers hold such a tile's heights, and its pairs add nothing to the
// convergence test (no excess above zero).  The flags live for one call.
//
// Between iterations the CTAs meet at a bounded grid barrier on one of three
// rotating 64-bit words: arrivals in the low half, CTAs that saw an excess above
// the tolerance in the high half, so one poll gives both.
#pragma once

#include "sb_relax.cuh"

namespace sb {

constexpr int kSweepHalo = 8;
constexpr int kSweepCols = 64;                            // box columns of a warp
constexpr int kSweepInner = kSweepCols - 2 * kSweepHalo;  // columns written back
// Box rows.  Fixed point, measured per sweep, a cut pile settling / every box
// moving (us): 701^2 20 rows 4.8 / 9.8, 24 rows 4.9 / 7.8, 28 rows 6.1 / 8.3, 32
// rows 7.0 / 9.1, 48 rows 10.1 / 14.7; 2048^2 20 rows 11.4 / 47, 24 rows 9.2 / 32,
// 28 rows 10.9 / 32, 32 rows 9.8 / 33.  More rows redo less halo, but the box's
// straight-line code outgrows the instruction cache.
constexpr int kSweepRows = 24;
constexpr int kSweepThreads = 128;
constexpr unsigned kSweepPolls = 1u << 22;

struct SweepConst {
  int n0, n1, pitch, tiles1, ntiles;
  int max_iterations;
  unsigned polls;    // of a wait at the barrier
  double crit[4];    // FP64: critical difference per direction
  double tol;
  unsigned C[4];     // FX: largest difference in quanta that does not move
  unsigned thr[4];   // FX: excess |d| - C from which a pair is above the tolerance
};

struct SweepControl {
  unsigned long long slot[3];
  unsigned int leave;
  int iterations;
  int converged;
  int status;  // 6: a wait gave up, in this or an earlier call; cleared by the host's report
};

// Arithmetic of one pair.  GEN = false: int32 differences (every height of the
// box within +-2^30 quanta) and no row outside the domain.  GEN = true: unsigned
// differences, exact for any int32 heights, and row limits.
template <bool FX, bool GEN>
struct SweepOp;

template <>
struct SweepOp<true, false> {
  using H = int;
  using L = int;
  struct Acc {
    int hi = 0, lo = 0;
  };
  static __device__ __forceinline__ L never() { return 0x7fffffff; }
  static __device__ __forceinline__ L limit(const SweepConst& c, int d, bool ok) {
    return ok ? (int)min(c.C[d], 0x7fffffffu) : never();
  }
  static __device__ __forceinline__ int excess(H a, H b, L C) {
    const int d = a - b;
    return d - min(max(d, -C), C);
  }
  static __device__ __forceinline__ void note(int r, Acc& m) {
    m.hi = max(m.hi, r);
    m.lo = min(m.lo, r);
  }
  // a moves by -t, b by +t with t = half the excess rounded away from zero =
  // r - trunc(r / 2)
  static __device__ __forceinline__ void pair(H& a, H& b, L C, bool count, Acc& m) {
    const int r = excess(a, b, C);
    const int q = (r + (int)((unsigned)r >> 31)) >> 1;
    a = a - r + q;
    b = b + r - q;
    if (count) note(r, m);
  }
  static __device__ __forceinline__ H transfer(H a, H b, L C, bool count, Acc& m) {
    const int r = excess(a, b, C);
    if (count) note(r, m);
    return r - ((r + (int)((unsigned)r >> 31)) >> 1);
  }
  static __device__ __forceinline__ void test(H a, H b, L C, const SweepConst&, Acc& m) {
    note(excess(a, b, C), m);
  }
  static __device__ __forceinline__ bool big(const Acc& m, const SweepConst& c, int d) {
    const int t = (int)min(c.thr[d], 0x7fffffffu);
    return m.hi >= t || -m.lo >= t;
  }
  static __device__ __forceinline__ bool any(const Acc& m) { return (m.hi | m.lo) != 0; }
};

template <>
struct SweepOp<true, true> {
  using H = int;
  using L = unsigned;
  struct Acc {
    unsigned m = 0;
  };
  static __device__ __forceinline__ L never() { return 0xffffffffu; }
  static __device__ __forceinline__ L limit(const SweepConst& c, int d, bool ok) {
    return ok ? c.C[d] : never();
  }
  static __device__ __forceinline__ unsigned excess(H a, H b, L C) {
    const unsigned u = a > b ? (unsigned)a - (unsigned)b : (unsigned)b - (unsigned)a;
    return max(u, C) - C;
  }
  static __device__ __forceinline__ H transfer(H a, H b, L C, bool count, Acc& m) {
    const unsigned x = excess(a, b, C);
    if (count) m.m = max(m.m, x);
    const int t = (int)((x >> 1) + (x & 1u));
    return a > b ? t : -t;
  }
  static __device__ __forceinline__ void pair(H& a, H& b, L C, bool count, Acc& m) {
    const int t = transfer(a, b, C, count, m);
    a -= t;
    b += t;
  }
  static __device__ __forceinline__ void test(H a, H b, L C, const SweepConst&, Acc& m) {
    m.m = max(m.m, excess(a, b, C));
  }
  static __device__ __forceinline__ bool big(const Acc& m, const SweepConst& c, int d) {
    return m.m >= c.thr[d];
  }
  static __device__ __forceinline__ bool any(const Acc& m) { return m.m != 0; }
};

// FP64: the reference's operations in its order (half of fmax(|a - b| - crit, 0)
// with the sign of a - b).
template <bool GEN>
struct SweepOp<false, GEN> {
  using H = double;
  using L = double;
  struct Acc {
    double tol = 0.0;
    bool over = false, moved = false;
  };
  static __device__ __forceinline__ L never() { return __longlong_as_double(0x7ff0000000000000ll); }
  static __device__ __forceinline__ L limit(const SweepConst& c, int d, bool ok) {
    return ok ? c.crit[d] : never();
  }
  static __device__ __forceinline__ H transfer(H a, H b, L C, bool count, Acc& m) {
    const double d = a - b;
    const double x = fabs(d) - C;
    const bool p = x > 0.0;
    if (count) {
      m.over |= x > m.tol;
      m.moved |= p;
    }
    return p ? copysign(0.5 * x, d) : 0.0;
  }
  static __device__ __forceinline__ void pair(H& a, H& b, L C, bool count, Acc& m) {
    const double d = a - b;
    const double x = fabs(d) - C;
    const bool p = x > 0.0;
    if (count) {
      m.over |= x > m.tol;
      m.moved |= p;
    }
    if (p) {
      const double t = copysign(0.5 * x, d);
      a -= t;
      b += t;
    }
  }
  static __device__ __forceinline__ void test(H a, H b, L C, const SweepConst&, Acc& m) {
    m.over |= fabs(a - b) - C > m.tol;
  }
  static __device__ __forceinline__ bool big(const Acc& m, const SweepConst&, int) { return m.over; }
  static __device__ __forceinline__ bool any(const Acc& m) { return m.moved; }
};

// One iteration of a warp's box.  okin: both columns of this lane lie in the
// domain; oknext / okprev: column 2l+1 and lane l+1's first (column 2l and lane
// l-1's second) do.  Columns outside hold zeros and never move: every pair
// across the border has an infinite limit.  [rlo, rhi): rows in the domain (GEN).
// hot: an excess above the tolerance among the tile's own pairs (lanes 4..27);
// chg: a transfer that touches the interior (lanes 3..28; conservative).
//
// Excesses of the idle parity count too, before each update.  Before a
// direction's first update that is parity 1; before the second, parity 0, whose
// pairs have just been brought to the critical difference: never above it in
// whole quanta, possibly by a rounding in FP64.  Once the tile is hot the
// outcome of the test is known, so they are only looked at while it is not.
template <bool FX, bool GEN>
__device__ __forceinline__ void sweep_box(const SweepConst& c,
                                          typename SweepOp<FX, GEN>::H (&e)[kSweepRows],
                                          typename SweepOp<FX, GEN>::H (&o)[kSweepRows], int lane,
                                          bool okin, bool oknext, bool okprev, int rlo, int rhi,
                                          bool& hot, bool& chg) {
  constexpr int R = kSweepRows;
  using S = SweepOp<FX, GEN>;
  using H = typename S::H;
  using L = typename S::L;
  const int nx = (lane + 1) & 31, pv = (lane - 1) & 31;
  constexpr unsigned kAll = 0xffffffffu;
  const bool own = lane >= 4 && lane < 28;
  bool moved = false;
  hot = false;
  auto rows = [&](int r, L lim) { return GEN && (r + 1 == rlo || r + 1 == rhi) ? S::never() : lim; };
  constexpr int r0 = kSweepHalo, r1 = R - kSweepHalo;  // interior rows
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    const L in = S::limit(c, d, d == 0 || okin);
    const L cross = S::limit(c, d, d == 3 ? okprev : oknext);
    typename S::Acc m;
    if constexpr (!FX) m.tol = c.tol;
    // pairs of rows r (and r + 1) without moving them
    auto look = [&](int par) {
      if (d == 1) {
#pragma unroll
        for (int r = r0; r < r1; ++r) {
          if (par == 0)
            S::test(e[r], o[r], in, c, m);
          else
            S::test(o[r], __shfl_sync(kAll, e[r], nx), cross, c, m);
        }
      } else {
#pragma unroll
        for (int r = r0; r < r1; ++r) {
          if ((r & 1) != par) continue;
          if (d == 0) {
            S::test(e[r], e[r + 1], rows(r, in), c, m);
            S::test(o[r], o[r + 1], rows(r, in), c, m);
          } else if (d == 2) {
            S::test(e[r], o[r + 1], rows(r, in), c, m);
            S::test(o[r], __shfl_sync(kAll, e[r + 1], nx), rows(r, cross), c, m);
          } else {
            S::test(o[r], e[r + 1], rows(r, in), c, m);
            S::test(e[r], __shfl_sync(kAll, o[r + 1], pv), rows(r, cross), c, m);
          }
        }
      }
    };
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      const int i = 2 * d + par;  // sub-phase: rows [i, R - i) are exact before it
      if (!hot && (par == 0 || !FX)) look(1 - par);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r < i || r >= R - i) continue;
        const bool count = r >= r0 - 1 && r < r1;
        if (d == 1) {
          if (par == 0) {
            S::pair(e[r], o[r], in, count, m);
          } else {
            const H t = S::transfer(o[r], __shfl_sync(kAll, e[r], nx), cross, count, m);
            o[r] -= t;
            e[r] += __shfl_sync(kAll, t, pv);
          }
        } else {
          if ((r & 1) != par || r + 1 >= R) continue;
          if (d == 0) {
            S::pair(e[r], e[r + 1], rows(r, in), count, m);
            S::pair(o[r], o[r + 1], rows(r, in), count, m);
          } else if (d == 2) {
            S::pair(e[r], o[r + 1], rows(r, in), count, m);
            const H t = S::transfer(o[r], __shfl_sync(kAll, e[r + 1], nx), rows(r, cross), count, m);
            o[r] -= t;
            e[r + 1] += __shfl_sync(kAll, t, pv);
          } else {
            S::pair(o[r], e[r + 1], rows(r, in), count, m);
            const H t = S::transfer(e[r], __shfl_sync(kAll, o[r + 1], pv), rows(r, cross), count, m);
            e[r] -= t;
            o[r + 1] += __shfl_sync(kAll, t, nx);
          }
        }
      }
      hot = hot || __any_sync(kAll, own && S::big(m, c, d));
    }
    moved |= S::any(m);
  }
  chg = __any_sync(kAll, moved && lane >= 3 && lane < 29);
}

template <bool FX>
__global__ void __launch_bounds__(kSweepThreads, FX ? 4 : 2)
    sweep_kernel(const SweepConst c, typename FvTypes<FX>::H* f0, typename FvTypes<FX>::H* f1,
                 int* act0, int* act1, SweepControl* ctl) {
  using H = typename FvTypes<FX>::H;
  using H2 = typename std::conditional<FX, int2, double2>::type;
  constexpr int R = kSweepRows, kRows = R - 2 * kSweepHalo;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // neighbouring tiles go to different SMs: active tiles come in clusters
  const int first = warp * gridDim.x + blockIdx.x, stride = gridDim.x * (kSweepThreads / 32);
  const int tiles0 = c.ntiles / c.tiles1;
  __shared__ int s_state;  // 0: next iteration, 1: converged, 2: stop, 3: a wait gave up
  int it = 0;
  for (;; ++it) {
    const H* src = (it & 1) ? f1 : f0;
    H* dst = (it & 1) ? f0 : f1;
    const int* prev = (it & 1) ? act0 : act1;
    int* next = (it & 1) ? act1 : act0;
    bool seen = false;
    for (int t = first; t < c.ntiles; t += stride) {
      const int t0 = t / c.tiles1, t1 = t - t0 * c.tiles1;
      bool self = true;
      if (it > 0) {
        int a = 0;
        if (lane < 9) {
          const int q0 = t0 + lane / 3 - 1, q1 = t1 + lane % 3 - 1;
          if (q0 >= 0 && q0 < tiles0 && q1 >= 0 && q1 < c.tiles1)
            a = __ldcg(prev + q0 * c.tiles1 + q1);
        }
        const unsigned near = __ballot_sync(0xffffffffu, a != 0);
        self = (near >> 4) & 1u;
        if (!near) {
          if (lane == 0) next[t] = 0;
          continue;
        }
      }
      const int g0 = t0 * kRows - kSweepHalo, g1 = t1 * kSweepInner - kSweepHalo + 2 * lane;
      const bool oke = g1 >= 0 && g1 < c.n1, oko = g1 + 1 >= 0 && g1 + 1 < c.n1;
      const int rlo = max(0, -g0), rhi = min(R, c.n0 - g0);
      H e[R], o[R];
      const H* p = src + (long long)g0 * c.pitch + g1;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        H2 v{0, 0};
        if (oke && r >= rlo && r < rhi)  // g1 is even and the pitch a multiple of 32: aligned, in the row
          v = __ldcg(reinterpret_cast<const H2*>(p + (long long)r * c.pitch));
        e[r] = v.x;
        o[r] = oko ? v.y : H(0);
      }
      bool gen = rlo > 0 || rhi < R;
      if constexpr (FX) {
        int hi = 0, lo = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          hi = max(hi, max(e[r], o[r]));
          lo = min(lo, min(e[r], o[r]));
        }
        gen = __any_sync(0xffffffffu, gen || hi >= (1 << 30) || lo < -(1 << 30));
      }
      const bool okin = oke && oko;
      const bool oknext = oko && g1 + 2 < c.n1 && lane < 31;
      const bool okprev = oke && g1 > 0 && lane > 0;
      bool hot, chg;
      if (gen)
        sweep_box<FX, true>(c, e, o, lane, okin, oknext, okprev, rlo, rhi, hot, chg);
      else
        sweep_box<FX, false>(c, e, o, lane, okin, oknext, okprev, rlo, rhi, hot, chg);
      seen |= hot;
      if (lane == 0) next[t] = chg ? 1 : 0;
      // the other buffer already holds the interior if it moved neither in this
      // iteration nor in the last
      if (chg || self) {
        if (lane >= kSweepHalo / 2 && lane < 32 - kSweepHalo / 2 && oke) {
          H* w = dst + (long long)g0 * c.pitch + g1;
#pragma unroll
          for (int r = kSweepHalo; r < R - kSweepHalo; ++r) {
            if (r < rhi) {
              if (oko) {
                H2 v;
                v.x = e[r];
                v.y = o[r];
                *reinterpret_cast<H2*>(w + (long long)r * c.pitch) = v;
              } else {
                w[(long long)r * c.pitch] = e[r];
              }
            }
          }
        }
      }
    }
    const int any = __syncthreads_or(seen);
    if (threadIdx.x == 0) {
      unsigned long long* slot = &ctl->slot[it % 3];
      // last read two barriers ago; in use again after this one
      if (blockIdx.x == 0) *(volatile unsigned long long*)&ctl->slot[(it + 1) % 3] = 0ull;
      __threadfence();
      unsigned long long v = atomicAdd(slot, 1ull + ((unsigned long long)(any ? 1 : 0) << 32));
      v += 1ull + ((unsigned long long)(any ? 1 : 0) << 32);
      unsigned polls = 0;
      while ((unsigned)v != gridDim.x) {
        if (++polls > c.polls) break;
        if (polls > 64) __nanosleep(32);
        v = *(volatile unsigned long long*)slot;
      }
      __threadfence();
      s_state = (unsigned)v != gridDim.x        ? 3
                : (v >> 32) == 0                ? 1
                : it + 1 >= c.max_iterations    ? 2
                                                : 0;
    }
    __syncthreads();
    if (s_state) break;
  }
  // leave the result in f0: only tiles that moved in the last iteration differ
  if (!(it & 1)) {
    for (int t = first; t < c.ntiles; t += stride) {
      if (!__ldcg(act0 + t)) continue;
      const int t0 = t / c.tiles1, t1 = t - t0 * c.tiles1;
      const int g0 = t0 * kRows, g1 = t1 * kSweepInner;
      for (int r = 0; r < kRows && g0 + r < c.n0; ++r)
        for (int k = lane; k < kSweepInner && g1 + k < c.n1; k += 32) {
          const size_t i = (size_t)(g0 + r) * c.pitch + g1 + k;
          f0[i] = __ldcg(f1 + i);
        }
    }
  }
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) {
      ctl->iterations = it + 1;
      ctl->converged = s_state == 1;
    }
    if (s_state == 3) atomicExch(&ctl->status, 6);  // SB_ERR_WAIT_LIMIT
    __threadfence();
    if (atomicAdd(&ctl->leave, 1u) == gridDim.x - 1) {  // the last CTA out: ready for the next call
      ctl->slot[0] = ctl->slot[1] = ctl->slot[2] = 0ull;
      ctl->leave = 0;
    }
  }
}

}  // namespace sb
