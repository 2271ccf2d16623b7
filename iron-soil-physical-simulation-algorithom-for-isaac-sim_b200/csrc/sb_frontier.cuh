// Compact-frontier repose rounds (production schedule: runtime/
// v2_physics_core.py:1172-1254 over solvers/warp_compact_frontier.py:56-130), all
// rounds of a call in one cooperative launch.
//
// A round works on a list of active tiles: eight colour sub-phases of
// reached-gated, weighted transfers, then a scan that finds the tiles of the next
// round.  A sub-phase runs the tiles that were listed when it started; tiles of
// the 3x3 cell stencil around moved endpoints join the list (a tile's stamp
// holds the last round that listed it, taken by atomicExch) and run from the next
// sub-phase on.  The scan appends straight to the next round's list the same way.
//
// A frontier is a few tiles (nine of 64^2 on a 192^2 pit), so a sub-phase has
// work for a few dozen CTAs and its time is latency.  The pairs of all listed
// tiles are therefore one index range over the whole grid (one pair per thread
// where it fits), a pair's four loads are issued together, and the sub-phases
// meet at a grid barrier instead of ten kernel boundaries with one CTA per tile:
// the 64-bit barrier word counts arrivals below and appended tiles above, so one
// poll gives the release and the new list length.  A round took 148 us as ten
// kernels of a graph loop and takes about 38 (192^2 pit, nine tiles): nine
// barriers of about 2.5 us and two dependent L2 round trips between them.
#pragma once

#include "sb_relax.cuh"

namespace sb {

constexpr unsigned kFrontierPolls = 1u << 22;

struct FrontierSync {
  unsigned long long slot[3];
  int count[2];          // entries of the two lists
  unsigned int leave;
  int pad;
};

// Records copied to mapped host memory by the last CTA of a step's last kernel.
struct PathRecordPtrs {
  const void* src[6];
  void* dst[6];
  int bytes[6];
};

__device__ __forceinline__ void copy_records(const PathRecordPtrs& p, int n) {
  for (int k = 0; k < n; ++k) {
    const unsigned* s = static_cast<const unsigned*>(p.src[k]);
    unsigned* d = static_cast<unsigned*>(p.dst[k]);
    for (int w = threadIdx.x; w < p.bytes[k] / 4; w += blockDim.x) d[w] = __ldcg(s + w);
  }
  __threadfence_system();
}

// One pair; returns whether it moved.
template <bool FX>
__device__ __forceinline__ bool frontier_pair(const RelaxConst& c, int dir, int a0, int a1, int b0,
                                              int b1, typename FvTypes<FX>::H* hf, int* reached) {
  using H = typename FvTypes<FX>::H;
  const size_t ia = (size_t)a0 * c.pitch + a1, ib = (size_t)b0 * c.pitch + b1;
  const int ra = __ldcg(reached + ia), rb = __ldcg(reached + ib);
  const H ha = __ldcg(hf + ia), hb = __ldcg(hf + ib);
  if (!ra && !rb) return false;
  if constexpr (FX) {
    const long long df = (long long)ha - (long long)hb;
    const double ex = (double)(df < 0 ? -df : df) - c.crit_q[dir];
    if (!(ex > 0.0)) return false;
    long long ua = 1, ub = 1;
    if (c.weighted) {
      const int wa = vertex_weight6(a0, a1, c.n0, c.n1), wb = vertex_weight6(b0, b1, c.n0, c.n1);
      if (wa != wb) {
        const long long g = gcd_ll(wa, wb);
        ua = wb / g;
        ub = wa / g;
      }
    }
    const long long kk = (long long)ceil(ex / (double)(ua + ub));
    const long long sg = df < 0 ? -1 : 1;
    hf[ia] = (H)(ha - sg * kk * ua);
    hf[ib] = (H)(hb + sg * kk * ub);
  } else {
    const double diff = ha - hb;
    const double ex = fabs(diff) - c.crit[dir];
    if (!(ex > 0.0)) return false;
    const double signed_ex = diff < 0.0 ? -ex : ex;
    double wa = 1.0, wb = 1.0;
    if (c.weighted) {
      wa = vertex_weight_fp64(a0, a1, c.n0, c.n1, c.f);
      wb = vertex_weight_fp64(b0, b1, c.n0, c.n1, c.f);
    }
    const double ws = wa + wb;
    const double ta = signed_ex * wb / ws, tb = signed_ex * wa / ws;
    hf[ia] = ha - ta;
    hf[ib] = hb + tb;
  }
  reached[ia] = 1;
  reached[ib] = 1;
  return true;
}

// Does cell (r, col) own a reachable pair whose excess is above the tolerance?
template <bool FX>
__device__ __forceinline__ bool frontier_unstable(const RelaxConst& c, int r, int col,
                                                  const typename FvTypes<FX>::H* hf,
                                                  const int* reached) {
  using H = typename FvTypes<FX>::H;
  const size_t ia = (size_t)r * c.pitch + col;
  const int ra = __ldcg(reached + ia);
  const H ha = __ldcg(hf + ia);
  int rb[4];
  H hb[4];
  bool in[4];
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    int d0, d1;
    dir_of(d, d0, d1);
    const int b0 = r + d0, b1 = col + d1;
    in[d] = b0 < c.n0 && b1 >= 0 && b1 < c.n1;
    const size_t ib = in[d] ? (size_t)b0 * c.pitch + b1 : ia;
    rb[d] = __ldcg(reached + ib);
    hb[d] = __ldcg(hf + ib);
  }
  bool found = false;
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    if (!in[d] || (!ra && !rb[d])) continue;
    if constexpr (FX) {
      const long long df = (long long)ha - (long long)hb[d];
      found |= (double)(df < 0 ? -df : df) - c.crit_q[d] > c.tol_q;
    } else {
      found |= fabs(ha - hb[d]) - c.crit[d] > c.tol;
    }
  }
  return found;
}

// pending: the tile flags of seeds (consumed); stamp, list0, list1: scratch of
// ntiles entries.  ctl->done set beforehand: nothing runs and the pending flags
// stay.  The last CTA to leave copies nrec records to the host.
template <bool FX>
__global__ void __launch_bounds__(kThreads)
    frontier_kernel(const RelaxConst c, typename FvTypes<FX>::H* hf, int* reached, int* pending,
                    int* stamp, int* list0, int* list1, RelaxControl* ctl, FrontierSync* sync,
                    const PathRecordPtrs rec, int nrec) {
  __shared__ int s_added, s_moved;
  __shared__ long long s_total;  // appended since the last barrier, or -1: a wait gave up
  __shared__ int s_last;
  const int T = c.ftile, lane = threadIdx.x & 31;
  const long long gtid = (long long)blockIdx.x * kThreads + threadIdx.x;
  const long long gthreads = (long long)gridDim.x * kThreads;
  int arrivals = 0, moved = 0, added = 0;
  if (threadIdx.x == 0) s_added = s_moved = 0;
  __syncthreads();
  // all CTAs; returns the tiles appended by anyone since the last call
  auto meet = [&]() {
    const int mine = warp_sum(added);
    added = 0;
    if (lane == 0 && mine) atomicAdd(&s_added, mine);
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long* slot = &sync->slot[arrivals % 3];
      // last read two barriers ago; in use again after this one
      if (blockIdx.x == 0)
        *(volatile unsigned long long*)&sync->slot[(arrivals + 1) % 3] = 0ull;
      __threadfence();
      const unsigned long long add = 1ull + ((unsigned long long)s_added << 32);
      s_added = 0;
      unsigned long long v = atomicAdd(slot, add) + add;
      unsigned polls = 0;
      while ((unsigned)v != gridDim.x) {
        if (++polls > kFrontierPolls) break;
        if (polls > 64) __nanosleep(32);
        v = *(volatile unsigned long long*)slot;
      }
      __threadfence();
      s_total = (unsigned)v != gridDim.x ? -1 : (long long)(v >> 32);
    }
    __syncthreads();
    ++arrivals;
    const long long total = s_total;
    __syncthreads();
    return total;
  };
  // lists tile t for round k unless that has happened already
  auto list_tile = [&](int t, int k) {
    if (__ldcg(stamp + t) == k || atomicExch(stamp + t, k) == k) return;
    (k & 1 ? list1 : list0)[atomicAdd(&sync->count[k & 1], 1)] = t;
    ++added;
  };
  if (!*(volatile int*)&ctl->done) {  // uniform across the grid
    for (long long t = gtid; t < c.ntiles; t += gthreads) {
      const int a = pending[t] != 0;
      stamp[t] = a;
      if (a) {
        pending[t] = 0;
        list1[atomicAdd(&sync->count[1], 1)] = (int)t;
        ++added;
      }
    }
    long long len = meet();
    int round = 0, status = 0;
    for (;;) {
      if (len < 0) {
        status = 6;  // SB_ERR_WAIT_LIMIT
        break;
      }
      if (len == 0) break;
      if (round >= c.max_iterations) {
        status = 4;  // SB_ERR_NONCONVERGENCE
        break;
      }
      ++round;
      const int* list = round & 1 ? list1 : list0;
      // the other list is written again by this round's scan
      if (gtid == 0) *(volatile int*)&sync->count[(round + 1) & 1] = 0;
      const int half = (T + 1) / 2;
      for (int s = 0; s < 8 && len >= 0; ++s) {
        const int dir = s >> 1, par = s & 1;
        int d0, d1;
        dir_of(dir, d0, d1);
        const long long items = len * half * T;
        for (long long i = gtid; i < items; i += gthreads) {
          const int e = (int)(i / (half * T)), k = (int)(i - (long long)e * (half * T));
          const int t = __ldcg(list + e);
          const int tr = t / c.tiles1, tc = t - tr * c.tiles1;
          // only the tile's rows (d0 != 0) or columns (d0 == 0) of parity par hold
          // an active endpoint a
          const int first = d0 ? ((par - tr * T) & 1) : ((par - tc * T) & 1);
          const int la0 = d0 ? first + 2 * (k / T) : k / half;
          const int la1 = d0 ? k % T : first + 2 * (k % half);
          const int a0 = tr * T + la0, a1 = tc * T + la1, b0 = a0 + d0, b1 = a1 + d1;
          if (la0 >= T || la1 >= T || a0 >= c.n0 || a1 >= c.n1) continue;
          if (b0 >= c.n0 || b1 < 0 || b1 >= c.n1) continue;
          if (!frontier_pair<FX>(c, dir, a0, a1, b0, b1, hf, reached)) continue;
          ++moved;
          // the 3x3 cell stencil of an endpoint inside the tile stays in the tile
          const int lo = min(la0, la1 + min(d1, 0)), hi = max(la0 + d0, la1 + max(d1, 0));
          if (lo >= 1 && hi <= T - 2) continue;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int p0 = q ? b0 : a0, p1 = q ? b1 : a1;
            for (int u = max(p0 - 1, 0) / T; u <= min(p0 + 1, c.n0 - 1) / T; ++u)
              for (int v = max(p1 - 1, 0) / T; v <= min(p1 + 1, c.n1 - 1) / T; ++v)
                list_tile(u * c.tiles1 + v, round);
          }
        }
        const long long more = meet();
        len = more < 0 ? -1 : len + more;
      }
      if (len < 0) continue;
      const long long cells = len * T * T;
      for (long long i = gtid; i < cells; i += gthreads) {
        const int e = (int)(i / (T * T)), k = (int)(i - (long long)e * (T * T));
        const int t = __ldcg(list + e);
        const int tr = t / c.tiles1, tc = t - tr * c.tiles1;
        const int r = tr * T + k / T, col = tc * T + k % T;
        if (r >= c.n0 || col >= c.n1) continue;
        if (frontier_unstable<FX>(c, r, col, hf, reached)) list_tile(t, round + 1);
      }
      len = meet();
    }
    if (!status)  // converged: the frontier ends here
      for (long long i = gtid; i < (long long)c.n0 * c.pitch; i += gthreads) reached[i] = 0;
    moved = warp_sum(moved);
    if (lane == 0 && moved) atomicAdd(&s_moved, moved);
    __syncthreads();
    if (threadIdx.x == 0) {
      if (s_moved) atomicAdd(&ctl->moved_edges, s_moved);
      if (status == 6) atomicExch(&ctl->status, 6);
      if (blockIdx.x == 0) {
        ctl->rounds = round;
        ctl->n_active = len < 0 ? 0 : (int)len;
        ctl->converged = status == 0;
        if (status == 4) ctl->status = 4;
        ctl->done = 1;
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&sync->leave, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (threadIdx.x < 3) sync->slot[threadIdx.x] = 0ull;
  if (threadIdx.x < 2) sync->count[threadIdx.x] = 0;
  if (threadIdx.x == 0) sync->leave = 0;
  copy_records(rec, nrec);
}

}  // namespace sb
