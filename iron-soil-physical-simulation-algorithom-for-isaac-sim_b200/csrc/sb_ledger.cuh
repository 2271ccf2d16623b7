// Per-step ledger / prologue reduction and field conversion kernels.
//
// One pass over the state computes, with a deterministic two-level reduction:
//   * the FP64 ledger of MobileV2ReferenceSolver.mass/momentum/energy_terms
//     (experimental/mobile_v2_reference.py:104-127) and of the production
//     ``summarize`` kernel (bulk_interaction/warp_mobile_v2.py:28-54); in the
//     fixed-point path mass and Triangle-A-C volume are exact int64 sums;
//   * the static short-circuit of ``_globally_static_below_start`` (:353-363);
//   * the wave speed that sets the first substep's dt (:239-253).
#pragma once

#include "sb_fv.cuh"

namespace sb {

// FX: a thread's ledger.  Every Triangle-A-C weighted sum is 6 times the plain one
// except at border cells, whose (w6 - 6) shares go to the thread's slots of edge
// (the fold's scratch): the inner cells keep 8 sums and maxima less in registers.
//
// grad: a before-step ledger decides the static short-circuit by whether the
// free-surface gradient exceeds the start slope anywhere; its maximum is used for
// nothing else.  A float32 value below the limit by 1e-4 settles a cell (its error
// is below 1e-6); the others are taken in FP64, until a lane has found one above
// the limit by 1e-9.
struct LedgerScan {
  bool grad;
  float sx0, sx1, sy0, sy1, limit2;
  double above2;
  int* wet;      // flags of the substep loop's blocks, or null
  double* edge;  // slots kFoldStride apart: qx, qy, hs2, hb, hh and (int64) h quanta
  double qx = 0.0, qy = 0.0, hs2 = 0.0, hb = 0.0, hh = 0.0, s2 = 0.0, grad2 = 0.0;
  float maxq = 0.f, wave = 0.f, ext = 0.f;
  int minh = 0x7fffffff;
  int quads = 0, wet_quads = 0;  // visited; with a wet cell
  long long mass = 0, rest6 = 0;
  __device__ __forceinline__ LedgerScan(const FvConst& c, bool grad_, double static_limit,
                                        int* wet_, double* fold)
      : grad(grad_), wet(wet_), edge(fold + threadIdx.x + (threadIdx.x >> 5)) {
    sx0 = (float)c.gsx[0];
    sx1 = (float)c.gsx[1];
    sy0 = (float)c.gsy[0];
    sy1 = (float)c.gsy[1];
    limit2 = (float)(static_limit * static_limit * (1.0 - 1.0e-4));
    above2 = static_limit * static_limit * (1.0 + 1.0e-9);
#pragma unroll
    for (int k = 0; k < 6; ++k) edge[k * kFoldStride] = 0.0;  // also the int64 zero
  }
  __device__ __forceinline__ void finish(const FvConst& c, double* v, long long* iq) const {
#pragma unroll
    for (int k = 0; k < L_NP; ++k) v[k] = 0.0;
    v[L_QX] = qx;
    v[L_QY] = qy;
    v[L_HS2] = hs2;
    v[L_HB] = hb;
    v[L_HH] = hh;
    v[L_QX_W] = 6.0 * qx + edge[0];
    v[L_QY_W] = 6.0 * qy + edge[kFoldStride];
    v[L_HS2_W] = 6.0 * hs2 + edge[2 * kFoldStride];
    v[L_HB_W] = 6.0 * hb + edge[3 * kFoldStride];
    v[L_HH_W] = 6.0 * hh + edge[4 * kFoldStride];
    v[L_MAXSPEED] = s2;
    v[L_NEGMINH] = minh == 0x7fffffff ? -1.0e300 : -((double)minh * c.Q);
    v[L_MAXQ] = maxq;
    v[L_MAXGRAD] = grad2;
    v[L_MAXWAVE] = wave;
    v[L_MAXEXT] = ext;
    iq[0] = mass;
    iq[1] = 6 * mass + __double_as_longlong(edge[5 * kFoldStride]);
    iq[2] = rest6;
  }
};

// Triangle-A-C weight: 6 wherever the cell has all its neighbours.
__device__ __forceinline__ int ledger_weight6(int r, int col, int ny, int nx) {
  if (r > 0 && r + 1 < ny && col > 0 && col + 1 < nx) return 6;
  return vertex_weight6(r, col, ny, nx);
}

// FX: sums and maxima of cell (r, col).  A cell with neither mobile material nor
// momentum contributes exact zeros.
__device__ __forceinline__ void ledger_cell_fx(const FvConst& c, int bq, int hq, float qxf,
                                               float qyf, double datum, int r, int col, bool inner,
                                               LedgerScan& scan) {
  const double hv = (double)hq * c.Q;
  const double bv = (double)bq * c.Q + datum;
  const double qxv = (double)qxf, qyv = (double)qyf;
  double s2 = 0.0, e = 0.0;
  float wave = 0.f;  // empty cell: no velocity, no celerity
  if (hq != 0) {
    const float hn = (float)hq * c.Qf;
    float vx = 0.f, vy = 0.f;
    if (hn > c.dryf) {
      const float inv = 1.0f / hn;
      vx = qxf * inv;
      vy = qyf * inv;
    }
    wave = sqrtf(vx * vx + vy * vy) + sqrtf(c.KGf * hn);
  }
  if (hv > c.dry) {  // one reciprocal: e = |q|^2 / h (= h |u|^2), s2 = e / h
    const double inv = 1.0 / hv;
    e = (qxv * qxv + qyv * qyv) * inv;
    s2 = e * inv;
  }
  const double hb = hv * bv, hh = hv * hv;
  scan.mass += hq;
  scan.qx += qxv;
  scan.qy += qyv;
  scan.hs2 += e;
  scan.hb += hb;
  scan.hh += hh;
  scan.s2 = fmax(scan.s2, s2);  // squared speed; sqrt after the max
  scan.maxq = fmaxf(scan.maxq, fmaxf(fabsf(qxf), fabsf(qyf)));
  scan.wave = fmaxf(scan.wave, wave);
  if (!inner) {
    const int less = ledger_weight6(r, col, c.ny, c.nx) - 6;
    if (less == 0) return;
    double* edge = scan.edge;
    edge[0] += qxv * less;
    edge[kFoldStride] += qyv * less;
    edge[2 * kFoldStride] += e * less;
    edge[3 * kFoldStride] += hb * less;
    edge[4 * kFoldStride] += hh * less;
    edge[5 * kFoldStride] = __longlong_as_double(
        __double_as_longlong(edge[5 * kFoldStride]) + (long long)hq * less);
  }
}

// Wrapping 32-bit sum and difference; the sign bit of over records a wrap.
__device__ __forceinline__ int wrap_add(int a, int b, int& over) {
  const int s = (int)((unsigned)a + (unsigned)b);
  over |= (a ^ s) & (b ^ s);
  return s;
}

__device__ __forceinline__ int wrap_sub(int a, int b, int& over) {
  const int d = (int)((unsigned)a - (unsigned)b);
  over |= (a ^ b) & (a ^ d);
  return d;
}

// FX: largest squared free-surface gradient (np.gradient, edge_order 1) of
// cells [col, col + n) of row r, from integer b + h differences scaled by
// Q / (2 dx) inside and Q / dx on the edges (c.gsx / c.gsy, from the host).
__device__ __forceinline__ double fx_grad2_max(const FvConst& c, const int32_t* __restrict__ b,
                                                const int32_t* __restrict__ h, int r, int col,
                                                int n) {
  const size_t row = (size_t)r * c.pitch;
  const size_t dn = r > 0 ? row - c.pitch : row, up = r + 1 < c.ny ? row + c.pitch : row;
  const double sy = r > 0 && r + 1 < c.ny ? c.gsy[0] : c.gsy[1];
  double most = 0.0;
#pragma unroll 1
  for (int x = col; x < col + n; ++x) {
    const int xl = x > 0 ? x - 1 : x, xr = x + 1 < c.nx ? x + 1 : x;
    const long long Hl = (long long)b[row + xl] + h[row + xl];
    const long long Hr = (long long)b[row + xr] + h[row + xr];
    const long long Hd = (long long)b[dn + x] + h[dn + x], Hu = (long long)b[up + x] + h[up + x];
    const double gx = (double)(Hr - Hl) * (x > 0 && x + 1 < c.nx ? c.gsx[0] : c.gsx[1]);
    const double gy = (double)(Hu - Hd) * sy;
    most = fmax(most, gx * gx + gy * gy);
  }
  return most;
}

// Columns of a warp's item of one row: a lane owns kLedgerQuad neighbours, read
// as 16-byte words (rows start on 128 bytes).
//
// Bound by DRAM in the end (20 B per cell; 51 us at 4096^2 and the measured copy
// rate), before that by instructions and by loads in flight: one cell per lane with
// its 13 scalar loads and 64-bit gradient took 234 instructions per 32 cells and 150
// us on a site that is nearly all dry; a quad per lane, 32-bit differences and one
// copy of the wet cells' code (two cells at a time) take 97 per 32 and 94 us (77 us
// after a step, without the gradient).  All wet, 2500 x 2300: 14 us less of 216 a
// step.  Two CTAs per SM (128 registers) against three with spills: 94 and 104 us;
// asking L2 for a warp's next item: 134 to 124 us.
constexpr int kLedgerQuad = 4;
constexpr int kLedgerCols = 32 * kLedgerQuad;
constexpr int kLedgerCtasFx = 2;  // resident CTAs per SM

// FX: cells [col, col + 4) of row r, col = a multiple of kLedgerCols + 4 lane.
// FULL: all four lie inside the grid (else the words past nx are the row's
// padding or, from a lane with no cell at all, not read).
template <bool FULL>
__device__ __forceinline__ void ledger_quad_fx(const FvConst& c, const int32_t* __restrict__ b,
                                               const int32_t* __restrict__ z,
                                               const int32_t* __restrict__ h,
                                               const float* __restrict__ qx,
                                               const float* __restrict__ qy,
                                               const float* __restrict__ ext_x,
                                               const float* __restrict__ ext_y, double datum, int r,
                                               int col, LedgerScan& scan) {
  const int n = FULL ? kLedgerQuad : min(c.nx - col, kLedgerQuad);
  if (!FULL && n <= 0) return;
  const unsigned gi = (unsigned)r * (unsigned)c.pitch + (unsigned)col;
  const int4 b4 = *reinterpret_cast<const int4*>(b + gi);
  const int4 z4 = *reinterpret_cast<const int4*>(z + gi);
  const int4 h4 = *reinterpret_cast<const int4*>(h + gi);
  const int4 x4 = *reinterpret_cast<const int4*>(qx + gi);
  const int4 y4 = *reinterpret_cast<const int4*>(qy + gi);
  const int bq[4] = {b4.x, b4.y, b4.z, b4.w}, zq[4] = {z4.x, z4.y, z4.z, z4.w};
  const int hq[4] = {h4.x, h4.y, h4.z, h4.w};
  const int qxb[4] = {x4.x, x4.y, x4.z, x4.w}, qyb[4] = {y4.x, y4.y, y4.z, y4.w};
  if (scan.grad) {
    // np.gradient, edge_order 1, of b + h
    const bool iny = r > 0 && r + 1 < c.ny;
    const unsigned dn = r > 0 ? gi - (unsigned)c.pitch : gi;
    const unsigned up = r + 1 < c.ny ? gi + (unsigned)c.pitch : gi;
    const int4 bd = *reinterpret_cast<const int4*>(b + dn);
    const int4 hd = *reinterpret_cast<const int4*>(h + dn);
    const int4 bu = *reinterpret_cast<const int4*>(b + up);
    const int4 hu = *reinterpret_cast<const int4*>(h + up);
    const unsigned gl = col > 0 ? gi - 1 : gi, gr = col + n < c.nx ? gi + n : gi + n - 1;
    int over = 0;  // sign bit: a 32-bit sum or difference wrapped
    int s[kLedgerQuad + 2];  // b + h of the cells and of their neighbours left and right
    s[0] = wrap_add(b[gl], h[gl], over);
    const int beyond = wrap_add(b[gr], h[gr], over);
#pragma unroll
    for (int k = 0; k < kLedgerQuad; ++k)
      s[k + 1] = FULL || k < n ? wrap_add(bq[k], hq[k], over) : beyond;
    s[kLedgerQuad + 1] = beyond;
    const int bdn[4] = {bd.x, bd.y, bd.z, bd.w}, hdn[4] = {hd.x, hd.y, hd.z, hd.w};
    const int bup[4] = {bu.x, bu.y, bu.z, bu.w}, hup[4] = {hu.x, hu.y, hu.z, hu.w};
    const float sy = iny ? scan.sy0 : scan.sy1;
    float most = 0.f;
#pragma unroll
    for (int k = 0; k < kLedgerQuad; ++k) {
      if (!FULL && k >= n) continue;
      const int dx = wrap_sub(s[k + 2], s[k], over);
      const int dy = wrap_sub(wrap_add(bup[k], hup[k], over), wrap_add(bdn[k], hdn[k], over), over);
      const bool inx = (k > 0 || col > 0) && ((FULL && k < 3) || col + k + 1 < c.nx);
      const float gx = (float)dx * (inx ? scan.sx0 : scan.sx1), gy = (float)dy * sy;
      most = fmaxf(most, gx * gx + gy * gy);
    }
    if ((over < 0 || most >= scan.limit2) && scan.grad2 <= scan.above2)
      scan.grad2 = fmax(scan.grad2, fx_grad2_max(c, b, h, r, col, n));
  }
  const bool inner = FULL && r > 0 && r + 1 < c.ny && col > 0 && col + kLedgerQuad < c.nx;
  long long rest6 = 0;
  int some = 0;  // 0: the four cells hold neither material nor momentum
#pragma unroll
  for (int k = 0; k < kLedgerQuad; ++k) {
    if (!FULL && k >= n) continue;
    const unsigned rest = (unsigned)max(bq[k], zq[k]) - (unsigned)zq[k];
    const int w6 = inner ? 1 : ledger_weight6(r, col + k, c.ny, c.nx);
    rest6 += (long long)rest * w6;
    scan.minh = min(scan.minh, hq[k]);
    some |= hq[k] | ((qxb[k] | qyb[k]) << 1);  // a momentum of -0 is none
    if (c.has_external)
      scan.ext = fmaxf(scan.ext, fmaxf(fabsf(ext_x[gi + k]), fabsf(ext_y[gi + k])));
  }
  scan.rest6 += inner ? rest6 * 6 : rest6;
  scan.quads += 1;
  if (some == 0) return;
  scan.wet_quads += 1;
  if (scan.wet) {  // the substep loop's blocks of these cells are not dry
    const int j = r / c.chunk_rows, i = (r - j * c.chunk_rows) / c.block_rows;
#pragma unroll
    for (int k = 0; k < kLedgerQuad; ++k)
      if ((FULL || k < n) && (hq[k] | ((qxb[k] | qyb[k]) << 1)) != 0)
        scan.wet[((col + k) / kStripOut * c.row_chunks + j) * c.chunk_blocks + i] = 1;
  }
#pragma unroll 1
  for (int k = 0; k < n; k += 2) {  // two cells at a time
    const bool k2 = k & 2;
    ledger_cell_fx(c, k2 ? bq[2] : bq[0], k2 ? hq[2] : hq[0],
                   __int_as_float(k2 ? qxb[2] : qxb[0]), __int_as_float(k2 ? qyb[2] : qyb[0]),
                   datum, r, col + k, inner, scan);
    if (FULL || k + 1 < n)
      ledger_cell_fx(c, k2 ? bq[3] : bq[1], k2 ? hq[3] : hq[1],
                     __int_as_float(k2 ? qxb[3] : qxb[1]), __int_as_float(k2 ? qyb[3] : qyb[1]),
                     datum, r, col + k + 1, inner, scan);
  }
}

// FP64 ledger contributions of cell (r, col): sums into v[0 .. L_NSUM), maxima
// into v[L_NSUM .. L_NP).
__device__ __forceinline__ void ledger_cell_fp64(const FvConst& c, const double* __restrict__ b,
                                                 const double* __restrict__ z,
                                                 const double* __restrict__ h,
                                                 const double* __restrict__ qx,
                                                 const double* __restrict__ qy,
                                                 const double* __restrict__ ext_x,
                                                 const double* __restrict__ ext_y, int r, int col,
                                                 double* v) {
  const size_t gi = (size_t)r * c.pitch + col;
  const int w6 = vertex_weight6(r, col, c.ny, c.nx);
  const double qxv = (double)qx[gi], qyv = (double)qy[gi];
  // gradient of the free surface b + h (np.gradient, edge_order 1)
  const int cl = col > 0 ? col - 1 : col, cr = col + 1 < c.nx ? col + 1 : col;
  const int rd = r > 0 ? r - 1 : r, ru = r + 1 < c.ny ? r + 1 : r;
  const double denx = (col > 0 && col + 1 < c.nx) ? 2.0 * c.dx : c.dx;
  const double deny = (r > 0 && r + 1 < c.ny) ? 2.0 * c.dy : c.dy;
  const size_t il = (size_t)r * c.pitch + cl, ir = (size_t)r * c.pitch + cr;
  const size_t idn = (size_t)rd * c.pitch + col, iup = (size_t)ru * c.pitch + col;
  const double hv = h[gi];
  const double bv = b[gi];
  v[L_HSUM] += hv;
  v[L_HSUM_W] += hv * w6;
  v[L_REST_W] += fmax(b[gi] - z[gi], 0.0) * w6;
  const double gx = ((b[ir] + h[ir]) - (b[il] + h[il])) / denx;
  const double gy = ((b[iup] + h[iup]) - (b[idn] + h[idn])) / deny;
  const double grad = hypot(gx, gy);
  const bool wet = hv > c.dry;
  double s2 = 0.0, spd = 0.0, e = 0.0;
  double vx = 0.0, vy = 0.0;
  if (wet) {
    vx = qxv / hv;
    vy = qyv / hv;
  }
  const double wave = sqrt(vx * vx + vy * vy) + sqrt(c.kg * fmax(hv, 0.0));
  if (wet) {
    s2 = (qxv * qxv + qyv * qyv) / (hv * hv);
    spd = sqrt(s2);
    e = hv * s2;
  }
  v[L_QX] += qxv;
  v[L_QY] += qyv;
  v[L_QX_W] += qxv * w6;
  v[L_QY_W] += qyv * w6;
  v[L_HS2] += e;
  v[L_HS2_W] += e * w6;
  v[L_HB] += hv * bv;
  v[L_HB_W] += hv * bv * w6;
  v[L_HH] += hv * hv;
  v[L_HH_W] += hv * hv * w6;
  v[L_MAXSPEED] = fmax(v[L_MAXSPEED], spd);
  v[L_NEGMINH] = fmax(v[L_NEGMINH], -hv);
  v[L_MAXQ] = fmax(v[L_MAXQ], fmax(fabs(qxv), fabs(qyv)));
  v[L_MAXGRAD] = fmax(v[L_MAXGRAD], grad);
  v[L_MAXWAVE] = fmax(v[L_MAXWAVE], wave);
  if (c.has_external)
    v[L_MAXEXT] = fmax(v[L_MAXEXT], fmax(fabs((double)ext_x[gi]), fabs((double)ext_y[gi])));
}

// Block reduction of per-thread ledger values into one block's partials, in a
// fixed order: slot k to part[k * stride], integer slot k to ipart[k * stride].
// fold: fold_words(L_NP) doubles of shared memory.
__device__ __forceinline__ void ledger_block_store(const double* v, const long long* iq,
                                                   double* fold, double* part, long long* ipart,
                                                   int stride) {
  const double* bt = block_fold<double, L_NP, L_NSUM>(v, fold);
  const double mine = threadIdx.x < L_NP ? bt[threadIdx.x] : 0.0;
  __syncthreads();  // the integer fold reuses the scratch
  const long long* it =
      block_fold<long long, kLedgerI64, kLedgerI64>(iq, reinterpret_cast<long long*>(fold));
  if (threadIdx.x < L_NP) part[(size_t)threadIdx.x * stride] = mine;
  if (threadIdx.x < kLedgerI64) ipart[(size_t)threadIdx.x * stride] = it[threadIdx.x];
}

// Final value of ledger slot k: the FX path accumulates squared gradient and
// squared speed maxima and takes the (monotone) square root after the max.
template <bool FX>
__device__ __forceinline__ double ledger_final_value(int k, double val) {
  if (FX && (k == L_MAXGRAD || k == L_MAXSPEED)) return sqrt(val);
  return val;
}

// Fixed-order fold of a ledger's slot-major block partials (nb blocks) into
// out.  Every thread of the block calls it; scratch: fold_words(L_NP) doubles.
template <bool FX>
__device__ void ledger_final_fold(const double* partials, const long long* ipartials, int nb,
                                  double* fold, LedgerOut* out) {
  const double* tot = reduce_partials<L_NP, L_NSUM>(partials, nb, fold);
  const double mine = threadIdx.x < L_NP ? tot[threadIdx.x] : 0.0;
  __syncthreads();  // the integer fold reuses the scratch
  long long a[kLedgerI64] = {0, 0, 0};
  for (int bk = threadIdx.x; bk < nb; bk += kThreads)
#pragma unroll
    for (int k = 0; k < kLedgerI64; ++k) a[k] += __ldcg(ipartials + (size_t)k * nb + bk);
  const long long* itot =
      block_fold<long long, kLedgerI64, kLedgerI64>(a, reinterpret_cast<long long*>(fold));
  if (threadIdx.x < L_NP) out->v[threadIdx.x] = ledger_final_value<FX>(threadIdx.x, mine);
  if (threadIdx.x < kLedgerI64) out->iq[threadIdx.x] = itot[threadIdx.x];
  __syncthreads();
}

// Static short-circuit and the first substep's dt from a "before" ledger
// (reference step :199-205, :239-253).  One thread.
__device__ __forceinline__ void ledger_prologue(const FvConst& c, const LedgerOut* out,
                                                double static_limit, FvControl* ctl) {
  const bool no_ext = !c.has_external || out->v[L_MAXEXT] <= 1.0e-14;
  const bool is_static = no_ext && out->v[L_MAXQ] <= 1.0e-14 && out->v[L_MAXGRAD] <= static_limit;
  ctl->wave = out->v[L_MAXWAVE];
  if (is_static) {
    ctl->static_skip = 1;
    ctl->done = 1;
  } else if (!(ctl->remaining > 1.0e-14)) {
    ctl->done = 1;
  } else if (c.max_substeps <= 0) {
    ctl->status = 2;
    ctl->done = 1;
  } else {
    plan_substep(c, ctl);
  }
}

// mode 0: "before" ledger of a step + prologue (static short-circuit, first
// dt, loop condition).  The prologue only needs four maxima, which the blocks
// send by atomicMax (order-free), so the last block plans the first substep
// at once; the before ledger's sums stay as block partials (part_before).
// mode 1: "after" ledger.  mode 2: "after" ledger, then the folds that the
// step deferred: the before ledger's partials into io->before and the step's
// substep impulse/energy sums (diag_acc, c.nblocks FV blocks) into ctl->diag.
template <bool FX>
__global__ void __launch_bounds__(kThreads, FX ? kLedgerCtasFx : 3)
    ledger_kernel(const FvConst c, const typename FvTypes<FX>::B* __restrict__ b,
                  const typename FvTypes<FX>::B* __restrict__ z,
                  const typename FvTypes<FX>::H* __restrict__ h0,
                  const typename FvTypes<FX>::H* __restrict__ h1,
                  const typename FvTypes<FX>::R* __restrict__ qx0,
                  const typename FvTypes<FX>::R* __restrict__ qx1,
                  const typename FvTypes<FX>::R* __restrict__ qy0,
                  const typename FvTypes<FX>::R* __restrict__ qy1,
                  const typename FvTypes<FX>::R* __restrict__ ext_x,
                  const typename FvTypes<FX>::R* __restrict__ ext_y, double datum,
                  double static_limit, int mode, FvControl* ctl, StepIO* io,
                  double* __restrict__ partials, long long* __restrict__ ipartials,
                  unsigned int* arrive, double* __restrict__ diag_acc,
                  double* __restrict__ part_before, long long* __restrict__ ipart_before,
                  cudaGraphConditionalHandle loop_handle, int use_handle) {
  using T = FvTypes<FX>;
  const int parity = ctl->parity;
  const typename T::H* h = parity ? h1 : h0;
  const typename T::R* qx = parity ? qx1 : qx0;
  const typename T::R* qy = parity ? qy1 : qy0;
  __shared__ double fold[fold_words(L_NP)];
  __shared__ int last;
  double v[L_NP];
  long long iq[kLedgerI64] = {0, 0, 0};
  bool seen = false, mostly_wet = false;  // a lane without a cell is neither wet nor dry
  const int nwarps = gridDim.x * (kThreads / 32);
  const int lane = threadIdx.x & 31;
  int it = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if constexpr (FX) {
    // a before-step ledger flags the wet blocks of the current buffer
    LedgerScan scan(c, mode == 0, static_limit,
                    mode == 0 && c.wet ? c.wet + parity * c.tiles_x * c.row_chunks * c.chunk_blocks
                                       : nullptr,
                    fold);
    // warp items = kLedgerCols columns of one row
    const int spans = (c.nx + kLedgerCols - 1) / kLedgerCols, items = spans * c.ny;
    int r = it / spans, s = it - r * spans;
    const int dr = nwarps / spans, ds = nwarps - dr * spans;
    // lane 4 a + l asks L2 for line l of array a of the warp's next item
    const void* ask = lane < 4    ? (const void*)b
                      : lane < 8  ? (const void*)z
                      : lane < 12 ? (const void*)h
                      : lane < 16 ? (const void*)qx
                                  : (const void*)qy;
    const int ask_col = 32 * (lane & 3);
    for (; it < items; it += nwarps) {
      const int row = r, col = s * kLedgerCols;
      r += dr;
      s += ds;
      if (s >= spans) {
        s -= spans;
        ++r;
      }
      if (lane < 20 && it + nwarps < items && s * kLedgerCols + ask_col < c.nx)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(
            (const char*)ask +
            4 * (size_t)((unsigned)r * (unsigned)c.pitch + s * kLedgerCols + ask_col)));
      if (col + kLedgerCols <= c.nx)
        ledger_quad_fx<true>(c, b, z, h, qx, qy, ext_x, ext_y, datum, row,
                             col + lane * kLedgerQuad, scan);
      else
        ledger_quad_fx<false>(c, b, z, h, qx, qy, ext_x, ext_y, datum, row,
                              col + lane * kLedgerQuad, scan);
    }
    scan.finish(c, v, iq);
    seen = scan.quads > 0;
    mostly_wet = seen && 2 * scan.wet_quads >= scan.quads;
  } else {
#pragma unroll
    for (int k = 0; k < L_NP; ++k) v[k] = 0.0;
    v[L_NEGMINH] = -1.0e300;
    // warp items = 32-column segments of one row; a lane owns one column
    const int strips = (c.nx + 31) >> 5, items = strips * c.ny;
    int r = it / strips, s = it - r * strips;
    const int dr = nwarps / strips, ds = nwarps - dr * strips;
#pragma unroll 2
    for (; it < items; it += nwarps) {
      const int col = (s << 5) + lane;
      if (col < c.nx) ledger_cell_fp64(c, b, z, h, qx, qy, ext_x, ext_y, r, col, v);
      r += dr;
      s += ds;
      if (s >= strips) {
        s -= strips;
        ++r;
      }
    }
  }
  // block partials slot-major: partials[k * gridDim.x + block]
  double* part = mode == 0 ? part_before : partials;
  long long* ipart = mode == 0 ? ipart_before : ipartials;
  ledger_block_store(v, iq, fold, part + blockIdx.x, ipart + blockIdx.x, gridDim.x);
  if (FX && mode == 0) {
    const int seen_threads = __syncthreads_count(seen);
    const int wet_threads = __syncthreads_count(mostly_wet);
    if (threadIdx.x == 4) {
      atomicAdd(&ctl->seen_threads, (unsigned)seen_threads);
      atomicAdd(&ctl->wet_threads, (unsigned)wet_threads);
    }
  } else {
    __syncthreads();
  }
  if (mode == 0 && threadIdx.x < 4) {  // the prologue's maxima (all >= 0: bits order like values)
    const int slot = threadIdx.x == 0 ? L_MAXEXT
                     : threadIdx.x == 1 ? L_MAXQ
                     : threadIdx.x == 2 ? L_MAXGRAD
                                        : L_MAXWAVE;
    const double m = part[(size_t)slot * gridDim.x + blockIdx.x];
    atomicMax(&ctl->pmax[threadIdx.x], (unsigned long long)__double_as_longlong(m));
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(arrive, 1u) == gridDim.x - 1) ? 1 : 0;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (mode == 0) {
    if (threadIdx.x == 0) {
      // prologue: static short-circuit and the first substep's dt
      LedgerOut pro;
      pro.v[L_MAXEXT] = __longlong_as_double((long long)atomicExch(&ctl->pmax[0], 0ull));
      pro.v[L_MAXQ] = __longlong_as_double((long long)atomicExch(&ctl->pmax[1], 0ull));
      pro.v[L_MAXGRAD] = ledger_final_value<FX>(
          L_MAXGRAD, __longlong_as_double((long long)atomicExch(&ctl->pmax[2], 0ull)));
      pro.v[L_MAXWAVE] = __longlong_as_double((long long)atomicExch(&ctl->pmax[3], 0ull));
      *arrive = 0;
      if (FX)
        ctl->dense =
            fv_dense(atomicExch(&ctl->wet_threads, 0u), atomicExch(&ctl->seen_threads, 0u));
      ledger_prologue(c, &pro, static_limit, ctl);
      __threadfence();
      if (use_handle) cudaGraphSetConditional(loop_handle, ctl->done ? 0u : 1u);
    }
    return;
  }
  ledger_final_fold<FX>(partials, ipartials, gridDim.x, fold, &io->after);
  if (mode == 2) {
    ledger_final_fold<FX>(part_before, ipart_before, gridDim.x, fold, &io->before);
    // the step's impulse/energy sums: fold the FV blocks' accumulators in a
    // fixed order and clear them for the next step
    const int nb = c.nblocks;
    double d[kFvDiag];
#pragma unroll
    for (int k = 0; k < kFvDiag; ++k) d[k] = 0.0;
    for (int bk = threadIdx.x; bk < nb; bk += kThreads) {
#pragma unroll
      for (int k = 0; k < kFvDiag; ++k) {
        double* a = diag_acc + (size_t)k * nb + bk;
        d[k] += __ldcg(a);
        *a = 0.0;
      }
    }
    const double* dt = block_fold<double, kFvDiag, kFvDiag>(d, fold);
    if (threadIdx.x < kFvDiag) ctl->diag[threadIdx.x] = dt[threadIdx.x];
    __syncthreads();
  }
  if (threadIdx.x == 0) *arrive = 0;
}

// Resets the loop control block for a new physics step of dt seconds (one thread).
__device__ __forceinline__ void fv_begin_body(FvControl* ctl, const double* dt) {
  {
    ctl->remaining = *dt;
    ctl->sub_dt = 0.0;
    ctl->max_cfl = 0.0;
    ctl->wave = 0.0;
    for (int k = 0; k < kFvDiag; ++k) ctl->diag[k] = 0.0;
    ctl->substeps = 0;
    ctl->done = 0;
    ctl->status = 0;
    ctl->cfl_limited = 0;
    ctl->static_skip = 0;
    ctl->arrive = 0;
    ctl->wait_fail = 0;
    ctl->arrive_wet = 0ull;
    for (int k = 0; k < 3; ++k) {
      ctl->wave3[k] = 0ull;
      ctl->wetn[k] = 0;
    }
  }
}

__global__ void fv_begin_kernel(FvControl* ctl, const double* dt) {
  if (threadIdx.x == 0 && blockIdx.x == 0) fv_begin_body(ctl, dt);
}

// ---------------------------------------------------------------------------
// Field conversion (host float64 layout <-> device storage).
// ---------------------------------------------------------------------------
__global__ void to_fixed_kernel(const double* __restrict__ src, int32_t* __restrict__ dst, int ny,
                                int nx, int pitch, double datum, double scale, int* range_error) {
  const long long n = (long long)ny * nx;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / nx), c = (int)(i % nx);
    const double x = rint((src[i] - datum) * scale);
    if (!(fabs(x) < 2147483647.0)) {
      atomicExch(range_error, 1);
      dst[(size_t)r * pitch + c] = 0;
    } else {
      dst[(size_t)r * pitch + c] = (int32_t)x;
    }
  }
}

__global__ void from_fixed_kernel(const int32_t* __restrict__ src, double* __restrict__ dst,
                                  int ny, int nx, int pitch, double datum, double quantum) {
  const long long n = (long long)ny * nx;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / nx), c = (int)(i % nx);
    dst[i] = (double)src[(size_t)r * pitch + c] * quantum + datum;
  }
}

__global__ void to_float_kernel(const double* __restrict__ src, float* __restrict__ dst, int ny,
                                int nx, int pitch) {
  const long long n = (long long)ny * nx;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / nx), c = (int)(i % nx);
    dst[(size_t)r * pitch + c] = (float)src[i];
  }
}

__global__ void from_float_kernel(const float* __restrict__ src, double* __restrict__ dst, int ny,
                                  int nx, int pitch) {
  const long long n = (long long)ny * nx;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / nx), c = (int)(i % nx);
    dst[i] = (double)src[(size_t)r * pitch + c];
  }
}

}  // namespace sb
