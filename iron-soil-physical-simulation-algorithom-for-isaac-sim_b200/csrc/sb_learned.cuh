// Learned repose proposal: a 4-layer 3x3 convolution net (4 -> 32 -> 32 ->
// 32 -> 4 channels, ReLU between, no bias, BF16 operands, FP32 accumulate)
// proposes per-edge outflows of a height field; they are applied in flux
// form (every transfer leaves one cell and enters its neighbour, in whole
// height quanta in the fixed-point state), and plain relaxation sweeps then
// finish to the repose tolerance.  The reference has no counterpart: its
// repose relaxation is the plain sweep (slope_model.py:273-343) alone.
//
// Convolutions are implicit GEMMs on the 5th-generation tensor cores
// (tcgen05.mma, kind::f16, operands in shared memory, accumulator in TMEM):
//
//   forward / data gradient: per output row of a 128-pixel tile, the nine
//     taps (dy, dx) are nine K-major operands (M = 128 pixels, K = input
//     channels) read straight out of the staged input rows -- a column
//     offset is a 16-byte start offset in the pixel-major staging layout --
//     against the tap's weights (N = output channels), accumulated in one
//     TMEM tile that is the output row.  The data gradient is the same kernel
//     run with the flipped, transposed weights and the ReLU mask of the
//     layer's input.
//   weight gradient: per input row, A = the row shifted by dx (M = (dx, ci),
//     K = 128 pixels) times B = output-gradient rows (N = co), accumulated in
//     TMEM over the CTA's band for the three row offsets; per-CTA partials
//     are summed in a fixed order by a second kernel.
//
// Operands use the canonical no-swizzle K-major layout: 8 x 16-byte core
// matrices, element (r, k) at ((r/8)*(K/8) + k/8)*128 + (r%8)*16 + (k%8)*2.
#pragma once

#include <cuda_bf16.h>

#include "sb_common.cuh"

namespace sb {

constexpr int kConvThreads = 128;   // 4 warps: TMEM lanes 0..127 = tile pixels
// Forward kernel: the four pixel warps plus one warp whose lane 0 issues the
// MMAs, so that a row's MMA issue overlaps the pixel warps' epilogue.
constexpr int kConvFwdThreads = 160;
constexpr int kConvTileOut = 128;   // output pixels per CTA row tile

// ---------------------------------------------------------------- tcgen05
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of sm_100; no swizzle, base offset 0
  return d;
}

// kind::f16 instruction descriptor: D f32, A/B bf16, both K-major or both
// MN-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n, bool mn_major = false) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major ? 3u << 15 : 0u) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                          int accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Warp 0 allocates ncols TMEM columns; the base address lands in *slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(slot)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols)
               : "memory");
}

// 16 consecutive f32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 consecutive f32 columns of this thread's TMEM lane (one load, one wait).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

struct ConvArgs {
  const __nv_bfloat16* in;      // [batch][h][w][cin]
  void* out;                    // bf16 [batch][h][w][cout], or f32 [batch][h][w][out_f32]
  const __nv_bfloat16* wpk;     // 3 row offsets x canonical B (n = dx*cout + co, k = ci)
  const __nv_bfloat16* mask;    // optional [batch][h][w][cout]: out *= (mask > 0)
  int batch, h, w;
  int rows_per_cta;
  int relu;
  int out_f32;                  // 0: bf16, all channels; k (multiple of 4): f32, first k channels
  int* status;                  // set to 1 if a bounded wait gave up
};

// Input rows are staged pixel-major: 130 pixels (x0-1 .. x0+128) of 16 bytes
// (8 channels) per K chunk, chunks kRowLbo bytes apart.  In the canonical
// K-major layout that is SBO = 128 B (8 consecutive pixels per core matrix,
// core matrices contiguous) and LBO = kRowLbo, so the operand for column
// offset dx is the same rows starting dx * 16 bytes later: no copies.
constexpr int kRowPixels = 130;
constexpr uint32_t kRowLbo = kRowPixels * 16;

template <int CIN, int COUT>
struct ConvSmem {
  static constexpr int W_BLOCK = COUT * CIN * 2;         // one tap's weights (canonical B)
  static constexpr int W_BYTES = 9 * W_BLOCK;
  static constexpr int ROW_BYTES = (CIN / 8) * kRowLbo;  // one staged input row
  static constexpr int SLOTS = 4;                        // rows y..y+2 in use + one in flight
  static constexpr int BYTES = W_BYTES + SLOTS * ROW_BYTES + 64;
  static constexpr uint32_t TMEM_COLS = 32;              // N = COUT <= 32 f32 columns
};

// Starts the copy of pixels [x, x + n) of an image row of C channels into a
// staged row: 16-byte pieces, neighbouring threads on neighbouring addresses
// (a thread per pixel instead asks L2 for every sector twice); zeros outside the
// image and where row is false.  ALIGNED = false: for images that do not start on 16
// bytes, whose elements are copied one by one (a 16-byte copy would fault).
template <int C, int NT, bool ALIGNED = true>
__device__ __forceinline__ void row_async(const __nv_bfloat16* __restrict__ image, int w, bool row,
                                          int r, int x, int n, uint32_t dst) {
  const __nv_bfloat16* src = image + (size_t)(row ? r : 0) * w * C;
  for (int i = threadIdx.x; i < n * (C / 8); i += NT) {
    const int p = i / (C / 8), c8 = i % (C / 8);
    const bool ok = row && x + p >= 0 && x + p < w;
    const __nv_bfloat16* from = src + (ok ? (size_t)(x + p) * C : 0) + c8 * 8;
    const uint32_t to = dst + c8 * kRowLbo + p * 16;
    if constexpr (ALIGNED) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from),
                   "r"(ok ? 16u : 0u)
                   : "memory");
    } else {
      uint32_t v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const unsigned short* e = reinterpret_cast<const unsigned short*>(from) + 2 * k;
        v[k] = ok ? (uint32_t)e[0] | (uint32_t)e[1] << 16 : 0u;
      }
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(v[0]), "r"(v[1]),
                   "r"(v[2]), "r"(v[3])
                   : "memory");
    }
  }
}

// Starts the asynchronous copy of input row r (pixels x0-1 .. x0+128) into
// a ring slot, as one group.
template <int CIN, int NT = kConvThreads>
__device__ __forceinline__ void conv_row_async(const __nv_bfloat16* __restrict__ in, int b, int h,
                                               int w, int r, int x0, unsigned char* slot) {
  row_async<CIN, NT>(in + (size_t)b * h * w * CIN, w, r >= 0 && r < h, r, x0 - 1, kRowPixels,
                     smem_u32(slot));
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ void conv_row_wait() {
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  fence_async_smem();  // the rows are read by the tensor core (async proxy)
}

// Waits until at most `pending` (0..2) of this thread's most recent row copies
// are still in flight.
__device__ __forceinline__ void conv_row_wait_pending(int pending) {
  if (pending >= 2)
    asm volatile("cp.async.wait_group 2;" ::: "memory");
  else if (pending == 1)
    asm volatile("cp.async.wait_group 1;" ::: "memory");
  else
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  fence_async_smem();
}

// Output row y of the tile at x0 from its accumulators: d = channels of pixel
// x0 + threadIdx.x, for 128 threads.  BF16: the lanes of a group of G = COUT / 8
// exchange 16-byte pieces (a transpose in log2 G steps), so that they write, and read
// the mask, side by side: a piece per lane every COUT * 2 bytes made two half-written
// sectors of each (32 -> 32 channels, 32 images of 128 x 128, 8 rows: 32.8 to 28.4 us, masked
// 39.4 to 33.5, and 10 rows: 26.2 and, the mask asked for before the exchange, 29.0).
template <int COUT>
__device__ __forceinline__ void conv_store_row(const ConvArgs& a, int b, int y, int x0,
                                               const float* d) {
  constexpr int G = COUT / 8;
  const size_t row = ((size_t)b * a.h + y) * a.w;
  if (a.out_f32) {
    const int xo = x0 + (int)threadIdx.x;
    if (xo >= a.w) return;
    const size_t pix = row + xo;
    float* op = reinterpret_cast<float*>(a.out) + pix * a.out_f32;
#pragma unroll
    for (int c = 0; c < COUT; c += 4) {
      if (c >= a.out_f32) break;
      float o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        o[j] = a.relu ? fmaxf(d[c + j], 0.f) : d[c + j];
        if (a.mask && !(__bfloat162float(a.mask[pix * COUT + c + j]) > 0.f)) o[j] = 0.f;
      }
      *reinterpret_cast<float4*>(op + c) = make_float4(o[0], o[1], o[2], o[3]);
    }
    return;
  }
  // after the exchange: piece threadIdx.x % G of the group's pixels
  const int first = x0 + (int)(threadIdx.x & ~(G - 1)), piece = (threadIdx.x & (G - 1)) * 8;
  uint4 mv[G];
  if (a.mask) {
#pragma unroll
    for (int k = 0; k < G; ++k)
      if (first + k < a.w)
        mv[k] = *reinterpret_cast<const uint4*>(a.mask + (row + first + k) * COUT + piece);
  }
  uint32_t v[G][4];
#pragma unroll
  for (int c = 0; c < G; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float lo = d[c * 8 + 2 * j], hi = d[c * 8 + 2 * j + 1];
      const __nv_bfloat162 p = a.relu ? __floats2bfloat162_rn(fmaxf(lo, 0.f), fmaxf(hi, 0.f))
                                      : __floats2bfloat162_rn(lo, hi);
      v[c][j] = *reinterpret_cast<const uint32_t*>(&p);
    }
#pragma unroll
  for (int bit = 1; bit < G; bit <<= 1) {
    const bool up = threadIdx.x & bit;
#pragma unroll
    for (int c = 0; c < G; ++c) {
      if (c & bit) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? v[c][j] : v[c | bit][j], bit);
        if (up)
          v[c][j] = got;
        else
          v[c | bit][j] = got;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < G; ++k) {
    if (first + k >= a.w) break;
    const size_t off = (row + first + k) * COUT + piece;
    if (a.mask) {
      const __nv_bfloat16* mk = reinterpret_cast<const __nv_bfloat16*>(&mv[k]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!(__bfloat162float(mk[2 * j]) > 0.f)) v[k][j] &= 0xffff0000u;
        if (!(__bfloat162float(mk[2 * j + 1]) > 0.f)) v[k][j] &= 0x0000ffffu;
      }
    }
    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + off) =
        make_uint4(v[k][0], v[k][1], v[k][2], v[k][3]);
  }
}

// D[pixel, co] for output row y: nine taps (dy, dx), each M = 128 pixels x
// K = CIN against the tap's weights (N = COUT), accumulated in TMEM.
template <int CIN, int COUT>
__device__ __forceinline__ void conv_issue_row(uint32_t tmem, uint32_t ring_base,
                                               uint32_t w_base, int y, uint32_t idesc) {
  using S = ConvSmem<CIN, COUT>;
  // descriptors are built once per row; a tap's operand is the same descriptor
  // with a 16-byte-multiple start offset added to its address field (bits
  // 0-13 hold addr >> 4; shared-memory offsets stay below 2^18, so no carry)
  const uint64_t bdesc0 = umma_desc(w_base, 128, (CIN / 8) * 128);
#pragma unroll
  for (int dy = 0; dy < 3; ++dy) {
    const uint32_t slot = ring_base + ((y - 1 + dy + S::SLOTS) % S::SLOTS) * S::ROW_BYTES;
    const uint64_t adesc0 = umma_desc(slot, kRowLbo, 128);
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) {
#pragma unroll
      for (int kk = 0; kk < CIN / 16; ++kk)
        umma_bf16(tmem, adesc0 + (uint64_t)((kk * 2 * kRowLbo + dx * 16) >> 4),
                  bdesc0 + (uint64_t)(((dy * 3 + dx) * S::W_BLOCK + kk * 256) >> 4), idesc,
                  (dy | dx | kk) != 0);
    }
  }
}

// Per CTA: one 128-pixel tile of rows [y0, y1).  Row y+1's MMAs are issued as
// soon as row y's accumulator has been read, so they run while row y's
// epilogue converts and stores; input rows are fetched by cp.async into a
// ring of SLOTS rows, SLOTS - 3 rows ahead of the rows the next MMA batch
// reads.  (Six slots measured slower than four: the extra 16 KB per CTA of
// the 32-channel layers cost a CTA per SM, and the per-row time is set by the
// tensor core's shared-memory operand reads -- 40 wavefronts per
// M128 x N32 x K16 MMA -- not by the copies.)
template <int CIN, int COUT>
__global__ void __launch_bounds__(kConvFwdThreads) conv3x3_tc_kernel(const ConvArgs a) {
  using S = ConvSmem<CIN, COUT>;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* wsm = smem;
  unsigned char* ring = smem + S::W_BYTES;
  uint64_t* bar = reinterpret_cast<uint64_t*>(ring + S::SLOTS * S::ROW_BYTES);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int x0 = blockIdx.x * kConvTileOut;
  const int y0 = blockIdx.y * a.rows_per_cta;
  const int y1 = min(y0 + a.rows_per_cta, a.h);
  const int b = blockIdx.z;
  auto slot = [&](int r) { return ring + ((r + S::SLOTS) % S::SLOTS) * S::ROW_BYTES; };

  // weights -> shared memory (already in canonical layout)
  {
    const uint4* src = reinterpret_cast<const uint4*>(a.wpk);
    uint4* dst = reinterpret_cast<uint4*>(wsm);
    for (int i = tid; i < S::W_BYTES / 16; i += kConvFwdThreads) dst[i] = src[i];
  }
  if (tid == 0) mbar_init(bar, 1);
  if (warp == 0) tmem_alloc(tslot, S::TMEM_COLS);
  conv_row_async<CIN, kConvFwdThreads>(a.in, b, a.h, a.w, y0 - 1, x0, slot(y0 - 1));
  conv_row_async<CIN, kConvFwdThreads>(a.in, b, a.h, a.w, y0, x0, slot(y0));
  conv_row_async<CIN, kConvFwdThreads>(a.in, b, a.h, a.w, y0 + 1, x0, slot(y0 + 1));
  conv_row_wait();
  fence_async_smem();  // the weights (generic stores) too
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = umma_idesc_bf16(128, COUT);
  const uint32_t w_base = smem_u32(wsm), ring_base = smem_u32(ring);
  const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const bool issuer = tid == 4 * 32;  // lane 0 of warp 4
  const bool pixel = warp < 4;         // the epilogue warps (TMEM lanes 0..127)
  unsigned phase = 0;
  bool ok = true;
  int issued = y0 + 1;  // last input row whose copy has been started
  if (y0 < y1) {
    if (issuer) {
      conv_issue_row<CIN, COUT>(tmem, ring_base, w_base, y0, idesc);
      umma_commit(bar);
    }
    // rows up to y1 are read (the last MMA batch, row y1-1, reads y1)
    for (int r = y0 + 2; r <= y0 + S::SLOTS - 2 && r <= y1; ++r) {
      conv_row_async<CIN, kConvFwdThreads>(a.in, b, a.h, a.w, r, x0, slot(r));
      issued = r;
    }
  }

  for (int y = y0; y < y1; ++y) {
    float d[COUT];  // this thread's pixel of the output row
    if (pixel) {
      ok = mbar_wait(bar, phase) && ok;
      tc_fence_after();
      if constexpr (COUT == 32)
        tmem_ld32(lane_addr, d);
      else
        tmem_ld16(lane_addr, d);
    }
    phase ^= 1;
    tc_fence_before();
    if (y + 1 < y1) conv_row_wait_pending(issued - (y + 2));  // row y+2 has landed
    __syncthreads();                                         // everyone has read the accumulator
    if (y + 1 < y1) {
      if (issuer) {
        tc_fence_after();
        conv_issue_row<CIN, COUT>(tmem, ring_base, w_base, y + 1, idesc);
        umma_commit(bar);
      }
      // the slot of row y-1 (= row y-1+SLOTS) is free: row y's MMAs have completed
      if (issued + 1 <= y1 && issued + 1 <= y + S::SLOTS - 1) {
        conv_row_async<CIN, kConvFwdThreads>(a.in, b, a.h, a.w, issued + 1, x0, slot(issued + 1));
        ++issued;
      }
    }
    if (pixel) conv_store_row<COUT>(a, b, y, x0, d);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (!ok && tid == 0 && a.status) atomicExch(a.status, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, S::TMEM_COLS);
}

// ------------------------------------------- forward, rotating accumulators
// Each staged input row is read by the tensor core once instead of three
// times.  Input row r feeds output rows r+1, r and r-1 through the kernel
// rows dy = 0, 1, 2; three TMEM accumulators of COUT columns (slot s holds
// output rows y with y % 3 == s) sit side by side, and for every column
// offset dx one MMA of N = 3 * COUT writes all three: its B operand is the
// three dy weight blocks in the order the slots want for this r.  The weights
// are staged per dx as five blocks W(2) W(1) W(0) W(2) W(1), so the operand
// for row r is the three consecutive blocks starting at block (1 - r) mod 3.
// Every MMA accumulates; a slot is cleared (tcgen05.st of zeros) right after
// its output row has been read, before the next row's MMAs add to it.  Per
// output row this issues 3 * CIN/16 MMAs (N = 3 * COUT) instead of
// 9 * CIN/16 (N = COUT): 2.1x less operand traffic from shared memory, which
// bounds the M128 x N32 form.  A CTA reads input rows y0-1 .. y1, so it runs
// two extra rows per row band.
template <int CIN, int COUT>
struct ConvRotSmem {
  static constexpr int W_BLOCK = COUT * CIN * 2;         // one (dy, dx) weight block
  static constexpr int W_BYTES = 15 * W_BLOCK;           // 3 dx x 5 staged blocks
  static constexpr int ROW_BYTES = (CIN / 8) * kRowLbo;  // one staged input row
  static constexpr int SLOTS = 4;                        // row in the MMA + three in flight
  static constexpr int BYTES = W_BYTES + SLOTS * ROW_BYTES + 64;
  static constexpr uint32_t TMEM_COLS = 3 * COUT <= 64 ? 64 : 128;
};

// Zeros COLS consecutive f32 columns of this thread's TMEM lane.
template <int COLS>
__device__ __forceinline__ void tmem_zero(uint32_t taddr) {
  static_assert(COLS == 16 || COLS == 32, "16 or 32 columns");
  const uint32_t z = 0u;
  if constexpr (COLS == 32) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
        "%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
        "r"(z)
        : "memory");
  } else {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
        "%1,%1};" ::"r"(taddr),
        "r"(z)
        : "memory");
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// MMAs of input row r (staged in its ring slot) into the three accumulators.
template <int CIN, int COUT>
__device__ __forceinline__ void conv_rot_issue(uint32_t tmem, uint32_t slot_addr, uint32_t w_base,
                                               int r, uint32_t idesc) {
  using S = ConvRotSmem<CIN, COUT>;
  const int first = ((1 - r) % 3 + 3) % 3;  // staged block that feeds accumulator slot 0
  const uint64_t adesc0 = umma_desc(slot_addr, kRowLbo, 128);
  const uint64_t bdesc0 = umma_desc(w_base, 128, (CIN / 8) * 128);
#pragma unroll
  for (int dx = 0; dx < 3; ++dx) {
#pragma unroll
    for (int kk = 0; kk < CIN / 16; ++kk)
      umma_bf16(tmem, adesc0 + (uint64_t)((kk * 2 * kRowLbo + dx * 16) >> 4),
                bdesc0 + (uint64_t)(((dx * 5 + first) * S::W_BLOCK + kk * 256) >> 4), idesc, 1);
  }
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(kConvThreads) conv3x3_rot_kernel(const ConvArgs a) {
  using S = ConvRotSmem<CIN, COUT>;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* wsm = smem;
  unsigned char* ring = smem + S::W_BYTES;
  uint64_t* bar = reinterpret_cast<uint64_t*>(ring + S::SLOTS * S::ROW_BYTES);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int x0 = blockIdx.x * kConvTileOut;
  const int y0 = blockIdx.y * a.rows_per_cta;
  const int y1 = min(y0 + a.rows_per_cta, a.h);
  const int b = blockIdx.z;
  auto slot = [&](int r) { return ring + ((r + S::SLOTS) % S::SLOTS) * S::ROW_BYTES; };

  // weights -> shared memory: per dx the blocks of dy = 2, 1, 0, 2, 1 (the
  // packed input holds block (dy * 3 + dx) for each (dy, dx))
  {
    constexpr int kDyOf[5] = {2, 1, 0, 2, 1};
    constexpr int kChunks = S::W_BLOCK / 16;
    const uint4* src = reinterpret_cast<const uint4*>(a.wpk);
    uint4* dst = reinterpret_cast<uint4*>(wsm);
    for (int i = tid; i < 15 * kChunks; i += kConvThreads) {
      const int blk = i / kChunks, off = i % kChunks;
      const int dx = blk / 5, j = blk % 5;
      dst[i] = src[(kDyOf[j] * 3 + dx) * kChunks + off];
    }
  }
  if (tid == 0) mbar_init(bar, 1);
  if (warp == 0) tmem_alloc(tslot, S::TMEM_COLS);
  const int r_first = y0 - 1, r_last = y1;  // input rows this CTA reads
  int issued = r_first - 1;                 // last input row whose copy has been started
  for (int r = r_first; r <= r_first + S::SLOTS - 1 && r <= r_last; ++r) {
    conv_row_async<CIN>(a.in, b, a.h, a.w, r, x0, slot(r));
    issued = r;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = umma_idesc_bf16(128, 3 * COUT);
  const uint32_t w_base = smem_u32(wsm);
  const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
  // all three accumulators start at zero
#pragma unroll
  for (int sl = 0; sl < 3; ++sl) tmem_zero<COUT>(lane_addr + (uint32_t)(sl * COUT));
  conv_row_wait_pending(issued - r_first);  // row r_first has landed
  fence_async_smem();                       // the weights (generic stores) too
  tc_fence_before();
  __syncthreads();
  unsigned phase = 0;
  bool ok = true;
  if (y0 < y1 && tid == 0) {
    tc_fence_after();
    conv_rot_issue<CIN, COUT>(tmem, smem_u32(slot(r_first)), w_base, r_first, idesc);
    umma_commit(bar);
  }
  for (int r = r_first; r <= r_last && y0 < y1; ++r) {
    ok = mbar_wait(bar, phase) && ok;
    phase ^= 1;
    tc_fence_after();
    // output row r - 1 is complete: read its accumulator, then clear the slot
    // for the output row r + 2 that the next MMAs start
    const int yo = r - 1;
    const uint32_t acc = lane_addr + (uint32_t)((((yo % 3) + 3) % 3) * COUT);
    float d[COUT];
    if constexpr (COUT == 32)
      tmem_ld32(acc, d);
    else
      tmem_ld16(acc, d);
    tmem_zero<COUT>(acc);
    tc_fence_before();
    if (r + 1 <= r_last) conv_row_wait_pending(issued - (r + 1));  // row r + 1 has landed
    __syncthreads();  // accumulator read and cleared by every thread, row r + 1 staged
    if (r + 1 <= r_last) {
      if (tid == 0) {
        tc_fence_after();
        conv_rot_issue<CIN, COUT>(tmem, smem_u32(slot(r + 1)), w_base, r + 1, idesc);
        umma_commit(bar);
      }
      // row r's MMAs have completed: its slot takes row r + SLOTS
      if (issued + 1 <= r_last && issued + 1 <= r + S::SLOTS) {
        conv_row_async<CIN>(a.in, b, a.h, a.w, issued + 1, x0, slot(issued + 1));
        ++issued;
      }
    }
    if (yo >= y0 && yo < y1) conv_store_row<COUT>(a, b, yo, x0, d);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (!ok && tid == 0 && a.status) atomicExch(a.status, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, S::TMEM_COLS);
}

// ------------------------------------------------------- packed weights
// The network's four layers (channels 16-32-32-32-16), one after another.
constexpr int kNetLayers = 4;
struct PackArgs {
  const float* w[kNetLayers];  // [3][3][ci][co]
  __nv_bfloat16* out;
};

// W[3][3][ci][co] -> the canonical K-major operand of each tap (rows n = output
// channel, k = input channel; 8 x 8 core matrices, (n / 8, k / 8) blocks).
// backward: of the data gradient's weights W'[dy][dx][co][ci] = W[2-dy][2-dx][ci][co].
// All layers in one launch: bound by launches, not by its 166 KB (as a gather, a cast
// and two flips per layer: 28 launches, 81 us of kernels in a training step).
__global__ void __launch_bounds__(256) learned_pack_kernel(const PackArgs a, int backward) {
  constexpr int kCh[kNetLayers + 1] = {16, 32, 32, 32, 16};
  int i = blockIdx.x * 256 + threadIdx.x;
  __nv_bfloat16* out = a.out + i;
#pragma unroll
  for (int l = 0; l < kNetLayers; ++l) {
    const int ci = kCh[l], co = kCh[l + 1], block = ci * co;
    if (i < 0 || i >= 9 * block) {
      i -= 9 * block;  // of a later layer, or (negative) already done
      continue;
    }
    const int kdim = backward ? co : ci;
    const int tap = i / block, off = i - tap * block, core = off >> 6;
    const int n = core / (kdim >> 3) * 8 + ((off >> 3) & 7);
    const int k = core % (kdim >> 3) * 8 + (off & 7);
    const int src = backward ? ((8 - tap) * ci + n) * co + k : (tap * ci + k) * co + n;
    *out = __float2bfloat16_rn(a.w[l][src]);
    return;
  }
}

// ----------------------------------------------------------- weight grad
struct WgradArgs {
  const __nv_bfloat16* in;    // layer input [batch][h][w][cin]
  const __nv_bfloat16* grad;  // gradient at the layer output [batch][h][w][cout]
  float* partial;             // per CTA: [3 dy][3 dx][cin][cout]
  int batch, h, w;
  int rows;    // output rows of a CTA's band
  int tiles;   // bands side by side (128 pixels each)
  int chunks;  // bands over the height
  int* status;
};

template <int CIN, int COUT>
struct WgradSmem {
  static constexpr uint32_t ROW = 4 * kRowLbo;  // input row: room for 32 channels
  static constexpr uint32_t G_ROW = (COUT / 8) * kRowLbo;
  static constexpr uint32_t STAGE = 4 * ROW + 2 * G_ROW;
  static constexpr uint32_t FOLD = 9 * CIN * (COUT + 1) * 4;  // in the place of the stages
  static constexpr uint32_t BYTES = (2 * STAGE > FOLD ? 2 * STAGE : FOLD) + 64;
  static constexpr uint32_t TMEM_COLS = COUT == 32 ? 256 : 128;  // 3 dx x 2 rows x COUT
};

// dW[dy][dx][ci][co] = sum over pixels of in[y + dy - 1][x + dx - 1][ci] g[y][x][co].
//
// Both operands are contracted over pixels, so both are MN-major in the staged rows
// as they lie in memory (16 bytes = 8 channels of a pixel; core matrices of 8 pixels,
// 128 B apart along K; channel groups kRowLbo apart along M and N): nothing is
// transposed, and a dx is the same rows dx * 16 bytes on.  A step takes two output
// rows y, y + 1 (N = 2 x COUT) against the four input rows y - 1 .. y + 2 (M = 4 x 32
// channels): six of the eight row pairs are the dy = 0, 1, 2 of the two rows, the other
// two are not read.  The next step's rows are in flight during the MMAs.
//
// An MMA of K = 16 costs about 75 cycles for any N up to 96 here, so two rows per MMA
// halve the tensor time; the two rows' windows share no buffer, which leaves one set of
// accumulators (192 columns) and room for two CTAs per SM.  32 images of 128 x 128 x 32
// (67 MB, 10 us at the copy rate): 31 to 40 us; one row per step and one CTA of two
// bands per SM 57 to 61 us; rows transposed with 2-byte stores 147 to 186 us.
template <int CIN, int COUT, bool ALIGNED>
__global__ void __launch_bounds__(kConvThreads) conv3x3_wgrad_tc_kernel(const WgradArgs a) {
  using S = WgradSmem<CIN, COUT>;
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + S::BYTES - 64);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = smem_u32(smem);
  const int q = blockIdx.x / a.tiles, img = q / a.chunks;
  const int x0 = ((int)blockIdx.x - q * a.tiles) * 128;
  const int y0 = (q - img * a.chunks) * a.rows, y1 = min(y0 + a.rows, a.h);
  const int npx = (min(a.w - x0, 128) + 15) / 16 * 16;  // K of a step's MMAs
  const int steps = (y1 - y0 + 1) / 2;
  const __nv_bfloat16* in = a.in + (size_t)img * a.h * a.w * CIN;
  const __nv_bfloat16* grad = a.grad + (size_t)img * a.h * a.w * COUT;
  auto load = [&](int i) {
    const uint32_t dst = base + (i & 1) * S::STAGE;
    const int y = y0 + 2 * i;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      row_async<CIN, kConvThreads, ALIGNED>(in, a.w, y - 1 + k >= 0 && y - 1 + k < a.h, y - 1 + k,
                                            x0 - 1, npx + 2, dst + k * S::ROW);
#pragma unroll
    for (int k = 0; k < 2; ++k)
      row_async<COUT, kConvThreads, ALIGNED>(grad, a.w, y + k < y1, y + k, x0, npx,
                                             dst + 4 * S::ROW + k * S::G_ROW);
  };
  load(0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 1, 1);
  }
  if (warp == 0) tmem_alloc(tslot, S::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
  // a band's last row without a partner is a step of its own columns alone (N =
  // COUT): against the zeros in the partner's place an infinite input would leave a
  // NaN in outputs that it has no part in
  const uint32_t idesc_two = umma_idesc_bf16(128, 2 * COUT, true);
  const uint32_t idesc_one = umma_idesc_bf16(128, COUT, true);
  bool ok = true;
  for (int i = 0; i < steps; ++i) {
    const uint32_t idesc = y0 + 2 * i + 1 < y1 ? idesc_two : idesc_one;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_async_smem();
    __syncthreads();  // step i's rows are staged
    if (tid == 0) {
      tc_fence_after();
      const uint32_t src = base + (i & 1) * S::STAGE;
      const uint64_t adesc = umma_desc(src, 128, kRowLbo);
      const uint64_t bdesc = umma_desc(src + 4 * S::ROW, 128, kRowLbo);
      for (int kk = 0; kk < npx / 16; ++kk)
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
          umma_bf16(tmem + dx * 2 * COUT, adesc + (uint64_t)(kk * 16 + dx),
                    bdesc + (uint64_t)(kk * 16), idesc, i > 0 || kk > 0);
      umma_commit(bar + (i & 1));
    }
    // step i - 1's MMAs have read the stage that step i + 1 takes
    if (i > 0) ok = mbar_wait(bar + ((i - 1) & 1), ((i - 1) >> 1) & 1) && ok;
    if (i + 1 < steps) load(i + 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  ok = mbar_wait(bar + ((steps - 1) & 1), ((steps - 1) >> 1) & 1) && ok;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  tc_fence_after();
  __syncthreads();  // every MMA has completed: the stages' place takes the sums
  // warp = input row of the window, lane = ci.  Row s and output row j (0, 1) of the
  // step are dy = s - j: first the shares of j = 0, then those of j = 1 on top (a band
  // of one row has none).
  float* fold = reinterpret_cast<float*>(smem);
#pragma unroll 1
  for (int j = 0; j < 2; ++j) {
    const int dy = warp - j;
    if (dy >= 0 && dy < 3 && y0 + j < y1) {
#pragma unroll 1
      for (int dx = 0; dx < 3; ++dx) {
        float v[COUT];
        if constexpr (COUT == 32)
          tmem_ld32(lane_addr + (uint32_t)((dx * 2 + j) * COUT), v);
        else
          tmem_ld16(lane_addr + (uint32_t)((dx * 2 + j) * COUT), v);
        if (lane < CIN) {
          float* f = fold + ((dy * 3 + dx) * CIN + lane) * (COUT + 1);
#pragma unroll
          for (int co = 0; co < COUT; ++co) f[co] = j == 0 ? v[co] : f[co] + v[co];
        }
      }
    }
    __syncthreads();
  }
  float* out = a.partial + (size_t)blockIdx.x * (9 * CIN * COUT);
  for (int i = tid; i < 9 * CIN * COUT; i += kConvThreads)
    out[i] = fold[i / COUT * (COUT + 1) + i % COUT];
  if (!ok && tid == 0 && a.status) atomicExch(a.status, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, S::TMEM_COLS);
}

// dw[i] = sum over CTAs of partial[cta][i], in FP64 and a fixed order: 32 outputs per
// block, eight threads each (one thread per output read 256 CTAs one after another:
// 25 us).
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* __restrict__ partial,
                                                           int nctas, int n,
                                                           float* __restrict__ dw) {
  __shared__ double part[8][32];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (i < n) {
#pragma unroll 4
    for (int c = slice; c < nctas; c += 8) s += (double)partial[(size_t)c * n + i];
  }
  part[slice][lane] = s;
  __syncthreads();
  if (slice == 0 && i < n) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += part[k][lane];
    dw[i] = (float)s;
  }
}

// --------------------------------------------------- features and fluxes
// Edges of cell (r, c): 0 east (r, c+1), 1 north (r+1, c), 2 north-east
// (r+1, c+1), 3 north-west (r+1, c-1); lengths dx, dy, and the diagonal.
__device__ __forceinline__ void edge_of(int k, int& dr, int& dc) {
  dr = k == 0 ? 0 : 1;
  dc = k == 0 ? 1 : (k == 1 ? 0 : (k == 2 ? 1 : -1));
}

struct LearnedGeom {
  int batch, h, w, pitch;       // height fields [batch][h][pitch]
  double dx, dy, tan_crit;
  double Q;                     // FX quantum (0 for FP64 heights)
  double datum;
};

// The per-pixel kernels below take one image row per block iteration
// (blockIdx.x strides over batch * h rows, threads over the row's columns), so
// no pixel index is divided into (batch, row, column).

// Features: per edge k, (H[c] - H[n_k]) / (L_k tan_crit) as BF16 channels
// 0..3 of a 16-channel pixel (12 zero channels); 0 for edges leaving the grid.
template <typename HT>
__global__ void learned_features_kernel(const LearnedGeom g, const HT* __restrict__ hgt,
                                        __nv_bfloat16* __restrict__ feat) {
  // a proposal's network kernel stages its weights meanwhile (it waits for this
  // kernel's end before it reads the features)
  cudaTriggerProgrammaticLaunchCompletion();
  const double diag = sqrt(g.dx * g.dx + g.dy * g.dy);
  const double scale = g.Q > 0.0 ? g.Q : 1.0;
  const double inv_l[4] = {scale / (g.dx * g.tan_crit), scale / (g.dy * g.tan_crit),
                           scale / (diag * g.tan_crit), scale / (diag * g.tan_crit)};
  for (int row = blockIdx.x; row < g.batch * g.h; row += gridDim.x) {
    const int bb = row / g.h, r = row - bb * g.h;
    const HT* H = hgt + (size_t)bb * g.h * g.pitch;
    for (int c = threadIdx.x; c < g.w; c += blockDim.x) {
      const double hc = (double)H[(size_t)r * g.pitch + c];
      __align__(16) __nv_bfloat16 f[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) f[k] = __float2bfloat16_rn(0.f);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        int dr, dc;
        edge_of(k, dr, dc);
        const int rn = r + dr, cn = c + dc;
        if (rn < g.h && cn >= 0 && cn < g.w)
          f[k] = __float2bfloat16_rn((float)((hc - (double)H[(size_t)rn * g.pitch + cn]) * inv_l[k]));
      }
      uint4* dst = reinterpret_cast<uint4*>(feat + ((size_t)row * g.w + c) * 16);
      dst[0] = reinterpret_cast<const uint4*>(f)[0];
      dst[1] = reinterpret_cast<const uint4*>(f)[1];
    }
  }
}

// Fixed point: transfers in whole quanta per edge (int32 [pixel][4]), rounded
// toward zero, then gathered -- every quantum leaves one cell and enters one
// neighbour.  Q is a power of two, so scaling by it commutes with every
// rounding, and truncation with the clamp to half the (whole)
// height difference: trunc(clamp(t, lim) / Q) = clamp(trunc(t / Q), |dq| / 2).
// Four dependent double operations instead of fifteen.
__device__ __forceinline__ int learned_quanta(float flux, int hc, int hn, double tan_crit,
                                              double dxq) {
  const int q = __double2int_rz((double)flux * tan_crit * dxq);  // saturates
  const unsigned u = hc > hn ? (unsigned)hc - (unsigned)hn : (unsigned)hn - (unsigned)hc;
  const int lim = (int)(u >> 1);
  return min(max(q, -lim), lim);
}

__global__ void learned_quantize_kernel(const LearnedGeom g, const int32_t* __restrict__ hq,
                                        const float* __restrict__ flux /*[pixel][4]*/,
                                        int32_t* __restrict__ tq /*[pixel][4]*/) {
  const double dxq = g.dx * (1.0 / g.Q);
  cudaGridDependencySynchronize();
  for (int row = blockIdx.x; row < g.batch * g.h; row += gridDim.x) {
    const int bb = row / g.h, r = row - bb * g.h;
    const int32_t* H = hq + (size_t)bb * g.h * g.pitch;
    for (int c = threadIdx.x; c < g.w; c += blockDim.x) {
      const size_t i = (size_t)row * g.w + c;
      const int hc = H[(size_t)r * g.pitch + c];
      const float4 fl = *reinterpret_cast<const float4*>(flux + i * 4);
      const float fk[4] = {fl.x, fl.y, fl.z, fl.w};
      int q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        int dr, dc;
        edge_of(k, dr, dc);
        const int rn = r + dr, cn = c + dc;
        q[k] = 0;
        if (rn < g.h && cn >= 0 && cn < g.w)
          q[k] = learned_quanta(fk[k], hc, H[(size_t)rn * g.pitch + cn], g.tan_crit, dxq);
      }
      *reinterpret_cast<int4*>(tq + i * 4) = make_int4(q[0], q[1], q[2], q[3]);
    }
  }
}

__global__ void learned_apply_fx_kernel(const LearnedGeom g, int32_t* __restrict__ hq,
                                        const int32_t* __restrict__ tq) {
  cudaGridDependencySynchronize();
  for (int row = blockIdx.x; row < g.batch * g.h; row += gridDim.x) {
    const int bb = row / g.h, r = row - bb * g.h;
    int32_t* H = hq + (size_t)bb * g.h * g.pitch;
    for (int c = threadIdx.x; c < g.w; c += blockDim.x) {
      const size_t i = (size_t)row * g.w + c;
      const int4 own = *reinterpret_cast<const int4*>(tq + i * 4);
      long long d = -(long long)own.x - own.y - own.z - own.w;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        int dr, dc;
        edge_of(k, dr, dc);
        const int rs = r - dr, cs = c - dc;  // the cell whose edge k ends here
        if (rs >= 0 && cs >= 0 && cs < g.w)
          d += tq[(((size_t)bb * g.h + rs) * g.w + cs) * 4 + k];
      }
      H[(size_t)r * g.pitch + c] = (int32_t)((long long)H[(size_t)r * g.pitch + c] + d);
    }
  }
}

// Training loss: predicted height change dH = -div(t) (unlimited transfers,
// f32) against the plain relaxation's change; writes the residual per pixel
// and the loss partial per block (blockDim a multiple of 32, at most 1024).
__global__ void learned_loss_kernel(const LearnedGeom g, const float* __restrict__ flux,
                                    const float* __restrict__ target_dh /*[pixel] metres*/,
                                    float* __restrict__ resid /*[pixel]*/,
                                    double* __restrict__ loss_part, float inv_scale2_n) {
  const long long n = (long long)g.batch * g.h * g.w;
  const float s = (float)(g.tan_crit * g.dx);
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % g.w);
    const int r = (int)((i / g.w) % g.h);
    const int bb = (int)(i / ((long long)g.w * g.h));
    float dh = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      int dr, dc;
      edge_of(k, dr, dc);
      if (r + dr < g.h && c + dc >= 0 && c + dc < g.w) dh -= flux[i * 4 + k] * s;
      const int rs = r - dr, cs = c - dc;
      if (rs >= 0 && cs >= 0 && cs < g.w)
        dh += flux[(((long long)bb * g.h + rs) * g.w + cs) * 4 + k] * s;
    }
    const float e = dh - target_dh[i];
    resid[i] = e;
    acc += (double)e * (double)e;
  }
  acc = warp_sum(acc);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w2 = 0; w2 < (int)(blockDim.x >> 5); ++w2) t += red[w2];
    loss_part[blockIdx.x] = t * (double)inv_scale2_n;
  }
}

// dL/dflux[c][k] = 2 s (e[n_k] - e[c]) / (scale^2 N) for edges inside the grid.
__global__ void learned_dflux_kernel(const LearnedGeom g, const float* __restrict__ resid,
                                     __nv_bfloat16* __restrict__ dflux, float inv_scale2_n) {
  const long long n = (long long)g.batch * g.h * g.w;
  const float s = (float)(g.tan_crit * g.dx);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % g.w);
    const int r = (int)((i / g.w) % g.h);
    const int bb = (int)(i / ((long long)g.w * g.h));
    __align__(16) __nv_bfloat16 f[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) f[k] = __float2bfloat16_rn(0.f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      int dr, dc;
      edge_of(k, dr, dc);
      const int rn = r + dr, cn = c + dc;
      if (rn < g.h && cn >= 0 && cn < g.w) {
        const float en = resid[((long long)bb * g.h + rn) * g.w + cn];
        f[k] = __float2bfloat16_rn(2.f * s * (en - resid[i]) * inv_scale2_n);
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(dflux + i * 16);
    dst[0] = reinterpret_cast<const uint4*>(f)[0];
    dst[1] = reinterpret_cast<const uint4*>(f)[1];
  }
}

}  // namespace sb
