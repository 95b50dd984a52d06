// Frame CDEF (src/coder/frame_cdef.rs:49-520 and src/cdef.rs).
//
// Device side, per frame:
//   cdef_dir_kernel      one thread per luma 8x8: the spec direction search
//                        (src/cdef.rs:89-178), plus the per-64x64-unit
//                        directional-variance sums of the non-skip blocks that
//                        the strength search gates on.
//   cdef_tab_kernel      a warp per 8x8 of a plane (two samples a lane), or per
//                        two or four smaller chroma blocks: all 12 (pri, sec) candidates of the block at once -- every tap
//                        is read and constrained once per strength, as the
//                        reference's fused candidate routine does
//                        (src/cdef.rs:651-800) -- then the decision distortion of
//                        each: the weighted SSE in the AVX2 lane order
//                        (src/avx/rd.rs:767-848) for whole blocks, plain SSE for
//                        blocks the visible window cuts; summed per unit with
//                        64-bit integer atomics (order-free).
//   cdef_apply_kernel    the same lanes: the chosen strengths filtered from a pre-CDEF snapshot into the
//                        reconstruction (src/coder/frame_cdef.rs:960-1125).
//   the strength search   the staged search over the unit tables
//                        (src/coder/frame_cdef.rs:116-520) as one cluster or a
//                        chain of small kernels, so that tables, search and apply
//                        run back to back on the stream and the host reads the
//                        decision once at the end.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "../../include/maroontree_b200.h"

namespace {

constexpr int kVeryLarge = 0x4000;  // the spec's out-of-frame tap value
constexpr int kNCand = 12;

// Cdef_Directions (row, col) per direction and tap distance.
__constant__ int8_t cDirs[8][2][2] = {
    {{-1, 1}, {-2, 2}}, {{0, 1}, {-1, 2}}, {{0, 1}, {0, 2}}, {{0, 1}, {1, 2}},
    {{1, 1}, {2, 2}},   {{1, 0}, {2, 1}},  {{1, 0}, {2, 0}}, {{1, 0}, {2, -1}},
};
__constant__ int8_t cUvDir422[8] = {7, 0, 2, 4, 5, 6, 6, 6};

// Weighted-SSE 4x4 DCT basis and weights (src/rd_sse.rs:1400-1430).
constexpr float kRawMean = 0.4625f;
__constant__ float cD[4][4] = {{0.5f, 0.5f, 0.5f, 0.5f},
                               {0.6532815f, 0.27059805f, -0.27059805f, -0.6532815f},
                               {0.5f, -0.5f, -0.5f, 0.5f},
                               {0.27059805f, -0.6532815f, 0.6532815f, -0.27059805f}};
__constant__ float cW[4][4] = {
    {1.8f / kRawMean, 1.0f / kRawMean, 0.4f / kRawMean, 0.2f / kRawMean},
    {1.0f / kRawMean, 0.8f / kRawMean, 0.2f / kRawMean, 0.2f / kRawMean},
    {0.4f / kRawMean, 0.2f / kRawMean, 0.2f / kRawMean, 0.2f / kRawMean},
    {0.2f / kRawMean, 0.2f / kRawMean, 0.2f / kRawMean, 0.2f / kRawMean},
};

__host__ __device__ __forceinline__ int log2_floor(int v) {
#ifdef __CUDA_ARCH__
  return v <= 0 ? 0 : 31 - __clz(v);
#else
  return v <= 0 ? 0 : 31 - __builtin_clz((unsigned)v);
#endif
}

// adjust_pri (src/cdef.rs:181-189): primary strength scaled by the block variance.
__host__ __device__ __forceinline__ int adjust_pri(int pri, int var) {
  if (var == 0) return 0;
  const int vs = var >> 6;
  const int l = vs != 0 ? min(log2_floor(vs), 12) : 0;
  return (pri * (4 + l) + 8) >> 4;
}

__device__ __forceinline__ int strength_shift(int s, int damping) {
  return s == 0 ? 0 : max(damping - log2_floor(s), 0);
}

struct Geo {
  int w8, h8, cw8, ch8, nbx, nby, uc, ur;
  int disp_w, disp_h, cw_vis, ch_vis;
  int sub_x, sub_y, bd, damping;
};

// ---------------------------------------------------------------------------
// Direction search: one thread per luma 8x8.
__global__ void __launch_bounds__(128) cdef_dir_kernel(const uint16_t* __restrict__ py, Geo g,
                                                       const uint8_t* __restrict__ skip8, uint8_t* __restrict__ dirs,
                                                       int32_t* __restrict__ vars,
                                                       unsigned long long* __restrict__ dv_sum,
                                                       int* __restrict__ dv_cnt) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= g.nbx * g.nby) return;
  const int bx = b % g.nbx, by = b / g.nbx;
  const int x = bx * 8, y = by * 8;
  const int cs = g.bd - 8;
  int part[8][15];
#pragma unroll
  for (int d = 0; d < 8; d++)
#pragma unroll
    for (int k = 0; k < 15; k++) part[d][k] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int yy = min(y + i, g.h8 - 1);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int xx = min(x + j, g.w8 - 1);
      const int p = (py[(size_t)yy * g.w8 + xx] >> cs) - 128;
      part[0][i + j] += p;
      part[1][i + j / 2] += p;
      part[2][i] += p;
      part[3][3 + i - j / 2] += p;
      part[4][7 + i - j] += p;
      part[5][3 - i / 2 + j] += p;
      part[6][j] += p;
      part[7][i / 2 + j] += p;
    }
  }
  long long cost[8];
#pragma unroll
  for (int d = 0; d < 8; d++) cost[d] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    cost[2] += (long long)part[2][i] * part[2][i];
    cost[6] += (long long)part[6][i] * part[6][i];
  }
  cost[2] *= 105;
  cost[6] *= 105;
  const long long kDiv[8] = {0, 840, 420, 280, 210, 168, 140, 120};
#pragma unroll
  for (int i = 0; i < 7; i++) {
    cost[0] += ((long long)part[0][i] * part[0][i] + (long long)part[0][14 - i] * part[0][14 - i]) * kDiv[i + 1];
    cost[4] += ((long long)part[4][i] * part[4][i] + (long long)part[4][14 - i] * part[4][14 - i]) * kDiv[i + 1];
  }
  cost[0] += (long long)part[0][7] * part[0][7] * 105;
  cost[4] += (long long)part[4][7] * part[4][7] * 105;
#pragma unroll
  for (int s = 1; s < 8; s += 2) {
#pragma unroll
    for (int i = 0; i < 5; i++) cost[s] += (long long)part[s][3 + i] * part[s][3 + i] * 105;
#pragma unroll
    for (int i = 0; i < 3; i++)
      cost[s] += ((long long)part[s][i] * part[s][i] + (long long)part[s][10 - i] * part[s][10 - i]) * kDiv[2 * i + 2];
  }
  int best_dir = 0;
  long long best = cost[0];
#pragma unroll
  for (int d = 1; d < 8; d++)
    if (cost[d] > best) {
      best = cost[d];
      best_dir = d;
    }
  long long opp = cost[0];
#pragma unroll
  for (int d = 0; d < 8; d++)
    if (d == ((best_dir + 4) & 7)) opp = cost[d];
  const int var = (int)((best - opp) >> 10);
  dirs[b] = (uint8_t)best_dir;
  vars[b] = var;
  if (dv_sum && !skip8[b]) {
    const int u = (by >> 3) * g.uc + (bx >> 3);
    atomicAdd(&dv_sum[u], (unsigned long long)(long long)var);
    atomicAdd(&dv_cnt[u], 1);
  }
}

// ---------------------------------------------------------------------------
// The candidate tables (src/cdef.rs:651-800 semantics): a warp per 8x8 block of
// a plane, or per two 4x8 or four 4x4 chroma blocks; a lane has two neighbouring
// samples, whose 16-bit halves go through the taps together.
//
// Integer work per sample bounds it (four primary taps under three strengths,
// eight secondary ones under two, eight more in direction 0, twelve outputs), so
// the halves share it: a tap's |difference| is the packed maximum less the
// packed minimum, max(s - (a >> shift), 0) is max(s, y) - y, and signed halves
// are summed as one linear 32-bit number, lo + 65536 hi, with a bias added before
// they are taken apart again.  The block and its surround are read once into
// shared memory, a second copy one sample to the left, so that a pair at any
// offset is one aligned word.  Errors are kept as floats (made by the exponent of
// 2^23, exact) for the weighted SSE, whose sums run over lanes in the reference's
// order.  Against a thread per sample with bounds-checked taps from global
// memory, integer errors converted by each of the transform's four readers and
// 48 of 64 threads in the SSE: 4096x4096 4:4:4 2.30 -> 1.66 ms, 1920x1080 4:2:0
// 269 -> 112 us (82 % of the issue slots, 1,700 instructions a block).
struct TabArgs {
  const uint16_t* rec[3];
  const uint16_t* src[3];
  unsigned long long* tab[3];
};

constexpr uint32_t kHalves = 0x00010001u;

__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("min.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// All ones in each half whose top bit is set.
__device__ __forceinline__ uint32_t half_signs(uint32_t v) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %1, 0xBB99;" : "=r"(r) : "r"(v));
  return r;
}

template <int BW, int BH>
struct TabShape {
  static constexpr int kLanes = BW * BH / 2;       // per block
  static constexpr int kBlocks = 32 / kLanes;      // per warp
  static constexpr int kPitch = BW + 4;            // words of a patch row: both copies
  static constexpr int kRows = BH + 4;
  static constexpr int kErr = BW == 8 ? 72 : BW * BH + 4;  // floats of a candidate's errors
};

// The word offset of the pair at (dr, dc) of a patch from the one at (0, 0).
template <int PITCH>
__host__ __device__ constexpr int pair_off(int dr, int dc) {
  return (dc & 1) * (PITCH / 2) + dr * PITCH + ((2 + dc) >> 1) - 1;
}

// A lane's pair of samples in its block's patch.
struct PairTaps {
  const uint32_t* C;  // its word
  uint32_t c2;        // the samples
  bool out;           // some lane's patch reaches out of the frame
  // The pair at offset off, its |differences| from the samples, and all ones in
  // the halves where it is not above them.
  __device__ __forceinline__ uint32_t at(int off, uint32_t& a, uint32_t& neg) const {
    uint32_t v = C[off];
    if (out) {  // out of the frame: no difference
      const uint32_t m = half_signs((v & 0x40004000u) << 1);
      v = (v & ~m) | (c2 & m);
    }
    a = max2(v, c2) - min2(v, c2);
    neg = half_signs((c2 | 0x80008000u) - v);
    return v;
  }
};

// sum += w times the differences constrained by strength s (both halves) with
// shift sh (mask: what a shifted half keeps).
__device__ __forceinline__ void add_constrained(uint32_t& sum, uint32_t a, uint32_t neg, uint32_t s, int sh,
                                                uint32_t mask, int w) {
  const uint32_t y = (a >> sh) & mask;
  const uint32_t r = min2(max2(s, y) - y, a);
  sum += (uint32_t)w * (r - 2 * (r & neg));
}

// c + ((8 + sum - (sum < 0)) >> 4) in each half, biased by 128.
__device__ __forceinline__ uint32_t filtered(uint32_t c2, uint32_t sum) {
  const uint32_t q = sum + 0x08000800u;  // halves 2048 + sum
  return c2 + (((q + 0x00070007u + ((q >> 11) & kHalves)) >> 4) & 0x0fff0fffu);
}

// The block at (x, y) of the plane with two samples around it, by the block's
// lanes (this one l).  The whole warp calls it.
template <int BW, int BH>
__device__ __forceinline__ PairTaps load_patch(const uint16_t* plane, int stride, int rows, int x, int y, int l,
                                               uint32_t* P) {
  using Sh = TabShape<BW, BH>;
  constexpr int kPitch = Sh::kPitch;
  bool out = false;
  uint16_t* const H = reinterpret_cast<uint16_t*>(P);
  for (int i = l; i < Sh::kRows * kPitch; i += Sh::kLanes) {
    const int r = i / kPitch, c = i - r * kPitch;
    const int xx = x + c - 2, yy = y + r - 2;
    const bool in = xx >= 0 && yy >= 0 && xx < stride && yy < rows;
    const uint16_t v = in ? plane[(size_t)yy * stride + xx] : (uint16_t)kVeryLarge;
    out |= !in;
    H[r * 2 * kPitch + c] = v;
    if (c) H[r * 2 * kPitch + kPitch + c - 1] = v;
  }
  out = __any_sync(0xffffffffu, out);
  __syncwarp();
  PairTaps t;
  t.C = P + (l / (BW / 2) + 2) * kPitch + l % (BW / 2) + 1;
  t.c2 = t.C[0];
  t.out = out;
  return t;
}

// The pair offsets of a direction's taps, by distance and side (a warp).
template <int PITCH>
__device__ __forceinline__ void stage_offsets(int16_t (&offs)[8][2][2], int t) {
  const int d = t >> 2, k = (t >> 1) & 1, sg = t & 1 ? -1 : 1;
  offs[d][k][t & 1] = (int16_t)pair_off<PITCH>(sg * cDirs[d][k][0], sg * cDirs[d][k][1]);
}

template <int BW, int BH>
__global__ void __launch_bounds__(128) cdef_tab_kernel(TabArgs ta, Geo g, const uint8_t* __restrict__ skip8,
                                                       const uint8_t* __restrict__ dirs,
                                                       const int32_t* __restrict__ vars, int pl0) {
  using Sh = TabShape<BW, BH>;
  constexpr int kPitch = Sh::kPitch, kLanes = Sh::kLanes;
  __shared__ __align__(16) uint32_t patch[4][Sh::kBlocks][Sh::kRows * kPitch];
  __shared__ __align__(16) float errs[4][Sh::kBlocks][kNCand * Sh::kErr];
  __shared__ int16_t offs[8][2][2];  // a direction's taps: distance, side
  const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
  if (t < 32) stage_offsets<kPitch>(offs, t);
  __syncthreads();
  const int sub = lane / kLanes, l = lane % kLanes;
  const int pl = pl0 + (int)blockIdx.z;
  const bool luma = pl == 0;
  const int nb = g.nbx * g.nby;
  const int bi = (blockIdx.x * 4 + wp) * Sh::kBlocks + sub, bc = min(bi, nb - 1);
  const int by = bc / g.nbx, bx = bc - by * g.nbx;
  const int x = bx * BW, y = by * BH;
  const int vis_w = luma ? g.disp_w : g.cw_vis, vis_h = luma ? g.disp_h : g.ch_vis;
  const int stride = luma ? g.w8 : g.cw8, rows = luma ? g.h8 : g.ch8;
  const bool live = bi < nb && !skip8[bc] && x < vis_w && y < vis_h;
  if (!__any_sync(0xffffffffu, live)) return;
  const int i0 = l / (BW / 2), j0 = 2 * (l % (BW / 2));  // this lane's samples (j0, i0) and (j0 + 1, i0)
  const PairTaps T = load_patch<BW, BH>(ta.rec[pl], stride, rows, x, y, l, patch[wp][sub]);
  const uint32_t c2 = T.c2;
  const int d0 = dirs[bc], var = vars[bc];
  const int dir = luma ? d0 : ((g.sub_x == 1 && g.sub_y == 0) ? (int)cUvDir422[d0] : d0);
  const int damp = max(luma ? g.damping : g.damping - 1, 1);
  // a strength's words: itself in both halves, its shift, the mask of what a
  // shifted half keeps
  uint32_t ps[3], pm[3], ss[2], sm[2];
  int psh[3], pw0[3], pw1[3], ssh[2];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const int e = luma ? adjust_pri(1 << q, var) : 1 << q;
    ps[q] = (uint32_t)e * kHalves;
    psh[q] = strength_shift(e, damp);
    pm[q] = (0xffffu >> psh[q]) * kHalves;
    pw0[q] = e & 1 ? 3 : 4;
    pw1[q] = e & 1 ? 3 : 2;
  }
#pragma unroll
  for (int q = 0; q < 2; q++) {
    ss[q] = (1u << q) * kHalves;
    ssh[q] = strength_shift(1 << q, damp);
    sm[q] = (0xffffu >> ssh[q]) * kHalves;
  }
  uint32_t mn = c2, mx = c2;
  uint32_t psum[3] = {0, 0, 0}, ssum[2] = {0, 0}, ssum0[2] = {0, 0};
#pragma unroll
  for (int k = 0; k < 2; k++) {
#pragma unroll
    for (int sg = 0; sg < 2; sg++) {
      uint32_t a, neg;
      const uint32_t v = T.at(offs[dir][k][sg], a, neg);
      mn = min2(mn, v);
      mx = max2(mx, v);
#pragma unroll
      for (int q = 0; q < 3; q++) add_constrained(psum[q], a, neg, ps[q], psh[q], pm[q], k == 0 ? pw0[q] : pw1[q]);
    }
#pragma unroll
    for (int dd = 2; dd <= 6; dd += 4)
#pragma unroll
      for (int sg = 0; sg < 2; sg++) {
        uint32_t a, neg;
        const uint32_t v = T.at(offs[(dir + dd) & 7][k][sg], a, neg);
        mn = min2(mn, v);
        mx = max2(mx, v);
#pragma unroll
        for (int q = 0; q < 2; q++) add_constrained(ssum[q], a, neg, ss[q], ssh[q], sm[q], 2 - k);
      }
  }
  if (__any_sync(0xffffffffu, dir != 0)) {  // the secondary taps of direction 0, where there is no primary strength
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
      for (int dd = 2; dd <= 6; dd += 4)
#pragma unroll
        for (int sg = 0; sg < 2; sg++) {
          uint32_t a, neg;
          T.at(offs[dd][k][sg], a, neg);
#pragma unroll
          for (int q = 0; q < 2; q++) add_constrained(ssum0[q], a, neg, ss[q], ssh[q], sm[q], 2 - k);
        }
  } else {
    ssum0[0] = ssum[0];
    ssum0[1] = ssum[1];
  }
  // the outputs, biased by 128, less the source: c + ((8 + sum - (sum < 0)) >> 4),
  // kept between the taps where both strengths are on
  const int vw = min(vis_w - x, BW), vh = min(vis_h - y, BH);
  const bool whole = vw == BW && vh == BH;
  const uint16_t* sp = ta.src[pl] + (size_t)(y + i0) * stride + x + j0;
  const float f0 = 8388736.0f + (float)(live ? sp[0] : 0), f1 = 8388736.0f + (float)(live ? sp[1] : 0);
  const uint32_t b128 = 128 * kHalves, b383 = 383 * kHalves;
  const uint32_t lo = min2(mn + b128, b383), hi = min2(mx + b128, b383);
  float* const E = errs[wp][sub] + l * 2;
#pragma unroll
  for (int si = 0; si < 3; si++)
#pragma unroll
    for (int pi = 0; pi < 4; pi++) {
      uint32_t sum = 0;
      if (si) sum = pi ? ssum[si - 1] : ssum0[si - 1];
      if (pi) sum += psum[pi - 1];
      uint32_t v = filtered(c2, sum);
      const bool clip = pi && si && ps[pi ? pi - 1 : 0] != 0;
      v = min2(max2(v, clip ? lo : b128), clip ? hi : b383);
      const float e0 = __fsub_rn(__uint_as_float(0x4b000000u | (v & 0xffffu)), f0);
      const float e1 = __fsub_rn(__uint_as_float(0x4b000000u | (v >> 16)), f1);
      *reinterpret_cast<float2*>(E + (si * 4 + pi) * Sh::kErr) = make_float2(e0, e1);
    }
  __syncwarp();
  const int u = (by >> 3) * g.uc + (bx >> 3);
  unsigned long long* const tab = ta.tab[pl] + (size_t)u * kNCand;
  if (__any_sync(0xffffffffu, live && !whole)) {  // blocks the visible window cuts: plain SSE of what is visible
    const bool v0 = i0 < vh && j0 < vw, v1 = i0 < vh && j0 + 1 < vw;
#pragma unroll 1
    for (int c = 0; c < kNCand; c++) {
      const float2 e = *reinterpret_cast<const float2*>(E + c * Sh::kErr);
      const int a = (int)e.x, b = (int)e.y;
      uint32_t r = (v0 ? (uint32_t)(a * a) : 0u) + (v1 ? (uint32_t)(b * b) : 0u);
#pragma unroll
      for (int o = kLanes / 2; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
      if (l == 0 && live && !whole) atomicAdd(&tab[c], (unsigned long long)r);
    }
  }
  if (!__any_sync(0xffffffffu, live && whole)) return;
  // the weighted SSE in the AVX2 kernel's float order
  const int k = lane & 3;
  if (BW == 8) {
    // Lanes (candidate, half row, row accumulator k): four of the eight lane
    // accumulators each, three rounds.
    float dk[4], wk[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      dk[m] = cD[k][m];
      wk[m] = cW[k][m];
    }
#pragma unroll 1
    for (int rd = 0; rd < 3; rd++) {
      const int task = rd * 8 + (lane >> 2), cand = task >> 1, hb = (task & 1) * 4;
      const float* e = errs[wp][0] + cand * Sh::kErr + hb;
      float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int r0 = 0; r0 < BH; r0 += 4) {
        float tt[4];
        const float4 a = *reinterpret_cast<const float4*>(e + r0 * 8);
        const float4 b = *reinterpret_cast<const float4*>(e + r0 * 8 + 8);
        const float4 c = *reinterpret_cast<const float4*>(e + r0 * 8 + 16);
        const float4 d = *reinterpret_cast<const float4*>(e + r0 * 8 + 24);
        tt[0] = __fmaf_rn(d.x, dk[3], __fmaf_rn(c.x, dk[2], __fmaf_rn(b.x, dk[1], __fmul_rn(a.x, dk[0]))));
        tt[1] = __fmaf_rn(d.y, dk[3], __fmaf_rn(c.y, dk[2], __fmaf_rn(b.y, dk[1], __fmul_rn(a.y, dk[0]))));
        tt[2] = __fmaf_rn(d.z, dk[3], __fmaf_rn(c.z, dk[2], __fmaf_rn(b.z, dk[1], __fmul_rn(a.z, dk[0]))));
        tt[3] = __fmaf_rn(d.w, dk[3], __fmaf_rn(c.w, dk[2], __fmaf_rn(b.w, dk[1], __fmul_rn(a.w, dk[0]))));
#pragma unroll
        for (int m = 0; m < 4; m++) {
          float cc = __fmul_rn(cD[m][0], tt[0]);
          cc = __fmaf_rn(cD[m][1], tt[1], cc);
          cc = __fmaf_rn(cD[m][2], tt[2], cc);
          cc = __fmaf_rn(cD[m][3], tt[3], cc);
          acc[m] = __fmaf_rn(__fmul_rn(wk[m], cc), cc, acc[m]);
        }
      }
      // the half rows, then the row accumulators (0 + 1) + (2 + 3)
#pragma unroll
      for (int m = 0; m < 4; m++) {
#pragma unroll
        for (int o = 4; o; o = o == 4 ? 1 : (o == 1 ? 2 : 0))
          acc[m] = __fadd_rn(acc[m], __shfl_xor_sync(0xffffffffu, acc[m], o));
      }
      const float res = __fadd_rn(__fadd_rn(acc[0], acc[2]), __fadd_rn(acc[1], acc[3]));
      if ((lane & 7) == 0) atomicAdd(&tab[cand], (unsigned long long)(long long)roundf(res));
    }
  } else {
    // Lanes (block, candidate, output lane k of the 4-wide path).
    float dl[4], wl[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      dl[m] = cD[k][m];
      wl[m] = cW[m][k];
    }
#pragma unroll 1
    for (int task = lane >> 2; task < Sh::kBlocks * kNCand; task += 8) {
      const int blk = task / kNCand, cand = task - blk * kNCand;
      const float* e = errs[wp][blk] + cand * Sh::kErr;
      float s = 0.0f;
#pragma unroll
      for (int r0 = 0; r0 < BH; r0 += 4) {
        const float4 a = *reinterpret_cast<const float4*>(e + r0 * 4);
        const float4 b = *reinterpret_cast<const float4*>(e + r0 * 4 + 4);
        const float4 c = *reinterpret_cast<const float4*>(e + r0 * 4 + 8);
        const float4 d = *reinterpret_cast<const float4*>(e + r0 * 4 + 12);
#pragma unroll
        for (int m = 0; m < 4; m++) {
          auto col = [&](float p, float q, float r, float w) {
            return __fmaf_rn(w, cD[m][3], __fmaf_rn(r, cD[m][2], __fmaf_rn(q, cD[m][1], __fmul_rn(p, cD[m][0]))));
          };
          float cc = __fmul_rn(dl[0], col(a.x, b.x, c.x, d.x));
          cc = __fmaf_rn(dl[1], col(a.y, b.y, c.y, d.y), cc);
          cc = __fmaf_rn(dl[2], col(a.z, b.z, c.z, d.z), cc);
          cc = __fmaf_rn(dl[3], col(a.w, b.w, c.w, d.w), cc);
          s = __fmaf_rn(__fmul_rn(wl[m], cc), cc, s);
        }
      }
      s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 2));
      s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 1));
      // the task's block is another lane's
      const int from = blk * kLanes;
      const bool ok = __shfl_sync(0xffffffffu, (int)(live && whole), from);
      const int tu = __shfl_sync(0xffffffffu, u, from);
      if (k == 0 && ok) atomicAdd(&ta.tab[pl][(size_t)tu * kNCand + cand], (unsigned long long)(long long)roundf(s));
    }
  }
}

// ---------------------------------------------------------------------------
// Apply: lanes as in the tables, over the blocks whose unit has a strength.
// ustr: per unit (luma pri, luma sec, chroma pri, chroma sec).  1920x1080 4:2:0
// 55 -> 30 us, 4096x4096 4:4:4 410 -> 230 us against a thread per sample with
// bounds-checked taps.
struct ApplyArgs {
  uint16_t* rec[3];
  const uint16_t* snap[3];
};

template <int BW, int BH>
__global__ void __launch_bounds__(128) cdef_apply_kernel(ApplyArgs aa, Geo g, const uint8_t* __restrict__ skip8,
                                                         const uint8_t* __restrict__ dirs,
                                                         const int32_t* __restrict__ vars,
                                                         const uint8_t* __restrict__ ustr, int pl0) {
  using Sh = TabShape<BW, BH>;
  __shared__ __align__(16) uint32_t patch[4][Sh::kBlocks][Sh::kRows * Sh::kPitch];
  __shared__ int16_t offs[8][2][2];
  const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
  if (t < 32) stage_offsets<Sh::kPitch>(offs, t);
  __syncthreads();
  const int sub = lane / Sh::kLanes, l = lane % Sh::kLanes;
  const int pl = pl0 + (int)blockIdx.z;
  const bool luma = pl == 0;
  const int nb = g.nbx * g.nby;
  const int bi = (blockIdx.x * 4 + wp) * Sh::kBlocks + sub, bc = min(bi, nb - 1);
  const int by = bc / g.nbx, bx = bc - by * g.nbx;
  const int u = (by >> 3) * g.uc + (bx >> 3);
  const int pri = ustr[u * 4 + (luma ? 0 : 2)], sec = ustr[u * 4 + (luma ? 1 : 3)];
  const bool live = bi < nb && !skip8[bc] && (pri != 0 || sec != 0);
  if (!__any_sync(0xffffffffu, live)) return;
  const int x = bx * BW, y = by * BH;
  const int stride = luma ? g.w8 : g.cw8, rows = luma ? g.h8 : g.ch8;
  const PairTaps T = load_patch<BW, BH>(aa.snap[pl], stride, rows, x, y, l, patch[wp][sub]);
  const int d0 = dirs[bc];
  const int bdir = luma ? d0 : ((g.sub_x == 1 && g.sub_y == 0) ? (int)cUvDir422[d0] : d0);
  const int dir = pri == 0 ? 0 : bdir;
  const int p_str = luma ? adjust_pri(pri, vars[bc]) : pri;
  const int damp = max(luma ? g.damping : g.damping - 1, 1);
  const int psh = strength_shift(p_str, damp), ssh = strength_shift(sec, damp);
  const uint32_t ps = (uint32_t)p_str * kHalves, ss = (uint32_t)sec * kHalves;
  const uint32_t pm = (0xffffu >> psh) * kHalves, sm = (0xffffu >> ssh) * kHalves;
  const int odd = p_str & 1;
  uint32_t sum = 0, mn = T.c2, mx = T.c2;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int w = k == 0 ? (odd ? 3 : 4) : (odd ? 3 : 2);
#pragma unroll
    for (int sg = 0; sg < 2; sg++) {
      uint32_t a, neg;
      const uint32_t v = T.at(offs[dir][k][sg], a, neg);
      add_constrained(sum, a, neg, ps, psh, pm, w);
      mn = min2(mn, v);
      mx = max2(mx, v);
    }
#pragma unroll
    for (int dd = 2; dd <= 6; dd += 4)
#pragma unroll
      for (int sg = 0; sg < 2; sg++) {
        uint32_t a, neg;
        const uint32_t v = T.at(offs[(dir + dd) & 7][k][sg], a, neg);
        add_constrained(sum, a, neg, ss, ssh, sm, 2 - k);
        mn = min2(mn, v);
        mx = max2(mx, v);
      }
  }
  const uint32_t b128 = 128 * kHalves, b383 = 383 * kHalves;
  const bool clip = p_str != 0 && sec != 0;  // between the taps
  const uint32_t lo = clip ? min2(mn + b128, b383) : b128, hi = clip ? min2(mx + b128, b383) : b383;
  const uint32_t v = min2(max2(filtered(T.c2, sum), lo), hi) - b128;
  if (!live) return;
  uint16_t* const d = aa.rec[pl] + (size_t)(y + l / (BW / 2)) * stride + x + 2 * (l % (BW / 2));
  d[0] = (uint16_t)v;
  d[1] = (uint16_t)(v >> 16);
}

// ---------------------------------------------------------------------------
// Host side.

int check_params(const mt_cdef_params* p) {
  if (!p) return MT_ERR_INVALID_INPUT;
  if (p->w8 <= 0 || p->h8 <= 0 || (p->w8 & 7) || (p->h8 & 7) || p->w8 > 16384 || p->h8 > 16384)
    return MT_ERR_INVALID_INPUT;
  if (p->disp_w <= p->w8 - 8 || p->disp_w > p->w8 || p->disp_h <= p->h8 - 8 || p->disp_h > p->h8)
    return MT_ERR_INVALID_INPUT;
  if (p->sub_x < 0 || p->sub_x > 1 || p->sub_y < 0 || p->sub_y > p->sub_x) return MT_ERR_INVALID_INPUT;
  if (p->base_q_idx < 1 || p->base_q_idx > 255) return MT_ERR_INVALID_INPUT;
  if (p->bd != 8) return MT_ERR_UNSUPPORTED;
  return MT_OK;
}

Geo make_geo(const mt_cdef_params* p) {
  Geo g;
  g.w8 = p->w8;
  g.h8 = p->h8;
  g.cw8 = p->w8 >> p->sub_x;
  g.ch8 = p->h8 >> p->sub_y;
  g.nbx = p->w8 / 8;
  g.nby = p->h8 / 8;
  g.uc = (p->w8 + 63) / 64;
  g.ur = (p->h8 + 63) / 64;
  g.disp_w = p->disp_w;
  g.disp_h = p->disp_h;
  g.cw_vis = (p->disp_w + (1 << p->sub_x) - 1) >> p->sub_x;
  g.ch_vis = (p->disp_h + (1 << p->sub_y) - 1) >> p->sub_y;
  g.sub_x = p->sub_x;
  g.sub_y = p->sub_y;
  g.bd = p->bd;
  g.damping = 3 + std::min(p->base_q_idx / 64, 3) + (p->bd - 8);
  return g;
}

constexpr int kMaxPairs = 144;  // 12 luma x 12 chroma candidates
constexpr long long kMargin = 40, kGate = 15000;
constexpr int kGreedySteps = 7;  // entries 2 .. 8
constexpr int kSearchThreads = 256;

struct SearchState {
  // the decision
  int32_t bits, n_strengths;
  uint8_t strengths[8][4];
  // unit statistics: signalling units, trusted units, distortion sums
  unsigned long long n_sig, n_trusted, total_off, unsig_off, gsum[3];
  // candidates: (pri, sec) and the table column of each
  int32_t nl, nc, np;
  uint8_t cand[12][2];
  int8_t col[12];
  // pass totals: [0] the single-entry pass, [1] and [2] alternate in the greedy passes
  unsigned long long tot[3][kMaxPairs];
  long long prefix[4];
  int32_t global_entry, nentries;
  int32_t entries[8];
  unsigned long long assign_total[4];  // the 2-, 4- and 8-entry sets at [1..3]
};

// Scratch layout of mt_cdef_frame_device (256-byte aligned pieces).
struct Layout {
  size_t dirs, vars, tabs, dv_sum, dv_cnt, ustr, snap_y, snap_u, snap_v, total;
  size_t state, d_off, thr, cm, sig, grids, grid;  // the strength search
  size_t tab_bytes;  // one plane's table
};

size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

Layout make_layout(const Geo& g, bool mono) {
  Layout L;
  const size_t nb = (size_t)g.nbx * g.nby, nu = (size_t)g.uc * g.ur;
  L.tab_bytes = nu * kNCand * 8;
  size_t o = 0;
  L.dirs = o;
  o += up256(nb);
  L.vars = o;
  o += up256(nb * 4);
  L.tabs = o;
  o += 3 * L.tab_bytes;
  L.dv_sum = o;
  o += nu * 8;
  L.dv_cnt = o;
  o += nu * 4;
  o = up256(o);
  L.ustr = o;
  o += up256(nu * 4);
  L.state = o;
  o += up256(sizeof(SearchState));
  L.d_off = o;
  o += up256(nu * 8);
  L.thr = o;
  o += up256(nu * 8);
  L.cm = o;
  o += up256(nu * 8);
  L.sig = o;
  o += up256(nu);
  L.grids = o;
  o += up256(3 * nu);
  L.grid = o;
  o += up256(nu);
  L.snap_y = o;
  o += up256((size_t)g.w8 * g.h8 * 2);
  L.snap_u = o;
  L.snap_v = o;
  if (!mono) {
    o += up256((size_t)g.cw8 * g.ch8 * 2);
    L.snap_v = o;
    o += up256((size_t)g.cw8 * g.ch8 * 2);
  }
  L.total = o;
  return L;
}

}  // namespace

namespace mth {
// Kernels the calling thread's last mt_cdef_frame_device launched (the
// direction and table kernels, the strength search's kernels and the apply
// kernel).
thread_local int cdef_last_launches = 0;
// Bytes mt_cdef_frame_device reads back to the host: the search's state
// (decision and statistics) and, when asked for, the per-unit grid.
void cdef_frame_transfer_bytes(const mt_cdef_params* p, size_t* d2h, size_t* h2d) {
  const Geo g = make_geo(p);
  *d2h = sizeof(SearchState) + (size_t)g.uc * g.ur;
  *h2d = 0;
}
}  // namespace mth

namespace {

int launch_tables(const uint16_t* y, const uint16_t* u, const uint16_t* v, const uint16_t* sy, const uint16_t* su,
                  const uint16_t* sv, const uint8_t* skip8, const Geo& g, bool mono, uint8_t* dirs, int32_t* vars,
                  int64_t* ltab, int64_t* utab, int64_t* vtab, unsigned long long* dv_sum, int* dv_cnt,
                  cudaStream_t st) {
  const size_t nu = (size_t)g.uc * g.ur;
  if (cudaMemsetAsync(ltab, 0, nu * kNCand * 8, st) != cudaSuccess) return MT_ERR_DEVICE;
  if (!mono) {
    if (cudaMemsetAsync(utab, 0, nu * kNCand * 8, st) != cudaSuccess) return MT_ERR_DEVICE;
    if (cudaMemsetAsync(vtab, 0, nu * kNCand * 8, st) != cudaSuccess) return MT_ERR_DEVICE;
  }
  if (dv_sum) {
    if (cudaMemsetAsync(dv_sum, 0, nu * 8, st) != cudaSuccess) return MT_ERR_DEVICE;
    if (cudaMemsetAsync(dv_cnt, 0, nu * 4, st) != cudaSuccess) return MT_ERR_DEVICE;
  }
  const int nb = g.nbx * g.nby;
  cdef_dir_kernel<<<(nb + 127) / 128, 128, 0, st>>>(y, g, skip8, dirs, vars, dv_sum, dv_cnt);
  TabArgs ta;
  ta.rec[0] = y;
  ta.rec[1] = u;
  ta.rec[2] = v;
  ta.src[0] = sy;
  ta.src[1] = su;
  ta.src[2] = sv;
  ta.tab[0] = reinterpret_cast<unsigned long long*>(ltab);
  ta.tab[1] = reinterpret_cast<unsigned long long*>(utab);
  ta.tab[2] = reinterpret_cast<unsigned long long*>(vtab);
  auto grid = [&](int per_warp, int planes) {
    return dim3((unsigned)((nb + 4 * per_warp - 1) / (4 * per_warp)), 1, (unsigned)planes);
  };
  cdef_tab_kernel<8, 8><<<grid(1, !mono && !g.sub_x ? 3 : 1), 128, 0, st>>>(ta, g, skip8, dirs, vars, 0);
  if (!mono && g.sub_x) {
    if (g.sub_y) cdef_tab_kernel<4, 4><<<grid(4, 2), 128, 0, st>>>(ta, g, skip8, dirs, vars, 1);
    else cdef_tab_kernel<4, 8><<<grid(2, 2), 128, 0, st>>>(ta, g, skip8, dirs, vars, 1);
  }
  return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

// frame lambda_d (src/coder.rs:259-271): mode_lambda_q(dc_q) *
// mode_lambda_weight(qidx, sub) / K_PART_LAMBDA with the shipped tuning.
float frame_lambda_d(int qidx, int bd, int sub_x, int sub_y, float dc_q) {
  const int sub = (sub_x == 1 && sub_y == 1) ? 2 : (sub_x == 1 ? 1 : 0);
  const float dc8 = dc_q / (float)(1u << (std::max(bd, 8) - 8));
  volatile float kf = 0.0015f * dc8;
  kf = 3.3f + kf;
  volatile float mlq = 0.009005174719460433f * 1.0f;
  mlq = mlq * dc_q;
  mlq = mlq * dc_q;
  mlq = mlq * kf;
  const float scale = sub == 2 ? 0.8f : (sub == 1 ? 0.65f : 0.6f);
  int wi = ((255 - qidx) * 3) / 4;
  wi = std::min(std::max(wi, 0), 72) + 128;
  const float w = (float)wi * (1.0f / 128.0f);
  float weight;
  if (sub == 1) {
    weight = w * scale;
  } else {
    volatile float r = ((float)qidx - 0.0f) / (72.0f - 0.0f);
    float rr = std::min(std::max((float)r, 0.0f), 1.0f);
    volatile float m = (w - 3.0f) * rr;
    weight = (3.0f + m) * scale;
  }
  volatile float num = mlq * weight;
  return num / 2.775f;
}

// ---------------------------------------------------------------------------
// The staged strength search (src/coder/frame_cdef.rs:116-520) on the device,
// as one cluster or a chain of small kernels on the stream (no host round trip): the unit
// statistics, the candidate list, the single-entry pass, seven greedy entry
// passes, the assignment of the 2-, 4- and 8-entry sets to the units, the rate
// decision and the per-unit strengths the apply kernel reads.  Integer sums
// are 64-bit atomics (order-free, exact); every choice is the first minimum in
// the reference's order, and the rate arithmetic is the reference's f32
// operations one by one.

struct SearchArgs {
  const long long* ltab;
  const long long* utab;
  const long long* vtab;
  const unsigned long long* dv_sum;
  const int* dv_cnt;
  int nu, mono, slow;
  float lambda;      // the frame lambda_d pricing the CDEF bits
  SearchState* S;
  long long* d_off;  // distortion with CDEF off, per unit
  long long* thr;    // its margin threshold
  long long* cm;     // the greedy set's best distortion so far
  uint8_t* sig;      // the unit signals a strength index (a non-skip block)
  uint8_t* grids;    // 3 x nu: the entry of each unit for the 2-, 4- and 8-entry sets
  uint8_t* grid;     // nu: the chosen set's entry per unit (0 unless bits > 0)
  uint8_t* ustr;     // nu x 4: the unit's strengths for the apply kernel
};

__host__ __device__ __forceinline__ long long sat_mul_pos(long long a, long long b) {  // b > 0
  if (a > LLONG_MAX / b) return LLONG_MAX;
  if (a < LLONG_MIN / b) return LLONG_MIN;
  return a * b;
}
__host__ __device__ __forceinline__ long long off_of(long long off) { return off - sat_mul_pos(off, kMargin) / 1000; }
__host__ __device__ __forceinline__ int cand_col(int pri, int sec) {  // sec_idx * 4 + pri_idx
  return sec * 4 + (pri == 4 ? 3 : pri);
}

__device__ __forceinline__ long long d_pair(const SearchArgs& a, const SearchState& S, int pp, int u) {
  long long d = a.ltab[(size_t)u * kNCand + S.col[pp / S.nc]];
  if (!a.mono) {
    const int c = S.col[pp % S.nc];
    d += a.utab[(size_t)u * kNCand + c] + a.vtab[(size_t)u * kNCand + c];
  }
  return d;
}

// The four strengths of pair pp (luma pri, sec, chroma pri, sec).
__device__ __forceinline__ void pair_strengths(const SearchState& S, int mono, int pp, int s[4]) {
  s[0] = S.cand[pp / S.nc][0];
  s[1] = S.cand[pp / S.nc][1];
  s[2] = mono ? 0 : S.cand[pp % S.nc][0];
  s[3] = mono ? 0 : S.cand[pp % S.nc][1];
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Sums of v[0..N) over the CTA into dst[0..N) with one atomic each
// (kSearchThreads threads).
template <int N>
__device__ __forceinline__ void block_add(unsigned long long (&v)[N], unsigned long long* const (&dst)[N]) {
  __shared__ unsigned long long part[N][kSearchThreads / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < N; k++) {
    const unsigned long long s = warp_sum(v[k]);
    if (l == 0) part[k][w] = s;
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < N; k++) {
      unsigned long long s = l < kSearchThreads / 32 ? part[k][l] : 0ull;
      s = warp_sum(s);
      if (l == 0 && s) atomicAdd(dst[k], s);
    }
  }
}

// Per unit: the signalling and trust flags (directional-variance gate), the
// CDEF-off distortion and its threshold, and the luma gains of pri 1 / 2 / 4
// that rank the Slow candidate list.
__global__ void __launch_bounds__(kSearchThreads) cdef_unit_stats_kernel(SearchArgs a) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  SearchState& S = *a.S;
  unsigned long long v[7] = {0, 0, 0, 0, 0, 0, 0};  // n_sig, n_trusted, total_off, unsig_off, gsum[3]
  if (u < a.nu) {
    const bool sg = a.dv_cnt[u] > 0;
    const long long cnt = a.dv_cnt[u] > 1 ? a.dv_cnt[u] : 1;
    const long long* lt = a.ltab + (size_t)u * kNCand;
    const long long lo = lt[0];
    const long long off = lo + (a.mono ? 0 : a.utab[(size_t)u * kNCand] + a.vtab[(size_t)u * kNCand]);
    a.d_off[u] = off;
    a.thr[u] = off_of(off);
    a.cm[u] = off;
    a.sig[u] = sg;
    v[0] = sg;
    v[1] = (long long)a.dv_sum[u] / cnt >= kGate;
    v[2] = (unsigned long long)off;
    v[3] = sg ? 0ull : (unsigned long long)off;
    const long long lim = off_of(lo);
#pragma unroll
    for (int i = 0; i < 3; i++) {  // pri 1, 2, 4 at sec 0: columns 1..3
      const long long on = lt[1 + i];
      v[4 + i] = on < lim ? (unsigned long long)(lo - on) : 0ull;
    }
  }
  unsigned long long* const dst[7] = {&S.n_sig, &S.n_trusted, &S.total_off, &S.unsig_off,
                                      &S.gsum[0], &S.gsum[1], &S.gsum[2]};
  block_add<7>(v, dst);
}

// The candidate list (one thread): Slow ranks pri 1 / 2 / 4 by their gains
// and pairs the useful ones with sec 1 and 2; otherwise all 12.
__device__ __forceinline__ void search_plan(const SearchArgs& a, SearchState& S) {
  int n = 0;
  auto push = [&](int pri, int sec) {
    S.cand[n][0] = (uint8_t)pri;
    S.cand[n][1] = (uint8_t)sec;
    S.col[n] = (int8_t)cand_col(pri, sec);
    ++n;
  };
  push(0, 0);
  if (a.slow) {
    const int pri_list[3] = {1, 2, 4};
    int r[3] = {0, 1, 2};  // stable: larger gain first, then list order
    for (int i = 1; i < 3; i++)
      for (int j = i; j > 0 && S.gsum[r[j]] > S.gsum[r[j - 1]]; j--) {
        const int t = r[j];
        r[j] = r[j - 1];
        r[j - 1] = t;
      }
    for (int i = 0; i < 3; i++) push(pri_list[i], 0);
    for (int sec = 1; sec <= 2; sec++) {
      push(0, sec);
      for (int k = 0; k < 3; k++)
        if (S.gsum[r[k]] > 0) push(pri_list[r[k]], sec);
    }
  } else {
    const int pl[4] = {0, 1, 2, 4};
    for (int i = 0; i < 4; i++)
      for (int sec = 0; sec <= 2; sec++)
        if (pl[i] || sec) push(pl[i], sec);
  }
  S.nl = n;
  S.nc = a.mono ? 1 : n;
  S.np = n * S.nc;
  for (int k = 0; k < 4; k++) S.prefix[k] = LLONG_MAX;
  S.entries[0] = 0;
  S.nentries = 1;
}
__global__ void cdef_plan_kernel(SearchArgs a) { search_plan(a, *a.S); }

// Per (pair, chunk of units): the pair's total over the signalling units.
// Pass 0 (the single-entry pass): its distortion.  Greedy passes: the set
// extended by the pair, each unit at the better of the set and the pair, or
// at CDEF off when that is within the margin.
__global__ void __launch_bounds__(kSearchThreads) cdef_pair_sum_kernel(SearchArgs a, int buf) {
  const SearchState& S = *a.S;
  const int pp = blockIdx.y;
  if (S.n_sig == 0 || pp >= S.np) return;
  unsigned long long v[1] = {0};
  for (int u = blockIdx.x * kSearchThreads + threadIdx.x; u < a.nu; u += gridDim.x * kSearchThreads) {
    if (!a.sig[u]) continue;
    const long long r = d_pair(a, S, pp, u);
    if (buf == 0) {
      v[0] += (unsigned long long)r;
    } else {
      const long long b = a.cm[u] < r ? a.cm[u] : r;
      v[0] += (unsigned long long)(b >= a.thr[u] ? a.d_off[u] : b);
    }
  }
  unsigned long long* const dst[1] = {&a.S->tot[buf][pp]};
  block_add<1>(v, dst);
}

// First minimum over the pairs of unsig_off + tot[buf][pair], by a whole warp
// (by one thread it was most of a greedy step's 9.4 us).
__device__ __forceinline__ int first_min(const SearchState& S, int buf, long long* best) {
  int bp = 0;
  long long bt = LLONG_MAX;
  for (int pp = threadIdx.x & 31; pp < S.np; pp += 32) {
    const long long t = (long long)(S.unsig_off + S.tot[buf][pp]);
    if (t < bt) {
      bt = t;
      bp = pp;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const long long t = __shfl_xor_sync(0xffffffffu, bt, o);
    const int p = __shfl_xor_sync(0xffffffffu, bp, o);
    if (t < bt || (t == bt && p < bp)) {
      bt = t;
      bp = p;
    }
  }
  *best = bt;
  return bp;
}

// The single-entry pass's best pair (one warp).
__global__ void cdef_global_entry_kernel(SearchArgs a) {
  SearchState& S = *a.S;
  if (S.n_sig == 0) return;
  long long bt;
  const int bp = first_min(S, 0, &bt);
  if (threadIdx.x == 0) {
    S.global_entry = bp;
    S.prefix[0] = bt;
  }
}

// One greedy step: every CTA finds the pass's best pair (the same one) and
// lowers its units' set distortion to it; CTA 0 records the entry and clears
// the other pass buffer for the next step.
__global__ void __launch_bounds__(kSearchThreads) cdef_greedy_step_kernel(SearchArgs a, int buf) {
  SearchState& S = *a.S;
  if (S.n_sig == 0) return;
  __shared__ int s_best;
  __shared__ long long s_tot;
  if (threadIdx.x < 32) {
    long long bt;
    const int bp = first_min(S, buf, &bt);
    if (threadIdx.x == 0) {
      s_best = bp;
      s_tot = bt;
    }
  }
  __syncthreads();
  const int bp = s_best;
  if (blockIdx.x == 0) {
    const int other = buf == 1 ? 2 : 1;
    for (int pp = threadIdx.x; pp < kMaxPairs; pp += blockDim.x) S.tot[other][pp] = 0;
    if (threadIdx.x == 0) {
      const int n = S.nentries + 1;
      S.entries[n - 1] = bp;
      S.nentries = n;
      if ((n & (n - 1)) == 0) S.prefix[__ffs(n) - 1] = s_tot;
    }
  }
  for (int u = blockIdx.x * kSearchThreads + threadIdx.x; u < a.nu; u += gridDim.x * kSearchThreads) {
    if (!a.sig[u]) continue;
    const long long r = d_pair(a, S, bp, u);
    if (r < a.cm[u]) a.cm[u] = r;
  }
}

// The 2-, 4- and 8-entry sets' entries of unit u and their distortions (dist:
// the unit's distortion of a pair): a unit takes the smallest-magnitude entry
// within its margin (ties by distortion, then list order), else the zero entry
// at CDEF off, else its best entry.
template <typename F>
__device__ __forceinline__ void assign_unit(const SearchArgs& a, const SearchState& S, int u, bool sig, long long off,
                                            long long thr, unsigned long long (&v)[3], F&& dist) {
  for (int b = 1; b <= 3; b++) {
    const int nset = 1 << b;
    uint8_t g = 0;
    if (!sig) {
      v[b - 1] += (unsigned long long)off;
    } else {
      int z = -1;
      for (int e = 0; e < nset; e++)
        if (S.entries[e] == 0) {
          z = e;
          break;
        }
      bool have = false;
      int pm = 0, pe = 0, rb_e = 0;
      long long pd = 0, rb_d = LLONG_MAX;
      for (int e = 0; e < nset; e++) {
        const long long d = dist(S.entries[e]);
        if (d < rb_d) {
          rb_d = d;
          rb_e = e;
        }
        if (d < thr) {
          int s[4];
          pair_strengths(S, a.mono, S.entries[e], s);
          const int mag = s[0] + s[1] + s[2] + s[3];
          if (!have || mag < pm || (mag == pm && d < pd)) {
            have = true;
            pm = mag;
            pd = d;
            pe = e;
          }
        }
      }
      long long t;
      if (have) {
        t = pd;
        g = (uint8_t)pe;
      } else if (z >= 0) {
        t = off;
        g = (uint8_t)z;
      } else {
        t = rb_d;
        g = (uint8_t)rb_e;
      }
      v[b - 1] += (unsigned long long)t;
    }
    a.grids[(size_t)(b - 1) * a.nu + u] = g;
  }
}

__global__ void __launch_bounds__(kSearchThreads) cdef_assign_kernel(SearchArgs a) {
  const SearchState& S = *a.S;
  if (S.n_sig == 0) return;
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long v[3] = {0, 0, 0};
  if (u < a.nu) assign_unit(a, S, u, a.sig[u], a.d_off[u], a.thr[u], v, [&](int pp) { return d_pair(a, S, pp, u); });
  unsigned long long* const dst[3] = {&a.S->assign_total[1], &a.S->assign_total[2], &a.S->assign_total[3]};
  block_add<3>(v, dst);
}

// The rate decision (one thread): CDEF off, the single entry, or 2 / 4 / 8
// entries, each priced as distortion + lambda_d x (entry bits + index bits).
__device__ __forceinline__ void search_decide(const SearchArgs& a, SearchState& S) {
  S.bits = -1;
  S.n_strengths = 0;
  for (int e = 0; e < 8; e++)
    for (int k = 0; k < 4; k++) S.strengths[e][k] = 0;
  if (S.n_sig == 0) return;
  const long long total_off = (long long)S.total_off;
  const float per_entry_bits = a.mono ? 6.0f : 12.0f;
  const int n_sig = (int)S.n_sig, n_trusted = (int)S.n_trusted;
  int best_bits = -1;
  float best_cost = __ll2float_rn(total_off);
  for (int b = 0; b <= 3; b++) {
    const int nb = 1 << b;
    const long long total = b == 0 ? S.prefix[0] : (long long)S.assign_total[b];
    if (total == LLONG_MAX) continue;
    if (b == 0 && (S.global_entry == 0 || n_trusted * 4 < n_sig * 3 || total >= off_of(total_off))) continue;
    const float e_bits = __fmul_rn(per_entry_bits, __int2float_rn(nb - 1));
    const float u_bits = __fmul_rn(__int2float_rn(b), __int2float_rn(n_sig));
    const float bits_f = __fadd_rn(e_bits, u_bits);
    const float lb = __fmul_rn(a.lambda, bits_f);
    const float cost = __fadd_rn(__ll2float_rn(total), lb);
    if (cost < best_cost) {
      best_cost = cost;
      best_bits = b;
    }
  }
  if (best_bits < 0) return;
  const int n = 1 << best_bits;
  S.bits = best_bits;
  S.n_strengths = n;
  for (int e = 0; e < n; e++) {
    int s[4];
    pair_strengths(S, a.mono, best_bits == 0 ? S.global_entry : S.entries[e], s);
    for (int k = 0; k < 4; k++) S.strengths[e][k] = (uint8_t)s[k];
  }
}

__global__ void cdef_decide_kernel(SearchArgs a) { search_decide(a, *a.S); }

// Each unit's entry and strengths under the decision (all zero when CDEF is
// off: the apply kernel then leaves the planes as they are).
__device__ __forceinline__ void unit_strengths(const SearchArgs& a, const SearchState& S, int u) {
  const int g = S.bits > 0 ? a.grids[(size_t)(S.bits - 1) * a.nu + u] : 0;
  a.grid[u] = (uint8_t)g;
#pragma unroll
  for (int k = 0; k < 4; k++) a.ustr[(size_t)u * 4 + k] = S.bits >= 0 ? S.strengths[g][k] : 0;
}
__global__ void __launch_bounds__(kSearchThreads) cdef_unit_strengths_kernel(SearchArgs a) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u < a.nu) unit_strengths(a, *a.S, u);
}

// The whole search in one launch of one cluster, for frames whose tables fit
// in a CTA's shared memory: every CTA holds all units' distortions (by
// candidate, the chroma planes' sums taken once), its own copy of the greedy
// set's best and of the search state, and sums every eighth pair, a warp per
// pair; the totals go to every CTA's memory and one cluster barrier ends a
// pass.  CTA 0 assigns and decides.  The chain of launches is bound by its
// launches (1080p, 510 units, 21 launches: 172 us; 150x101: 118 us).
constexpr int kSearchCtas = 8, kClusterThreads = 512;
constexpr size_t search_smem(int nu) { return (size_t)nu * (2 * kNCand + 3) * 8 + (size_t)nu; }
constexpr size_t kSearchSmemMax = 200 * 1024;

__global__ void __cluster_dims__(kSearchCtas, 1, 1) __launch_bounds__(kClusterThreads)
    cdef_search_cluster_kernel(SearchArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char search_dyn[];
  __shared__ SearchState S;
  __shared__ unsigned long long sums[7];
  __shared__ int s_best;
  const int nu = a.nu, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int rank = (int)cluster.block_rank();
  long long* const lt = reinterpret_cast<long long*>(search_dyn);  // [candidate][unit]
  long long* const uv = lt + (size_t)kNCand * nu;
  long long* const off = uv + (size_t)kNCand * nu;
  long long* const thr = off + nu;
  long long* const cm = thr + nu;
  uint8_t* const sig = reinterpret_cast<uint8_t*>(cm + nu);
  for (int i = t; i < nu * kNCand; i += kClusterThreads) {
    const int u = i / kNCand, k = i - u * kNCand;
    lt[(size_t)k * nu + u] = a.ltab[i];
    uv[(size_t)k * nu + u] = a.mono ? 0 : a.utab[i] + a.vtab[i];
  }
  if (t < 7) sums[t] = 0;
  __syncthreads();
  {
    unsigned long long v[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int u = t; u < nu; u += kClusterThreads) {
      const bool sg = a.dv_cnt[u] > 0;
      const long long cnt = a.dv_cnt[u] > 1 ? a.dv_cnt[u] : 1;
      const long long lo = lt[u], o = lo + uv[u], lim = off_of(lo);
      off[u] = cm[u] = o;
      thr[u] = off_of(o);
      sig[u] = sg;
      v[0] += sg;
      v[1] += (long long)a.dv_sum[u] / cnt >= kGate;
      v[2] += (unsigned long long)o;
      v[3] += sg ? 0ull : (unsigned long long)o;
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const long long on = lt[(size_t)(1 + i) * nu + u];
        v[4 + i] += on < lim ? (unsigned long long)(lo - on) : 0ull;
      }
    }
#pragma unroll
    for (int k = 0; k < 7; k++) {
      const unsigned long long s = warp_sum(v[k]);
      if (lane == 0 && s) atomicAdd(&sums[k], s);
    }
  }
  __syncthreads();
  if (t == 0) {
    S.n_sig = sums[0];
    S.n_trusted = sums[1];
    S.total_off = sums[2];
    S.unsig_off = sums[3];
    for (int k = 0; k < 3; k++) S.gsum[k] = sums[4 + k];
    search_plan(a, S);
  }
  // every CTA has started, and its state is set
  cluster.sync();
  const bool any = S.n_sig != 0;  // the same in every CTA
  for (int pass = 0; any && pass <= kGreedySteps; pass++) {
    const int buf = pass & 1;
    for (int pp = rank + kSearchCtas * w; pp < S.np; pp += kSearchCtas * (kClusterThreads / 32)) {
      const long long* l = lt + (size_t)S.col[pp / S.nc] * nu;
      const long long* c = uv + (size_t)S.col[pp % S.nc] * nu;
      unsigned long long v = 0;
      for (int u = lane; u < nu; u += 32) {
        if (!sig[u]) continue;
        const long long r = l[u] + (a.mono ? 0 : c[u]);
        if (pass == 0) {
          v += (unsigned long long)r;
        } else {
          const long long b = cm[u] < r ? cm[u] : r;
          v += (unsigned long long)(b >= thr[u] ? off[u] : b);
        }
      }
      v = __shfl_sync(0xffffffffu, warp_sum(v), 0);
      if (lane < kSearchCtas) *cluster.map_shared_rank(&S.tot[buf][pp], lane) = v;
    }
    cluster.sync();
    if (w == 0) {
      long long bt;
      const int bp = first_min(S, buf, &bt);
      if (lane == 0) {
        s_best = bp;
        if (pass == 0) {
          S.global_entry = bp;
          S.prefix[0] = bt;
        } else {
          const int n = S.nentries + 1;
          S.entries[n - 1] = bp;
          S.nentries = n;
          if ((n & (n - 1)) == 0) S.prefix[__ffs(n) - 1] = bt;
        }
      }
    }
    __syncthreads();
    if (pass) {
      const long long* l = lt + (size_t)S.col[s_best / S.nc] * nu;
      const long long* c = uv + (size_t)S.col[s_best % S.nc] * nu;
      for (int u = t; u < nu; u += kClusterThreads) {
        const long long r = l[u] + (a.mono ? 0 : c[u]);
        if (sig[u] && r < cm[u]) cm[u] = r;
      }
    }
    __syncthreads();
  }
  if (rank) return;  // nobody writes to this CTA's memory any more
  if (t < 3) sums[t] = 0;
  __syncthreads();
  if (any) {
    unsigned long long v[3] = {0, 0, 0};
    for (int u = t; u < nu; u += kClusterThreads)
      assign_unit(a, S, u, sig[u], off[u], thr[u], v, [&](int pp) {
        return lt[(size_t)S.col[pp / S.nc] * nu + u] + (a.mono ? 0 : uv[(size_t)S.col[pp % S.nc] * nu + u]);
      });
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const unsigned long long s = warp_sum(v[k]);
      if (lane == 0 && s) atomicAdd(&sums[k], s);
    }
  }
  __syncthreads();
  if (t == 0) {
    for (int k = 0; k < 3; k++) S.assign_total[1 + k] = sums[k];
    search_decide(a, S);
    SearchState& out = *a.S;
    out.bits = S.bits;
    out.n_strengths = S.n_strengths;
    for (int e = 0; e < 8; e++)
      for (int k = 0; k < 4; k++) out.strengths[e][k] = S.strengths[e][k];
  }
  __syncthreads();
  for (int u = t; u < nu; u += kClusterThreads) unit_strengths(a, S, u);
}

// The search's launches on the stream, after the tables: one cluster where the
// units' tables fit in shared memory (up to 943 units), else the chain, which
// spreads the units over the SMs.
constexpr int kSearchLaunches = 7 + 2 * kGreedySteps;

int launch_search(const SearchArgs& a, cudaStream_t st, int* launches) {
  if (search_smem(a.nu) <= kSearchSmemMax) {
    if (cudaFuncSetAttribute(cdef_search_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kSearchSmemMax) != cudaSuccess)
      return MT_ERR_DEVICE;
    cdef_search_cluster_kernel<<<kSearchCtas, kClusterThreads, search_smem(a.nu), st>>>(a);
    *launches = 1;
    return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
  }
  *launches = kSearchLaunches;
  if (cudaMemsetAsync(a.S, 0, sizeof(SearchState), st) != cudaSuccess) return MT_ERR_DEVICE;
  const int ublocks = (a.nu + kSearchThreads - 1) / kSearchThreads;
  const int chunks = std::min(ublocks, 16);  // unit chunks per pair in the pass sums
  cdef_unit_stats_kernel<<<ublocks, kSearchThreads, 0, st>>>(a);
  cdef_plan_kernel<<<1, 1, 0, st>>>(a);
  cdef_pair_sum_kernel<<<dim3(chunks, kMaxPairs), kSearchThreads, 0, st>>>(a, 0);
  cdef_global_entry_kernel<<<1, 32, 0, st>>>(a);
  for (int k = 0; k < kGreedySteps; k++) {
    const int buf = 1 + (k & 1);
    cdef_pair_sum_kernel<<<dim3(chunks, kMaxPairs), kSearchThreads, 0, st>>>(a, buf);
    cdef_greedy_step_kernel<<<std::min(ublocks, 64), kSearchThreads, 0, st>>>(a, buf);
  }
  cdef_assign_kernel<<<ublocks, kSearchThreads, 0, st>>>(a);
  cdef_decide_kernel<<<1, 1, 0, st>>>(a);
  cdef_unit_strengths_kernel<<<ublocks, kSearchThreads, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

}  // namespace

extern "C" {

int mt_quant_init(uint8_t base_q_idx, uint8_t bd, uint8_t qm_level, mt_quant* out);

int mt_cdef_tables_device(const uint16_t* d_y, const uint16_t* d_u, const uint16_t* d_v, const uint16_t* d_src_y,
                          const uint16_t* d_src_u, const uint16_t* d_src_v, const uint8_t* d_skip8,
                          const mt_cdef_params* prm, uint8_t* d_dirs, int32_t* d_vars, int64_t* d_luma_tab,
                          int64_t* d_u_tab, int64_t* d_v_tab, void* stream) {
  int rc = check_params(prm);
  if (rc != MT_OK) return rc;
  const bool mono = prm->mono != 0;
  if (!d_y || !d_src_y || !d_skip8 || !d_dirs || !d_vars || !d_luma_tab) return MT_ERR_INVALID_INPUT;
  if (!mono && (!d_u || !d_v || !d_src_u || !d_src_v || !d_u_tab || !d_v_tab)) return MT_ERR_INVALID_INPUT;
  const Geo g = make_geo(prm);
  return launch_tables(d_y, d_u, d_v, d_src_y, d_src_u, d_src_v, d_skip8, g, mono, d_dirs, d_vars, d_luma_tab,
                       d_u_tab, d_v_tab, nullptr, nullptr, reinterpret_cast<cudaStream_t>(stream));
}

size_t mt_cdef_scratch_bytes(const mt_cdef_params* prm) {
  if (check_params(prm) != MT_OK) return 0;
  return make_layout(make_geo(prm), prm->mono != 0).total;
}

}  // extern "C"

namespace mth {

// mt_cdef_frame_device up to the filtered planes, on the stream and without a
// wait: `decided` (when given) is recorded once the strength search's decision
// is on the device (*d_bits, and *d_grid per 64x64 unit), ahead of the filter.
int cdef_frame_enqueue(uint16_t* d_y, uint16_t* d_u, uint16_t* d_v, const uint16_t* d_src_y, const uint16_t* d_src_u,
                       const uint16_t* d_src_v, const uint8_t* d_skip8, const mt_cdef_params* prm, void* d_scratch,
                       cudaEvent_t decided, const int32_t** d_bits, const uint8_t** d_grid, cudaStream_t st) {
  int rc = check_params(prm);
  if (rc != MT_OK) return rc;
  const bool mono = prm->mono != 0;
  if (!d_y || !d_src_y || !d_skip8 || !d_scratch) return MT_ERR_INVALID_INPUT;
  if (!mono && (!d_u || !d_v || !d_src_u || !d_src_v)) return MT_ERR_INVALID_INPUT;
  const Geo g = make_geo(prm);
  const Layout L = make_layout(g, mono);
  uint8_t* s = static_cast<uint8_t*>(d_scratch);
  const size_t nu = (size_t)g.uc * g.ur;
  uint8_t* dirs = s + L.dirs;
  int32_t* vars = reinterpret_cast<int32_t*>(s + L.vars);
  int64_t* tabs = reinterpret_cast<int64_t*>(s + L.tabs);
  unsigned long long* dv_sum = reinterpret_cast<unsigned long long*>(s + L.dv_sum);
  int* dv_cnt = reinterpret_cast<int*>(s + L.dv_cnt);
  mth::cdef_last_launches = 0;
  rc = launch_tables(d_y, d_u, d_v, d_src_y, d_src_u, d_src_v, d_skip8, g, mono, dirs, vars, tabs, tabs + nu * kNCand,
                     tabs + 2 * nu * kNCand, dv_sum, dv_cnt, st);
  if (rc != MT_OK) return rc;
  mth::cdef_last_launches = !mono && prm->sub_x ? 3 : 2;
  // the strength search on the stream
  mt_quant q;
  if (mt_quant_init((uint8_t)prm->base_q_idx, (uint8_t)prm->bd, 15, &q) != MT_OK) return MT_ERR_INVALID_INPUT;
  SearchArgs sa;
  sa.ltab = reinterpret_cast<const long long*>(tabs);
  sa.utab = reinterpret_cast<const long long*>(tabs + nu * kNCand);
  sa.vtab = reinterpret_cast<const long long*>(tabs + 2 * nu * kNCand);
  sa.dv_sum = dv_sum;
  sa.dv_cnt = dv_cnt;
  sa.nu = (int)nu;
  sa.mono = mono;
  sa.slow = prm->slow != 0;
  sa.lambda = frame_lambda_d(prm->base_q_idx, prm->bd, prm->sub_x, prm->sub_y, (float)q.dc_q);
  sa.S = reinterpret_cast<SearchState*>(s + L.state);
  sa.d_off = reinterpret_cast<long long*>(s + L.d_off);
  sa.thr = reinterpret_cast<long long*>(s + L.thr);
  sa.cm = reinterpret_cast<long long*>(s + L.cm);
  sa.sig = s + L.sig;
  sa.grids = s + L.grids;
  sa.grid = s + L.grid;
  sa.ustr = s + L.ustr;
  int search_launches = 0;
  if ((rc = launch_search(sa, st, &search_launches)) != MT_OK) return rc;
  mth::cdef_last_launches += search_launches;
  if (d_bits) *d_bits = &sa.S->bits;
  if (d_grid) *d_grid = sa.grid;
  if (decided && cudaEventRecord(decided, st) != cudaSuccess) return MT_ERR_DEVICE;
  // the filter from a pre-CDEF snapshot, with each unit's strengths (all zero:
  // the planes stay as they are)
  ApplyArgs aa;
  aa.rec[0] = d_y;
  aa.rec[1] = d_u;
  aa.rec[2] = d_v;
  aa.snap[0] = reinterpret_cast<uint16_t*>(s + L.snap_y);
  aa.snap[1] = reinterpret_cast<uint16_t*>(s + L.snap_u);
  aa.snap[2] = reinterpret_cast<uint16_t*>(s + L.snap_v);
  const size_t ny = (size_t)g.w8 * g.h8 * 2, nc = (size_t)g.cw8 * g.ch8 * 2;
  if (cudaMemcpyAsync(s + L.snap_y, d_y, ny, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return MT_ERR_DEVICE;
  if (!mono) {
    if (cudaMemcpyAsync(s + L.snap_u, d_u, nc, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return MT_ERR_DEVICE;
    if (cudaMemcpyAsync(s + L.snap_v, d_v, nc, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return MT_ERR_DEVICE;
  }
  auto grid = [&](int per_warp, int planes) {
    return dim3((unsigned)((g.nbx * g.nby + 4 * per_warp - 1) / (4 * per_warp)), 1, (unsigned)planes);
  };
  const uint8_t* us = s + L.ustr;
  cdef_apply_kernel<8, 8><<<grid(1, !mono && !g.sub_x ? 3 : 1), 128, 0, st>>>(aa, g, d_skip8, dirs, vars, us, 0);
  mth::cdef_last_launches += 1;
  if (!mono && g.sub_x) {
    if (g.sub_y) cdef_apply_kernel<4, 4><<<grid(4, 2), 128, 0, st>>>(aa, g, d_skip8, dirs, vars, us, 1);
    else cdef_apply_kernel<4, 8><<<grid(2, 2), 128, 0, st>>>(aa, g, d_skip8, dirs, vars, us, 1);
    mth::cdef_last_launches += 1;
  }
  return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

// The decision of the last cdef_frame_enqueue over d_scratch, read back; waits
// for the stream.
int cdef_frame_decision(const mt_cdef_params* prm, void* d_scratch, mt_cdef_decision* out, uint8_t* grid,
                        cudaStream_t st) {
  const Geo g = make_geo(prm);
  const Layout L = make_layout(g, prm->mono != 0);
  uint8_t* s = static_cast<uint8_t*>(d_scratch);
  SearchState hs;
  if (cudaMemcpyAsync(&hs, s + L.state, sizeof(hs), cudaMemcpyDeviceToHost, st) != cudaSuccess) return MT_ERR_DEVICE;
  if (grid && cudaMemcpyAsync(grid, s + L.grid, (size_t)g.uc * g.ur, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return MT_ERR_DEVICE;
  if (cudaStreamSynchronize(st) != cudaSuccess) return MT_ERR_DEVICE;
  out->bits = hs.bits;
  out->damping = 3 + std::min(prm->base_q_idx / 64, 3);
  out->n_strengths = hs.n_strengths;
  out->unit_cols = g.uc;
  out->unit_rows = g.ur;
  memcpy(out->strengths, hs.strengths, sizeof(out->strengths));
  return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

}  // namespace mth

extern "C" {

int mt_cdef_frame_device(uint16_t* d_y, uint16_t* d_u, uint16_t* d_v, const uint16_t* d_src_y,
                         const uint16_t* d_src_u, const uint16_t* d_src_v, const uint8_t* d_skip8,
                         const mt_cdef_params* prm, void* d_scratch, mt_cdef_decision* out, uint8_t* grid,
                         void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (!out) {
    const int rc = check_params(prm);
    return rc != MT_OK ? rc : MT_ERR_INVALID_INPUT;
  }
  const int rc = mth::cdef_frame_enqueue(d_y, d_u, d_v, d_src_y, d_src_u, d_src_v, d_skip8, prm, d_scratch, nullptr,
                                         nullptr, nullptr, st);
  return rc != MT_OK ? rc : mth::cdef_frame_decision(prm, d_scratch, out, grid, st);
}

int mt_cdef_frame(uint16_t* y, uint16_t* u, uint16_t* v, const uint16_t* src_y, const uint16_t* src_u,
                  const uint16_t* src_v, const uint8_t* skip8, const mt_cdef_params* prm, mt_cdef_decision* out,
                  uint8_t* grid) {
  int rc = check_params(prm);
  if (rc != MT_OK) return rc;
  const bool mono = prm->mono != 0;
  if (!y || !src_y || !skip8 || !out) return MT_ERR_INVALID_INPUT;
  if (!mono && (!u || !v || !src_u || !src_v)) return MT_ERR_INVALID_INPUT;
  const Geo g = make_geo(prm);
  const size_t ny = (size_t)g.w8 * g.h8 * 2, nc = mono ? 0 : (size_t)g.cw8 * g.ch8 * 2, nsk = (size_t)g.nbx * g.nby;
  const size_t scratch = mt_cdef_scratch_bytes(prm);
  const size_t o_y = 0, o_sy = up256(ny), o_u = o_sy + up256(ny), o_v = o_u + up256(nc), o_su = o_v + up256(nc),
               o_sv = o_su + up256(nc), o_sk = o_sv + up256(nc), o_scr = o_sk + up256(nsk);
  uint8_t* d = nullptr;
  if (cudaMalloc(&d, o_scr + scratch) != cudaSuccess) return MT_ERR_ALLOC;
  cudaError_t e = cudaMemcpy(d + o_y, y, ny, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_sy, src_y, ny, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_sk, skip8, nsk, cudaMemcpyHostToDevice);
  if (!mono) {
    if (e == cudaSuccess) e = cudaMemcpy(d + o_u, u, nc, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + o_v, v, nc, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + o_su, src_u, nc, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + o_sv, src_v, nc, cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess) {
    rc = mt_cdef_frame_device((uint16_t*)(d + o_y), mono ? nullptr : (uint16_t*)(d + o_u),
                              mono ? nullptr : (uint16_t*)(d + o_v), (const uint16_t*)(d + o_sy),
                              mono ? nullptr : (const uint16_t*)(d + o_su), mono ? nullptr : (const uint16_t*)(d + o_sv),
                              d + o_sk, prm, d + o_scr, out, grid, nullptr);
    if (rc == MT_OK) {
      e = cudaMemcpy(y, d + o_y, ny, cudaMemcpyDeviceToHost);
      if (!mono && e == cudaSuccess) e = cudaMemcpy(u, d + o_u, nc, cudaMemcpyDeviceToHost);
      if (!mono && e == cudaSuccess) e = cudaMemcpy(v, d + o_v, nc, cudaMemcpyDeviceToHost);
    }
  }
  cudaFree(d);
  if (rc != MT_OK) return rc;
  return e == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

}  // extern "C"
