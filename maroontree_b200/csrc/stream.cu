// The encoder's entropy coding on the device, from the blocks' decisions and
// levels to every tile's payload bytes:
//
//   1. units_kernel (count): each transform block's token count and the
//      context byte it leaves its neighbours; a scan places the blocks in
//      coding order (tiles, superblocks and 8x8 blocks in z-order).
//   2. units_kernel (write): the block syntax (code_split always splitting down
//      to 8x8, src/coder/superblock.rs:950-990) and the coefficient symbols
//      (src/coeffs.rs:109-420, :583) as 16-bit tokens; hist / part_scan /
//      scatter put the tokens of each CDF in a list of their own, in order;
//      trace and fix adapt every CDF along its list (update_cdf) and write
//      the range coder's store (fl, fh, nms) of each token at its place.
//   3. map / compose / walk / ranges: the coder's range before every piece of
//      256 stores and the piece's share of the code value; shift_scan: the bit
//      position of every piece.
//   4. digits_kernel: the shares added into 16-bit digits; bytes_kernel: the
//      carries resolved and the bytes written.
//
// What makes each step parallel.  A token's contexts depend only on the levels
// and modes of its block and its left and top neighbours, all final, so no
// block waits for another.  A CDF depends only on the symbols coded with it:
// the 246 CDFs this encoder uses adapt side by side.  The coder's
// state (src/odec.rs:315-615) is its 16-bit range and the code value so far.
// The code value is a sum (each symbol adds r - u at its bit position), so
// pieces add up in any order.  The range is a serial chain, but a symbol other
// than the first of its CDF leaves a range that depends only on the top eight
// bits of the one before: 128 classes.  A piece therefore starts at such a
// symbol, is run from all 128 classes (four per lane), and the pieces' maps
// are composed; the range before every piece follows exactly, and the pieces
// are run again from it.
//
// Figures (quality 60; what a whole encode spends outside its decision
// kernel, upload and filters included, against the syntax walk, CDF adaptation
// and range coder on host threads that this replaces): 1920x1080 4:2:0, 0.83 M
// tokens, 10.0 -> 1.3 ms; 512x512 4:4:4, 0.23 M, 2.9 -> 0.54 ms; 4096x4096
// 4:4:4, 5.97 M in two tiles, 89 -> 8.3 ms.
#include "stream.h"

#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "../../include/maroontree_b200.h"
#include "av1_tables.h"
#include "chain4.cuh"
#include "chain8.cuh"

namespace mth {
struct StreamPlan {
  uint32_t* off;        // [3 nb] counts, then offsets inside a scan block
  uint32_t* bpre;       // [scan blocks] tokens before each scan block
  uint32_t* delta;      // [tiles] what places a tile's offsets in the token buffer
  uint32_t* cdef_at;    // [superblocks] first cdef_idx place
  uint8_t* res;         // [3 nb] context bytes
  StreamTile* tile;     // [tiles]
  StreamTotals* total;
};
}  // namespace mth

namespace {

using mth::StreamGeom;
using mth::StreamGroup;
using mth::StreamInput;
using mth::StreamPlan;
using mth::StreamTile;
using mth::StreamTotals;

// The CDFs this encoder codes with, by a dense id; the symbol of a token is in
// bits 8-12, bit 12 marking a gathered partition bool (split; bit 8: top).
enum Id : int {
  kPartBl8 = 0,
  kPartSplit = 1,       // 12: level x ctx
  kSkip = 13,
  kKfY = 14,            // 25: above * 5 + left
  kAngle = 39,          // 8
  kUvMode = 47,         // 13, CfL allowed
  kPalY = 60,
  kPalUv = 61,
  kFilterIntra = 62,    // BLOCK_8X8
  kTxsz = 63,           // 3
  kTxtp = 66,           // 13
  kTxbSkip = 79,        // luma, then chroma contexts 7-9
  kBase = 83,           // 41 per plane type
  kBr = 165,            // 21 per plane type
  kEobBase = 207,       // 4 per plane type
  kEobHi = 215,         // 11 per plane type
  kDcSign = 237,        // 3 per plane type
  kEobBin = 243,        // luma 2-D, luma 1-D, chroma
  kIds = 246,
  kBool = 254,          // equiprobable bit
  kNop = 255,           // a place for a cdef_idx bit, or padding
};
constexpr uint32_t kGathered = 16;

constexpr int kScanBlock = 4096;      // counts per scan block
constexpr int kPart = 2048;           // tokens a warp partitions
constexpr int kSeg = 1024;            // list entries a warp adapts a CDF along,
constexpr int kWarm = 2 * kSeg;       // after this many before them
constexpr int kChunk = 256;           // stores per piece of the range chain
constexpr int kGroup = 64;            // pieces per group
constexpr int kGroupTokens = kChunk * kGroup;  // tiles start at multiples of this
constexpr int kClasses = 128;
constexpr uint32_t kNoStart = 0xFFFFFFFFu;

__constant__ uint8_t cModeCtx[13] = {0, 1, 2, 3, 4, 4, 4, 4, 3, 0, 1, 2, 0};  // src/intrapred.rs:1088

// A store of the coder in 24 bits: fl >> 6 (512: no symbol below), fh >> 6,
// nms; 0 stands for no store.
__device__ __forceinline__ uint32_t store_word(uint32_t fl, uint32_t fh, uint32_t nms) {
  return (fl >> 6) | ((fh >> 6) << 10) | (nms << 20);
}
__device__ __forceinline__ uint32_t bool_word(bool v) {  // probability 1/2
  return v ? store_word(16384, 0, 1) : store_word(32768, 16384, 2);
}

// ---------------------------------------------------------------------------
// Tokens.

struct Place {
  int tx0, ty0, tx1, ty1, tile;
  uint32_t pos;  // coding-order position of the block in the frame
};

__device__ __forceinline__ int zrank(int x, int y, int w, int h) {  // z-order rank of (x, y) among the w x h blocks
  int r = 0;
#pragma unroll
  for (int s = 4; s >= 1; s >>= 1) {
    if (y >= s) r += w * min(s, h);
    const int hh = y >= s ? h - s : min(s, h);
    if (x >= s) r += min(s, w) * hh;
    w = x >= s ? w - s : min(s, w);
    h = hh;
    x = x >= s ? x - s : x;
    y = y >= s ? y - s : y;
  }
  return r;
}

__device__ __forceinline__ Place place_of(const StreamGeom& g, int x, int y) {
  Place p;
  const int tc = x / g.tile_w8, tr = y / g.tile_h8;
  p.tile = tr * g.tcols + tc;
  p.tx0 = tc * g.tile_w8;
  p.ty0 = tr * g.tile_h8;
  p.tx1 = min(p.tx0 + g.tile_w8, g.nbx);
  p.ty1 = min(p.ty0 + g.tile_h8, g.nby);
  const int tw = p.tx1 - p.tx0, th = p.ty1 - p.ty0;
  const int sx = x & ~7, sy = y & ~7;  // tiles are whole superblocks
  const int sw = min(8, p.tx1 - sx), sh = min(8, p.ty1 - sy);
  p.pos = (uint32_t)(g.nbx * p.ty0 + p.tx0 * th + (sy - p.ty0) * tw + (sx - p.tx0) * sh + zrank(x - sx, y - sy, sw, sh));
  return p;
}

__device__ __forceinline__ int hi_count(uint32_t m) { return m < 3 ? 0 : min(4, (int)(min(m - 3, 12u) / 3) + 1); }
__device__ __forceinline__ int golomb_count(uint32_t m) { return m < 15 ? 0 : 2 * (32 - __clz(m - 14)) - 1; }

// A transform block's levels as context bytes: 12 x 10, zero past the block.
constexpr int kLevStride = 12, kLevRows = 10;

// Eight lanes per N x N transform block of one plane, PER = N * N / 8
// consecutive scan positions per lane.  The context of a coefficient reads
// positions coded before it only, whose magnitudes are final, so every
// position's tokens are written at once at offsets from a scan over the lanes.
// Bound by the levels' read (256 bytes a block, coalesced) and the 2-byte
// token writes.
template <int N, bool LUMA, bool WRITE>
__global__ void __launch_bounds__(128) units_kernel(const StreamGeom g, const StreamInput in, const StreamPlan p,
                                                    const StreamGroup grp, uint16_t* __restrict__ tokens) {
  constexpr int PER = N * N / 8, LG = N == 8 ? 3 : 2;
  __shared__ __align__(16) int32_t cfs[16][64];
  __shared__ uint8_t lev[16][kLevStride * kLevRows];
  __shared__ uint8_t scan[64];
  const int t = threadIdx.x, l = t & 7, ul = t >> 3;
  const int nb = g.nbx * g.nby, u = min((int)blockIdx.x * 16 + ul, nb - 1);
  const bool live = (int)blockIdx.x * 16 + ul < nb;
  const int plane = LUMA ? 0 : 1 + (int)blockIdx.y;
  if (t < N * N) scan[t] = N == 8 ? mtd::kScan8[t] : mtd::kScan4[t];
  {
    const int32_t* cf = (LUMA ? in.lv[0] : (plane == 1 ? in.lv[1] : in.lv[2])) + (size_t)u * (N * N) + l * PER;
    if (PER == 8) {
      *reinterpret_cast<int4*>(&cfs[ul][l * 8]) = *reinterpret_cast<const int4*>(cf);
      *reinterpret_cast<int4*>(&cfs[ul][l * 8 + 4]) = *reinterpret_cast<const int4*>(cf + 4);
    } else {
      *reinterpret_cast<int2*>(&cfs[ul][l * 2]) = *reinterpret_cast<const int2*>(cf);
    }
  }
  if (WRITE)
    for (int i = l; i < kLevStride * kLevRows; i += 8) lev[ul][i] = 0;
  __syncthreads();
  const int y = u / g.nbx, x = u - y * g.nbx;
  const int ty = in.tx[u], m = in.mode[u];
  const int cls = LUMA && ty == MT_TX_V_DCT ? 1 : (LUMA && ty == MT_TX_H_DCT ? 2 : 0);
  // this lane's positions i = l * PER + j of the coding order
  auto raster = [&](int i) {
    return cls == 0 ? (int)scan[i] : (cls == 1 ? ((i & (N - 1)) << LG) | (i >> LG) : i);
  };
  int32_t v[PER];
  int eob = -1;
  uint32_t cul = 0, na = 0, nbits = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int k = raster(l * PER + j);
    v[j] = cfs[ul][k];
    const uint32_t a = (uint32_t)abs(v[j]);
    if (a) eob = l * PER + j;
    cul += a;
    na += hi_count(a);
    nbits += a ? 1 + golomb_count(a) : 0;
    if (WRITE) {
      const int cx = cls == 2 ? k & (N - 1) : k >> LG, cy = cls == 2 ? k >> LG : k & (N - 1);
      lev[ul][cx * kLevStride + cy] = a == 0 ? 0 : (a <= 2 ? (uint8_t)(a * 0x41) : (uint8_t)(min(a, 15u) + 0xC0));
    }
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    eob = max(eob, __shfl_xor_sync(~0u, eob, o));
    cul += __shfl_xor_sync(~0u, cul, o);
  }
  const int bin = eob < 2 ? max(eob, 0) : 32 - __clz(eob);
  const int head = eob < 0 ? 1 : 2 + (LUMA ? 1 : 0) + (bin > 1 ? bin - 1 : 0);
  // base and ladder tokens of this lane's positions (one base token each up
  // to the end of block), signs and remainders after them
  na += (uint32_t)max(0, min(PER, eob + 1 - l * PER));
  uint32_t run = na | (nbits << 16);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const uint32_t w = __shfl_up_sync(~0u, run, o, 8);
    if (l >= o) run += w;
  }
  const uint32_t tot = __shfl_sync(~0u, run, 7, 8);
  const uint32_t totA = tot & 0xffff, totB = tot >> 16;
  const Place pl = place_of(g, x, y);
  const bool dir = m >= MT_V_PRED && m <= MT_D67_PRED, dc = m == MT_DC_PRED;
  // the partition nodes that start at this block
  const bool first = ((x | y) & 7) == 0;
  int nodes = 0;
  if (LUMA)
#pragma unroll
    for (int s = 8; s >= 2; s >>= 1)
      if (((x | y) & (s - 1)) == 0) nodes += (x + s / 2 < g.nbx || y + s / 2 < g.nby) ? 1 : 0;
  const int syntax = LUMA ? nodes + 6 + (first ? 3 : 0) + (dir ? 1 : 0) + (dc ? 2 : 0) : 0;
  const uint32_t slot = 3 * pl.pos + plane;
  if (!WRITE) {
    if (live && l == 0) {
      const int c0 = cfs[ul][0];
      p.off[slot] = (uint32_t)(syntax + head) + totA + totB;
      p.res[3 * (size_t)u + plane] =
          eob < 0 ? 0x40 : (uint8_t)(min(cul, 63u) | (c0 == 0 ? 0x40 : (c0 < 0 ? 0 : 0x80)));
    }
    return;
  }
  __syncwarp();
  if (!live || (uint32_t)(pl.tile - grp.tile0) >= (uint32_t)grp.ntiles) return;
  uint32_t o = p.off[slot] + p.bpre[slot / kScanBlock] + p.delta[pl.tile];
  auto tok = [&](uint32_t at, int id, uint32_t s) { tokens[at] = (uint16_t)(id | (s << 8)); };
  const bool has_t = y > pl.ty0, has_l = x > pl.tx0;
  const uint32_t A = has_t ? p.res[3 * (size_t)(u - g.nbx) + plane] : 0x40;
  const uint32_t Lc = has_l ? p.res[3 * (size_t)(u - 1) + plane] : 0x40;
  const int s = (int)(A >> 6) + (int)(Lc >> 6) - 2, dcs = (s != 0) + (s > 0);
  const int ctx0 = cls == 0 ? 0 : 1;  // which end-of-block CDF
  constexpr int P = LUMA ? 0 : 1;
  if (l == 0) {
    uint32_t q = o;
    if (LUMA) {
#pragma unroll
      for (int sz = 8, bl = 1; sz >= 2; sz >>= 1, ++bl)
        if (((x | y) & (sz - 1)) == 0) {
          const bool h = x + sz / 2 < g.nbx, w = y + sz / 2 < g.nby;
          const int id = kPartSplit + (bl - 1) * 4 + has_t + 2 * has_l;
          if (h && w) tok(q++, id, 3);
          else if (h || w) tok(q++, id, kGathered | (h ? 1 : 0));
        }
      tok(q++, kPartBl8, 0);
      tok(q++, kSkip, 0);
      if (first) {  // read_cdef() follows the superblock's first skip flag
        p.cdef_at[(y >> 3) * g.sb_cols + (x >> 3)] = q;
        for (int k = 0; k < 3; ++k) tok(q++, kNop, 0);
      }
      const int ma = has_t ? in.mode[u - g.nbx] : 0, ml = has_l ? in.mode[u - 1] : 0;
      tok(q++, kKfY + cModeCtx[ma] * 5 + cModeCtx[ml], (uint32_t)m);
      if (dir) tok(q++, kAngle + m - MT_V_PRED, 3);  // delta 0
      tok(q++, kUvMode + m, MT_DC_PRED);
      if (dc) tok(q++, kPalY, 0);
      tok(q++, kPalUv, 0);
      if (dc) tok(q++, kFilterIntra, 0);
      tok(q++, kTxsz + has_l + has_t, 0);
    }
    tok(q++, kTxbSkip + (LUMA ? 0 : 1 + (A != 0x40) + (Lc != 0x40)), eob < 0 ? 1 : 0);
    if (eob >= 0) {
      if (LUMA) tok(q++, kTxtp + m, cls == 1 ? 2 : (cls == 2 ? 3 : ty));
      tok(q++, kEobBin + (LUMA ? ctx0 : 2), bin);
      if (bin > 1) {
        tok(q++, kEobHi + P * 11 + bin, (eob >> (bin - 2)) & 1);
        for (int b = bin - 3; b >= 0; --b) tok(q++, kBool, (eob >> b) & 1);
      }
    }
  }
  if (eob < 0) return;
  o += syntax + head;
  uint32_t qa = o + totA - (run & 0xffff);           // after the positions of the lanes above
  uint32_t qb = o + totA + (run >> 16) - nbits;      // after the signs of the lanes below
  const uint8_t* lv = lev[ul];
#pragma unroll
  for (int j = PER - 1; j >= 0; --j) {
    const int i = l * PER + j;
    if (i > eob) continue;
    const int k = raster(i);
    const int cx = cls == 2 ? k & (N - 1) : k >> LG, cy = cls == 2 ? k >> LG : k & (N - 1);
    const uint8_t* c = lv + cx * kLevStride + cy;
    const uint32_t a = (uint32_t)abs(v[j]);
    uint32_t hi, mag;
    int far;
    if (cls == 0) {
      hi = (uint32_t)c[1] + c[kLevStride] + c[kLevStride + 1];
      mag = hi + c[2] + c[2 * kLevStride];
      far = (cx | cy) > 1;
    } else {
      hi = (uint32_t)c[1] + c[kLevStride] + c[2];
      mag = hi + c[3] + c[4];
      far = cy != 0;
    }
    int br;
    if (i == eob) {
      const int ce = eob == 0 ? 0 : 1 + (eob > (N * N >> 3)) + (eob > (N * N >> 2));
      tok(qa++, kEobBase + P * 4 + ce, min(a, 3u) - 1);
      br = eob == 0 ? 0 : (far ? 14 : 7);
    } else {
      const int lo = mag > 512 ? 4 : (int)((mag + 64) >> 7);
      int ctx;
      if (cls == 0) {
        // eLoOff by min(diagonal): 1 and 6 near the origin, 21 further out, 0 at DC
        const int d = min(cx, 4) + min(cy, 4);
        ctx = i == 0 ? 0 : lo + (d < 2 ? 1 : (d < 4 ? 6 : 21));
      } else {
        ctx = 26 + (cy > 1 ? 10 : cy * 5) + lo;
      }
      tok(qa++, kBase + P * 41 + ctx, min(a, 3u));
      const uint32_t mg = hi & 63;
      br = (i == 0 ? 0 : (far ? 14 : 7)) + (mg > 12 ? 6 : (int)((mg + 1) >> 1));
    }
    if (a >= 3) {
      const int total = min((int)a - 3, 12);
      int coded = 0;
      for (int e = 0; e < 4; ++e) {
        const int sy = min(total - coded, 3);
        tok(qa++, kBr + P * 21 + br, sy);
        coded += sy;
        if (sy < 3) break;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int i = l * PER + j;
    const uint32_t a = (uint32_t)abs(v[j]);
    if (!a) continue;
    if (i == 0) tok(qb++, kDcSign + P * 3 + dcs, v[j] < 0);
    else tok(qb++, kBool, v[j] < 0);
    if (a >= 15) {
      const uint32_t xg = a - 14;
      const int len = 32 - __clz(xg);
      for (int e = 0; e < len - 1; ++e) tok(qb++, kBool, 0);
      for (int e = len - 1; e >= 0; --e) tok(qb++, kBool, (xg >> e) & 1);
    }
  }
}

// ---------------------------------------------------------------------------
// Placement: an exclusive scan of the 3 nb counts, 4096 per CTA, then of the
// CTAs' sums, which also lays the tiles out, in groups of whole tiles that the
// following steps take one after the other in the same buffers.  A frame's total
// may pass 32 bits (from some 75 Mpx of 4:4:4 noise at quality 99 on), and the
// running sums here wrap; a tile's extent and its place in its group do not:
// at most 31 tokens per coefficient (levels below 2^13 at the finest steps) and
// 2,376 superblocks make under 2^30, and differences of wrapped sums are exact.

__device__ __forceinline__ uint32_t block_scan_1024(uint32_t v, uint32_t* warp_sum, uint32_t* total) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  uint32_t s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t q = __shfl_up_sync(~0u, s, o);
    if (lane >= o) s += q;
  }
  if (lane == 31) warp_sum[w] = s;
  __syncthreads();
  if (w == 0) {
    uint32_t q = warp_sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t r = __shfl_up_sync(~0u, q, o);
      if (lane >= o) q += r;
    }
    warp_sum[lane] = q;
  }
  __syncthreads();
  const uint32_t ex = s - v + (w ? warp_sum[w - 1] : 0);
  *total = warp_sum[31];
  __syncthreads();
  return ex;
}

__global__ void __launch_bounds__(1024) scan_local_kernel(uint32_t* __restrict__ off, int n,
                                                          uint32_t* __restrict__ sums) {
  __shared__ uint32_t ws[32];
  const int i = blockIdx.x * kScanBlock + threadIdx.x * 4;
  uint32_t c[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) c[k] = i + k < n ? off[i + k] : 0;
  uint32_t total;
  uint32_t run = block_scan_1024(c[0] + c[1] + c[2] + c[3], ws, &total);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i + k < n) off[i + k] = run;
    run += c[k];
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) scan_blocks_kernel(const StreamGeom g, const StreamPlan p, int nblk) {
  __shared__ uint32_t ws[32];
  uint32_t carry = 0;
  for (int b = 0; b < nblk; b += 1024) {
    const int i = b + (int)threadIdx.x;
    uint32_t total;
    const uint32_t ex = block_scan_1024(i < nblk ? p.bpre[i] : 0, ws, &total);
    if (i < nblk) p.bpre[i] = carry + ex;
    carry += total;
  }
  __syncthreads();
  const int nt = g.tcols * g.trows;
  for (int k = threadIdx.x; k < nt; k += 1024) {  // each tile's first token in the unpadded order
    const int ty0 = (k / g.tcols) * g.tile_h8, tx0 = (k % g.tcols) * g.tile_w8;
    const int th = min(g.tile_h8, g.nby - ty0);
    const uint32_t i = 3u * (uint32_t)(g.nbx * ty0 + tx0 * th);
    p.delta[k] = p.off[i] + p.bpre[i / kScanBlock];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t base = 0, most = 0, groups = 1;
    for (int k = 0; k < nt; ++k) {
      const uint32_t start = p.delta[k], end = k + 1 < nt ? p.delta[k + 1] : carry;
      const uint32_t n = (end - start + kGroupTokens - 1) / kGroupTokens * kGroupTokens;
      if (base && (base >= g.max_tokens || n > g.max_tokens - base)) {  // the next group
        base = 0;
        ++groups;
      }
      p.tile[k].base = base;
      p.tile[k].ntok = end - start;
      p.delta[k] = base - start;
      base += n;
      most = max(most, base);
    }
    p.total->tokens = most;
    p.total->groups = groups;
  }
}

// ---------------------------------------------------------------------------
// Partition of the tokens by CDF, keeping their order: a histogram per 2048
// tokens, a scan of the histograms, and the scatter.

struct Lists {
  uint16_t* tok;    // [padded] tokens
  uint32_t* st;     // [padded] stores
  uint32_t* idx;    // [padded] a list entry's token
  uint8_t* sym;     // [padded] a list entry's symbol
  uint32_t* hist;   // [padded / kPart][256]
  uint2* list;      // [tiles][256] (first entry, entries)
  uint32_t* seg0;   // [tiles][256] segments of the tile's lists before a list
  uint16_t* seg_a;  // [segments][16] a CDF before a segment (entry 15: updates so far, 32 at most)
  uint16_t* seg_b;  // [segments][16] and after it
  uint16_t* seg_m;  // [segments] its largest symbol, and the smallest << 8
  uint16_t* map;    // [padded / kChunk][128] the range after a piece, by class before it
  uint32_t* spos;   // [padded / kChunk] first store of a piece, or kNoStart
  uint16_t* gmap;   // [groups][128]
  uint16_t* gr;     // [groups] the range before a group
  uint32_t* cd;     // [padded / kChunk] bits shifted out before a piece, in its group
  uint32_t* nd;     // [padded / kChunk] digits of a piece
  uint32_t* loc;    // [padded + 4 pieces] every piece's digits, its first bit at the top of a digit
  uint32_t* gd;     // [groups] bits shifted out by a group, then before it
};

__device__ __forceinline__ int tile_of(const StreamTile* __restrict__ tile, int nt, uint32_t i) {
  int k = 0;
  while (k + 1 < nt && tile[k + 1].base <= i) ++k;
  return k;
}

__global__ void __launch_bounds__(128) hist_kernel(const Lists L, const StreamTile* __restrict__ tile, int nt) {
  __shared__ uint32_t h[4][256];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunk = blockIdx.x * 4 + w, a = chunk * kPart;
  for (int i = lane; i < 256; i += 32) h[w][i] = 0;
  __syncwarp();
  const StreamTile ti = tile[tile_of(tile, nt, a)];
  const uint32_t end = min(a + kPart, ti.base + ti.ntok);
  for (uint32_t i = a + lane; i < end; i += 32) atomicAdd(&h[w][L.tok[i] & 255], 1u);
  __syncwarp();
  for (int i = lane; i < 256; i += 32) L.hist[(size_t)chunk * 256 + i] = h[w][i];
}

// A CTA per tile, four threads per CDF each over a quarter of the chunks.
__global__ void __launch_bounds__(1024) part_scan_kernel(const Lists L, const StreamTile* __restrict__ tile) {
  __shared__ uint32_t part[4][256], first[256], segs[256];
  const StreamTile ti = tile[blockIdx.x];
  const int id = threadIdx.x & 255, q = threadIdx.x >> 8;
  const int c0 = (int)(ti.base / kPart), n = (int)((ti.ntok + kPart - 1) / kPart);
  const int lo = c0 + n * q / 4, hi = c0 + n * (q + 1) / 4;
  uint32_t s = 0;
#pragma unroll 8
  for (int c = lo; c < hi; ++c) s += L.hist[(size_t)c * 256 + id];
  part[q][id] = s;
  __syncthreads();
  if (q == 0) {
    const uint32_t total = id < kIds ? part[0][id] + part[1][id] + part[2][id] + part[3][id] : 0;
    first[id] = total;
    segs[id] = (total + kSeg - 1) / kSeg;
  }
  __syncthreads();
  if (threadIdx.x < 64) {  // exclusive scans over the CDFs, eight per lane: entries and segments
    uint32_t* a = threadIdx.x < 32 ? first : segs;
    const int l = threadIdx.x & 31;
    uint32_t v[8], sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k] = a[l * 8 + k];
      sum += v[k];
    }
    uint32_t ex = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t w = __shfl_up_sync(~0u, ex, o);
      if (l >= o) ex += w;
    }
    ex -= sum;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      a[l * 8 + k] = ex;
      ex += v[k];
    }
  }
  __syncthreads();
  uint32_t run = ti.base + first[id];
  if (q == 1) L.seg0[blockIdx.x * 256 + id] = segs[id];
  if (q == 0)
    L.list[blockIdx.x * 256 + id] = make_uint2(run, part[0][id] + part[1][id] + part[2][id] + part[3][id]);
  for (int k = 0; k < q; ++k) run += part[k][id];
#pragma unroll 8
  for (int c = lo; c < hi; ++c) {
    const uint32_t v = L.hist[(size_t)c * 256 + id];
    L.hist[(size_t)c * 256 + id] = run;
    run += v;
  }
}

__global__ void __launch_bounds__(128) scatter_kernel(const Lists L, const StreamTile* __restrict__ tile, int nt) {
  __shared__ uint32_t at[4][256];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunk = blockIdx.x * 4 + w, a = chunk * kPart;
  const StreamTile ti = tile[tile_of(tile, nt, a)];
  const uint32_t end = ti.base + ti.ntok;
  if (a < end)
    for (int i = lane; i < 256; i += 32) at[w][i] = L.hist[(size_t)chunk * 256 + i];
  __syncwarp();
  for (int b = 0; b < kPart; b += 32) {
    const uint32_t i = a + b + lane;
    const uint32_t t = i < end ? L.tok[i] : (uint32_t)kNop;
    const int id = t & 255;
    const uint32_t same = __match_any_sync(~0u, id);
    if (id < kIds) {
      const uint32_t e = at[w][id] + __popc(same & ((1u << lane) - 1));
      L.idx[e] = i;
      L.sym[e] = (uint8_t)(t >> 8);
    } else {
      L.st[i] = id == kBool ? bool_word((t >> 8) != 0) : 0;
    }
    __syncwarp();
    if (id < kIds && (same >> lane) == 1) at[w][id] += __popc(same);  // the last lane of each CDF
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// update_cdf along a CDF's list.  Lanes i and 16 + i of a warp hold entry i:
// entries below the symbol move up by (32768 - c) >> rate, the others down by
// c >> rate.  With v the distance from where the entry is moving, 32768 - c or
// c, both are v -= v >> rate, and only a change of direction costs a third
// operation.  The distances before each of 32 updates go to shared memory and
// lane k takes the k-th symbol's.
//
// The chain along a list is serial (16 cycles a symbol, 25 with the two
// directions computed apart), but a CDF forgets: two states that see the same
// symbols move together by 1/128 (1/64 for short CDFs) a symbol and, being whole
// numbers, meet; only an entry within 1 << rate of its end of the range rests
// where it is until a symbol moves it away, and then comes back to just that
// distance.  So a long list is cut into segments of 1024.  The first of each list
// is adapted by itself; the others by a warp each, along the 2048 symbols before
// the segment from the state after the first one, its entries at rest put at
// that distance if a symbol has moved them since.  fix_kernel then compares every
// segment's first state with the last one of the segment before and adapts
// again, from the true state, those that differ (none of 659 segments at
// 1920x1080, 1 of 2,960 in a tile of 4096x4096; from the initial CDF 16 and 66,
// most of them in a row).

// 32 updates of entry c; bit k of up: the k-th moves it up.
template <int RATE, bool STORE>
__device__ __forceinline__ int trace_batch(int c, uint32_t up, uint32_t* buf) {
  const int lane = threadIdx.x & 15;
  const uint32_t last = up >> 31;
  uint32_t turn = up ^ (up >> 1) ^ (last << 31);
  int v = (up & 1) ? 32768 - c : c;
#pragma unroll 1
  for (int g = 0; g < 4; ++g) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (STORE) buf[(g * 8 + k) * 17 + lane] = (uint32_t)v;  // twice the same
      v -= v >> RATE;
      if ((turn >> k) & 1) v = 32768 - v;
    }
    turn >>= 8;
  }
  return last ? 32768 - v : v;
}

// Entries [from, to) of the list li from state c (updates so far: done).
template <bool STORE>
__device__ __forceinline__ void trace_span(const Lists& L, const uint2 li, uint32_t from, uint32_t to, int n,
                                           bool updating, uint32_t* buf, int& c, uint32_t& done) {
  const int lane = threadIdx.x & 31, rate0 = 3 + min(n >> 1, 2);
  // four batches of 32 at a time, the next four loaded ahead: a batch is shorter
  // than the way to L2
  uint32_t nidx[4], nsym[4], idx[4], syms[4];
  auto ahead = [&](uint32_t b) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t e = b + j * 32 + lane;
      nidx[j] = STORE && e < to ? L.idx[li.x + e] : 0;
      nsym[j] = e < to ? L.sym[li.x + e] : 0;
    }
  };
  ahead(from);
  for (uint32_t b = from; b < to; b += 32) {
    const uint32_t q4 = ((b - from) >> 5) & 3;
    if (q4 == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        idx[j] = nidx[j];
        syms[j] = nsym[j];
      }
      ahead(b + 128);
    }
    const uint32_t i = q4 < 2 ? (q4 ? idx[1] : idx[0]) : (q4 == 2 ? idx[2] : idx[3]);
    const uint32_t sym = q4 < 2 ? (q4 ? syms[1] : syms[0]) : (q4 == 2 ? syms[2] : syms[3]);
    const bool live = b + lane < to;
    const bool upd = live && updating && sym < kGathered;
    const uint32_t um = __ballot_sync(~0u, upd);
    uint32_t mask = 0;  // bit k: symbol k is above this lane's entry
    for (int e = 0; e < n - 1; ++e) {
      const uint32_t q = __ballot_sync(~0u, (int)sym > e);
      if ((lane & 15) == e) mask = q;
    }
    if (um == ~0u && done >= 32) {
      if (rate0 == 5) c = trace_batch<7, STORE>(c, mask, buf);
      else c = trace_batch<6, STORE>(c, mask, buf);
    } else {
      const uint32_t ord = done + __popc(um & ((1u << lane) - 1));
      const int myrate = rate0 + (int)(min(ord, 32u) >> 4);
#pragma unroll 1
      for (int k = 0; k < 32; ++k) {
        const int rate = __shfl_sync(~0u, myrate, k);
        const bool up = (mask >> k) & 1;
        int v = up ? 32768 - c : c;
        if (STORE) buf[k * 17 + (lane & 15)] = (uint32_t)v;
        if ((um >> k) & 1) v -= v >> rate;
        c = up ? 32768 - v : v;
      }
    }
    done = min(done + __popc(um), 32u);
    if (!STORE) continue;
    __syncwarp();
    if (live) {
      const uint32_t* row = buf + lane * 17;
      uint32_t wd;
      if (sym < kGathered) {
        wd = store_word(sym ? 32768 - row[sym - 1] : 32768u, row[sym], (uint32_t)n - sym);
      } else {  // gather_split_prob_icdf (src/coeffs.rs:2927-2935), the split taken
        auto r = [&](int s) { return 32768 - (int)row[s]; };
        const int out = (sym & 1) ? (r(1) - r(4)) + r(5) + (r(8) - r(7)) : (r(0) - r(1)) + (r(2) - r(6)) + (r(7) - r(8));
        wd = store_word((uint32_t)min(max(out, 1), 32767), 0, 1);
      }
      L.st[i] = wd;
    }
    __syncwarp();
  }
}

constexpr int kCdfEntries = 16;
__device__ __forceinline__ size_t seg_slot(const StreamTile* tile, int t, uint32_t k) {
  return (size_t)tile[t].base / kSeg + 256 * t + k;
}

// The list and segment of a warp's slot; false past the tile's segments.
__device__ __forceinline__ bool find_segment(const Lists& L, const StreamTile* __restrict__ tile, int nt,
                                             uint32_t slot, int& t, int& id, uint32_t& seg) {
  const int lane = threadIdx.x & 31;
  t = 0;
  while (t + 1 < nt && seg_slot(tile, t + 1, 0) <= slot) ++t;
  const uint32_t k = slot - (uint32_t)seg_slot(tile, t, 0);
  // the list: the last one with its first segment at or before k (the ids past
  // the CDFs hold the tile's number of segments)
  const uint32_t* seg0 = L.seg0 + t * 256;
  if (k >= seg0[255]) return false;
  const int hi = __popc(__ballot_sync(~0u, seg0[lane * 8] <= k)) - 1;
  id = hi * 8 + __popc(__ballot_sync(~0u, lane < 8 && seg0[hi * 8 + (lane & 7)] <= k)) - 1;
  seg = k - seg0[id];
  return true;
}

// The first segment of every list, and the symbols' extremes of the others.
__global__ void __launch_bounds__(128) first_kernel(const Lists L, const StreamTile* __restrict__ tile, int nt,
                                                    const uint16_t* __restrict__ cdfs, int updating) {
  __shared__ uint32_t bufs[4][32 * 17];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t slot = blockIdx.x * 4 + w;
  int t, id;
  uint32_t seg;
  if (!find_segment(L, tile, nt, slot, t, id, seg)) return;
  const uint2 li = L.list[t * 256 + id];
  const uint32_t from = seg * kSeg, to = min(from + kSeg, li.y);
  if (seg == 0) {
    const int n = cdfs[id * kCdfEntries + 15];  // symbols
    int c = (lane & 15) < n - 1 ? cdfs[id * kCdfEntries + (lane & 15)] : 0;
    uint32_t done = 0;
    trace_span<true>(L, li, from, to, n, updating, bufs[w], c, done);
    if (lane < 16) L.seg_b[(size_t)slot * 16 + lane] = (uint16_t)(lane == 15 ? done : (uint32_t)c);
  } else {
    uint32_t hi = 0, lo = 255;
#pragma unroll 8
    for (uint32_t i = from + lane; i < to; i += 32) {
      const uint32_t s = L.sym[li.x + i];
      hi = max(hi, s < kGathered ? s : 0);
      lo = min(lo, s);
    }
    hi = __reduce_max_sync(~0u, hi);
    lo = __reduce_min_sync(~0u, lo);
    if (lane == 0) L.seg_m[slot] = (uint16_t)(hi | (lo << 8));
  }
}

// A warp per later segment.
__global__ void __launch_bounds__(128) trace_kernel(const Lists L, const StreamTile* __restrict__ tile, int nt,
                                                    const uint16_t* __restrict__ cdfs, int updating) {
  __shared__ uint32_t bufs[4][32 * 17];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t slot = blockIdx.x * 4 + w;
  int t, id;
  uint32_t seg;
  if (!find_segment(L, tile, nt, slot, t, id, seg) || seg == 0) return;
  const uint2 li = L.list[t * 256 + id];
  const int n = cdfs[id * kCdfEntries + 15], e = lane & 15;
  const uint32_t start = seg > kWarm / kSeg ? seg - kWarm / kSeg : 1;  // the warm-up's first segment
  const uint32_t first = slot - seg;
  uint32_t hi = 0, lo = 255;
  for (uint32_t k = 1 + lane; k < start; k += 32) {
    const uint32_t m = L.seg_m[first + k];
    hi = max(hi, m & 255);
    lo = min(lo, m >> 8);
  }
  hi = __reduce_max_sync(~0u, hi);
  lo = __reduce_min_sync(~0u, lo);
  const uint32_t v = L.seg_b[(size_t)first * 16 + e];
  uint32_t done = __shfl_sync(~0u, v, 15);
  int c = e < n - 1 ? (int)v : 0;
  const int rest = (1 << (5 + min(n >> 1, 2))) - 1;
  if (e < n - 1 && updating) {
    if (hi > (uint32_t)e && c < rest) c = rest;
    if (lo <= (uint32_t)e && c > 32768 - rest) c = 32768 - rest;
  }
  const uint32_t from = seg * kSeg, to = min(from + kSeg, li.y);
  trace_span<false>(L, li, start * kSeg, from, n, updating, nullptr, c, done);
  if (lane < 16) L.seg_a[(size_t)slot * 16 + lane] = (uint16_t)(lane == 15 ? done : (uint32_t)c);
  trace_span<true>(L, li, from, to, n, updating, bufs[w], c, done);
  if (lane < 16) L.seg_b[(size_t)slot * 16 + lane] = (uint16_t)(lane == 15 ? done : (uint32_t)c);
}

// A CTA per list of several segments, 256 of them at a time: the segments whose
// first state is not the last one before them, eight at once (a warp each),
// until there are none; the first of them is right after one turn.
__global__ void __launch_bounds__(256) fix_kernel(const Lists L, const StreamTile* __restrict__ tile,
                                                  const uint16_t* __restrict__ cdfs, int updating) {
  __shared__ uint32_t bufs[8][32 * 17], bad[8];
  const int id = blockIdx.x, t = blockIdx.y, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint2 li = L.list[t * 256 + id];
  const uint32_t nseg = (li.y + kSeg - 1) / kSeg;
  if (nseg < 2) return;
  const int n = cdfs[id * kCdfEntries + 15];
  const size_t slot = seg_slot(tile, t, L.seg0[t * 256 + id]);
  uint16_t* const A = L.seg_a + slot * 16;
  uint16_t* const B = L.seg_b + slot * 16;
  for (uint32_t s0 = 1; s0 < nseg; s0 += 256) {
    for (;;) {
      const uint32_t s = s0 + threadIdx.x;
      bool differs = false;
      if (s < nseg) {
        const uint4* a = reinterpret_cast<const uint4*>(A + s * 16);
        const uint4* b = reinterpret_cast<const uint4*>(B + s * 16 - 16);
        const uint4 a0 = a[0], a1 = a[1], b0 = b[0], b1 = b[1];
        differs = ((a0.x ^ b0.x) | (a0.y ^ b0.y) | (a0.z ^ b0.z) | (a0.w ^ b0.w) | (a1.x ^ b1.x) | (a1.y ^ b1.y) |
                   (a1.z ^ b1.z) | (a1.w ^ b1.w)) != 0;
      }
      const uint32_t m = __ballot_sync(~0u, differs);
      if (lane == 0) bad[w] = m;
      __syncthreads();
      // this warp's segment: the w-th differing one
      int left = w, k = -1;
      bool any = false;
      for (int i = 0; i < 8; ++i) {
        uint32_t q = bad[i];
        any = any || q;
        const int c = __popc(q);
        if (k < 0 && left < c) {
          for (; left; --left) q &= q - 1;
          k = i * 32 + __ffs(q) - 1;
        } else if (k < 0) {
          left -= c;
        }
      }
      if (!any) break;
      const uint32_t seg = s0 + (uint32_t)k;
      const uint32_t v = k >= 0 ? B[(seg - 1) * 16 + (lane & 15)] : 0;
      __syncthreads();
      if (k >= 0) {
        if (lane < 16) A[seg * 16 + lane] = (uint16_t)v;
        uint32_t done = __shfl_sync(~0u, v, 15);
        int c = (lane & 15) < n - 1 ? (int)v : 0;
        trace_span<true>(L, li, seg * kSeg, min((seg + 1) * kSeg, li.y), n, updating, bufs[w], c, done);
        if (lane < 16) B[seg * 16 + lane] = (uint16_t)(lane == 15 ? done : (uint32_t)c);
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// The range coder.

__global__ void cdef_fill_kernel(const StreamGeom g, const StreamPlan p, const StreamGroup grp,
                                 uint32_t* __restrict__ st, const int32_t* __restrict__ bits,
                                 const uint8_t* __restrict__ grid, int nsb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = *bits;
  if (i >= nsb || n <= 0 || n > 3) return;
  const int tile = i / g.sb_cols * 8 / g.tile_h8 * g.tcols + i % g.sb_cols * 8 / g.tile_w8;
  if ((uint32_t)(tile - grp.tile0) >= (uint32_t)grp.ntiles) return;
  for (int k = 0; k < n; ++k) st[p.cdef_at[i] + k] = bool_word((grid[i] >> (n - 1 - k)) & 1);
}

// A store after which the range depends on the top byte before it only.
__device__ __forceinline__ bool is_start(uint32_t w) { return w != 0 && (w & 1023) < 512; }

// The sub-range of store w (not 0) at range r: l below it, nr its size.
__device__ __forceinline__ void sub_range(uint32_t w, uint32_t r, uint32_t& l, uint32_t& nr) {
  const uint32_t fl = w & 1023, fh = (w >> 10) & 1023, nms = w >> 20, R = r >> 8;
  const uint32_t u = fl == 512 ? r : ((R * fl) >> 1) + 4 * nms;
  const uint32_t v = ((R * fh) >> 1) + 4 * (nms - 1);
  l = r - u;
  nr = u - v;
}

// N states per lane over n stores, unpacked in shared memory: (fl, fh, 4 nms -
// 4, set without a symbol below).  Ranges are kept with their top bit at bit 31.
template <int N>
__device__ __forceinline__ void map_batch(uint32_t* r, const uint4* w, int n) {
#pragma unroll 2
  for (int k = 0; k < n; ++k) {
    const uint4 q = w[k];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const uint32_t R = r[j] >> 24;
      const uint32_t top = q.w ? (r[j] >> 16) - q.z : ((R * q.x) >> 1) + 4;
      const uint32_t nr = top - ((R * q.y) >> 1);
      r[j] = nr << __clz(nr);
    }
  }
}

// A warp per piece: the range after it from each of the 128 classes before
// it, at first four per lane.  Ranges meet as the stores go by (50 to 60
// different ones of the 128 are left after 32 stores, 35 after 64, under 30
// after 128, mostly neighbours), so between batches of 32 equal neighbours are
// merged whenever that halves the states per lane.  A piece runs from its first
// start store (a tile's first piece from the tile's first store) to the next
// piece's.
__global__ void __launch_bounds__(128) map_kernel(const Lists L, const StreamTile* __restrict__ tile, int nt) {
  __shared__ uint32_t sh_r[4][kClasses];
  __shared__ uint8_t sh_i[4][kClasses];
  __shared__ uint4 sh_w[4][32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const uint32_t c = blockIdx.x * 4 + wp, a = c * kChunk;
  const StreamTile ti = tile[tile_of(tile, nt, a)];
  const uint32_t end = ti.base + ti.ntok;
  uint32_t r[4], cls[4];  // the states of this lane; where its classes' states are
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    r[j] = (uint32_t)(kClasses + j * 32 + lane) << 24;
    cls[j] = j * 32 + lane;
  }
  int per = 4, cnt = kClasses;
  bool started = false;
  for (uint32_t b = a; b < end; b += 32) {
    const uint32_t w = b + lane < end ? L.st[b + lane] : 0;
    uint32_t live = __ballot_sync(~0u, w != 0);
    const uint32_t starts = __ballot_sync(~0u, is_start(w));
    if (!started) {
      if (b >= a + kChunk) break;
      const bool tile_first = a == ti.base;
      if (!tile_first && !starts) continue;
      const int f = tile_first ? 0 : __ffs(starts) - 1;
      live &= ~0u << f;
      started = true;
      if (lane == 0) L.spos[c] = b + f;
    } else if (b >= a + kChunk && starts) {  // the next piece starts here
      live &= (1u << (__ffs(starts) - 1)) - 1;
    }
    if ((live >> lane) & 1) {
      const uint32_t fl = w & 1023, nms = w >> 20;
      sh_w[wp][__popc(live & ((1u << lane) - 1))] =
          make_uint4(fl, (w >> 10) & 1023, 4 * (nms - 1), fl == 512);
    }
    __syncwarp();
    const int nw = __popc(live);
    if (per == 4) map_batch<4>(r, sh_w[wp], nw);
    else if (per == 2) map_batch<2>(r, sh_w[wp], nw);
    else map_batch<1>(r, sh_w[wp], nw);
    __syncwarp();
    if (b >= a + kChunk && starts) break;
    if (per > 1) {
      uint32_t at[4];  // a state's place after merging
      int n = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t before = __shfl_up_sync(~0u, r[j], 1);
        const uint32_t last = __shfl_sync(~0u, r[j ? j - 1 : 0], 31);
        if (lane == 0) before = j ? last : 0;
        const uint32_t m = __ballot_sync(~0u, j * 32 + lane < cnt && r[j] != before);
        at[j] = (uint32_t)(n + __popc(m & ((2u << lane) - 1)) - 1);
        n += __popc(m);
      }
      if (n <= 16 * per) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j * 32 + lane < cnt) {  // equal states write the same value
            sh_r[wp][at[j]] = r[j];
            sh_i[wp][j * 32 + lane] = (uint8_t)at[j];
          }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          cls[j] = sh_i[wp][cls[j]];
          r[j] = sh_r[wp][min(j * 32 + lane, n - 1)];
        }
        __syncwarp();
        cnt = n;
        per = n <= 32 ? 1 : 2;
      }
    }
  }
  if (!started && lane == 0) L.spos[c] = kNoStart;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < per) sh_r[wp][j * 32 + lane] = r[j] >> 16;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j) L.map[(size_t)c * kClasses + j * 32 + lane] = started ? (uint16_t)sh_r[wp][cls[j]] : 0;
}

// A group's map from its pieces' (0: the range is unchanged).
__global__ void __launch_bounds__(kClasses) compose_kernel(const Lists L) {
  __shared__ uint16_t m[kGroup][kClasses];
  const int t = threadIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(L.map + (size_t)blockIdx.x * kGroup * kClasses);
  uint4* dst = reinterpret_cast<uint4*>(&m[0][0]);
  for (int i = t; i < kGroup * kClasses / 8; i += kClasses) dst[i] = src[i];
  __syncthreads();
  uint32_t cur = 0;
  for (int k = 0; k < kGroup; ++k) {
    const uint32_t v = m[k][cur ? (cur >> 8) - kClasses : t];
    cur = v ? v : cur;
  }
  L.gmap[(size_t)blockIdx.x * kClasses + t] = (uint16_t)cur;
}

// A CTA per tile walks its groups.
__global__ void __launch_bounds__(256) walk_kernel(const Lists L, const StreamTile* __restrict__ tile) {
  __shared__ uint16_t m[kGroup][kClasses];
  const StreamTile ti = tile[blockIdx.x];
  const int g0 = (int)(ti.base / kGroupTokens), n = (int)((ti.ntok + kGroupTokens - 1) / kGroupTokens);
  uint32_t r = 0x8000;
  for (int b = 0; b < n; b += kGroup) {
    const int k1 = min(kGroup, n - b);
    const uint4* src = reinterpret_cast<const uint4*>(L.gmap + (size_t)(g0 + b) * kClasses);
    uint4* dst = reinterpret_cast<uint4*>(&m[0][0]);
    __syncthreads();
    for (int i = threadIdx.x; i < k1 * kClasses / 8; i += 256) dst[i] = src[i];
    __syncthreads();
    if (threadIdx.x == 0)
      for (int k = 0; k < k1; ++k) {
        L.gr[g0 + b + k] = (uint16_t)r;
        const uint32_t v = m[k][(r >> 8) - kClasses];
        r = v ? v : r;
      }
  }
}

// Calls f(l, d) for the stores of a piece from its range r (l = d = 0 for a word
// that is none): one thread per piece, sixteen bytes of stores at a time, the
// next ones loaded ahead; straight-line code, as every lane of the warp is at
// another store.
template <class F>
__device__ __forceinline__ void run_piece(const uint32_t* __restrict__ st, uint32_t from, uint32_t next,
                                          uint32_t end, uint32_t r, F&& f) {
  const uint4* v = reinterpret_cast<const uint4*>(st);
  uint32_t q = from >> 2;
  uint4 cur = v[q];
  bool run = true;
  while (run && q * 4 < end) {
    const uint4 nx = (q + 1) * 4 < end ? v[q + 1] : make_uint4(0, 0, 0, 0);
    const uint32_t w[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t i = q * 4 + k;
      run = run && !(i >= next && is_start(w[k]));
      const bool on = run && i >= from && i < end && w[k] != 0;
      uint32_t l, nr;
      sub_range(w[k], r, l, nr);
      const int d = on ? __clz(nr) - 16 : 0;
      r = on ? nr << d : r;
      f(on ? l : 0u, d);
    }
    cur = nx;
    ++q;
  }
}

// The range before every piece of a group, the bits each piece shifts out and
// its share of the code value: the sum of its l, each at its bit position,
// streamed through a window of two 16-bit digits.  A piece's first l ends at
// bit 30 of its digits (the most significant first), so that it cannot overflow
// the first digit; n stores shift at most 15 n bits and give n + 4 digits at
// most.
__global__ void __launch_bounds__(kGroup) ranges_kernel(const Lists L, const StreamTile* __restrict__ tile, int nt) {
  __shared__ uint16_t m[kGroup][kClasses];
  __shared__ uint16_t rs[kGroup];
  __shared__ uint32_t half;
  const int t = threadIdx.x;
  const uint32_t c = blockIdx.x * kGroup + t;
  const uint4* src = reinterpret_cast<const uint4*>(L.map + (size_t)blockIdx.x * kGroup * kClasses);
  uint4* dst = reinterpret_cast<uint4*>(&m[0][0]);
  for (int i = t; i < kGroup * kClasses / 8; i += kGroup) dst[i] = src[i];
  __syncthreads();
  if (t == 0) {
    uint32_t r = L.gr[blockIdx.x];
    for (int k = 0; k < kGroup; ++k) {
      rs[k] = (uint16_t)r;
      const uint32_t v = m[k][(r >> 8) - kClasses];
      r = v ? v : r;
    }
  }
  __syncthreads();
  const StreamTile ti = tile[tile_of(tile, nt, blockIdx.x * kGroupTokens)];
  const uint32_t from = L.spos[c];
  uint32_t bits = 0;
  if (from != kNoStart) {
    uint32_t* dg = L.loc + from + 4 * c;
    uint32_t q = 1;
    int b = 15;  // bits of digit q in the window
    unsigned long long acc = 0;
    run_piece(L.st, from, (c + 1) * kChunk, ti.base + ti.ntok, rs[t], [&](uint32_t l, int d) {
      bits += d;
      acc = (acc + l) << d;
      b += d;
      const bool out = b > 16;
      if (out) dg[q - 1] = (uint32_t)(acc >> b);
      acc = out ? acc & ((1ull << b) - 1) : acc;
      q += out;
      b -= out ? 16 : 0;
    });
    dg[q - 1] = (uint32_t)(acc >> b);
    dg[q] = (uint32_t)(acc & ((1ull << b) - 1)) << (16 - b);
    L.nd[c] = q + 1;
  }
  uint32_t s = bits;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t q = __shfl_up_sync(~0u, s, o);
    if ((t & 31) >= o) s += q;
  }
  if (t == 31) half = s;
  __syncthreads();
  if (t >= 32) s += half;
  L.cd[c] = s - bits;
  if (t == kGroup - 1) L.gd[blockIdx.x] = s;
}

// The bits before every group of its tile, and where the tiles' digits and
// bytes go.
__global__ void __launch_bounds__(1024) shift_scan_kernel(const Lists L, const StreamPlan p, const StreamGroup grp) {
  __shared__ uint32_t ws[32];
  uint32_t digit = 0, byte = 0;
  for (int k = grp.tile0; k < grp.tile0 + grp.ntiles; ++k) {
    const StreamTile ti = p.tile[k];
    const int g0 = (int)(ti.base / kGroupTokens), n = (int)((ti.ntok + kGroupTokens - 1) / kGroupTokens);
    uint32_t carry = 0;
    for (int b = 0; b < n; b += 1024) {
      const int i = b + (int)threadIdx.x;
      uint32_t total;
      const uint32_t ex = block_scan_1024(i < n ? L.gd[g0 + i] : 0, ws, &total);
      if (i < n) L.gd[g0 + i] = carry + ex;
      carry += total;
    }
    const uint32_t nbytes = (carry + 8) >> 3;
    if (threadIdx.x == 0) {
      p.tile[k].shift = carry;
      p.tile[k].digit = digit;
      p.tile[k].byte = byte;
      p.tile[k].nbytes = nbytes;
    }
    digit += ((carry + 30) >> 4) + 2;
    byte += nbytes;
  }
  if (threadIdx.x == 0) {
    p.total->digits = digit;
    p.total->bytes = byte;
  }
}

// The code value after all stores, its units bit at digit bit 15 of digit 0
// and the payload from digit 1 on: a warp adds each piece's digits, shifted by
// the bits shifted out before it.
__global__ void __launch_bounds__(128) digits_kernel(const Lists L, const StreamTile* __restrict__ tile, int nt,
                                                     uint32_t* __restrict__ digits) {
  const uint32_t c = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const StreamTile ti = tile[tile_of(tile, nt, c * kChunk)];
  uint32_t* dg = digits + ti.digit;
  if (c * kChunk == ti.base && lane == 0) {  // done(): the sum is rounded up before its last bits are dropped
    const uint32_t at = ti.shift + 30, v = 0x3FFFu << (15 - (at & 15));
    atomicAdd(&dg[at >> 4], v & 0xffff);
    atomicAdd(&dg[(at >> 4) - 1], v >> 16);
  }
  const uint32_t from = L.spos[c];
  if (from == kNoStart) return;
  const uint32_t* loc = L.loc + from + 4 * c;
  const uint32_t n = L.nd[c], before = L.gd[c / kGroup] + L.cd[c], sh = before & 15;
  dg += before >> 4;
  for (uint32_t i = lane; i <= n; i += 32) {
    const uint32_t v = (i < n ? loc[i] >> sh : 0) + (i ? (loc[i - 1] << (16 - sh)) & 0xffff : 0);
    if (v) atomicAdd(&dg[i], v);
  }
}

// Two payload bytes per thread: digit i with the overflow of the digit below
// it and the carry from further below, found by looking down past digits of
// all ones.
__global__ void __launch_bounds__(256) bytes_kernel(const StreamTile* __restrict__ tile,
                                                    const uint32_t* __restrict__ digits, uint8_t* __restrict__ out) {
  const StreamTile ti = tile[blockIdx.y];
  const uint32_t i = blockIdx.x * 256 + threadIdx.x + 1;
  const uint32_t k = 2 * (i - 1);
  if (k >= ti.nbytes) return;
  const uint32_t* dg = digits + ti.digit;
  const uint32_t last = (ti.shift + 30) >> 4;  // digit last + 1 is zero
  auto part = [&](uint32_t j) { return (dg[j] & 0xffff) + (dg[j + 1] >> 16); };
  uint32_t carry = 0;
  for (uint32_t j = i + 1; j <= last; ++j) {
    const uint32_t x = part(j);
    if (x != 0xffff) {
      carry = x > 0xffff;
      break;
    }
  }
  uint32_t x = (part(i) + carry) & 0xffff;
  // done(): bit `shift` + 16 is set, what follows it is not coded
  const uint32_t e = ti.shift + 16;
  if (i == e >> 4) {
    const uint32_t bit = 0x8000u >> (e & 15);
    x = (x & ~(2 * bit - 1)) | bit;
  } else if (i > e >> 4) {
    x = 0;
  }
  out[ti.byte + k] = (uint8_t)(x >> 8);
  if (k + 1 < ti.nbytes) out[ti.byte + k + 1] = (uint8_t)x;
}

// ---------------------------------------------------------------------------

size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

struct Carve {
  uint8_t* base;
  size_t at = 0;
  template <class T>
  T* take(size_t n) {
    T* p = reinterpret_cast<T*>(base + at);
    at += up256(n * sizeof(T));
    return p;
  }
};

size_t carve_plan(const StreamGeom& g, void* mem, StreamPlan* p) {
  const size_t nb = (size_t)g.nbx * g.nby, nt = (size_t)g.tcols * g.trows;
  Carve c{static_cast<uint8_t*>(mem)};
  p->total = c.take<StreamTotals>(1);
  p->tile = c.take<StreamTile>(nt);
  p->delta = c.take<uint32_t>(nt);
  p->cdef_at = c.take<uint32_t>((size_t)g.sb_cols * g.sb_rows);
  p->off = c.take<uint32_t>(3 * nb);
  p->bpre = c.take<uint32_t>((3 * nb + kScanBlock - 1) / kScanBlock);
  p->res = c.take<uint8_t>(3 * nb);
  return c.at;
}

size_t carve_lists(const StreamGeom& g, uint32_t padded, void* mem, Lists* L) {
  const size_t n = padded, nt = (size_t)g.tcols * g.trows, nc = n / kChunk, ng = n / kGroupTokens;
  Carve c{static_cast<uint8_t*>(mem)};
  L->st = c.take<uint32_t>(n);
  L->idx = c.take<uint32_t>(n);
  L->tok = c.take<uint16_t>(n);
  L->sym = c.take<uint8_t>(n);
  L->hist = c.take<uint32_t>(n / kPart * 256);
  L->list = c.take<uint2>(nt * 256);
  L->seg0 = c.take<uint32_t>(nt * 256);
  const size_t ns = n / kSeg + 256 * nt;
  L->seg_a = c.take<uint16_t>(ns * 16);
  L->seg_b = c.take<uint16_t>(ns * 16);
  L->seg_m = c.take<uint16_t>(ns);
  L->map = c.take<uint16_t>(nc * kClasses);
  L->spos = c.take<uint32_t>(nc);
  L->gmap = c.take<uint16_t>(ng * kClasses);
  L->gr = c.take<uint16_t>(ng);
  L->cd = c.take<uint32_t>(nc);
  L->nd = c.take<uint32_t>(nc);
  L->loc = c.take<uint32_t>(n + 4 * nc);
  L->gd = c.take<uint32_t>(ng);
  return c.at;
}

int status() { return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE; }

template <bool WRITE>
void launch_units(const StreamGeom& g, const StreamInput& in, const StreamPlan& p, const StreamGroup& grp,
                  uint16_t* tokens, cudaStream_t st) {
  const unsigned n = (unsigned)(((size_t)g.nbx * g.nby + 15) / 16);
  units_kernel<8, true, WRITE><<<n, 128, 0, st>>>(g, in, p, grp, tokens);
  if (g.sub)
    units_kernel<4, false, WRITE><<<dim3(n, 2), 128, 0, st>>>(g, in, p, grp, tokens);
  else
    units_kernel<8, false, WRITE><<<dim3(n, 2), 128, 0, st>>>(g, in, p, grp, tokens);
}

uint16_t g_cdfs[8][256 * kCdfEntries];  // by quantiser context and chroma transform size
std::once_flag g_cdfs_once;

void build_cdf_tables();

}  // namespace

extern "C" {
int mt_cdf_layout(mt_cdf_slot_layout* out);
int mt_cdfs_default(int32_t qctx, uint16_t* data, size_t data_cap, uint32_t* offsets, uint16_t* lens,
                    int32_t slots_cap, size_t* data_len, int32_t* nslots);
}

namespace mth {

size_t stream_plan_bytes(const StreamGeom& g) {
  StreamPlan p;
  return carve_plan(g, nullptr, &p);
}
size_t stream_token_bytes(const StreamGeom& g, uint32_t padded) {
  Lists L;
  return carve_lists(g, padded, nullptr, &L);
}
size_t stream_digit_bytes(const StreamTotals& t) { return up256((size_t)t.digits * 4) + t.bytes; }

size_t stream_cdf_bytes() { return sizeof(g_cdfs[0]); }
const void* stream_cdf_table(int qctx, int sub) {
  std::call_once(g_cdfs_once, build_cdf_tables);
  return g_cdfs[2 * qctx + (sub ? 1 : 0)];
}

int stream_count(const StreamGeom& g, const StreamInput& in, void* plan, cudaStream_t st, int* launches) {
  StreamPlan p;
  carve_plan(g, plan, &p);
  launch_units<false>(g, in, p, StreamGroup{}, nullptr, st);
  *launches += 2;
  return stream_place(g, plan, st, launches);
}

int stream_place(const StreamGeom& g, void* plan, cudaStream_t st, int* launches) {
  StreamPlan p;
  carve_plan(g, plan, &p);
  const int n = 3 * g.nbx * g.nby, nblk = (n + kScanBlock - 1) / kScanBlock;
  scan_local_kernel<<<nblk, 1024, 0, st>>>(p.off, n, p.bpre);
  scan_blocks_kernel<<<1, 1024, 0, st>>>(g, p, nblk);
  *launches += 2;
  return status();
}

uint32_t* stream_counts(const StreamGeom& g, void* plan) {
  StreamPlan p;
  carve_plan(g, plan, &p);
  return p.off;
}
const StreamTotals* stream_totals(const StreamGeom& g, void* plan) {
  StreamPlan p;
  carve_plan(g, plan, &p);
  return p.total;
}
const StreamTile* stream_tiles(const StreamGeom& g, void* plan) {
  StreamPlan p;
  carve_plan(g, plan, &p);
  return p.tile;
}

StreamGroup stream_group(const StreamTile* tiles, int ntiles, int tile0) {
  StreamGroup grp;
  grp.tile0 = tile0;
  for (int k = tile0; k < ntiles && (k == tile0 || tiles[k].base != 0); ++k) {
    grp.ntiles += 1;
    grp.tokens = tiles[k].base + (tiles[k].ntok + kGroupTokens - 1) / kGroupTokens * kGroupTokens;
  }
  return grp;
}

int stream_trace(const StreamGeom& g, const StreamInput& in, void* plan, void* tokens, const StreamGroup& grp,
                 const void* d_cdfs, bool updating, cudaStream_t st, int* launches) {
  StreamPlan p;
  Lists L;
  carve_plan(g, plan, &p);
  carve_lists(g, grp.tokens, tokens, &L);
  const StreamTile* tile = p.tile + grp.tile0;
  const int nt = grp.ntiles;
  launch_units<true>(g, in, p, grp, L.tok, st);
  hist_kernel<<<grp.tokens / kPart / 4, 128, 0, st>>>(L, tile, nt);
  part_scan_kernel<<<nt, 1024, 0, st>>>(L, tile);
  scatter_kernel<<<grp.tokens / kPart / 4, 128, 0, st>>>(L, tile, nt);
  const uint16_t* cdfs = static_cast<const uint16_t*>(d_cdfs);
  const unsigned ns = grp.tokens / kSeg + 256 * nt;
  first_kernel<<<ns / 4, 128, 0, st>>>(L, tile, nt, cdfs, updating);
  trace_kernel<<<ns / 4, 128, 0, st>>>(L, tile, nt, cdfs, updating);
  fix_kernel<<<dim3(kIds, nt), 256, 0, st>>>(L, tile, cdfs, updating);
  *launches += 8;
  return status();
}

int stream_ranges(const StreamGeom& g, void* plan, void* tokens, const StreamGroup& grp, const int32_t* bits,
                  const uint8_t* grid, cudaStream_t st, int* launches) {
  StreamPlan p;
  Lists L;
  carve_plan(g, plan, &p);
  carve_lists(g, grp.tokens, tokens, &L);
  const StreamTile* tile = p.tile + grp.tile0;
  const int nt = grp.ntiles, nsb = g.sb_cols * g.sb_rows;
  if (bits) {
    cdef_fill_kernel<<<(nsb + 127) / 128, 128, 0, st>>>(g, p, grp, L.st, bits, grid, nsb);
    *launches += 1;
  }
  map_kernel<<<grp.tokens / kChunk / 4, 128, 0, st>>>(L, tile, nt);
  compose_kernel<<<grp.tokens / kGroupTokens, kClasses, 0, st>>>(L);
  walk_kernel<<<nt, 256, 0, st>>>(L, tile);
  ranges_kernel<<<grp.tokens / kGroupTokens, kGroup, 0, st>>>(L, tile, nt);
  shift_scan_kernel<<<1, 1024, 0, st>>>(L, p, grp);
  *launches += 5;
  return status();
}

const uint8_t* stream_bytes(const StreamGeom& g, void* plan, void* tokens, const StreamGroup& grp, void* digits,
                            const StreamTotals& t, uint32_t max_bytes, cudaStream_t st, int* launches) {
  StreamPlan p;
  Lists L;
  carve_plan(g, plan, &p);
  carve_lists(g, grp.tokens, tokens, &L);
  const StreamTile* tile = p.tile + grp.tile0;
  uint32_t* dg = static_cast<uint32_t*>(digits);
  uint8_t* out = static_cast<uint8_t*>(digits) + up256((size_t)t.digits * 4);
  if (cudaMemsetAsync(dg, 0, (size_t)t.digits * 4, st) != cudaSuccess) return nullptr;
  digits_kernel<<<grp.tokens / kChunk / 4, 128, 0, st>>>(L, tile, grp.ntiles, dg);
  bytes_kernel<<<dim3((max_bytes + 511) / 512, grp.ntiles), 256, 0, st>>>(tile, dg, out);
  *launches += 2;
  return status() == MT_OK ? out : nullptr;
}

}  // namespace mth

namespace {

// A CDF's inverse values in entries 0.., its symbol count in entry 15.
void build_cdf_tables() {
  mt_cdf_slot_layout S;
  mt_cdf_layout(&S);
  for (int q = 0; q < 4; ++q) {
    size_t len = 0;
    int32_t ns = 0;
    mt_cdfs_default(q, nullptr, 0, nullptr, nullptr, 0, &len, &ns);
    std::vector<uint16_t> data(len), lens((size_t)ns);
    std::vector<uint32_t> offs((size_t)ns);
    mt_cdfs_default(q, data.data(), len, offs.data(), lens.data(), ns, &len, &ns);
    for (int sub = 0; sub < 2; ++sub) {
      auto put = [&](int id, int slot, int n) {
        for (int k = 0; k < n; ++k) {
          uint16_t* d = g_cdfs[2 * q + sub] + (size_t)(id + k) * kCdfEntries;
          const size_t s = (size_t)(slot + k);
          memcpy(d, data.data() + offs[s], (size_t)(lens[s] - 1) * 2);
          d[kCdfEntries - 1] = lens[s];
        }
      };
      put(kPartBl8, S.part_bl8, 1);
      put(kPartSplit, S.part_split, 12);
      put(kSkip, S.skip, 1);
      put(kKfY, S.kf_y, 25);
      put(kAngle, S.angle_delta, 8);
      put(kUvMode, S.uv_mode + 13, 13);
      put(kPalY, S.palette_y_mode, 1);
      put(kPalUv, S.palette_uv_mode, 1);
      put(kFilterIntra, S.filter_intra + 3, 1);
      put(kTxsz, S.txsz, 3);
      put(kTxtp, S.txtp8, 13);
      const int cc = sub ? 0 : 1;  // chroma: TX_4X4 or TX_8X8
      put(kTxbSkip, S.txb_skip[1], 1);
      put(kTxbSkip + 1, S.txb_skip[cc] + 7, 3);
      for (int p = 0; p < 2; ++p) {
        const int c = p ? cc : 1;
        put(kBase + 41 * p, S.base_tok[c][p], 41);
        put(kBr + 21 * p, S.br_tok[c][p], 21);
        put(kEobBase + 4 * p, S.eob_base[c][p], 4);
        put(kEobHi + 11 * p, S.eob_hi[c][p], 11);
        put(kDcSign + 3 * p, S.dc_sign[p], 3);
      }
      put(kEobBin, S.eob_bin + 4, 1);                     // 64 luma
      put(kEobBin + 1, S.eob_bin + 6, 1);                 // 64 luma, 1-D classes
      put(kEobBin + 2, S.eob_bin + (sub ? 0 : 8), 1);     // 16 or 64 chroma
    }
  }
}

}  // namespace
