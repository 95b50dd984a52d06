// The encoder's 8x8 candidate chain (chain8.cuh) with EIGHT lanes per candidate
// (an octet), for a launch whose latency, not its throughput, bounds the run:
// the wavefront of the encoder, where a few dozen blocks per dependency level
// are all the work there is.
//
// The four octets of a warp run one transform type, so the warp never splits:
// every sync is the whole warp's and every loop has a warp-wide bound.  Lane j
// of an octet holds a row or a column of the block in registers from the
// residual to the cost; shared memory carries the two transposes, the terms of
// the ordered float sums, and tables.
//
// Same arithmetic, same order, same results as the one-thread chain (bit for
// bit):
//   * the trellis round-down decisions are per coefficient (the reference's
//     AVX2 chunks decide each position from the chunk's starting values, so
//     only the chunk's "any level > 63" flag is shared);
//   * the float chains that have an order (the trellis suffix sums of the
//     zeroing distortion, its running prefix cost, the rate walk's sum) keep
//     it: their terms are computed by all lanes and added by one lane in the
//     reference's order, positions outside a chain's range adding an exact +0;
//     integer sums (SATD, counts) are reduced across lanes in any order.
#pragma once
#include <stdint.h>

#include "chain4.cuh"
#include "chain8.cuh"

namespace mtd {

// Shared-memory working set of one octet.  t: transposes (stride 9, or 5 at
// 4x4).  Trellis: sr[4 + k] = the suffix sum from scan index 63 - k (sr[3] = 0
// is the empty sum), b / r the prefix terms.  Rate: b, r and t hold the walk's
// three terms, at 63 - scan index.  296 words: the octets of a warp start 8
// banks apart.
struct OctBuf {
  int32_t t[72];
  float sr[68];
  float b[64];
  float r[64];
  float pad[28];
};
static_assert(sizeof(OctBuf) / 4 % 32 == 8 && sizeof(OctBuf) % 16 == 0, "octet bank offset");

// What one plane of an image needs beside its quantiser: per coefficient the
// forward QM scale and the dequantisation step (rc = 8 x + y, or 4 x + y), per
// level and per scan index lambda times the static rate and the end-of-block
// cost, and the reciprocals of the two IDTX divisions.
struct CoopPlane {
  float qs[64];
  int32_t step[64];
  float lrate[64];  // lambda * rate(level)
  float lsig[64];   // lambda * (0.9 bin + extra + 2) of an end of block at scan index e
  float lambda;     // 0: no trellis
  float dq2, aq2;
  uint32_t idiv[2];  // 2^32 / dc_q, 2^32 / ac_q, rounded up
  int has_qm;
  mt_quant q;

  // Thread t of 64: qm the plane's inverse QM row (NULL: flat), n its samples.
  __device__ __forceinline__ void stage(int t, const mt_quant& quant, float lam, const uint8_t* qm, int n) {
    const int w = qm && t < n ? qm[t] : 32;
    qs[t] = fwd_qm_scale(w);
    const int32_t base = t == 0 ? quant.dc_q : quant.ac_q;
    step[t] = qm ? (base * w + 16) >> 5 : base;
    lrate[t] = __fmul_rn(lam, kCoefRateLut[t]);
    const int bin = t < 2 ? t : 32 - __clz(t), extra = bin > 1 ? bin - 2 : 0;
    lsig[t] = __fmul_rn(lam, __fadd_rn(__fmul_rn((float)bin, 0.9f), __fadd_rn((float)extra, 2.0f)));
    if (t == 0) {
      lambda = lam;
      dq2 = __fmul_rn((float)quant.dc_q, (float)quant.dc_q);
      aq2 = __fmul_rn((float)quant.ac_q, (float)quant.ac_q);
      idiv[0] = 0xffffffffu / (uint32_t)quant.dc_q + 1u;
      idiv[1] = 0xffffffffu / (uint32_t)quant.ac_q + 1u;
      has_qm = qm != nullptr;
      q = quant;
    }
  }
};

// Inverse scans by row: row[y][x] is the scan index of (x, y).
struct CoopScan {
  alignas(8) uint8_t row8[8][8];
  uint8_t row4[4][4];
  __device__ __forceinline__ void stage(int t) {  // thread t of 64
    row8[t & 7][t >> 3] = kIScan8[t];
    if (t < 16) {
      const int rc = kScan4[t];
      row4[rc & 3][rc >> 2] = (uint8_t)t;
    }
  }
};

// A group of W lanes of a warp (W = 8 an octet; 4 for the 4x4 chroma block).
template <int W>
struct Coop {
  int j;
  __device__ __forceinline__ Coop() : j(threadIdx.x & (W - 1)) {}
  __device__ __forceinline__ int max(int v) const {
#pragma unroll
    for (int s = W / 2; s; s >>= 1) v = ::max(v, __shfl_xor_sync(0xffffffffu, v, s));
    return v;
  }
  __device__ __forceinline__ uint32_t sum(uint32_t v) const {
#pragma unroll
    for (int s = W / 2; s; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    return v;
  }
};

// Eight int16 of a row or column as one 16-byte load.
__device__ __forceinline__ void load8(const int16_t* p, int32_t* v) {
  const int4 w = *reinterpret_cast<const int4*>(p);
  const int32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    v[2 * k] = (int16_t)(x[k] & 0xffff);
    v[2 * k + 1] = x[k] >> 16;
  }
}

// The transpose of a W x W block: lane j hands in one line and gets the line
// across it (bank-conflict free over the warp's groups).
template <int W>
__device__ __forceinline__ void coop_transpose(int32_t* v, int32_t* t, int j) {
#pragma unroll
  for (int k = 0; k < W; k++) t[j * (W + 1) + k] = v[k];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < W; k++) v[k] = t[k * (W + 1) + j];
  __syncwarp();
}

// Quantisation of 8-bit residuals' coefficients: every |coefficient| is below
// 2^15 and every multiplier at most 65536 / 4, so the products stay in 32 bits.
__device__ __forceinline__ int32_t quant_half32(int32_t d, int32_t m) {
  const int32_t p = d * m, l = (abs(p) + 32768) >> 16;
  return p < 0 ? -l : l;
}

// Forward transform and quantisation of type TX from the residual (col / row:
// columns and rows of eight int16): lane j gets row j of the levels (c) and of
// the targets' magnitudes (at).
__device__ __forceinline__ void coop8_fwd(int TX, const int16_t* col, const int16_t* row, const CoopPlane& P, int32_t* c,
                                          float* at, OctBuf& o, const Coop<8>& g) {
  const int j = g.j;
  int32_t v[8];
  if (TX == MT_TX_IDTX) {
    load8(row + j * 8, v);
#pragma unroll
    for (int x = 0; x < 8; x++) {
      const bool dc = x == 0 && j == 0;
      const int32_t qd = dc ? P.q.dc_q : P.q.ac_q, num = v[x] * 8;
      at[x] = fabsf(__fdiv_rn((float)num, (float)qd));
      const uint32_t am = (uint32_t)abs(num);
      // (am + qd / 2) / qd: exact for am + qd / 2 < 2^16 and qd < 2^12
      const int32_t level = (int32_t)__umulhi(am + (uint32_t)(qd >> 1), dc ? P.idiv[0] : P.idiv[1]);
      c[x] = (int32_t)am < qd ? 0 : (num < 0 ? -level : level);
    }
    return;
  }
  const bool one_d = TX == MT_TX_V_DCT || TX == MT_TX_H_DCT;
  if (TX == MT_TX_H_DCT) {
    load8(row + j * 8, v);
  } else {
    load8(col + j * 8, v);
    if (TX == MT_TX_ADST_ADST || TX == MT_TX_ADST_DCT) fadst8(v); else fdct8(v);
    coop_transpose<8>(v, o.t, j);
  }
  if (TX == MT_TX_ADST_ADST || TX == MT_TX_DCT_ADST) fadst8(v);
  else if (TX != MT_TX_V_DCT) fdct8(v);
#pragma unroll
  for (int x = 0; x < 8; x++) {
    const int32_t m = x == 0 && j == 0 ? P.q.q_mult_dc : P.q.q_mult_ac;
    if (one_d) {
      const int32_t p = v[x] * 2 * m, l = (abs(p) + 32768) >> 16;
      at[x] = fabsf(__fmul_rn((float)p, 1.0f / 65536.0f));
      c[x] = abs(p) < 65536 ? 0 : (p < 0 ? -l : l);
    } else {
      float tf = __fmul_rn(__fmul_rn((float)v[x], (float)m), 1.0f / 65536.0f);
      if (P.has_qm) {  // apply_qm
        tf = __fmul_rn(tf, P.qs[x * 8 + j]);
        const float tr = truncf(tf);
        const float st = fabsf(__fsub_rn(tf, tr)) >= 0.5f ? copysignf(1.0f, tf) : 0.0f;
        c[x] = (int32_t)__fadd_rn(tr, st);
      } else {
        c[x] = quant_half32(v[x], m);
      }
      at[x] = fabsf(tf);
    }
  }
}

// The 4x4 DCT_DCT of the same form (multipliers doubled, src/dct.rs:3076-3100).
__device__ __forceinline__ void coop4_fwd(int32_t* v, const CoopPlane& P, int32_t* c, float* at, OctBuf& o,
                                          const Coop<4>& g) {
  const int j = g.j;
  fdct4v(v);
  coop_transpose<4>(v, o.t, j);
  fdct4v(v);
#pragma unroll
  for (int x = 0; x < 4; x++) {
    const int32_t m = 2 * (x == 0 && j == 0 ? P.q.q_mult_dc : P.q.q_mult_ac);
    float tf = __fmul_rn(__fmul_rn((float)v[x], (float)m), 1.0f / 65536.0f);
    if (P.has_qm) {
      tf = __fmul_rn(tf, P.qs[x * 4 + j]);
      const float tr = truncf(tf);
      const float st = fabsf(__fsub_rn(tf, tr)) >= 0.5f ? copysignf(1.0f, tf) : 0.0f;
      c[x] = (int32_t)__fadd_rn(tr, st);
    } else {
      c[x] = quant_half32(v[x], m);
    }
    at[x] = fabsf(tf);
  }
}

// trellis_optimize (trellis8 / trellis4) over row-wise levels c and target
// magnitudes at, e the scan indexes.  Returns the final end of block (-1: all
// zero).
template <int W>
__device__ __forceinline__ int coop_trellis(int32_t* c, const float* at, const int* e, const CoopPlane& P, OctBuf& o,
                                            const Coop<W>& g) {
  constexpr unsigned kAll = 0xffffffffu;
  const int j = g.j;
  int e1 = 0;
#pragma unroll
  for (int x = 0; x < W; x++)
    if (c[x] != 0) e1 = ::max(e1, e[x] + 1);
  const int m = g.max(e1);
  if (!(P.lambda > 0.0f)) return m - 1;
  const int M8 = ((int)__reduce_max_sync(kAll, (unsigned)m) + 7) & ~7;
  if (M8 == 0) return -1;
  const int full8 = m & ~7, chunked = full8 + ((m - full8) >= 4 ? 4 : 0);
  // step A.  The reference decides each position of a chunk (of eight, then one
  // of four) from the chunk's starting values, in the AVX2 FMA form unless the
  // chunk holds a level above 63; then, and in the scalar tail, the plain form.
  unsigned bigb = 0;  // bit k: chunk k holds one
#pragma unroll
  for (int x = 0; x < W; x++)
    if (abs(c[x]) > 63 && e[x] < chunked) bigb |= 1u << (e[x] >> 3);
  if (__any_sync(kAll, bigb != 0)) {
#pragma unroll
    for (int s = W / 2; s; s >>= 1) bigb |= __shfl_xor_sync(kAll, bigb, s);
  }
#pragma unroll
  for (int x = 0; x < W; x++) {
    const float q2 = x == 0 && j == 0 ? P.dq2 : P.aq2;
    const int32_t l = abs(c[x]), ld = ::max(l - 1, 0);
    const float el = __fsub_rn(at[x], (float)l), ed = __fsub_rn(at[x], (float)ld);
    const float rl = l < 64 ? P.lrate[l] : __fmul_rn(P.lambda, coef_rate_bits((uint32_t)l));
    const float rd = ld < 64 ? P.lrate[ld] : __fmul_rn(P.lambda, coef_rate_bits((uint32_t)ld));
    const bool fma_form = e[x] < chunked && !((bigb >> (e[x] >> 3)) & 1u);
    const float l2 = __fmul_rn(el, el), d2 = __fmul_rn(ed, ed);
    const float cl = fma_form ? __fmaf_rn(q2, l2, rl) : __fadd_rn(__fmul_rn(q2, l2), rl);
    const float cd = fma_form ? __fmaf_rn(q2, d2, rd) : __fadd_rn(__fmul_rn(q2, d2), rd);
    if (l != 0 && cd < cl) c[x] = c[x] < 0 ? c[x] + 1 : c[x] - 1;
    // the terms of the ordered sums, +0 past the end of block: S = q2 at^2 (the
    // zeroing distortion), B = q2 (at - l)^2, R = lambda rate(l)
    const int32_t l1 = abs(c[x]);
    const float ec = __fsub_rn(at[x], (float)l1);
    const bool in = e[x] < m;
    o.sr[67 - e[x]] = in ? __fmul_rn(q2, __fmul_rn(at[x], at[x])) : 0.0f;
    o.b[e[x]] = in ? __fmul_rn(q2, __fmul_rn(ec, ec)) : 0.0f;
    o.r[e[x]] = in ? (l1 < 64 ? P.lrate[l1] : __fmul_rn(P.lambda, coef_rate_bits((uint32_t)l1))) : 0.0f;
  }
  if (j == 0) o.sr[3] = 0.0f;
  if (W == 4 && j == 0) o.sr[67 - 16] = 0.0f;  // S(16): the scan ends there
  __syncwarp();
  // Lane 0: the suffix sums right to left (acc += S; S = acc).  Lane 1: the
  // prefix cost left to right (b = pre + B; B = b; pre = b + R).
  if (j < 2) {
    float* arr = j == 0 ? o.sr + 4 + (64 - M8) : o.b;
    float acc = 0.0f;
#pragma unroll 1
    for (int s = 0; s < M8; s += 8) {
      float v[8], r[8];
#pragma unroll
      for (int u = 0; u < 8; u += 4) {
        const float4 a = *reinterpret_cast<const float4*>(arr + s + u);
        float4 q = *reinterpret_cast<const float4*>(o.r + s + u);
        if (j == 0) q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        v[u] = a.x, v[u + 1] = a.y, v[u + 2] = a.z, v[u + 3] = a.w;
        r[u] = q.x, r[u + 1] = q.y, r[u + 2] = q.z, r[u + 3] = q.w;
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        v[u] = __fadd_rn(acc, v[u]);
        acc = __fadd_rn(v[u], r[u]);
      }
#pragma unroll
      for (int u = 0; u < 8; u += 4)
        *reinterpret_cast<float4*>(arr + s + u) = make_float4(v[u], v[u + 1], v[u + 2], v[u + 3]);
    }
  }
  __syncwarp();
  // candidate ends: the lowest cost, the first position on ties
  float best = __int_as_float(0x7f800000);
  int best_e = 64;
#pragma unroll
  for (int x = 0; x < W; x++) {
    if (c[x] != 0) {
      const float cst = __fadd_rn(__fadd_rn(o.b[e[x]], P.lsig[e[x]]), o.sr[66 - e[x]]);
      if (cst < best || (cst == best && e[x] < best_e)) {
        best = cst;
        best_e = e[x];
      }
    }
  }
#pragma unroll
  for (int s = W / 2; s; s >>= 1) {
    const float ob = __shfl_xor_sync(kAll, best, s);
    const int oe = __shfl_xor_sync(kAll, best_e, s);
    if (ob < best || (ob == best && oe < best_e)) {
      best = ob;
      best_e = oe;
    }
  }
  const float skip = __fadd_rn(o.sr[67], P.lambda);
  const int keep = (best_e == 64 || skip < best) ? 0 : best_e + 1;
#pragma unroll
  for (int x = 0; x < W; x++)
    if (e[x] >= keep) c[x] = 0;
  __syncwarp();
  return keep - 1;
}

// Dequantised row j of c (step: per coefficient, or the flat step).
template <int W>
__device__ __forceinline__ void coop_dequant(const int32_t* c, bool flat, const CoopPlane& P, int32_t* v, int j) {
#pragma unroll
  for (int x = 0; x < W; x++) {
    const int32_t l = c[x];
    const int32_t step = flat ? (x == 0 && j == 0 ? P.q.dc_q : P.q.ac_q) : P.step[x * W + j];
    int32_t mag = (int32_t)(((uint32_t)abs(l) * (uint32_t)step) & 0xffffffu);
    mag = ::min(mag, P.q.cf_max + (l < 0 ? 1 : 0));
    v[x] = l < 0 ? -mag : mag;
  }
}

// Dequantisation + inverse transform of type TX: lane j gets column j of the
// inverse residual.
__device__ __forceinline__ void coop8_inv(int TX, const int32_t* c, const CoopPlane& P, int32_t* v, OctBuf& o,
                                          const Coop<8>& g) {
  const mt_quant& q = P.q;
  coop_dequant<8>(c, TX == MT_TX_IDTX || TX == MT_TX_V_DCT || TX == MT_TX_H_DCT, P, v, g.j);
  if (TX == MT_TX_IDTX || TX == MT_TX_V_DCT) {
#pragma unroll
    for (int x = 0; x < 8; x++) v[x] *= 2;
  } else if (TX == MT_TX_ADST_ADST || TX == MT_TX_DCT_ADST) {
    iadst8s(v, 1, q.rmin, q.rmax);
  } else {
    idct8s(v, 1, q.rmin, q.rmax);
  }
#pragma unroll
  for (int x = 0; x < 8; x++) v[x] = clampi((v[x] + 1) >> 1, q.cmin, q.cmax);
  coop_transpose<8>(v, o.t, g.j);
  if (TX == MT_TX_IDTX || TX == MT_TX_H_DCT) {
#pragma unroll
    for (int y = 0; y < 8; y++) v[y] *= 2;
  } else if (TX == MT_TX_ADST_ADST || TX == MT_TX_ADST_DCT) {
    iadst8s(v, 1, q.cmin, q.cmax);
  } else {
    idct8s(v, 1, q.cmin, q.cmax);
  }
#pragma unroll
  for (int y = 0; y < 8; y++) v[y] = (v[y] + 8) >> 4;
}
__device__ __forceinline__ void coop4_inv(const int32_t* c, const CoopPlane& P, int32_t* v, OctBuf& o,
                                          const Coop<4>& g) {
  const mt_quant& q = P.q;
  coop_dequant<4>(c, false, P, v, g.j);
  idct4s(v, 1, q.rmin, q.rmax);
#pragma unroll
  for (int x = 0; x < 4; x++) v[x] = clampi(v[x], q.cmin, q.cmax);
  coop_transpose<4>(v, o.t, g.j);
  idct4s(v, 1, q.cmin, q.cmax);
#pragma unroll
  for (int y = 0; y < 4; y++) v[y] = (v[y] + 8) >> 4;
}

// satd8 of the error columns d (lane j column j): 4x4 Hadamards, the vertical
// half in registers, the horizontal one over lanes.
__device__ __forceinline__ uint32_t coop8_satd(int32_t* d, const Coop<8>& g) {
  uint32_t satd = 0;
#pragma unroll
  for (int h = 0; h < 8; h += 4) {
    const int32_t a = d[h] + d[h + 2], b = d[h] - d[h + 2], cc = d[h + 1] + d[h + 3], f = d[h + 1] - d[h + 3];
    d[h] = a + cc;
    d[h + 1] = b + f;
    d[h + 2] = b - f;
    d[h + 3] = a - cc;
  }
#pragma unroll
  for (int s = 1; s < 4; s <<= 1) {
    const int32_t sg = g.j & s ? -1 : 1;
#pragma unroll
    for (int k = 0; k < 8; k++) d[k] = __shfl_xor_sync(0xffffffffu, d[k], s) + sg * d[k];
  }
#pragma unroll
  for (int k = 0; k < 8; k++) satd += (uint32_t)abs(d[k]);
  return g.sum(satd);
}

// b + 1 + 1 + ... (n times, one rounding each): inside a binade of [1, 2^23)
// the sums are exact, so each binade takes one addition and one for the step
// across its end.
__device__ __forceinline__ float add_ones(float b, int n) {
  while (n > 0) {
    int s = 0;
    if (b >= 1.0f && b < 8388608.0f) {
      const float top = __int_as_float((__float_as_int(b) & 0x7f800000) + 0x00800000);
      s = ::min((int)ceilf(__fsub_rn(top, b)) - 1, n);
    }
    if (s > 0) {
      b = __fadd_rn(b, (float)s);
      n -= s;
    } else {
      b = __fadd_rn(b, 1.0f);
      n--;
    }
  }
  return b;
}

// rate8 (txb_skip and dc_sign context 0, no skip price) over the octet, lane j
// holding row j of the levels.  The reference's reverse walk has entered
// exactly the later scan positions when it reads a context, and the five
// neighbours of a position inside the block are later ones (past a column's
// end its map holds nothing yet), so contexts come from the final levels: own
// columns from registers, rows j + 1 and j + 2 by shuffles of packed level
// bytes.  Lane 0 returns the bits.
__device__ __forceinline__ float coop8_rate(const int32_t* c, const int* e, int eob, const mt_coef_costs& T, int mode,
                                            int tx, OctBuf& o, const Coop<8>& g) {
  constexpr unsigned kAll = 0xffffffffu;
  const int j = g.j;
  const int E = (int)__reduce_max_sync(kAll, (unsigned)(eob + 1));  // the longest walk of the warp, + 1
  uint32_t lo = 0, hi = 0;  // level bytes of columns 0..3 and 4..7
#pragma unroll
  for (int x = 0; x < 4; x++) {
    lo |= level_byte((uint32_t)abs(c[x])) << (8 * x);
    hi |= level_byte((uint32_t)abs(c[x + 4])) << (8 * x);
  }
  uint32_t lo1 = __shfl_down_sync(kAll, lo, 1, 8), hi1 = __shfl_down_sync(kAll, hi, 1, 8);
  uint32_t lo2 = __shfl_down_sync(kAll, lo, 2, 8), hi2 = __shfl_down_sync(kAll, hi, 2, 8);
  if (j == 7) lo1 = hi1 = 0;
  if (j >= 6) lo2 = hi2 = 0;
  auto at = [](uint32_t l, uint32_t h, int x) -> uint32_t {
    return x > 7 ? 0u : (x < 4 ? (l >> (8 * (x & 3))) & 255u : (h >> (8 * (x & 3))) & 255u);
  };
  const uint32_t dcmag = (at(lo1, hi1, 0) + at(lo, hi, 1) + at(lo1, hi1, 1)) & 63;  // lane 0's: (0,1), (1,0), (1,1)
  float* T1 = o.b;
  float* T2 = o.r;
  float* T3 = reinterpret_cast<float*>(o.t);
  bool any3 = false;
  uint32_t nz = 0, me = 0;
  if (E > 1) {
#pragma unroll
    for (int x = 0; x < 8; x++) {
      const uint32_t m = (uint32_t)abs(c[x]);
      const bool in = e[x] >= 1 && e[x] < eob;
      any3 |= in && m >= 3;
      nz += in && m != 0;
      me |= e[x] == eob ? m : 0u;
    }
    any3 = __any_sync(kAll, any3);
    nz = g.sum(nz);
    me = g.sum(me);
#pragma unroll
    for (int x = 0; x < 8; x++) {
      const uint32_t m = (uint32_t)abs(c[x]);
      const bool in = e[x] >= 1 && e[x] < eob;
      const uint32_t hm = at(lo1, hi1, x) + at(lo, hi, x + 1) + at(lo1, hi1, x + 1);
      const uint32_t mag = hm + at(lo2, hi2, x) + at(lo, hi, x + 2);
      const int d = x + j;
      const int ctx = (d < 2 ? d : (d < 4 ? 6 : 21)) + ::min((int)((mag + 64) >> 7), 4);
      const float t1 = T.base_tok[ctx][::min(m, 3u)];
      T1[63 - e[x]] = in ? t1 : 0.0f;
      if (any3) {
        float t2 = 0.0f, t3 = 0.0f;
        if (in && m >= 3) {
          const uint32_t hmag = hm & 63;
          t2 = T.br_cum[((j | x) > 1 ? 14 : 7) + (hmag > 12 ? 6 : (int)((hmag + 1) >> 1))][::min((int32_t)m - 3, 12)];
          if (m >= 15) t3 = golomb_cost(m - 15);
        }
        T2[63 - e[x]] = t2;
        T3[63 - e[x]] = t3;
      }
    }
  }
  __syncwarp();
  float bits = 0.0f;
  if (j == 0) {
    if (eob < 0) {
      bits = T.txb_skip[0][1];
    } else {
      bits = __fadd_rn(T.txb_skip[0][0], T.txtp[mode][tx]);
      const uint32_t dm = (uint32_t)abs(c[0]);
      const float sign = T.dc_sign[0][c[0] < 0];
      auto hi_tok = [&](uint32_t m, int bc) -> float {
        float h = T.br_cum[bc][::min((int32_t)m - 3, 12)];
        if (m >= 15) h = __fadd_rn(h, golomb_cost(m - 15));
        return h;
      };
      if (eob == 0) {
        bits = __fadd_rn(bits, T.eob_bin[0]);
        bits = __fadd_rn(bits, T.eob_base[0][::min(dm, 3u) - 1]);
        if (dm >= 3) bits = __fadd_rn(bits, hi_tok(dm, 0));
        bits = __fadd_rn(bits, sign);
      } else {
        const int eob_bin = eob < 2 ? eob : 32 - __clz(eob);
        bits = __fadd_rn(bits, T.eob_bin[eob_bin]);
        if (eob_bin > 1) {
          const int nb = eob_bin - 2;
          bits = __fadd_rn(bits, T.eob_hi[eob_bin][(eob >> nb) & 1]);
          bits = __fadd_rn(bits, (float)nb);
        }
        bits = __fadd_rn(bits, T.eob_base[1 + (eob > 8) + (eob > 16)][::min(me, 3u) - 1]);
        // the end of block's br context: 7 inside the first 2 x 2, else 14
        if (me >= 3) bits = __fadd_rn(bits, hi_tok(me, eob == 1 || eob == 2 || eob == 4 ? 7 : 14));
        const int first = 64 - ((E + 7) & ~7);
        if (!any3) {
#pragma unroll 2
          for (int k = first; k < 64; k += 4) {
            const float4 a = *reinterpret_cast<const float4*>(T1 + k);
            bits = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(bits, a.x), a.y), a.z), a.w);
          }
        } else {
#pragma unroll 2
          for (int k = first; k < 64; k += 4) {
            const float4 a = *reinterpret_cast<const float4*>(T1 + k);
            const float4 b = *reinterpret_cast<const float4*>(T2 + k);
            const float4 d = *reinterpret_cast<const float4*>(T3 + k);
            bits = __fadd_rn(__fadd_rn(__fadd_rn(bits, a.x), b.x), d.x);
            bits = __fadd_rn(__fadd_rn(__fadd_rn(bits, a.y), b.y), d.y);
            bits = __fadd_rn(__fadd_rn(__fadd_rn(bits, a.z), b.z), d.z);
            bits = __fadd_rn(__fadd_rn(__fadd_rn(bits, a.w), b.w), d.w);
          }
        }
        bits = __fadd_rn(bits, T.base_tok[0][::min(dm, 3u)]);
        if (dm >= 3) bits = __fadd_rn(bits, hi_tok(dm, dcmag > 12 ? 6 : (int)((dcmag + 1) >> 1)));
        if (dm != 0) bits = __fadd_rn(bits, sign);
        bits = add_ones(bits, 1 + (int)nz);
      }
    }
  }
  __syncwarp();
  return bits;
}

// The block's neighbours as predict_sq_at<8> builds them, at index 2 (logical
// -2 .. 15; -1 the corner): above along the row, left down the column, with
// the fills of unavailable sides.
struct CoopEdges {
  int16_t a[20], l[20];
};

// Scratch of one predicting warp: the filtered and the upsampled edges.
struct CoopPredBuf {
  int32_t fa[20], fl[20], ua[36], ul[36];
};

// One entry of filter_edge (src/intrapred.rs:977-1012) at position o of an
// edge of `size` entries, e logical index 0.
template <typename I>
__device__ __forceinline__ int32_t edge_tap(const I* e, int o, int size, int strength) {
  const int32_t k0 = strength == 3 ? 2 : 0, k1 = strength == 1 ? 4 : (strength == 2 ? 5 : 4),
                k2 = strength == 1 ? 8 : (strength == 2 ? 6 : 4);
  const int last = size - 1;
  const int32_t a = e[::max(o - 1, 0) - 1], b = e[::min(::max(o, 0), last) - 1], c = e[::min(o + 1, last) - 1];
  const int32_t d = e[::min(o + 2, last) - 1], f = e[::min(o + 3, last) - 1];
  return (k0 * a + k1 * b + k2 * c + k1 * d + k0 * f + 8) >> 4;
}

// predict_sq_at<8> of one mode (angle delta 0) by a whole warp: lane l writes
// samples (2 (l >> 3), l & 7) and the one right of it, as the prediction by
// columns (pcol) and the residual against src (by columns) by columns and by
// rows.
__device__ __forceinline__ void coop8_predict(int mode, const CoopEdges& E, bool have_top, bool have_left, bool ft,
                                              const int16_t* src, int16_t* pcol, int16_t* rcol, int16_t* rrow,
                                              CoopPredBuf& B) {
  const int lane = threadIdx.x & 31, y = lane & 7, x0 = (lane >> 3) * 2;
  const int16_t* A = E.a + 2;
  const int16_t* L = E.l + 2;
  int32_t p[2];
  if (mode == MT_DC_PRED) {
    const int32_t s = lane < 8 ? (have_top ? A[lane] : 0) : (lane < 16 && have_left ? L[lane - 8] : 0);
    const int32_t sum = __reduce_add_sync(0xffffffffu, s);
    p[0] = p[1] = (have_top && have_left) ? (8 + sum) >> 4 : ((have_top || have_left) ? (4 + sum) >> 3 : 128);
  } else if (mode == MT_V_PRED) {
    p[0] = A[x0];
    p[1] = A[x0 + 1];
  } else if (mode == MT_H_PRED) {
    p[0] = p[1] = L[y];
  } else if (mode <= MT_D67_PRED) {
    const int angle = mode == MT_D45_PRED ? 45 : mode == MT_D135_PRED ? 135 : mode == MT_D113_PRED ? 113
                    : mode == MT_D157_PRED ? 157 : mode == MT_D203_PRED ? 203 : 67;
    {  // lanes 0..15 filter the above edge, 16..31 the left one
      const bool ab = lane < 16;
      const int o = lane & 15;
      const int n = 9 + ((ab ? angle < 90 : angle > 180) ? 8 : 0);
      const int s = edge_strength(8, 8, ft, angle - (ab ? 90 : 180));
      const int16_t* e = ab ? A : L;
      int32_t* f = (ab ? B.fa : B.fl) + 2;
      f[o] = s && o < n - 1 ? edge_tap(e, o, n, s) : e[o];
      if (o == 0) f[-1] = e[-1];
    }
    __syncwarp();
    const int da = abs(angle - 90), dl = abs(angle - 180);
    const bool up_a = da < 40 && !ft, up_l = dl < 40 && !ft;  // w + h is 16
    const int32_t* a = B.fa + 2;
    const int32_t* l = B.fl + 2;
    if (up_a || up_l) {  // upsample_edge (src/intrapred.rs:1026-1048); one side at most
      const int num = 8 + ((up_a ? angle < 90 : angle > 180) ? 8 : 0);
      const int32_t* f = up_a ? a : l;
      int32_t* u = (up_a ? B.ua : B.ul) + 2;
      if (lane < num) {
        auto in = [&](int k) { return f[(k <= 1 ? 0 : ::min(k - 1, num)) - 1]; };
        const int32_t v = -in(lane) + 9 * in(lane + 1) + 9 * in(lane + 2) - in(lane + 3);
        u[2 * lane - 1] = clampi((v + 8) >> 4, 0, 255);
        u[2 * lane] = in(lane + 2);
        if (lane == 0) u[-2] = f[-1];
      }
      __syncwarp();
      if (up_a) a = u; else l = u;
    }
    if (angle < 90) {
      const int dx = kDrDeriv[angle >> 1], lastb = 15 << up_a;
      const int xpos = dx * (y + 1), shift = ((xpos << up_a) & 0x3f) >> 1;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int b = (xpos >> (6 - up_a)) + ((x0 + k) << up_a);
        p[k] = b < lastb ? (a[b] * (32 - shift) + a[b + 1] * shift + 16) >> 5 : a[lastb];
      }
    } else if (angle > 180) {
      const int dy = kDrDeriv[(270 - angle) >> 1], lastb = 15 << up_l;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int ypos = dy * (x0 + k + 1), shift = ((ypos << up_l) & 0x3f) >> 1;
        const int b = (ypos >> (6 - up_l)) + (y << up_l);
        p[k] = b >= lastb ? l[lastb] : (l[b] * (32 - shift) + l[b + 1] * shift + 16) >> 5;
      }
    } else {
      const int dy = kDrDeriv[(angle - 90) >> 1], dx = kDrDeriv[(180 - angle) >> 1];
      const int t = (y + 1) * dx - 64;
      const int xs = t <= 0 ? 0 : ::min((t + 63) >> 6, 8);  // left edge before xs, above edge from it
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int x = x0 + k;
        const bool lf = x < xs;
        const int pos = lf ? (y << 6) - (x + 1) * dy : (xs << 6) - (y + 1) * dx;
        const int up = lf ? up_l : up_a;
        const int32_t* e = lf ? l : a;
        const int b = (pos >> (6 - up)) + (lf ? 0 : (x - xs) << up_a);
        const int sh = ((pos * (1 << up)) & 0x3f) >> 1;
        p[k] = (e[b] * (32 - sh) + e[b + 1] * sh + 16) >> 5;
      }
    }
  } else if (mode == MT_PAETH_PRED) {
    const int32_t lv = L[y], cn = A[-1];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int32_t tv = A[x0 + k], b = lv + tv - cn;
      const int32_t ld = abs(lv - b), td = abs(tv - b), cd = abs(cn - b);
      p[k] = (ld <= td && ld <= cd) ? lv : (td <= cd ? tv : cn);
    }
  } else {
    const int32_t right = A[7], bottom = L[7], wv = kSmW8[y], lv = L[y];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int32_t wh = kSmW8[x0 + k];
      const int32_t v = wv * A[x0 + k] + (256 - wv) * bottom, h = wh * lv + (256 - wh) * right;
      p[k] = mode == MT_SMOOTH_PRED ? (v + h + 256) >> 9 : ((mode == MT_SMOOTH_V_PRED ? v : h) + 128) >> 8;
    }
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int i = (x0 + k) * 8 + y;
    const int16_t r = (int16_t)(src[i] - p[k]);
    pcol[i] = (int16_t)p[k];
    rcol[i] = r;
    rrow[y * 8 + x0 + k] = r;
  }
}

}  // namespace mtd
