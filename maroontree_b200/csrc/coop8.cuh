// The encoder's 8x8 candidate chain (chain8.cuh) with EIGHT lanes per candidate,
// for a launch whose latency, not its throughput, bounds the run: the wavefront
// of the encoder, where a few dozen blocks per dependency level are all the work
// there is.
//
// The four groups of a warp run one transform type, so the warp never splits:
// every sync is the whole warp's.  Lane j of a group holds row j of the block in
// registers from the quantisation to the cost (column j after the inverse).
// Shared memory carries the two transposes, the terms of the ordered float sums,
// and tables.  Sixteen lanes per candidate (half rows) were slower (512x512 4:4:4
// 8.8 against 8.4 us a dependency level, 1080p 9.9 against 8.8): both halves
// have to run the row and column passes, and a block's warps share the issue
// slots of the SMs it runs on.
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
//     integer sums (SATD, counts) are reduced across lanes in any order;
//   * levels become floats, and targets levels, by adding and subtracting 2^23
//     (exact for them), which spares the conversion unit.
#pragma once
#include <stdint.h>

#include "chain4.cuh"
#include "chain8.cuh"

namespace mtd {

// Shared-memory working set of one group.  t: transposes (stride 9, or 5 at
// 4x4).  Trellis: sr[4 + k] = the suffix sum from scan index 63 - k (sr[3] = 0
// is the empty sum), b[e] and r[e] the prefix terms.  Rate: the walk's terms at
// 63 - scan index, the first of each position in b, or where some level has two
// the pairs over b and r; the third ones in t.  296 words: the groups of a warp
// start 8 banks apart.
struct GroupBuf {
  int32_t t[72];
  float sr[68];
  float b[64];
  float r[64];
  float pad[28];
};
static_assert(sizeof(GroupBuf) / 4 % 32 == 8 && sizeof(GroupBuf) % 16 == 0, "bank offset of a group");

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
  float mdc, mac;    // the multipliers / 65536 (exact, so scaling by them rounds once, as the reference's two steps do)
  uint32_t idiv[2];  // 2^32 / dc_q, 2^32 / ac_q, rounded up
  int has_qm;
  mt_quant q;
  alignas(16) float zero[64];  // the suffix chain's empty second terms
  float idt[2][256];           // IDTX targets 8 m / ac_q and 8 m / dc_q of a residual of magnitude m

  // Thread t of 64: qm the plane's inverse QM row (NULL: flat), n its samples.
  __device__ __forceinline__ void stage(int t, const mt_quant& quant, float lam, const uint8_t* qm, int n) {
    const int w = qm && t < n ? qm[t] : 32;
    qs[t] = fwd_qm_scale(w);
    const int32_t base = t == 0 ? quant.dc_q : quant.ac_q;
    step[t] = qm ? (base * w + 16) >> 5 : base;
    zero[t] = 0.0f;
    lrate[t] = __fmul_rn(lam, kCoefRateLut[t]);
    const int bin = t < 2 ? t : 32 - __clz(t), extra = bin > 1 ? bin - 2 : 0;
    lsig[t] = __fmul_rn(lam, __fadd_rn(__fmul_rn((float)bin, 0.9f), __fadd_rn((float)extra, 2.0f)));
    for (int m = t; m < 256; m += 64) {
      idt[0][m] = __fdiv_rn((float)(m * 8), (float)quant.ac_q);
      idt[1][m] = __fdiv_rn((float)(m * 8), (float)quant.dc_q);
    }
    if (t == 0) {
      lambda = lam;
      dq2 = __fmul_rn((float)quant.dc_q, (float)quant.dc_q);
      aq2 = __fmul_rn((float)quant.ac_q, (float)quant.ac_q);
      mdc = (float)quant.q_mult_dc / 65536.0f;
      mac = (float)quant.q_mult_ac / 65536.0f;
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

// Lane j of a group of W lanes (8 for an 8x8 block, 4 for a 4x4 one).
template <int W>
struct Coop {
  int j;
  __device__ __forceinline__ Coop() : j(threadIdx.x & (W - 1)) {}
  __device__ __forceinline__ uint32_t max(uint32_t v) const {
#pragma unroll
    for (int s = W / 2; s; s >>= 1) v = ::max(v, __shfl_xor_sync(0xffffffffu, v, s));
    return v;
  }
  __device__ __forceinline__ uint32_t min(uint32_t v) const {
#pragma unroll
    for (int s = W / 2; s; s >>= 1) v = ::min(v, __shfl_xor_sync(0xffffffffu, v, s));
    return v;
  }
  __device__ __forceinline__ uint32_t sum(uint32_t v) const {
#pragma unroll
    for (int s = W / 2; s; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    return v;
  }
  __device__ __forceinline__ uint32_t any_of(uint32_t v) const {
#pragma unroll
    for (int s = W / 2; s; s >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, s);
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

// float(v) of |v| < 2^22, and floor(x) of 0 <= x < 2^22 as an integer and as a
// float.
__device__ __forceinline__ float small_float(int32_t v) {
  return __fsub_rn(__int_as_float(0x4b400000 + v), 12582912.0f);
}
__device__ __forceinline__ int32_t small_floor(float x, float* f) {
  const float y = __fadd_rz(x, 8388608.0f);
  *f = __fsub_rn(y, 8388608.0f);
  return __float_as_int(y) - 0x4b000000;
}

// Quantisation (+ QM) of row j of 2-D coefficients v, |v| < 2^16 (8-bit
// residuals) and multipliers of at most 2^15, so that the products stay in 32
// bits: levels c and target magnitudes at.  scale: 1, or 2 at 4x4
// (src/dct.rs:3076-3100).
template <int W>
__device__ __forceinline__ void coop_quant(const int32_t* v, const CoopPlane& P, int scale, int32_t* c, float* at,
                                           const Coop<W>& g) {
#pragma unroll
  for (int k = 0; k < W; k++) {
    const bool dc = k == 0 && g.j == 0;
    const float tf = __fmul_rn(small_float(v[k]), (dc ? P.mdc : P.mac) * (float)scale);
    if (P.has_qm) {  // apply_qm: round half away from zero by the fraction
      at[k] = fabsf(__fmul_rn(tf, P.qs[k * W + g.j]));
      float tr;
      int32_t l = small_floor(at[k], &tr);
      l += __fsub_rn(at[k], tr) >= 0.5f;
      c[k] = v[k] < 0 ? -l : l;
    } else {
      const int32_t p = v[k] * ((dc ? P.q.q_mult_dc : P.q.q_mult_ac) * scale), l = (abs(p) + 32768) >> 16;
      at[k] = fabsf(tf);
      c[k] = p < 0 ? -l : l;
    }
  }
}

// Whether a type's forward transform starts from the rows of the residual.
__device__ __forceinline__ bool coop8_by_rows(int TX) { return TX == MT_TX_IDTX || TX == MT_TX_H_DCT; }

// Forward transform and quantisation of type TX from column j (or row j:
// coop8_by_rows) of the residual, magnitudes below 256.  The two passes are one
// loop, so that a warp runs the second from the instructions it has just
// fetched: the kernels' code is larger than the instruction caches.
__device__ __forceinline__ void coop8_fwd(int TX, int32_t* v, const CoopPlane& P, int32_t* c, float* at, GroupBuf& o,
                                          const Coop<8>& g) {
  const int j = g.j;
  if (TX == MT_TX_IDTX) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const bool dc = k == 0 && j == 0;
      const int32_t qd = dc ? P.q.dc_q : P.q.ac_q;
      const uint32_t m = (uint32_t)abs(v[k]), am = m * 8;
      at[k] = P.idt[dc][::min(m, 255u)];
      // (am + qd / 2) / qd: exact for am + qd / 2 < 2^16 and qd < 2^12
      const int32_t level = (int32_t)__umulhi(am + (uint32_t)(qd >> 1), dc ? P.idiv[0] : P.idiv[1]);
      c[k] = (int32_t)am < qd ? 0 : (v[k] < 0 ? -level : level);
    }
    return;
  }
  const bool one = TX == MT_TX_V_DCT || TX == MT_TX_H_DCT;  // one pass, quant_fullstep
#pragma unroll 1
  for (int pass = TX == MT_TX_H_DCT; pass < 2; pass++) {
    const bool adst = TX == MT_TX_ADST_ADST || TX == (pass ? MT_TX_DCT_ADST : MT_TX_ADST_DCT);
    if (adst) fadst8(v);
    else if (!(pass && TX == MT_TX_V_DCT)) fdct8(v);
    if (!pass) coop_transpose<8>(v, o.t, j);
  }
  if (one) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int32_t p = v[k] * 2 * (k == 0 && j == 0 ? P.q.q_mult_dc : P.q.q_mult_ac), l = (abs(p) + 32768) >> 16;
      at[k] = fabsf(__fmul_rn((float)p, 1.0f / 65536.0f));
      c[k] = abs(p) < 65536 ? 0 : (p < 0 ? -l : l);
    }
  } else {
    coop_quant<8>(v, P, 1, c, at, g);
  }
}

// The 4x4 DCT_DCT of the same form from column j (v).
__device__ __forceinline__ void coop4_fwd(int32_t* v, const CoopPlane& P, int32_t* c, float* at, GroupBuf& o,
                                          const Coop<4>& g) {
  fdct4v(v);
  coop_transpose<4>(v, o.t, g.j);
  fdct4v(v);
  coop_quant<4>(v, P, 2, c, at, g);
}

// trellis_optimize (trellis8 / trellis4) over row j's levels c and target
// magnitudes at, e their scan indexes; without `run` the levels stay.  Returns
// the final end of block (-1: all zero).
template <int W>
__device__ __forceinline__ int coop_trellis(int32_t* c, const float* at, const int* e, const CoopPlane& P, GroupBuf& o,
                                            const Coop<W>& g, bool run = true) {
  constexpr unsigned kAll = 0xffffffffu;
  int e1 = 0;
  bool big = false;
#pragma unroll
  for (int k = 0; k < W; k++) {
    if (c[k] != 0) e1 = ::max(e1, e[k] + 1);
    big |= abs(c[k]) > 63;
  }
  const int m = (int)g.max((unsigned)e1);
  if (!run || !(P.lambda > 0.0f) || !__any_sync(kAll, m != 0)) return m - 1;
  const int full8 = m & ~7, chunked = full8 + ((m - full8) >= 4 ? 4 : 0);
  // step A.  The reference decides each position of a chunk (of eight, then one
  // of four) from the chunk's starting values, in the AVX2 FMA form unless the
  // chunk holds a level above 63; then, and in the scalar tail, the plain form.
  const bool any_big = __any_sync(kAll, big);
  unsigned bigb = 0;  // bit k: chunk k holds one
  if (any_big) {
#pragma unroll
    for (int k = 0; k < W; k++)
      if (abs(c[k]) > 63 && e[k] < chunked) bigb |= 1u << (e[k] >> 3);
    bigb = g.any_of(bigb);
  }
#pragma unroll
  for (int k = 0; k < W; k++) {
    const float q2 = k == 0 && g.j == 0 ? P.dq2 : P.aq2;
    const int32_t l = abs(c[k]), ld = ::max(l - 1, 0);
    const float fl = small_float(l), fd = fmaxf(__fsub_rn(fl, 1.0f), 0.0f);
    const float el = __fsub_rn(at[k], fl), ed = __fsub_rn(at[k], fd);
    float rl, rd;
    bool fma_form = e[k] < chunked;
    if (!any_big) {
      rl = P.lrate[l];
      rd = P.lrate[ld];
    } else {
      rl = l < 64 ? P.lrate[l] : __fmul_rn(P.lambda, coef_rate_bits((uint32_t)l));
      rd = ld < 64 ? P.lrate[ld] : __fmul_rn(P.lambda, coef_rate_bits((uint32_t)ld));
      fma_form = fma_form && !((bigb >> (e[k] >> 3)) & 1u);
    }
    const float l2 = __fmul_rn(el, el), d2 = __fmul_rn(ed, ed);
    const float ql = __fmul_rn(q2, l2), qd = __fmul_rn(q2, d2);
    const float cl = fma_form ? __fmaf_rn(q2, l2, rl) : __fadd_rn(ql, rl);
    const float cd = fma_form ? __fmaf_rn(q2, d2, rd) : __fadd_rn(qd, rd);
    const bool dn = l != 0 && cd < cl;
    if (dn) c[k] = c[k] < 0 ? c[k] + 1 : c[k] - 1;
    // the terms of the ordered sums: S = q2 at^2 (the zeroing distortion, +0
    // past the end of block), B = q2 (at - l)^2, R = lambda rate(l)
    o.sr[67 - e[k]] = e[k] < m ? __fmul_rn(q2, __fmul_rn(at[k], at[k])) : 0.0f;
    o.b[e[k]] = dn ? qd : ql;
    o.r[e[k]] = dn ? rd : rl;
  }
  if (g.j == 0) o.sr[W == 4 ? 67 - 16 : 3] = 0.0f;  // the empty sum past the whole scan
  __syncwarp();
  // Lane 0: the suffix sums right to left (acc += S; S = acc).  Lane 1: the
  // prefix cost left to right (b = pre + B; B = b; pre = b + R).
  if (g.j < 2) {
    const int m8 = (m + 7) & ~7;
    float* arr = g.j == 0 ? o.sr + 4 + (64 - m8) : o.b;
    const float* add = g.j == 0 ? P.zero : o.r;
    float acc = 0.0f;
#pragma unroll 1
    for (int s = 0; s < m8; s += 8) {
      float v[8], r[8];
#pragma unroll
      for (int u = 0; u < 8; u += 4) {
        const float4 x = *reinterpret_cast<const float4*>(arr + s + u), y = *reinterpret_cast<const float4*>(add + s + u);
        v[u] = x.x, v[u + 1] = x.y, v[u + 2] = x.z, v[u + 3] = x.w;
        r[u] = y.x, r[u + 1] = y.y, r[u + 2] = y.z, r[u + 3] = y.w;
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
  // candidate ends: the lowest cost (costs are not negative, so their bits order
  // like their values), the first position on ties
  uint32_t cost[W], low = 0x7f800000u;
#pragma unroll
  for (int k = 0; k < W; k++) {
    cost[k] = 0x7f800000u;
    if (c[k] != 0) cost[k] = __float_as_uint(__fadd_rn(__fadd_rn(o.b[e[k]], P.lsig[e[k]]), o.sr[66 - e[k]]));
    low = ::min(low, cost[k]);
  }
  low = g.min(low);
  uint32_t first = 64;
#pragma unroll
  for (int k = 0; k < W; k++)
    if (cost[k] == low && c[k] != 0) first = ::min(first, (uint32_t)e[k]);
  const int best_e = (int)g.min(first);
  const float best = __uint_as_float(low);
  const float skip = __fadd_rn(o.sr[67], P.lambda);
  const int keep = (best_e == 64 || skip < best) ? 0 : best_e + 1;
#pragma unroll
  for (int k = 0; k < W; k++)
    if (e[k] >= keep) c[k] = 0;
  __syncwarp();
  return keep - 1;
}

// Dequantised row j of c (flat: without the QM).
template <int W>
__device__ __forceinline__ void coop_dequant(const int32_t* c, bool flat, const CoopPlane& P, int32_t* v, int j) {
#pragma unroll
  for (int k = 0; k < W; k++) {
    const int32_t l = c[k];
    const int32_t step = flat ? (k == 0 && j == 0 ? P.q.dc_q : P.q.ac_q) : P.step[k * W + j];
    int32_t mag = (int32_t)(((uint32_t)abs(l) * (uint32_t)step) & 0xffffffu);
    mag = ::min(mag, P.q.cf_max + (l < 0 ? 1 : 0));
    v[k] = l < 0 ? -mag : mag;
  }
}

// Dequantisation + inverse transform of type TX: lane j gets column j of the
// inverse residual.  Both passes in one loop, as in the forward transform.
__device__ __forceinline__ void coop8_inv(int TX, const int32_t* c, const CoopPlane& P, int32_t* v, GroupBuf& o,
                                          const Coop<8>& g) {
  const mt_quant& q = P.q;
  coop_dequant<8>(c, TX == MT_TX_IDTX || TX == MT_TX_V_DCT || TX == MT_TX_H_DCT, P, v, g.j);
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {  // rows, columns
    const int32_t lo = pass ? q.cmin : q.rmin, hi = pass ? q.cmax : q.rmax;
    if (TX == MT_TX_IDTX || TX == (pass ? MT_TX_H_DCT : MT_TX_V_DCT)) {
#pragma unroll
      for (int x = 0; x < 8; x++) v[x] *= 2;
    } else if (TX == MT_TX_ADST_ADST || TX == (pass ? MT_TX_ADST_DCT : MT_TX_DCT_ADST)) {
      iadst8s(v, 1, lo, hi);
    } else {
      idct8s(v, 1, lo, hi);
    }
    if (!pass) {
#pragma unroll
      for (int x = 0; x < 8; x++) v[x] = clampi((v[x] + 1) >> 1, q.cmin, q.cmax);
      coop_transpose<8>(v, o.t, g.j);
    }
  }
#pragma unroll
  for (int y = 0; y < 8; y++) v[y] = (v[y] + 8) >> 4;
}
__device__ __forceinline__ void coop4_inv(const int32_t* c, const CoopPlane& P, int32_t* v, GroupBuf& o,
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

// The first terms of a coded block's rate, in the walk's order: txb_skip, the
// tx-type symbol, the end-of-block position (rate8); coded: the price of the
// first.
__device__ __forceinline__ float coop8_rate_head(const mt_coef_costs& T, float coded, int mode, int tx, int eob) {
  float bits = __fadd_rn(coded, T.txtp[mode][tx]);
  const int bin = eob < 2 ? eob : 32 - __clz(eob);
  bits = __fadd_rn(bits, T.eob_bin[bin]);
  if (bin > 1) {
    const int nb = bin - 2;
    bits = __fadd_rn(bits, T.eob_hi[bin][(eob >> nb) & 1]);
    bits = __fadd_rn(bits, (float)nb);
  }
  return bits;
}

// rate8 over the group; none: the bits of a block without levels; head(eob): the
// first terms of one with levels (coop8_rate_head); sign: the dc_sign context's
// row.  The
// reference's reverse walk has entered exactly the later scan positions when it
// reads a context, and the five neighbours of a position inside the block are
// later ones (past a column's end its map holds nothing yet), so contexts come
// from the final levels: the row's from registers, rows j + 1 and j + 2 by
// shuffles of packed level bytes, summed two to a register.  Every position up
// to the end of block puts its terms (the base token; of a level of 3 or more
// the br cost; of one of 15 or more the golomb cost, which the end of block and
// DC add to the br cost first) in shared memory in the walk's order, an absent
// one as +0, and lane 0 adds them, DC's sign and the sign bits behind them, and
// returns the bits.
template <typename Head>
__device__ __forceinline__ float coop8_rate(const int32_t* c, const int* e, int eob, const mt_coef_costs& T,
                                            float none, Head&& head, const float* sign, GroupBuf& o,
                                            const Coop<8>& g) {
  constexpr unsigned kAll = 0xffffffffu;
  const int j = g.j;
  uint32_t m[8], w[2] = {0, 0}, nz = 0, top = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    m[k] = (uint32_t)abs(c[k]);
    const uint32_t t = ::min(m[k], 15u);
    w[k >> 2] |= (t >= 3 ? t + 0xc0u : t * 0x41u) << (8 * (k & 3));  // level_byte
    nz += m[k] != 0;
    top = ::max(top, m[k]);
  }
  uint32_t a[2], b[2];  // rows j + 1 and j + 2
#pragma unroll
  for (int i = 0; i < 2; i++) {
    a[i] = __shfl_down_sync(kAll, w[i], 1, 8);
    b[i] = __shfl_down_sync(kAll, w[i], 2, 8);
    if (j == 7) a[i] = 0;
    if (j >= 6) b[i] = 0;
  }
  nz = g.sum(nz);  // DC, the end of block and the interior
  const bool any3 = __any_sync(kAll, top >= 3), any15 = __any_sync(kAll, top >= 15);
  auto even = [](uint32_t v) { return __byte_perm(v, 0, 0x4140); };  // bytes 0, 1 as halves
  auto odd = [](uint32_t v) { return __byte_perm(v, 0, 0x4342); };   // bytes 2, 3
  const uint32_t w1[2] = {__funnelshift_r(w[0], w[1], 8), w[1] >> 8}, w2[2] = {__funnelshift_r(w[0], w[1], 16), w[1] >> 16};
  const uint32_t a1[2] = {__funnelshift_r(a[0], a[1], 8), a[1] >> 8};
  uint32_t hm2[4], mg2[4];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    hm2[2 * i] = even(a[i]) + even(w1[i]) + even(a1[i]);
    hm2[2 * i + 1] = odd(a[i]) + odd(w1[i]) + odd(a1[i]);
    mg2[2 * i] = hm2[2 * i] + even(b[i]) + even(w2[i]);
    mg2[2 * i + 1] = hm2[2 * i + 1] + odd(b[i]) + odd(w2[i]);
  }
  // the end of block's base row (one column on), and its br context: 0 at DC, 7
  // inside the first 2 x 2, else 14
  const int eob_row = eob <= 0 ? 0 : 1 + (eob > 8) + (eob > 16);
  const int eob_bc = eob <= 0 ? 0 : (eob == 1 || eob == 2 || eob == 4 ? 7 : 14);
  float* T3 = reinterpret_cast<float*>(o.t);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const bool in = e[k] <= eob, end = e[k] == eob, dc = k == 0 && j == 0;
    const uint32_t hm = (hm2[k >> 1] >> (16 * (k & 1))) & 0xffffu, mag = (mg2[k >> 1] >> (16 * (k & 1))) & 0xffffu;
    const int d = k + j;
    const int ctx = dc ? 0 : (d < 2 ? d : (d < 4 ? 6 : 21)) + ::min((int)((mag + 64) >> 7), 4);
    const int tok = (int)::min(m[k], 3u);
    const float* t1p = end ? &T.eob_base[eob_row][::max(tok - 1, 0)] : &T.base_tok[ctx][tok];
    const float t1 = in ? *t1p : 0.0f;
    if (!any3) {
      o.b[63 - e[k]] = t1;
    } else {
      float t2 = 0.0f, t3 = 0.0f;
      if (m[k] >= 3) {
        const int mg = (int)(hm & 63);
        const int bc = end ? eob_bc : (dc ? 0 : (d > 1 && !(d == 2 && j == 1) ? 14 : 7)) + ::min((mg + 1) >> 1, 6);
        t2 = T.br_cum[bc][::min((int32_t)m[k] - 3, 12)];
        if (m[k] >= 15) {
          t3 = golomb_cost(m[k] - 15);
          if (end || dc) {
            t2 = __fadd_rn(t2, t3);
            t3 = 0.0f;
          }
        }
      }
      *reinterpret_cast<float2*>(o.b + 2 * (63 - e[k])) = make_float2(t1, t2);
      if (any15) T3[63 - e[k]] = t3;
    }
  }
  __syncwarp();
  float bits = 0.0f;
  if (j == 0) {
    bits = eob < 0 ? none : head(eob);
    if (eob >= 0) {
      const int first = (63 - eob) & ~3;
      if (!any3) {
#pragma unroll 2
        for (int k = first; k < 64; k += 4) {
          const float4 x = *reinterpret_cast<const float4*>(o.b + k);
          bits = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(bits, x.x), x.y), x.z), x.w);
        }
      } else if (!any15) {
#pragma unroll 2
        for (int k = first; k < 64; k += 4) {
          const float4 x = *reinterpret_cast<const float4*>(o.b + 2 * k);
          const float4 y = *reinterpret_cast<const float4*>(o.b + 2 * k + 4);
          bits = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(bits, x.x), x.y), x.z), x.w);
          bits = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(bits, y.x), y.y), y.z), y.w);
        }
      } else {
#pragma unroll 1
        for (int k = first; k < 64; k++)
          bits = __fadd_rn(__fadd_rn(__fadd_rn(bits, o.b[2 * k]), o.b[2 * k + 1]), T3[k]);
      }
      if (c[0] != 0) bits = __fadd_rn(bits, sign[c[0] < 0]);
      if (eob > 0) bits = add_ones(bits, (int)nz - (c[0] != 0));
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
