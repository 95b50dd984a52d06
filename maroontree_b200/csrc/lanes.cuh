// The leaf searches' stages for one N x N transform block (N = 8, 16, 32)
// evaluated by N lanes of a warp: 32 / N blocks per warp, every lane of the
// warp in step (all syncs are whole-warp syncs, all loops with a sync run to a
// warp-wide bound).
//
// Why N lanes: a block's stages have N-wide work almost everywhere.  The
// transforms are N independent rows or columns, the prediction N columns, and
// on the default scan an anti-diagonal holds at most N positions, none of
// which reads another one's level: the scan runs diagonal by diagonal (odd
// ones by rising row, even ones by rising column), and the five neighbours a
// coefficient context reads lie one or two diagonals on, or, past a column's
// end, N - 3 or more diagonals back.  So the context trellis walks 2N - 1
// diagonals instead of N * N positions.
// A thread per block keeps 7 to 50 KB of working set per thread, in local
// memory that overflows L1 or in shared memory that few threads fit; here the
// set of a block is 1.2, 4.5 or 20 KB and serves N lanes.
//
// The float chains with a fixed order (the trellis' suffix and prefix sums,
// the rate walk) keep it: their terms are computed by all lanes, compacted in
// the walk's order, and one lane adds them.
//
// Results equal the one-thread stages (leaf8.cuh, chain16.cuh, wsse.cuh) bit
// for bit.
#pragma once
#include <stdint.h>

#include <type_traits>

#include "coop8.cuh"
#include "leaf8.cuh"
#include "txfm32.cuh"
#include "wsse.cuh"

namespace mtd {

constexpr unsigned kFull = 0xffffffffu;

// The lanes of one block.
template <int N>
struct Lanes {
  int j;           // lane of the block, 0 .. N - 1
  unsigned first;  // its lane 0 in the warp
  __device__ __forceinline__ Lanes() : j(threadIdx.x & (N - 1)), first(threadIdx.x & 31u & ~(unsigned)(N - 1)) {}
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  template <typename T>
  __device__ __forceinline__ T sum(T v) const {
#pragma unroll
    for (int s = N / 2; s; s >>= 1) v += __shfl_xor_sync(kFull, v, s);
    return v;
  }
  __device__ __forceinline__ int max(int v) const {
#pragma unroll
    for (int s = N / 2; s; s >>= 1) v = ::max(v, __shfl_xor_sync(kFull, v, s));
    return v;
  }
  // The block's lanes of a warp ballot.
  __device__ __forceinline__ unsigned ballot(bool p) const {
    const unsigned b = __ballot_sync(kFull, p);
    return N == 32 ? b : (b >> first) & ((1u << (N & 31)) - 1u);
  }
  template <typename T>
  __device__ __forceinline__ T from(T v, int lane) const {
    return __shfl_sync(kFull, v, lane, N);
  }
};
__device__ __forceinline__ int warp_max_all(int v) { return __reduce_max_sync(kFull, v); }

// The default scan by diagonals: the first scan index of diagonal d, its
// first row / column, and the scan index of (x, y).
template <int N>
__device__ __forceinline__ int diag_base(int d) {
  const int r = 2 * N - 1 - d;
  return d < N ? (d * (d + 1)) >> 1 : N * N - ((r * (r + 1)) >> 1);
}
template <int N>
__device__ __forceinline__ int scan_index(int x, int y) {
  const int d = x + y, lo = ::max(0, d - (N - 1));
  return diag_base<N>(d) + ((d & 1) ? y : x) - lo;
}
// Diagonal of scan index i.
template <int N>
__device__ __forceinline__ int diag_of(int i) {
  const int rc = scan_rc<N>(i);
  return (rc & (N - 1)) + (rc >> log2w<N>());
}

// kLoCtxOff by diagonal (its entries depend on x + y alone).
__device__ __forceinline__ int lo_ctx_off(int d) { return d < 2 ? d : (d < 4 ? 6 : 21); }

// Shared working set of one block.  tf, a and t are one run of at least 3 N^2
// words: the prediction edges, then targets | prefix terms | transform scratch
// and suffix sums, then the error block (tf) or the rate walk's terms (all
// three).  KEEP: the reconstruction gets room of its own (several types are
// tried on one prediction), else it replaces the prediction.  The size is N
// words mod 32, so the blocks of a warp start N banks apart.
template <int N, bool KEEP = false>
struct LaneBuf {
  static constexpr int NN = N * N;
  // levels are 32-bit at 32x32 (a full-scale DC at the smallest steps passes 16 bits)
  using Coef = std::conditional_t<N == 32, int32_t, int16_t>;
  static constexpr int kWords = 2 * NN + N * (N + 1) + NN * (int)sizeof(Coef) / 4 + NN / 2 * (KEEP ? 2 : 1) +
                                (N + 2) * N / 4 + NN / 32 + 1;
  static constexpr int kPad = ((N - kWords) % 32 + 32) % 32;
  float tf[NN];
  float a[NN];
  int32_t t[N * (N + 1)];
  Coef cf[NN];
  int16_t pred[NN];
  int16_t kept[KEEP ? NN : 2 * kPad + 2];
  uint8_t lv[(N + 2) * N];
  uint16_t ck[NN / 16 + (KEEP ? 2 * kPad + 2 : 0)];  // rate checkpoints; the plain trellis' chunk flags
  __device__ __forceinline__ int16_t* rec() { return KEEP ? kept : pred; }
};
static_assert(sizeof(LaneBuf<16>) / 4 % 32 == 16 && sizeof(LaneBuf<16, true>) / 4 % 32 == 16, "bank offset of 16x16");
static_assert(sizeof(LaneBuf<8>) / 4 % 32 == 8 && sizeof(LaneBuf<32>) % 128 == 0, "bank offset of 8x8 and 32x32");

// predict_sq_at over the block's lanes: the edges position by position in
// shared memory, then lane j writes column j of pred (row-major).
template <int N, typename R>
__device__ __forceinline__ void lane_predict(const R& rd, int fw, int fh, int ox, int oy, int mode, int delta,
                                             bool have_tr, bool have_bl, bool ft, int bd, int16_t* pred,
                                             int32_t* scratch, const Lanes<N>& g) {
  constexpr int cap = edge_cap<N>(), edge_len = 2 * N, L = log2w<N>();
  static_assert(2 * cap <= 3 * N * N, "the edges fit the scratch");
  const int j = g.j;
  int32_t* A = scratch + kEdgeOrigin;
  int32_t* Lf = scratch + cap + kEdgeOrigin;
  const bool have_top = oy > 0, have_left = ox > 0;
  const int32_t base = 1 << (bd - 1);
  const bool dir = mode >= MT_V_PRED && mode <= MT_D67_PRED;
  const int base_angle = mode == MT_V_PRED ? 90 : mode == MT_H_PRED ? 180 : mode == MT_D45_PRED ? 45
                       : mode == MT_D135_PRED ? 135 : mode == MT_D113_PRED ? 113 : mode == MT_D157_PRED ? 157
                       : mode == MT_D203_PRED ? 203 : 67;
  const int angle = base_angle + delta * 3;
  const bool slanted = dir && angle != 90 && angle != 180;
  int32_t a0, a1, l0, l1;  // entries j and N + j of the two edges
  if (have_top) {
    const int px_have = have_tr ? ::min(N, ::max(fw - (ox + N), 0)) : 0;
    a0 = rd(ox + j, oy - 1);
    a1 = rd(ox + N + (j < px_have ? j : px_have - 1), oy - 1);  // the last available sample repeated
  } else {
    a0 = a1 = have_left ? rd(ox - 1, oy) : base - 1;
  }
  if (have_left) {
    const int px_have = have_bl ? ::min(N, ::max(fh - (oy + N), 0)) : 0;
    l0 = rd(ox - 1, oy + j);
    l1 = rd(ox - 1, oy + N + (j < px_have ? j : px_have - 1));
  } else {
    l0 = l1 = have_top ? rd(ox, oy - 1) : base + 1;
  }
  int32_t corner =
      have_left ? (have_top ? rd(ox - 1, oy - 1) : rd(ox - 1, oy)) : (have_top ? rd(ox, oy - 1) : base);
  A[j] = a0;
  A[N + j] = a1;
  Lf[j] = l0;
  Lf[N + j] = l1;
  if (j == 0) {
    // the corner filter of the middle zone, before the edges are smoothed
    if (edge_len >= 24 && slanted && angle > 90 && angle < 180) corner = (5 * l0 + 6 * corner + 5 * a0 + 8) >> 4;
    A[-1] = Lf[-1] = corner;
  }
  int32_t dc = 0;
  {
    const int32_t s = g.sum((have_top ? a0 : 0) + (have_left ? l0 : 0));
    dc = (have_top && have_left) ? (N + s) >> (L + 1) : ((have_top || have_left) ? ((N >> 1) + s) >> L : base);
  }
  g.sync();
  int up_a = 0, up_l = 0;
  if (__any_sync(kFull, slanted)) {
    const int na = N + 1 + (angle < 90 ? N : 0), nl = N + 1 + (angle > 180 ? N : 0);
    const int sa = slanted ? edge_strength(N, N, ft, angle - 90) : 0;
    const int sl = slanted ? edge_strength(N, N, ft, angle - 180) : 0;
    int32_t fa[2], fl[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int o = j + i * N;
      fa[i] = sa && o < na - 1 ? edge_tap(A, o, na, sa) : 0;
      fl[i] = sl && o < nl - 1 ? edge_tap(Lf, o, nl, sl) : 0;
    }
    g.sync();
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int o = j + i * N;
      if (sa && o < na - 1) A[o] = fa[i];
      if (sl && o < nl - 1) Lf[o] = fl[i];
    }
    g.sync();
    if constexpr (N == 8) {  // upsample_edge (never on larger blocks)
      const int da = abs(angle - 90), dl = abs(angle - 180), lim = ft ? 8 : 16;
      up_a = slanted && da < 40 && 2 * N <= lim;
      up_l = slanted && dl < 40 && 2 * N <= lim;
      const int32_t maxv = (1 << bd) - 1;
      const int numa = N + (angle < 90 ? N : 0), numl = N + (angle > 180 ? N : 0);
      auto in = [](const int32_t* e, int k, int num) { return e[(k <= 1 ? 0 : ::min(k - 1, num)) - 1]; };
      int32_t ha[2], va[2], hl[2], vl[2];
      const int32_t am = A[-1], lm = Lf[-1];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int k = j + i * N;
        if (up_a && k < numa) {
          va[i] = in(A, k + 2, numa);
          ha[i] = clampi((-in(A, k, numa) + 9 * in(A, k + 1, numa) + 9 * va[i] - in(A, k + 3, numa) + 8) >> 4, 0, maxv);
        }
        if (up_l && k < numl) {
          vl[i] = in(Lf, k + 2, numl);
          hl[i] =
              clampi((-in(Lf, k, numl) + 9 * in(Lf, k + 1, numl) + 9 * vl[i] - in(Lf, k + 3, numl) + 8) >> 4, 0, maxv);
        }
      }
      g.sync();
      if (j == 0 && up_a) A[-2] = am;
      if (j == 0 && up_l) Lf[-2] = lm;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int k = j + i * N;
        if (up_a && k < numa) A[2 * k - 1] = ha[i], A[2 * k] = va[i];
        if (up_l && k < numl) Lf[2 * k - 1] = hl[i], Lf[2 * k] = vl[i];
      }
      g.sync();
    }
  }
  const int x = j;
  int16_t* out = pred + x;
  if (mode == MT_DC_PRED) {
#pragma unroll 8
    for (int y = 0; y < N; y++) out[y * N] = (int16_t)dc;
  } else if (dir) {
    const int32_t* a = A;
    const int32_t* l = Lf;
    if (angle == 90) {
#pragma unroll 8
      for (int y = 0; y < N; y++) out[y * N] = (int16_t)a0;
    } else if (angle == 180) {
#pragma unroll 8
      for (int y = 0; y < N; y++) out[y * N] = (int16_t)l[y];
    } else if (angle < 90) {
      const int dx = kDrDeriv[angle >> 1];
      const int max_base_x = (edge_len - 1) << up_a, frac_bits = 6 - up_a;
      const int32_t last = a[max_base_x];
#pragma unroll 2
      for (int y = 0; y < N; y++) {
        const int xpos = dx * (y + 1), shift = ((xpos << up_a) & 0x3f) >> 1;
        const int b = (xpos >> frac_bits) + (x << up_a);
        out[y * N] = (int16_t)(b < max_base_x ? (a[b] * (32 - shift) + a[b + 1] * shift + 16) >> 5 : last);
      }
    } else if (angle > 180) {
      const int dy = kDrDeriv[(270 - angle) >> 1];
      const int max_base_y = (edge_len - 1) << up_l, frac_bits = 6 - up_l;
      const int ypos = dy * (x + 1), shift = ((ypos << up_l) & 0x3f) >> 1, b0 = ypos >> frac_bits;
      const int32_t last = l[max_base_y];
#pragma unroll 2
      for (int y = 0; y < N; y++) {
        const int b = b0 + (y << up_l);
        out[y * N] = (int16_t)(b >= max_base_y ? last : (l[b] * (32 - shift) + l[b + 1] * shift + 16) >> 5);
      }
    } else {
      const int dy = kDrDeriv[(angle - 90) >> 1], dx = kDrDeriv[(180 - angle) >> 1];
#pragma unroll 2
      for (int y = 0; y < N; y++) {
        const int t = (y + 1) * dx - 64;
        const int x0 = t <= 0 ? 0 : ::min((t + 63) >> 6, N);
        // left edge before x0, above edge from it
        const int pos = x < x0 ? (y << 6) - (x + 1) * dy : (x0 << 6) - (y + 1) * dx;
        const int up = x < x0 ? up_l : up_a;
        const int32_t* e = x < x0 ? l : a;
        const int b = (pos >> (6 - up)) + (x < x0 ? 0 : (x - x0) << up_a);
        const int sh = ((pos * (1 << up)) & 0x3f) >> 1;
        out[y * N] = (int16_t)((e[b] * (32 - sh) + e[b + 1] * sh + 16) >> 5);
      }
    }
  } else if (mode == MT_PAETH_PRED) {
    const int32_t tv = a0, cn = A[-1];
#pragma unroll 2
    for (int y = 0; y < N; y++) {
      const int32_t lv = Lf[y], b = lv + tv - cn;
      const int32_t ld = abs(lv - b), td = abs(tv - b), cd = abs(cn - b);
      out[y * N] = (int16_t)((ld <= td && ld <= cd) ? lv : (td <= cd ? tv : cn));
    }
  } else {
    const int32_t right = A[N - 1], bottom = Lf[N - 1], wh = sm_weight<N>(x);
#pragma unroll 2
    for (int y = 0; y < N; y++) {
      const int32_t wv = sm_weight<N>(y);
      const int32_t v = wv * a0 + (256 - wv) * bottom, h = wh * Lf[y] + (256 - wh) * right;
      out[y * N] = (int16_t)(mode == MT_SMOOTH_PRED ? (v + h + 256) >> 9
                                                    : ((mode == MT_SMOOTH_V_PRED ? v : h) + 128) >> 8);
    }
  }
  g.sync();
}

// Forward transform + quantisation (+ the QM of the 2-D types) of src - pred
// into w.cf / w.tf: fwd8x8 / fwd16x16 and apply_qm; at 32x32 the residual gets
// 6 bits of headroom and each output the 64-bit rounding (x * 16384 + 2^21) >>
// 22 of dct32x32_quant_t_direct (src/dct.rs:705-736).  qs: the forward scale of
// each QM weight value.  32x32 takes DCT_DCT only, 16x16 no V_DCT / H_DCT.
// Returns the sum of the residual.
template <int N, typename W>
__device__ __forceinline__ int32_t lane_fwd(const uint16_t* __restrict__ src, int stride, int tx, const mt_quant& q,
                                            const uint8_t* qm, const float* qs, W& w, const Lanes<N>& g) {
  using Coef = typename W::Coef;
  const int j = g.j;
  int32_t v[N];
  int32_t sum = 0;
#pragma unroll
  for (int r = 0; r < N; r++) {
    v[r] = (int32_t)src[(size_t)r * stride + j] - w.pred[r * N + j];
    sum += v[r];
    v[r] = (int16_t)v[r];
  }
  sum = g.sum(sum);
  g.sync();  // the edges of the prediction are done with
  if (N != 32 && tx == MT_TX_IDTX) {
#pragma unroll
    for (int y = 0; y < N; y++) {
      const int rc = y + j * N;
      const int32_t qd = rc == 0 ? q.dc_q : q.ac_q;
      const int32_t num = v[y] * 8;
      w.tf[rc] = __fdiv_rn((float)num, (float)qd);
      const int32_t am = (int32_t)uabs(num);
      const int32_t level = (am + qd / 2) / qd;
      w.cf[rc] = (Coef)(am < qd ? 0 : (num < 0 ? -level : level));
    }
    g.sync();
    return sum;
  }
  const bool col_adst = N != 32 && (tx == MT_TX_ADST_ADST || tx == MT_TX_ADST_DCT);
  const bool row_adst = N != 32 && (tx == MT_TX_ADST_ADST || tx == MT_TX_DCT_ADST);
  const bool one = N == 8 && (tx == MT_TX_V_DCT || tx == MT_TX_H_DCT);  // one pass, quant_fullstep
  auto pass = [&](bool adst) {
    if constexpr (N == 32) {
      fdct32(v);
    } else if constexpr (N == 16) {
      if (adst) fadst16(v); else fdct16(v);
    } else {
      if (adst) fadst8(v); else fdct8(v);
    }
  };
  if constexpr (N == 32) {
#pragma unroll
    for (int r = 0; r < N; r++) v[r] *= 64;
  }
  // one copy of the transform for both passes: the chain's code is larger than
  // the instruction caches
#pragma unroll 1
  for (int ps = 0; ps < 2; ps++) {
    if (!one || tx == (ps ? MT_TX_H_DCT : MT_TX_V_DCT)) pass(ps ? row_adst : col_adst);
    if (ps == 0) {
#pragma unroll
      for (int r = 0; r < N; r++) w.t[r * (N + 1) + j] = v[r];
      g.sync();
#pragma unroll
      for (int u = 0; u < N; u++) v[u] = w.t[j * (N + 1) + u];
    }
  }
#pragma unroll
  for (int u = 0; u < N; u++) w.t[j * (N + 1) + u] = v[u];  // the lane's own row: a loop over it stays short
#pragma unroll 4
  for (int u = 0; u < N; u++) {
    const int idx = u * N + j;
    const int32_t m = idx == 0 ? q.q_mult_dc : q.q_mult_ac;
    int32_t c = w.t[j * (N + 1) + u];
    if constexpr (N == 16) c = mul_q16(c, 32768);
    if constexpr (N == 32) c = (int32_t)(((long long)c * 16384 + (1ll << 21)) >> 22);
    float x;
    Coef l;
    if (one) {
      const int32_t p = c * 2 * m, lv = (abs(p) + 32768) >> 16;
      x = __fmul_rn((float)p, 1.0f / 65536.0f);
      l = (Coef)(abs(p) < 65536 ? 0 : (p < 0 ? -lv : lv));
    } else {
      x = __fmul_rn(__fmul_rn((float)c, (float)m), 1.0f / 65536.0f);
      l = (Coef)quant_q16(c, m);
    }
    if (qm && !one) {
      x = __fmul_rn(x, qs[qm[idx]]);
      const float tr = truncf(x);
      const float step = fabsf(__fsub_rn(x, tr)) >= 0.5f ? copysignf(1.0f, x) : 0.0f;
      l = (Coef)(int32_t)__fadd_rn(tr, step);
    }
    w.tf[idx] = x;
    w.cf[idx] = l;
  }
  g.sync();
  return sum;
}

// Last nonzero scan index of w.cf, -1 when all are zero.
template <int N, typename W>
__device__ __forceinline__ int lane_eob(const W& w, const Lanes<N>& g) {
  int e1 = 0;
#pragma unroll 8
  for (int x = 0; x < N; x++)
    if (w.cf[x * N + g.j] != 0) e1 = ::max(e1, scan_index<N>(x, g.j) + 1);
  return g.max(e1) - 1;
}

// The level map of w.cf (trellis_ctx / rate_bounded: stride N, two zero
// columns).
template <int N, typename W>
__device__ __forceinline__ void lane_level_map(W& w, const Lanes<N>& g) {
#pragma unroll 8
  for (int x = 0; x < N; x++) w.lv[x * N + g.j] = (uint8_t)level_byte(uabs(w.cf[x * N + g.j]));
  w.lv[N * N + g.j] = 0;
  w.lv[N * N + N + g.j] = 0;
}

// trellis_ctx8 at side N over the block's lanes (same parameters).  Returns the final
// end of block (-1: all zero).
template <int N, typename W>
__device__ __forceinline__ int lane_trellis_ctx(W& w, float dc_q, float ac_q, float lambda, const mt_coef_costs& T,
                                                int dcs, const uint8_t* qm, bool qm_full, float band_t,
                                                const Lanes<N>& g) {
  using Coef = typename W::Coef;
  constexpr int L = log2w<N>(), NN = N * N;
  constexpr float kCap = 2.0f, kNInv = 1.0f / (float)NN;
  const int j = g.j;
  auto* cf = w.cf;
  const float* tf = w.tf;
  uint8_t* lv = w.lv;
  const int eob = lane_eob<N>(w, g), m = eob + 1;
  const int M = warp_max_all(m);
  if (M == 0) return -1;
  const int D = diag_of<N>(M - 1);
  const float dq2_dc = __fmul_rn(dc_q, dc_q), dq2_ac = __fmul_rn(ac_q, ac_q);
  auto qm_at = [&](int rc) -> float {
    const float wq = __fmul_rn((float)qm[rc], 1.0f / 32.0f);  // exact
    return qm_full ? __fmul_rn(wq, wq) : wq;
  };
  auto distw = [&](int idx, int rc, uint32_t lev) -> float {
    const float at = fabsf(tf[rc]);
    const float e = __fsub_rn(at, (float)lev);
    float d = __fmul_rn(rc == 0 ? dq2_dc : dq2_ac, __fmul_rn(e, e));
    if (qm) d = __fmul_rn(d, qm_at(rc));
    if (band_t != 0.0f && at < kCap) d = __fdiv_rn(d, __fadd_rn(1.0f, __fmul_rn(band_t, __fmul_rn((float)idx, kNInv))));
    return d;
  };
  lane_level_map<N>(w, g);
  g.sync();
  auto interior_ctx = [&](int rc, int& bc) -> int {
    const int x = rc >> L, y = rc & (N - 1);
    const uint32_t hm = (uint32_t)lv[rc + 1] + lv[rc + N] + lv[rc + N + 1];
    const uint32_t mag = hm + lv[rc + 2] + lv[rc + 2 * N];
    const uint32_t hm6 = hm & 63;
    bc = ((y | x) > 1 ? 14 : 7) + (hm6 > 12 ? 6 : (int)((hm6 + 1) >> 1));
    return lo_ctx_off(x + y) + (mag > 512 ? 4 : (int)((mag + 64) >> 7));
  };
  auto dc_brc = [&]() -> int {
    const uint32_t mag = ((uint32_t)lv[1] + lv[N] + lv[N + 1]) & 63;
    return mag > 12 ? 6 : (int)((mag + 1) >> 1);
  };

  // Step A, a diagonal at a time from the last one down: a position's context
  // reads final levels of later diagonals (and, past a column's end, starting
  // levels of much earlier ones).
  for (int d = D; d >= 1; d--) {
    const int lo = ::max(0, d - (N - 1)), len = ::min(d + 1, 2 * N - 1 - d);
    const int i = diag_base<N>(d) + j;
    const int p = lo + j, x = (d & 1) ? d - p : p, y = d - x;
    const int rc = x * N + y;
    const bool in = j < len && i < eob;
    const uint32_t l = in ? uabs(cf[rc]) : 0u;
    if (!__any_sync(kFull, l != 0)) continue;
    if (l != 0) {
      int bc;
      const int ctx = interior_ctx(rc, bc);
      const float* bt = T.base_tok[ctx];
      auto rate_k = [&](uint32_t k) -> float {
        if (k == 0) return bt[0];
        if (k < 3) return __fadd_rn(bt[k], 1.0f);
        return __fadd_rn(__fadd_rn(bt[3], hi_cost(T, k, bc)), 1.0f);
      };
      uint32_t best_k = l;
      float best_c = 0.0f;
#pragma unroll 1
      for (int32_t k = (int32_t)l; k >= 0; k--) {  // the level itself, then the lower ones
        const bool first = k == (int32_t)l;
        const float dk = distw(i, rc, (uint32_t)k);
        if (!first && dk >= best_c) break;
        const float c = __fadd_rn(dk, __fmul_rn(lambda, rate_k((uint32_t)k)));
        if (first || c < best_c) {
          best_c = c;
          best_k = (uint32_t)k;
        }
      }
      if (best_k != l) {
        cf[rc] = (Coef)(cf[rc] < 0 ? -(int32_t)best_k : (int32_t)best_k);
        lv[rc] = (uint8_t)level_byte(best_k);
      }
    }
    g.sync();
  }
  if (j == 0 && m > 0) {
    const uint32_t l = uabs(cf[0]);
    if (l != 0) {
      const int bc = dc_brc();
      const float sgn_bits = T.dc_sign[dcs][cf[0] < 0];
      auto dc_rate = [&](uint32_t k) -> float {
        if (k == 0) return T.base_tok[0][0];
        float b = T.base_tok[0][::min(k, 3u)];
        if (k >= 3) b = __fadd_rn(b, hi_cost(T, k, bc));
        return __fadd_rn(b, sgn_bits);
      };
      uint32_t best_k = l;
      float best_c = 0.0f;
#pragma unroll 1
      for (int32_t k = (int32_t)l; k >= 0; k--) {
        const bool first = k == (int32_t)l;
        const float dk = distw(0, 0, (uint32_t)k);
        if (!first && dk >= best_c) break;
        const float c = __fadd_rn(dk, __fmul_rn(lambda, dc_rate((uint32_t)k)));
        if (first || c < best_c) {
          best_c = c;
          best_k = (uint32_t)k;
        }
      }
      if (best_k != l) {
        cf[0] = (Coef)(cf[0] < 0 ? -(int32_t)best_k : (int32_t)best_k);
        lv[0] = (uint8_t)level_byte(best_k);
      }
    }
  }
  g.sync();

  // Step B: every position's zeroing distortion (S) and rate + distortion (A),
  // then the two ordered sums.
  float* S = reinterpret_cast<float*>(w.t);
  float* A = w.a;
  float cur0 = 0.0f, zero0 = 0.0f;
  for (int x = 0; x <= ::min(D, N - 1); x++) {
    const int rc = x * N + j, i = scan_index<N>(x, j);
    if (i < m) {
      const float dq2 = rc == 0 ? dq2_dc : dq2_ac;
      const float at = fabsf(tf[rc]);
      const uint32_t k = uabs(cf[rc]);
      const float e = __fsub_rn(at, (float)k);
      float cur = __fmul_rn(dq2, __fmul_rn(e, e));
      float zero = __fmul_rn(dq2, __fmul_rn(at, at));
      if (qm) {
        const float w2 = qm_at(rc);
        cur = __fmul_rn(cur, w2);
        zero = __fmul_rn(zero, w2);
      }
      if (band_t != 0.0f && at < kCap) {
        const float wgt = __fdiv_rn(1.0f, __fadd_rn(1.0f, __fmul_rn(band_t, __fmul_rn((float)i, kNInv))));
        zero = __fmul_rn(zero, wgt);
        cur = __fmul_rn(cur, wgt);
      }
      if (i == 0) {
        cur0 = cur;
        zero0 = zero;
      } else {
        int bc;
        const int ctx = interior_ctx(rc, bc);
        float r = T.base_tok[ctx][::min(k, 3u)];
        if (k >= 3) r = __fadd_rn(r, hi_cost(T, k, bc));
        if (k != 0) r = __fadd_rn(r, 1.0f);
        S[i] = zero;
        A[i] = __fadd_rn(__fmul_rn(lambda, r), cur);
      }
    }
  }
  cur0 = g.from(cur0, 0);
  zero0 = g.from(zero0, 0);
  g.sync();
  // lane 0: S[i] = the sum of S from m - 1 down to i; lane 1: A[e] = the sum of A[1 .. e - 1]
  if (j < 2) {
    if (j == 0) S[m] = 0.0f;
    float* arr = j == 0 ? S : A;
    float acc = 0.0f;
    int s = 1;
    for (; s + 8 <= m; s += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = arr[j == 0 ? m - (s + u) : s + u];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const float nx = __fadd_rn(acc, v[u]);
        arr[j == 0 ? m - (s + u) : s + u] = j == 0 ? nx : acc;
        acc = nx;
      }
    }
    for (; s < m; s++) {
      const int e = j == 0 ? m - s : s;
      const float nx = __fadd_rn(acc, arr[e]);
      arr[e] = j == 0 ? nx : acc;
      acc = nx;
    }
  }
  g.sync();
  const uint32_t dc_m = uabs(cf[0]);
  const bool dc_neg = cf[0] < 0;
  float dc_cost;
  if (dc_m == 0) {
    dc_cost = __fmul_rn(lambda, T.base_tok[0][0]);
  } else {
    float b = T.base_tok[0][::min(dc_m, 3u)];
    if (dc_m >= 3) b = __fadd_rn(b, hi_cost(T, dc_m, dc_brc()));
    b = __fadd_rn(b, T.dc_sign[dcs][dc_neg]);
    dc_cost = __fmul_rn(lambda, b);
  }
  dc_cost = __fadd_rn(dc_cost, cur0);
  auto eob_coeff_cost = [&](int e, int rc, uint32_t k) -> float {
    const int ctx_e = 1 + (e > (NN >> 3)) + (e > (NN >> 2));
    const uint32_t tok = ::min(k, 3u);
    float c = T.eob_base[ctx_e][tok - 1];
    if (tok == 3) c = __fadd_rn(c, hi_cost(T, k, ((rc >> L) | (rc & (N - 1))) > 1 ? 14 : 7));
    return __fadd_rn(c, 1.0f);
  };
  auto eob_pt_cost = [&](int e) -> float {
    const int bin = e < 2 ? e : 32 - __clz(e);
    float c = T.eob_bin[bin];
    if (bin > 1) {
      const int nb = bin - 2;
      c = __fadd_rn(c, T.eob_hi[bin][(e >> nb) & 1]);
      c = __fadd_rn(c, (float)nb);
    }
    return c;
  };
  float best_cost = __int_as_float(0x7f800000);
  int best_e = NN;
  uint32_t best_m = 0;
  for (int x = 0; x <= ::min(D, N - 1); x++) {
    const int rc = x * N + j, e = scan_index<N>(x, j);
    const uint32_t k = e >= 1 && e < m ? uabs(cf[rc]) : 0u;
    if (k != 0) {
      const float base = __fadd_rn(__fadd_rn(__fadd_rn(dc_cost, A[e]), __fmul_rn(lambda, eob_pt_cost(e))), S[e + 1]);
      uint32_t m_best = k;
      float c = 0.0f;
#pragma unroll 1
      for (uint32_t lv1 = k; lv1 >= ::max(k - 1, 1u); lv1--) {  // the level, and the one below where it is not zero
        const float cl =
            __fadd_rn(base, __fadd_rn(__fmul_rn(lambda, eob_coeff_cost(e, rc, lv1)), distw(e, rc, lv1)));
        if (lv1 == k || cl < c) {
          c = cl;
          m_best = lv1;
        }
      }
      if (c < best_cost) {  // rising e: the first one on ties; never an infinite cost
        best_cost = c;
        best_e = e;
        best_m = m_best;
      }
    }
  }
#pragma unroll
  for (int s = N / 2; s; s >>= 1) {
    const float oc = __shfl_xor_sync(kFull, best_cost, s);
    const int oe = __shfl_xor_sync(kFull, best_e, s);
    const uint32_t om = __shfl_xor_sync(kFull, best_m, s);
    if (oc < best_cost || (oc == best_cost && oe < best_e)) {
      best_cost = oc;
      best_e = oe;
      best_m = om;
    }
  }
  if (best_e == NN) best_e = -1;
  const float suf1 = S[1];  // (m == 1: S[m])
  if (dc_m != 0) {
    float c0 = __fadd_rn(T.eob_bin[0], T.eob_base[0][::min(dc_m, 3u) - 1]);
    if (dc_m >= 3) c0 = __fadd_rn(c0, hi_cost(T, dc_m, 0));
    const float r = __fadd_rn(c0, T.dc_sign[dcs][dc_neg]);
    const float total0 = __fadd_rn(__fadd_rn(__fmul_rn(lambda, r), cur0), suf1);
    if (total0 < best_cost) {
      best_cost = total0;
      best_e = 0;
      best_m = dc_m;
    }
  }
  const float skip_cost = __fadd_rn(__fadd_rn(suf1, zero0), __fmul_rn(lambda, 1.0f));
  if (best_e < 0 || skip_cost < best_cost) best_e = -1;
  g.sync();  // every lane has read cf[0]
  for (int x = 0; x <= ::min(D, N - 1); x++) {
    const int rc = x * N + j, i = scan_index<N>(x, j);
    if (i < m) {
      if (i > best_e) {
        cf[rc] = 0;
      } else if (i == best_e && best_m != uabs(cf[rc])) {
        const bool neg = cf[rc] != 0 ? cf[rc] < 0 : tf[rc] < 0.0f;
        cf[rc] = (Coef)(neg ? -(int32_t)best_m : (int32_t)best_m);
      }
    }
  }
  g.sync();
  return best_e;
}

// trellis_sq (trellis_optimize) over the block's lanes.  Returns the final end
// of block (-1: all zero).
template <int N, typename W>
__device__ __forceinline__ int lane_trellis_plain(W& w, float dc_q, float ac_q, float lambda, const float* lut,
                                                  const Lanes<N>& g) {
  using Coef = typename W::Coef;
  constexpr int NN = N * N, kFlagWords = NN / 256 ? NN / 256 : 1;
  const int j = g.j;
  auto* cf = w.cf;
  const float dq2 = __fmul_rn(dc_q, dc_q), aq2 = __fmul_rn(ac_q, ac_q);
  const int m = lane_eob<N>(w, g) + 1;
  const int M = warp_max_all(m);
  if (M == 0) return -1;
  const int xmax = ::min(diag_of<N>(M - 1), N - 1);  // the last column that holds a scan index below M
  const int full8 = m & ~7;
  const bool has4 = (m - full8) >= 4;
  const int chunked = full8 + (has4 ? 4 : 0);
  // step A: each chunk of eight (and one of four) positions takes the FMA form
  // unless it holds a level above 63; the rest the plain form
  unsigned* flags = reinterpret_cast<unsigned*>(w.a);
  bool big = false;
  for (int x = 0; x <= xmax; x++) big |= uabs(cf[x * N + j]) > 63u;
  const bool any_big = __any_sync(kFull, big);
  if (any_big) {
    if (j < kFlagWords) flags[j] = 0;
    g.sync();
    for (int x = 0; x <= xmax; x++) {
      const int e = scan_index<N>(x, j);
      if (e < chunked && uabs(cf[x * N + j]) > 63u) atomicOr(&flags[e >> 8], 1u << ((e >> 3) & 31));
    }
    g.sync();
  }
  for (int x = 0; x <= xmax; x++) {
    const int rc = x * N + j, e = scan_index<N>(x, j);
    const int32_t c = cf[rc];
    if (e < m && c != 0) {
      const float at = fabsf(w.tf[rc]), q2 = rc == 0 ? dq2 : aq2;
      bool dn;
      if (e < chunked && !(any_big && ((flags[e >> 8] >> ((e >> 3) & 31)) & 1u))) {
        const int32_t li = (int32_t)uabs(c), ldi = ::max(li - 1, 0);
        const float el = __fsub_rn(at, (float)li), ed = __fsub_rn(at, (float)ldi);
        const float cl = __fmaf_rn(q2, __fmul_rn(el, el), __fmul_rn(lambda, lut[li]));
        const float cd = __fmaf_rn(q2, __fmul_rn(ed, ed), __fmul_rn(lambda, lut[ldi]));
        dn = cd < cl;
      } else {
        dn = round_down_plain(at, uabs(c), q2, lambda);
      }
      if (dn) cf[rc] = (Coef)(c < 0 ? c + 1 : c - 1);
    }
  }
  g.sync();  // the flags are read
  float* S = reinterpret_cast<float*>(w.t);
  float* B = w.a;
  float* R = w.tf;
  for (int x = 0; x <= xmax; x++) {
    const int rc = x * N + j, e = scan_index<N>(x, j);
    if (e < m) {
      const float at = fabsf(w.tf[rc]), q2 = rc == 0 ? dq2 : aq2;
      const float ecur = __fsub_rn(at, (float)uabs(cf[rc]));
      S[e] = __fmul_rn(q2, __fmul_rn(at, at));
      B[e] = __fmul_rn(q2, __fmul_rn(ecur, ecur));
    }
  }
  g.sync();  // the targets are read
  for (int x = 0; x <= xmax; x++) {
    const int e = scan_index<N>(x, j);
    if (e < m) {
      const uint32_t l = uabs(cf[x * N + j]);
      R[e] = __fmul_rn(lambda, l < 64 ? lut[l] : coef_rate_bits(l));
    }
  }
  g.sync();
  // lane 0: S[e] = the sum of S from m - 1 down to e; lane 1: B[e] += the
  // running cost before it, which then takes R[e] too
  if (j < 2) {
    if (j == 0) S[m] = 0.0f;
    float* arr = j == 0 ? S : B;
    float acc = 0.0f;
    int s = 0;
    for (; s + 8 <= m; s += 8) {
      float v[8], r[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        v[u] = arr[j == 0 ? m - 1 - (s + u) : s + u];
        r[u] = j == 0 ? 0.0f : R[s + u];
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const float x = __fadd_rn(acc, v[u]);
        arr[j == 0 ? m - 1 - (s + u) : s + u] = x;
        acc = __fadd_rn(x, r[u]);
      }
    }
    for (; s < m; s++) {
      const int e = j == 0 ? m - 1 - s : s;
      const float x = __fadd_rn(acc, arr[e]);
      arr[e] = x;
      acc = __fadd_rn(x, j == 0 ? 0.0f : R[e]);
    }
  }
  g.sync();
  float best = __int_as_float(0x7f800000);
  int best_e = NN;
  for (int x = 0; x <= xmax; x++) {
    const int e = scan_index<N>(x, j);
    if (e < m && cf[x * N + j] != 0) {
      const int bin = e < 2 ? e : 32 - __clz(e);
      const int extra = bin > 1 ? bin - 2 : 0;
      const float sig = __fadd_rn(__fmul_rn((float)bin, 0.9f), __fadd_rn((float)extra, 2.0f));
      const float c = __fadd_rn(__fadd_rn(B[e], __fmul_rn(lambda, sig)), S[e + 1]);
      if (c < best) {  // rising e: the first one on ties; never an infinite cost
        best = c;
        best_e = e;
      }
    }
  }
#pragma unroll
  for (int s = N / 2; s; s >>= 1) {
    const float oc = __shfl_xor_sync(kFull, best, s);
    const int oe = __shfl_xor_sync(kFull, best_e, s);
    if (oc < best || (oc == best && oe < best_e)) {
      best = oc;
      best_e = oe;
    }
  }
  const float skip = __fadd_rn(S[0], lambda);
  const int keep = (m == 0 || best_e == NN || skip < best) ? 0 : best_e + 1;
  for (int x = 0; x <= xmax; x++) {
    const int e = scan_index<N>(x, j);
    if (e >= keep && e < m) cf[x * N + j] = 0;
  }
  g.sync();
  return keep - 1;
}

// Dequantisation and inverse transform of w.cf (inv8x8 / inv16x16; TX_32X32
// halves the masked product, src/idct.rs:2281-2320), the reconstruction clamp(pred + inverse) into w.rec() and the error against
// the displayed part (vw x vh) of the source, 0 past it, into w.tf (int32,
// row-major).
template <int N, typename W>
__device__ __forceinline__ void lane_inv_err(const uint16_t* __restrict__ src, int stride, int tx, const mt_quant& q,
                                             const uint8_t* qm, int vw, int vh, int32_t maxv, W& w,
                                             const Lanes<N>& g) {
  const int j = g.j;
  const bool idtx = N != 32 && tx == MT_TX_IDTX;
  const bool one = N == 8 && (tx == MT_TX_V_DCT || tx == MT_TX_H_DCT);
  const uint8_t* wq = idtx || one ? nullptr : qm;
  const bool col_adst = N != 32 && (tx == MT_TX_ADST_ADST || tx == MT_TX_ADST_DCT);
  const bool row_adst = N != 32 && (tx == MT_TX_ADST_ADST || tx == MT_TX_DCT_ADST);
#pragma unroll 4
  for (int u = 0; u < N; u++) {
    const int rc = u * N + j;
    const int32_t l = w.cf[rc];
    const int32_t base = rc == 0 ? q.dc_q : q.ac_q;
    const int32_t step = wq ? ((base * (int32_t)wq[rc] + 16) >> 5) : base;
    int32_t mag = (int32_t)((uabs(l) * (uint32_t)step) & 0xffffffu);
    if constexpr (N == 32) mag >>= 1;
    mag = ::min(mag, q.cf_max + (l < 0 ? 1 : 0));
    w.t[j * (N + 1) + u] = l == 0 ? 0 : (l < 0 ? -mag : mag);
  }
  int32_t v[N];
#pragma unroll
  for (int u = 0; u < N; u++) v[u] = w.t[j * (N + 1) + u];
  auto pass = [&](bool adst, int32_t mn, int32_t mx) {
    if constexpr (N == 32) {
      idct32s(v, 1, mn, mx);
    } else if constexpr (N == 16) {
      if (adst) iadst16s(v, 1, mn, mx); else idct16s(v, 1, mn, mx);
    } else {
      if (adst) iadst8s(v, 1, mn, mx); else idct8s(v, 1, mn, mx);
    }
  };
  auto ident = [](int32_t x) { return N == 8 ? 2 * x : 2 * x + ((x * 1697 + 1024) >> 11); };
#pragma unroll 1
  for (int ps = 0; ps < 2; ps++) {  // rows, columns
    if (idtx || (one && tx == (ps ? MT_TX_H_DCT : MT_TX_V_DCT))) {
#pragma unroll
      for (int u = 0; u < N; u++) v[u] = ident(v[u]);
    } else {
      pass(ps ? col_adst : row_adst, ps ? q.cmin : q.rmin, ps ? q.cmax : q.rmax);
    }
    if (ps == 0) {
#pragma unroll
      for (int u = 0; u < N; u++)
        w.t[j * (N + 1) + u] = clampi(N == 8 ? (v[u] + 1) >> 1 : (v[u] + 2) >> 2, q.cmin, q.cmax);
      g.sync();
#pragma unroll
      for (int y = 0; y < N; y++) v[y] = w.t[y * (N + 1) + j];
    }
  }
  int32_t* err = reinterpret_cast<int32_t*>(w.tf);
  int16_t* rec = w.rec();
#pragma unroll
  for (int y = 0; y < N; y++) w.t[y * (N + 1) + j] = v[y];  // the lane's own column
#pragma unroll 4
  for (int y = 0; y < N; y++) {
    const int32_t r = clampi((int32_t)w.pred[y * N + j] + (int16_t)((w.t[y * (N + 1) + j] + 8) >> 4), 0, maxv);
    rec[y * N + j] = (int16_t)r;
    err[y * N + j] = j < vw && y < vh ? (int32_t)src[(size_t)y * stride + j] - r : 0;
  }
  g.sync();
}

// sse_recon_block of the error block that lane_inv_err left.
template <int N, typename W>
__device__ __forceinline__ long long lane_sse(const W& w, int vw, int vh, float scale, const Lanes<N>& g) {
  const int32_t* err = reinterpret_cast<const int32_t*>(w.tf);
  const int j = g.j;
  if (!(scale > 0.0f)) {  // the same for every block of a launch
    long long s = 0;
#pragma unroll 8
    for (int y = 0; y < N; y++) {
      const long long v = err[y * N + j];
      s += v * v;
    }
    return g.sum(s);
  }
  // Lane (k, ln) holds accumulators of row-transform index k and tile-pair lane
  // ln: 32 of them, 32 / N per lane (k, k + N / 8, ...).
  constexpr int K = 32 / N, KS = N / 8;
  const int pw = (::max(vw, 0) + 3) & ~3, ph = (::max(vh, 0) + 3) & ~3;
  const int pairs = pw & ~7;
  const int ln = j & 7, l = j & 3, lane4 = (int)(threadIdx.x & 31u) & ~3;
  float tot[K];
  float D[K][4], Wt[K], Dl[4];
#pragma unroll
  for (int i = 0; i < 4; i++) Dl[i] = kWsseD[l][i];
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int k = (j >> 3) + i * KS;
    tot[i] = 0.0f;
    Wt[i] = kWsseW[k][l];
#pragma unroll
    for (int r = 0; r < 4; r++) D[i][r] = kWsseD[k][r];
  }
#pragma unroll 1
  for (int r0 = 0; r0 < N; r0 += 4)
#pragma unroll 2
    for (int c0 = 0; c0 < N; c0 += 8) {
      // tile pairs past the displayed part add exact zeros
      float e[4];
#pragma unroll
      for (int r = 0; r < 4; r++) e[r] = c0 < pairs ? (float)err[(r0 + r) * N + c0 + ln] : 0.0f;
#pragma unroll
      for (int i = 0; i < K; i++) {
        float v = __fmul_rn(e[0], D[i][0]);
        v = __fmaf_rn(e[1], D[i][1], v);
        v = __fmaf_rn(e[2], D[i][2], v);
        v = __fmaf_rn(e[3], D[i][3], v);
        float c = __fmul_rn(Dl[0], __shfl_sync(kFull, v, lane4));
        c = __fmaf_rn(Dl[1], __shfl_sync(kFull, v, lane4 + 1), c);
        c = __fmaf_rn(Dl[2], __shfl_sync(kFull, v, lane4 + 2), c);
        c = __fmaf_rn(Dl[3], __shfl_sync(kFull, v, lane4 + 3), c);
        tot[i] = __fmaf_rn(__fmul_rn(Wt[i], c), c, tot[i]);
      }
    }
#pragma unroll
  for (int i = 0; i < K; i++) tot[i] = __fadd_rn(tot[i], __shfl_xor_sync(kFull, tot[i], 4));
  float sum;
  if constexpr (N == 32) {
    sum = __fadd_rn(tot[0], __shfl_xor_sync(kFull, tot[0], 8));
    sum = __fadd_rn(sum, __shfl_xor_sync(kFull, sum, 16));
  } else if constexpr (N == 16) {
    const float s0 = __fadd_rn(tot[0], __shfl_xor_sync(kFull, tot[0], 8));
    const float s1 = __fadd_rn(tot[1], __shfl_xor_sync(kFull, tot[1], 8));
    sum = __fadd_rn(s0, s1);
  } else {
    sum = __fadd_rn(__fadd_rn(tot[0], tot[1]), __fadd_rn(tot[2], tot[3]));
  }
  const bool tail = pairs < pw;
  if (__any_sync(kFull, tail)) {  // the 4-wide tail tiles, into the four sums
#pragma unroll 1
    for (int r0 = 0; r0 < N; r0 += 4) {
      float e[4];
#pragma unroll
      for (int r = 0; r < 4; r++) e[r] = tail && r0 < ph ? (float)err[(r0 + r) * N + pairs + l] : 0.0f;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        float v = __fmul_rn(e[0], kWsseD[k][0]);
        v = __fmaf_rn(e[1], kWsseD[k][1], v);
        v = __fmaf_rn(e[2], kWsseD[k][2], v);
        v = __fmaf_rn(e[3], kWsseD[k][3], v);
        float c = __fmul_rn(Dl[0], __shfl_sync(kFull, v, lane4));
        c = __fmaf_rn(Dl[1], __shfl_sync(kFull, v, lane4 + 1), c);
        c = __fmaf_rn(Dl[2], __shfl_sync(kFull, v, lane4 + 2), c);
        c = __fmaf_rn(Dl[3], __shfl_sync(kFull, v, lane4 + 3), c);
        sum = __fmaf_rn(__fmul_rn(kWsseW[k][l], c), c, sum);
      }
    }
  }
  const float s2 = __fadd_rn(sum, __shfl_xor_sync(kFull, sum, 2));
  const float d = __fadd_rn(s2, __shfl_xor_sync(kFull, s2, 1));
  return vw <= 0 || vh <= 0 ? 0 : __float2ll_rz(roundf(__fmul_rn(d, scale)));
}

// rate_bounded<N> over the block's lanes: the terms of the reverse walk are
// compacted in its order over tf | a | t, then lane 0 adds them.  eob: the
// block's last nonzero scan index (-1: none).  BOUNDED: a block leaves with
// +inf where the one-thread walk does.  Every lane gets the bits.
template <int N, bool BOUNDED, typename W>
__device__ __forceinline__ float lane_rate(W& w, int eob, const mt_coef_costs& T, int skip_ctx, int dcs, int mode,
                                           int tx, bool use_skip_bits, float skip1, float skip0, float bound,
                                           const Lanes<N>& g) {
  constexpr int NN = N * N;
  const int j = g.j;
  const auto* cf = w.cf;
  const int E = warp_max_all(eob);
  int nterm = 0, ac_nz = 1;
  if (E > 0) {
    float* P = reinterpret_cast<float*>(&w);  // tf | a | t
    const uint8_t* lv = w.lv;
    lane_level_map<N>(w, g);
    g.sync();
    for (int d = diag_of<N>(E); d >= 1; d--) {
      const int lo = ::max(0, d - (N - 1)), len = ::min(d + 1, 2 * N - 1 - d);
      // lanes in the walk's order: falling scan index
      const int kk = len - 1 - j;
      const int i = diag_base<N>(d) + kk;
      const bool act = kk >= 0 && i < eob;
      const int p = lo + kk, x = (d & 1) ? d - p : p, y = d - x;
      uint32_t m = 0;
      float t1 = 0.0f, t2 = 0.0f, t3 = 0.0f;
      if (act) {
        const int rc = x * N + y;
        // the walk's map holds the positions already walked: not those that
        // follow a column's end, which have lower scan indexes
        const uint32_t n1 = y + 1 < N ? lv[rc + 1] : 0u, n9 = y + 1 < N ? lv[rc + N + 1] : 0u;
        const uint32_t hm = n1 + lv[rc + N] + n9;
        const uint32_t mag = hm + (y + 2 < N ? lv[rc + 2] : 0u) + lv[rc + 2 * N];
        const int ctx = lo_ctx_off(x + y) + (mag > 512 ? 4 : (int)((mag + 64) >> 7));
        m = uabs(cf[rc]);
        t1 = T.base_tok[ctx][::min(m, 3u)];
        if (m >= 3) {
          const uint32_t hmag = hm & 63;
          const int bc = ((y | x) > 1 ? 14 : 7) + (hmag > 12 ? 6 : (int)((hmag + 1) >> 1));
          t2 = T.br_cum[bc][::min((int32_t)m - 3, 12)];
          if (m >= 15) t3 = golomb_cost(m - 15);
        }
      }
      const unsigned lt = (1u << j) - 1u;
      const unsigned b1 = g.ballot(act), b2 = g.ballot(m >= 3), b3 = g.ballot(m >= 15);
      ac_nz += __popc(g.ballot(m != 0));
      if (act) {
        const int o = nterm + __popc(b1 & lt) + __popc(b2 & lt) + __popc(b3 & lt);
        P[o] = t1;
        if (m >= 3) P[o + 1] = t2;
        if (m >= 15) P[o + 2] = t3;
        if (BOUNDED && (i & 15) == 0) w.ck[i >> 4] = (uint16_t)o;
      }
      nterm += __popc(b1) + __popc(b2) + __popc(b3);
    }
    g.sync();
  }
  float bits = 0.0f;
  if (j == 0) {
    if (eob < 0) {
      bits = use_skip_bits ? skip1 : T.txb_skip[skip_ctx][1];
    } else {
      bits = use_skip_bits ? skip0 : T.txb_skip[skip_ctx][0];
      if (tx >= 0) bits = __fadd_rn(bits, T.txtp[mode][tx]);
      const uint32_t dm = uabs(cf[0]);
      const float* dcs_c = T.dc_sign[dcs];
      if (eob == 0) {
        bits = __fadd_rn(bits, T.eob_bin[0]);
        bits = __fadd_rn(bits, T.eob_base[0][::min(dm, 3u) - 1]);
        if (dm >= 3) bits = __fadd_rn(bits, hi_cost(T, dm, 0));
        bits = __fadd_rn(bits, dcs_c[cf[0] < 0]);
      } else {
        const int eob_bin = eob < 2 ? eob : 32 - __clz(eob);
        bits = __fadd_rn(bits, T.eob_bin[eob_bin]);
        if (eob_bin > 1) {
          const int nb = eob_bin - 2;
          bits = __fadd_rn(bits, T.eob_hi[eob_bin][(eob >> nb) & 1]);
          bits = __fadd_rn(bits, (float)nb);
        }
        bool out = BOUNDED && bits > bound;
        const int rc = scan_rc<N>(eob);
        const uint32_t me = uabs(cf[rc]);
        bits = __fadd_rn(bits, T.eob_base[1 + (eob > (NN >> 3)) + (eob > (NN >> 2))][::min(me, 3u) - 1]);
        if (me >= 3) bits = __fadd_rn(bits, hi_cost(T, me, ((rc >> log2w<N>()) | (rc & (N - 1))) > 1 ? 14 : 7));
        const float* P = reinterpret_cast<const float*>(&w);
        int o = 0;
        auto add_to = [&](int end) {
          for (; o + 8 <= end; o += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = P[o + u];
#pragma unroll
            for (int u = 0; u < 8; u++) bits = __fadd_rn(bits, v[u]);
          }
          for (; o < end; o++) bits = __fadd_rn(bits, P[o]);
        };
        if (BOUNDED) {
          for (int i = (eob - 1) & ~15; i >= 16 && !out; i -= 16) {
            add_to(w.ck[i >> 4]);
            out = bits > bound;
          }
        }
        if (out) {
          bits = __int_as_float(0x7f800000);
        } else {
          add_to(nterm);
          bits = __fadd_rn(bits, T.base_tok[0][::min(dm, 3u)]);
          if (dm >= 3) {
            const uint32_t mag = ((uint32_t)w.lv[1] + w.lv[N] + w.lv[N + 1]) & 63;
            bits = __fadd_rn(bits, hi_cost(T, dm, mag > 12 ? 6 : (int)((mag + 1) >> 1)));
          }
          if (dm != 0) bits = __fadd_rn(bits, dcs_c[cf[0] < 0]);
          bits = add_ones(bits, ac_nz);
        }
      }
    }
  }
  bits = g.from(bits, 0);
  g.sync();
  return bits;
}

// Stages the tables of a launch: the cost slice, the QM weights (32 = flat)
// and the forward scale of each weight value.
template <int NN>
struct LaneTables {
  mt_coef_costs T;
  float qs[256];
  uint8_t qm[NN];
  __device__ __forceinline__ void load(const mt_coef_costs* __restrict__ costs, const uint8_t* __restrict__ qm_row,
                                       bool has_qm) {
    const float* s = reinterpret_cast<const float*>(costs);
    float* d = reinterpret_cast<float*>(&T);
    for (int i = threadIdx.x; i < (int)(sizeof(mt_coef_costs) / 4); i += blockDim.x) d[i] = s[i];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) qs[i] = fwd_qm_scale(i ? i : 1);
    for (int i = threadIdx.x; i < NN; i += blockDim.x) qm[i] = has_qm ? qm_row[i] : (uint8_t)32;
    __syncthreads();
  }
};

}  // namespace mtd
