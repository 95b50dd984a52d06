// The leaves' chroma searches, batched over leaves: pick_uv16_420
// (src/coder/block16.rs:980-1381), pick_uv16_444 (:437-978), pick_uv32_420
// (src/coder/block32.rs:2797-3120) and pick_uv32_444 (:2264-2720) with the
// shipped tuning (uv16_joint on, uv8_joint_k 4, cfl_alpha_rd_steps 0).  Each
// leaf runs the DC path, the CfL path (the AC of the leaf's luma
// reconstruction, the closed-form alphas) and the SATD-ranked directional
// stage; every priced candidate goes through the same per-plane chain
// (plane_chain).  A leaf is a CTA, a plane of a candidate N lanes of it.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/maroontree_b200.h"
#include "common.cuh"
#include "lanes.cuh"

namespace mth {
float scaled_trellis_lambda_host(float dc_q, float lambda0);
}

namespace {

using namespace mtd;

constexpr int kJointModes = 12;
constexpr int kMaxJoint = 12;

struct UvArgs {
  mt_split16_params p;  // the chroma planes
  mt_uv16_params u;
  mt_quant q;           // the chroma quantiser
  float lambda;         // scaled_trellis_lambda of the chroma trellis (0: off)
  int has_qm;
};

// The shortlist's modes in the reference's order (block16.rs:1143-1156).
__constant__ uint8_t kJointList[kJointModes] = {MT_SMOOTH_V_PRED, MT_PAETH_PRED, MT_SMOOTH_PRED, MT_SMOOTH_H_PRED,
                                                MT_V_PRED,        MT_H_PRED,     MT_D135_PRED,   MT_D113_PRED,
                                                MT_D157_PRED,     MT_D45_PRED,   MT_D67_PRED,    MT_D203_PRED};

__device__ __forceinline__ bool directional(int m) { return m >= MT_V_PRED && m <= MT_D67_PRED; }

// chroma_tx_for_mode (src/coder/chroma_tx.rs:46-66): dav1d's uv-mode map.
__device__ __forceinline__ int chroma_tx(int m) {
  if (m == MT_PAETH_PRED || m == MT_SMOOTH_PRED || m == MT_D135_PRED) return MT_TX_ADST_ADST;
  if (m == MT_SMOOTH_V_PRED || m == MT_V_PRED || m == MT_D113_PRED || m == MT_D67_PRED) return MT_TX_ADST_DCT;
  if (m == MT_SMOOTH_H_PRED || m == MT_H_PRED || m == MT_D157_PRED || m == MT_D203_PRED) return MT_TX_DCT_ADST;
  return MT_TX_DCT_DCT;
}

__device__ __forceinline__ float rd_cost_i64(long long d, float lam, float rate) {
  return __fadd_rn((float)d, __fmul_rn(lam, rate));
}

// uv_mode_bits (src/coder/lossy_state.rs:1302-1349); cfl: the alphas' form.
__device__ float uv_mode_bits(const mt_uv_mode_costs& C, int y_mode, int uv, bool cfl, int au, int av) {
  if (!cfl) {
    float bits = C.uv_mode[y_mode][uv];
    if (directional(uv)) bits = __fadd_rn(bits, C.angle_delta[uv - MT_V_PRED][3]);
    return bits;
  }
  const int su = au == 0 ? 0 : (au < 0 ? 1 : 2), sv = av == 0 ? 0 : (av < 0 ? 1 : 2);
  const int sign = su * 3 + sv;
  if (sign == 0) return C.uv_mode[y_mode][MT_DC_PRED];
  float bits = __fadd_rn(C.uv_mode[y_mode][MT_UV_CFL_PRED], C.cfl_sign[sign - 1]);
  if (su != 0) bits = __fadd_rn(bits, C.cfl_alpha[(su == 2) * 3 + sv][abs(au) - 1]);
  if (sv != 0) bits = __fadd_rn(bits, C.cfl_alpha[(sv == 2) * 3 + su][abs(av) - 1]);
  return bits;
}

// One plane of a leaf: source / reconstruction origins, displayed extent,
// coefficient contexts.
struct UvPlane {
  const uint16_t* src;  // block origin
  const uint16_t* rec;  // plane base
  int vw, vh;
  int sk, ds;           // txb_skip context 7 + above nz + left nz, dc_sign_ctx_span
  float skip1, skip0;
};

struct PlaneCost {
  long long sse;
  float bits;
};

// The four searches.
enum class UvForm { k16_420, k32_420, k16_444, k32_444 };

// Shape of a search: N the chroma block's side, CTX the context trellis (4:2:0)
// or the plain one (4:4:4), Slots the blocks a CTA evaluates at a time, each on
// N lanes: consecutive slots are U and V of one candidate.
// A leaf is a CTA and its candidates go Slots / 2 at a time: DC and CfL
// together, the ranking's predictions, the ranked modes, the deltas.  Six slots
// of 16x16 (3 warps, 27 KB, 6 CTAs per SM) take the three ranked modes in one
// step and the six deltas in two; at 32x32 six would leave one CTA per SM, four
// (4 warps, 79 KB) leave two.  Eight of 8x8 (2 warps) take the default
// shortlist of four at once.
template <UvForm F>
struct UvShape {
  static constexpr int N = F == UvForm::k16_420 ? 8 : (F == UvForm::k32_444 ? 32 : 16);
  static constexpr bool k420 = F == UvForm::k16_420 || F == UvForm::k32_420;
  static constexpr bool kCtx = k420;
  static constexpr int kSlots = N == 8 ? 8 : (N == 16 ? 6 : 4);
  static constexpr int kThreads = kSlots * N;
  // CTAs per SM that ptxas keeps registers for.  Shared memory decides it for
  // the wider blocks; the 8x8 form would take 117 registers (8 CTAs).  At 1080p
  // 8, 10, 11, 12, 14, 16 CTAs: 939, 907, 870, 872, 891, 917 us (80 registers
  // hold the chain, below that it spills).
  static constexpr int kMinCtas = F == UvForm::k16_420 ? 11 : 1;
};

// One N x N plane of a candidate after its prediction (w.pred): the transform
// with the QM (DCT_DCT only at 32x32), trellis_optimize_ctx against the chroma
// costs in the plane's dc_sign context (CTX) or the plain trellis_optimize (the
// 4:4:4 chroma_rect_trellis), preserve_dc (src/rd_sse.rs:759-765) when
// `keep_dc`, the inverse, sse_recon and chroma_bits.
// Called, not inlined, as is the predictor: a search prices candidates in three
// places, and one copy of the chain in the instruction cache beats three
// (1080p: pick_uv16_444 3.45 -> 2.27 ms, pick_uv32_420 1.11 -> 0.78 ms).
template <int N, bool CTX>
__device__ __noinline__ PlaneCost plane_chain(const UvArgs& a, const UvPlane& P, const LaneTables<N * N>& S,
                                                 const float* lut, int tx, bool keep_dc, LaneBuf<N>& w,
                                                 const Lanes<N>& g) {
  const mt_split16_params& p = a.p;
  const mt_quant& q = a.q;
  const uint8_t* qm = a.has_qm ? S.qm : nullptr;
  const int32_t sum = lane_fwd<N>(P.src, p.stride, tx, q, qm, S.qs, w, g);
  int eob;
  if (a.lambda > 0.0f) {
    if constexpr (CTX)
      eob = lane_trellis_ctx<N>(w, (float)q.dc_q, (float)q.ac_q, a.lambda, S.T, P.ds, qm, q.qm_level >= 5, p.band_tilt,
                                g);
    else
      eob = lane_trellis_plain<N>(w, (float)q.dc_q, (float)q.ac_q, a.lambda, lut, g);
  } else {
    eob = lane_eob<N>(w, g);
  }
  const int32_t mean = sum / (N * N);  // truncating, as the reference's i32 division
  const bool keep = keep_dc && w.cf[0] == 0 && abs(mean) >= 8;
  g.sync();
  if (keep) {
    if (g.j == 0) w.cf[0] = mean > 0 ? 1 : -1;
    eob = max(eob, 0);
  }
  g.sync();
  lane_inv_err<N>(P.src, p.stride, tx, q, qm, P.vw, P.vh, (1 << p.bd) - 1, w, g);
  PlaneCost c;
  c.sse = lane_sse<N>(w, P.vw, P.vh, p.wsse_scale, g);
  c.bits = lane_rate<N, false>(w, eob, S.T, P.sk, P.ds, 0, -1, p.use_skip_bits != 0, P.skip1, P.skip0,
                               __int_as_float(0x7f800000), g);
  return c;
}

// The CfL prediction of a plane into w.pred: the AC of the leaf's luma
// reconstruction at l (4:2:0: the 2x2 sums << 1, cfl_ac_sub; 4:4:4: << 3), less
// its rounded mean, and cfl_best_alpha (src/intrapred.rs:1211-1258) over the
// displayed part: the closed-form alpha, then the first minimum of the
// prediction's SSE over alpha - 3 .. alpha + 3 within +-16.  Returns the alpha.
template <int N, bool SUB>
__device__ __forceinline__ int lane_cfl(const uint16_t* __restrict__ l, int ls, const UvPlane& P, int stride, int32_t dc,
                                        int32_t maxv, LaneBuf<N>& w, const Lanes<N>& g) {
  constexpr int L = log2w<N>();
  const int x = g.j;
  // the lane's column of the AC, over the scratch that the transform takes next:
  // loops a few rows at a time instead of the column in registers (at 32x32 the
  // seven alphas written out were 40 KB of code)
  int32_t* const ac = reinterpret_cast<int32_t*>(w.a) + x;
  int32_t sum = 0;
#pragma unroll 4
  for (int y = 0; y < N; y++) {
    int32_t v;
    if constexpr (SUB) {
      const uint16_t* q = l + (size_t)(2 * y) * ls + 2 * x;
      v = ((int32_t)q[0] + q[1] + q[ls] + q[ls + 1]) << 1;
    } else {
      v = (int32_t)l[(size_t)y * ls + x] << 3;
    }
    ac[y * N] = (int16_t)v;
    sum += v;
  }
  const int32_t mean = (g.sum(sum) + N * N / 2) >> (2 * L);
  const bool vis_x = x < P.vw;
  long long num = 0, den = 0;
#pragma unroll 4
  for (int y = 0; y < N; y++) {
    const int16_t a = (int16_t)(ac[y * N] - mean);
    ac[y * N] = a;
    if (vis_x && y < P.vh) {
      const long long v = a;
      num += (long long)((int32_t)P.src[(size_t)y * stride + x] - dc) * v;
      den += v * v;
    }
  }
  num = g.sum(num);
  den = g.sum(den);
  int alpha = 0;
  const long long sg = num > 0 ? 1 : (num < 0 ? -1 : 0);
  long long a0 = den == 0 ? 0 : (64 * num + (den >> 1) * sg) / den;
  a0 = a0 < -16 ? -16 : (a0 > 16 ? 16 : a0);
  long long e[7];
#pragma unroll
  for (int k = 0; k < 7; k++) e[k] = 0;
#pragma unroll 1
  for (int y = 0; y < N; y++) {
    if (vis_x && y < P.vh) {
      const int32_t a = ac[y * N];
      const int32_t s = P.src[(size_t)y * stride + x];
#pragma unroll
      for (int k = 0; k < 7; k++) {
        const long long d = s - cfl_pred_pixel(dc, a, (int)a0 - 3 + k, maxv);
        e[k] += d * d;
      }
    }
  }
  long long best_e = 0x7fffffffffffffffLL;
#pragma unroll
  for (int k = 0; k < 7; k++) {
    const long long ek = g.sum(e[k]);
    const int c = (int)a0 - 3 + k;
    if (c >= -16 && c <= 16 && ek < best_e) {
      best_e = ek;
      alpha = c;
    }
  }
  if (den == 0) alpha = 0;
#pragma unroll 4
  for (int y = 0; y < N; y++) w.pred[y * N + x] = (int16_t)cfl_pred_pixel(dc, ac[y * N], alpha, maxv);
  g.sync();
  return alpha;
}

// satd_sad_proxy of w.pred over the block's lanes, a 4x4 tile at a time each.
template <int N>
__device__ __forceinline__ unsigned long long lane_satd_sad(const UvPlane& P, int stride, const LaneBuf<N>& w,
                                                            const Lanes<N>& g) {
  uint32_t sad = 0, satd = 0;
  for (int tile = g.j; tile < (N / 4) * (N / 4); tile += N) {
    const int ty = (tile / (N / 4)) * 4, tx = (tile % (N / 4)) * 4;
    int32_t r[4][4];
#pragma unroll
    for (int y = 0; y < 4; y++) {
      int32_t d[4];
#pragma unroll
      for (int x = 0; x < 4; x++) {
        const bool vis = tx + x < P.vw && ty + y < P.vh;
        d[x] = vis ? (int32_t)P.src[(size_t)(ty + y) * stride + tx + x] - w.pred[(ty + y) * N + tx + x] : 0;
        sad += uabs(d[x]);
      }
      const int32_t e = d[0] + d[2], f = d[0] - d[2], gg = d[1] + d[3], h = d[1] - d[3];
      r[y][0] = e + gg;
      r[y][1] = f + h;
      r[y][2] = f - h;
      r[y][3] = e - gg;
    }
#pragma unroll
    for (int x = 0; x < 4; x++) {
      const int32_t e = r[0][x] + r[2][x], f = r[0][x] - r[2][x], gg = r[1][x] + r[3][x], h = r[1][x] - r[3][x];
      satd += uabs(e + gg) + uabs(f + h) + uabs(f - h) + uabs(e - gg);
    }
  }
  return (unsigned long long)g.sum((unsigned long long)sad) + (g.sum((unsigned long long)satd) >> 2);
}

// The prediction of (mode, delta) into w.pred.
template <int N>
__device__ __noinline__ void plane_predict(const uint16_t* __restrict__ rec, int stride, int fw, int fh, int cx, int cy,
                                              int mode, int delta, bool tr, bool bl, bool ft, int bd, LaneBuf<N>& w,
                                              const Lanes<N>& g) {
  lane_predict<N>(PlaneRead{rec, stride}, fw, fh, cx, cy, mode, delta, tr, bl, ft, bd, w.pred,
                  reinterpret_cast<int32_t*>(&w), g);
}

// A leaf's chroma search.  Every thread follows the decisions on the costs that
// the slots leave in shared memory; a candidate that wins is written out at
// once, over the winner before it.
// k16_444 is pick_uv16_444 (block16.rs:437-978), k32_444 pick_uv32_444
// (block32.rs:2264-2720): DC, CfL against DC on the chroma lambda (the 16x16
// search on the summed SSE and bits, the 32x32 one on the planes' costs), the
// 12 modes ranked by SATD into a top-3 priced in list order on dir_lambda, the
// zone-2 deltas of a directional winner.  k32_420 is pick_uv32_420
// (block32.rs:2797-3120): the same on the one chroma lambda with the context
// trellis, DC's total without mode bits, no deltas after CfL.  k16_420 is
// pick_uv16_420 (block16.rs:980-1381): the joint (mode, delta) shortlist of the
// SATD ranking in place of the top-3 and the deltas.
// Bound by issue, instruction fetch and the chains' latency, HBM is idle.
// Measured at 1080p against a thread per leaf with its working set in shared
// memory (3, 10 or 50 KB, so 55, 21 or 4 leaves per SM): k16_420 2.83 -> 0.87 ms,
// k16_444 25.2 -> 2.1, k32_420 24.2 -> 0.7, k32_444 56 -> 1.72 ms; of that, code
// kept short (one transform for both passes, rows four at a time, CfL's column in
// shared memory; 185 to 350 KB -> 158 to 173) k16_420 1.09 -> 0.94 ms and k32_444
// 2.18 -> 1.72.
template <UvForm F, typename J>
__global__ void __launch_bounds__(UvShape<F>::kThreads, UvShape<F>::kMinCtas) uv_kernel(
    const uint16_t* __restrict__ src_u, const uint16_t* __restrict__ src_v, const uint16_t* __restrict__ rec_u,
    const uint16_t* __restrict__ rec_v, const uint16_t* __restrict__ luma, const __grid_constant__ UvArgs a,
    const uint8_t* __restrict__ qm_row, const mt_coef_costs* __restrict__ costs,
    const mt_uv_mode_costs* __restrict__ mode_costs, const J* __restrict__ jobs, int n,
    mt_uv16_result* __restrict__ res, int32_t* __restrict__ cf_out, uint16_t* __restrict__ rec_out) {
  constexpr int N = UvShape<F>::N, NN = N * N, U = N / 4, kSlots = UvShape<F>::kSlots, kCands = kSlots / 2;
  constexpr bool kCtx = UvShape<F>::kCtx, k420 = UvShape<F>::k420, kJoint = F == UvForm::k16_420;
  __shared__ LaneTables<NN> S;
  __shared__ mt_uv_mode_costs M;
  __shared__ float lut[64];
  __shared__ PlaneCost cost[kCands][2];
  __shared__ int salpha[2];
  __shared__ unsigned long long score[kJoint ? 60 : 12][2];
  __shared__ uint8_t list[kMaxJoint];  // the joint shortlist, as indexes of the ranking
  extern __shared__ __align__(128) unsigned char lane_smem[];
  const int job = blockIdx.x;
  const mt_split16_params& p = a.p;
  const J jb = jobs[job];
  constexpr int kLeaf = k420 ? 2 * N : N;
  const int cx = k420 ? jb.px >> 1 : jb.px, cy = k420 ? jb.py >> 1 : jb.py;
  const bool ok = (jb.px & (kLeaf - 1)) == 0 && (jb.py & (kLeaf - 1)) == 0 && cx + N <= p.frame_w &&
                  cy + N <= p.frame_h && jb.y_mode <= MT_PAETH_PRED;
  if (!ok) {
    if (threadIdx.x == 0) {
      mt_uv16_result r = {};
      r.total = r.dc_total = r.cfl_total = __int_as_float(0x7f800000);
      r.uv_mode = 255;
      res[job] = r;
    }
    for (int i = threadIdx.x; i < 2 * NN; i += blockDim.x) {
      if (cf_out) cf_out[(size_t)job * 2 * NN + i] = 0;
      if (rec_out) rec_out[(size_t)job * 2 * NN + i] = 0;
    }
    return;
  }
  {
    const float* gm = reinterpret_cast<const float*>(mode_costs);
    float* sm = reinterpret_cast<float*>(&M);
    for (int i = threadIdx.x; i < (int)(sizeof(mt_uv_mode_costs) / 4); i += blockDim.x) sm[i] = gm[i];
    for (int i = threadIdx.x; i < 64; i += blockDim.x) lut[i] = kCoefRateLut[i];
  }
  S.load(costs, qm_row, a.has_qm);
  const Lanes<N> g;
  const int slot = threadIdx.x / N, pl = slot & 1;
  LaneBuf<N>& w = reinterpret_cast<LaneBuf<N>*>(lane_smem)[slot];
  const int32_t maxv = (1 << p.bd) - 1;
  const float mlam = p.rd_lambda, dlam = k420 ? p.rd_lambda : a.u.dir_lambda;
  const bool have_tr = jb.flags & MT_CAND_HAVE_TR, have_bl = jb.flags & MT_CAND_HAVE_BL;
  const bool ft = jb.flags & MT_CAND_FILTER_TYPE;
  const int vis_w = p.vis_w > 0 ? p.vis_w : p.frame_w, vis_h = p.vis_h > 0 ? p.vis_h : p.frame_h;
  UvPlane P;  // this slot's plane
  P.src = (pl ? src_v : src_u) + (size_t)cy * p.stride + cx;
  P.rec = pl ? rec_v : rec_u;
  P.vw = min(max(vis_w - cx, 0), N);
  P.vh = min(max(vis_h - cy, 0), N);
  {
    bool anz = false, lnz = false;
    int s = -2 * U;
    for (int k = 0; k < U; k++) {
      anz |= jb.a_coef[pl][k] != 0x40;
      lnz |= jb.l_coef[pl][k] != 0x40;
      s += (jb.a_coef[pl][k] >> 6) + (jb.l_coef[pl][k] >> 6);
    }
    P.sk = 7 + anz + lnz;       // the chroma txb_skip context over the block's units
    P.ds = (s != 0) + (s > 0);  // dc_sign_ctx_span over U + U units
    P.skip1 = p.use_skip_bits ? p.skip_bits[P.sk][0] : 0.0f;
    P.skip0 = p.use_skip_bits ? p.skip_bits[P.sk][1] : 0.0f;
  }
  auto predict = [&](int m, int d, bool tr, bool bl) {
    plane_predict<N>(P.rec, p.stride, p.frame_w, p.frame_h, cx, cy, m, d, tr, bl, ft, p.bd, w, g);
  };
  // candidate c of the last step becomes the leaf's output
  auto put = [&](int c) {
    if (slot >> 1 != c) return;
    const size_t o = (size_t)job * 2 * NN + pl * NN;
    if (cf_out)
      for (int i = g.j; i < NN; i += N) cf_out[o + i] = w.cf[i];
    if (rec_out)
      for (int i = g.j; i < NN; i += N) rec_out[o + i] = (uint16_t)w.pred[i];
  };
  auto plane_rd = [&](const PlaneCost& c, float lam) { return rd_cost_i64(c.sse, lam, c.bits); };
  // Evaluates one candidate per pair of slots: f(c) predicts candidate c.
  // `step` counts the candidates of this step; the spare slots of a warp that
  // holds a candidate repeat one.
  auto evaluate = [&](int step, auto f) {
    const int c0 = (int)(threadIdx.x & ~31u) / N >> 1;  // the warp's first candidate
    if (c0 < step) {
      const int c = min(slot >> 1, step - 1);
      int tx = MT_TX_DCT_DCT;
      const bool keep_dc = f(c, &tx);
      const PlaneCost pc = plane_chain<N, kCtx>(a, P, S, lut, tx, keep_dc, w, g);
      if (slot >> 1 < step && g.j == 0) cost[slot >> 1][pl] = pc;
    }
    __syncthreads();
  };

  // DC (slots 0, 1) and CfL (slots 2, 3)
  evaluate(2, [&](int c, int*) {
    predict(MT_DC_PRED, 0, have_tr, have_bl);
    const int32_t dc = w.pred[0];
    g.sync();
    if (__any_sync(kFull, c == 1)) {
      // a warp that holds both candidates runs both and keeps DC's prediction
      int16_t flat[N];
#pragma unroll
      for (int y = 0; y < N; y++) flat[y] = (int16_t)dc;
      const int al = lane_cfl<N, k420>(luma + (size_t)jb.py * a.u.luma_stride + jb.px, a.u.luma_stride, P, p.stride, dc,
                                       maxv, w, g);
      if (c == 1) {
        if (g.j == 0 && slot >> 1 == 1) salpha[pl] = al;
      } else {
#pragma unroll
        for (int y = 0; y < N; y++) w.pred[y * N + g.j] = flat[y];
      }
      g.sync();
    }
    return c == 0;  // preserve_dc
  });
  const int au = salpha[0], av = salpha[1];
  const float sig = uv_mode_bits(M, jb.y_mode, MT_UV_CFL_PRED, true, au, av);
  const float dc_bits = uv_mode_bits(M, jb.y_mode, MT_DC_PRED, false, 0, 0);
  float dc_total, cfl_total, best_total;
  bool use_cfl;
  if constexpr (F == UvForm::k16_444) {
    // rd_cost_i64 of the summed SSE and bits (block16.rs:587-597)
    dc_total = rd_cost_i64(cost[0][0].sse + cost[0][1].sse, mlam,
                           __fadd_rn(__fadd_rn(cost[0][0].bits, cost[0][1].bits), dc_bits));
    cfl_total = rd_cost_i64(cost[1][0].sse + cost[1][1].sse, mlam,
                            __fadd_rn(__fadd_rn(cost[1][0].bits, cost[1][1].bits), sig));
    use_cfl = cfl_total < dc_total && (au != 0 || av != 0);
  } else if constexpr (F == UvForm::k32_444) {
    // the planes' rd_cost_i64 summed, then the mode bits (block32.rs:2399-2404)
    dc_total = __fadd_rn(__fadd_rn(plane_rd(cost[0][0], mlam), plane_rd(cost[0][1], mlam)), __fmul_rn(mlam, dc_bits));
    cfl_total = __fadd_rn(__fadd_rn(plane_rd(cost[1][0], mlam), plane_rd(cost[1][1], mlam)), __fmul_rn(mlam, sig));
    use_cfl = cfl_total < dc_total && (au != 0 || av != 0);
  } else {
    // no mode bits in DC's total (block16.rs:999-1046)
    dc_total = __fadd_rn(__fadd_rn(0.0f, plane_rd(cost[0][0], mlam)), plane_rd(cost[0][1], mlam));
    const float body = __fadd_rn(__fadd_rn(0.0f, plane_rd(cost[1][0], mlam)), plane_rd(cost[1][1], mlam));
    cfl_total = __fsub_rn(__fadd_rn(body, __fmul_rn(mlam, sig)), __fmul_rn(mlam, dc_bits));
    use_cfl = (au != 0 || av != 0) && cfl_total < dc_total;
  }
  if constexpr (k420) {
    best_total = use_cfl ? cfl_total : dc_total;
  } else {
    // the directional stage on dir_lambda: the current choice's total, then the ranked modes
    const PlaneCost* cur = cost[use_cfl ? 1 : 0];
    best_total = __fmul_rn(dlam, use_cfl ? sig : dc_bits);
    for (int k = 0; k < 2; k++) best_total = __fadd_rn(best_total, plane_rd(cur[k], dlam));
  }
  put(use_cfl ? 1 : 0);
  int mode = MT_DC_PRED, delta = 0;
  __syncthreads();  // the choice is written and the costs are read

  // the SATD ranking: the 12 modes, or (joint) the directional ones at 7 deltas
  const bool deltas = a.u.angle_deltas;
  const int nrank = kJoint && deltas ? 60 : 12;
  auto ranked = [&](int i, int* m, int* d) {  // entry i of the ranking
    if (nrank == 12) {
      *m = kJointList[i];
      *d = 0;
    } else if (i < 4) {  // the list's first four have no angle
      *m = kJointList[i];
      *d = 0;
    } else {
      *m = kJointList[4 + (i - 4) / 7];
      *d = (i - 4) % 7 - 3;
    }
  };
  for (int b = 0; b < nrank; b += kCands) {
    const int i = min(b + (slot >> 1), nrank - 1);
    int m, d;
    ranked(i, &m, &d);
    predict(m, d, have_tr, have_bl);
    const unsigned long long sc = lane_satd_sad<N>(P, p.stride, w, g);
    if (b + (slot >> 1) < nrank && g.j == 0) score[i][pl] = sc;
    g.sync();  // the prediction is read
  }
  __syncthreads();
  if constexpr (kJoint) {
    // the first joint_k entries by (score, mode, delta), each priced in full
    const int nk = min(min(max(a.u.joint_k, 1), kMaxJoint), nrank);
    for (int i = threadIdx.x; i < nrank; i += blockDim.x) {
      int m, d;
      ranked(i, &m, &d);
      const unsigned long long sc = score[i][0] + score[i][1];
      int before = 0;
      for (int k = 0; k < nrank; k++) {
        int mk, dk;
        ranked(k, &mk, &dk);
        const unsigned long long sk = score[k][0] + score[k][1];
        before += sk < sc || (sk == sc && (mk < m || (mk == m && dk < d)));
      }
      if (before < nk) list[before] = (uint8_t)i;
    }
    __syncthreads();
    for (int b = 0; b < nk; b += kCands) {
      const int step = min(kCands, nk - b);
      evaluate(step, [&](int c, int* tx) {
        int m, d;
        ranked(list[b + c], &m, &d);
        *tx = chroma_tx(m);
        predict(m, d, have_tr, have_bl);
        return true;
      });
      int win = -1;
      for (int c = 0; c < step; c++) {
        int m, d;
        ranked(list[b + c], &m, &d);
        float ad_bits = 0.0f;
        if (directional(m)) ad_bits = __fsub_rn(M.angle_delta[m - MT_V_PRED][d + 3], M.angle_delta[m - MT_V_PRED][3]);
        float total = __fmul_rn(mlam, __fadd_rn(uv_mode_bits(M, jb.y_mode, m, false, 0, 0), ad_bits));
        total = __fadd_rn(total, plane_rd(cost[c][0], mlam));
        // once U's total reaches the best, V is not looked at
        if (!(total >= best_total)) total = __fadd_rn(total, plane_rd(cost[c][1], mlam));
        if (total < best_total) {
          best_total = total;
          mode = m;
          delta = d;
          use_cfl = false;
          win = c;
        }
      }
      if (win >= 0) put(win);
      __syncthreads();
    }
  } else {
    // rank_chroma_modes (superblock.rs:469-513) into DirectionalTopK
    // (coder.rs:326-365), K = 3: earlier list entries win ties; priced in list order
    uint32_t top = 0;
    {
      unsigned long long tc[3];
      int ti[3], tn = 0;
      for (int i = 0; i < 12; i++) {
        const unsigned long long sc = score[i][0] + score[i][1];
        if (tn == 3 && sc >= tc[2]) continue;
        int pos = tn < 3 ? tn++ : 2;
        for (; pos > 0 && sc < tc[pos - 1]; pos--) {
          tc[pos] = tc[pos - 1];
          ti[pos] = ti[pos - 1];
        }
        tc[pos] = sc;
        ti[pos] = i;
      }
      for (int k = 0; k < tn; k++) top |= 1u << ti[k];
    }
    auto top_mode = [&](int c) { return (int)kJointList[__fns(top, 0, c + 1)]; };
    for (int b = 0; b < 3; b += kCands) {
      const int step = min(kCands, 3 - b);
      evaluate(step, [&](int c, int* tx) {
        const int m = top_mode(b + c);
        *tx = N == 32 ? MT_TX_DCT_DCT : chroma_tx(m);  // forced DCT_DCT at TX_32X32
        predict(m, 0, have_tr, have_bl);
        return true;
      });
      int win = -1;
      for (int c = 0; c < step; c++) {
        const int m = top_mode(b + c);
        float total = __fmul_rn(dlam, uv_mode_bits(M, jb.y_mode, m, false, 0, 0));
        for (int k = 0; k < 2; k++) total = __fadd_rn(total, plane_rd(cost[c][k], dlam));
        if (total < best_total) {
          best_total = total;
          mode = m;
          if (k420) use_cfl = false;
          win = c;
        }
      }
      if (win >= 0) put(win);
      __syncthreads();
    }
    // the zone-2 angle deltas of a directional winner (uv_ad; uv_ad32 at 32x32)
    if (!(k420 && use_cfl) && deltas && directional(mode)) {
      const int m = mode, tx0 = N == 32 ? MT_TX_DCT_DCT : chroma_tx(m);
      int lo = 0, nd = 0;  // deltas lo, lo + 1, ... without 0
      if (m == MT_V_PRED) lo = 1, nd = 3;
      else if (m == MT_H_PRED) lo = -3, nd = 3;
      else if (m == MT_D113_PRED || m == MT_D135_PRED || m == MT_D157_PRED) lo = -3, nd = 6;
      auto nth = [&](int i) { return lo + i + (lo < 0 && lo + i >= 0); };
      const float base_sig = __fsub_rn(uv_mode_bits(M, jb.y_mode, m, false, 0, 0), M.angle_delta[m - MT_V_PRED][3]);
      for (int b = 0; b < nd; b += kCands) {
        const int step = min(kCands, nd - b);
        evaluate(step, [&](int c, int* tx) {
          *tx = tx0;
          predict(m, nth(b + c), false, false);
          return true;
        });
        int win = -1;
        for (int c = 0; c < step; c++) {
          const int d = nth(b + c);
          float total = __fmul_rn(dlam, __fadd_rn(base_sig, M.angle_delta[m - MT_V_PRED][d + 3]));
          for (int k = 0; k < 2; k++) total = __fadd_rn(total, plane_rd(cost[c][k], dlam));
          if (total < best_total) {
            best_total = total;
            delta = d;
            win = c;
          }
        }
        if (win >= 0) put(win);
        __syncthreads();
      }
    }
  }
  if (threadIdx.x == 0) {
    mt_uv16_result r;
    r.total = best_total;
    r.dc_total = dc_total;
    r.cfl_total = cfl_total;
    r.uv_mode = (uint8_t)(mode != MT_DC_PRED ? mode : (use_cfl ? MT_UV_CFL_PRED : MT_DC_PRED));
    r.angle_delta = (int8_t)delta;
    r.cfl_alpha[0] = (int8_t)au;
    r.cfl_alpha[1] = (int8_t)av;
    res[job] = r;
  }
}

int uv_check(const mt_split16_params* p, const mt_uv16_params* u, const mt_quant* q, int32_t n) {
  if (!p || !u || !q || n < 0) return MT_ERR_INVALID_INPUT;
  if (p->bd != 8) return MT_ERR_UNSUPPORTED;
  if (p->frame_w < 8 || p->frame_h < 8 || p->stride < p->frame_w || p->vis_w < 0 || p->vis_h < 0)
    return MT_ERR_INVALID_INPUT;
  if (u->luma_stride < 2 * p->frame_w) return MT_ERR_INVALID_INPUT;
  if (!(p->rd_lambda > 0.0f) || !(p->wsse_scale >= 0.0f)) return MT_ERR_INVALID_INPUT;
  return MT_OK;
}

// 4:4:4: the chroma planes have the luma size, so the luma stride needs only
// the frame width.
int uv_check_444(const mt_split16_params* p, const mt_uv16_params* u, const mt_quant* q, int32_t n) {
  if (!p || !u || !q || n < 0) return MT_ERR_INVALID_INPUT;
  if (p->bd != 8) return MT_ERR_UNSUPPORTED;
  if (p->frame_w < 16 || p->frame_h < 16 || p->stride < p->frame_w || p->vis_w < 0 || p->vis_h < 0)
    return MT_ERR_INVALID_INPUT;
  if (u->luma_stride < p->frame_w) return MT_ERR_INVALID_INPUT;
  if (!(p->rd_lambda > 0.0f) || !(p->wsse_scale >= 0.0f)) return MT_ERR_INVALID_INPUT;
  return MT_OK;
}

size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

template <UvForm F, typename J>
int uv_device(const uint16_t* su, const uint16_t* sv, const uint16_t* ru, const uint16_t* rv, const uint16_t* luma,
              const mt_split16_params* prm, const mt_uv16_params* uvp, const mt_quant* quant, const uint8_t* d_qm,
              const mt_coef_costs* d_costs, const mt_uv_mode_costs* d_mc, const J* d_jobs, int32_t n,
              mt_uv16_result* d_res, int32_t* d_cf, uint16_t* d_rec, void* stream) {
  using Shape = UvShape<F>;
  const int rc = Shape::k420 ? uv_check(prm, uvp, quant, n) : uv_check_444(prm, uvp, quant, n);
  if (rc != MT_OK) return rc;
  if (n == 0) return MT_OK;
  if (!su || !sv || !ru || !rv || !luma || !d_costs || !d_mc || !d_jobs || !d_res) return MT_ERR_INVALID_INPUT;
  if (!Shape::k420 && (!(uvp->dir_lambda > 0.0f) || prm->frame_w < Shape::N || prm->frame_h < Shape::N))
    return MT_ERR_INVALID_INPUT;
  UvArgs a;
  a.p = *prm;
  a.u = *uvp;
  a.q = *quant;
  a.lambda = prm->trellis_lambda0 > 0.0f ? mth::scaled_trellis_lambda_host((float)quant->dc_q, prm->trellis_lambda0)
                                         : 0.0f;
  a.has_qm = quant->qm_level < 15 && d_qm != nullptr;
  auto* kern = uv_kernel<F, J>;
  constexpr size_t dyn = sizeof(LaneBuf<Shape::N>) * Shape::kSlots;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn) != cudaSuccess)
    return MT_ERR_DEVICE;
  kern<<<(unsigned)n, Shape::kThreads, dyn, reinterpret_cast<cudaStream_t>(stream)>>>(
      su, sv, ru, rv, luma, a, d_qm, d_costs, d_mc, d_jobs, n, d_res, d_cf, d_rec);
  return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

// Host-buffer form of either search: the planes, tables and jobs copied to one
// device allocation, the launch, the results (and levels / reconstruction,
// per_job entries each) copied back.
template <typename J, typename L>
int uv_host(const uint16_t* src_u, const uint16_t* src_v, const uint16_t* rec_u, const uint16_t* rec_v,
            const uint16_t* luma, size_t luma_rows, const mt_split16_params* prm, const mt_uv16_params* uvp,
            const mt_quant* quant, const uint8_t* qm_row, size_t qm_len, const mt_coef_costs* costs,
            const mt_uv_mode_costs* mode_costs, const J* jobs, int32_t n, mt_uv16_result* results, int32_t* cf_out,
            uint16_t* rec_out, size_t per_job, L launch) {
  if (!prm || !uvp || !quant || n < 0) return MT_ERR_INVALID_INPUT;
  if (n == 0) return MT_OK;
  if (!src_u || !src_v || !rec_u || !rec_v || !luma || !costs || !mode_costs || !jobs || !results)
    return MT_ERR_INVALID_INPUT;
  if (prm->stride <= 0 || prm->frame_h <= 0 || uvp->luma_stride <= 0) return MT_ERR_INVALID_INPUT;
  const size_t plane = (size_t)prm->stride * prm->frame_h * 2;
  const size_t lplane = (size_t)uvp->luma_stride * luma_rows * 2;
  size_t o = 0;
  const size_t o_su = o, o_sv = (o += up256(plane)), o_ru = (o += up256(plane)), o_rv = (o += up256(plane));
  const size_t o_l = (o += up256(plane)), o_qm = (o += up256(lplane)), o_c = (o += up256(qm_len));
  const size_t o_mc = (o += up256(sizeof(mt_coef_costs))), o_j = (o += up256(sizeof(mt_uv_mode_costs)));
  const size_t o_r = (o += up256((size_t)n * sizeof(J)));
  const size_t o_cf = (o += up256((size_t)n * sizeof(mt_uv16_result)));
  const size_t o_rec = (o += cf_out ? up256((size_t)n * per_job * 4) : 0);
  const size_t total = o + (rec_out ? up256((size_t)n * per_job * 2) : 0);
  uint8_t* d = nullptr;
  if (cudaMalloc(&d, total) != cudaSuccess) return MT_ERR_ALLOC;
  const bool has_qm = quant->qm_level < 15 && qm_row != nullptr;
  cudaError_t e = cudaMemcpy(d + o_su, src_u, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_sv, src_v, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_ru, rec_u, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_rv, rec_v, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_l, luma, lplane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && has_qm) e = cudaMemcpy(d + o_qm, qm_row, qm_len, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_c, costs, sizeof(mt_coef_costs), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_mc, mode_costs, sizeof(mt_uv_mode_costs), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_j, jobs, (size_t)n * sizeof(J), cudaMemcpyHostToDevice);
  int rc = MT_OK;
  if (e == cudaSuccess) {
    auto U = [&](size_t off) { return reinterpret_cast<const uint16_t*>(d + off); };
    rc = launch(U(o_su), U(o_sv), U(o_ru), U(o_rv), U(o_l), has_qm ? d + o_qm : nullptr,
                reinterpret_cast<const mt_coef_costs*>(d + o_c), reinterpret_cast<const mt_uv_mode_costs*>(d + o_mc),
                reinterpret_cast<const J*>(d + o_j), reinterpret_cast<mt_uv16_result*>(d + o_r),
                cf_out ? reinterpret_cast<int32_t*>(d + o_cf) : nullptr,
                rec_out ? reinterpret_cast<uint16_t*>(d + o_rec) : nullptr);
    if (rc == MT_OK) e = cudaMemcpy(results, d + o_r, (size_t)n * sizeof(mt_uv16_result), cudaMemcpyDeviceToHost);
    if (rc == MT_OK && e == cudaSuccess && cf_out)
      e = cudaMemcpy(cf_out, d + o_cf, (size_t)n * per_job * 4, cudaMemcpyDeviceToHost);
    if (rc == MT_OK && e == cudaSuccess && rec_out)
      e = cudaMemcpy(rec_out, d + o_rec, (size_t)n * per_job * 2, cudaMemcpyDeviceToHost);
  }
  cudaFree(d);
  if (rc != MT_OK) return rc;
  return e == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

}  // namespace

extern "C" {

int mt_pick_uv16_420_device(const uint16_t* d_src_u, const uint16_t* d_src_v, const uint16_t* d_rec_u,
                            const uint16_t* d_rec_v, const uint16_t* d_luma, const mt_split16_params* prm,
                            const mt_uv16_params* uvp, const mt_quant* quant, const uint8_t* d_qm_row,
                            const mt_coef_costs* d_costs, const mt_uv_mode_costs* d_mode_costs,
                            const mt_uv16_job* d_jobs, int32_t n, mt_uv16_result* d_results, int32_t* d_cf,
                            uint16_t* d_rec, void* stream) {
  return uv_device<UvForm::k16_420>(d_src_u, d_src_v, d_rec_u, d_rec_v, d_luma, prm, uvp, quant, d_qm_row, d_costs, d_mode_costs,
                     d_jobs, n, d_results, d_cf, d_rec, stream);
}

int mt_pick_uv16_420(const uint16_t* src_u, const uint16_t* src_v, const uint16_t* rec_u, const uint16_t* rec_v,
                     const uint16_t* luma, const mt_split16_params* prm, const mt_uv16_params* uvp,
                     const mt_quant* quant, const uint8_t* qm_row, const mt_coef_costs* costs,
                     const mt_uv_mode_costs* mode_costs, const mt_uv16_job* jobs, int32_t n,
                     mt_uv16_result* results, int32_t* cf_out, uint16_t* rec_out) {
  const int rc = uv_check(prm, uvp, quant, n);
  if (rc != MT_OK) return rc;
  return uv_host(src_u, src_v, rec_u, rec_v, luma, 2 * (size_t)prm->frame_h, prm, uvp, quant, qm_row, 64, costs,
                 mode_costs, jobs, n, results, cf_out, rec_out, 128,
                 [&](const uint16_t* su, const uint16_t* sv, const uint16_t* ru, const uint16_t* rv, const uint16_t* l,
                     const uint8_t* qm, const mt_coef_costs* c, const mt_uv_mode_costs* mc, const mt_uv16_job* j,
                     mt_uv16_result* r, int32_t* cf, uint16_t* rec) {
                   return uv_device<UvForm::k16_420>(su, sv, ru, rv, l, prm, uvp, quant, qm, c, mc, j, n, r, cf, rec, nullptr);
                 });
}

int mt_pick_uv32_444_device(const uint16_t* d_src_u, const uint16_t* d_src_v, const uint16_t* d_rec_u,
                            const uint16_t* d_rec_v, const uint16_t* d_luma, const mt_split16_params* prm,
                            const mt_uv16_params* uvp, const mt_quant* quant, const uint8_t* d_qm_row,
                            const mt_coef_costs* d_costs, const mt_uv_mode_costs* d_mode_costs,
                            const mt_uv32_444_job* d_jobs, int32_t n, mt_uv16_result* d_results, int32_t* d_cf,
                            uint16_t* d_rec, void* stream) {
  return uv_device<UvForm::k32_444>(d_src_u, d_src_v, d_rec_u, d_rec_v, d_luma, prm, uvp, quant, d_qm_row, d_costs,
                          d_mode_costs, d_jobs, n, d_results, d_cf, d_rec, stream);
}

int mt_pick_uv32_444(const uint16_t* src_u, const uint16_t* src_v, const uint16_t* rec_u, const uint16_t* rec_v,
                     const uint16_t* luma, const mt_split16_params* prm, const mt_uv16_params* uvp,
                     const mt_quant* quant, const uint8_t* qm_row, const mt_coef_costs* costs,
                     const mt_uv_mode_costs* mode_costs, const mt_uv32_444_job* jobs, int32_t n,
                     mt_uv16_result* results, int32_t* cf_out, uint16_t* rec_out) {
  const int rc = uv_check_444(prm, uvp, quant, n);
  if (rc != MT_OK) return rc;
  if (n > 0 && !(uvp->dir_lambda > 0.0f)) return MT_ERR_INVALID_INPUT;
  return uv_host(src_u, src_v, rec_u, rec_v, luma, (size_t)prm->frame_h, prm, uvp, quant, qm_row, 1024, costs,
                 mode_costs, jobs, n, results, cf_out, rec_out, 2048,
                 [&](const uint16_t* su, const uint16_t* sv, const uint16_t* ru, const uint16_t* rv, const uint16_t* l,
                     const uint8_t* qm, const mt_coef_costs* c, const mt_uv_mode_costs* mc,
                     const mt_uv32_444_job* j, mt_uv16_result* r, int32_t* cf, uint16_t* rec) {
                   return uv_device<UvForm::k32_444>(su, sv, ru, rv, l, prm, uvp, quant, qm, c, mc, j, n, r, cf, rec, nullptr);
                 });
}

int mt_pick_uv32_420_device(const uint16_t* d_src_u, const uint16_t* d_src_v, const uint16_t* d_rec_u,
                            const uint16_t* d_rec_v, const uint16_t* d_luma, const mt_split16_params* prm,
                            const mt_uv16_params* uvp, const mt_quant* quant, const uint8_t* d_qm_row,
                            const mt_coef_costs* d_costs, const mt_uv_mode_costs* d_mode_costs,
                            const mt_uv32_420_job* d_jobs, int32_t n, mt_uv16_result* d_results, int32_t* d_cf,
                            uint16_t* d_rec, void* stream) {
  return uv_device<UvForm::k32_420>(d_src_u, d_src_v, d_rec_u, d_rec_v, d_luma, prm, uvp, quant, d_qm_row, d_costs, d_mode_costs,
                     d_jobs, n, d_results, d_cf, d_rec, stream);
}

int mt_pick_uv32_420(const uint16_t* src_u, const uint16_t* src_v, const uint16_t* rec_u, const uint16_t* rec_v,
                     const uint16_t* luma, const mt_split16_params* prm, const mt_uv16_params* uvp,
                     const mt_quant* quant, const uint8_t* qm_row, const mt_coef_costs* costs,
                     const mt_uv_mode_costs* mode_costs, const mt_uv32_420_job* jobs, int32_t n,
                     mt_uv16_result* results, int32_t* cf_out, uint16_t* rec_out) {
  const int rc = uv_check(prm, uvp, quant, n);
  if (rc != MT_OK) return rc;
  return uv_host(src_u, src_v, rec_u, rec_v, luma, 2 * (size_t)prm->frame_h, prm, uvp, quant, qm_row, 256, costs,
                 mode_costs, jobs, n, results, cf_out, rec_out, 512,
                 [&](const uint16_t* su, const uint16_t* sv, const uint16_t* ru, const uint16_t* rv, const uint16_t* l,
                     const uint8_t* qm, const mt_coef_costs* c, const mt_uv_mode_costs* mc,
                     const mt_uv32_420_job* j, mt_uv16_result* r, int32_t* cf, uint16_t* rec) {
                   return uv_device<UvForm::k32_420>(su, sv, ru, rv, l, prm, uvp, quant, qm, c, mc, j, n, r, cf, rec, nullptr);
                 });
}

int mt_pick_uv16_444_device(const uint16_t* d_src_u, const uint16_t* d_src_v, const uint16_t* d_rec_u,
                            const uint16_t* d_rec_v, const uint16_t* d_luma, const mt_split16_params* prm,
                            const mt_uv16_params* uvp, const mt_quant* quant, const uint8_t* d_qm_row,
                            const mt_coef_costs* d_costs, const mt_uv_mode_costs* d_mode_costs,
                            const mt_uv16_444_job* d_jobs, int32_t n, mt_uv16_result* d_results, int32_t* d_cf,
                            uint16_t* d_rec, void* stream) {
  return uv_device<UvForm::k16_444>(d_src_u, d_src_v, d_rec_u, d_rec_v, d_luma, prm, uvp, quant, d_qm_row, d_costs,
                          d_mode_costs, d_jobs, n, d_results, d_cf, d_rec, stream);
}

int mt_pick_uv16_444(const uint16_t* src_u, const uint16_t* src_v, const uint16_t* rec_u, const uint16_t* rec_v,
                     const uint16_t* luma, const mt_split16_params* prm, const mt_uv16_params* uvp,
                     const mt_quant* quant, const uint8_t* qm_row, const mt_coef_costs* costs,
                     const mt_uv_mode_costs* mode_costs, const mt_uv16_444_job* jobs, int32_t n,
                     mt_uv16_result* results, int32_t* cf_out, uint16_t* rec_out) {
  const int rc = uv_check_444(prm, uvp, quant, n);
  if (rc != MT_OK) return rc;
  if (n > 0 && !(uvp->dir_lambda > 0.0f)) return MT_ERR_INVALID_INPUT;
  return uv_host(src_u, src_v, rec_u, rec_v, luma, (size_t)prm->frame_h, prm, uvp, quant, qm_row, 256, costs,
                 mode_costs, jobs, n, results, cf_out, rec_out, 512,
                 [&](const uint16_t* su, const uint16_t* sv, const uint16_t* ru, const uint16_t* rv, const uint16_t* l,
                     const uint8_t* qm, const mt_coef_costs* c, const mt_uv_mode_costs* mc,
                     const mt_uv16_444_job* j, mt_uv16_result* r, int32_t* cf, uint16_t* rec) {
                   return uv_device<UvForm::k16_444>(su, sv, ru, rv, l, prm, uvp, quant, qm, c, mc, j, n, r, cf, rec, nullptr);
                 });
}

}  // extern "C"
