// The leaf luma searches, batched: pick_block8's (src/coder/block8.rs:689-1420),
// pick_luma16's and pick_luma32's Slow mode-loop candidates and winner
// transform-type refinements (leaf_lanes_kernel, N lanes per job), and the 64x64
// leaf's two legs (leaf64_kernel).
// The stages are the split trial's (leaf8.cuh, over lanes in lanes.cuh):
// DCT_DCT + QM with trellis_optimize_ctx, the dav1d inverse, sse_recon, the
// bounded 2-D and the 1-D rate walks; every type runs through one loop body.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../../include/maroontree_b200.h"
#include "lanes.cuh"
#include "leaf8.cuh"
#include "wsse.cuh"

namespace mth {
float scaled_trellis_lambda_host(float dc_q, float lambda0);
}

namespace {

using namespace mtd;

struct LeafArgs {
  mt_split16_params p;
  mt_quant q;
  float lambda;  // scaled_trellis_lambda (0: no trellis)
  int has_qm;
};

__device__ __forceinline__ float rd_cost_i64(long long d, float lam, float rate) {
  return __fadd_rn((float)d, __fmul_rn(lam, rate));
}

// Blocks per CTA of the lane kernels: 32 of 8x8 (8 warps: the tables that a CTA
// stages are a tenth of its work), 8 of 16x16 (4 warps) or 5 of 32x32 (5 warps),
// two CTAs of the latter filling an SM's shared memory.
template <int N>
__host__ __device__ constexpr int lane_blocks() {
  return N == 32 ? 5 : (N == 16 ? 8 : 32);
}
template <int N>
__host__ __device__ constexpr int lane_threads() {
  return lane_blocks<N>() * N;
}
// The 16x16 mode loop in large CTAs: two of 24 jobs (12 warps) fill an SM's
// shared memory with 48 jobs, where five of 8 hold 40, and stage a third of the
// tables: 104,520 jobs 1.08 -> 0.86 ms (14 jobs: 1.01), 22,568 jobs 262 -> 244
// us.  Where they would fill the device less than twice, small CTAs spread
// better: 11,440 jobs 146 us in CTAs of 8, 151 of 24; 468 jobs 69 and 76.
constexpr int kModes16 = 24;
template <int N, bool REFINE>
__host__ __device__ constexpr int leaf_max_blocks() {
  return N == 16 && !REFINE ? kModes16 : lane_blocks<N>();
}

// The leaves' mode-loop candidates -- pick_block8's
// (src/coder/block8.rs:738-808), pick_luma16's
// (src/coder/partition_search.rs:4802-4880) and pick_luma32's
// (src/coder/block32.rs:776-836: TX_32X32 DCT_DCT, the only intra type of that
// size, trellis_optimize_ctx of class 3, no tx-type symbol in the rate) -- and
// their winner refinements (REFINE; block8.rs:1183-1404: ADST_ADST, ADST_DCT,
// DCT_ADST, IDTX and, with tx_search, V_DCT and H_DCT;
// partition_search.rs:5252-5474: the first five).  N lanes per job.  A rejected
// job of a warp that holds a good one runs along on the block at the origin and
// writes its rejection.
// Bound by instruction issue and fetch and the diagonals' latency; HBM is idle.
// Measured on the 1080p mode loops, against a thread per job with its working
// set in local memory: 8x8 (421,200 jobs) 1.38 -> 0.98 ms (300x200: 239 -> 60
// us), 16x16 (104,520 jobs) 7.7 -> 0.86 ms, 32x32 (25,740 jobs) 33.0 -> 1.40 ms;
// refinements: 8x8 (32,400 jobs, 7 types) 0.97 -> 0.64 ms (300x200: 796 -> 145
// us), 16x16 (8,040) 3.84 -> 0.72 ms.
template <int N, bool REFINE>
__global__ void __launch_bounds__(leaf_max_blocks<N, REFINE>() * N) leaf_lanes_kernel(
    const uint16_t* __restrict__ src, const uint16_t* __restrict__ rec, LeafArgs a,
    const uint8_t* __restrict__ qm_row, const mt_coef_costs* __restrict__ costs,
    const mt_leaf8_job* __restrict__ jobs, int n, mt_leaf8_result* __restrict__ res, int32_t* __restrict__ cf_out,
    uint16_t* __restrict__ rec_out) {
  static_assert(N != 32 || !REFINE, "32x32 has one transform type");
  constexpr int NN = N * N;
  using Buf = LaneBuf<N, REFINE>;
  __shared__ LaneTables<NN> S;
  extern __shared__ __align__(128) unsigned char lane_smem[];
  S.load(costs, qm_row, a.has_qm);
  const Lanes<N> g;
  Buf& w = reinterpret_cast<Buf*>(lane_smem)[threadIdx.x / N];
  const int job = blockIdx.x * (blockDim.x / N) + threadIdx.x / N;
  const bool live = job < n;
  const mt_split16_params& p = a.p;
  const mt_quant& q = a.q;
  mt_leaf8_job jb = {};
  if (live) jb = jobs[job];
  const bool ok = live && jb.px + N <= p.frame_w && jb.py + N <= p.frame_h && jb.mode <= MT_PAETH_PRED &&
                  jb.angle_delta >= -3 && jb.angle_delta <= 3 &&
                  (jb.angle_delta == 0 || (jb.mode >= MT_V_PRED && jb.mode <= MT_D67_PRED)) && jb.dcs_ctx < 3;
  if (live && !ok) {
    if (g.j == 0) {
      mt_leaf8_result r = {};
      r.bits = r.cost = __int_as_float(0x7f800000);
      r.tx_type = 255;
      res[job] = r;
    }
    if (cf_out)
      for (int i = g.j; i < NN; i += N) cf_out[(size_t)job * NN + i] = 0;
    if (rec_out)
      for (int i = g.j; i < NN; i += N) rec_out[(size_t)job * NN + i] = 0;
  }
  if (!__any_sync(kFull, ok)) return;
  if (!ok) jb = {};
  const uint8_t* qm = a.has_qm ? S.qm : nullptr;
  const int32_t maxv = (1 << p.bd) - 1;
  const float rd_lam = p.rd_lambda;
  const int vis_w = p.vis_w > 0 ? p.vis_w : p.frame_w, vis_h = p.vis_h > 0 ? p.vis_h : p.frame_h;
  const int vw = min(max(vis_w - jb.px, 0), N), vh = min(max(vis_h - jb.py, 0), N);
  const uint16_t* s0 = src + (size_t)jb.py * p.stride + jb.px;
  const float skip1 = p.use_skip_bits ? p.skip_bits[0][0] : 0.0f;
  const float skip0 = p.use_skip_bits ? p.skip_bits[0][1] : 0.0f;
  const int ds = jb.dcs_ctx;
  lane_predict<N>(PlaneRead{rec, p.stride}, p.frame_w, p.frame_h, jb.px, jb.py, jb.mode, jb.angle_delta, jb.flags & 1,
                  (jb.flags >> 1) & 1, (jb.flags >> 2) & 1, p.bd, w.pred, reinterpret_cast<int32_t*>(&w), g);
  // DCT_DCT, then (refinement) ADST_ADST, ADST_DCT, DCT_ADST, IDTX and at 8x8
  // V_DCT, H_DCT (the 16x16 intra set has none); nibble k: the k-th type
  constexpr uint32_t kTypeOrder = 0x3206541u;
  const int ntypes = !REFINE ? 1 : (N == 8 && p.tx_search ? 7 : 5);
  int btx = MT_TX_DCT_DCT;
  long long bsse = 0, dct_sse = 0, dct_guard = 0;
  float bbits = 0.0f;
#pragma unroll 1
  for (int k = 0; k < ntypes; k++) {
    const int t = REFINE ? (int)((kTypeOrder >> (4 * k)) & 15u) : MT_TX_DCT_DCT;
    lane_fwd<N>(s0, p.stride, t, q, qm, S.qs, w, g);
    const bool one = REFINE && N == 8 && (t == MT_TX_V_DCT || t == MT_TX_H_DCT);
    int eob;
    if (t != MT_TX_IDTX && !one && a.lambda > 0.0f)
      eob = lane_trellis_ctx<N>(w, (float)q.dc_q, (float)q.ac_q, a.lambda, S.T, ds, qm, q.qm_level >= 5, p.band_tilt,
                                g);
    else
      eob = lane_eob<N>(w, g);
    lane_inv_err<N>(s0, p.stride, t, q, qm, vw, vh, maxv, w, g);
    const long long asse = lane_sse<N>(w, vw, vh, p.wsse_scale, g);
    bool gate = true;
    if (REFINE && k > 0) {
      // the ADST family within tx_guard of the DCT's SSE, IDTX within tx_guard
      // of the current best's (partition_search.rs:5320-5470,
      // block8.rs:1214-1396), V / H at most the current best's
      gate = one ? asse <= bsse
                 : (t == MT_TX_IDTX ? asse <= bsse + (p.tx_guard_shift >= 63 ? 0 : (bsse >> p.tx_guard_shift))
                                    : asse <= dct_sse + dct_guard);
      if (!__any_sync(kFull, gate)) continue;
    }
    const float base_rd = k == 0 ? 0.0f : rd_cost_i64(bsse, rd_lam, bbits);
    // bounded: the ADST family at 8x8, ADST_ADST at 16x16 (ADST_DCT / DCT_ADST
    // are priced with luma_bits there, partition_search.rs:5396-5404).  tx-type
    // symbol: the 5-type TX_16X16 set drops V_DCT / H_DCT; TX_32X32 codes none.
    const bool bounded = REFINE && (N == 8 ? t >= MT_TX_ADST_ADST : t == MT_TX_ADST_ADST);
    const float bound = bounded ? __fdiv_rn(__fsub_rn(base_rd, (float)asse), rd_lam) : __int_as_float(0x7f800000);
    const int sym = N == 32 ? -1 : (N == 16 && t >= MT_TX_ADST_ADST ? t - 2 : t);
    float abits = 0.0f;
    if (one) {  // the 1-D walk, few of them past their gate, on one lane
      if (g.j == 0 && gate)
        abits = rate_1d<N>(w.cf, t == MT_TX_V_DCT, S.T, ds, jb.mode, reinterpret_cast<uint8_t*>(w.t));
      abits = g.from(abits, 0);
      g.sync();
    } else {
      abits = lane_rate<N, REFINE>(w, eob, S.T, 0, ds, jb.mode, sym, p.use_skip_bits != 0, skip1, skip0, bound, g);
    }
    if (k == 0 || (gate && rd_cost_i64(asse, rd_lam, abits) < base_rd)) {
      bsse = asse;
      bbits = abits;
      btx = t;
      if (ok && cf_out)
        for (int i = g.j; i < NN; i += N) cf_out[(size_t)job * NN + i] = w.cf[i];
      if (ok && rec_out)
        for (int i = g.j; i < NN; i += N) rec_out[(size_t)job * NN + i] = (uint16_t)w.rec()[i];
    }
    if (k == 0) {
      dct_sse = asse;
      dct_guard = p.tx_guard_shift >= 63 ? 0 : (asse >> p.tx_guard_shift);
    }
    g.sync();  // the levels and the reconstruction are read
  }
  if (ok && g.j == 0) {
    mt_leaf8_result r = {};
    r.sse = bsse;
    r.bits = bbits;
    r.cost = REFINE ? rd_cost_i64(bsse, rd_lam, bbits) : rd_cost_i64(bsse, rd_lam, __fadd_rn(bbits, jb.syntax_bits));
    r.tx_type = (uint8_t)btx;
    res[job] = r;
  }
}

// Neighbour reads of the transforms inside a 64x64 block: the last row and
// column of each coded transform from shared memory, all else from the plane.
// A transform's edges read no other sample of the block.
template <int N>
struct Grid64Read {
  const uint16_t* __restrict__ rec;
  int stride, px, py;
  const uint16_t* edge;  // rows (y / N) * 64 + x, then columns (x / N) * 64 + y
  __device__ __forceinline__ int32_t operator()(int x, int y) const {
    const int dx = x - px, dy = y - py;
    if ((unsigned)dx < 64u && (unsigned)dy < 64u)
      return (dy & (N - 1)) == N - 1 ? edge[(dy / N) * 64 + dx] : edge[64 * (64 / N) + (dx / N) * 64 + dy];
    return rec[(size_t)y * stride + x];
  }
};

// N = 32: the 64x64 leaf's four-TX_32X32 leg (rd_pick_luma64's candidate loop,
// src/coder/block64.rs:1906-1958): for a (64x64 block, mode, delta), the
// quadrants in raster order (Q64, :328), each predicted at 32x32 from the
// running reconstruction with the per-transform edge flags (quad_edges,
// :2731-2745), TX_32X32 DCT_DCT with the QM and trellis_optimize_ctx in the
// quadrant's dc_sign context, the inverse, the decision distortion
// (luma_pick_distortion with luma64_wsse: chroma_sse's value, i.e. sse_recon,
// times K_PART_LAMBDA, src/coder/lossy_state.rs:2363-2382), luma_bits.  total =
// mlam * mode_bits (+ mlam * delta_bits) + sum of (dist + mlam * bits), f32 in
// that order.
// N = 16: the sixteen-TX_16X16 leg (the tx_depth-2 trial,
// src/coder/block64.rs:1983-2010, through grid16_luma_pass, :1670-1805): the
// dc_sign and txb_skip (skip_ctx_split) contexts from the running above / left
// context bytes, the DCT_DCT symbol (1) of the mode's TX_16X16 tx-type CDF;
// coef_res_ctx then fills the transform's context bytes.  total = mode cost +
// (dist + mlam x bits) + mlam x depth_bits, f32 in that order.
// The transforms of a job are a chain; the jobs fill the GPU.  Measured at
// 1080p against a thread per job: N = 32 (6,240 jobs) 80 -> 1.72 ms,
// N = 16 (480 jobs) 8.4 -> 0.65 ms.
template <int N, typename J, typename R>
__global__ void __launch_bounds__(lane_threads<N>()) leaf64_kernel(
    const uint16_t* __restrict__ src, const uint16_t* __restrict__ rec, LeafArgs a,
    const uint8_t* __restrict__ qm_row, const mt_coef_costs* __restrict__ costs, const J* __restrict__ jobs, int n,
    R* __restrict__ res, int32_t* __restrict__ cf_out) {
  constexpr int NN = N * N, G = 64 / N;
  constexpr bool kGrid = N == 16;
  using Buf = LaneBuf<N>;
  __shared__ LaneTables<NN> S;
  __shared__ uint16_t edges[lane_blocks<N>()][2 * G * 64];
  extern __shared__ __align__(128) unsigned char lane_smem[];
  S.load(costs, qm_row, a.has_qm);
  const Lanes<N> g;
  const int slot = threadIdx.x / N;
  Buf& w = reinterpret_cast<Buf*>(lane_smem)[slot];
  uint16_t* edge = edges[slot];
  const int job = blockIdx.x * lane_blocks<N>() + slot;
  const bool live = job < n;
  const mt_split16_params& p = a.p;
  const mt_quant& q = a.q;
  const float kInf = __int_as_float(0x7f800000);
  J jb = {};
  if (live) jb = jobs[job];
  const bool directional = jb.mode >= MT_V_PRED && jb.mode <= MT_D67_PRED;
  bool ok = live && jb.px + 64 <= p.frame_w && jb.py + 64 <= p.frame_h && jb.mode <= MT_PAETH_PRED &&
            jb.angle_delta >= -3 && jb.angle_delta <= 3 && (jb.angle_delta == 0 || directional);
  if constexpr (!kGrid)
    ok = ok && jb.dcs_ctx[0] < 3 && jb.dcs_ctx[1] < 3 && jb.dcs_ctx[2] < 3 && jb.dcs_ctx[3] < 3;
  if (live && !ok) {
    if (g.j == 0) {
      R r = {};
      r.total = kInf;
      if constexpr (kGrid) {
        r.dist = r.bits = kInf;
      } else {
        for (int k = 0; k < 4; k++) r.bits[k] = kInf;
      }
      res[job] = r;
    }
    if constexpr (kGrid) {
      if (cf_out)
        for (int i = g.j; i < 4096; i += N) cf_out[(size_t)job * 4096 + i] = 0;
    }
  }
  if (!__any_sync(kFull, ok)) return;
  if (!ok) jb = {};
  const Grid64Read<N> rd{rec, p.stride, jb.px, jb.py, edge};
  const uint8_t* qm = a.has_qm ? S.qm : nullptr;
  const int32_t maxv = (1 << p.bd) - 1;
  const float mlam = p.rd_lambda;
  const int vis_w = p.vis_w > 0 ? p.vis_w : p.frame_w, vis_h = p.vis_h > 0 ? p.vis_h : p.frame_h;
  const bool have_tr = jb.flags & MT_CAND_HAVE_TR, have_bl = jb.flags & MT_CAND_HAVE_BL;
  const bool ft = jb.flags & MT_CAND_FILTER_TYPE;
  uint32_t actx[G], lctx[G];  // N = 16: four context bytes per transform column / row
  if constexpr (kGrid) {
#pragma unroll
    for (int i = 0; i < G; i++) {
      actx[i] = lctx[i] = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        actx[i] |= (uint32_t)jb.a_coef[4 * i + k] << (8 * k);
        lctx[i] |= (uint32_t)jb.l_coef[4 * i + k] << (8 * k);
      }
    }
  }
  float total = __fmul_rn(mlam, jb.mode_bits), dist = 0.0f, bits = 0.0f;
  if (directional) total = __fadd_rn(total, __fmul_rn(mlam, jb.delta_bits));
  long long sse_sum = 0;
#pragma unroll 1
  for (int ty = 0; ty < G; ty++)
#pragma unroll 1
    for (int tx = 0; tx < G; tx++) {
      const int t = ty * G + tx;
      const int sx = tx * N, sy = ty * N, bx = jb.px + sx, by = jb.py + sy;
      const bool tr = ty == 0 ? (jb.py > 0 && (tx < G - 1 || have_tr)) : tx < G - 1;
      const bool bl = tx == 0 && jb.px > 0 && (ty < G - 1 || have_bl);
      const uint16_t* s0 = src + (size_t)by * p.stride + bx;
      const int vw = min(max(vis_w - bx, 0), N), vh = min(max(vis_h - by, 0), N);
      lane_predict<N>(rd, p.frame_w, p.frame_h, bx, by, jb.mode, jb.angle_delta, tr, bl, ft, p.bd, w.pred,
                      reinterpret_cast<int32_t*>(&w), g);
      int ds, sk = 0;
      if constexpr (kGrid) {
        const uint32_t la4 = tx == 0 ? actx[0] : (tx == 1 ? actx[1] : (tx == 2 ? actx[2] : actx[3]));
        const uint32_t ll4 = ty == 0 ? lctx[0] : (ty == 1 ? lctx[1] : (ty == 2 ? lctx[2] : lctx[3]));
        uint32_t la = 0, ll = 0;
        int s = -8;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t av = (la4 >> (8 * k)) & 255u, lv = (ll4 >> (8 * k)) & 255u;
          la |= av;
          ll |= lv;
          s += (int)(av >> 6) + (int)(lv >> 6);
        }
        sk = kSkipCtxTbl[min(la & 0x3fu, 4u)][min(ll & 0x3fu, 4u)];
        ds = (s != 0) + (s > 0);
      } else {
        ds = jb.dcs_ctx[t];
      }
      lane_fwd<N>(s0, p.stride, MT_TX_DCT_DCT, q, qm, S.qs, w, g);
      int eob;
      if (a.lambda > 0.0f)
        eob = lane_trellis_ctx<N>(w, (float)q.dc_q, (float)q.ac_q, a.lambda, S.T, ds, qm, q.qm_level >= 5,
                                  p.band_tilt, g);
      else
        eob = lane_eob<N>(w, g);
      lane_inv_err<N>(s0, p.stride, MT_TX_DCT_DCT, q, qm, vw, vh, maxv, w, g);
      const long long sse = lane_sse<N>(w, vw, vh, p.wsse_scale, g);
      const float d1 = __fmul_rn(__ll2float_rn(sse), 2.775f);  // proxy_wsse: K_PART_LAMBDA
      const float skip1 = p.use_skip_bits ? p.skip_bits[sk][0] : 0.0f;
      const float skip0 = p.use_skip_bits ? p.skip_bits[sk][1] : 0.0f;
      const float b1 = lane_rate<N, false>(w, eob, S.T, sk, ds, jb.mode, kGrid ? 1 : -1, p.use_skip_bits != 0, skip1,
                                           skip0, kInf, g);
      edge[ty * 64 + sx + g.j] = (uint16_t)w.pred[(N - 1) * N + g.j];
      edge[64 * G + tx * 64 + sy + g.j] = (uint16_t)w.pred[g.j * N + N - 1];
      if constexpr (kGrid) {
        dist = __fadd_rn(dist, d1);
        bits = __fadd_rn(bits, b1);
        sse_sum += sse;
        // coef_res_ctx: min(cumulative level, 63) | the dc-sign marker
        uint32_t cul = 0;
#pragma unroll
        for (int i = 0; i < N; i++) cul += uabs(w.cf[i * N + g.j]);
        cul = g.sum(cul);
        const int32_t c0 = w.cf[0];
        const uint32_t rc = eob < 0 ? 0x40u : (min(cul, 63u) | (c0 == 0 ? 0x40u : (c0 < 0 ? 0u : 0x80u)));
        const uint32_t rc4 = rc * 0x01010101u;
#pragma unroll
        for (int i = 0; i < G; i++) {
          if (i == tx) actx[i] = rc4;
          if (i == ty) lctx[i] = rc4;
        }
        if (ok && cf_out)
          for (int i = g.j; i < NN; i += N) cf_out[(size_t)job * 4096 + t * NN + i] = w.cf[i];
      } else {
        total = __fadd_rn(total, __fadd_rn(d1, __fmul_rn(mlam, b1)));
        if (ok && g.j == 0) {
          res[job].bits[t] = b1;
          res[job].sse[t] = sse;
        }
      }
      g.sync();  // the block's edges are written, its levels and samples read
    }
  if (ok && g.j == 0) {
    R& r = res[job];
    r.reserved = 0;
    if constexpr (kGrid) {
      total = __fadd_rn(total, __fadd_rn(dist, __fmul_rn(mlam, bits)));
      r.total = __fadd_rn(total, __fmul_rn(mlam, jb.depth_bits));
      r.dist = dist;
      r.bits = bits;
      r.sse = sse_sum;
    } else {
      r.total = total;
    }
  }
}

// Shared memory of a CTA of `blocks`, opted in for: always for the kernel's
// largest CTA, since another thread may be about to launch one.
template <typename B, typename K>
bool lane_smem_bytes(K kernel, int blocks, int max_blocks, size_t* dyn) {
  *dyn = sizeof(B) * (size_t)blocks;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(B) * max_blocks)) ==
         cudaSuccess;
}

int check(const mt_split16_params* p, const mt_quant* q, int32_t n) {
  if (!p || !q || n < 0) return MT_ERR_INVALID_INPUT;
  if (p->bd != 8) return MT_ERR_UNSUPPORTED;
  if (p->frame_w < 4 || p->frame_h < 4 || p->stride < p->frame_w || p->vis_w < 0 || p->vis_h < 0)
    return MT_ERR_INVALID_INPUT;
  if (!(p->rd_lambda > 0.0f) || !(p->wsse_scale >= 0.0f) || p->tx_guard_shift < 0) return MT_ERR_INVALID_INPUT;
  return MT_OK;
}

size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

template <int N, bool REFINE>
int leaf_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm, const mt_quant* quant,
                 const uint8_t* d_qm_row, const mt_coef_costs* d_costs, const mt_leaf8_job* d_jobs, int32_t n,
                 mt_leaf8_result* d_results, int32_t* d_cf, uint16_t* d_rec, void* stream) {
  const int rc = check(prm, quant, n);
  if (rc != MT_OK) return rc;
  if (n == 0) return MT_OK;
  if (!d_src || !d_recon || !d_costs || !d_jobs || !d_results) return MT_ERR_INVALID_INPUT;
  LeafArgs a;
  a.p = *prm;
  a.q = *quant;
  a.lambda = prm->trellis_lambda0 > 0.0f ? mth::scaled_trellis_lambda_host((float)quant->dc_q, prm->trellis_lambda0)
                                         : 0.0f;
  a.has_qm = quant->qm_level < 15 && d_qm_row != nullptr;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int B = lane_blocks<N>();
  if constexpr (leaf_max_blocks<N, REFINE>() > lane_blocks<N>()) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return MT_ERR_DEVICE;
    if (n >= 2 * 2 * leaf_max_blocks<N, REFINE>() * sms) B = leaf_max_blocks<N, REFINE>();
  }
  size_t dyn = 0;
  if (!lane_smem_bytes<LaneBuf<N, REFINE>>(leaf_lanes_kernel<N, REFINE>, B, leaf_max_blocks<N, REFINE>(), &dyn))
    return MT_ERR_DEVICE;
  leaf_lanes_kernel<N, REFINE><<<(unsigned)((n + (int64_t)B - 1) / B), (unsigned)(B * N), dyn, st>>>(
      d_src, d_recon, a, d_qm_row, d_costs, d_jobs, n, d_results, d_cf, d_rec);
  return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

template <int N>
int leaf_host(const uint16_t* src, const uint16_t* recon, const mt_split16_params* prm, const mt_quant* quant,
              const uint8_t* qm_row, const mt_coef_costs* costs, const mt_leaf8_job* jobs, int32_t n, int32_t refine,
              mt_leaf8_result* results, int32_t* cf_out, uint16_t* rec_out);

template <int N, typename J, typename R>
int leaf64_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm, const mt_quant* quant,
                  const uint8_t* d_qm_row, const mt_coef_costs* d_costs, const J* d_jobs, int32_t n, R* d_results,
                  int32_t* d_cf, void* stream) {
  const int rc = check(prm, quant, n);
  if (rc != MT_OK) return rc;
  if (n == 0) return MT_OK;
  if (!d_src || !d_recon || !d_costs || !d_jobs || !d_results) return MT_ERR_INVALID_INPUT;
  LeafArgs a;
  a.p = *prm;
  a.q = *quant;
  a.lambda = prm->trellis_lambda0 > 0.0f ? mth::scaled_trellis_lambda_host((float)quant->dc_q, prm->trellis_lambda0)
                                         : 0.0f;
  a.has_qm = quant->qm_level < 15 && d_qm_row != nullptr;
  constexpr int B = lane_blocks<N>();
  size_t dyn = 0;
  if (!lane_smem_bytes<LaneBuf<N>>(leaf64_kernel<N, J, R>, B, B, &dyn)) return MT_ERR_DEVICE;
  leaf64_kernel<N, J, R><<<(unsigned)((n + B - 1) / B), lane_threads<N>(), dyn,
                           reinterpret_cast<cudaStream_t>(stream)>>>(d_src, d_recon, a, d_qm_row, d_costs, d_jobs, n,
                                                                     d_results, d_cf);
  return cudaGetLastError() == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

int quad32_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm, const mt_quant* quant,
                  const uint8_t* d_qm_row, const mt_coef_costs* d_costs, const mt_quad32_job* d_jobs, int32_t n,
                  mt_quad32_result* d_results, void* stream) {
  return leaf64_device<32>(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, nullptr, stream);
}

int grid16_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm, const mt_quant* quant,
                  const uint8_t* d_qm_row, const mt_coef_costs* d_costs, const mt_grid16_job* d_jobs, int32_t n,
                  mt_grid16_result* d_results, int32_t* d_cf, void* stream) {
  return leaf64_device<16>(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, d_cf, stream);
}

}  // namespace

extern "C" {

int mt_leaf8_luma_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm,
                         const mt_quant* quant, const uint8_t* d_qm_row, const mt_coef_costs* d_costs,
                         const mt_leaf8_job* d_jobs, int32_t n, mt_leaf8_result* d_results, int32_t* d_cf,
                         uint16_t* d_rec, void* stream) {
  return leaf_device<8, false>(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, d_cf, d_rec, stream);
}

int mt_leaf8_tx_refine_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm,
                              const mt_quant* quant, const uint8_t* d_qm_row, const mt_coef_costs* d_costs,
                              const mt_leaf8_job* d_jobs, int32_t n, mt_leaf8_result* d_results, int32_t* d_cf,
                              uint16_t* d_rec, void* stream) {
  return leaf_device<8, true>(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, d_cf, d_rec, stream);
}

int mt_leaf8(const uint16_t* src, const uint16_t* recon, const mt_split16_params* prm, const mt_quant* quant,
             const uint8_t* qm_row, const mt_coef_costs* costs, const mt_leaf8_job* jobs, int32_t n, int32_t refine,
             mt_leaf8_result* results, int32_t* cf_out, uint16_t* rec_out) {
  return leaf_host<8>(src, recon, prm, quant, qm_row, costs, jobs, n, refine, results, cf_out, rec_out);
}

int mt_leaf16_luma_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm,
                          const mt_quant* quant, const uint8_t* d_qm_row, const mt_coef_costs* d_costs,
                          const mt_leaf8_job* d_jobs, int32_t n, mt_leaf8_result* d_results, int32_t* d_cf,
                          uint16_t* d_rec, void* stream) {
  return leaf_device<16, false>(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, d_cf, d_rec,
                                stream);
}

int mt_leaf16_tx_refine_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm,
                               const mt_quant* quant, const uint8_t* d_qm_row, const mt_coef_costs* d_costs,
                               const mt_leaf8_job* d_jobs, int32_t n, mt_leaf8_result* d_results, int32_t* d_cf,
                               uint16_t* d_rec, void* stream) {
  return leaf_device<16, true>(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, d_cf, d_rec,
                               stream);
}

int mt_leaf16(const uint16_t* src, const uint16_t* recon, const mt_split16_params* prm, const mt_quant* quant,
              const uint8_t* qm_row, const mt_coef_costs* costs, const mt_leaf8_job* jobs, int32_t n, int32_t refine,
              mt_leaf8_result* results, int32_t* cf_out, uint16_t* rec_out) {
  return leaf_host<16>(src, recon, prm, quant, qm_row, costs, jobs, n, refine, results, cf_out, rec_out);
}

int mt_leaf32_luma_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm,
                          const mt_quant* quant, const uint8_t* d_qm_row, const mt_coef_costs* d_costs,
                          const mt_leaf8_job* d_jobs, int32_t n, mt_leaf8_result* d_results, int32_t* d_cf,
                          uint16_t* d_rec, void* stream) {
  return leaf_device<32, false>(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, d_cf, d_rec,
                                stream);
}

int mt_leaf32(const uint16_t* src, const uint16_t* recon, const mt_split16_params* prm, const mt_quant* quant,
              const uint8_t* qm_row, const mt_coef_costs* costs, const mt_leaf8_job* jobs, int32_t n,
              mt_leaf8_result* results, int32_t* cf_out, uint16_t* rec_out) {
  return leaf_host<32>(src, recon, prm, quant, qm_row, costs, jobs, n, 0, results, cf_out, rec_out);
}

int mt_quad32_luma_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm,
                          const mt_quant* quant, const uint8_t* d_qm_row, const mt_coef_costs* d_costs,
                          const mt_quad32_job* d_jobs, int32_t n, mt_quad32_result* d_results, void* stream) {
  return quad32_device(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, stream);
}

int mt_quad32_luma(const uint16_t* src, const uint16_t* recon, const mt_split16_params* prm, const mt_quant* quant,
                   const uint8_t* qm_row, const mt_coef_costs* costs, const mt_quad32_job* jobs, int32_t n,
                   mt_quad32_result* results) {
  int rc = check(prm, quant, n);
  if (rc != MT_OK) return rc;
  if (n == 0) return MT_OK;
  if (!src || !recon || !costs || !jobs || !results) return MT_ERR_INVALID_INPUT;
  const size_t plane = (size_t)prm->stride * prm->frame_h * sizeof(uint16_t);
  const size_t o_src = 0, o_rec = up256(plane), o_qm = o_rec + up256(plane), o_cost = o_qm + up256(1024);
  const size_t o_jobs = o_cost + up256(sizeof(mt_coef_costs));
  const size_t o_res = o_jobs + up256((size_t)n * sizeof(mt_quad32_job));
  const size_t total = o_res + up256((size_t)n * sizeof(mt_quad32_result));
  uint8_t* d = nullptr;
  if (cudaMalloc(&d, total) != cudaSuccess) return MT_ERR_ALLOC;
  const bool has_qm = quant->qm_level < 15 && qm_row != nullptr;
  cudaError_t e = cudaMemcpy(d + o_src, src, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_rec, recon, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && has_qm) e = cudaMemcpy(d + o_qm, qm_row, 1024, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_cost, costs, sizeof(mt_coef_costs), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_jobs, jobs, (size_t)n * sizeof(mt_quad32_job), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    rc = quad32_device(reinterpret_cast<const uint16_t*>(d + o_src), reinterpret_cast<const uint16_t*>(d + o_rec),
                       prm, quant, has_qm ? d + o_qm : nullptr, reinterpret_cast<const mt_coef_costs*>(d + o_cost),
                       reinterpret_cast<const mt_quad32_job*>(d + o_jobs), n,
                       reinterpret_cast<mt_quad32_result*>(d + o_res), nullptr);
    if (rc == MT_OK) e = cudaMemcpy(results, d + o_res, (size_t)n * sizeof(mt_quad32_result), cudaMemcpyDeviceToHost);
  }
  cudaFree(d);
  if (rc != MT_OK) return rc;
  return e == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

int mt_grid16_luma_device(const uint16_t* d_src, const uint16_t* d_recon, const mt_split16_params* prm,
                          const mt_quant* quant, const uint8_t* d_qm_row, const mt_coef_costs* d_costs,
                          const mt_grid16_job* d_jobs, int32_t n, mt_grid16_result* d_results, int32_t* d_cf,
                          void* stream) {
  return grid16_device(d_src, d_recon, prm, quant, d_qm_row, d_costs, d_jobs, n, d_results, d_cf, stream);
}

int mt_grid16_luma(const uint16_t* src, const uint16_t* recon, const mt_split16_params* prm, const mt_quant* quant,
                   const uint8_t* qm_row, const mt_coef_costs* costs, const mt_grid16_job* jobs, int32_t n,
                   mt_grid16_result* results, int32_t* cf_out) {
  int rc = check(prm, quant, n);
  if (rc != MT_OK) return rc;
  if (n == 0) return MT_OK;
  if (!src || !recon || !costs || !jobs || !results) return MT_ERR_INVALID_INPUT;
  const size_t plane = (size_t)prm->stride * prm->frame_h * sizeof(uint16_t);
  const size_t o_src = 0, o_rec = up256(plane), o_qm = o_rec + up256(plane), o_cost = o_qm + up256(256);
  const size_t o_jobs = o_cost + up256(sizeof(mt_coef_costs));
  const size_t o_res = o_jobs + up256((size_t)n * sizeof(mt_grid16_job));
  const size_t o_cf = o_res + up256((size_t)n * sizeof(mt_grid16_result));
  const size_t total = o_cf + (cf_out ? up256((size_t)n * 4096 * 4) : 0);
  uint8_t* d = nullptr;
  if (cudaMalloc(&d, total) != cudaSuccess) return MT_ERR_ALLOC;
  const bool has_qm = quant->qm_level < 15 && qm_row != nullptr;
  cudaError_t e = cudaMemcpy(d + o_src, src, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_rec, recon, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && has_qm) e = cudaMemcpy(d + o_qm, qm_row, 256, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_cost, costs, sizeof(mt_coef_costs), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_jobs, jobs, (size_t)n * sizeof(mt_grid16_job), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    rc = grid16_device(reinterpret_cast<const uint16_t*>(d + o_src), reinterpret_cast<const uint16_t*>(d + o_rec),
                       prm, quant, has_qm ? d + o_qm : nullptr, reinterpret_cast<const mt_coef_costs*>(d + o_cost),
                       reinterpret_cast<const mt_grid16_job*>(d + o_jobs), n,
                       reinterpret_cast<mt_grid16_result*>(d + o_res),
                       cf_out ? reinterpret_cast<int32_t*>(d + o_cf) : nullptr, nullptr);
    if (rc == MT_OK) e = cudaMemcpy(results, d + o_res, (size_t)n * sizeof(mt_grid16_result), cudaMemcpyDeviceToHost);
    if (rc == MT_OK && e == cudaSuccess && cf_out)
      e = cudaMemcpy(cf_out, d + o_cf, (size_t)n * 4096 * 4, cudaMemcpyDeviceToHost);
  }
  cudaFree(d);
  if (rc != MT_OK) return rc;
  return e == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

}  // extern "C"

namespace {

// Host-buffer form of the leaf searches.
template <int N>
int leaf_host(const uint16_t* src, const uint16_t* recon, const mt_split16_params* prm, const mt_quant* quant,
              const uint8_t* qm_row, const mt_coef_costs* costs, const mt_leaf8_job* jobs, int32_t n, int32_t refine,
              mt_leaf8_result* results, int32_t* cf_out, uint16_t* rec_out) {
  constexpr size_t NN = (size_t)N * N;
  int rc = check(prm, quant, n);
  if (rc != MT_OK) return rc;
  if (n == 0) return MT_OK;
  if (!src || !recon || !costs || !jobs || !results) return MT_ERR_INVALID_INPUT;
  const size_t plane = (size_t)prm->stride * prm->frame_h * sizeof(uint16_t);
  const size_t o_src = 0, o_rec = up256(plane), o_qm = o_rec + up256(plane), o_cost = o_qm + up256(NN);
  const size_t o_jobs = o_cost + up256(sizeof(mt_coef_costs));
  const size_t o_res = o_jobs + up256((size_t)n * sizeof(mt_leaf8_job));
  const size_t o_cf = o_res + up256((size_t)n * sizeof(mt_leaf8_result));
  const size_t o_out = o_cf + (cf_out ? up256((size_t)n * NN * 4) : 0);
  const size_t total = o_out + (rec_out ? up256((size_t)n * NN * 2) : 0);
  uint8_t* d = nullptr;
  if (cudaMalloc(&d, total) != cudaSuccess) return MT_ERR_ALLOC;
  const bool has_qm = quant->qm_level < 15 && qm_row != nullptr;
  cudaError_t e = cudaMemcpy(d + o_src, src, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_rec, recon, plane, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && has_qm) e = cudaMemcpy(d + o_qm, qm_row, NN, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_cost, costs, sizeof(mt_coef_costs), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + o_jobs, jobs, (size_t)n * sizeof(mt_leaf8_job), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    auto fn = refine ? leaf_device<N, N != 32> : leaf_device<N, false>;
    rc = fn(reinterpret_cast<const uint16_t*>(d + o_src), reinterpret_cast<const uint16_t*>(d + o_rec), prm, quant,
            has_qm ? d + o_qm : nullptr, reinterpret_cast<const mt_coef_costs*>(d + o_cost),
            reinterpret_cast<const mt_leaf8_job*>(d + o_jobs), n, reinterpret_cast<mt_leaf8_result*>(d + o_res),
            cf_out ? reinterpret_cast<int32_t*>(d + o_cf) : nullptr,
            rec_out ? reinterpret_cast<uint16_t*>(d + o_out) : nullptr, nullptr);
    if (rc == MT_OK) e = cudaMemcpy(results, d + o_res, (size_t)n * sizeof(mt_leaf8_result), cudaMemcpyDeviceToHost);
    if (rc == MT_OK && e == cudaSuccess && cf_out) e = cudaMemcpy(cf_out, d + o_cf, (size_t)n * NN * 4, cudaMemcpyDeviceToHost);
    if (rc == MT_OK && e == cudaSuccess && rec_out) e = cudaMemcpy(rec_out, d + o_out, (size_t)n * NN * 2, cudaMemcpyDeviceToHost);
  }
  cudaFree(d);
  if (rc != MT_OK) return rc;
  return e == cudaSuccess ? MT_OK : MT_ERR_DEVICE;
}

}  // namespace
