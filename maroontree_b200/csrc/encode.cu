// mt_encode_rgb8: an end-to-end AVIF encode on the device with this library's
// kernels and the reference's bitstream, entropy coder and container.
//
// What it decides, and what it does not: the reference's superblock decision
// engine (src/coder/superblock.rs:813 decode_sb and its partition / leaf
// searches) is not restated here.  This encoder codes every 64x64 superblock
// as a full split down to 8x8 blocks; each 8x8 luma block takes the lowest RD
// cost (strict <, first in (mode, type) order) of the 13 intra modes at angle
// delta 0 times the seven 8x8 intra transform types, as priced by the batched
// candidate chain (prediction, forward transform, quantisation and QM,
// trellis, inverse, SATD bridge, coefficient rate); chroma is UV_DC_PRED with
// DCT_DCT (8x8 in 4:4:4, 4x4 in 4:2:0).  Everything after the decisions is the
// reference's: the coefficient coders and block syntax with their contexts,
// the adaptive range coder and tile packer, the shipped loop-filter levels,
// the CDEF strength search with its per-unit cdef_idx replay, the sequence and
// frame headers and the AVIF container.  The result decodes under any AV1
// decoder to the reconstruction this encoder computed.
//
// Schedule: one persistent launch of 4-CTA clusters takes the frame's 8x8
// blocks from a ticket counter in dependency-level order (a block after its
// left, top, top-left and, where its edges use them, top-right and
// bottom-left neighbours inside its tile) and waits for those neighbours'
// edge records with bounded polls.  The 13 modes of a block are split over the
// cluster's CTAs and the seven transform types over a CTA's warps, each (mode,
// type) candidate on eight lanes; the cluster minimum picks the winner.  Frames
// code in the spec-minimum uniform tiling (one tile up to 64 superblocks wide
// and 2304 in area), tiles independent.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "../../include/maroontree_b200.h"
#include "av1_tables.h"
#include "coop8.cuh"
#include "stream.h"

namespace mth {
float scaled_trellis_lambda_host(float dc_q, float lambda0);
}

namespace {

namespace cg = cooperative_groups;

struct EncArgs {
  const uint16_t* src[3];
  uint16_t* rec[3];
  mt_chain_params py, pc;  // luma / chroma plane parameters
  mt_quant qy, qc;
  float tly, tlc;          // scaled trellis lambdas
  int has_qm_y, has_qm_c;  // a QM row for luma / chroma (level < 15)
  int sub;                 // 0 4:4:4, 2 4:2:0
  int w8, h8;
  int tile_w8, tile_h8;    // the uniform tile size in 8x8 blocks (the last tile may be smaller)
  uint8_t* mode;           // per 8x8 block (frame raster of 8x8 blocks)
  uint8_t* tx;
  int32_t* lv_y;           // 64 per block
  int32_t* lv_u;           // 64 (4:4:4) or 16 (4:2:0) per block
  int32_t* lv_v;
};

// One image of a launch: its arguments, its tables and its blocks' edge
// records (zero at the launch).
struct JobDesc {
  EncArgs a;
  const mt_coef_costs* cy;
  const uint8_t* qmy;
  const uint8_t* qmc;
  uint4* edges;
};

// The z-order position of the k-th 8x8 block of a superblock and its
// intra-edge flags down the quadtree (src/coder/superblock.rs:958-987: root
// (top-right 1, bottom-left 0); children TL (1, 1), TR (parent's, 0),
// BL (1, parent's), BR (0, 0)).
__host__ __device__ constexpr void zorder(int k, int* bx, int* by, bool* thr, bool* lhb) {
  int x = 0, y = 0;
  bool t = true, l = false;
  for (int lvl = 2; lvl >= 0; --lvl) {
    const int c = (k >> (2 * lvl)) & 3;
    const int h = 1 << lvl;
    if (c == 0) {
      t = true;
      l = true;
    } else if (c == 1) {
      x += h;
      l = false;
    } else if (c == 2) {
      y += h;
      t = true;
    } else {
      x += h;
      y += h;
      t = false;
      l = false;
    }
  }
  *bx = x;
  *by = y;
  *thr = t;
  *lhb = l;
}

// The order in which the blocks are taken: block (x, y) of superblock (c, r)
// of a tile comes at kWaveCol c + kWaveRow r + t[y][x].  The numbers are the
// dependency levels (one more than the highest of a block's left, top, top-left
// and, where its intra edges use them, top-right and bottom-left neighbours)
// inside a large frame, where a superblock further right or down adds the same
// to every level; at a tile's edges some of the neighbours are missing, so the
// order holds there too, a few steps late.  With it the list is made on the
// device (three launches, 10 us) instead of level by level on the host (0.4 ms
// at 1080p, 3.6 ms at 4096x4096).
constexpr int kWaveCol = 22, kWaveRow = 30;
struct Wave {
  uint8_t t[8][8];
  int last;
};
constexpr Wave make_wave() {
  int t[8][8] = {};
  bool moved = true;
  for (int pass = 0; moved && pass < 256; ++pass) {
    moved = false;
    for (int k = 0; k < 64; ++k) {
      int x = 0, y = 0;
      bool thr = false, lhb = false;
      zorder(k, &x, &y, &thr, &lhb);
      int lv = t[y][x];
      const int dx[5] = {-1, 0, -1, 1, -1}, dy[5] = {0, -1, -1, -1, 1};
      for (int d = 0; d < 5; ++d) {
        if ((d == 3 && !thr) || (d == 4 && !lhb)) continue;
        const int xx = x + dx[d] + 8, yy = y + dy[d] + 8;  // 8 .. 15 inside the superblock
        const int at = t[yy & 7][xx & 7] + kWaveCol * (xx / 8 - 1) + kWaveRow * (yy / 8 - 1);
        if (at + 1 > lv) lv = at + 1;
      }
      if (lv != t[y][x]) {
        t[y][x] = lv;
        moved = true;
      }
    }
  }
  Wave w = {};
  for (int k = 0; k < 64; ++k) {
    w.t[k / 8][k % 8] = (uint8_t)t[k / 8][k % 8];
    if (t[k / 8][k % 8] > w.last) w.last = t[k / 8][k % 8];
  }
  w.last = moved ? -1 : w.last;  // never moved again: every block is after its neighbours
  return w;
}
constexpr Wave kWave = make_wave();
static_assert(kWave.last > 0 && kWave.last < 256, "the wave has an order");
__constant__ Wave cWave = kWave;

// A list entry: the block's column and row (11 bits each), and which of its
// left, top, top-right and bottom-left neighbours it may use (inside its tile;
// the last two also coded before it).
constexpr uint32_t kHasL = 1u << 22, kHasT = 1u << 23, kHasTr = 1u << 24, kHasBl = 1u << 25;

__device__ __forceinline__ bool is_smooth(int m) { return m == MT_SMOOTH_PRED || m == MT_SMOOTH_V_PRED || m == MT_SMOOTH_H_PRED; }

// A block is a cluster of kClusterCtas CTAs (on as many SMs).  CTA r takes the
// modes [mode_lo(r), mode_lo(r + 1)), a warp each transform type of them, eight
// lanes per mode: a warp runs one transform path, a CTA predicts each mode once
// for the seven types.  One more warp codes a chroma plane in CTAs 2 and 3 and
// fetches the cluster's next block in CTA 0.
// Candidate index = mode * 7 + type, the order ties are broken in.
constexpr int kClusterCtas = 4;
// CTAs of the decision kernel resident per SM (its register budget follows).
#ifndef MT_ENC_CTAS_PER_SM
#define MT_ENC_CTAS_PER_SM 2
#endif
constexpr int kTypes = 7;  // MT_TX_IDTX .. MT_TX_DCT_ADST
constexpr int kSideWarp = kTypes;  // the chroma / next-block warp, behind one per type
constexpr int kLumaThreads = kTypes * 32;
constexpr int kStepThreads = kLumaThreads + 32;
constexpr int kGroupBufs = 4 * kTypes + 8;  // one per candidate, and eight groups of four lanes for chroma
__device__ __forceinline__ int mode_lo(int rank) { return rank ? 3 * rank + 1 : 0; }  // 0, 4, 7, 10
__device__ __forceinline__ int mode_rank(int m) { return m < 4 ? 0 : (m - 1) / 3; }

// What the clusters tell each other about a finished block: per block and
// plane two 16-byte records, the bottom row and the right column as bytes, then
// a set word and, in luma, the mode.  A record is written and read whole, so
// seeing the set word is seeing the samples: a reader polls the record itself
// and needs no count, no fence and no second read.
__device__ __forceinline__ uint4* edge_rec(uint4* base, int b, int plane, int right) {
  return base + ((size_t)b * 3 + plane) * 2 + right;
}
__device__ __forceinline__ void put_rec(uint4* p, uint32_t lo, uint32_t hi, uint32_t mode) {
  const unsigned __int128 v = ((unsigned __int128)(((unsigned long long)mode << 32) | 1u) << 64) |
                              (((unsigned long long)hi << 32) | lo);
  asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(v) : "memory");
}
__device__ __forceinline__ uint4 get_rec(const uint4* p) {
  unsigned __int128 v;
  asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(v) : "l"(p) : "memory");
  return make_uint4((uint32_t)v, (uint32_t)(v >> 32), (uint32_t)(v >> 64), (uint32_t)(v >> 96));
}

// What the CTAs of a cluster write into each other's shared memory.  A warp's
// minimum key (cost, candidate) is stored with its bytes counted by the reading
// CTA's barrier of the block: the barrier opens when all 28 keys are there, and
// a waiting warp is suspended meanwhile (polling the keys instead took the
// issue slots of the warps still at work: 1080p 8.8, 4096x4096 42.8 ms).  The
// next block and the chroma warps' marks are words with the block's sequence
// number in them, polled by a warp per CTA that has nothing else to do: sequence
// (24 bits), end (1), image (7), list entry (32).
constexpr uint32_t kSeqMask = 0xffffffu;
__device__ __forceinline__ void put_word(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.cluster.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long get_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.cluster.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Everything one CTA keeps in shared memory beside the groups' buffers.
struct StepShared {
  alignas(16) int16_t pcol[4][64];  // the predictions of this CTA's modes, by columns
  alignas(16) int16_t rcol[4][64];  // their residuals by columns
  alignas(16) int16_t rrow[4][64];  // and by rows
  alignas(16) int16_t ccol[64];     // the chroma residual by columns (4:4:4)
  alignas(16) int16_t src[64], csrc[64];  // the block's luma and chroma source samples, by columns
  mtd::CoopEdges edge;
  mtd::CoopPredBuf pb[4];
  mtd::CoopPlane py, pc;
  mtd::CoopScan scan;
  mt_coef_costs cy;
  float head[4][kTypes][64];                 // coop8_rate_head of this CTA's modes, by type and end of block
  alignas(8) unsigned long long key[2][32];  // by block parity: the cluster's luma warps' minima
  unsigned long long key_bar[2];             // their barriers
  unsigned long long mark[2][2];             // by block parity: the chroma warps' marks
  unsigned long long next[2];                // by block parity
  uint32_t begun;                            // the block whose edges the luma warps last had
  uint8_t nb_mode[2];             // modes of the blocks above and to the left
  JobDesc job;                    // the descriptor of the image whose tables are staged
};

__device__ __forceinline__ void luma_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kLumaThreads) : "memory"); }

// Every wait gives up after a number of polls and sets *err.  Of them only the
// waits for records, which depend on other clusters, end early on a set *err:
// what a cluster's CTAs tell each other (keys, marks, words) still comes, late
// by one such wait at most, since every warp goes on to its key or mark, and
// cutting those waits short would let a word be overwritten, or a barrier armed
// twice, before all have seen it.  Their limits are there for what cannot
// happen, each several times what it waits for: a record's wait lasts some
// 0.2 s, the fetching warp's waits 3 to 4 s each, the one for its word 27 s.
constexpr int kMaxPolls = 1 << 20, kMaxWordPolls = 1 << 24, kMaxBarPolls = 1 << 23;

__device__ __forceinline__ uint4 wait_rec(const uint4* p, uint32_t* err) {
  uint4 v = get_rec(p);
  for (int it = 1; v.z == 0; ++it) {
    if ((it & 15) == 0 && *(volatile uint32_t*)err) break;
    if (it > kMaxPolls) {
      atomicExch(err, 1u);
      break;
    }
    v = get_rec(p);
  }
  return v;
}

constexpr int kLumaKeys = kClusterCtas * kTypes;

// The barriers of the luma keys: one arrival (arm) and 28 keys of 8 bytes each
// a block, two barriers taken in turn.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void key_bar_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void key_bar_arm(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "n"(kLumaKeys * 8)
               : "memory");
}
__device__ __forceinline__ void put_key(const unsigned long long* slot, const unsigned long long* bar, int cta,
                                        unsigned long long key) {
  uint32_t rs, rb;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rs) : "r"(smem_addr(slot)), "r"(cta));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(smem_addr(bar)), "r"(cta));
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u64 [%0], %1, [%2];" ::"r"(rs), "l"(key), "r"(rb)
               : "memory");
}
// False when the limit has passed.
__device__ __forceinline__ bool wait_keys(const unsigned long long* bar, uint32_t phase, uint32_t* err) {
  for (int it = 1;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(phase)
        : "memory");
    if (__all_sync(0xffffffffu, ok != 0)) return true;
    if (it > kMaxBarPolls) {
      if ((threadIdx.x & 31) == 0) atomicExch(err, 1u);
      return false;
    }
    if (it > 1024) __nanosleep(500);
  }
}

// The chroma warps' marks of a block (the fetching warp; lanes 0 and 1).
__device__ __forceinline__ bool wait_marks(const unsigned long long* mark, uint32_t seq, uint32_t* err) {
  const int lane = threadIdx.x & 31;
  for (int it = 1; !__all_sync(0xffffffffu, lane >= 2 || (uint32_t)get_word(mark + (lane & 1)) == seq); ++it) {
    if (it > kMaxWordPolls) {
      if (lane == 0) atomicExch(err, 1u);
      return false;
    }
    __nanosleep(200);
  }
  return true;
}

// Until the CTA's luma warps have block seq's edges: a ticket taken earlier
// would sit behind a block that is still waiting, while another cluster may be
// free to code it.
__device__ __forceinline__ bool wait_begun(const uint32_t* begun, uint32_t seq, uint32_t* err) {
  for (int it = 1; !__all_sync(0xffffffffu, *(volatile const uint32_t*)begun == seq); ++it) {
    if (it > 2 * kMaxWordPolls) {
      if ((threadIdx.x & 31) == 0) atomicExch(err, 1u);
      return false;
    }
    __nanosleep(100);
  }
  return true;
}

// The block of sequence number seq (a warp, all lanes the same).  Its word comes
// from the cluster's fetching warp, which writes it to every CTA or, when one of
// its own waits has run out, to none: every warp of the cluster gets the same
// blocks and leaves at the same one.
constexpr unsigned long long kEnd = 1ull << 39;
__device__ __forceinline__ unsigned long long wait_next(const unsigned long long* next, uint32_t seq, uint32_t* err) {
  unsigned long long v = get_word(next);
  for (int it = 1; !__all_sync(0xffffffffu, (uint32_t)(v >> 40) == (seq & kSeqMask)); ++it) {
    if (it > 4 * kMaxWordPolls) {
      if ((threadIdx.x & 31) == 0) atomicExch(err, 1u);
      return kEnd;
    }
    if (it > 4) __nanosleep(it > 4096 ? 400 : 100);
    v = get_word(next);
  }
  return v;
}

// One chroma plane of a block on the last warp: UV_DC_PRED and DCT_DCT, 8x8 in
// 4:4:4 and 4x4 in 4:2:0.  Only the levels and the reconstruction are wanted,
// so the chain stops after the inverse.  Every group of lanes computes the
// block; the first one writes it.
struct ChromaBlock {
  uint16_t* rec;
  int32_t* lv;
  int stride, n;
  int32_t dc;
};

// The source and the DC prediction.
__device__ __forceinline__ ChromaBlock chroma_start(StepShared& S, const EncArgs& a, uint4* edges, int pl, int b,
                                                    int nbx, int px, int py, bool has_t, bool has_l, uint32_t* err) {
  const int lane = threadIdx.x & 31;
  const int n = a.sub ? 4 : 8, ln = a.sub ? 2 : 3;
  const int cx = a.sub ? px / 2 : px, cy = a.sub ? py / 2 : py, stride = a.pc.stride;
  for (int i = lane; i < n * n; i += 32) {
    const int y = i >> ln, x = i & (n - 1);
    S.csrc[x * n + y] = (int16_t)a.src[1 + pl][(size_t)(cy + y) * stride + cx + x];
  }
  uint32_t s = 0;  // dc_pred_sq_at
  if ((lane == 0 && has_t) || (lane == 1 && has_l)) {
    const uint4 v = wait_rec(edge_rec(edges, lane == 0 ? b - nbx : b - 1, 1 + pl, lane), err);
    s = __dp4a(v.x, 0x01010101u, __dp4a(v.y, 0x01010101u, 0u));  // 4:2:0 leaves the upper four bytes 0
  }
  s = __reduce_add_sync(0xffffffffu, s);
  ChromaBlock k;
  k.rec = a.rec[1 + pl] + (size_t)cy * stride + cx;
  k.lv = (pl == 0 ? a.lv_u : a.lv_v) + (size_t)b * n * n;
  k.stride = stride;
  k.n = n;
  k.dc = (has_t && has_l) ? (n + (int)s) >> (ln + 1) : ((has_t || has_l) ? ((n >> 1) + (int)s) >> ln : 128);
  return k;
}

// The reconstruction from the inverse's columns v, the records, the block.
template <int N>
__device__ __forceinline__ void chroma_finish(const ChromaBlock& k, uint4* edges, int pl, int b, const int32_t* c,
                                              int32_t* v) {
  const int lane = threadIdx.x & 31;
  uint32_t col[2] = {0, 0};
#pragma unroll
  for (int y = 0; y < N; y++) {
    v[y] = min(max(k.dc + v[y], 0), 255);
    col[y >> 2] |= (uint32_t)v[y] << (8 * (y & 3));
  }
  uint32_t row = (uint32_t)v[N - 1] << (8 * (lane & 3));
  row |= __shfl_xor_sync(0xffffffffu, row, 1);
  row |= __shfl_xor_sync(0xffffffffu, row, 2);
  const uint32_t hi = N == 8 ? __shfl_sync(0xffffffffu, row, 4) : 0;
  if (lane == 0) put_rec(edge_rec(edges, b, 1 + pl, 0), row, hi, 0);
  if (lane == N - 1) put_rec(edge_rec(edges, b, 1 + pl, 1), col[0], col[1], 0);
  if (lane < N) {
#pragma unroll
    for (int y = 0; y < N; y++) {
      k.lv[y * N + lane] = c[y];
      k.rec[(size_t)y * k.stride + lane] = (uint16_t)v[y];
    }
  }
  __syncwarp();
}

// The 8x8 blocks of the frame in dependency order, coded by persistent
// clusters (one block per cluster at a time).  CTA 0's last warp takes blocks
// from the ticket counter, one ahead of the block being evaluated (`late`: only
// once that block has its edges), and writes them to every CTA.  A block's luma warps wait for the edge records of its
// left, top, top-left and, where its intra edges use them, top-right and
// bottom-left neighbours, which are its intra edges; predict the CTA's modes (a
// warp each); evaluate the candidates; and write their minimum keys (cost,
// candidate index) to every CTA.  Every warp takes the minimum of the cluster's
// 28 keys, and the lanes that hold it write the block's records first and the
// block itself behind them.  The chroma warps run beside, on their own records.
//
// What keeps the shared buffers apart: a key is written when its warp has read
// all it reads of the block, so a warp that has waited for all the keys may
// overwrite the block's source, edges and predictions.  The next block's words
// and the keys alternate between two slots: the fetching warp writes block
// n + 2 over block n's word after the luma keys and the chroma marks of block n,
// and a key of block n + 2 needs that word.
//
// Tickets follow the dependency levels, so the lowest unfinished ticket's
// cluster has nothing left to wait for: a cluster holds a later ticket only
// while it works on an earlier one.  A wait for a record that runs out of polls
// sets *err; once it is set the other waits for records stop, the blocks in hand
// are coded from what there is, and every cluster leaves at the end that its
// fetching warp writes.
// list[i] = (entry, image).
//
// Bound by the dependency chain: a level's latency is the record's way between
// two SMs, the prediction, one candidate chain and the keys' way in the
// cluster; with more blocks per level than clusters, by instruction latency and
// fetch.  Measured against done counts (a release per CTA, the edges read behind
// them) and a cluster barrier per block: 512x512 4:4:4 (402 levels) 3.37 -> 2.80
// ms, 1080p 4:2:0 (1,148) 10.05 -> 8.68; with late tickets 2.70 and 8.53.  The
// kernel's code is kept small (118 KB; 153 KB with chroma's own copy of the chain,
// both passes of the transforms written out and a poll and an edge writer per
// neighbour): 4096x4096 4:4:4 (2,354 levels of 111 blocks) 41.4 -> 31.7 ms, 1080p
// 8.53 -> 8.04.  Three CTAs per SM (80 registers) are slower: 4096x4096 44.3 ms at
// 153 KB; at 118 KB 1080p 8.63 against 8.01, 512x512 3.08 against 2.82.
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kStepThreads, MT_ENC_CTAS_PER_SM)
    encode_blocks_kernel(const JobDesc* __restrict__ jobs, const uint2* __restrict__ list, int nlist,
                         uint32_t* ticket_ctr, uint32_t* err, int late) {
  __shared__ StepShared S;
  extern __shared__ __align__(16) unsigned char group_smem[];
  mtd::GroupBuf* bufs = reinterpret_cast<mtd::GroupBuf*>(group_smem);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t < 64) S.scan.stage(t);
  if (t < 2) {  // sequence numbers start at 1
    S.next[t] = 0;
    S.begun = 0;
    S.mark[t][0] = S.mark[t][1] = 0;
    key_bar_init(&S.key_bar[t]);
    key_bar_arm(&S.key_bar[t]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster.sync();  // every CTA of the cluster has its slots set
  if (warp == kSideWarp && rank < 2) {
    if (rank == 0) {  // the fetching warp
      for (uint32_t seq = 1;; ++seq) {
        if (seq > 2 && (!wait_keys(&S.key_bar[seq & 1], ((seq - 3) >> 1) & 1, err) ||
                        !wait_marks(S.mark[seq & 1], (seq - 2) & kSeqMask, err)))
          break;
        if (late && seq > 1 && !wait_begun(&S.begun, seq - 1, err)) break;
        uint32_t stop = 0;
        if (lane == 0) {
          const uint32_t tk = atomicAdd(ticket_ctr, 1u);
          stop = *(volatile uint32_t*)err != 0 || tk >= (uint32_t)nlist;
          unsigned long long v = kEnd;
          if (!stop) {
            const uint2 ent = list[tk];
            v = ((unsigned long long)ent.y << 32) | ent.x;
          }
          v |= (unsigned long long)(seq & kSeqMask) << 40;
          for (int q = 0; q < kClusterCtas; ++q) put_word(cluster.map_shared_rank(&S.next[seq & 1], q), v);
        }
        if (__any_sync(0xffffffffu, stop != 0)) break;
      }
    }
    cluster.sync();
    return;
  }
  const int nthr = rank < 2 ? kLumaThreads : kStepThreads;
  auto cta_bar = [&]() { asm volatile("bar.sync 2, %0;" ::"r"(nthr) : "memory"); };
  const EncArgs& a = S.job.a;
  const int mlo = mode_lo(rank), nm = mode_lo(rank + 1) - mlo;  // this CTA's modes
  int cur = -1;                                                 // the image whose tables are staged
  unsigned long long ahead = 0;                                 // the next block's word, if it was there early
  for (uint32_t seq = 1;; ++seq) {
    unsigned long long nx = ahead;
    if (!__all_sync(0xffffffffu, (uint32_t)(ahead >> 40) == (seq & kSeqMask)))
      nx = wait_next(&S.next[seq & 1], seq, err);
    if (nx & kEnd) break;  // the same for every warp of the cluster
    const int img = (int)(nx >> 32) & 127;
    if (img != cur) {  // another image: its descriptor, then its tables
      cta_bar();
      const int* gj = reinterpret_cast<const int*>(jobs + img);
      int* sj = reinterpret_cast<int*>(&S.job);
      for (int i = t; i < (int)(sizeof(JobDesc) / 4); i += nthr) sj[i] = gj[i];
      cta_bar();
      const float* gy = reinterpret_cast<const float*>(S.job.cy);
      float* sy = reinterpret_cast<float*>(&S.cy);
      for (int i = t; i < (int)(sizeof(mt_coef_costs) / 4); i += nthr) sy[i] = gy[i];
      if (t < 64) S.py.stage(t, a.qy, a.tly, a.has_qm_y ? S.job.qmy : nullptr, 64);
      else if (t < 128) S.pc.stage(t - 64, a.qc, a.tlc, a.has_qm_c ? S.job.qmc : nullptr, a.sub ? 16 : 64);
      cta_bar();
      for (int i = t; i < nm * kTypes * 64; i += nthr) {
        const int m = i / (kTypes * 64), x = i / 64 % kTypes;
        S.head[m][x][i & 63] = mtd::coop8_rate_head(S.cy, S.cy.txb_skip[0][0], mlo + m, x, i & 63);
      }
      cta_bar();
      cur = img;
    }
    uint4* const edges = S.job.edges;
    const int nbx = a.w8 / 8;
    const uint32_t ent = (uint32_t)nx;
    const int bx = (int)(ent & 2047), by = (int)(ent >> 11) & 2047, b = by * nbx + bx;
    const int px = bx * 8, py = by * 8;
    // neighbours outside the block's tile are unavailable (AV1 intra edges and
    // contexts stop at tile edges)
    const bool has_l = ent & kHasL, has_t = ent & kHasT, have_tr = ent & kHasTr, have_bl = ent & kHasBl;
    const bool chroma = warp == kSideWarp;
    auto chroma_done = [&]() {
      if (lane == 0) put_word(cluster.map_shared_rank(&S.mark[seq & 1][rank - 2], 0), seq & kSeqMask);
    };
    ChromaBlock cb;
    if (chroma) {
      cb = chroma_start(S, a, edges, rank - 2, b, nbx, px, py, has_t, has_l, err);
      __syncwarp();
      if (a.sub) {
        const mtd::Coop<4> g;
        mtd::GroupBuf& o = bufs[4 * kTypes + (lane >> 2)];
        int32_t c[4], v[4];
        float at[4];
        int e[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
          e[x] = S.scan.row4[g.j][x];
          v[x] = S.csrc[g.j * 4 + x] - cb.dc;
        }
        mtd::coop4_fwd(v, S.pc, c, at, o, g);
        mtd::coop_trellis<4>(c, at, e, S.pc, o, g);
        mtd::coop4_inv(c, S.pc, v, o, g);
        chroma_finish<4>(cb, edges, rank - 2, b, c, v);
        chroma_done();
        continue;
      }
      for (int i = lane; i < 64; i += 32) S.ccol[i] = (int16_t)(S.csrc[i] - cb.dc);
      __syncwarp();
    }
    if (!chroma) {
      // the intra edges with their fills (predict_sq_at), a warp per neighbour
      // (left, top, top-left, top-right, bottom-left), a lane per sample, and the
      // source block
      if (warp < 5) {
        int16_t* const A = S.edge.a + 2;
        int16_t* const L = S.edge.l + 2;
        const bool up = warp == 1 || warp == 3;  // a row of the above edge, else a column of the left one
        int16_t* const e = (up ? A : L) + (warp > 2 ? 8 : 0);
        const bool have = warp == 0 ? has_l : (warp == 1 ? has_t : (warp == 2 ? has_l && has_t : (up ? have_tr : have_bl)));
        const int from = b + (warp == 1 ? -nbx : (warp == 2 ? -nbx - 1 : (warp == 3 ? 1 - nbx : (warp == 4 ? nbx - 1 : -1))));
        if (have) {
          const uint4 r = wait_rec(edge_rec(edges, from, 0, !(up || warp == 2)), err);
          const int k = min(lane, 7);  // an unavailable far side repeats the last sample
          const int16_t v = (int16_t)(((k < 4 ? r.x : r.y) >> (8 * (k & 3))) & 255);
          if (warp == 2) {
            if (lane == 7) A[-1] = L[-1] = v;
          } else {
            if (lane < (warp < 2 && !(up ? have_tr : have_bl) ? 16 : 8)) e[lane] = v;
            if (warp < 2) {
              if (!(up ? has_l : has_t)) {  // the other side repeats this one's first sample
                if (lane < 17) (up ? L : A)[lane - 1] = (int16_t)(r.x & 255);
                if (lane == 0) e[-1] = v;
              }
              if (lane == 0) S.nb_mode[1 - warp] = (uint8_t)r.w;
            }
          }
        } else if (warp < 2) {
          if (lane == 0) S.nb_mode[1 - warp] = MT_DC_PRED;
          if (!has_l && !has_t && lane < 17) e[lane - 1] = (int16_t)(lane == 0 ? 128 : (up ? 127 : 129));
        }
      } else {
        const int i = t - 160, y = i >> 3, x = i & 7;
        S.src[x * 8 + y] = (int16_t)a.src[0][(size_t)(py + y) * a.py.stride + px + x];
      }
      luma_bar();
      if (t == 0) *(volatile uint32_t*)&S.begun = seq;
      if (warp < nm)
        mtd::coop8_predict(mlo + warp, S.edge, has_t, has_l, is_smooth(S.nb_mode[0]) || is_smooth(S.nb_mode[1]), S.src,
                           S.pcol[warp], S.rcol[warp], S.rrow[warp], S.pb[warp]);
      luma_bar();
    }
    const mtd::Coop<8> g;
    const int slot = lane >> 3, ms = min(slot, nm - 1), TX = chroma ? MT_TX_DCT_DCT : warp;
    mtd::GroupBuf& o = bufs[4 * warp + slot];
    const mtd::CoopPlane& P = chroma ? S.pc : S.py;
    int32_t c[8], rv[8];  // this lane's levels (row j) and reconstruction (column j)
    int e[8];
    {
      const uint2 w = *reinterpret_cast<const uint2*>(S.scan.row8[g.j]);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        e[k] = (w.x >> (8 * k)) & 255;
        e[k + 4] = (w.y >> (8 * k)) & 255;
      }
    }
    float at[8];
    {
      int32_t v[8];
      mtd::load8((chroma ? S.ccol : (mtd::coop8_by_rows(TX) ? S.rrow[ms] : S.rcol[ms])) + g.j * 8, v);
      mtd::coop8_fwd(TX, v, P, c, at, o, g);
    }
    const int eob = mtd::coop_trellis<8>(c, at, e, P, o, g);
    mtd::coop8_inv(TX, c, P, rv, o, g);
    if (chroma) {
      chroma_finish<8>(cb, edges, rank - 2, b, c, rv);
      chroma_done();
      continue;
    }
    int32_t d[8], pr[8];
    mtd::load8(S.pcol[ms] + g.j * 8, pr);
    mtd::load8(S.src + g.j * 8, d);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      rv[k] = min(max(pr[k] + rv[k], 0), 255);
      d[k] -= rv[k];
    }
    const uint32_t satd = mtd::coop8_satd(d, g);
    float price = __fmul_rn(__fmul_rn(__fmul_rn((float)satd, fmaxf((float)S.py.q.ac_q, 1.0f)), 0.25f), a.py.satd_scale);
    if (a.py.satd_bridge != 0.0f) price = __fmul_rn(price, a.py.satd_bridge);
    const float* const head = S.head[ms][TX];
    const float bits = mtd::coop8_rate(c, e, eob, S.cy, S.cy.txb_skip[0][1], [head](int k) { return head[k]; },
                                       S.cy.dc_sign[0], o, g);
    const float cost = __fadd_rn(price, __fmul_rn(a.py.mode_lambda, bits));
    unsigned long long k = ~0ull;
    if (g.j == 0 && slot < nm)
      k = ((unsigned long long)__float_as_uint(cost) << 32) | (unsigned)((mlo + ms) * kTypes + TX);
#pragma unroll
    for (int s = 8; s < 32; s <<= 1) {
      const unsigned long long ok = __shfl_xor_sync(0xffffffffu, k, s);
      k = ok < k ? ok : k;
    }
    k = __shfl_sync(0xffffffffu, k, 0);
    if (lane < kClusterCtas) put_key(&S.key[seq & 1][rank * kTypes + warp], &S.key_bar[seq & 1], lane, k);
    // every group's records, while the keys are on their way
    uint32_t row = (uint32_t)rv[7] << (8 * (g.j & 3)), col[2] = {0, 0};
    row |= __shfl_xor_sync(0xffffffffu, row, 1);
    row |= __shfl_xor_sync(0xffffffffu, row, 2);
    const uint32_t row_hi = __shfl_sync(0xffffffffu, row, 4, 8);
#pragma unroll
    for (int q = 0; q < 8; ++q) col[q >> 2] |= (uint32_t)rv[q] << (8 * (q & 3));
    ahead = get_word(&S.next[(seq + 1) & 1]);
    const bool complete = wait_keys(&S.key_bar[seq & 1], ((seq - 1) >> 1) & 1, err);
    if (t == 0 && complete) key_bar_arm(&S.key_bar[seq & 1]);  // for block seq + 2
    const unsigned long long all = S.key[seq & 1][lane];
    const uint32_t cst = lane < kLumaKeys ? (uint32_t)(all >> 32) : 0xffffffffu;
    const uint32_t low = __reduce_min_sync(0xffffffffu, cst);
    const int wi = (int)__reduce_min_sync(0xffffffffu, cst == low && lane < kLumaKeys ? (uint32_t)all : 255u);
    const int wm = wi / kTypes;
    if (rank == mode_rank(wm) && warp == wi - wm * kTypes && slot == wm - mlo) {
      const int j = g.j;
      if (j == 0) put_rec(edge_rec(edges, b, 0, 0), row, row_hi, (uint32_t)wm);
      if (j == 7) put_rec(edge_rec(edges, b, 0, 1), col[0], col[1], (uint32_t)wm);
      int32_t* lv = a.lv_y + (size_t)b * 64 + j;
      uint16_t* r = a.rec[0] + (size_t)py * a.py.stride + px + j;
#pragma unroll
      for (int q = 0; q < 8; ++q) r[(size_t)q * a.py.stride] = (uint16_t)rv[q];
#pragma unroll
      for (int q = 0; q < 8; ++q) lv[q * 8] = c[q];
      if (j == 0) {
        a.mode[b] = (uint8_t)wm;
        a.tx[b] = (uint8_t)warp;
      }
    }
    __syncwarp();
  }
  // None may leave while another CTA can still write to its shared memory: the
  // keys of the last block have been waited for, unless that wait has run out.
  if (*(volatile uint32_t*)err)
    for (int i = 0; i < 32; ++i) __nanosleep(1000);
  cluster.sync();
}

// One plane of 8-bit samples into the coder's padded u16 plane, edge samples
// replicated past the displayed size (pad_to_mult8_u16, src/dispatch.rs:113-131).
__global__ void pad_plane_kernel(const uint8_t* __restrict__ in, int w, int h, uint16_t* __restrict__ out, int pw,
                                 int ph) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= pw || y >= ph) return;
  out[(size_t)y * pw + x] = in[(size_t)min(y, h - 1) * w + min(x, w - 1)];
}

// The deblocking maps of a frame of 8x8 blocks and transforms, per 4x4 unit: the
// block's width and height in units (2), whether the unit starts a block's
// column or row, and the width and height for chroma.  Four units per thread
// (w4 is even, n4 a multiple of four); written here instead of on the host
// (4096x4096: 2.6 ms of loops and a 6.3 MB copy).
__global__ void block_maps_kernel(uint32_t* __restrict__ maps, int w4, int n4) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, q = n4 / 4;
  if (i >= q) return;
  uint32_t rows = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) rows |= (uint32_t)(((4 * i + k) / w4 & 1) == 0) << (8 * k);
  maps[i] = maps[q + i] = maps[4 * q + i] = maps[5 * q + i] = 0x02020202u;
  maps[2 * q + i] = 0x00010001u;
  maps[3 * q + i] = rows;
}

// The ticket list, wave by wave over all images of a launch: a count per wave,
// a scan, and a place for each block (any order inside a wave).
template <bool PLACE>
__global__ void __launch_bounds__(256) list_kernel(const JobDesc* __restrict__ jobs, uint32_t* __restrict__ wave,
                                                   uint2* __restrict__ list) {
  const EncArgs& a = jobs[blockIdx.y].a;
  const int nbx = a.w8 / 8, nby = a.h8 / 8;
  const int b = blockIdx.x * 256 + threadIdx.x;
  if (b >= nbx * nby) return;
  const int y = b / nbx, x = b - y * nbx;
  const int tx0 = x - x % a.tile_w8, ty0 = y - y % a.tile_h8;
  const int at = kWaveCol * ((x - tx0) >> 3) + kWaveRow * ((y - ty0) >> 3) + cWave.t[y & 7][x & 7];
  if (!PLACE) {
    atomicAdd(&wave[at], 1u);
    return;
  }
  int k = 0;  // z-order index
#pragma unroll
  for (int i = 0; i < 3; ++i) k |= ((x >> i) & 1) << (2 * i) | ((y >> i) & 1) << (2 * i + 1);
  int zx, zy;
  bool thr, lhb;
  zorder(k, &zx, &zy, &thr, &lhb);
  const bool l = x > tx0, t = y > ty0;
  uint32_t e = (uint32_t)x | ((uint32_t)y << 11) | (l ? kHasL : 0) | (t ? kHasT : 0);
  if (thr && t && x + 1 < min(tx0 + a.tile_w8, nbx)) e |= kHasTr;
  if (lhb && l && y + 1 < min(ty0 + a.tile_h8, nby)) e |= kHasBl;
  list[atomicAdd(&wave[at], 1u)] = make_uint2(e, blockIdx.y);
}

__global__ void __launch_bounds__(1024) wave_scan_kernel(uint32_t* __restrict__ wave, int n) {
  __shared__ uint32_t part[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  uint32_t carry = 0;
  for (int b = 0; b < n; b += 1024) {
    const uint32_t v = b + t < n ? wave[b + t] : 0;
    uint32_t s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t q = __shfl_up_sync(~0u, s, o);
      if (lane >= o) s += q;
    }
    if (lane == 31) part[w] = s;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int i = 0; i < 32; ++i) {
      if (i < w) before += part[i];
      all += part[i];
    }
    if (b + t < n) wave[b + t] = carry + before + s - v;
    carry += all;
    __syncthreads();
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side.

namespace {

// The device buffers of the images of an encode call.  Each device keeps
// sets of them -- one per image of the largest batch seen, each grown to the
// largest frame it carried, each with two streams -- until
// mt_encode_release_buffers or exit.  A call uses them when no other call on
// that device holds them; otherwise it allocates its own for the call.
constexpr int kSlots = 16;
enum Slot { kRgb, kPlanes, kTables, kDecisions, kLevels, kSched, kPlan, kTokens, kMaps, kDeblock, kFiltered, kSkip8,
            kCdef, kDigits, kList, kJobs };
struct BufSet {
  void* p[kSlots] = {};
  size_t cap[kSlots] = {};
  cudaStream_t st[2] = {nullptr, nullptr};
};
struct Arena {
  std::mutex mu;
  std::vector<BufSet> sets;
};
Arena g_arenas[16];

class Buffers {
 public:
  explicit Buffers(int n) : own_((size_t)n) {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 16 && g_arenas[dev].mu.try_lock()) {
      ar_ = &g_arenas[dev];
      if ((int)ar_->sets.size() < n) ar_->sets.resize((size_t)n);
    }
  }
  ~Buffers() {
    if (ar_) ar_->mu.unlock();
    for (BufSet& b : own_) {
      for (void* q : b.p) cudaFree(q);
      for (cudaStream_t s : b.st)
        if (s) cudaStreamDestroy(s);
    }
  }
  // slack: what a buffer whose size follows the picture's content gets beside,
  // so that the next picture seldom has to grow it (a free waits for the device).
  template <class T>
  T* get(int i, Slot s, size_t n, bool slack = false) {
    BufSet& b = set(i);
    n = n ? n : 1;
    if (b.cap[s] < n) {
      cudaFree(b.p[s]);
      b.p[s] = nullptr;
      b.cap[s] = 0;
      const size_t more = slack ? n + n / 4 : n;
      if (cudaMalloc(&b.p[s], more) == cudaSuccess) {
        b.cap[s] = more;
      } else {  // where the slack does not fit, without it
        cudaGetLastError();
        if (more == n || cudaMalloc(&b.p[s], n) != cudaSuccess) return nullptr;
        b.cap[s] = n;
      }
    }
    return reinterpret_cast<T*>(b.p[s]);
  }
  cudaStream_t stream(int i, int k) {  // 0: the image's own, 1: its entropy coding beside the filters
    BufSet& b = set(i);
    if (!b.st[k] && cudaStreamCreateWithFlags(&b.st[k], cudaStreamNonBlocking) != cudaSuccess) b.st[k] = nullptr;
    return b.st[k];
  }

 private:
  BufSet& set(int i) { return ar_ ? ar_->sets[(size_t)i] : own_[(size_t)i]; }
  Arena* ar_ = nullptr;
  std::vector<BufSet> own_;
};

// The stats of one call: copies, launches and CUDA-event times (the events
// exist only when the caller asked for stats).
struct CallStats {
  mt_encode_stats* s;
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};  // call start, blocks start, blocks end, call end
  explicit CallStats(mt_encode_stats* st) : s(st) {
    if (!s) return;
    memset(s, 0, sizeof(*s));
    for (auto& e : ev) cudaEventCreate(&e);
  }
  ~CallStats() {
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
  }
  void h2d(size_t n) {
    if (s) s->h2d_bytes += n;
  }
  void d2h(size_t n) {
    if (s) s->d2h_bytes += n;
  }
  void launches(int n) {
    if (s) s->kernel_launches += (uint32_t)n;
  }
  void mark(int k, cudaStream_t st) {
    if (s) cudaEventRecord(ev[k], st);
  }
  void finish() {
    if (!s) return;
    cudaEventSynchronize(ev[3]);
    cudaEventElapsedTime(&s->blocks_ms, ev[1], ev[2]);
    cudaEventElapsedTime(&s->call_ms, ev[0], ev[3]);
  }
};


// One image of an encode call, through its three phases.
struct Job {
  // the call's inputs
  const uint8_t* rgb = nullptr;
  bool rgb_on_device = false;
  const uint8_t* const* yuv = nullptr;
  uint32_t width = 0, height = 0;
  const mt_encode_config* cfg = nullptr;
  uint8_t** out = nullptr;
  size_t* out_len = nullptr;
  uint16_t** recon_out = nullptr;
  mt_encode_stats* stats = nullptr;
  // the frame
  mt_encode_plan plan = {};
  int sub = 0, sx = 0, nbx = 0, nby = 0, nb = 0, sb_cols = 0, sb_rows = 0, cl = 0;
  int32_t tcl = 0, trl = 0;      // TileColsLog2, TileRowsLog2
  int tile_sb_w = 0, tile_sb_h = 0;  // the uniform tile size in superblocks
  int32_t pw = 0, ph = 0, pcw = 0, pch = 0;
  size_t ny = 0, nc = 0;
  EncArgs a = {};
  JobDesc desc = {};
  uint16_t* src[3] = {};
  uint16_t* rec[3] = {};
  mth::StreamGeom sg = {};
  mth::StreamInput si = {};
  void* d_plan = nullptr;
  uint8_t* d_cdfs = nullptr;
  cudaStream_t st = nullptr, st_code = nullptr;
  std::unique_ptr<CallStats> cs;
  int rc = MT_OK;
};

}  // namespace

namespace mth {
int cdef_frame_enqueue(uint16_t* d_y, uint16_t* d_u, uint16_t* d_v, const uint16_t* d_src_y, const uint16_t* d_src_u,
                       const uint16_t* d_src_v, const uint8_t* d_skip8, const mt_cdef_params* prm, void* d_scratch,
                       cudaEvent_t decided, const int32_t** d_bits, const uint8_t** d_grid, cudaStream_t st);
int cdef_frame_decision(const mt_cdef_params* prm, void* d_scratch, mt_cdef_decision* out, uint8_t* grid,
                        cudaStream_t st);
void cdef_frame_transfer_bytes(const mt_cdef_params* p, size_t* d2h, size_t* h2d);
extern thread_local int cdef_last_launches;
extern thread_local int deblock_last_launches;
}  // namespace mth

extern "C" {
int mt_coef_costs_build(const mt_coef_cdfs* cdfs, mt_coef_costs* out);
const uint8_t* mt_qm_row(int32_t qm_level, int32_t chroma, int32_t w, int32_t h);
}

namespace {

// The dependency levels of a w x h-block tile (a statistic: the length of the
// critical path).  From five superblocks on, one more column or row adds the
// same number, so a larger tile's count follows from those of small ones.
int tile_levels(int w, int h) {
  const int more_c = std::max(0, (w + 7) / 8 - 4), more_r = std::max(0, (h + 7) / 8 - 4);
  auto count = [](int nbx, int nby) {
    std::vector<int> T((size_t)nbx * nby, 0);
    int last = 0;
    for (int sb = 0; sb < ((nbx + 7) / 8) * ((nby + 7) / 8); ++sb)
      for (int k = 0; k < 64; ++k) {
        int bx, by;
        bool thr, lhb;
        zorder(k, &bx, &by, &thr, &lhb);
        const int x = sb % ((nbx + 7) / 8) * 8 + bx, y = sb / ((nbx + 7) / 8) * 8 + by;
        if (x >= nbx || y >= nby) continue;
        int lv = 0;
        auto dep = [&](int xx, int yy) { lv = std::max(lv, T[(size_t)yy * nbx + xx] + 1); };
        if (x) dep(x - 1, y);
        if (y) dep(x, y - 1);
        if (x && y) dep(x - 1, y - 1);
        if (thr && y && x + 1 < nbx) dep(x + 1, y - 1);
        if (lhb && x && y + 1 < nby) dep(x - 1, y + 1);
        T[(size_t)y * nbx + x] = lv;
        last = std::max(last, lv);
      }
    return last + 1;
  };
  w -= 8 * more_c;
  h -= 8 * more_r;
  const int n = count(w, h);
  return n + (more_c ? more_c * (n - count(w - 8, h)) : 0) + (more_r ? more_r * (n - count(w, h - 8)) : 0);
}

}  // namespace

namespace mth {
// The most blocks that a tile of cols x rows superblocks has in one wave (a
// tile's partial superblocks have fewer): a superblock's blocks by their wave,
// then along a row and over the rows as running sums at the waves' strides.
int widest_wave(int cols, int rows) {
  const int n = kWaveCol * (cols - 1) + kWaveRow * (rows - 1) + kWave.last + 1;
  std::vector<int> sum((size_t)n), at((size_t)n, 0);
  for (const auto& row : kWave.t)
    for (uint8_t t : row) at[t] += 1;
  auto along = [&](int stride, int count) {
    for (int i = 0; i < n; ++i)
      sum[(size_t)i] = at[(size_t)i] + (i >= stride ? sum[(size_t)(i - stride)] : 0) -
                       (i >= stride * count ? at[(size_t)(i - stride * count)] : 0);
    at.swap(sum);
  };
  along(kWaveCol, cols);
  along(kWaveRow, rows);
  return *std::max_element(at.begin(), at.end());
}
}  // namespace mth

namespace {

int frame_levels(int nbx, int nby, int tile_w8, int tile_h8) {
  int n = 0;  // the full tiles and the last ones of the rows and columns
  for (int w : {std::min(tile_w8, nbx), nbx - (nbx - 1) / tile_w8 * tile_w8})
    for (int h : {std::min(tile_h8, nby), nby - (nby - 1) / tile_h8 * tile_h8}) n = std::max(n, tile_levels(w, h));
  return n;
}

// Validation, device buffers, the input on the device (colour conversion or
// padding), the frame laws' tables and the kernel arguments of image i.
int job_setup(Job& j, Buffers& buf, int i) {
  if (!j.out || !j.out_len) return MT_ERR_INVALID_INPUT;
  *j.out = nullptr;
  *j.out_len = 0;
  int rc = mt_encode_config_validate(j.cfg);
  if (rc != MT_OK) return rc;
  const mt_encode_config* cfg = j.cfg;
  const uint32_t width = j.width, height = j.height;
  rc = mt_validate_rgb8_input(width, height, (size_t)width * height * 3);
  if (rc != MT_OK) return rc;
  if (!j.rgb && (!j.yuv || !j.yuv[0] || !j.yuv[1] || !j.yuv[2])) return MT_ERR_INVALID_INPUT;
  if (cfg->chroma != MT_CHROMA_420 && cfg->chroma != MT_CHROMA_444) return MT_ERR_UNSUPPORTED_CHROMA_FORMAT;
  if ((rc = mt_encode_config_effective(cfg, &j.plan)) != MT_OK) return rc;
  if (j.plan.base_q_idx == 0) return MT_ERR_UNSUPPORTED;  // lossless is a separate encoder
  const int sub = j.sub = cfg->chroma == MT_CHROMA_420 ? 2 : 0;
  const int sx = j.sx = sub ? 1 : 0;
  if ((rc = mt_padded_plane_dims((int)width, (int)height, sub, &j.pw, &j.ph, &j.pcw, &j.pch)) != MT_OK) return rc;
  const int32_t pw = j.pw, ph = j.ph, pcw = j.pcw, pch = j.pch;
  const int nbx = j.nbx = pw / 8, nby = j.nby = ph / 8, nb = j.nb = nbx * nby;
  const int sb_cols = j.sb_cols = (pw + 63) / 64, sb_rows = j.sb_rows = (ph + 63) / 64;
  // the spec-minimum uniform tiling (src/coder/frame_encode.rs:75-80): one
  // tile unless the frame exceeds the AV1 maximum tile width (64 superblocks)
  // or area (2304 superblocks)
  if ((rc = mt_tiling_spec_min(pw, ph, &j.tcl, &j.trl)) != MT_OK) return rc;
  j.tile_sb_w = (sb_cols + (1 << j.tcl) - 1) >> j.tcl;
  j.tile_sb_h = (sb_rows + (1 << j.trl) - 1) >> j.trl;
  const int cl = j.cl = sub ? 16 : 64;  // chroma levels per block
  // quantisers, QM rows, the default luma CDF slice and its bit costs, lambdas
  mt_quant qy, qc;
  if (mt_quant_init(j.plan.base_q_idx, 8, j.plan.qm_y, &qy) != MT_OK) return MT_ERR_INVALID_INPUT;
  if (mt_quant_init_chroma(j.plan.base_q_idx, 0, 0, 8, j.plan.qm_u, &qc) != MT_OK) return MT_ERR_INVALID_INPUT;
  mt_coef_cdfs cdy;
  mt_coef_costs cy;
  const int qctx = mt_qcat(j.plan.base_q_idx);
  mt_coef_cdfs_default(qctx, 8, 8, 0, &cdy);
  mt_coef_costs_build(&cdy, &cy);
  mt_rd_lambdas lam;
  if (mt_rd_lambdas_init(j.plan.base_q_idx, qy.dc_q, sub, 8, &lam) != MT_OK) return MT_ERR_INVALID_INPUT;
  const uint8_t* qmy = mt_qm_row(j.plan.qm_y, 0, 8, 8);
  const uint8_t* qmc = mt_qm_row(j.plan.qm_u, 1, sub ? 4 : 8, sub ? 4 : 8);
  // device buffers
  const size_t ny = j.ny = (size_t)pw * ph, nc = j.nc = (size_t)pcw * pch;
  const size_t in_bytes = j.rgb ? (size_t)width * height * 3
                                : (size_t)width * height + 2 * (size_t)((width + sx) >> sx) * ((height + sx) >> sx);
  uint8_t* d_rgbbuf = buf.get<uint8_t>(i, kRgb, j.rgb_on_device ? 1 : in_bytes);
  uint16_t* d_planes = buf.get<uint16_t>(i, kPlanes, (ny + 2 * nc) * 2 * 2);
  constexpr size_t cost_bytes = (sizeof(mt_coef_costs) + 128 + 15) & ~(size_t)15;
  const size_t cdf_bytes = mth::stream_cdf_bytes();
  uint8_t* d_tabs = buf.get<uint8_t>(i, kTables, cost_bytes + cdf_bytes);
  uint8_t* d_decs = buf.get<uint8_t>(i, kDecisions, (size_t)nb * 2);
  int32_t* d_levels = buf.get<int32_t>(i, kLevels, (size_t)nb * (64 + 2 * cl) * 4);
  mth::StreamGeom& sg = j.sg;
  sg.nbx = nbx;
  sg.nby = nby;
  sg.sub = sub;
  sg.sb_cols = sb_cols;
  sg.sb_rows = sb_rows;
  sg.tile_w8 = j.tile_sb_w * 8;
  sg.tile_h8 = j.tile_sb_h * 8;
  sg.tcols = (sb_cols + j.tile_sb_w - 1) / j.tile_sb_w;
  sg.trows = (sb_rows + j.tile_sb_h - 1) / j.tile_sb_h;
  j.d_plan = buf.get<void>(i, kPlan, mth::stream_plan_bytes(sg));
  uint4* d_edges = buf.get<uint4>(i, kSched, (size_t)nb * 6 * sizeof(uint4));
  const cudaStream_t st = j.st = buf.stream(i, 0);
  j.st_code = buf.stream(i, 1);
  if (!d_rgbbuf || !d_planes || !d_tabs || !d_decs || !d_levels || !j.d_plan || !d_edges || !st || !j.st_code)
    return MT_ERR_DEVICE;
  uint16_t* const* src = j.src;
  for (int p = 0; p < 3; ++p) {
    j.src[p] = d_planes + (p == 0 ? 0 : ny + (size_t)(p - 1) * nc);
    j.rec[p] = d_planes + ny + 2 * nc + (p == 0 ? 0 : ny + (size_t)(p - 1) * nc);
  }
  mt_coef_costs* d_cy = reinterpret_cast<mt_coef_costs*>(d_tabs);
  uint8_t* d_qmy = reinterpret_cast<uint8_t*>(d_cy + 1);
  uint8_t* d_qmc = d_qmy + 64;
  j.cs.reset(new CallStats(j.stats));
  CallStats& cs = *j.cs;
  cs.mark(0, st);
  if (j.rgb) {
    const uint8_t* d_in = j.rgb;
    if (!j.rgb_on_device) {
      if (cudaMemcpyAsync(d_rgbbuf, j.rgb, in_bytes, cudaMemcpyHostToDevice, st) != cudaSuccess) return MT_ERR_DEVICE;
      cs.h2d(in_bytes);
      d_in = d_rgbbuf;
    }
    if ((rc = mt_csc_rgb8_device(d_in, (int)width, (int)height, sub, src[0], src[1], src[2], st)) != MT_OK) return rc;
    cs.launches(2);
  } else {
    const int cw = (int)((width + sx) >> sx), ch = (int)((height + sx) >> sx);
    uint8_t* d_in = d_rgbbuf;
    const size_t n0 = (size_t)width * height, n1 = (size_t)cw * ch;
    if (cudaMemcpyAsync(d_in, j.yuv[0], n0, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(d_in + n0, j.yuv[1], n1, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(d_in + n0 + n1, j.yuv[2], n1, cudaMemcpyHostToDevice, st) != cudaSuccess)
      return MT_ERR_DEVICE;
    pad_plane_kernel<<<dim3((pw + 127) / 128, ph), 128, 0, st>>>(d_in, (int)width, (int)height, src[0], pw, ph);
    pad_plane_kernel<<<dim3((pcw + 127) / 128, pch), 128, 0, st>>>(d_in + n0, cw, ch, src[1], pcw, pch);
    pad_plane_kernel<<<dim3((pcw + 127) / 128, pch), 128, 0, st>>>(d_in + n0 + n1, cw, ch, src[2], pcw, pch);
    cs.h2d(n0 + 2 * n1);
    cs.launches(3);
  }
  cudaMemsetAsync(d_tabs, 32, sizeof(mt_coef_costs) + 128, st);  // flat QM weights past a 4x4 row
  cudaMemcpyAsync(d_cy, &cy, sizeof(cy), cudaMemcpyHostToDevice, st);
  if (qmy) cudaMemcpyAsync(d_qmy, qmy, 64, cudaMemcpyHostToDevice, st);
  if (qmc) cudaMemcpyAsync(d_qmc, qmc, sub ? 16 : 64, cudaMemcpyHostToDevice, st);
  j.d_cdfs = d_tabs + cost_bytes;
  cudaMemcpyAsync(j.d_cdfs, mth::stream_cdf_table(qctx, sub), cdf_bytes, cudaMemcpyHostToDevice, st);
  cs.h2d(sizeof(mt_coef_costs) + cdf_bytes + (qmy ? 64 : 0) + (qmc ? (sub ? 16 : 64) : 0));
  EncArgs& a = j.a;
  a = EncArgs{};
  for (int p = 0; p < 3; ++p) {
    a.src[p] = j.src[p];
    a.rec[p] = j.rec[p];
  }
  a.py = {};
  a.py.tx_size = 8;
  a.py.bd = 8;
  a.py.frame_w = pw;
  a.py.frame_h = ph;
  a.py.stride = pw;
  a.py.trellis_lambda0 = lam.trellis_lambda0;
  a.py.mode_lambda = lam.mode_lambda;
  a.py.satd_scale = lam.satd_scale;
  a.py.satd_bridge = lam.satd_bridge;
  a.pc = a.py;
  a.pc.tx_size = sub ? 4 : 8;
  a.pc.frame_w = pcw;
  a.pc.frame_h = pch;
  a.pc.stride = pcw;
  a.qy = qy;
  a.qc = qc;
  a.tly = mth::scaled_trellis_lambda_host((float)qy.dc_q, lam.trellis_lambda0);
  a.tlc = mth::scaled_trellis_lambda_host((float)qc.dc_q, lam.trellis_lambda0);
  a.has_qm_y = qmy != nullptr;
  a.has_qm_c = qmc != nullptr;
  a.sub = sub;
  a.w8 = pw;
  a.h8 = ph;
  a.tile_w8 = j.tile_sb_w * 8;
  a.tile_h8 = j.tile_sb_h * 8;
  a.mode = d_decs;
  a.tx = a.mode + nb;
  a.lv_y = d_levels;
  a.lv_u = a.lv_y + (size_t)nb * 64;
  a.lv_v = a.lv_u + (size_t)nb * cl;
  j.si.mode = a.mode;
  j.si.tx = a.tx;
  j.si.lv[0] = a.lv_y;
  j.si.lv[1] = a.lv_u;
  j.si.lv[2] = a.lv_v;
  j.desc.a = a;
  j.desc.cy = d_cy;
  j.desc.qmy = d_qmy;
  j.desc.qmc = d_qmc;
  j.desc.edges = d_edges;
  if (cudaMemsetAsync(a.mode, 0, (size_t)nb * 2, st) != cudaSuccess ||
      cudaMemsetAsync(d_edges, 0, (size_t)nb * 6 * sizeof(uint4), st) != cudaSuccess)
    return MT_ERR_DEVICE;
  if (j.stats) {
    j.stats->blocks = (uint32_t)nb;
    j.stats->levels = (uint32_t)frame_levels(nbx, nby, a.tile_w8, a.tile_h8);
  }
  return MT_OK;
}

// The decisions of every image that set up, in one launch: the images'
// blocks merged wave by wave into one ticket list (each image's order is
// still a dependency order), the persistent clusters taking tickets across
// images.
// skip: tickets left out at the list's start (none but to test the waits' end).
int decide_all(std::vector<Job>& jobs, Buffers& buf, int skip) {
  std::vector<JobDesc> descs;
  std::vector<int> slot;  // job index per descriptor
  size_t total = 0;
  int waves = 0, nb_max = 0, width_max = 0;
  for (size_t i = 0; i < jobs.size(); ++i)
    if (jobs[i].rc == MT_OK) {
      const Job& j = jobs[i];
      slot.push_back((int)i);
      descs.push_back(j.desc);
      total += (size_t)j.nb;
      nb_max = std::max(nb_max, j.nb);
      const int tc = std::min(j.tile_sb_w, j.sb_cols), tr = std::min(j.tile_sb_h, j.sb_rows);
      waves = std::max(waves, kWaveCol * (tc - 1) + kWaveRow * (tr - 1) + kWave.last + 1);
      width_max += j.sg.tcols * j.sg.trows * mth::widest_wave(tc, tr);
    }
  if (slot.empty()) return MT_OK;
  const int i0 = slot[0];
  const cudaStream_t ks = jobs[(size_t)i0].st;
  uint2* d_list = buf.get<uint2>(i0, kList, total * sizeof(uint2) + ((size_t)waves + 2) * 4);
  JobDesc* d_jobs = buf.get<JobDesc>(i0, kJobs, descs.size() * sizeof(JobDesc));
  if (!d_list || !d_jobs) return MT_ERR_DEVICE;
  uint32_t* d_ctl = reinterpret_cast<uint32_t*>(d_list + total);  // [0] ticket counter, [1] timeout flag
  uint32_t* d_wave = d_ctl + 2;
  // the launch waits for every image's set-up on its own stream
  std::vector<cudaEvent_t> evs;
  for (size_t d = 1; d < slot.size(); ++d) {
    cudaEvent_t e;
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return MT_ERR_DEVICE;
    evs.push_back(e);
    cudaEventRecord(e, jobs[(size_t)slot[d]].st);
    cudaStreamWaitEvent(ks, e, 0);
  }
  if (cudaMemcpyAsync(d_jobs, descs.data(), descs.size() * sizeof(JobDesc), cudaMemcpyHostToDevice, ks) !=
          cudaSuccess ||
      cudaMemsetAsync(d_ctl, 0, ((size_t)waves + 2) * 4, ks) != cudaSuccess)
    return MT_ERR_DEVICE;
  const dim3 lg((unsigned)((nb_max + 255) / 256), (unsigned)descs.size());
  list_kernel<false><<<lg, 256, 0, ks>>>(d_jobs, d_wave, nullptr);
  wave_scan_kernel<<<1, 1024, 0, ks>>>(d_wave, waves);
  list_kernel<true><<<lg, 256, 0, ks>>>(d_jobs, d_wave, d_list);
  // one cluster per block that can run at once (no merged wave is wider than the
  // tiles' widest together) and a quarter more, since a cluster that writes its
  // block is not free yet (512x512 4:4:4, 20 blocks: 2.84 ms with 20 clusters, 2.82
  // with 25), at most as many as the SMs hold
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    return MT_ERR_DEVICE;
  const int most = std::max(1, sms * MT_ENC_CTAS_PER_SM / kClusterCtas);
  const int nclusters = std::min(width_max + width_max / 4, most);
  // With a cluster for every block that can run, a ticket is better left to the
  // cluster that can start it (1080p 9.05 -> 8.59 ms, 512x512 4:4:4 2.88 -> 2.71,
  // 2048x2048 13.3 -> 12.4); with fewer, the next ticket is wanted at once
  // (4096x4096 42.1 -> 41.0 ms).
  const int late = width_max <= most;
  for (int d : slot) {
    jobs[(size_t)d].cs->h2d(sizeof(JobDesc));
    jobs[(size_t)d].cs->mark(1, ks);
  }
  constexpr int dyn = kGroupBufs * (int)sizeof(mtd::GroupBuf);
  if (cudaFuncSetAttribute(encode_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess)
    return MT_ERR_DEVICE;
  encode_blocks_kernel<<<nclusters * kClusterCtas, kStepThreads, dyn, ks>>>(d_jobs, d_list + skip, (int)total - skip,
                                                                            d_ctl, d_ctl + 1, late);
  for (int d : slot) {
    jobs[(size_t)d].cs->mark(2, ks);
    jobs[(size_t)d].cs->launches(4);
    jobs[(size_t)d].cs->d2h(4);
  }
  // every image's finishing work waits for the launch
  cudaEvent_t done_ev;
  if (cudaEventCreateWithFlags(&done_ev, cudaEventDisableTiming) != cudaSuccess) return MT_ERR_DEVICE;
  evs.push_back(done_ev);
  cudaEventRecord(done_ev, ks);
  for (int d : slot) cudaStreamWaitEvent(jobs[(size_t)d].st, done_ev, 0);
  uint32_t timed_out = 0;
  const bool ok = cudaMemcpyAsync(&timed_out, d_ctl + 1, 4, cudaMemcpyDeviceToHost, ks) == cudaSuccess &&
                  cudaStreamSynchronize(ks) == cudaSuccess && cudaGetLastError() == cudaSuccess;
  for (cudaEvent_t e : evs) cudaEventDestroy(e);
  if (!ok || timed_out) return MT_ERR_DEVICE;
  return MT_OK;
}

// A CUDA event destroyed with its scope.
struct EventGuard {
  cudaEvent_t e = nullptr;
  ~EventGuard() {
    if (e) cudaEventDestroy(e);
  }
};

// A stream waited for when its scope ends, on every return path: the buffers
// its work uses are the next call's.
struct StreamGuard {
  cudaStream_t s;
  ~StreamGuard() { cudaStreamSynchronize(s); }
};

// Everything after the decisions for image i: the filters, with the entropy
// coding beside them on the image's second stream, headers and container.
int job_finish(Job& j, Buffers& buf, int i) {
  int rc = MT_OK;
  const cudaStream_t st = j.st;
  CallStats& cs = *j.cs;
  const mt_encode_config* cfg = j.cfg;
  const uint32_t width = j.width, height = j.height;
  const int sub = j.sub, sx = j.sx, nb = j.nb;
  const int32_t pw = j.pw, ph = j.ph;
  const size_t ny = j.ny, nc = j.nc;
  uint16_t* const* src = j.src;
  uint16_t* const* rec = j.rec;
  const cudaStream_t sc = j.st_code;
  StreamGuard code_guard{sc};
  // every token's place; its total sizes the buffers of the entropy coding
  int nl = 0;
  if ((rc = mth::stream_count(j.sg, j.si, j.d_plan, st, &nl)) != MT_OK) return rc;
  mth::StreamTotals tot = {};
  const int ntiles = j.sg.tcols * j.sg.trows;
  std::vector<mth::StreamTile> tile((size_t)ntiles);
  EventGuard counted, decided;
  for (EventGuard* e : {&counted, &decided})
    if (cudaEventCreateWithFlags(&e->e, cudaEventDisableTiming) != cudaSuccess) return MT_ERR_DEVICE;
  if (cudaMemcpyAsync(&tot, mth::stream_totals(j.sg, j.d_plan), sizeof(tot), cudaMemcpyDeviceToHost, st) !=
          cudaSuccess ||
      cudaEventRecord(counted.e, st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess ||
      cudaStreamWaitEvent(sc, counted.e, 0) != cudaSuccess)
    return MT_ERR_DEVICE;
  cs.d2h(sizeof(tot));
  // the tiles that go through the entropy coding together: all, but for a frame
  // of very many tokens
  mth::StreamGroup grp;
  grp.ntiles = ntiles;
  grp.tokens = tot.tokens;
  if (tot.groups > 1) {
    if (cudaMemcpyAsync(tile.data(), mth::stream_tiles(j.sg, j.d_plan), tile.size() * sizeof(tile[0]),
                        cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return MT_ERR_DEVICE;
    cs.d2h(tile.size() * sizeof(tile[0]));
    grp = mth::stream_group(tile.data(), ntiles, 0);
  }
  void* d_tok = buf.get<void>(i, kTokens, mth::stream_token_bytes(j.sg, tot.tokens), true);
  if (!d_tok) return MT_ERR_DEVICE;
  if ((rc = mth::stream_trace(j.sg, j.si, j.d_plan, d_tok, grp, j.d_cdfs, cfg->updating_cdf != 0, sc, &nl)) != MT_OK)
    return rc;
  // deblocking (uniform 8x8 blocks and transforms) and the CDEF decision
  int32_t ly, luv, sharp;
  mt_loop_filter_levels(j.plan.base_q_idx, sx, sx, &ly, &luv, &sharp);
  const int n4 = (pw / 4) * (ph / 4);
  mt_deblock_frame_params g = {};
  g.w8 = pw;
  g.h8 = ph;
  g.disp_w = (int)width;
  g.disp_h = (int)height;
  g.sub_x = g.sub_y = sx;
  g.bd = 8;
  const size_t dbs = mt_deblock_frame_scratch_bytes(&g);
  uint8_t* d_maps = buf.get<uint8_t>(i, kMaps, (size_t)n4 * 6);
  void* d_db = buf.get<void>(i, kDeblock, dbs);
  if (!d_maps || !d_db) return MT_ERR_DEVICE;
  block_maps_kernel<<<(unsigned)((n4 / 4 + 255) / 256), 256, 0, st>>>(reinterpret_cast<uint32_t*>(d_maps), pw / 4, n4);
  cs.launches(1);
  // the recon planes are kept: the filters write planes of their own
  uint16_t* d_flt = buf.get<uint16_t>(i, kFiltered, (ny + 2 * nc) * 2);
  if (!d_flt) return MT_ERR_DEVICE;
  uint16_t* flt[3] = {d_flt, d_flt + ny, d_flt + ny + nc};
  const uint8_t* m0 = d_maps;
  if ((rc = mt_deblock_frame_device_to(rec[0], rec[1], rec[2], flt[0], flt[1], flt[2], m0, m0 + n4,
                                       m0 + 2 * (size_t)n4, m0 + 3 * (size_t)n4, m0 + 4 * (size_t)n4,
                                       m0 + 5 * (size_t)n4, &g, ly, luv, luv, d_db, st)) != MT_OK)
    return rc;
  cs.launches(mth::deblock_last_launches);
  mt_cdef_params cp = {};
  cp.w8 = pw;
  cp.h8 = ph;
  cp.disp_w = (int)width;
  cp.disp_h = (int)height;
  cp.sub_x = cp.sub_y = sx;
  cp.base_q_idx = j.plan.base_q_idx;
  cp.bd = 8;
  cp.slow = cfg->speed <= MT_SPEED_SLOW;
  uint8_t* d_skip8 = buf.get<uint8_t>(i, kSkip8, (size_t)nb);
  void* d_cs = buf.get<void>(i, kCdef, mt_cdef_scratch_bytes(&cp));
  if (!d_skip8 || !d_cs) return MT_ERR_DEVICE;
  if (cudaMemsetAsync(d_skip8, 0, (size_t)nb, st) != cudaSuccess) return MT_ERR_DEVICE;
  mt_cdef_decision dec = {};
  const int32_t* d_bits = nullptr;
  const uint8_t* d_grid = nullptr;
  if (j.plan.cdef) {
    if ((rc = mth::cdef_frame_enqueue(flt[0], flt[1], flt[2], src[0], src[1], src[2], d_skip8, &cp, d_cs, decided.e,
                                      &d_bits, &d_grid, st)) != MT_OK)
      return rc;
    cs.launches(mth::cdef_last_launches);
    // the coder needs the decision, not the filtered planes
    if (cudaStreamWaitEvent(sc, decided.e, 0) != cudaSuccess) return MT_ERR_DEVICE;
  } else {
    dec.bits = -1;
  }
  if ((rc = mth::stream_ranges(j.sg, j.d_plan, d_tok, grp, d_bits, d_grid, sc, &nl)) != MT_OK) return rc;
  if (j.recon_out) {  // the decoder's output: deblocked and CDEF-filtered
    if (cudaMemcpyAsync(j.recon_out[0], flt[0], ny * 2, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(j.recon_out[1], flt[1], nc * 2, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(j.recon_out[2], flt[2], nc * 2, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return MT_ERR_DEVICE;
    cs.d2h((ny + 2 * nc) * 2);
  }
  size_t ntok = 0;
  std::vector<std::vector<uint8_t>> payloads;  // by group
  std::vector<const uint8_t*> ctiles;
  std::vector<size_t> tile_lens;
  for (;;) {
    mth::StreamTile* const gt = tile.data() + grp.tile0;
    const size_t gt_bytes = (size_t)grp.ntiles * sizeof(tile[0]);
    if (cudaMemcpyAsync(&tot, mth::stream_totals(j.sg, j.d_plan), sizeof(tot), cudaMemcpyDeviceToHost, sc) !=
            cudaSuccess ||
        cudaMemcpyAsync(gt, mth::stream_tiles(j.sg, j.d_plan) + grp.tile0, gt_bytes, cudaMemcpyDeviceToHost, sc) !=
            cudaSuccess ||
        cudaStreamSynchronize(sc) != cudaSuccess)
      return MT_ERR_DEVICE;
    uint32_t longest = 0;
    for (int k = 0; k < grp.ntiles; ++k) {
      longest = std::max(longest, gt[k].nbytes);
      ntok += gt[k].ntok;
    }
    void* d_dig = buf.get<void>(i, kDigits, mth::stream_digit_bytes(tot), true);
    if (!d_dig) return MT_ERR_DEVICE;
    const uint8_t* d_pay = mth::stream_bytes(j.sg, j.d_plan, d_tok, grp, d_dig, tot, longest, sc, &nl);
    payloads.emplace_back(tot.bytes);
    uint8_t* const payload = payloads.back().data();
    if (!d_pay || cudaMemcpyAsync(payload, d_pay, tot.bytes, cudaMemcpyDeviceToHost, sc) != cudaSuccess ||
        cudaStreamSynchronize(sc) != cudaSuccess)
      return MT_ERR_DEVICE;
    for (int k = 0; k < grp.ntiles; ++k) {
      ctiles.push_back(payload + gt[k].byte);
      tile_lens.push_back(gt[k].nbytes);
    }
    cs.d2h(sizeof(tot) + gt_bytes + tot.bytes);
    if (grp.tile0 + grp.ntiles == ntiles) break;
    grp = mth::stream_group(tile.data(), ntiles, grp.tile0 + grp.ntiles);
    if ((rc = mth::stream_trace(j.sg, j.si, j.d_plan, d_tok, grp, j.d_cdfs, cfg->updating_cdf != 0, sc, &nl)) !=
            MT_OK ||
        (rc = mth::stream_ranges(j.sg, j.d_plan, d_tok, grp, d_bits, d_grid, sc, &nl)) != MT_OK)
      return rc;
  }
  cs.launches(nl);
  if (j.plan.cdef) {
    if ((rc = mth::cdef_frame_decision(&cp, d_cs, &dec, nullptr, st)) != MT_OK) return rc;
    size_t cd2h = 0, ch2d = 0;
    mth::cdef_frame_transfer_bytes(&cp, &cd2h, &ch2d);
    cs.d2h(cd2h - (size_t)j.sg.sb_cols * j.sg.sb_rows);
  }
  // headers and container
  mt_sequence_header_params sp = {};
  sp.width = width;
  sp.height = height;
  sp.profile = sub ? 0 : 1;
  sp.bit_depth = 8;
  sp.color_present = cfg->color_present;
  sp.primaries = cfg->primaries;
  sp.transfer = cfg->transfer;
  sp.matrix = cfg->matrix;
  sp.full_range = cfg->full_range;
  sp.chroma_sample_position = cfg->chroma_sample_position;
  sp.ss_x = sp.ss_y = (uint32_t)sx;
  sp.enable_filter_intra = sp.enable_intra_edge_filter = 1;
  mt_frame_header_params fp = {};
  fp.w8 = pw;
  fp.h8 = ph;
  fp.base_q_idx = j.plan.base_q_idx;
  fp.qm_y = j.plan.qm_y;
  fp.qm_u = fp.qm_v = j.plan.qm_u;
  fp.updating_cdf = cfg->updating_cdf;
  fp.lf_y = ly;
  fp.lf_u = fp.lf_v = luv;
  fp.lf_sharpness = sharp;
  fp.cdef_bits = dec.bits;
  fp.cdef_damping = dec.bits >= 0 ? dec.damping : 3;
  for (int e = 0; e < dec.n_strengths && e < 8; ++e)
    for (int q = 0; q < 4; ++q) fp.cdef_strengths[e][q] = dec.strengths[e][q];
  fp.tile_cols_log2 = j.tcl;
  fp.tile_rows_log2 = j.trl;
  uint8_t* obu = nullptr;
  size_t obu_len = 0;
  rc = mt_av1_stream(&sp, &fp, ctiles.data(), tile_lens.data(), ntiles, &obu, &obu_len);
  if (rc != MT_OK) return rc;
  mt_avif_item_params ip = {};
  ip.width = width;
  ip.height = height;
  ip.bit_depth = 8;
  ip.channels = 3;
  ip.seq_profile = (uint8_t)sp.profile;
  ip.seq_level_idx = mt_av1_level_for(width, height);
  ip.chroma_sub_x = ip.chroma_sub_y = sx;
  ip.color_present = cfg->color_present;
  ip.primaries = (uint16_t)cfg->primaries;
  ip.transfer = (uint16_t)cfg->transfer;
  ip.matrix = (uint16_t)cfg->matrix;
  ip.full_range = cfg->full_range;
  ip.icc = cfg->icc;
  ip.icc_len = cfg->icc_len;
  ip.exif = cfg->exif;
  ip.exif_len = cfg->exif_len;
  ip.imir_axis = -1;
  ip.clli_present = cfg->clli_present;
  ip.max_content_light_level = cfg->max_content_light_level;
  ip.max_pic_average_light_level = cfg->max_pic_average_light_level;
  rc = mt_wrap_av1_image(obu, obu_len, &ip, j.out, j.out_len);
  free(obu);
  if (j.stats) j.stats->tokens = (uint32_t)(ntok - 3 * (size_t)j.sg.sb_cols * j.sg.sb_rows);
  cs.mark(3, st);
  cs.finish();
  return rc;
}

// The encode of a batch of images: set-up per image, one launch for all
// their decisions, then each image's finishing work on a host thread of its
// own (the calling thread for one image).  Every image's bytes are those of
// encoding it alone.
void encode_jobs(std::vector<Job>& jobs, int skip = 0) {
  const int n = (int)jobs.size();
  Buffers buf(n);
  for (int i = 0; i < n; ++i) jobs[(size_t)i].rc = job_setup(jobs[(size_t)i], buf, i);
  const int rc = decide_all(jobs, buf, skip);
  for (Job& j : jobs)
    if (j.rc == MT_OK && rc != MT_OK) j.rc = rc;
  if (n == 1) {
    if (jobs[0].rc == MT_OK) jobs[0].rc = job_finish(jobs[0], buf, 0);
    return;
  }
  int dev = 0;  // a new thread starts on device 0; the streams and buffers are the caller's device's
  const bool have_dev = cudaGetDevice(&dev) == cudaSuccess;
  std::vector<std::thread> pool;
  for (int i = 0; i < n; ++i)
    if (jobs[(size_t)i].rc == MT_OK)
      pool.emplace_back([&jobs, &buf, i, dev, have_dev]() {
        jobs[(size_t)i].rc =
            have_dev && cudaSetDevice(dev) == cudaSuccess ? job_finish(jobs[(size_t)i], buf, i) : MT_ERR_DEVICE;
      });
  for (std::thread& t : pool) t.join();
}

int encode_one(const uint8_t* rgb, bool rgb_on_device, const uint8_t* const* yuv, uint32_t width, uint32_t height,
               const mt_encode_config* cfg, uint8_t** out, size_t* out_len, uint16_t* recon_out[3],
               mt_encode_stats* stats, int skip = 0) {
  std::vector<Job> jobs(1);
  Job& j = jobs[0];
  j.rgb = rgb;
  j.rgb_on_device = rgb_on_device;
  j.yuv = yuv;
  j.width = width;
  j.height = height;
  j.cfg = cfg;
  j.out = out;
  j.out_len = out_len;
  j.recon_out = recon_out;
  j.stats = stats;
  encode_jobs(jobs, skip);
  return j.rc;
}

}  // namespace

namespace mth {
// mt_encode_rgb8 of a frame whose first block nobody codes: the waits for its
// records run out, and the call returns MT_ERR_DEVICE.
int encode_without_first_block(const uint8_t* rgb, uint32_t width, uint32_t height, const mt_encode_config* cfg) {
  uint8_t* out = nullptr;
  size_t len = 0;
  const int rc = encode_one(rgb, false, nullptr, width, height, cfg, &out, &len, nullptr, nullptr, 1);
  free(out);
  return rc;
}
}  // namespace mth

extern "C" {

int mt_encode_rgb8_ex(const uint8_t* rgb, uint32_t width, uint32_t height, const mt_encode_config* cfg,
                      uint8_t** out, size_t* out_len, uint16_t* recon_out[3], mt_encode_stats* stats) {
  if (!rgb) return MT_ERR_INVALID_INPUT;
  return encode_one(rgb, false, nullptr, width, height, cfg, out, out_len, recon_out, stats);
}

int mt_encode_rgb8(const uint8_t* rgb, uint32_t width, uint32_t height, const mt_encode_config* cfg, uint8_t** out,
                   size_t* out_len) {
  return mt_encode_rgb8_ex(rgb, width, height, cfg, out, out_len, nullptr, nullptr);
}

int mt_encode_rgb8_device(const uint8_t* d_rgb, uint32_t width, uint32_t height, const mt_encode_config* cfg,
                          uint8_t** out, size_t* out_len, mt_encode_stats* stats) {
  if (!d_rgb) return MT_ERR_INVALID_INPUT;
  return encode_one(d_rgb, true, nullptr, width, height, cfg, out, out_len, nullptr, stats);
}

int mt_encode_rgb8_batch(int32_t n, const uint8_t* const* rgb, const uint32_t* widths, const uint32_t* heights,
                         const mt_encode_config* cfgs, uint8_t** outs, size_t* out_lens, int32_t* rcs,
                         mt_encode_stats* stats) {
  if (n < 1 || n > 64 || !rgb || !widths || !heights || !cfgs || !outs || !out_lens) return MT_ERR_INVALID_INPUT;
  std::vector<Job> jobs((size_t)n);
  for (int i = 0; i < n; ++i) {
    Job& j = jobs[(size_t)i];
    outs[i] = nullptr;
    out_lens[i] = 0;
    j.rgb = rgb[i];
    j.width = widths[i];
    j.height = heights[i];
    j.cfg = &cfgs[i];
    j.out = &outs[i];
    j.out_len = &out_lens[i];
    j.stats = stats ? &stats[i] : nullptr;
    if (!rgb[i]) j.rc = MT_ERR_INVALID_INPUT;
  }
  std::vector<Job> live;  // images with an input: the others keep their code
  std::vector<int> idx;
  for (int i = 0; i < n; ++i)
    if (jobs[(size_t)i].rgb) {
      idx.push_back(i);
      live.push_back(std::move(jobs[(size_t)i]));
    }
  encode_jobs(live);
  int first = MT_OK;
  for (size_t k = 0; k < live.size(); ++k) jobs[(size_t)idx[k]].rc = live[k].rc;
  for (int i = 0; i < n; ++i) {
    if (rcs) rcs[i] = jobs[(size_t)i].rc;
    if (first == MT_OK && jobs[(size_t)i].rc != MT_OK) first = jobs[(size_t)i].rc;
  }
  return first;
}

void mt_encode_release_buffers(void) {
  int cur = 0;
  cudaGetDevice(&cur);
  for (int d = 0; d < 16; ++d) {
    Arena& ar = g_arenas[d];
    std::lock_guard<std::mutex> lock(ar.mu);
    if (ar.sets.empty()) continue;
    cudaSetDevice(d);
    for (BufSet& b : ar.sets) {
      for (void*& q : b.p) {
        cudaFree(q);
        q = nullptr;
      }
      for (cudaStream_t s : b.st)
        if (s) cudaStreamDestroy(s);
    }
    ar.sets.clear();
  }
  cudaSetDevice(cur);
}

int mt_encode_yuv8(const uint8_t* y, const uint8_t* u, const uint8_t* v, uint32_t width, uint32_t height,
                   const mt_encode_config* cfg, uint8_t** out, size_t* out_len, uint16_t* recon_out[3]) {
  const uint8_t* planes[3] = {y, u, v};
  if (!y || !u || !v) return MT_ERR_INVALID_INPUT;
  return encode_one(nullptr, false, planes, width, height, cfg, out, out_len, recon_out, nullptr);
}

}  // extern "C"
