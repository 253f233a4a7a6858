// dQ kernel: the query-stationary half of the backward pass.
//
// A work item is one 128-row query tile of one head; the CTA walks the key tiles the item's rows can
// see, over every KV span of the call (sink | halo | local), so that dQ is accumulated on chip and
// written exactly once -- no atomics, no fp32 accumulator in global memory:
//
//   S  = Q K^T          A = Q  (smem, K-major)   B = K (smem, K-major)     two TMEM buffers
//   dP = dO V^T         A = dO (smem, K-major)   B = V (smem, K-major)
//   P  = exp2(S * scale_log2 - lse2[row]),  dS = P * (dP - delta[row])      (16 compute warps)
//   dQ += dS K          A = dS (TMEM, written over S)   B = K (smem, MN-major)
//
// P is recomputed from the final log-sum-exp, so the result is exact for any set of spans
// (the property the reference's per-hop backward relies on, ring_swa/ops/attn.py:63-126).
//
// The kernel is persistent: one CTA per SM keeps taking items from a counter in global memory and
// every pipeline (K/V rings, S buffers, barrier phases) keeps running across item boundaries, so
// the fill and drain of one item (first loads, last dQ product, dQ write-out) overlap the next
// item's loads and products instead of leaving the SM idle.  Roles:
//   warp 0      key-tile list of each item (two-slot ring) and TMA producer (Q, dO once per item;
//               K ring of 3, V ring of 2)
//   warps 1-3   issue the S, dP and dQ products, one warp each (all 32 lanes run the loop and one
//               elected lane issues: a converged warp is scheduled better than a lone lane when the
//               compute warps next to it are in an FMA-heavy phase)
//   warps 4-19  compute, four warps per TMEM lane quadrant, 32 key columns each
// Three warps issue MMAs because the issue path, not the tensor pipe, is what one thread saturates
// first: with S and dQ on one thread, that thread was the longest chain of a key tile.  TMEM: [0,128) S_0/dS_0, [128,256) S_1/dS_1, [256,384) dP, [384,512) dQ.
#include "rswa_common.cuh"
#include "rswa_tiles.cuh"
#include "tc05.cuh"

namespace rswa {
using namespace tc05;

RSWA_TRACE_DECL(dq)
#ifndef RSWA_TRACE_G0
#define RSWA_TRACE_G0 200
#endif
#define DQ_TRC(cond, g, s) RSWA_TRC(dq, (cond) && (g) >= RSWA_TRACE_G0 && (g) < RSWA_TRACE_G0 + 32, ((g) - RSWA_TRACE_G0) * 32 + (s))

namespace {

constexpr int kDqThreads = 640;
constexpr int kDqTmemCols = 512;
constexpr int kDqKStages = 3;
constexpr int kDqSmemTiles = 7 * kTileBytes;  // Q, dO, K x 3, V x 2
constexpr int kDqCompute = 512;
// The MMA-issuing threads poll their barriers without back-off: they sit on the critical path of
// every key tile, and a sleeping poll was measured slower.
constexpr int kMmaPollNs = 0;
constexpr int kCmpPollNs = 0;
#ifndef RSWA_DQ_POLY
#define RSWA_DQ_POLY 1
#endif
constexpr bool kDqPoly = RSWA_DQ_POLY != 0;  // a quarter of the exponentials on the FMA pipe
constexpr int kDqGeomUsers = 4 + kDqCompute / 32;  // producer, three MMA issuers, one lane per compute warp

struct DqCtl {
  uint64_t q_full, do_full, q_free, do_free;
  uint64_t k_full[kDqKStages], v_full[2], k_free[kDqKStages], v_free[2];
  uint64_t s_ready[2], s_free[2], dp_ready, dp_loaded, ds_ready, done, dq_drained;
  uint64_t geom_full[2], geom_free[2];
  uint32_t tmem_base;
  int err;
  int item[2];  // work item of each geometry slot, -1: no more work
  QBlockGeom geom[2];
};

constexpr int kDqSmemBytes = kDqSmemTiles + 1024;
static_assert(sizeof(DqCtl) <= 1024, "control block too large");
static_assert(kDqSmemBytes <= 232448, "shared memory budget");

struct DqItem {
  int qt, h, b, hk, row0;
};
__device__ __forceinline__ DqItem dq_item(const BwdKernelParams& p, int n_q_tiles, int it) {
  DqItem d;  // query tile fastest, then head, then batch row
  d.qt = it % n_q_tiles;
  it /= n_q_tiles;
  d.h = it % p.hq;
  d.b = it / p.hq;
  d.hk = d.h / (p.hq / p.hkv);
  d.row0 = d.qt * kTile;
  return d;
}

// kPlain: one KV span, no packed sequences, no sink tokens (the plain sliding window of one GPU).  The
// SM's instruction cache holds 32 KB and this kernel's five roles together execute more than that per
// work item, so what such a call cannot need is compiled out of its variant.
// kD: width of a head, 128 or 64.
template <int kD, bool kBf16, bool kPlain>
__global__ void __launch_bounds__(kDqThreads, 1)
rswa_dq_kernel(const __grid_constant__ BwdKernelParams p, int n_q_tiles, int n_items) {
  constexpr uint32_t kLoadBytes = kD / 64 * kBoxBytes;  // what a tile holds (its slots in shared memory are kTileBytes apart)
  const int* const cu_seq = kPlain ? nullptr : p.cu;
  const int n_seqs = kPlain ? 0 : p.n_seqs;
  const int n_spans = kPlain ? 1 : p.n_spans;
  const int n_sink = kPlain ? 0 : p.n_sink;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sDO = smem + kTileBytes;
  uint8_t* sK = smem + 2 * kTileBytes;  // three stages
  uint8_t* sV = smem + 5 * kTileBytes;  // two stages
  DqCtl* ctl = reinterpret_cast<DqCtl*>(smem + kDqSmemTiles);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&ctl->q_full, 1);
    mbar_init(&ctl->do_full, 1);
    mbar_init(&ctl->q_free, 1);
    mbar_init(&ctl->do_free, 1);
    for (int i = 0; i < kDqKStages; ++i) {
      mbar_init(&ctl->k_full[i], 1);
      mbar_init(&ctl->k_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl->v_full[i], 1);
      mbar_init(&ctl->v_free[i], 1);
      mbar_init(&ctl->s_ready[i], 1);
      mbar_init(&ctl->s_free[i], 1);
      mbar_init(&ctl->geom_full[i], 1);
      mbar_init(&ctl->geom_free[i], kDqGeomUsers);
    }
    mbar_init(&ctl->dp_ready, 1);
    mbar_init(&ctl->dp_loaded, kDqCompute / 32);  // one arrival per compute warp
    mbar_init(&ctl->ds_ready, kDqCompute / 32);  // one arrival per compute warp
    mbar_init(&ctl->done, 1);
    mbar_init(&ctl->dq_drained, kDqCompute / 32);  // one arrival per compute warp
    mbar_fence_init();
    // No griddep_wait() here: when this kernel starts early, the kernel it overlaps is the dK/dV kernel of the same
    // call, which it needs nothing from.  What the delta kernel and everything before the call wrote comes through the
    // gate: acquired here, by the other threads through the barrier below.  The wait is at the end instead.
    const bool open = p.gate == nullptr || gate_wait(p.gate);
    ctl->err = (smem_u32(smem) & 1023u) ? 199 : !open ? kErrWaitProducer : status_code(p.status, p.mirror);
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, kDqTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const uint32_t tmem = ctl->tmem_base;
  const uint32_t tDP = tmem + 256, tDQ = tmem + 384;
  volatile int* err = &ctl->err;
  // Items are handed out through a counter in global memory rather than by a fixed stride: a CTA
  // whose SM is busy with another kernel (a collective of the ring, say) starts late and simply takes
  // fewer items, instead of leaving its whole share for the end.
  const int n_work = (ctl->err != 0) ? 0 : n_items;

  if (warp < 4) {
    setmaxnreg_dec<56>();
    if (warp == 0 && lane == 0) {
      // ------------------------------------------------------------------ key-tile lists + TMA producer
      // One loop turn per key tile and ONE copy of each load's code (this thread runs through its code
      // at the pace of instruction fetch, and the kernel has to fit the instruction cache).
      if (p.gate != nullptr) fence_proxy_async_global();  // what came through the gate is read by TMA here
      int n = -1, kc = 0, ic = 0;  // item of this CTA, K/V tiles loaded so far, items with work so far
      int j = 0, n_tiles = 0, slot = 0;
      DqItem w = {};
      QBlockGeom* geom = nullptr;
      TileCursor c = {};
      for (;;) {
        if (j >= n_tiles) {  // next item
          if (n >= 0) mbar_arrive(&ctl->geom_free[slot]);  // this role is done with the list of the item before
          ++n;
          slot = n & 1;
          // The list of item n goes into slot n & 1 once every role is done with item n - 2.  This
          // thread has spare time exactly here: its last loads of the previous item are issued and
          // the ring stages for this one are still in use.
          if (n >= 2 && !mbar_wait<200>(&ctl->geom_free[slot], ((n >> 1) - 1) & 1, err, kErrWaitProducer)) break;
          const int it = n_work > 0 ? atomicAdd(p.dq_counter, 1) : n_work;
          j = 0;
          n_tiles = 0;
          if (it >= n_work) {  // tell every role that the work has run out
            ctl->item[slot] = -1;
            mbar_arrive(&ctl->geom_full[slot]);
            break;
          }
          ctl->item[slot] = it;
          geom = &ctl->geom[slot];
          w = dq_item(p, n_q_tiles, it);
          // a block of one query tile: the second tile of the geometry stays empty
          qblock_geometry<kTile>(geom, cu_seq, n_seqs, n_spans, p.span_pos, p.span_len, p.q_pos_start, p.q_len,
                                 p.window, n_sink, w.qt, w.qt + 1);
          mbar_arrive(&ctl->geom_full[slot]);
          n_tiles = geom->n_tiles;
          if (n_tiles == 0) continue;
          cursor_begin<kTile>(geom, p.span_pos, p.span_len, c);
          // Q may be replaced once the last S product of the previous item has read it
          if (ic > 0 && !mbar_wait<200>(&ctl->q_free, (ic - 1) & 1, err, kErrWaitProducer)) break;
          mbar_expect_tx(&ctl->q_full, kLoadBytes);
          tma_load_4d(sQ, &p.q_map, &ctl->q_full, 0, w.h, w.row0, w.b);
          if (kD > 64) tma_load_4d(sQ + kBoxBytes, &p.q_map, &ctl->q_full, 64, w.h, w.row0, w.b);
        }
        const int sk = kc % kDqKStages, sv = kc & 1;
        if (kc >= kDqKStages && !mbar_wait<200>(&ctl->k_free[sk], ((kc / kDqKStages) - 1) & 1, err, kErrWaitProducer)) break;
        mbar_expect_tx(&ctl->k_full[sk], kLoadBytes);
        tma_load_4d(sK + sk * kTileBytes, &p.k_map[c.span], &ctl->k_full[sk], 0, w.hk, c.tok, w.b);
        if (kD > 64) tma_load_4d(sK + sk * kTileBytes + kBoxBytes, &p.k_map[c.span], &ctl->k_full[sk], 64, w.hk, c.tok, w.b);
        if (j == 0) {
          // dO likewise, after the last dP product of the previous item
          if (ic > 0 && !mbar_wait<200>(&ctl->do_free, (ic - 1) & 1, err, kErrWaitProducer)) break;
          ++ic;
          mbar_expect_tx(&ctl->do_full, kLoadBytes);
          tma_load_4d(sDO, &p.do_map, &ctl->do_full, 0, w.h, w.row0, w.b);
          if (kD > 64) tma_load_4d(sDO + kBoxBytes, &p.do_map, &ctl->do_full, 64, w.h, w.row0, w.b);
        }
        if (kc >= 2 && !mbar_wait<200>(&ctl->v_free[sv], ((kc >> 1) - 1) & 1, err, kErrWaitProducer)) break;
        mbar_expect_tx(&ctl->v_full[sv], kLoadBytes);
        tma_load_4d(sV + sv * kTileBytes, &p.v_map[c.span], &ctl->v_full[sv], 0, w.hk, c.tok, w.b);
        if (kD > 64) tma_load_4d(sV + sv * kTileBytes + kBoxBytes, &p.v_map[c.span], &ctl->v_full[sv], 64, w.hk, c.tok, w.b);
        ++j;
        ++kc;
        cursor_next<kTile>(geom, p.span_pos, p.span_len, c, j < n_tiles);
      }
    } else if (warp == 1 && elect_one()) {
      // ------------------------------------------------------------------ MMA issuer 1: S = Q K^T
      constexpr uint32_t id_kk = idesc_f16(128, 128, kBf16 ? 1 : 0, 0, 0);
      constexpr uint32_t kTile16 = kTileBytes >> 4;
      const uint64_t dQd = smem_desc_sw128(smem_u32(sQ), 16, 1024);
      const uint64_t dKk = smem_desc_sw128(smem_u32(sK), 16, 1024);  // K as K-major B operand
      uint64_t dqa[kD / 16];  // the A operands never change: Q has one buffer
#pragma unroll
      for (int k = 0; k < kD / 16; ++k) dqa[k] = dQd + ((((k >> 2) * kBoxBytes + (k & 3) * 32)) >> 4);
      bool ok = true;
      int n = 0, kc = 0, ic = 0;  // kc: key tiles of earlier items = running index of this item's tile 0
      for (;; ++n) {
        const int slot = n & 1;
        ok = mbar_wait<kMmaPollNs>(&ctl->geom_full[slot], (n >> 1) & 1, err, kErrWaitMma);
        if (!ok || ctl->item[slot] < 0) break;
        const int n_tiles = ctl->geom[slot].n_tiles;
        if (n_tiles > 0) {
          ok = mbar_wait<kMmaPollNs>(&ctl->q_full, ic & 1, err, kErrWaitMma);
          for (int j = 0; j < n_tiles && ok; ++j) {
            const int g = kc + j;
            const int sk = g % kDqKStages;
            // every operand of the instructions is in a register BEFORE the waits: what this
            // thread executes between the last barrier and the last instruction is on the chain that
            // bounds the kernel, and it gets an instruction through only every few cycles
            uint64_t db[kD / 16];
            const uint32_t td = tmem + 128 * (g & 1);
#pragma unroll
            for (int k = 0; k < kD / 16; ++k) {
              db[k] = dKk + sk * kTile16 + ((((k >> 2) * kBoxBytes + (k & 3) * 32)) >> 4);
              asm volatile("" : "+l"(db[k]));
            }
            ok = mbar_wait<kMmaPollNs>(&ctl->k_full[sk], (g / kDqKStages) & 1, err, kErrWaitMma);
            // S buffer g & 1 last held dS of tile g - 2: the dQ product that reads it must be complete
            if (ok && g >= 2) ok = mbar_wait<kMmaPollNs>(&ctl->s_free[g & 1], ((g >> 1) - 1) & 1, err, kErrWaitMma);
            if (!ok) break;
            DQ_TRC(true, g, 0);
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < kD / 16; ++k) mma_ss(td, dqa[k], db[k], id_kk, k > 0 ? 1u : 0u);
            DQ_TRC(true, g, 1);
            mma_commit(&ctl->s_ready[g & 1]);
            if (j + 1 == n_tiles) mma_commit(&ctl->q_free);  // that was the item's last read of Q
          }
          kc += n_tiles;
          ++ic;
        }
        if (ok) mbar_arrive(&ctl->geom_free[slot]);
      }
    } else if (warp == 3 && elect_one()) {
      // ------------------------------------------------------------------ MMA issuer 3: dQ += dS K
      constexpr uint32_t id_tn = idesc_f16(128, kD, kBf16 ? 1 : 0, 0, 1);
      constexpr uint32_t kTile16 = kTileBytes >> 4;
      const uint64_t dKm = smem_desc_sw128(smem_u32(sK), kBoxBytes, 1024);  // K as MN-major B operand
      bool ok = true;
      int n = 0, kc = 0, ic = 0;
      for (;; ++n) {
        const int slot = n & 1;
        ok = mbar_wait<kMmaPollNs>(&ctl->geom_full[slot], (n >> 1) & 1, err, kErrWaitMma);
        if (!ok || ctl->item[slot] < 0) break;
        const int n_tiles = ctl->geom[slot].n_tiles;
        if (n_tiles > 0) {
          for (int j = 0; j < n_tiles && ok; ++j) {
            const int g = kc + j;
            // (operands in registers before the waits, as for S)
            uint64_t db[8];
            uint32_t ta[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              db[k] = dKm + (g % kDqKStages) * kTile16 + k * 128;
              ta[k] = tmem + 128 * (g & 1) + (k >> 1) * 32 + (k & 1) * 8;
              asm volatile("" : "+l"(db[k]), "+r"(ta[k]));
            }
            const uint32_t acc0 = j > 0 ? 1u : 0u;
            ok = mbar_wait<kMmaPollNs>(&ctl->ds_ready, g & 1, err, kErrWaitMma);
            // the first product of an item overwrites dQ: the previous item's must have been read out
            if (ok && j == 0 && ic > 0) ok = mbar_wait<kMmaPollNs>(&ctl->dq_drained, (ic - 1) & 1, err, kErrWaitMma);
            if (!ok) break;
            DQ_TRC(true, g, 2);
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < 8; ++k) mma_ts(tDQ, ta[k], db[k], id_tn, k > 0 ? 1u : acc0);
            DQ_TRC(true, g, 3);
            mma_commit(&ctl->k_free[g % kDqKStages]);
            mma_commit(&ctl->s_free[g & 1]);
          }
          if (ok) mma_commit(&ctl->done);
          kc += n_tiles;
          ++ic;
        }
        if (ok) mbar_arrive(&ctl->geom_free[slot]);
      }
    } else if (warp == 2 && elect_one()) {
      // ------------------------------------------------------------------ MMA issuer 2: dP
      constexpr uint32_t id_kk = idesc_f16(128, 128, kBf16 ? 1 : 0, 0, 0);
      constexpr uint32_t kTile16 = kTileBytes >> 4;
      const uint64_t dDO = smem_desc_sw128(smem_u32(sDO), 16, 1024);
      const uint64_t dVk = smem_desc_sw128(smem_u32(sV), 16, 1024);
      bool ok = true;
      int n = 0, kc = 0, ic = 0;
      for (;; ++n) {
        const int slot = n & 1;
        ok = mbar_wait<kMmaPollNs>(&ctl->geom_full[slot], (n >> 1) & 1, err, kErrWaitMma);
        if (!ok || ctl->item[slot] < 0) break;
        const int n_tiles = ctl->geom[slot].n_tiles;
        if (n_tiles > 0) {
          ok = mbar_wait<kMmaPollNs>(&ctl->do_full, ic & 1, err, kErrWaitMma);
          for (int j = 0; j < n_tiles && ok; ++j) {
            const int g = kc + j;
            const int sv = g & 1;
            ok = mbar_wait<kMmaPollNs>(&ctl->v_full[sv], (g >> 1) & 1, err, kErrWaitMma);
            // the compute warps must have read dP of the previous tile out of TMEM
            if (ok && g > 0) ok = mbar_wait<kMmaPollNs>(&ctl->dp_loaded, (g - 1) & 1, err, kErrWaitMma);
            if (!ok) break;
            DQ_TRC(true, g, 4);
            tc_fence_after();
            const uint64_t dVs = dVk + sv * kTile16;
#pragma unroll
            for (int k = 0; k < kD / 16; ++k) {
              const uint32_t off = ((k >> 2) * kBoxBytes + (k & 3) * 32) >> 4;
              mma_ss(tDP, dDO + off, dVs + off, id_kk, k > 0 ? 1u : 0u);
            }
            mma_commit(&ctl->dp_ready);
            DQ_TRC(true, g, 5);
            mma_commit(&ctl->v_free[sv]);
          }
          if (ok) mma_commit(&ctl->do_free);
          kc += n_tiles;
          ++ic;
        }
        if (ok) mbar_arrive(&ctl->geom_free[slot]);
      }
    }
  } else {
    // -------------------------------------------------------------------- compute warps
    // Four warps per TMEM lane quadrant, each owning 32 of the tile's 128 key columns.
    setmaxnreg_inc<104>();  // 128 x 56 + 512 x 104 <= 640 x 96 (the launch allocation)
    const int quad = warp & 3;
    const int part = (warp - 4) >> 2;       // which 32 key columns of the tile this warp handles
    const int row = quad * 32 + lane;       // query row inside the tile
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const float sl2 = p.scale_log2;
    const float mul = p.scale;
    bool ok = true;
    int n = 0, kc = 0, ic = 0;
    // row statistics of the item after this one, fetched while this one's last products still run
    float lse2_nx = 0.f, delta_nx = 0.f;
    auto row_stats = [&](int it_, float& l2, float& dl) {
      const DqItem w_ = dq_item(p, n_q_tiles, it_);
      const long long roff = w_.b * p.d_sb + w_.h * p.d_sh + w_.row0 + row;  // rows are padded to whole tiles
      l2 = p.lse2[roff];  // (negated) -inf past q_len: P vanishes
      dl = p.delta[roff];
    };
    // An item's dQ is read out of tensor memory and stored only after the first exponentials of the
    // NEXT item: its last product is still running when its last dS has been handed over, and waiting
    // for it right there left every compute warp idle.
    uint16_t* pend_row = nullptr;  // where this thread's kD / 4 values of the pending item go (null: row does not exist)
    bool pend = false;
    int pend_ic = 0;
    auto drain = [&]() -> bool {
      bool k = mbar_wait<kCmpPollNs>(&ctl->done, pend_ic & 1, err, kErrWaitEpilogue);
      k = __all_sync(0xffffffffu, k);
      if (!k) return false;
      tc_fence_after();
      uint32_t r[kD / 4];
      if constexpr (kD == 128) tmem_ld32(tDQ + lane_off + part * 32, r);
      else tmem_ld16(tDQ + lane_off + part * 16, r);
      tmem_ld_wait();
      // the accumulator is released as soon as it is in registers
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->dq_drained);
      if (pend_row != nullptr) {
        // (32-byte stores: whole sectors, half as many requests as 16-byte ones)
#pragma unroll
        for (int v = 0; v < kD / 64; ++v) {
          uint32_t o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            o[i] = pack2<kBf16>(__uint_as_float(r[v * 16 + 2 * i]) * mul, __uint_as_float(r[v * 16 + 2 * i + 1]) * mul);
          st_global_v8(pend_row + v * 16, o);
        }
      }
      pend = false;
      return true;
    };
    for (;; ++n) {
      const int slot = n & 1;
      ok = mbar_wait<kCmpPollNs>(&ctl->geom_full[slot], (n >> 1) & 1, err, kErrWaitSoftmax);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const int it = ctl->item[slot];
      if (it < 0) break;
      const DqItem w = dq_item(p, n_q_tiles, it);
      if (n == 0) row_stats(it, lse2_nx, delta_nx);
      const float lse2_r = lse2_nx, delta_r = delta_nx;
      const QBlockGeom* geom = &ctl->geom[slot];
      const int n_tiles = geom->n_tiles;
      const bool valid = row < geom->n_valid[0];
      const int pos = geom->p0[0] + row;
      int s_p = 0, e_p = 0;
      if (valid) seq_of(cu_seq, n_seqs, pos, s_p, e_p);
      const int hi = valid ? pos : -1;
      const int lo = valid ? max(s_p, pos - p.window) : 0x7fffffff;
      const int sink_end = valid ? s_p + n_sink : -0x7fffffff;
      TileCursor cur;
      cursor_begin<kTile>(geom, p.span_pos, p.span_len, cur);
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int g = kc + j;
        const int kt0 = cur.kt0 + part * 32;
        const int span_end = cur.kt_last + 1;
        const uint32_t tSj = tmem + 128 * (g & 1) + lane_off;
        ok = mbar_wait<kCmpPollNs>(&ctl->s_ready[g & 1], (g >> 1) & 1, err, kErrWaitSoftmax);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        DQ_TRC(warp == 4 && lane == 0, g, 8);
        DQ_TRC(warp == 17 && lane == 0, g, 12);
        tc_fence_after();
        float pr[32];
        {
          uint32_t s0[32];
          tmem_ld32(tSj + part * 32, s0);
          tmem_ld_wait();
          // one pair in four goes through the FMA pipe instead of the special-function unit
          // (two values per instruction wherever the pipe has a packed form: the compute warps are bound
          // by their instruction count, 16 warps on four schedulers)
          const float2 sl2v = make_float2(sl2, sl2), nlv = make_float2(lse2_r, lse2_r);  // (the rows arrive negated, see the delta kernel)
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 x = __ffma2_rn(make_float2(__uint_as_float(s0[i]), __uint_as_float(s0[i + 1])), sl2v, nlv);
            if (kDqPoly && ((i >> 1) & 3) == 3) {
              const float2 e = ex2_poly2(x);
              pr[i] = e.x, pr[i + 1] = e.y;
            } else {
              pr[i] = ex2f(x.x), pr[i + 1] = ex2f(x.y);
            }
          }
        }
        const bool my_mask = !(kt0 >= lo && kt0 + 31 <= hi && kt0 + 31 < span_end);
        if (__any_sync(0xffffffffu, my_mask)) {
          // this row sees the positions [lo, top] (its window) and [s_p, s_p + sn) (sink tokens below it)
          const int top = min(hi, span_end - 1);
          const uint32_t wn = static_cast<uint32_t>(max(top - lo + 1, 0));
          const uint32_t sn = kPlain ? 0u : static_cast<uint32_t>(max(min(sink_end, top + 1) - s_p, 0));
          const int c0 = kt0 - lo, c1 = kt0 - s_p;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const bool vis = static_cast<uint32_t>(c0 + i) < wn || (!kPlain && static_cast<uint32_t>(c1 + i) < sn);
            pr[i] = vis ? pr[i] : 0.f;
          }
        }
        DQ_TRC(warp == 4 && lane == 0, g, 9);
        DQ_TRC(warp == 17 && lane == 0, g, 13);
        if (j == 0 && pend) {
          ok = drain();
          if (!ok) break;
        }
        ok = mbar_wait<kCmpPollNs>(&ctl->dp_ready, g & 1, err, kErrWaitSoftmax);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        DQ_TRC(warp == 4 && lane == 0, g, 10);
        DQ_TRC(warp == 17 && lane == 0, g, 14);
        tc_fence_after();
        uint32_t dpk[16];
        {
          uint32_t d0[32];
          tmem_ld32(tDP + lane_off + part * 32, d0);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->dp_loaded);  // dP of the next tile may overwrite these columns now
          const float2 ndv = make_float2(delta_r, delta_r);
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 ds = __fmul2_rn(make_float2(pr[i], pr[i + 1]),
                                         __fadd2_rn(make_float2(__uint_as_float(d0[i]), __uint_as_float(d0[i + 1])), ndv));
            dpk[i >> 1] = pack2<kBf16>(ds.x, ds.y);
          }
        }
        // dS (16-bit) goes over the first half of the very S columns this warp has read, so no
        // other warp has to be waited for: keys [32 part, +32) sit in columns [32 part, +16)
        tmem_st16(tSj + part * 32, dpk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->ds_ready);
        DQ_TRC(warp == 4 && lane == 0, g, 11);
        DQ_TRC(warp == 17 && lane == 0, g, 15);
        cursor_next<kTile>(geom, p.span_pos, p.span_len, cur, j + 1 < n_tiles);
      }
      if (!ok) break;

      {
        // the next item's list is ready long before this point (the producer runs an item ahead): its
        // rows' lse and delta are on their way while the epilogue below runs
        const int slot_nx = (n + 1) & 1;
        ok = mbar_wait<kCmpPollNs>(&ctl->geom_full[slot_nx], ((n + 1) >> 1) & 1, err, kErrWaitSoftmax);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const int it_nx = ctl->item[slot_nx];
        if (it_nx >= 0) row_stats(it_nx, lse2_nx, delta_nx);
      }
      uint16_t* drow = reinterpret_cast<uint16_t*>(p.dq) + w.b * p.dq_sb +
                       static_cast<long long>(w.row0 + row) * p.dq_st + w.h * p.dq_sh + part * (kD / 4);
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->geom_free[slot]);  // (the list is not needed any more)
      if (n_tiles > 0) {
        // the item's dQ * softmax_scale -> dq: later (see above)
        pend = true;
        pend_ic = ic;
        pend_row = valid ? drow : nullptr;
        kc += n_tiles;
        ++ic;
      } else if (valid) {
        // no key of the given spans is visible to this query tile
        uint4* dst = reinterpret_cast<uint4*>(drow);
#pragma unroll
        for (int v = 0; v < kD / 32; ++v) dst[v] = make_uint4(0, 0, 0, 0);
      }
    }
    if (ok && pend) ok = drain();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kDqTmemCols);
  }
  // (this kernel must not be finished before the dK/dV kernel is: what follows on the stream waits for this one)
  griddep_wait();
  if (threadIdx.x == 0 && ctl->err != 0) raise_status(p.status, p.mirror, ctl->err);
}

}  // namespace

int launch_dq(const BwdKernelParams& kp, int dtype, bool early, cudaStream_t stream) {
  const int n_q_tiles = (kp.q_len + kTile - 1) / kTile;
  const long long n_items = static_cast<long long>(n_q_tiles) * kp.hq * kp.batch;
  if (n_items <= 0) return RSWA_OK;
  if (n_items > 0x7fffffffLL) {
    set_error("rswa_bwd: too many query tiles (%lld)", n_items);
    return RSWA_E_ARG;
  }
  const bool plain = kp.n_spans == 1 && kp.cu == nullptr && kp.n_sink == 0;
  const int variant = (dtype == RSWA_DTYPE_BF16 ? 1 : 0) + (plain ? 2 : 0) + (kp.head_dim == kNarrowHeadDim ? 4 : 0);
  using Kern = void (*)(const BwdKernelParams, int, int);
  static const Kern kerns[8] = {rswa_dq_kernel<128, false, false>, rswa_dq_kernel<128, true, false>,
                                rswa_dq_kernel<128, false, true>,  rswa_dq_kernel<128, true, true>,
                                rswa_dq_kernel<64, false, false>,  rswa_dq_kernel<64, true, false>,
                                rswa_dq_kernel<64, false, true>,   rswa_dq_kernel<64, true, true>};
  const Kern kern = kerns[variant];
  // (the attribute is a property of the function on a device: set once per kernel variant and device)
  static bool attr_set[8][64] = {{false}};
  int dev_id = 0;
  cudaError_t e = cudaGetDevice(&dev_id);
  if (e == cudaSuccess && (dev_id < 0 || dev_id >= 64 || !attr_set[variant][dev_id])) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kDqSmemBytes);
    if (e == cudaSuccess && dev_id >= 0 && dev_id < 64) attr_set[variant][dev_id] = true;
  }
  if (e != cudaSuccess) {
    set_error("rswa_bwd(dq): cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return RSWA_E_CUDA;
  }
  // one CTA per SM (shared memory and TMEM allow no more), each striding over the items
  const long long n_cta = n_items < sm_count() ? n_items : sm_count();
  e = launch_kernel(kern, dim3(static_cast<unsigned>(n_cta)), kDqThreads, kDqSmemBytes, stream, early, kp, n_q_tiles, static_cast<int>(n_items));
  count_launches(1);
  if (e != cudaSuccess) {
    set_error("rswa_bwd(dq): launch: %s", cudaGetErrorString(e));
    return RSWA_E_CUDA;
  }
  return RSWA_OK;
}

}  // namespace rswa
