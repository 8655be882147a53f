// Per-root Bron-Kerbosch search with Tomita pivoting, one warp per root.
//
// Replaces the block-per-root kernels mce_kernel_l1_ip_{nowl,wl}
// (mce/mce_kernel_nowl.cuh:9-109, mce/mce_kernel_wl.cuh:9-154) and the
// helpers they call in mce/mce_utils.cuh.  The search rules are the
// reference's (cited inline); the execution model is not:
//  - a warp, not a 128/256-thread block, owns a root, so a tree step costs
//    a few warp instructions instead of several __syncthreads;
//  - the induced subgraph of the root's later neighbours lives in registers
//    (lane i holds adjacency row i, and row i+32 for the 64-bit engine) or,
//    for wide roots, in a per-warp slab, instead of per-block global arrays;
//  - the pivot is the candidate u maximising popc(P & N(u)), found with one
//    __reduce_max_sync over (score, -index) keys: every lane scores its own
//    row(s) in parallel;
//  - the DFS stack is an explicit array of (P, X, branch set, chosen set)
//    frames in shared memory (register engine) or the slab (wide engine);
//  - earlier neighbours of the root (the reference's Xx list, tested with a
//    binary search per tree node, mce/mce_utils.cuh:265-292) are encoded once
//    per root as bitmaps over the root's later neighbours, duplicates
//    dropped; a leaf is maximal only if none of them contains the clique;
//  - load balance: a warp about to descend into a child with many candidates
//    hands the child to the device task queue instead while other warps are
//    idle (queue.cuh), the counterpart of the reference's worker list.
// Tie-breaking: the pivot with the lowest index among the best scores, so
// per-root tree sizes are deterministic and independent of who walks them.
#include <climits>
#include <cstddef>
#include <cstring>

#include "common.cuh"
#include "engine.cuh"
#include "kernels.h"
#include "queue.cuh"

namespace mce {

__global__ void queue_init_kernel(QueueView q) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < q.cap; i += gridDim.x * blockDim.x)
    q.seq[i] = i;
}

namespace {

// Blocks per SM: the 32-bit engine runs 6 (48 warps: more warps hide the
// encode's memory latency better than the registers they give up), the
// 64-bit engine 4.
// EV (opts.warp_log): 0 none, 1 per-warp load and donations, 2 plus the
// per-phase cycle breakdown.
// OPS (opts.count_ops): the variant that sums the algorithmic word
// operations of every walk (reg_tree / mem_tree), run outside timed calls.
// SPLIT: the variant for several warps per root (opts.warps_per_root > 1);
// the others keep no state for it.  STAGE (opts.stage_lists): the encode's
// lists are staged in shared memory by 1-D bulk copies (flat_walk_staged).
// L2 (-p l2): the edge-rooted variant.
template <typename Word, int NR, int EV = 0, bool LIST = false, bool XP = false, bool OPS = false,
          bool SPLIT = false, bool STAGE = false, bool L2 = false>
__global__ void __launch_bounds__(REG_BLOCK, (NR == 1 && sizeof(Word) == 4) ? 6 : (NR == 2 ? 4 : 1))
    bk_reg_kernel(BKArgs a, int cls) {
  __shared__ RegSmem<Word, NR> sm_all[REG_BLOCK / 32];
  RegSmem<Word, NR> &sm = sm_all[threadIdx.x >> 5];
  const int lane = (int)lane_id();
  if constexpr (STAGE) stage_init();
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const RegSlab<Word> sl = reg_slab<Word>(a, gw);
  const uint32_t beg = a.shape->cls_off[cls], end = a.shape->cls_off[cls + 1];
  const bool share = a.q.hdr != nullptr;
  u64 h0 = 0, h1 = 0, nodes = 0, ops = 0;
  RegRoot<Word> rt;
  Bd bdv, *bd = &bdv;
  if constexpr (EV == 2) bdv.start();
  if (share && lane == 0) atomicAdd(&a.q.hdr->work, 1u);
  // units of work: (root, part) pairs, the parts of a root fetched one
  // after the other so that different warps take them
  const uint32_t parts = SPLIT && a.parts > 1 ? (uint32_t)a.parts : 1u;
  const uint32_t units = (end - beg) * parts;
  for (;;) {
    uint32_t i0 = 0;
    if (lane == 0) i0 = atomicAdd(&a.fetch[cls], (uint32_t)REG_CHUNK);
    i0 = __shfl_sync(MCE_FULL, i0, 0);
    if (i0 >= units) break;
    for (int k = 0; k < REG_CHUNK; ++k) {
      const uint32_t u = i0 + k;
      if (u >= units) break;
      const int32_t r = a.roots[beg + u / parts];
      MCE_BD(BD_ENCODE);
      if (parts == 1 || r != rt.r) reg_encode<Word, NR, STAGE>(a, sm, sl, r, rt);
      MCE_BD(BD_OTHER);
      u64 nd = 0, cnt = 0, op = 0;
      if constexpr (L2) {  // -p l2: the root's edges are the units
        reg_l2_units<Word, NR, LIST>(a, sm, sl, rt, h0, cnt, [&](Word Pv, Word Sv, Word XOv) {
          if (share && wants_task(a.q)) {  // offered to idle warps at once
            const u64 w0 = (u64)(uint32_t)rt.r, w1 = (u64)Pv, w3 = (u64)Sv, w4 = (u64)XOv;
            if (q_push(a.q, a.err, a.wait_limit_ns, [&](uint32_t k2) {
                  return k2 == 0 ? w0 : k2 == 1 ? w1 : k2 == 2 ? 0ull : k2 == 3 ? w3 : w4;
                }) != Q_KEPT) {
              if (EV && lane == 0) warp_record(a)[2] += 1;
              return;
            }
          }
          reg_tree<Word, NR, false, EV, LIST, XP, OPS, SPLIT, true>(a, sm, sl, rt, Pv, (Word)0, Sv,
                                                                    h0, h1, nd, cnt, bd, &op, 0, 1,
                                                                    XOv);
        });
      } else {
        reg_tree<Word, NR, false, EV, LIST, XP, OPS, SPLIT>(a, sm, sl, rt, WOps<Word>::low(rt.d),
                                                            (Word)0, (Word)0, h0, h1, nd, cnt, bd,
                                                            &op, (int)(u % parts), (int)parts);
      }
      nodes += nd;
      root_done(a, r, nd, cnt);
      if constexpr (OPS) {
        ops += op;
        root_ops_done(a, r, op);
      }
    }
  }
  if constexpr (NR == 1 && sizeof(Word) == 4 && EV == 0 && !LIST && !XP && !OPS && !SPLIT &&
                !STAGE && !L2) {
    // frames the lane engine handed over (a.resume)
    const uint32_t frames = a.resume ? min(*a.resume_count, a.resume_cap) : 0u;
    while (frames) {
      uint32_t i = 0;
      if (lane == 0) i = atomicAdd(a.resume_next, 1u);
      i = __shfl_sync(MCE_FULL, i, 0);
      if (i >= frames) break;
      const uint32_t *f = a.resume + (size_t)i * RESUME_WORDS;
      const int32_t r = (int32_t)f[0];
      if (r < 0) continue;  // a slot that was given up
      if (r != rt.r) reg_encode<Word, NR, STAGE>(a, sm, sl, r, rt, false);
      u64 nd = 0, cnt = 0, op = 0;
      reg_tree<Word, NR, false, EV, LIST, XP, OPS, false>(a, sm, sl, rt, f[1], f[2], f[3], h0, h1,
                                                          nd, cnt, bd, &op, 0, 1, (Word)0, true,
                                                          f[4], f[5]);
      nodes += nd;
      root_done(a, r, nd, cnt);
    }
  }
  if (share) {
    root_phase_done(a.q);
    u64 t0 = 0, t1 = 0, t2 = 0, t3 = 0, t4 = 0;
    MCE_BD(BD_QUEUE);
    idle_phase(
        a,
        [&](uint32_t k, u64 w) {  // lane k receives word k
          if (k == 0) t0 = w;
          if (k == 1) t1 = w;
          if (k == 2) t2 = w;
          if (k == 3) t3 = w;
          if (k == 4) t4 = w;
        },
        [&]() {
          // word k of the task arrived on lane k
          const int32_t r = (int32_t)__shfl_sync(MCE_FULL, t0, 0);
          const Word P = (Word)__shfl_sync(MCE_FULL, t1, 1);
          const Word X = (Word)__shfl_sync(MCE_FULL, t2, 2);
          const Word S = (Word)__shfl_sync(MCE_FULL, t3, 3);
          const Word XO = L2 ? (Word)__shfl_sync(MCE_FULL, t4, 4) : (Word)0;  // L2 unit's outside rows
          MCE_BD(BD_ENCODE);
          if (r != rt.r) reg_encode<Word, NR, STAGE>(a, sm, sl, r, rt, false);
          u64 nd = 0, cnt = 0, op = 0;
          reg_tree<Word, NR, false, EV, LIST, XP, OPS, false, L2>(a, sm, sl, rt, P, X, S, h0, h1, nd,
                                                                  cnt, bd, &op, 0, 1, XO);
          nodes += nd;
          root_done(a, r, nd, cnt);
          if constexpr (OPS) {
            ops += op;
            root_ops_done(a, r, op);
          }
          MCE_BD(BD_QUEUE);
        });
  }
  MCE_BD(BD_OTHER);
  if (h0) atomicAdd(&a.hist[lane + 2], h0);
  if (h1) atomicAdd(&a.hist[lane + 34], h1);
  if (lane == 0 && nodes) atomicAdd(a.nodes, nodes);  // warp-uniform count
  if (OPS && lane == 0 && ops) atomicAdd(a.ops, ops);
  if (EV && lane == 0) {  // opts.warp_log
    u64 *w = warp_record(a);
    w[0] = sm_id();
    w[1] = nodes;
    if constexpr (EV == 2)
      for (int i = 0; i < 7; ++i) w[3 + i] = bdv.acc[i];
  }
}

// The wide engine at 4 blocks per SM (96 registers) or, with
// opts.wide_blocks = 8, at 8 (64 registers): more warps pay on graphs whose
// wide roots have large shared subtrees (R-MAT), fewer on many small ones.
template <int EV = 0, int MINB = 1, bool LIST = false, bool OPS = false, bool SPLIT = false,
          bool XP = false, bool L2 = false>
__global__ void __launch_bounds__(MEM_BLOCK, MINB) bk_mem_kernel(BKArgs a, int cls) {
  __shared__ MemSmem sm_all[MEM_BLOCK / 32];
  __shared__ u64 srows_all[MEM_BLOCK / 32][2 * MEM_SROWS_D];
  MemSmem &sm = sm_all[threadIdx.x >> 5];
  u64 *srows = srows_all[threadIdx.x >> 5];
  const int lane = (int)lane_id();
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const Slab sl = slab_of(a, gw);
  const uint32_t beg = a.shape->cls_off[cls], end = a.shape->cls_off[cls + 1];
  const bool share = a.q.hdr != nullptr;
  u64 h0 = 0, h1 = 0, nodes = 0, ops = 0;
  MemRoot rt;
  Bd bdv, *bd = &bdv;
  if constexpr (EV == 2) bdv.start();
  if (share && lane == 0) atomicAdd(&a.q.hdr->work, 1u);
  const uint32_t parts = SPLIT && a.parts > 1 ? (uint32_t)a.parts : 1u;  // warps per root
  const uint32_t units = (end - beg) * parts;
  for (;;) {
    uint32_t i0 = 0;
    if (lane == 0) i0 = atomicAdd(&a.fetch[cls], 1u);
    i0 = __shfl_sync(MCE_FULL, i0, 0);
    if (i0 >= units) break;
    const int32_t r = a.roots[beg + i0 / parts];
    MCE_BD(BD_ENCODE);
    if (a.d_lo && a.rp[r + 1] - a.split[r] <= a.d_lo) continue;
    if (parts == 1 || r != rt.r) mem_encode(a, sm, sl, r, rt, srows);
    MCE_BD(BD_OTHER);
    if (rt.d == 0) continue;
    const int Wr = rt.Wr;
    u64 nd = 0, cnt = 0, op = 0;
    if constexpr (L2) {  // -p l2: the root's edges are the units
      const int WM = (a.dcap + 63) >> 6;
      mem_l2_units<LIST>(a, sl, rt, h0, h1, cnt, [&](bool xo_any) {
        if (share && wants_task(a.q)) {  // offered to idle warps at once
          const u64 *F0 = sl.stk;
          if (q_push(a.q, a.err, a.wait_limit_ns, [&](uint32_t k2) -> u64 {
                if (k2 == 0) return (u64)(uint32_t)r;
                const uint32_t part = (k2 - 1) / WM, w = (k2 - 1) % WM;
                if ((int)w >= Wr) return 0ull;
                return part == 0 ? F0[w] : part == 1 ? 0ull : part == 2 ? F0[3 * Wr + w] : sl.xo[w];
              }) != Q_KEPT) {
            if (EV && lane == 0) warp_record(a)[2] += 1;
            return;
          }
        }
        mem_tree<false, EV, LIST, OPS, SPLIT, XP, true>(a, sl, rt, h0, h1, nd, cnt, bd, &op, 0, 1,
                                                        xo_any);
      });
    } else {
      if (lane < Wr) {  // root frame: P = all of N+(r), X = 0, S = 0
        const u64 all = (lane == Wr - 1 && (rt.d & 63)) ? ((1ull << (rt.d & 63)) - 1ull) : ~0ull;
        sl.stk[lane] = all;
        sl.stk[Wr + lane] = 0;
        sl.stk[3 * Wr + lane] = 0;
      }
      __syncwarp();
      mem_tree<false, EV, LIST, OPS, SPLIT, XP>(a, sl, rt, h0, h1, nd, cnt, bd, &op, (int)(i0 % parts),
                                            (int)parts);
    }
    nodes += nd;
    root_done(a, r, nd, cnt);
    if constexpr (OPS) {
      ops += op;
      root_ops_done(a, r, op);
    }
  }
  if (share) {
    root_phase_done(a.q);
    const int WM = (a.dcap + 63) >> 6;
    int32_t task_root = -1;
    MCE_BD(BD_QUEUE);
    idle_phase(
        a,
        [&](uint32_t k, u64 w) {
          if (k == 0) {
            task_root = (int32_t)w;  // lane 0 reads word 0
          } else {
            const uint32_t part = (k - 1) / WM, ww = (k - 1) % WM;
            sl.xs[part * WM + ww] = w;  // staged; moved to frame 0 after encode
          }
        },
        [&]() {
          const int32_t r = __shfl_sync(MCE_FULL, task_root, 0);
          __syncwarp();
          // the staging area is rewritten by mem_encode: keep the task first
          u64 tp = 0, tx = 0, ts = 0, to = 0;
          if (lane < WM) {
            tp = sl.xs[lane];
            tx = sl.xs[WM + lane];
            ts = sl.xs[2 * WM + lane];
            to = sl.xs[3 * WM + lane];  // an L2 unit's outside rows (0 otherwise)
          }
          __syncwarp();
          MCE_BD(BD_ENCODE);
          if (r != rt.r) mem_encode(a, sm, sl, r, rt, srows);
          MCE_BD(BD_QUEUE);
          if (rt.d == 0) return;
          const int Wr = rt.Wr;
          if (lane < Wr) {
            sl.stk[lane] = tp;
            sl.stk[Wr + lane] = tx;
            sl.stk[3 * Wr + lane] = ts;
            sl.xo[lane] = to;
          }
          const bool xo_any = __any_sync(MCE_FULL, lane < Wr && to != 0);
          __syncwarp();
          u64 nd = 0, cnt = 0, op = 0;
          mem_tree<false, EV, LIST, OPS, false, XP, L2>(a, sl, rt, h0, h1, nd, cnt, bd, &op, 0, 1,
                                                        xo_any);
          nodes += nd;
          root_done(a, r, nd, cnt);
          if constexpr (OPS) {
            ops += op;
            root_ops_done(a, r, op);
          }
          MCE_BD(BD_QUEUE);
        });
  }
  MCE_BD(BD_OTHER);
  if (h0) atomicAdd(&a.hist[lane + 2], h0);
  if (h1) atomicAdd(&a.hist[lane + 34], h1);
  if (lane == 0 && nodes) atomicAdd(a.nodes, nodes);  // warp-uniform count
  if (OPS && lane == 0 && ops) atomicAdd(a.ops, ops);
  if (EV && lane == 0) {  // opts.warp_log
    u64 *w = warp_record(a);
    w[0] = sm_id();
    w[1] = nodes;
    if constexpr (EV == 2)
      for (int i = 0; i < 7; ++i) w[3 + i] = bdv.acc[i];
  }
}

}  // namespace

size_t bk_slab_words(int cls, int dcap, int xcap, int rxcap) {
  if (cls == CLS_R32 || cls == CLS_R64) return 4 * (size_t)rxcap;  // hash, rows, leaf list
  const size_t WM = (size_t)(dcap + 63) / 64;
  size_t w = (size_t)dcap * WM + (size_t)(dcap + 1) * 4 * WM + 32 * WM + (size_t)xcap * WM;
  w += WM;                                          // xo (an L2 unit's outside rows)
  w += (size_t)hash_cap(xcap);                      // hash set (one-word rows)
  w += (3 * (size_t)dcap + (size_t)xcap + 1) / 2 + 1;  // pl, xl (xcap + dcap) and pk (int32)
  w += (size_t)p_cap(dcap);                         // hash of P: keys and indices (int32)
  w = w > 3 * WM + 1 ? w : 3 * WM + 1;
  return (w + 31) & ~(size_t)31;                    // 256-byte aligned slabs
}

uint32_t bk_task_words(int cls, int dcap) {
  if (cls == CLS_R32 || cls == CLS_R64) return 5;  // root, P, X, chosen set, L2 outside rows
  return 1 + 4 * (uint32_t)((dcap + 63) / 64);     // the same, W words each
}

int bk_warps_for_class(int cls, int sms, int wide_blocks, int *warps, int *block, int *smem) {
  int per_sm = 0;
  if (cls == CLS_R32 || cls == CLS_R64) {
    *block = REG_BLOCK;
    *smem = 0;
    if (cls == CLS_R32)
      MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bk_reg_kernel<uint32_t, 1>, REG_BLOCK, 0));
    else
      MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bk_reg_kernel<u64, 2>, REG_BLOCK, 0));
    if (per_sm < 1) per_sm = 1;
    *warps = sms * per_sm * (REG_BLOCK / 32);
  } else {
    *block = MEM_BLOCK;
    *smem = 0;
    // the variant's resident blocks per SM (its registers decide), at most 4 or 8
    if (wide_blocks == 8)
      MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bk_mem_kernel<0, 8>, MEM_BLOCK, 0));
    else
      MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bk_mem_kernel<>, MEM_BLOCK, 0));
    const int cap = wide_blocks == 8 ? 8 : 4;
    if (per_sm > cap) per_sm = cap;
    if (per_sm < 1) per_sm = 1;
    *warps = sms * per_sm * (MEM_BLOCK / 32);
  }
  return MCE_OK;
}

namespace {

// One engine-class launch of the variant <EV, LIST, XP, OPS, SPLIT, STAGE, L2>.
template <int EV, bool LIST, bool XP, bool OPS, bool SPLIT, bool STAGE, bool L2>
int launch_cls(int cls, int word_bits, const BKArgs &a, int grid, int block, int smem,
               cudaStream_t s) {
  if (cls == CLS_R32 && word_bits == 64)
    bk_reg_kernel<u64, 1, EV, LIST, XP, OPS, SPLIT, false, L2><<<grid, block, smem, s>>>(a, cls);
  else if (cls == CLS_R32)
    bk_reg_kernel<uint32_t, 1, EV, LIST, XP, OPS, SPLIT, STAGE, L2><<<grid, block, smem, s>>>(a, cls);
  else if (cls == CLS_R64)
    bk_reg_kernel<u64, 2, EV, LIST, XP, OPS, SPLIT, false, L2><<<grid, block, smem, s>>>(a, cls);
  else if (cls == CLS_MEM && a.wide8 && EV == 0)
    bk_mem_kernel<EV, 8, LIST, OPS, SPLIT, XP, L2><<<grid, block, smem, s>>>(a, cls);
  else if (cls == CLS_MEM)
    bk_mem_kernel<EV, 1, LIST, OPS, SPLIT, XP, L2><<<grid, block, smem, s>>>(a, cls);
  else
    return MCE_EINVAL;
  MCE_CUDA(cudaGetLastError());
  return MCE_OK;
}

}  // namespace

// The variant a call needs: listing, the evaluation logs (per-warp load, and
// cycles), the word-op count, several warps per root, -i px, staged lists,
// L2 units.  Modes that do not combine: the evaluation and listing variants
// run with one warp per root and IP pivots; the word-op count with IP and L1.
int bk_launch(int cls, int word_bits, const BKArgs &a, int grid, int block, int smem,
              cudaStream_t s, int *launches) {
  if (grid <= 0) return MCE_OK;
  const int ev = a.warp_log == nullptr ? 0 : (a.warp_cycles ? 2 : 1);
  const bool xp = a.x_pivot != 0, split = a.parts > 1;
  int rc;
  if (a.level2) {
    if (a.list_buf)
      rc = launch_cls<0, true, false, false, false, false, true>(cls, word_bits, a, grid, block, smem, s);
    else if (ev == 2)
      rc = launch_cls<2, false, false, false, false, false, true>(cls, word_bits, a, grid, block, smem, s);
    else if (ev == 1)
      rc = launch_cls<1, false, false, false, false, false, true>(cls, word_bits, a, grid, block, smem, s);
    else if (xp)
      rc = launch_cls<0, false, true, false, false, false, true>(cls, word_bits, a, grid, block, smem, s);
    else
      rc = launch_cls<0, false, false, false, false, false, true>(cls, word_bits, a, grid, block, smem, s);
  } else if (a.list_buf) {
    rc = launch_cls<0, true, false, false, false, false, false>(cls, word_bits, a, grid, block, smem, s);
  } else if (a.count_ops) {
    rc = launch_cls<0, false, false, true, true, false, false>(cls, word_bits, a, grid, block, smem, s);
  } else if (ev == 2) {
    rc = launch_cls<2, false, false, false, false, false, false>(cls, word_bits, a, grid, block, smem, s);
  } else if (ev == 1) {
    rc = launch_cls<1, false, false, false, false, false, false>(cls, word_bits, a, grid, block, smem, s);
  } else if (split) {
    if (xp)
      rc = launch_cls<0, false, true, false, true, false, false>(cls, word_bits, a, grid, block, smem, s);
    else
      rc = launch_cls<0, false, false, false, true, false, false>(cls, word_bits, a, grid, block, smem, s);
  } else if (xp) {
    rc = launch_cls<0, false, true, false, false, false, false>(cls, word_bits, a, grid, block, smem, s);
  } else if (a.stage) {
    rc = launch_cls<0, false, false, false, false, true, false>(cls, word_bits, a, grid, block, smem, s);
  } else {
    rc = launch_cls<0, false, false, false, false, false, false>(cls, word_bits, a, grid, block, smem, s);
  }
  if (rc == MCE_OK && launches) *launches += 1;
  return rc;
}

int queue_launch_init(const QueueView &q, cudaStream_t s, int *launches, bool keep_pushed) {
  MCE_CUDA(cudaMemsetAsync(q.hdr, 0, keep_pushed ? offsetof(QueueHdr, pushed) : sizeof(QueueHdr), s));
  queue_init_kernel<<<(q.cap + 255) / 256, 256, 0, s>>>(q);
  MCE_CUDA(cudaGetLastError());
  if (launches) *launches += 1;
  return MCE_OK;
}

// ===========================================================================
// Allocation-free search entry point.
//
// For callers that cannot allocate device memory: processes whose GPU memory
// is owned entirely by another allocator (a framework's caching allocator
// that has reserved the device), and latency-critical loops in which
// cudaMalloc's implicit device-wide synchronisation is not acceptable.  The
// caller passes an oriented graph, a root list and a histogram, all already
// in device memory; the search runs the 32-wide register engine with its
// per-warp scratch in the file-scope array below, which every GPU that loads
// this library holds until the process exits.
//
// Every call resolves the array's device address on the current device with
// cudaGetSymbolAddress, checks the root ids against the vertex count before
// any read at them, and synchronises its stream twice (the root check, the
// status) before it returns.  Every call shares
// the array and clears the part that must start at zero, so calls whose work
// overlaps on the GPU race with each other: serialise them (one stream, or
// events).
// ===========================================================================
namespace {

constexpr size_t NOALLOC_CTL_BYTES = 1024;  // ShapeInfo, fetch counters, status, nodes
constexpr size_t NOALLOC_SLAB_WORDS = 2 * REG_XCAP;  // u64 words per warp: 4 x REG_XCAP u32 words
static_assert(MCE_NOALLOC_SCRATCH_BYTES % 256 == 0, "scratch size");

static __device__ __align__(256) unsigned long long g_noalloc_scratch[MCE_NOALLOC_SCRATCH_BYTES / 8];

struct NoallocCtl {
  ShapeInfo shape;
  uint32_t fetch[8];
  uint32_t err[4];
  unsigned long long nodes[4];
};
static_assert(sizeof(NoallocCtl) <= NOALLOC_CTL_BYTES, "control block");

// The host-side name g_noalloc_scratch is not a device address; the address
// of the current device's copy is looked up on every call (cheap next to the
// call's two stream synchronisations), so there is no host-side cache to
// guard between threads or to go stale after a device reset.
int noalloc_scratch(unsigned long long **out) {
  void *p = nullptr;
  MCE_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
  *out = (unsigned long long *)p;
  return MCE_OK;
}

// Every root id must lie in [0, n) - tested before anything is read at that
// id (bit 2 of err[0]) - and fit the 32-wide engine: 1..32 later and
// <= REG_XCAP earlier neighbours (bit 1).
__global__ void noalloc_check_kernel(const int32_t *rp, const int32_t *split, int64_t n,
                                     const int32_t *roots, uint32_t num_roots, NoallocCtl *ctl) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    ctl->shape.cls_off[CLS_R32] = 0;
    ctl->shape.cls_off[CLS_R32 + 1] = num_roots;
  }
  if (i >= num_roots) return;
  const int32_t r = roots[i];
  if (r < 0 || (int64_t)r >= n) {
    atomicOr(&ctl->err[0], 2u);
    return;
  }
  const int32_t dplus = rp[r + 1] - split[r], dminus = split[r] - rp[r];
  if (dplus < 1 || dplus > 32 || dminus > REG_XCAP) atomicOr(&ctl->err[0], 1u);
}

}  // namespace

extern "C" int mce_count_oriented_noalloc(const int32_t *d_row_ptr, const int32_t *d_split,
                                          const int32_t *d_col_split, int64_t n,
                                          const int32_t *d_roots, int64_t num_roots,
                                          uint64_t *d_hist, void *stream) {
  if (num_roots < 0 || n < 0 || !d_hist ||
      (num_roots > 0 && (!d_row_ptr || !d_split || !d_col_split || !d_roots)))
    return MCE_EINVAL;
  if (num_roots >= ((int64_t)1 << 31) || n >= ((int64_t)1 << 31)) return MCE_ELIMIT;
  int dev = 0, sms = 0, per_sm = 0;
  MCE_CUDA(cudaGetDevice(&dev));
  unsigned long long *base = nullptr;
  int rc = noalloc_scratch(&base);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  NoallocCtl *ctl = (NoallocCtl *)base;
  MCE_CUDA(cudaMemsetAsync(ctl, 0, NOALLOC_CTL_BYTES, s));
  const uint32_t nr = (uint32_t)num_roots;
  noalloc_check_kernel<<<(nr + 255) / 256 + 1, 256, 0, s>>>(d_row_ptr, d_split, n, d_roots, nr,
                                                             ctl);
  MCE_CUDA(cudaGetLastError());
  uint32_t err = 0;
  MCE_CUDA(cudaMemcpyAsync(&err, &ctl->err[0], sizeof(err), cudaMemcpyDeviceToHost, s));
  MCE_CUDA(cudaStreamSynchronize(s));
  if (err & 2u) return MCE_EINVAL;
  if (err) return MCE_ELIMIT;
  MCE_CUDA(cudaMemsetAsync(d_hist, 0, sizeof(uint64_t) * MCE_HIST_MAX, s));
  if (nr == 0) {
    MCE_CUDA(cudaStreamSynchronize(s));
    return MCE_OK;
  }
  // as many whole blocks of warps as the occupancy, the roots and the array allow
  MCE_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bk_reg_kernel<uint32_t, 1>,
                                                         REG_BLOCK, 0));
  const int wpb = REG_BLOCK / 32;
  const int64_t slab_warps =
      (int64_t)((MCE_NOALLOC_SCRATCH_BYTES - NOALLOC_CTL_BYTES) / (NOALLOC_SLAB_WORDS * 8));
  int64_t blocks = (int64_t)sms * (per_sm > 0 ? per_sm : 1);
  blocks = blocks < slab_warps / wpb ? blocks : slab_warps / wpb;
  const int64_t want = ((int64_t)nr + REG_CHUNK * wpb - 1) / (REG_CHUNK * wpb);
  if (want < blocks) blocks = want;
  BKArgs a;
  memset(&a, 0, sizeof(a));
  a.rp = d_row_ptr;
  a.split = d_split;
  a.cs = d_col_split;
  a.roots = d_roots;
  a.shape = &ctl->shape;
  a.fetch = ctl->fetch;
  a.hist = (unsigned long long *)d_hist;
  a.nodes = ctl->nodes;
  a.err = &ctl->err[1];
  a.slab = base + NOALLOC_CTL_BYTES / 8;
  a.slab_words = NOALLOC_SLAB_WORDS;
  a.dcap = 32;
  a.xcap = REG_XCAP;
  a.rxcap = REG_XCAP;
  bk_reg_kernel<uint32_t, 1><<<(unsigned)blocks, REG_BLOCK, 0, s>>>(a, CLS_R32);
  MCE_CUDA(cudaGetLastError());
  MCE_CUDA(cudaMemcpyAsync(&err, &ctl->err[1], sizeof(err), cudaMemcpyDeviceToHost, s));
  MCE_CUDA(cudaStreamSynchronize(s));
  return err ? MCE_ELIMIT : MCE_OK;
}

}  // namespace mce
