// Degeneracy order by synchronous k-core peeling: one cooperative launch.
//
// Replaces graph::SingleGPU_Kcore::findKcoreIncremental_async
// (include/kcore.cuh:233-316), which drives every peel round from the host
// with several launches and a cudaDeviceSynchronize + scalar read-backs per
// round.  Here all levels and rounds run inside one persistent kernel whose
// blocks meet at a bounded grid barrier between phases; the host launches
// once and reads nothing until the end.
//
// Semantics kept from the reference (so priorities are bit-identical):
//  - at level k, round 0 is every remaining vertex of remaining degree k
//    (filter_window + filter_with_random_append, include/kcore.cuh:21-48);
//  - removing a round lowers neighbour degrees; a neighbour whose degree
//    falls from k+1 to k joins the next round (process_degree, :80-95);
//  - rounds are numbered over all levels; priority[v] = v's round number,
//    and the round that empties the graph is not processed, so its vertices
//    keep priority = m (:258, :276);
//  - a level with no vertex of degree k runs no round (the scan below jumps
//    straight to the smallest remaining degree, which numbers rounds the
//    same way).
// Decrements of a vertex that is already removed or queued change no round's
// membership: its degree is at most its level and only falls, while a vertex
// joins a round only when its degree falls from level + 1.  So no core number
// is read before a decrement, and a scan tells the remaining vertices by
// their degree alone.
#include <climits>

#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace mce {

struct PeelCtl {
  uint32_t arrived;    // blocks that reached a phase barrier so far, over all phases
  uint32_t err;
  uint32_t fcnt[3];    // light frontier sizes, one slot per phase mod 3
  unsigned long long hpack[3];  // heavy frontier: (count << 32) | 32-edge chunks
  uint32_t acnt[3];    // alive-list sizes, one slot per scan mod 3
  uint32_t amin[3];    // min degree over the alive list written by a scan
  int32_t degeneracy;
  uint32_t rounds;
  uint32_t levels;
  // state handed back by a solo section (written by block 0, read by all)
  uint32_t solo_q, solo_cnt, solo_priority, solo_rounds;
  int64_t solo_todo;
  int32_t solo_degen;
  uint32_t solo_sections;
  unsigned long long t_scan, t_round, t_wait;  // ns seen by block 0 (diagnostics)
  uint32_t seg_next;   // batches: next graph to peel
  uint32_t seg_part[MAX_BATCH_PARTS];  // ... the same per part of a batch still arriving
  uint32_t seg_mid_next;       // the same for the middle and small graphs' launches
  uint32_t seg_mid_part[MAX_BATCH_PARTS];
  uint32_t seg_small_next;
  uint32_t seg_small_part[MAX_BATCH_PARTS];
};

namespace {

// One block per SM: a phase costs one arrival per block at the barrier.  The
// grid-wide peel is bounded by the latency of its phases (a barrier, then some
// six dependent accesses); with one counter that only grows, one reader of the
// phase's counters per block and no core number read before a decrement, a
// round of BA n = 1e6 takes 10 us instead of 17 (peel 3.1 -> 1.77 ms) and the
// order of R-MAT 17 3.1 ms instead of 6.4.
constexpr int PEEL_BLOCK = 1024;
// A frontier of at most solo_max vertices is peeled by block 0 alone, round
// after round with __syncthreads between them, for up to SOLO_ROUNDS rounds
// (well inside the other blocks' barrier wait limit).
constexpr uint32_t SOLO_ROUNDS = 65536;
// A frontier vertex with more neighbours than this is "heavy": it is stored
// from the back of the frontier buffer, its first chunk number goes to the
// slot's chunk-base array, and the round spreads all heavy chunks (32 edges
// each) over every warp, so no single warp serialises a hub while the rest
// of the grid waits at the next barrier.  One 64-bit atomic hands out both
// the slot and the chunk base, so bases increase with the slot.
constexpr int32_t HEAVY_DEG = 256;
// Light frontier vertices a warp takes at a time in a large frontier.
constexpr int PEEL_GROUP = 8;

// A warp's staging buffer for the next frontier: appends gather here and
// reach the list STAGE at a time, one atomic on its counter per flush
// instead of one per 32-edge window (the counter is shared by the grid).
constexpr uint32_t STAGE = 256;
struct Stage {
  int32_t *buf;  // STAGE entries of shared memory, one buffer per warp
  uint32_t n;    // warp-uniform fill
};

__device__ __forceinline__ void stage_flush(Stage &st, int32_t *list, uint32_t *cnt) {
  if (!st.n) return;
  const uint32_t lane = lane_id();
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(cnt, st.n);
  base = __shfl_sync(MCE_FULL, base, 0);
  for (uint32_t i = lane; i < st.n; i += 32) list[base + i] = st.buf[i];
  __syncwarp();
  st.n = 0;
}

__device__ __forceinline__ void stage_append(Stage &st, bool pred, int32_t val, int32_t *list,
                                             uint32_t *cnt) {
  const uint32_t mask = __ballot_sync(MCE_FULL, pred);
  if (!mask) return;
  const uint32_t k = __popc(mask);
  if (st.n + k > STAGE) stage_flush(st, list, cnt);
  if (pred) st.buf[st.n + __popc(mask & ((1u << lane_id()) - 1u))] = val;
  __syncwarp();
  st.n += k;
}

// Block-aggregated appends to two lists (one atomic per list per block);
// every thread of the block must call it.
__device__ __forceinline__ void block_append2(bool p1, int32_t v1, int32_t *l1, uint32_t *c1,
                                              bool p2, int32_t v2, int32_t *l2, uint32_t *c2) {
  __shared__ uint32_t w1[PEEL_BLOCK / 32], w2[PEEL_BLOCK / 32], base1, base2;
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t m1 = __ballot_sync(MCE_FULL, p1), m2 = __ballot_sync(MCE_FULL, p2);
  if (lane == 0) {
    w1[wid] = __popc(m1);
    w2[wid] = __popc(m2);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t a = 0, b = 0;
    for (uint32_t w = 0; w < nw; ++w) {
      const uint32_t x = w1[w], y = w2[w];
      w1[w] = a;
      w2[w] = b;
      a += x;
      b += y;
    }
    base1 = a ? atomicAdd(c1, a) : 0;
    base2 = b ? atomicAdd(c2, b) : 0;
  }
  __syncthreads();
  if (p1) l1[base1 + w1[wid] + __popc(m1 & lt)] = v1;
  if (p2) l2[base2 + w2[wid] + __popc(m2 & lt)] = v2;
  __syncthreads();  // the shared counters are reused by the next call
}

// Append a heavy vertex: slot k at list[cap - 1 - k], first chunk at base[k].
__device__ __forceinline__ void heavy_append(bool pred, int32_t v, int32_t degv, int32_t *list,
                                             int32_t *base, int64_t cap,
                                             unsigned long long *pack) {
  if (!pred) return;
  const unsigned long long chunks = (unsigned long long)((degv + 31) / 32);
  const unsigned long long old = atomicAdd(pack, (1ull << 32) | chunks);
  const uint32_t slot = (uint32_t)(old >> 32);
  list[cap - 1 - (int64_t)slot] = v;
  base[slot] = (int32_t)(uint32_t)old;
}

__device__ __forceinline__ unsigned long long ld_volatile64(const unsigned long long *p) {
  return *(const volatile unsigned long long *)p;
}

// What a phase left behind, read by one thread per block (thousands of warps
// reading the same few words would queue at one L2 slice).
struct PhaseOut {
  uint32_t light, heavy, chunks;  // the frontier: light and heavy vertices, 32-edge chunks
  uint32_t alive, lowest;         // a scan's survivors and their lowest degree
  uint32_t ok;
};

__device__ __forceinline__ void read_frontier(const PeelCtl *ctl, uint32_t slot, PhaseOut &o) {
  const unsigned long long hp = ld_volatile64(&ctl->hpack[slot]);
  o.light = ld_volatile(&ctl->fcnt[slot]);
  o.heavy = (uint32_t)(hp >> 32);
  o.chunks = (uint32_t)hp;
}

// Grid barrier at the end of a phase (all blocks are resident: cooperative
// launch) and the counters of its output: frontier slot q, alive slot s.  One
// counter that only grows, one release add per block and one acquiring reader
// per block; bounded: false (and MCE_ERR_WAIT_TIMEOUT) after limit_ns.
__device__ __forceinline__ bool phase_sync(PeelCtl *ctl, uint32_t nblocks, uint32_t &target,
                                           uint32_t q, uint32_t s, PhaseOut &out,
                                           uint64_t limit_ns) {
  __syncthreads();
  target += nblocks;
  if (threadIdx.x == 0) {
    red_release(&ctl->arrived, 1u);
    uint32_t ok = 1, spins = 0;
    uint64_t t0 = 0;
    while ((int32_t)(ld_acquire(&ctl->arrived) - target) < 0) {
      if ((++spins & 255u) == 0) {
        const uint64_t now = globaltimer_ns();
        if (!t0) t0 = now;
        if (ld_volatile(&ctl->err) & MCE_ERR_WAIT_TIMEOUT) {
          ok = 0;
          break;
        }
        if (now - t0 > limit_ns) {
          atomicOr(&ctl->err, MCE_ERR_WAIT_TIMEOUT);
          ok = 0;
          break;
        }
      }
    }
    read_frontier(ctl, q, out);
    out.alive = ld_volatile(&ctl->acnt[s]);
    out.lowest = ld_volatile(&ctl->amin[s]);
    out.ok = ok;
  }
  __syncthreads();
  return out.ok != 0;
}

// Lower the degree of neighbour col[j] of a vertex being removed; true if it
// falls to `level` (it then joins the next round).
__device__ __forceinline__ bool peel_edge(int32_t j, int32_t e, int32_t level,
                                          const int32_t *__restrict__ col, int32_t *deg,
                                          int32_t &u) {
  u = 0;
  if (j >= e) return false;
  u = col[j];
  return atomicSub(&deg[u], 1) == level + 1;
}

// One peel round (phase q) over the frontier in slot q % 3 (its counters in
// `in`), executed by the threads [t0, t0 + nt) (the whole grid, or block 0
// alone): set the round's priority, lower the neighbours' degrees and append
// every neighbour whose degree falls to `level` to the frontier in slot
// (q + 1) % 3.
__device__ __noinline__ void peel_round(uint32_t q, int32_t level, uint32_t priority,
                                        const PhaseOut &in, int64_t t0, int64_t nt, int64_t cap,
                                        const int32_t *__restrict__ rp,
                                        const int32_t *__restrict__ col, int32_t *deg,
                                        int32_t *core, uint32_t *prio, int32_t *const *fr,
                                        int32_t *const *hb, PeelCtl *ctl, int32_t *stage) {
  const uint32_t lane = lane_id();
  Stage st{stage, 0};
  const int fn = (q + 1) % 3;
  if (t0 == 0) {
    ctl->fcnt[(q + 2) % 3] = 0;
    ctl->hpack[(q + 2) % 3] = 0;
  }
  const uint32_t lc = in.light, hc = in.heavy, hch = in.chunks;
  const int32_t *Fc = fr[q % 3], *HB = hb[q % 3];
  int32_t *Fn = fr[fn], *HBn = hb[fn];
  for (int64_t i = t0; i < (int64_t)lc + hc; i += nt) {
    const int32_t v = i < lc ? Fc[i] : Fc[cap - 1 - (i - lc)];
    prio[v] = priority;
    core[v] = level;
  }
  auto push = [&](bool p, int32_t u) {
    int32_t du = 0;
    if (p) du = rp[u + 1] - rp[u];
    const bool heavy = p && du > HEAVY_DEG;
    stage_append(st, p && !heavy, u, Fn, &ctl->fcnt[fn]);
    heavy_append(heavy, u, du, Fn, HBn, cap, &ctl->hpack[fn]);
  };
  // light vertices: a warp each; in a frontier with at least PEEL_GROUP of
  // them per warp, a warp takes PEEL_GROUP at a time and keeps the loads
  // and degree updates of their first windows in flight together (one chain
  // of dependent accesses per group instead of one per vertex)
  const int64_t nwarp = nt >> 5;
  if (lc >= (int64_t)PEEL_GROUP * nwarp) {
    constexpr int R = PEEL_GROUP;
    const int64_t groups = (lc + R - 1) / R;
    for (int64_t gi = t0 >> 5; gi < groups; gi += nwarp) {
      const int64_t i0 = gi * R;
      const int rows = lc - i0 < R ? (int)(lc - i0) : R;
      int32_t v = 0, b = 0, e = 0;
      if ((int)lane < rows) {
        v = Fc[i0 + lane];
        b = rp[v];
        e = rp[v + 1];
      }
      int32_t U[R];
      bool live[R];
#pragma unroll
      for (int k = 0; k < R; ++k) {  // every row's first window
        const int32_t j = __shfl_sync(MCE_FULL, b, k) + (int32_t)lane;
        const bool in = k < rows && j < __shfl_sync(MCE_FULL, e, k);
        U[k] = in ? col[j] : 0;
        live[k] = in;
      }
      int32_t old[R];
#pragma unroll
      for (int k = 0; k < R; ++k) old[k] = live[k] ? atomicSub(&deg[U[k]], 1) : 0;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        push(live[k] && old[k] == level + 1, U[k]);
      }
      for (int k = 0; k < rows; ++k) {  // the rest of rows longer than a window
        const int32_t bk = __shfl_sync(MCE_FULL, b, k), ek = __shfl_sync(MCE_FULL, e, k);
        for (int32_t j0 = bk + 32; j0 < ek; j0 += 32) {
          int32_t u;
          const bool p = peel_edge(j0 + (int32_t)lane, ek, level, col, deg, u);
          push(p, u);
        }
      }
    }
  } else {
    for (int64_t i = t0 >> 5; i < lc; i += nwarp) {
      const int32_t v = Fc[i];
      const int32_t b = rp[v], e = rp[v + 1];
      for (int32_t j0 = b; j0 < e; j0 += 32) {
        int32_t u;
        const bool p = peel_edge(j0 + (int32_t)lane, e, level, col, deg, u);
        push(p, u);
      }
    }
  }
  // heavy vertices: chunk c belongs to the last slot whose base is <= c
  for (int64_t c = t0 >> 5; c < hch; c += nt >> 5) {
    int lo = 0, hi = (int)hc;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (HB[mid] <= (int32_t)c)
        lo = mid + 1;
      else
        hi = mid;
    }
    const int h = lo - 1;
    const int32_t v = Fc[cap - 1 - h];
    const int32_t e = rp[v + 1];
    const int32_t j = rp[v] + ((int32_t)c - HB[h]) * 32 + (int32_t)lane;
    int32_t u;
    const bool p = peel_edge(j, e, level, col, deg, u);
    push(p, u);
  }
  stage_flush(st, Fn, &ctl->fcnt[fn]);
}

__global__ void __launch_bounds__(PEEL_BLOCK)
    peel_kernel(int32_t n, uint32_t m, const int32_t *__restrict__ rp,
                const int32_t *__restrict__ col, int32_t *deg, int32_t *core, uint32_t *prio,
                int32_t *alistA, int32_t *alistB, int32_t *front0, int32_t *front1,
                int32_t *front2, int32_t *hb0, int32_t *hb1, int32_t *hb2, PeelCtl *ctl,
                uint64_t limit_ns, uint32_t solo_max) {
  __shared__ int32_t stage_all[PEEL_BLOCK / 32][STAGE];
  __shared__ PhaseOut out;  // of the latest phase
  int32_t *const stage = stage_all[threadIdx.x >> 5];
  const uint32_t nblocks = gridDim.x;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthr = (int64_t)gridDim.x * blockDim.x;
  const uint32_t lane = lane_id();
  int32_t *const fr[3] = {front0, front1, front2};
  int32_t *const hb[3] = {hb0, hb1, hb2};
  int32_t *alist[2] = {alistA, alistB};

  for (int64_t v = tid; v < n; v += nthr) {
    deg[v] = rp[v + 1] - rp[v];
    core[v] = -1;
    prio[v] = m;
    alistA[v] = (int32_t)v;
  }
  if (tid == 0) {  // phase/scan 0 reads acnt[0]; every other counter starts at 0
    ctl->fcnt[0] = ctl->fcnt[1] = ctl->fcnt[2] = 0;
    ctl->hpack[0] = ctl->hpack[1] = ctl->hpack[2] = 0;
    ctl->acnt[0] = (uint32_t)n;
    ctl->acnt[1] = ctl->acnt[2] = 0;
    ctl->amin[0] = ctl->amin[1] = ctl->amin[2] = 0xFFFFFFFFu;
  }
  uint32_t target = 0;  // arrivals at the end of the current phase
  if (!phase_sync(ctl, nblocks, target, 0, 0, out, limit_ns)) return;

  // phase timers of block 0 (diagnostics only)
  unsigned long long t_ts = 0, t_tr = 0, t_w = 0, mark = tid == 0 ? globaltimer_ns() : 0;
  auto tick = [&](unsigned long long &acc) {
    if (tid == 0) {
      const unsigned long long now = globaltimer_ns();
      acc += now - mark;
      mark = now;
    }
  };
  int64_t todo = n;
  int32_t level = 0, degen = 0;
  uint32_t priority = 0, rounds = 0, levels = 0;
  // Phases (scans and rounds) are numbered q = 0, 1, 2, ...  Phase q appends
  // its output frontier to buffer/counter slot (q + 1) % 3 and resets slot
  // (q + 2) % 3; after barrier q every thread reads slot (q + 1) % 3.  A
  // slot is reset two phases after it was read, so a slow reader can never
  // see a counter that another block has already started to refill.  Scans
  // are numbered s the same way for the alive-list counters (3 slots) and
  // buffers (2 slots).
  uint32_t q = 0, s = 0;
  while (todo > 0) {
    // ---- scan: split the alive list into {deg == level} and {deg > level}
    const uint32_t nalive = out.alive;
    const int32_t *A = alist[s & 1];
    int32_t *A2 = alist[(s + 1) & 1];
    const int fo = (q + 1) % 3, ao = (s + 1) % 3;
    int32_t *F = fr[fo];
    if (tid == 0) {
      ctl->acnt[(s + 2) % 3] = 0;
      ctl->amin[(s + 2) % 3] = 0xFFFFFFFFu;
      ctl->fcnt[(q + 2) % 3] = 0;
      ctl->hpack[(q + 2) % 3] = 0;
    }
    {
      uint32_t mymin = 0xFFFFFFFFu;
      // block-strided so that every thread of a block runs the same number
      // of iterations: appends are aggregated per block (one atomic each)
      const int64_t bs = blockDim.x;
      const int64_t lim = ((int64_t)nalive + bs - 1) / bs * bs;
      for (int64_t i = tid; i < lim; i += nthr) {
        int32_t v = 0, d = 0;
        bool live = false;
        if (i < nalive) {
          v = A[i];
          live = true;
          d = deg[v];
        }
        const bool inF = live && d == level;
        const bool keep = live && d > level;
        const int32_t dv = inF ? rp[v + 1] - rp[v] : 0;
        const bool heavy = inF && dv > HEAVY_DEG;
        block_append2(inF && !heavy, v, F, &ctl->fcnt[fo], keep, v, A2, &ctl->acnt[ao]);
        heavy_append(heavy, v, dv, F, hb[fo], (int64_t)n + 1, &ctl->hpack[fo]);
        if (keep) mymin = min(mymin, (uint32_t)d);
      }
      mymin = __reduce_min_sync(MCE_FULL, mymin);
      if (lane == 0 && mymin != 0xFFFFFFFFu) atomicMin(&ctl->amin[ao], mymin);
    }
    tick(t_ts);
    ++q;
    ++s;
    if (!phase_sync(ctl, nblocks, target, q % 3, s % 3, out, limit_ns)) return;
    tick(t_w);
    uint32_t cnt = out.light + out.heavy;
    if (cnt == 0) {
      // no vertex of degree `level` remains: jump to the smallest degree
      // (a rescan at that level always finds the vertex that attains it)
      const uint32_t mn = out.lowest;
      if (mn == 0xFFFFFFFFu || (int32_t)mn <= level) {
        if (tid == 0) atomicOr(&ctl->err, MCE_ERR_QUEUE);  // inconsistent state: stop
        break;
      }
      level = (int32_t)mn;
      continue;
    }
    ++levels;
    // ---- rounds of this level: phase q reads frontier q % 3
    while (cnt > 0) {
      degen = level;
      todo -= cnt;
      if (todo == 0) {  // the final round keeps priority = m
        const int32_t *Fc = fr[q % 3];
        for (int64_t i = tid; i < (int64_t)out.light + out.heavy; i += nthr)
          core[i < out.light ? Fc[i] : Fc[n - (i - out.light)]] = level;
        break;
      }
      if (cnt <= solo_max) {
        // Small frontier: block 0 peels consecutive rounds alone.  The first
        // barrier lets every block read `cnt` before block 0 recycles slots.
        tick(t_tr);
        if (!phase_sync(ctl, nblocks, target, q % 3, s % 3, out, limit_ns)) return;
        tick(t_w);
        if (blockIdx.x == 0) {
          uint32_t it = 0;
          for (;;) {
            peel_round(q, level, priority, out, threadIdx.x, blockDim.x, (int64_t)n + 1, rp, col,
                       deg, core, prio, fr, hb, ctl, stage);
            __syncthreads();
            ++q;
            if (threadIdx.x == 0) read_frontier(ctl, q % 3, out);
            __syncthreads();
            cnt = out.light + out.heavy;
            ++priority;
            ++rounds;
            if (cnt == 0 || cnt > solo_max || ++it >= SOLO_ROUNDS) break;  // cnt not yet counted
            degen = level;
            todo -= cnt;
            if (todo == 0) {  // the final round keeps priority = m
              const int32_t *Fc = fr[q % 3];
              for (int64_t i = threadIdx.x; i < (int64_t)cnt; i += blockDim.x)
                core[i < out.light ? Fc[i] : Fc[n - (i - out.light)]] = level;
              break;
            }
            __syncthreads();       // every thread has read cnt before slots rotate
          }
          if (threadIdx.x == 0) {
            ctl->solo_q = q;
            ctl->solo_cnt = cnt;
            ctl->solo_priority = priority;
            ctl->solo_rounds = rounds;
            ctl->solo_todo = todo;
            ctl->solo_degen = degen;
            ++ctl->solo_sections;
          }
        }
        tick(t_tr);
        if (!phase_sync(ctl, nblocks, target, q % 3, s % 3, out, limit_ns)) return;
        tick(t_w);
        q = ld_volatile(&ctl->solo_q);
        cnt = ld_volatile(&ctl->solo_cnt);
        __syncthreads();  // every thread is past the barrier's output
        if (threadIdx.x == 0) read_frontier(ctl, q % 3, out);
        __syncthreads();
        priority = ld_volatile(&ctl->solo_priority);
        rounds = ld_volatile(&ctl->solo_rounds);
        todo = *(volatile int64_t *)&ctl->solo_todo;
        degen = *(volatile int32_t *)&ctl->solo_degen;
        if (todo == 0) break;
        continue;
      }
      peel_round(q, level, priority, out, tid, nthr, (int64_t)n + 1, rp, col, deg, core, prio, fr,
                 hb, ctl, stage);
      tick(t_tr);
      ++q;
      if (!phase_sync(ctl, nblocks, target, q % 3, s % 3, out, limit_ns)) return;
      tick(t_w);
      cnt = out.light + out.heavy;
      ++priority;
      ++rounds;
    }
    if (todo == 0) break;
    ++level;
  }
  if (tid == 0) {
    ctl->degeneracy = degen;
    ctl->t_scan = t_ts;
    ctl->t_round = t_tr;
    ctl->t_wait = t_w;
    ctl->rounds = rounds;
    ctl->levels = levels;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Batches: one block peels one graph of the disjoint union at a time.
//
// The graphs of a batch share no edge, so each can be peeled alone; a block
// runs a graph's synchronous rounds with __syncthreads between them instead
// of grid barriers, and blocks take graphs largest first.  Rounds are
// numbered per graph and a graph's final round keeps priority m_g (its own
// arc count): each graph gets the numbering the reference gives it when it
// is the whole input.  Orientation only compares vertices of one graph.
// ---------------------------------------------------------------------------
namespace {

// 16 warps per graph: on the 4,096-graph batch the per-graph peel took
// 5.6 ms with 256 threads, 3.6 ms with 512 and 5.0 ms with 1,024 (its length
// is the round chain of the largest graphs; more threads shorten each round,
// fewer resident blocks leave fewer graphs running at once).
constexpr int SEG_BLOCK = 512;

// Rows longer than SEG_HEAVY arcs are walked by every warp of the block
// together, up to SEG_HEAVY_MAX of them per round.
constexpr int SEG_HEAVY = 256, SEG_HEAVY_MAX = 32;
// Frontier vertices whose rows a warp has in flight together.
constexpr int SEG_GROUP = 8;

struct SegShared {
  int32_t todo, level, minv, fcnt, ncnt;
  uint32_t g;
  // peel_graph_smem: one slot per phase (scan or round) mod 3, reset one
  // phase before it is used, one phase after it was last read
  uint32_t cnt[3], mn[3], hcnt[3];
  uint16_t heavy[SEG_HEAVY_MAX];
};

// Graphs of at most SEG_SMEM_N vertices keep their remaining degrees (16-bit
// halves of 32-bit words, decremented by one atomic on the word; bit 15 marks
// a vertex that is queued or removed, whose further decrements change
// nothing) and the order in which vertices are queued (16-bit local ids) in
// shared memory.  The frontier of a round is a slice of that order.
constexpr int SEG_SMEM_N = 16384;
constexpr uint32_t SEG_GONE = 0x8000u;

// One graph (local vertices 0..n-1 = union vertices vb..vb+n-1) peeled by one
// block; the rounds and their numbering are those of the global-memory path
// below.  What bounds it is the chain of dependent loads (row offsets, arcs)
// of each round, so a warp takes up to SEG_GROUP frontier vertices at a time
// and has their rows' first windows in flight together, one block barrier
// ends the light rows of a round and one the long ones (long rows are spread
// over the warps), and the tests and decrements stay on the SM.
__device__ void peel_graph_smem(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                                int32_t *core, uint32_t *prio, int64_t vb, int n, uint32_t mg,
                                uint32_t *sdeg, uint16_t *order, SegShared &sh, PeelCtl *ctl) {
  const int lane = (int)lane_id(), w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const int words = (n + 1) >> 1;
  for (int k = threadIdx.x; k < words; k += blockDim.x) {
    const int64_t v = vb + 2 * k;
    const int32_t r0 = rp[v], r1 = rp[v + 1], r2 = 2 * k + 1 < n ? rp[v + 2] : r1;
    const uint32_t d0 = (uint32_t)min(r1 - r0, 0x7FFF);
    const uint32_t d1 = 2 * k + 1 < n ? (uint32_t)min(r2 - r1, 0x7FFF) : 0xFFFFu;
    sdeg[k] = d0 | (d1 << 16);
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) prio[vb + i] = mg;
  if (threadIdx.x < 3) {
    sh.cnt[threadIdx.x] = sh.hcnt[threadIdx.x] = 0;
    sh.mn[threadIdx.x] = 0xFFFFFFFFu;
  }
  __syncthreads();
  int head = 0, level = 0, last_level = 0;  // order[0, head) has been processed
  uint32_t priority = 0, ph = 0;            // ph: this phase's slot
  auto next_phase = [&]() { ph = ph == 2 ? 0 : ph + 1; };
  auto reset_next = [&]() {
    if (threadIdx.x == 0) {
      const uint32_t q = ph == 2 ? 0 : ph + 1;
      sh.cnt[q] = sh.hcnt[q] = 0;
      sh.mn[q] = 0xFFFFFFFFu;
    }
  };
  while (head < n) {
    // scan: the remaining vertices of degree `level` are the level's first round
    reset_next();
    uint32_t mn = 0xFFFFFFFFu;
    for (int k0 = 32 * w; k0 < words; k0 += 32 * nw) {
      const int k = k0 + lane;
      const uint32_t x = k < words ? sdeg[k] : 0xFFFFFFFFu;
      const uint32_t d0 = x & 0xFFFFu, d1 = x >> 16;
      // == level: a remaining vertex never has less
      const bool t0 = d0 < SEG_GONE && d0 <= (uint32_t)level;
      const bool t1 = d1 < SEG_GONE && d1 <= (uint32_t)level;
      if (!t0 && d0 < SEG_GONE) mn = min(mn, d0);
      if (!t1 && d1 < SEG_GONE) mn = min(mn, d1);
      const uint32_t m0 = __ballot_sync(MCE_FULL, t0), m1 = __ballot_sync(MCE_FULL, t1);
      if (m0 | m1) {
        if (t0 || t1) sdeg[k] = x | (t0 ? SEG_GONE : 0u) | (t1 ? SEG_GONE << 16 : 0u);
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&sh.cnt[ph], (uint32_t)(__popc(m0) + __popc(m1)));
        base = __shfl_sync(MCE_FULL, base, 0) + (uint32_t)head;
        // below n, unless repeated or one-sided arcs wore a removed vertex's mark down
        const uint32_t p0 = base + __popc(m0 & lt), p1 = base + __popc(m0) + __popc(m1 & lt);
        if (t0 && p0 < (uint32_t)n) order[p0] = (uint16_t)(2 * k);
        if (t1 && p1 < (uint32_t)n) order[p1] = (uint16_t)(2 * k + 1);
      }
    }
    mn = __reduce_min_sync(MCE_FULL, mn);
    if (lane == 0 && mn != 0xFFFFFFFFu) atomicMin(&sh.mn[ph], mn);
    __syncthreads();
    int cnt = min((int)sh.cnt[ph], n - head);
    const uint32_t lowest = sh.mn[ph];
    next_phase();
    if (cnt == 0) {  // no vertex at this level: go to the lowest remaining degree
      if (lowest == 0xFFFFFFFFu) break;
      level = (int)lowest;
      continue;
    }
    last_level = level;
    while (cnt > 0) {
      reset_next();
      const int end = head + cnt;  // this round's slice; the next one's begins here
      const bool last = end >= n;  // the final round keeps priority m_g
      for (int i = head + (int)threadIdx.x; i < end; i += blockDim.x) {
        const int v = order[i];
        core[vb + v] = level;
        if (!last) prio[vb + v] = priority;
      }
      if (last) {
        head = end;
        break;
      }
      // lower the degree of neighbour c (in: this lane has one); a vertex whose
      // degree falls to `level` joins the next round
      auto lower = [&](bool in, int32_t c) {
        const uint32_t u = (uint32_t)(c - (int32_t)vb);
        bool p = false;
        if (in && u < (uint32_t)n) {  // else: not this graph's vertex (invalid input)
          const uint32_t s = (u & 1u) * 16u;
          p = ((atomicSub(&sdeg[u >> 1], 1u << s) >> s) & 0xFFFFu) == (uint32_t)level + 1u;
          if (p) atomicOr(&sdeg[u >> 1], SEG_GONE << s);
        }
        const uint32_t mask = __ballot_sync(MCE_FULL, p);
        if (mask) {
          uint32_t base = 0;
          if (lane == 0) base = atomicAdd(&sh.cnt[ph], (uint32_t)__popc(mask));
          base = __shfl_sync(MCE_FULL, base, 0) + (uint32_t)(end + __popc(mask & lt));
          if (p && base < (uint32_t)n) order[base] = (uint16_t)u;
        }
      };
      const int g = min(SEG_GROUP, (cnt + nw - 1) / nw);  // spread small rounds over the warps
      for (int i0 = head + w * g; i0 < end; i0 += nw * g) {
        const int rows = min(g, end - i0);
        int32_t b = 0, e = 0;
        if (lane < rows) {
          const int v = order[i0 + lane];
          b = rp[vb + v];
          e = rp[vb + v + 1];
          if (e - b > SEG_HEAVY) {
            const uint32_t hp = atomicAdd(&sh.hcnt[ph], 1u);
            if (hp < (uint32_t)SEG_HEAVY_MAX) {
              sh.heavy[hp] = (uint16_t)v;
              e = b;
            }
          }
        }
        int32_t U[SEG_GROUP];
#pragma unroll
        for (int k = 0; k < SEG_GROUP; ++k) {  // every row's first window
          const int32_t j = __shfl_sync(MCE_FULL, b, k) + lane;
          const bool in = k < rows && j < __shfl_sync(MCE_FULL, e, k);
          U[k] = in ? col[j] : -1;
        }
#pragma unroll
        for (int k = 0; k < SEG_GROUP; ++k)
          if (k < rows) lower(U[k] >= 0, U[k]);
        for (uint32_t lm = __ballot_sync(MCE_FULL, e - b > 32); lm; lm &= lm - 1) {
          const int k = __ffs(lm) - 1;  // the rest of rows longer than a window
          const int32_t bk = __shfl_sync(MCE_FULL, b, k), ek = __shfl_sync(MCE_FULL, e, k);
          for (int32_t j0 = bk + 32; j0 < ek; j0 += 128) {
            int32_t c[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) c[q] = j0 + 32 * q + lane < ek ? col[j0 + 32 * q + lane] : -1;
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (j0 + 32 * q < ek) lower(c[q] >= 0, c[q]);
          }
        }
      }
      __syncthreads();
      const int hc = min((int)sh.hcnt[ph], SEG_HEAVY_MAX);
      if (hc > 0) {
        for (int h = 0; h < hc; ++h) {
          const int64_t v = vb + sh.heavy[h];
          const int32_t bk = rp[v], ek = rp[v + 1];
          for (int32_t j0 = bk + 32 * w; j0 < ek; j0 += 32 * nw) {
            const int32_t c = j0 + lane < ek ? col[j0 + lane] : -1;
            lower(c >= 0, c);
          }
        }
        __syncthreads();
      }
      head = end;
      cnt = min((int)sh.cnt[ph], n - head);
      next_phase();
      ++priority;
    }
    ++level;
  }
  if (threadIdx.x == 0) {
    atomicMax(&ctl->rounds, priority);
    atomicMax(&ctl->degeneracy, last_level);
  }
  __syncthreads();
}

// A single graph of at most SEG_SMEM_N vertices and PEEL_ONE_M arcs: one
// block, whose rounds cost a block barrier each instead of a grid barrier.
// One block against the grid: ER n = 200, 1,000 and 10,000 (degree 10 to 20)
// 0.027, 0.053 and 0.195 ms against 0.094, 0.231 and 0.251; ER n = 16,384 of
// 492 k and 982 k arcs 0.383 and 0.494 against 0.329 and 0.400; with many
// rounds (R-MAT 13 of 204 k arcs, BA of 1.02 M) 0.437 and 0.941 against 1.359
// and 1.528: the limit lies between.
constexpr int PEEL_ONE_BLOCK = 1024;
constexpr int64_t PEEL_ONE_M = 1 << 19;
__global__ void __launch_bounds__(PEEL_ONE_BLOCK)
    peel_one_kernel(int n, uint32_t m, const int32_t *__restrict__ rp,
                    const int32_t *__restrict__ col, int32_t *core, uint32_t *prio, PeelCtl *ctl) {
  __shared__ SegShared sh;
  extern __shared__ uint32_t seg_dyn[];
  const int n2 = (n + 1) & ~1;
  peel_graph_smem(rp, col, core, prio, 0, n, m, seg_dyn, (uint16_t *)(seg_dyn + n2 / 2), sh, ctl);
}

__global__ void __launch_bounds__(SEG_BLOCK)
    peel_segments_kernel(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                         int32_t *deg, int32_t *core, uint32_t *prio, int32_t *fa, int32_t *fb,
                         const int64_t *__restrict__ vtx_off, const int64_t *__restrict__ arc_off,
                         const int32_t *__restrict__ order, int32_t G, PeelCtl *ctl,
                         uint32_t *next, int smem_n) {
  __shared__ SegShared sh;
  extern __shared__ uint32_t seg_dyn[];  // smem_n / 2 degree words, then smem_n ids
  uint32_t *sdeg = seg_dyn;
  uint16_t *vord = (uint16_t *)(seg_dyn + smem_n / 2);
  const int lane = (int)lane_id(), w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (;;) {
    if (threadIdx.x == 0) sh.g = atomicAdd(next, 1u);  // next graph, largest first
    __syncthreads();
    const uint32_t gi = sh.g;
    if (gi >= (uint32_t)G) break;
    const int32_t gr = order[gi];
    const int64_t vb = vtx_off[gr] - gr, n = vtx_off[gr + 1] - vtx_off[gr] - 1;
    const uint32_t mg = (uint32_t)(arc_off[gr + 1] - arc_off[gr]);
    if (n <= smem_n) {
      peel_graph_smem(rp, col, core, prio, vb, (int)n, mg, sdeg, vord, sh, ctl);
      continue;
    }
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
      const int64_t v = vb + i;
      deg[v] = rp[v + 1] - rp[v];
      core[v] = -1;
      prio[v] = mg;
    }
    if (threadIdx.x == 0) {
      sh.todo = (int32_t)n;
      sh.level = 0;
    }
    __syncthreads();
    int32_t *F0 = fa + vb, *G0 = fb + vb;  // this graph's slice of the frontier buffers
    uint32_t priority = 0;
    int last_level = -1;
    while (sh.todo > 0) {
      const int level = sh.level;
      __syncthreads();
      if (threadIdx.x == 0) {
        sh.fcnt = 0;
        sh.minv = INT_MAX;
      }
      __syncthreads();
      for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const int64_t v = vb + i;
        if (core[v] == -1) {
          if (deg[v] <= level) {  // == level: a remaining vertex never has less
            core[v] = level;
            F0[atomicAdd(&sh.fcnt, 1)] = (int32_t)v;
          } else {
            atomicMin(&sh.minv, deg[v]);
          }
        }
      }
      __syncthreads();
      if (sh.fcnt == 0) {  // no vertex at this level: go to the lowest remaining degree
        __syncthreads();
        if (threadIdx.x == 0) sh.level = sh.minv;
        __syncthreads();
        continue;
      }
      int32_t *F = F0, *Gq = G0;
      for (;;) {
        const int cnt = sh.fcnt;
        __syncthreads();
        if (cnt == 0) break;
        last_level = level;
        if (threadIdx.x == 0) {
          sh.todo -= cnt;
          sh.ncnt = 0;
        }
        __syncthreads();
        if (sh.todo == 0) break;  // the final round keeps priority m_g
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) prio[F[i]] = priority;
        for (int i = w; i < cnt; i += nw) {
          const int32_t v = F[i];
          for (int32_t j = rp[v] + lane; j < rp[v + 1]; j += 32) {
            const int32_t u = col[j];
            if (*(volatile int32_t *)&core[u] == -1) {
              const int old = atomicSub(&deg[u], 1);
              if (old == level + 1) {
                core[u] = level;
                Gq[atomicAdd(&sh.ncnt, 1)] = u;
              }
            }
          }
        }
        __syncthreads();
        if (threadIdx.x == 0) sh.fcnt = sh.ncnt;
        int32_t *t = F;
        F = Gq;
        Gq = t;
        ++priority;
        __syncthreads();
      }
      if (threadIdx.x == 0) sh.level = level + 1;
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      atomicMax(&ctl->rounds, priority);
      atomicMax(&ctl->degeneracy, last_level < 0 ? 0 : last_level);
    }
    __syncthreads();
  }
}

}  // namespace

// 128 threads per small graph (at most PEEL_SMALL_N vertices) and 256 per
// middle one (at most PEEL_MID_N): blocks that need 8 or 32 KB of shared
// memory, so many more of them fit on an SM than of the 512-thread blocks
// with room for 16,384 vertices.
constexpr int SEG_SMALL_BLOCK = 128, SEG_MID_BLOCK = 256;

int peel_segments_launch(const PeelArgs &a, const int64_t *vtx_off, const int64_t *arc_off,
                         const int32_t *order, int32_t G, int32_t g_big, int32_t g_mid,
                         cudaStream_t s, const PeelSide &ps, int *launches, int part,
                         int64_t max_n) {
  int dev = 0, sms = 0;
  MCE_CUDA(cudaGetDevice(&dev));
  MCE_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // set on every call: the attribute belongs to the current device
  MCE_CUDA(cudaFuncSetAttribute(peel_segments_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                SEG_SMEM_N * 4));
  if (part >= MAX_BATCH_PARTS) return MCE_EINVAL;
  if (g_big < 0 || g_mid < 0 || g_big + g_mid > G) return MCE_EINVAL;
  PeelCtl *ctl = (PeelCtl *)a.ctl;
  if (part < 0) MCE_CUDA(cudaMemsetAsync(ctl, 0, sizeof(PeelCtl), s));
  // one launch: `cnt` graphs of order[first..], blocks of `threads`, shared
  // state for graphs of up to `nmax` vertices
  auto launch = [&](int32_t first, int32_t cnt, int threads, int64_t nmax, uint32_t *next,
                    cudaStream_t st) -> int {
    if (cnt <= 0) return MCE_OK;
    const int smem_n = nmax <= 0 ? 0 : (int)((std::min<int64_t>(nmax, SEG_SMEM_N) + 1) & ~1);
    const size_t smem = (size_t)smem_n * 4;  // 2 bytes of degree + 2 of order per vertex
    int per_sm = 0;
    MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, peel_segments_kernel, threads,
                                                           smem));
    if (per_sm < 1) return MCE_ECUDA;
    int blocks = sms * per_sm;
    if (blocks > cnt) blocks = cnt;
    peel_segments_kernel<<<blocks, threads, smem, st>>>(a.rp, a.col, a.deg, a.core, a.prio,
                                                        a.front0, a.front1, vtx_off, arc_off,
                                                        order + first, cnt, ctl, next, smem_n);
    MCE_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
    return MCE_OK;
  };
  const bool p0 = part < 0;
  const int32_t g_small = G - g_big - g_mid;
  const bool fork = ps.side[0] && ps.side[1] && ps.fork && ps.join[0] && ps.join[1] &&
                    (g_mid > 0 || g_small > 0);
  if (fork) {
    MCE_CUDA(cudaEventRecord(ps.fork, s));
    MCE_CUDA(cudaStreamWaitEvent(ps.side[0], ps.fork, 0));
    MCE_CUDA(cudaStreamWaitEvent(ps.side[1], ps.fork, 0));
  }
  int rc = launch(0, g_big, SEG_BLOCK, max_n, p0 ? &ctl->seg_next : &ctl->seg_part[part], s);
  if (rc) return rc;
  rc = launch(g_big, g_mid, SEG_MID_BLOCK, std::min<int64_t>(max_n, PEEL_MID_N),
              p0 ? &ctl->seg_mid_next : &ctl->seg_mid_part[part], fork ? ps.side[0] : s);
  if (rc) return rc;
  rc = launch(g_big + g_mid, g_small, SEG_SMALL_BLOCK, std::min<int64_t>(max_n, PEEL_SMALL_N),
              p0 ? &ctl->seg_small_next : &ctl->seg_small_part[part], fork ? ps.side[1] : s);
  if (rc) return rc;
  if (fork) {
    MCE_CUDA(cudaEventRecord(ps.join[0], ps.side[0]));
    MCE_CUDA(cudaEventRecord(ps.join[1], ps.side[1]));
    MCE_CUDA(cudaStreamWaitEvent(s, ps.join[0], 0));
    MCE_CUDA(cudaStreamWaitEvent(s, ps.join[1], 0));
  }
  return MCE_OK;
}

size_t peel_ctl_bytes() { return sizeof(PeelCtl); }

int peel_launch(const PeelArgs &a, cudaStream_t s, int *launches) {
  int dev = 0, sms = 0, per_sm = 0, coop = 0;
  if (a.n <= SEG_SMEM_N && a.m <= PEEL_ONE_M && a.solo_max == 0) {
    const size_t smem = (size_t)((a.n + 1) & ~(int64_t)1) * 4;
    // set on every call: the attribute belongs to the current device
    MCE_CUDA(cudaFuncSetAttribute(peel_one_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  SEG_SMEM_N * 4));
    MCE_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(PeelCtl), s));
    peel_one_kernel<<<1, PEEL_ONE_BLOCK, smem, s>>>((int)a.n, (uint32_t)a.m, a.rp, a.col, a.core,
                                                    a.prio, (PeelCtl *)a.ctl);
    MCE_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
    return MCE_OK;
  }
  MCE_CUDA(cudaGetDevice(&dev));
  MCE_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MCE_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  if (!coop) return MCE_ENODEV;
  MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, peel_kernel, PEEL_BLOCK, 0));
  if (per_sm < 1) return MCE_ECUDA;
  per_sm = 1;
  int32_t n = (int32_t)a.n;
  uint32_t m = (uint32_t)a.m;
  PeelCtl *ctl = (PeelCtl *)a.ctl;
  MCE_CUDA(cudaMemsetAsync(ctl, 0, sizeof(PeelCtl), s));
  uint64_t limit = a.wait_limit_ns;
  uint32_t solo_max = a.solo_max;
  void *args[] = {(void *)&n,        (void *)&m,        (void *)&a.rp,     (void *)&a.col,
                  (void *)&a.deg,    (void *)&a.core,   (void *)&a.prio,   (void *)&a.alistA,
                  (void *)&a.alistB, (void *)&a.front0, (void *)&a.front1, (void *)&a.front2,
                  (void *)&a.hb0,    (void *)&a.hb1,    (void *)&a.hb2,
                  (void *)&ctl,      (void *)&limit,    (void *)&solo_max};
  MCE_CUDA(cudaLaunchCooperativeKernel((void *)peel_kernel, dim3(sms * per_sm), dim3(PEEL_BLOCK),
                                       args, 0, s));
  if (launches) *launches += 1;
  return MCE_OK;
}

int peel_read(const void *ctl_dev, int32_t *degeneracy, uint32_t *err, uint32_t *rounds,
              uint32_t *solo_sections, cudaStream_t s, double *phase_ms) {
  PeelCtl h;
  MCE_CUDA(cudaMemcpyAsync(&h, ctl_dev, sizeof(PeelCtl), cudaMemcpyDeviceToHost, s));
  MCE_CUDA(cudaStreamSynchronize(s));
  if (degeneracy) *degeneracy = h.degeneracy;
  if (err) *err = h.err;
  if (rounds) *rounds = h.rounds;
  if (solo_sections) *solo_sections = h.solo_sections;
  if (phase_ms) {
    phase_ms[0] = h.t_scan * 1e-6;
    phase_ms[1] = h.t_round * 1e-6;
    phase_ms[2] = h.t_wait * 1e-6;
  }
  return MCE_OK;
}

}  // namespace mce
