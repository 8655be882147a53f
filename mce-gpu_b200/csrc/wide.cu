// The search of roots with 65 to 256 later neighbours, one warp per root.
//
// The trees of such roots are most of the work on graphs with a dense core.
// The sets of a node (P, X, branches, chosen) are W 64-bit words that every
// lane holds; the adjacency rows (enc.cu) lie in shared memory, and lane i
// scores candidates i, i + 32, ...: the words of a candidate's row are one
// vector load, groups of 32 without a candidate are skipped, and one
// reduction picks the pivot (best score, lowest index).  The frames lie in
// shared memory as far as WIDE_FRAMES reach, then in the warp's slab.
//
// What bounds it: instruction issue per node (61 % of the slots on R-MAT 13, 5
// warps per scheduler at 94 registers).  bk_mem_kernel keeps its frames
// in global memory, loads row words one by one and walks every leaf; with this
// engine in its place a count of R-MAT 13 went from 28.5 to 12.5 ms and one of
// R-MAT 12 with -i px from 6.05 to 3.55.  For 33 to 64 later neighbours the
// register engine stays: this code with one word per set took 5 % longer.
//
// The tree and its tallies are those of bk_mem_kernel, which takes the wider
// roots and the logging, listing and edge-rooted variants; what differs is
// how a node is done.  Branches without a neighbour in P are settled together
// (reg_tree's rule), and a long list of earlier-neighbour rows keeps only the
// rows containing the chosen set on the way down.
#include <climits>

#include "common.cuh"
#include "engine.cuh"
#include "kernels.h"
#include "queue.cuh"

namespace mce {

namespace {

constexpr int W_BLOCK = 128;      // 4 warps
constexpr int WIDE_FRAMES = 20;   // frames per warp in shared memory

template <int W>
struct WSet {
  u64 w[W];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int j = 0; j < W; ++j) w[j] = 0;
  }
  __device__ __forceinline__ bool any() const {
    u64 x = 0;
#pragma unroll
    for (int j = 0; j < W; ++j) x |= w[j];
    return x != 0;
  }
  __device__ __forceinline__ int count() const {
    int c = 0;
#pragma unroll
    for (int j = 0; j < W; ++j) c += __popcll(w[j]);
    return c;
  }
  __device__ __forceinline__ int lowest() const {  // of a non-empty set
    int v = 0;
#pragma unroll
    for (int j = W - 1; j >= 0; --j)
      if (w[j]) v = 64 * j + __ffsll((long long)w[j]) - 1;
    return v;
  }
  // the 32 bits that start at 32 k
  __device__ __forceinline__ uint32_t half(int k) const { return (uint32_t)(w[k >> 1] >> (32 * (k & 1))); }
  __device__ __forceinline__ void set_half(int k, uint32_t m) { w[k >> 1] |= (u64)m << (32 * (k & 1)); }
};

template <int W>
__device__ __forceinline__ u64 bit_word(int v, int j) {  // word j of {v}
  return (v >> 6) == j ? 1ull << (v & 63) : 0ull;
}
template <int W>
__device__ __forceinline__ u64 low_word(int v, int j) {  // word j of {0 .. v - 1}
  const int s = v - 64 * j;
  return s >= 64 ? ~0ull : s <= 0 ? 0ull : (1ull << s) - 1ull;
}

template <int W>
struct WSmem {
  alignas(16) u64 rows[64 * W][W];
  alignas(16) u64 xl0[32][W];
  u64 stk[WIDE_FRAMES][5 * W + 1];  // P, X, branches, settled leaves, chosen; list start and length
};

// A task of this engine: the root, then P, X and the chosen set, W words each.
// Its size does not depend on the graph's widest root (bk_mem_kernel's does),
// so that a lane of the taker holds one word.
template <int W>
constexpr uint32_t wide_task_words() {
  static_assert(1 + 3 * W <= WIDE_TASK_WORDS && WIDE_TASK_WORDS <= 32, "one word per lane");
  return 1 + 3 * W;
}

// Slab of a warp, in words: the frames past the shared ones, then the lists
// of earlier-neighbour rows (xcap rows).
template <int W>
constexpr size_t deep_words() {
  return (size_t)(64 * W) * (5 * W + 1);
}

struct WRoot {
  int32_t r = -1;
  int d = 0, u = 0, Wr = 0;  // later and earlier neighbours, words per row as built
  const u64 *xr = nullptr;   // the earlier neighbours' rows
};

template <int W, bool XP>
__device__ void w_tree(const BKArgs &a, WSmem<W> &sm, u64 *slab, const WRoot &rt, WSet<W> Pc, WSet<W> Xc, WSet<W> Sc, u64 &h0, u64 &h1, u64 &nodes, u64 &cnt) {
  const int lane = (int)lane_id();
  const uint32_t lt = (1u << lane) - 1u;
  const bool share = a.q.hdr != nullptr;
  const int nX = rt.u;
  u64 *const xl = slab + deep_words<W>();
  auto frame = [&](int f) { return f < WIDE_FRAMES ? sm.stk[f] : slab + (size_t)(f - WIDE_FRAMES) * (5 * W + 1); };
  // row i of the current list: lb < 0: the first 32 in xl0, the rest in xl
  int lb = -1, nL = 0;
  auto lrow = [&](int i) {
    const u64 *p = lb < 0 ? (i < 32 ? sm.xl0[i] : xl + (size_t)i * W) : xl + (size_t)(lb + i) * W;
    WSet<W> row;
#pragma unroll
    for (int j = 0; j < W; ++j) row.w[j] = p[j];
    return row;
  };
  auto xrow = [&](int i) {  // earlier-neighbour row i as built (rt.Wr words)
    WSet<W> row;
#pragma unroll
    for (int j = 0; j < W; ++j) row.w[j] = j < rt.Wr ? rt.xr[(size_t)i * rt.Wr + j] : 0ull;
    return row;
  };
  auto has = [&](const WSet<W> &row, const WSet<W> &s) {
    u64 miss = 0;
#pragma unroll
    for (int j = 0; j < W; ++j) miss |= s.w[j] & ~row.w[j];
    return miss == 0;
  };
  // the list of the rows of xr that contain s
  auto filter = [&](const WSet<W> &s) {
    __syncwarp();
    lb = -1;
    nL = 0;
    for (int i0 = 0; i0 < nX; i0 += 32) {
      const int i = i0 + lane;
      WSet<W> row;
      bool h = false;
      if (i < nX) {
        row = xrow(i);
        h = has(row, s);
      }
      const uint32_t m = __ballot_sync(MCE_FULL, h);
      if (h) {
        const int at = nL + __popc(m & lt);
        u64 *o = at < 32 ? sm.xl0[at] : xl + (size_t)at * W;
#pragma unroll
        for (int j = 0; j < W; ++j) o[j] = row.w[j];
      }
      nL += __popc(m);
    }
    __syncwarp();
  };
  auto covered = [&](const WSet<W> &s, bool root) {
    const int n = root ? nX : nL;
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int i = i0 + lane;
      if (__any_sync(MCE_FULL, i < n && has(root ? xrow(i) : lrow(i), s))) return true;
    }
    return false;
  };
  auto leaf = [&](int bin, u64 k) {  // k cliques of bin + 2 vertices
    cnt += k;
    if (bin < 64) {
      if (lane == (bin & 31)) {
        if (bin < 32)
          h0 += k;
        else
          h1 += k;
      }
    } else if (lane == 0) {
      atomicAdd(&a.hist[bin + 2], k);
    }
  };
  int lvl = Sc.count();           // vertices chosen above the node to enter
  const bool per_branch = lvl == 0;
  if (!per_branch && nX > 0) filter(Sc);
  WSet<W> P, X, B, Lp, S;
  P.clear();
  X.clear();
  B.clear();
  Lp.clear();
  S.clear();
  int sp = 0, recheck = 0, cl = lvl;  // cl: vertices chosen above the current frame
  bool want = false, start = true;
  for (;;) {
    if (!start) {
      if (!B.any()) {
        if (sp == 0) break;
        --sp;
        const u64 *f = frame(sp);
#pragma unroll
        for (int j = 0; j < W; ++j) {
          P.w[j] = f[j];
          X.w[j] = f[W + j];
          B.w[j] = f[2 * W + j];
          Lp.w[j] = f[3 * W + j];
          S.w[j] = f[4 * W + j];
        }
        const u64 l = f[5 * W];
        lb = (int)(uint32_t)(l >> 32);
        nL = (int)(uint32_t)l;
        cl = S.count();
      }
      const int v = B.lowest();
      const u64 *rv = sm.rows[v];
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const u64 vb = bit_word<W>(v, j), mv = Lp.w[j] & low_word<W>(v, j);
        B.w[j] &= ~vb;
        P.w[j] &= ~mv;  // the settled leaves before v have left P for X
        X.w[j] |= mv;
        Lp.w[j] &= ~mv;
        const u64 row = rv[j];
        Pc.w[j] = P.w[j] & row;
        Xc.w[j] = X.w[j] & row;
        Sc.w[j] = S.w[j] | vb;
        P.w[j] &= ~vb;
        X.w[j] |= vb;
      }
      ++nodes;
      if (cl == 0 && nX > 0) filter(Sc);  // earlier neighbours adjacent to v
      lvl = cl + 1;
      if (!Pc.any()) {  // test_maximality (mce/mce_utils.cuh:507-524)
        if (!Xc.any() && !covered(Sc, false)) leaf(lvl - 1, 1);
        continue;
      }
    }
    // enter (Pc, Xc, Sc): pivot over P' | X' (:366-402)
    const int pc = Pc.count();
    int key = 0;
    uint32_t vote = 0, iso = 0;  // vote bit 0: an X' vertex covers P'; bit 1: P' is not a clique
#pragma unroll
    for (int k = 0; k < 2 * W; ++k) {
      const uint32_t pw = Pc.half(k), xw = Xc.half(k);
      if ((pw | xw) == 0) continue;
      if (((pw | xw) >> lane) & 1u) {
        const u64 *row = sm.rows[32 * k + lane];
        int s = 0;
#pragma unroll
        for (int j = 0; j < W; ++j) s += __popcll(Pc.w[j] & row[j]);
        key = max(key, ((s + 1) << 8) | (255 - (32 * k + lane)));
        if ((pw >> lane) & 1u) {
          if (s != pc - 1) vote |= 2u;
          if (s == 0) iso |= 1u << k;
        } else if (s == pc) {
          vote |= 1u;
        }
      }
    }
    vote = __reduce_or_sync(MCE_FULL, vote);
    if ((vote & 1u) || pc == 0) {
      if (start) break;
      continue;
    }
    if (vote == 0) {  // P' is a clique: one path of pc nodes ends in S' | P'
      WSet<W> U;
#pragma unroll
      for (int j = 0; j < W; ++j) U.w[j] = Sc.w[j] | Pc.w[j];
      const bool cov = covered(U, lvl == 0);
      if (!(XP && cov)) nodes += (u64)pc;  // -i px prunes where a row covers P'
      if (!cov) leaf(lvl + pc - 1, 1);
      if (start) break;
      continue;
    }
    key = (int)__reduce_max_sync(MCE_FULL, (unsigned)key);
    const u64 *prow = sm.rows[255 - (key & 255)];
    WSet<W> piv;
#pragma unroll
    for (int j = 0; j < W; ++j) piv.w[j] = prow[j];
    if constexpr (XP) {  // earlier neighbours adjacent to the whole chosen set (:404-472)
      const bool root = lvl == 0;
      const int n = root ? nX : nL;
      int best = 0;
      uint32_t bid = 0xFFFFFFFFu;
      bool el = false;
      for (int i = lane; i < n; i += 32) {
        const WSet<W> row = root ? xrow(i) : lrow(i);
        if (!has(row, Sc)) continue;
        int s = 0;
#pragma unroll
        for (int j = 0; j < W; ++j) s += __popcll(Pc.w[j] & row.w[j]);
        el |= s == pc;
        if (s + 1 > best) {  // ids ascend within a lane: ties keep the lowest
          best = s + 1;
          bid = (uint32_t)i;
        }
      }
      if (__any_sync(MCE_FULL, el)) {
        if (start) break;
        continue;
      }
      const int mb = (int)__reduce_max_sync(MCE_FULL, (unsigned)best);
      if (mb > (key >> 8)) {
        const int id = (int)__reduce_min_sync(MCE_FULL, best == mb ? bid : 0xFFFFFFFFu);
        piv = root ? xrow(id) : lrow(id);
      }
    }
    // hand the child to an idle warp (mce/mce_utils.cuh:872-880,1063-1113)
    if (!start && share && pc >= a.donate_min &&
        (nodes >= a.donate_after || (a.policy && a.policy[rt.r]))) {
      if (--recheck <= 0) {  // the queue state is read every 32 candidate nodes
        want = wants_task(a.q);
        recheck = 32;
      }
      if (want) {
        const int pushed = q_push(a.q, a.err, a.wait_limit_ns, [&](uint32_t k2) -> u64 {
          u64 x = (u64)(uint32_t)rt.r;
#pragma unroll
          for (int j = 0; j < W; ++j) {
            if ((int)k2 == 1 + j) x = Pc.w[j];
            if ((int)k2 == 1 + W + j) x = Xc.w[j];
            if ((int)k2 == 1 + 2 * W + j) x = Sc.w[j];
          }
          return x;
        });
        want = pushed == Q_PUSHED;
        if (pushed != Q_KEPT) continue;
      }
    }
    if (B.any()) {  // come back to the frame's other branches
      u64 *f = frame(sp);
      __syncwarp();
      if (lane == 0) {
#pragma unroll
        for (int j = 0; j < W; ++j) {
          f[j] = P.w[j];
          f[W + j] = X.w[j];
          f[2 * W + j] = B.w[j];
          f[3 * W + j] = Lp.w[j];
          f[4 * W + j] = S.w[j];
        }
        f[5 * W] = (u64)(uint32_t)lb << 32 | (u64)(uint32_t)nL;
      }
      __syncwarp();
      ++sp;
    }
    P = Pc;
    X = Xc;
    S = Sc;
    cl = lvl;
    WSet<W> Bn;
#pragma unroll
    for (int j = 0; j < W; ++j) Bn.w[j] = P.w[j] & ~piv.w[j];
    // a long list keeps only the rows containing the chosen set (:265-292); a
    // depth-0 branch's list holds exactly those already
    if (nL > 32 && lvl >= (per_branch ? 2 : 1) && !start) {
      const int top = lb < 0 ? nL : lb + nL;
      if (top + nL <= a.xcap) {
        int k = 0;
        for (int i0 = 0; i0 < nL; i0 += 32) {
          const int i = i0 + lane;
          const WSet<W> row = lrow(i < nL ? i : 0);
          const bool h = i < nL && has(row, S);
          const uint32_t m = __ballot_sync(MCE_FULL, h);
          if (h) {
            u64 *o = xl + (size_t)(top + k + __popc(m & lt)) * W;
#pragma unroll
            for (int j = 0; j < W; ++j) o[j] = row.w[j];
          }
          k += __popc(m);
        }
        __syncwarp();
        lb = top;
        nL = k;
      }
    }
    // the branches that are leaves: no neighbour in P
    Lp.clear();
#pragma unroll
    for (int k = 0; k < 2 * W; ++k) {
      if (Bn.half(k) == 0) continue;
      Lp.set_half(k, __ballot_sync(MCE_FULL, (iso >> k) & 1u) & Bn.half(k));
    }
    if (Lp.any()) {
      WSet<W> M;
      M.clear();
#pragma unroll
      for (int k = 0; k < 2 * W; ++k) {
        const uint32_t lw = Lp.half(k);
        if (lw == 0) continue;
        bool m = false;
        if ((lw >> lane) & 1u) {
          const int i = 32 * k + lane;
          const u64 *row = sm.rows[i];
          u64 x = 0;
#pragma unroll
          for (int j = 0; j < W; ++j) x |= (X.w[j] | (Bn.w[j] & low_word<W>(i, j))) & row[j];
          m = x == 0;
        }
        M.set_half(k, __ballot_sync(MCE_FULL, m));
      }
      nodes += (u64)Lp.count();
      if (M.any()) {  // minus those an earlier neighbour of the root covers
        const bool root = cl == 0;
        const int n = root ? nX : nL;
        if (n > 0) {
          WSet<W> acc;
          acc.clear();
          for (int i = lane; i < n; i += 32) {
            const WSet<W> row = root ? xrow(i) : lrow(i);
            if (has(row, S)) {
#pragma unroll
              for (int j = 0; j < W; ++j) acc.w[j] |= row.w[j];
            }
          }
#pragma unroll
          for (int j = 0; j < W; ++j) {
            const u64 c = (u64)__reduce_or_sync(MCE_FULL, (uint32_t)acc.w[j]) |
                          (u64)__reduce_or_sync(MCE_FULL, (uint32_t)(acc.w[j] >> 32)) << 32;
            M.w[j] &= ~c;
          }
        }
        const int k = M.count();
        if (k) leaf(cl, (u64)k);
      }
    }
#pragma unroll
    for (int j = 0; j < W; ++j) B.w[j] = Bn.w[j] & ~Lp.w[j];
    start = false;
  }
  __syncwarp();
}

// The root's rows into shared memory; its earlier rows stay where they are.
// False, with a status bit, for a root that is not this engine's: wider than
// its sets, without rows, or with more earlier neighbours than the lists hold.
template <int W>
__device__ __forceinline__ bool w_load(const BKArgs &a, WSmem<W> &sm, int32_t r, WRoot &rt) {
  const int lane = (int)lane_id();
  const int32_t ub = a.rp[r], sb = a.split[r];
  const int d = a.rp[r + 1] - sb, u = sb - ub;
  const u64 *rows = a.wptr[r];
  if (d > 64 * W || !rows || u > a.xcap) {
    if (lane == 0) atomicOr(a.err, d > 64 * W || !rows ? MCE_ERR_DEGREE : MCE_ERR_XROWS);
    return false;
  }
  rt.r = r;
  rt.d = d;
  rt.u = u;
  rt.Wr = (rt.d + 63) >> 6;
  rt.xr = rows + (size_t)rt.d * rt.Wr;
  __syncwarp();
  for (int i = lane; i < rt.d; i += 32) {
#pragma unroll
    for (int j = 0; j < W; ++j) sm.rows[i][j] = j < rt.Wr ? rows[(size_t)i * rt.Wr + j] : 0ull;
  }
  __syncwarp();
  return true;
}

// The roots of the wide class with more than d_lo and at most 64 W later
// neighbours.
template <int W, bool XP>
__global__ void __launch_bounds__(W_BLOCK, W == 2 ? 5 : 4) wide_kernel(BKArgs a, int d_lo, int fetch) {
  extern __shared__ __align__(16) unsigned char w_dyn[];
  WSmem<W> &sm = reinterpret_cast<WSmem<W> *>(w_dyn)[threadIdx.x >> 5];
  const int lane = (int)lane_id();
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  u64 *slab = a.slab + (size_t)gw * a.slab_words;
  const uint32_t beg = a.shape->cls_off[CLS_MEM], end = a.shape->cls_off[CLS_MEM + 1];
  const bool share = a.q.hdr != nullptr;
  u64 h0 = 0, h1 = 0, nodes = 0;
  WRoot rt;
  if (share && lane == 0) atomicAdd(&a.q.hdr->work, 1u);
  for (;;) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(&a.fetch[fetch], 1u);
    i = beg + __shfl_sync(MCE_FULL, i, 0);
    if (i >= end) break;
    const int32_t r = a.roots[i];
    const int d = a.rp[r + 1] - a.split[r];
    if (d <= d_lo || d > 64 * W) continue;  // another launch's
    if (!w_load<W>(a, sm, r, rt)) continue;
    WSet<W> P, none;
    none.clear();
#pragma unroll
    for (int j = 0; j < W; ++j) P.w[j] = low_word<W>(d, j);
    u64 nd = 0, cnt = 0;
    w_tree<W, XP>(a, sm, slab, rt, P, none, none, h0, h1, nd, cnt);
    nodes += nd;
    root_done(a, r, nd, cnt);
  }
  if (share) {
    root_phase_done(a.q);
    u64 t = 0;  // lane k: word k of the task
    idle_phase(
        a, [&](uint32_t, u64 w) { t = w; },
        [&]() {
          const int32_t r = (int32_t)__shfl_sync(MCE_FULL, t, 0);
          WSet<W> P, X, S;
#pragma unroll
          for (int j = 0; j < W; ++j) {
            P.w[j] = __shfl_sync(MCE_FULL, t, 1 + j);
            X.w[j] = __shfl_sync(MCE_FULL, t, 1 + W + j);
            S.w[j] = __shfl_sync(MCE_FULL, t, 1 + 2 * W + j);
          }
          if (r != rt.r && !w_load<W>(a, sm, r, rt)) return;
          u64 nd = 0, cnt = 0;
          w_tree<W, XP>(a, sm, slab, rt, P, X, S, h0, h1, nd, cnt);
          nodes += nd;
          root_done(a, r, nd, cnt);
        });
  }
  if (h0) atomicAdd(&a.hist[lane + 2], h0);
  if (h1) atomicAdd(&a.hist[lane + 34], h1);
  if (lane == 0 && nodes) atomicAdd(a.nodes, nodes);
}

}  // namespace

// Launches for 64 W later neighbours, W = 2 or 4: resident warps and slab
// words per warp.
template <int W, bool XP>
int w_plan(int sms, int *grid) {
  int per_sm = 0;
  MCE_CUDA(cudaFuncSetAttribute(wide_kernel<W, XP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(WSmem<W>) * (W_BLOCK / 32))));
  MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wide_kernel<W, XP>, W_BLOCK,
                                                         sizeof(WSmem<W>) * (W_BLOCK / 32)));
  *grid = sms * (per_sm > 0 ? per_sm : 1);
  return MCE_OK;
}

int wide_plan(int W, bool xp, int sms, int xcap, int *grid, size_t *slab_words) {
  const size_t deep = W == 2 ? deep_words<2>() : deep_words<4>();
  *slab_words = (deep + (size_t)W * (size_t)xcap + 31) & ~(size_t)31;
  if (W == 2) return xp ? w_plan<2, true>(sms, grid) : w_plan<2, false>(sms, grid);
  return xp ? w_plan<4, true>(sms, grid) : w_plan<4, false>(sms, grid);
}

int wide_launch(int W, bool xp, const BKArgs &args, int d_lo, int fetch, int grid, cudaStream_t s,
                int *launches) {
  BKArgs a = args;
  if (a.q.hdr) {
    a.q.words = W == 2 ? wide_task_words<2>() : wide_task_words<4>();
    if (a.q.slot < a.q.words) return MCE_EINVAL;
  }
  const size_t smem = (W == 2 ? sizeof(WSmem<2>) : sizeof(WSmem<4>)) * (W_BLOCK / 32);
  if (W == 2 && xp)
    wide_kernel<2, true><<<grid, W_BLOCK, smem, s>>>(a, d_lo, fetch);
  else if (W == 2)
    wide_kernel<2, false><<<grid, W_BLOCK, smem, s>>>(a, d_lo, fetch);
  else if (xp)
    wide_kernel<4, true><<<grid, W_BLOCK, smem, s>>>(a, d_lo, fetch);
  else
    wide_kernel<4, false><<<grid, W_BLOCK, smem, s>>>(a, d_lo, fetch);
  MCE_CUDA(cudaGetLastError());
  if (launches) *launches += 1;
  return MCE_OK;
}

}  // namespace mce
