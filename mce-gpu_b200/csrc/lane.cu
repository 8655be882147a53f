// The search of narrow roots, one lane per root.
//
// A root with few later neighbours has a small tree (7 nodes on average in
// power-law graphs) over rows of a few bits, and a warp that walks it uses a
// few of its lanes.  Here every lane walks a tree of its own: the rows
// (enc.cu) lie in shared memory, one bank per lane, the frames in local
// memory, and a node's pivot scores are a loop over its candidates.  The rows
// of the root's earlier neighbours are kept as columns - bit k of the column
// of vertex i: the k-th earlier neighbour is adjacent to i - so the set of
// earlier neighbours adjacent to everything chosen is one AND per node, and a
// leaf is maximal when it is empty.
//
// The tree, its pivots (best score, lowest index) and its tallies are those of
// the warp engine (reg_tree, engine.cuh), shortcuts included: a candidate set
// that is a clique is settled where it is found, and so are the branches
// without a neighbour in P.
//
// Lanes that have finished are refilled together once enough of them wait.  A
// root that walks more than LANE_NODES nodes hands its open frames to the
// warp engine, which can share them; so do the roots with too many earlier
// neighbours, whole.
//
// What bounds it: the latency of loading the next roots' rows (20 warps stalled
// on loads per issue, 34 % of issue slots, on 512 graphs), then the divergence
// of 32 trees (11 lanes active per instruction) and a lane's last long tree at
// the end of a launch (hence LANE_DRAIN).  On the 2.86 M roots of
// 1,024 Chung-Lu graphs the launch of up to 16 later neighbours takes 0.79 ms,
// that of up to 32 (and 64 earlier ones) 0.50 ms and the warp engine's rest
// 1.15 ms; the warp engine alone took 3.98 ms for all of them.
#include "common.cuh"
#include "kernels.h"
#include "queue.cuh"

namespace mce {

namespace {

constexpr uint32_t LANE_FULL = 0xFFFFFFFFu;
constexpr int LANE_NODES = 512;     // nodes of a root before its frames are handed over
constexpr int LANE_DRAIN = 8;       // ... or lanes left in a warp that has no roots to come
// The second launch's roots: up to MID_D later and 32 MID_K earlier neighbours.
constexpr int MID_D = 32, MID_K = 2;
constexpr int LANE_HSLOT = 8;       // copies of the histogram per warp (fewer same-word atomics)

template <int D, int K, int WARPS>
struct LaneSmem {
  uint32_t row[WARPS][D][32];
  uint32_t col[WARPS][K][D][32];
  uint32_t hist[WARPS][D][LANE_HSLOT];  // by clique size - 2
};

template <int D, int K, int WARPS, int REFILL>
__global__ void __launch_bounds__(32 * WARPS) lane_kernel(LaneArgs a) {
  __shared__ LaneSmem<D, K, WARPS> sm;
  const int lane = (int)lane_id(), wid = (int)(threadIdx.x >> 5);
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t *const row = &sm.row[wid][0][lane];
  uint32_t *const hist = &sm.hist[wid][0][lane & (LANE_HSLOT - 1)];
  auto R = [&](int i) { return row[i * 32]; };
  for (int i = lane; i < D * LANE_HSLOT; i += 32) (&sm.hist[wid][0][0])[i] = 0;
  __syncwarp();
  const uint32_t total = *a.count;
  uint32_t stk[D][5 + K];
  uint32_t P = 0, X = 0, B = 0, Lp = 0, S = 0, XA[K];  // the current frame
  uint32_t Pc = 0, Xc = 0, Sc = 0, XAc[K];             // the node to enter (pend)
  int sp = 0;
  int32_t r = 0;
  uint32_t nodes = 0, cnt = 0, cap = 0;
  unsigned long long all_nodes = 0;
  bool live = false, pend = false, more = true;
#pragma unroll
  for (int k = 0; k < K; ++k) XA[k] = XAc[k] = 0;
  auto emit = [&](int bin) {  // a maximal clique of bin + 2 vertices
    ++cnt;
    atomicAdd(&hist[bin * LANE_HSLOT], 1u);
  };
  for (;;) {
    uint32_t act = __ballot_sync(LANE_FULL, live);
    if (more && __popc(act) <= 32 - REFILL) {
      const uint32_t idle = ~act;
      uint32_t i0 = 0;
      if (lane == 0) i0 = atomicAdd(a.next, (uint32_t)__popc(idle));
      i0 = __shfl_sync(LANE_FULL, i0, 0);
      more = i0 + (uint32_t)__popc(idle) < total;
      const uint32_t i = i0 + (uint32_t)__popc(idle & lt);
      if (!live && i < total) {
        r = a.roots[i];
        const int32_t ub = a.rp[r], sb = a.split[r];
        const int d = a.rp[r + 1] - sb, u = sb - ub;
        if (d > D || u > 32 * K) {  // not for this kernel
          if (a.mid && d <= MID_D && u <= 32 * MID_K)
            a.mid[atomicAdd(a.mid_count, 1u)] = r;
          else
            a.rest[atomicAdd(a.rest_count, 1u)] = r;
        } else {
          for (int j = 0; j < d; ++j) {
            row[j * 32] = a.enc[sb + j];
#pragma unroll
            for (int k = 0; k < K; ++k) sm.col[wid][k][j][lane] = 0;
          }
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int uk = min(u - 32 * k, 32);
            XAc[k] = uk >= 32 ? 0xFFFFFFFFu : uk > 0 ? (1u << uk) - 1u : 0u;
            for (int t = 0; t < uk; ++t) {
              uint32_t w = a.enc[ub + 32 * k + t];
              while (w) {
                const int j = __ffs((int)w) - 1;
                w &= w - 1;
                sm.col[wid][k][j][lane] |= 1u << t;
              }
            }
          }
          Pc = d >= 32 ? 0xFFFFFFFFu : (1u << d) - 1u;
          Xc = Sc = 0;
          B = 0;
          sp = 0;
          nodes = cnt = 0;
          cap = LANE_NODES;
          live = pend = true;
        }
      }
      __syncwarp();
      act = __ballot_sync(LANE_FULL, live);
    }
    if (act == 0) {
      if (!more) break;
      continue;
    }
    const bool drain = !more && __popc(act) <= LANE_DRAIN;
    if (live) {
      if (!pend) {
        if (B == 0) {  // the frame is done
          if (sp == 0) {
            live = false;
            all_nodes += nodes;
            if (a.root_nodes && nodes) atomicAdd(&a.root_nodes[r], (unsigned long long)nodes);
            if (a.root_count && cnt) atomicAdd(&a.root_count[r], (unsigned long long)cnt);
            if (a.graph_count && cnt)
              atomicAdd(&a.graph_count[a.graph_of[r]], (unsigned long long)cnt);
          } else {
            --sp;
            P = stk[sp][0];
            X = stk[sp][1];
            B = stk[sp][2];
            Lp = stk[sp][3];
            S = stk[sp][4];
#pragma unroll
            for (int k = 0; k < K; ++k) XA[k] = stk[sp][5 + k];
          }
        }
        if (live && (nodes > cap || (drain && cap == LANE_NODES))) {  // hand the open frames to the warp engine
          const uint32_t at = atomicAdd(a.resume_count, (uint32_t)sp + 1u);
          if (at + (uint32_t)sp + 1u <= RESUME_CAP) {
            for (int f = 0; f <= sp; ++f) {
              uint32_t *o = a.resume + (size_t)(at + f) * RESUME_WORDS;
              const bool top = f == sp;
              o[0] = (uint32_t)r;
              o[1] = top ? P : stk[f][0];
              o[2] = top ? X : stk[f][1];
              o[3] = top ? S : stk[f][4];
              o[4] = top ? B : stk[f][2];
              o[5] = top ? Lp : stk[f][3];
            }
            sp = 0;
            B = 0;
            all_nodes += nodes;
            if (a.root_nodes && nodes) atomicAdd(&a.root_nodes[r], (unsigned long long)nodes);
            if (a.root_count && cnt) atomicAdd(&a.root_count[r], (unsigned long long)cnt);
            if (a.graph_count && cnt)
              atomicAdd(&a.graph_count[a.graph_of[r]], (unsigned long long)cnt);
            live = false;
          } else {  // no room: the slots stay unused (marked), the lane goes on
            for (uint32_t f = at; f < at + (uint32_t)sp + 1u && f < RESUME_CAP; ++f)
              a.resume[(size_t)f * RESUME_WORDS] = 0xFFFFFFFFu;
            cap = 0xFFFFFFFFu;
          }
        }
        if (live) {  // branch on the lowest vertex of B
          const int v = __ffs((int)B) - 1;
          const uint32_t vb = 1u << v, rv = R(v);
          B &= B - 1;
          const uint32_t mv = Lp & (vb - 1u);  // the settled leaves before v have left P for X
          P &= ~mv;
          X |= mv;
          Lp &= ~mv;
          Pc = P & rv;
          Xc = X & rv;
          Sc = S | vb;
          uint32_t out = 0;
#pragma unroll
          for (int k = 0; k < K; ++k) {
            XAc[k] = XA[k] & sm.col[wid][k][v][lane];
            out |= XAc[k];
          }
          P &= ~vb;
          X |= vb;
          ++nodes;
          pend = Pc != 0;
          if (!pend && Xc == 0 && out == 0) emit(__popc(Sc) - 1);
        }
      }
      if (pend) {  // enter (Pc, Xc, Sc)
        pend = false;
        const int pc = __popc(Pc);
        int best = -1;
        uint32_t prow = 0, iso = 0, notc = 0;
        bool cov = false;
        for (uint32_t c = Pc | Xc; c; c &= c - 1) {
          const uint32_t bit = c & (0u - c);
          const uint32_t ru = R(__ffs((int)c) - 1);
          const int s = __popc(Pc & ru);
          if (s > best) {  // ascending index: ties keep the lowest
            best = s;
            prow = ru;
          }
          if (Xc & bit) {
            cov |= s == pc;
          } else {
            notc |= (uint32_t)(s != pc - 1);
            if (s == 0) iso |= bit;
          }
        }
        if (!cov) {
          if (!notc) {  // P' is a clique: one path of pc nodes ends in S' | P'
            uint32_t out = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
              uint32_t x = XAc[k];
              for (uint32_t c = Pc; c && x; c &= c - 1) x &= sm.col[wid][k][__ffs((int)c) - 1][lane];
              out |= x;
            }
            nodes += (uint32_t)pc;
            if (out == 0) emit(__popc(Sc) + pc - 1);
          } else {
            if (B) {  // come back to the frame's other branches
              stk[sp][0] = P;
              stk[sp][1] = X;
              stk[sp][2] = B;
              stk[sp][3] = Lp;
              stk[sp][4] = S;
#pragma unroll
              for (int k = 0; k < K; ++k) stk[sp][5 + k] = XA[k];
              ++sp;
            }
            P = Pc;
            X = Xc;
            S = Sc;
#pragma unroll
            for (int k = 0; k < K; ++k) XA[k] = XAc[k];
            const uint32_t Bn = Pc & ~prow;
            Lp = iso & Bn;
            B = Bn & ~Lp;
            nodes += (uint32_t)__popc(Lp);
            for (uint32_t c = Lp; c; c &= c - 1) {  // the branches that are leaves
              const uint32_t bit = c & (0u - c);
              const int u = __ffs((int)c) - 1;
              uint32_t out = (X | (Bn & (bit - 1u))) & R(u);
#pragma unroll
              for (int k = 0; k < K; ++k) out |= XA[k] & sm.col[wid][k][u][lane];
              if (out == 0) emit(__popc(S));
            }
          }
        }
      }
    }
  }
  __syncwarp();
  for (int b = lane; b < D; b += 32) {
    unsigned long long h = 0;
#pragma unroll
    for (int k = 0; k < LANE_HSLOT; ++k) h += sm.hist[wid][b][k];
    if (h) atomicAdd(&a.hist[b + 2], h);
  }
  for (int o = 16; o; o >>= 1) all_nodes += __shfl_down_sync(LANE_FULL, all_nodes, o);
  if (lane == 0 && all_nodes) atomicAdd(a.nodes, all_nodes);
}

// One launch: as many blocks as are resident at once, or as `roots` fill.
template <int D, int K, int WARPS, int REFILL>
int launch(const LaneArgs &a, int sms, cudaStream_t s, int *launches) {
  int per_sm = 0;
  MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &per_sm, lane_kernel<D, K, WARPS, REFILL>, 32 * WARPS, 0));
  lane_kernel<D, K, WARPS, REFILL><<<(unsigned)(sms * (per_sm > 0 ? per_sm : 1)), 32 * WARPS, 0, s>>>(a);
  MCE_CUDA(cudaGetLastError());
  if (launches) *launches += 1;
  return MCE_OK;
}

}  // namespace

int lane_launch(const BKArgs &b, const uint32_t *count, int32_t *mid, int32_t *rest,
                uint32_t *resume, LaneCtl *ctl, int sms, cudaStream_t s, int *launches) {
  MCE_CUDA(cudaMemsetAsync(ctl, 0, sizeof(LaneCtl), s));
  LaneArgs a;
  a.rp = b.rp;
  a.split = b.split;
  a.roots = b.roots;
  a.count = count;
  a.next = &ctl->next[0];
  a.enc = b.enc;
  a.hist = b.hist;
  a.nodes = b.nodes;
  a.root_nodes = b.root_nodes;
  a.root_count = b.root_count;
  a.graph_count = b.graph_count;
  a.graph_of = b.graph_of;
  a.mid = mid;
  a.rest = rest;
  a.mid_count = &ctl->mid_count;
  a.rest_count = &ctl->rest.cls_off[CLS_R32 + 1];
  a.resume = resume;
  a.resume_count = &ctl->resume_count;
  int rc = launch<16, 1, 4, 16>(a, sms, s, launches);
  if (rc) return rc;
  a.roots = mid;
  a.count = &ctl->mid_count;
  a.next = &ctl->next[1];
  a.mid = nullptr;
  return launch<MID_D, MID_K, 2, 12>(a, sms, s, launches);
}

}  // namespace mce
