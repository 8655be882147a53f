// The search's induced subgraphs, built before it for every root at once.
//
// Replaces, for the whole graph, the per-root encode of the reference
// (warp_sorted_count_and_encode_full, mce/mce_utils.cuh:90-117, run by the
// block that owns the root) and its list of earlier neighbours tested with a
// binary search per tree node (:265-292).  Let x come before v and v before w
// in the degeneracy order, all three adjacent.  One walk of v's later list
// against a hash of x's later list finds the triangle, and the triangle is
// used three times:
//   - bit w of row v (and bit v of row w) of root x's induced subgraph;
//   - bit w of the row of v's earlier neighbour x, over v's later neighbours
//     (the rows that decide whether a leaf of root v is maximal).
// So nothing walks the later lists of a root's earlier neighbours a second
// time, a hub's thousands of earlier neighbours cost no warp a serial walk,
// and a warp that takes a shared subtree reads its root's rows instead of
// building them again.
//
// Layout.  A root with at most 32 later neighbours has 32-bit words in enc,
// at its own CSR positions: enc[rp[v] + k] the row of its k-th earlier
// neighbour, enc[split[v] + i] adjacency row i.  A wider root (d later, u
// earlier neighbours) has a region of 64-bit words, W = ceil(d / 64) per row:
// wptr[v] points at its d adjacency rows, then its u earlier rows.  Rows of
// earlier neighbours keep the list's order, zero where nothing is common.
//
// What bounds it: instruction issue (77 % of the slots, L1 65 % busy on 512
// Chung-Lu graphs of 28 M arcs; on 1,024 graphs of 65 M arcs 2.1 ms for the
// narrow roots, 0.46 ms for the wide ones), most of it the lookups of list
// elements that are not in the hash - hence the bitmap before it (2.43 -> 2.08
// ms) and two windows per step.  It took the place of the search's own encode and the hub rows: the
// search of those graphs' 32-bit class 6.4 -> 4.0 ms, BA n = 1e6 5.3 -> 3.8
// ms a call, R-MAT 13 59.7 -> 29.1 ms (a taken subtree reads its rows).
#include <algorithm>

#include "common.cuh"
#include "engine.cuh"
#include "kernels.h"

namespace mce {

namespace {

constexpr int ENC_BLOCK = 256;
constexpr int ENC_WARPS = ENC_BLOCK / 32;
constexpr int ENC_SLOTS = 128;  // hash slots per warp: 4 per item
// Vertex ids below 2^26 leave five bits of a hash key for the root's place
// in the warp's group; with more vertices a warp takes one root at a time.
constexpr int ENC_ID_BITS = 26;
constexpr int ENC_LIST = 64;    // longest list walked by the flattened walk
constexpr int WIDE_BLOCK = 128;
constexpr int WIDE_SLOTS = 4096;  // hash slots of a wide root: 2 per later neighbour at least

// Per-warp scratch of a flattened walk over the lists of up to 32 items.
struct WalkSmem {
  uint32_t start[ENC_LIST + 2];  // bit e: a list starts at element e of the walk
  int2 base[32];                 // by rank among non-empty lists: {list start - offset, key bits}
  int32_t off[32];               // ... the list's first element
  uint8_t item[32];              // ... and its item
};

// A hash of ids (linear probing, -1: empty) whose most frequent answer is no:
// an element is looked up only if its bit of the keys' bitmap is set (1,024
// bits for up to 32 keys: 3 % of the others pass; null: no bitmap).
struct IdHash {
  const int32_t *hkey;
  uint32_t mask;          // slots - 1
  uint32_t shift;         // the slot is the hash's bits from here on
  const uint32_t *bits;
};

__device__ __forceinline__ uint32_t id_hash(int32_t key) { return (uint32_t)key * 0x9E3779B1u; }

// Looks two keys per lane up: the slots that hold them, or -1; a lane without
// a key passes -1.  The warp probes together until every lane's are settled: a
// loop per lane lost hits (a lane in a further probe was missed by the warp's
// next ballot and shuffles).
__device__ __forceinline__ void find2(const IdHash &t, int32_t ka, int32_t kb, int &at_a,
                                      int &at_b) {
  const uint32_t xa = id_hash(ka), xb = id_hash(kb);
  bool ca = ka != -1, cb = kb != -1;
  if (t.bits) {
    ca = ca && ((t.bits[xa >> 27] >> ((xa >> 22) & 31u)) & 1u);
    cb = cb && ((t.bits[xb >> 27] >> ((xb >> 22) & 31u)) & 1u);
  }
  at_a = at_b = -1;
  if (!__any_sync(MCE_FULL, ca || cb)) return;
  const int32_t *const hkey = t.hkey;
  const uint32_t mask = t.mask;
  uint32_t ha = (xa >> t.shift) & mask, hb = (xb >> t.shift) & mask;
  int32_t fa = ca ? hkey[ha] : -1, fb = cb ? hkey[hb] : -1;
  bool ga = ca && fa != ka && fa != -1, gb = cb && fb != kb && fb != -1;
  while (__any_sync(MCE_FULL, ga || gb)) {
    if (ga) {
      ha = (ha + 1) & mask;
      fa = hkey[ha];
      ga = fa != ka && fa != -1;
    }
    if (gb) {
      hb = (hb + 1) & mask;
      fb = hkey[hb];
      gb = fb != kb && fb != -1;
    }
  }
  if (ca && fa == ka) at_a = (int)ha;
  if (cb && fb == kb) at_b = (int)hb;
}

// Looks every element of the items' lists up (lane t holds item t: list start
// b, length len <= ENC_LIST, key bits kb) in the hash and calls hit(rank,
// slot, position) for those found.  Two windows of 32 elements are in flight;
// an element's list is found from a bitmap of list starts (rank = set bits up
// to it).
template <typename F>
__device__ __forceinline__ void walk_lists(WalkSmem &sm, const int32_t *__restrict__ cs, int32_t b,
                                           int len, int32_t kb, const IdHash &tab, F hit) {
  const int lane = (int)lane_id();
  const uint32_t lt = (1u << lane) - 1u, le = lt | (1u << lane);
  const int incl = warp_incl_scan(len);
  const int T = __shfl_sync(MCE_FULL, incl, 31);
  const int off = incl - len;
  sm.start[lane] = 0;
  sm.start[lane + 32] = 0;
  const uint32_t ne = __ballot_sync(MCE_FULL, len > 0);
  if (len > 0) {
    const int k = __popc(ne & lt);
    sm.base[k] = make_int2(b - off, kb);
    sm.off[k] = off;
    sm.item[k] = (uint8_t)lane;
  }
  __syncwarp();
  if (len > 0) atomicOr(&sm.start[off >> 5], 1u << (off & 31));
  __syncwarp();
  int before = -1;  // lists that start before the window, minus one
  for (int e0 = 0; e0 < T; e0 += 64) {
    const uint32_t m0 = sm.start[e0 >> 5], m1 = sm.start[(e0 >> 5) + 1];
    const int c0 = __popc(m0);
    const int ra = before + __popc(m0 & le), rb = before + c0 + __popc(m1 & le);
    before += c0 + __popc(m1);
    const int ea = e0 + lane, eb = ea + 32;
    const bool ia = ea < T, ib = eb < T;
    int32_t ka = -1, kb2 = -1;
    if (ia) {
      const int2 p = sm.base[ra];
      ka = cs[p.x + ea] | p.y;
    }
    if (ib) {
      const int2 p = sm.base[rb];
      kb2 = cs[p.x + eb] | p.y;
    }
    int ta, tb;
    find2(tab, ka, kb2, ta, tb);
    if (ta >= 0) hit(ra, ta, ea);
    if (tb >= 0) hit(rb, tb, eb);
    __syncwarp();
  }
  __syncwarp();
}

__device__ __forceinline__ int32_t lower_bound_g(const int32_t *__restrict__ a, int32_t len,
                                                 int32_t key) {
  int32_t lo = 0;
  while (len > 0) {
    const int32_t half = len >> 1;
    if (a[lo + half] < key) {
      lo += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return lo;
}

// The row of v's earlier neighbour x (its place in v's earlier list found by
// binary search), at most 64 bits wide.  In a CSR that is not symmetric x may
// not be there: its place past the list has no row.
__device__ __forceinline__ void put_row(const EncArgs &a, int32_t x, int32_t v, int32_t rv,
                                        int dv, int uv, uint32_t lo, uint32_t hi) {
  const int32_t pos = lower_bound_g(a.cs + rv, uv, x);
  if (pos >= uv) return;
  if (dv <= 32 && uv <= REG_XCAP_MAX) {
    a.enc[rv + pos] = lo;
  } else {
    unsigned long long *p = a.wptr[v];
    if (p) p[dv + pos] = (unsigned long long)hi << 32 | lo;
  }
}

// One item with a list longer than ENC_LIST, walked by the whole warp against
// the hash of x's later list (key bits kb): hit(slot) records the pair (this
// item, the id in the slot).  The row's words are the windows' ballots.
template <typename Hit>
__device__ __forceinline__ void long_item(const EncArgs &a, int32_t x, int32_t v, int32_t rv,
                                          int32_t sv, int32_t ev, int32_t kb, const IdHash &tab,
                                          Hit hit) {
  const int lane = (int)lane_id();
  const int dv = ev - sv, W = (dv + 63) >> 6;
  uint32_t w0 = 0, w1 = 0;  // lane k: 32-bit words k and k + 32 of the row
  for (int q = 0; q * 32 < dv; q += 2) {
    const int ja = q * 32 + lane, jb = ja + 32;
    const int32_t ka = ja < dv ? a.cs[sv + ja] | kb : -1, kc = jb < dv ? a.cs[sv + jb] | kb : -1;
    int ta, tb;
    find2(tab, ka, kc, ta, tb);
    const uint32_t ma = __ballot_sync(MCE_FULL, ta >= 0), mb = __ballot_sync(MCE_FULL, tb >= 0);
    if (ta >= 0) hit(ta);
    if (tb >= 0) hit(tb);
    __syncwarp();
    if (lane == (q & 31)) {
      if (q < 32)
        w0 = ma;
      else
        w1 = ma;
    }
    if (lane == ((q + 1) & 31)) {
      if (q + 1 < 32)
        w0 = mb;
      else
        w1 = mb;
    }
  }
  if (!__any_sync(MCE_FULL, (w0 | w1) != 0)) return;
  unsigned long long *p = a.wptr[v];
  if (!p) return;
  const int32_t pos = lower_bound_g(a.cs + rv, sv - rv, x);  // the same for every lane
  if (pos >= sv - rv) return;  // as in put_row
  uint32_t *dst = reinterpret_cast<uint32_t *>(p + ((size_t)dv + pos) * W);
  if (lane < 2 * W) dst[lane] = w0;
  if (lane + 32 < 2 * W) dst[lane + 32] = w1;
}

struct EncSmem {
  WalkSmem walk;
  int32_t hkey[ENC_SLOTS];  // the items' ids, tagged with their root's place (-1: empty) ...
  uint8_t hidx[ENC_SLOTS];  // ... and their lanes
  uint8_t first[32];        // first lane of an item's root
  uint32_t rows[32], lo[32], hi[32];
  uint32_t bits[32];        // the ids' bitmap
};

// Roots with at most 32 later neighbours.  A warp takes up to 32 of them,
// and of those as many at a time as have 32 later neighbours together: a lane
// per (root, later neighbour).  Small roots (8 later neighbours on average in
// power-law graphs) so share one set of loads, one scan and full windows.
__global__ void __launch_bounds__(ENC_BLOCK) enc_small_kernel(EncArgs a, uint32_t fetch_n) {
  __shared__ EncSmem sm_all[ENC_WARPS];
  EncSmem &sm = sm_all[threadIdx.x >> 5];
  const int lane = (int)lane_id();
  const uint32_t le = 0xFFFFFFFFu >> (31 - lane);
  const uint32_t beg = a.shape->cls_off[CLS_R32], end = a.shape->cls_off[CLS_R32 + 1];
  const bool pack = a.n <= ((int64_t)1 << ENC_ID_BITS);
  for (;;) {
    uint32_t i0 = 0;
    if (lane == 0) i0 = atomicAdd(a.next, fetch_n);
    i0 = beg + __shfl_sync(MCE_FULL, i0, 0);
    if (i0 >= end) break;
    const int nr = (int)min(fetch_n, end - i0);
    int32_t r = 0, sb = 0;
    int d = 0;
    if (lane < nr) {
      r = a.roots[i0 + lane];
      sb = a.split[r];
      d = a.rp[r + 1] - sb;
    }
    const int cum = warp_incl_scan(d);
    for (int s0 = 0; s0 < nr;) {
      const int base = s0 ? __shfl_sync(MCE_FULL, cum, s0 - 1) : 0;
      const uint32_t fit = __ballot_sync(MCE_FULL, lane >= s0 && lane < nr && cum - base <= 32);
      const int ns = pack ? __popc(fit) : 1;  // at least one: a root has 1..32
      const int I = __shfl_sync(MCE_FULL, cum, s0 + ns - 1) - base;
      const bool mine = lane >= s0 && lane < s0 + ns;
      const uint32_t starts = __reduce_or_sync(MCE_FULL, mine ? 1u << (cum - d - base) : 0u);
      const int s = s0 + __popc(starts & le) - 1;          // this item's root
      const int first = 31 - __clz(starts & le);           // ... and its first lane
      const int32_t x = __shfl_sync(MCE_FULL, r, s), xs = __shfl_sync(MCE_FULL, sb, s);
      const int dx = __shfl_sync(MCE_FULL, d, s);
      const bool item = lane < I;
      const int32_t tag = pack ? (s - s0) << ENC_ID_BITS : 0;
      const int32_t at = xs + lane - first;
      int32_t v = 0, rv = 0, sv = 0, ev = 0;
      if (item) {
        v = a.cs[at];
        rv = a.rp[v];
        sv = a.split[v];
        ev = a.rp[v + 1];
      }
      const int dv = ev - sv, uv = sv - rv;
      // one later neighbour: it has no row and no common neighbour
      const bool walked = item && dx > 1 && dv > 0;
      const bool narrow = dv <= ENC_LIST && uv <= REG_XCAP_MAX;
#pragma unroll
      for (int i = 0; i < ENC_SLOTS; i += 32) sm.hkey[i + lane] = -1;
      sm.rows[lane] = 0;
      sm.lo[lane] = 0;
      sm.hi[lane] = 0;
      sm.bits[lane] = 0;
      sm.first[lane] = (uint8_t)first;
      __syncwarp();
      if (item && dx > 1) {
        const int32_t key = v | tag;
        const uint32_t xh = id_hash(key);
        uint32_t h = xh >> 25;
        while (atomicCAS(&sm.hkey[h], -1, key) != -1) h = (h + 1) & (ENC_SLOTS - 1);
        sm.hidx[h] = (uint8_t)lane;
        atomicOr(&sm.bits[xh >> 27], 1u << ((xh >> 22) & 31u));
      }
      __syncwarp();
      const IdHash tab{sm.hkey, ENC_SLOTS - 1, 25, sm.bits};
      auto pair = [&](int t, int i) {  // items t and i of one root are adjacent
        const int f = sm.first[t];
        atomicOr(&sm.rows[t], 1u << (i - f));
        atomicOr(&sm.rows[i], 1u << (t - f));
      };
      walk_lists(sm.walk, a.cs, sv, walked && narrow ? dv : 0, tag, tab,
                 [&](int k, int h, int e) {
                   const int t = sm.walk.item[k], j = e - sm.walk.off[k];
                   pair(t, sm.hidx[h]);
                   if (j < 32)
                     atomicOr(&sm.lo[t], 1u << j);
                   else
                     atomicOr(&sm.hi[t], 1u << (j - 32));
                 });
      __syncwarp();
      if (walked && narrow && (sm.lo[lane] | sm.hi[lane]))
        put_row(a, x, v, rv, dv, uv, sm.lo[lane], sm.hi[lane]);
      for (uint32_t wm = __ballot_sync(MCE_FULL, walked && !narrow); wm; wm &= wm - 1) {
        const int t = __ffs(wm) - 1;
        const int32_t tg = __shfl_sync(MCE_FULL, tag, t);
        long_item(a, __shfl_sync(MCE_FULL, x, t), __shfl_sync(MCE_FULL, v, t),
                  __shfl_sync(MCE_FULL, rv, t), __shfl_sync(MCE_FULL, sv, t),
                  __shfl_sync(MCE_FULL, ev, t), tg, tab, [&](int h) { pair(t, sm.hidx[h]); });
      }
      __syncwarp();
      if (item) a.enc[at] = sm.rows[lane];
      __syncwarp();
      s0 += ns;
    }
  }
}

// Wider roots: a block per (root, WIDE_BLOCK of its later neighbours), a warp
// per 32 of those; the root's hash is the block's, its rows are completed
// with atomics in its region (both directions of a pair may come from
// different blocks).
struct WideSmem {
  int32_t hkey[WIDE_SLOTS];
  uint16_t hidx[WIDE_SLOTS];
  WalkSmem walk[WIDE_BLOCK / 32];
  uint32_t lo[WIDE_BLOCK], hi[WIDE_BLOCK];
};

__global__ void __launch_bounds__(WIDE_BLOCK) enc_wide_kernel(EncArgs a, uint32_t groups) {
  __shared__ WideSmem sm;
  const int lane = (int)lane_id(), w = (int)(threadIdx.x >> 5);
  const uint32_t beg = a.shape->cls_off[CLS_R64], end = a.shape->cls_off[CLS_MEM + 1];
  const uint64_t units = (uint64_t)(end - beg) * groups;
  int32_t have = -1;  // root whose hash is built
  uint32_t mask = 0;
  for (uint64_t un = blockIdx.x; un < units; un += gridDim.x) {
    const int32_t x = a.roots[beg + (uint32_t)(un / groups)];
    const int32_t sx = a.split[x];
    const int dx = a.rp[x + 1] - sx, t0 = (int)(un % groups) * WIDE_BLOCK;
    if (t0 >= dx) continue;
    if (have != x) {
      int cap = 128;
      while (cap < 4 * dx && cap < WIDE_SLOTS) cap <<= 1;
      mask = (uint32_t)cap - 1u;
      __syncthreads();
      for (int i = threadIdx.x; i < cap; i += WIDE_BLOCK) sm.hkey[i] = -1;
      __syncthreads();
      for (int i = threadIdx.x; i < dx; i += WIDE_BLOCK) {
        const int32_t id = a.cs[sx + i];
        uint32_t h = (id_hash(id) >> 16) & mask;
        while (atomicCAS(&sm.hkey[h], -1, id) != -1) h = (h + 1) & mask;
        sm.hidx[h] = (uint16_t)i;
      }
      __syncthreads();
      have = x;
    }
    unsigned long long *rows = a.wptr[x];
    const int Wx = (dx + 63) >> 6;
    const int t = t0 + (int)threadIdx.x;  // this lane's item
    const bool item = t < dx;
    int32_t v = 0, rv = 0, sv = 0, ev = 0;
    if (item) {
      v = a.cs[sx + t];
      rv = a.rp[v];
      sv = a.split[v];
      ev = a.rp[v + 1];
    }
    const int dv = ev - sv, uv = sv - rv;
    const bool narrow = dv <= ENC_LIST && uv <= REG_XCAP_MAX;
    uint32_t *lo = sm.lo + 32 * w, *hi = sm.hi + 32 * w;
    lo[lane] = 0;
    hi[lane] = 0;
    __syncwarp();
    const IdHash tab{sm.hkey, mask, 16, nullptr};
    auto pair = [&](int j, int i) {  // later neighbours j and i of x are adjacent
      if (!rows) return;             // no region: the search builds this root's rows
      atomicOr(&rows[(size_t)j * Wx + (i >> 6)], 1ull << (i & 63));
      atomicOr(&rows[(size_t)i * Wx + (j >> 6)], 1ull << (j & 63));
    };
    walk_lists(sm.walk[w], a.cs, sv, item && narrow ? dv : 0, 0, tab,
               [&](int k, int h, int e) {
                 const int tl = sm.walk[w].item[k], j = e - sm.walk[w].off[k];
                 pair(t0 + 32 * w + tl, sm.hidx[h]);
                 if (j < 32)
                   atomicOr(&lo[tl], 1u << j);
                 else
                   atomicOr(&hi[tl], 1u << (j - 32));
               });
    __syncwarp();
    if (item && narrow && (lo[lane] | hi[lane])) put_row(a, x, v, rv, dv, uv, lo[lane], hi[lane]);
    for (uint32_t wm = __ballot_sync(MCE_FULL, item && !narrow && dv > 0); wm; wm &= wm - 1) {
      const int tl = __ffs(wm) - 1;
      long_item(a, x, __shfl_sync(MCE_FULL, v, tl), __shfl_sync(MCE_FULL, rv, tl),
                __shfl_sync(MCE_FULL, sv, tl), __shfl_sync(MCE_FULL, ev, tl), 0, tab,
                [&](int h) { pair(t0 + 32 * w + tl, sm.hidx[h]); });
    }
    __syncwarp();
  }
}

// The wide roots' regions: woff (from orientation) words past base, as far as
// cap words reach; the roots past it have none and are encoded by the search.
__global__ void wide_regions_kernel(const int32_t *__restrict__ list, uint32_t cnt,
                                    const int32_t *__restrict__ rp,
                                    const int32_t *__restrict__ split,
                                    const unsigned long long *__restrict__ woff,
                                    unsigned long long *base, unsigned long long cap,
                                    unsigned long long **wptr) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  const int32_t v = list[i];
  const unsigned long long rows = (unsigned long long)(rp[v + 1] - rp[v]);
  const unsigned long long words = rows * (unsigned long long)((rp[v + 1] - split[v] + 63) >> 6);
  const unsigned long long off = woff[i];
  wptr[v] = off + words <= cap ? base + off : nullptr;
}

}  // namespace

int enc_launch(const EncArgs &a, const int32_t *wide_list, uint32_t wide_cnt,
               const unsigned long long *woff, unsigned long long *wbase, unsigned long long wcap,
               uint32_t small_cnt, uint32_t max_dplus, int64_t arc0, int64_t arc1, int64_t v0,
               int64_t v1, int sms, cudaStream_t s, int *launches) {
  // rows and earlier rows that no triangle touches stay zero; nx: not yet known
  if (arc1 > arc0) MCE_CUDA(cudaMemsetAsync(a.enc + arc0, 0, sizeof(uint32_t) * (size_t)(arc1 - arc0), s));
  if (v1 > v0) MCE_CUDA(cudaMemsetAsync(a.nx + v0, 0xFF, sizeof(int32_t) * (size_t)(v1 - v0), s));
  MCE_CUDA(cudaMemsetAsync(a.next, 0, sizeof(uint32_t), s));
  if (wide_cnt > 0) {
    if (wcap > 0) MCE_CUDA(cudaMemsetAsync(wbase, 0, sizeof(unsigned long long) * (size_t)wcap, s));
    wide_regions_kernel<<<(wide_cnt + 255) / 256, 256, 0, s>>>(wide_list, wide_cnt, a.rp, a.split,
                                                               woff, wbase, wcap, a.wptr);
    MCE_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
  }
  if (small_cnt > 0) {
    int per_sm = 0;
    MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, enc_small_kernel, ENC_BLOCK, 0));
    const int64_t warps = (int64_t)sms * (per_sm > 0 ? per_sm : 1) * ENC_WARPS;
    // few roots: spread them over the warps rather than packing them
    int64_t f = ((int64_t)small_cnt + 4 * warps - 1) / (4 * warps);
    f = f < 1 ? 1 : f > 32 ? 32 : f;
    const int64_t want = (((int64_t)small_cnt + f - 1) / f + ENC_WARPS - 1) / ENC_WARPS;
    const int64_t blocks = std::min<int64_t>(want, warps / ENC_WARPS);
    enc_small_kernel<<<(unsigned)blocks, ENC_BLOCK, 0, s>>>(a, (uint32_t)f);
    MCE_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
  }
  if (wide_cnt > 0) {
    int per_sm = 0;
    MCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, enc_wide_kernel, WIDE_BLOCK, 0));
    const uint32_t groups = (max_dplus + WIDE_BLOCK - 1) / WIDE_BLOCK;
    const int64_t units = (int64_t)wide_cnt * groups;
    const int64_t blocks = std::min<int64_t>(units, (int64_t)sms * (per_sm > 0 ? per_sm : 1));
    enc_wide_kernel<<<(unsigned)blocks, WIDE_BLOCK, 0, s>>>(a, groups);
    MCE_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
  }
  return MCE_OK;
}

}  // namespace mce
