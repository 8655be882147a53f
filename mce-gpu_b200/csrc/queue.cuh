// Device task queue for sharing search subtrees between warps.
//
// Replaces the reference's worker list (include/queue.cuh:17-56: a ticket
// ring of idle block ids plus a per-block mailbox that a donor fills while
// the idle block spins, mce/mce_utils.cuh:241-263,1063-1113).  There, an idle
// block waits on its own mailbox without a limit, and the kernel only ends
// when every block of the grid sits in the ring, so the whole grid must be
// resident.  Here the queue holds self-contained tasks - a root and one node
// of its search tree (P, X and the chosen set as bitmaps over the root's
// later neighbours) - so any warp can take any task, and termination is a
// single counter:
//   work = warps still in their root phase + tasks queued or running.
// A warp that has run out of roots draws a ticket - the ring position of the
// next task nobody waits for - and polls that position alone, so thousands of
// idle warps do not meet at one word; donors push while tickets are ahead of
// tasks, each at a position of its own too (one atomic add).  What bounds the
// sharing is the chain of dependent accesses from one push to the next: with
// donors agreeing on the ring's tail by compare-and-swap the device made one
// push per 0.9 us, and the time of the search of an R-MAT graph of scale 13
// was its number of pushes.  An idle warp's poll is bounded by a no-progress
// time limit, a donor's wait for its slot by the same time.
#pragma once

#include "common.cuh"

namespace mce {

struct QueueHdr {  // one word per 128-byte line
  uint32_t head;   // tickets drawn (ring positions, modulo 2^32) ...
  uint32_t pad0[31];
  uint32_t tail;   // ... and tasks pushed
  uint32_t pad1[31];
  uint32_t work;   // see above
  uint32_t pad2[31];
  uint32_t pushed; // tasks pushed, over all launches of a search on this ring (statistics)
};

struct QueueView {
  QueueHdr *hdr = nullptr;
  uint32_t *seq = nullptr;           // cap entries
  unsigned long long *pay = nullptr; // cap x words
  uint32_t cap = 0;                  // power of two
  uint32_t words = 0;                // u64 words per task
  uint32_t slot = 0;                 // ... and the most that `pay` has room for
};

__global__ void queue_init_kernel(QueueView q);

// A ring slot at position pos (modulo cap): seq = pos when empty, pos + 1 with
// the task there, pos + cap once the task was taken.
//
// Claim a position and publish `words` task words held by the warp (lane k
// holds words k, k+32, ...; supplied by `get(k)`).
//
// Positions stay less than a lap ahead of tickets, so that the ticket of a
// slot's last task is drawn and the wait for the slot is one for a running warp
// to copy a task out: each claim follows a look at both counters that found
// positions less than a lap, minus one per warp of the launch, ahead, and each
// look is good for one claim, so at most every warp claims after the last one.
// The look is q_wants' or that of the warp's last push, which has it in flight
// beside the slot's word (with a look of its own before each claim a count of
// BA n = 1,155 took 1,040 us, with this one 1,023).
//
// The wait is bounded by limit_ns: when it runs out the search ends with
// MCE_ERR_WAIT_TIMEOUT.  The slot's word is read without acquire (an acquire
// empties the SM's L1: those graphs 9.64 ms a count, 9.62 without): nothing is
// read after it, and the task is written only where it has the awaited value,
// which its last reader released.
enum QPush : int { Q_KEPT = 0, Q_PUSHED = 1, Q_PUSHED_LAST = 2 };  // ... and no room for the next

template <typename Get>
__device__ __forceinline__ int q_push(const QueueView &q, uint32_t *err, uint64_t limit_ns,
                                      Get get) {
  const uint32_t lane = lane_id();
  uint32_t pos = 0;
  int ok = Q_KEPT;
  if (lane == 0) {
    pos = atomicAdd(&q.hdr->tail, 1u);
    const uint32_t head = ld_volatile(&q.hdr->head);
    const uint32_t *s = &q.seq[pos & (q.cap - 1)];
    bool free = ld_volatile(s) == pos;
    if (!free) {
      const uint64_t t0 = globaltimer_ns();
      do {
        __nanosleep(64);
        free = ld_volatile(s) == pos;
      } while (!free && globaltimer_ns() - t0 <= limit_ns);
    }
    if (free) {
      atomicAdd(&q.hdr->work, 1u);  // counted before anyone can take it
      atomicAdd(&q.hdr->pushed, 1u);
      const int32_t room = (int32_t)q.cap - (int32_t)(gridDim.x * (blockDim.x >> 5));
      ok = (int32_t)(pos + 1 - head) < room ? Q_PUSHED : Q_PUSHED_LAST;
    } else {
      atomicOr(err, MCE_ERR_WAIT_TIMEOUT);
    }
  }
  ok = __shfl_sync(MCE_FULL, ok, 0);
  if (ok == Q_KEPT) return ok;
  pos = __shfl_sync(MCE_FULL, pos, 0);
  unsigned long long *dst = q.pay + (size_t)(pos & (q.cap - 1)) * q.words;
  for (uint32_t k = lane; k < q.words; k += 32) dst[k] = get(k);
  __syncwarp();
  if (lane == 0) {
    __threadfence();
    st_release(&q.seq[pos & (q.cap - 1)], pos + 1);
  }
  __syncwarp();
  return ok;
}

// Whether the task of ticket `pos` is there (lane 0's answer).
__device__ __forceinline__ bool q_ready(const QueueView &q, uint32_t pos) {
  return ld_acquire(&q.seq[pos & (q.cap - 1)]) == pos + 1;
}

// Take the task of ticket `pos` (q_ready on lane 0 said so): put(k, word)
// receives every word, lane-strided.
template <typename Put>
__device__ __forceinline__ void q_take(const QueueView &q, uint32_t pos, Put put) {
  const uint32_t lane = lane_id();
  __syncwarp();  // the other lanes read after lane 0's acquire
  const volatile unsigned long long *src = q.pay + (size_t)(pos & (q.cap - 1)) * q.words;
  for (uint32_t k = lane; k < q.words; k += 32) put(k, src[k]);
  __syncwarp();
  if (lane == 0) st_release(&q.seq[pos & (q.cap - 1)], pos + q.cap);  // slot free again
  __syncwarp();
}

// Donate a child only while more warps are waiting than tasks are queued.  (A
// look that allows one claim: a ring has more slots than the device warps.)
__device__ __forceinline__ bool q_wants(const QueueView &q) {
  if (!q.hdr) return false;
  return (int32_t)(ld_volatile(&q.hdr->head) - ld_volatile(&q.hdr->tail)) > 0;
}

}  // namespace mce
