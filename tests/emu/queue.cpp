// queue MODE: the task ring on the CPU.  Prints what the mode says.
//   full   a donor that nobody takes from, a ticket drawn: {accepted, positions
//          handed out}
//   laps   two donors and two takers over many laps: {tasks pushed, sum of the
//          tasks taken}
//   stale  a taker without work whose slot is still an earlier lap's: {status}
//   held   a donor whose slot is never given back: {accepted, status}
#include <string>

#include "common.cuh"
#include "engine.cuh"
#include "kernels.h"
#include "queue.cuh"

using namespace mce;

int main(int argc, char **argv) {
  const std::string mode = argc > 1 ? argv[1] : "";
  emu::max_rounds = 20000000;
  const uint32_t cap = 64, words = 3;
  QueueHdr hdr;
  memset(&hdr, 0, sizeof hdr);
  std::vector<uint32_t> seq(cap);
  for (uint32_t i = 0; i < cap; ++i) seq[i] = i;
  std::vector<unsigned long long> pay(cap * words);
  uint32_t err = 0;
  BKArgs a;
  memset(&a, 0, sizeof a);
  a.err = &err;
  a.wait_limit_ns = 10000000;
  a.q.hdr = &hdr;
  a.q.seq = seq.data();
  a.q.pay = pay.data();
  a.q.cap = cap;
  a.q.words = words;
  a.q.slot = words;
  auto push = [&](unsigned long long x) {
    return q_push(a.q, a.err, a.wait_limit_ns, [&](uint32_t k) { return x + k; });
  };
  unsigned long long accepted = 0, taken = 0;
  if (mode == "full") {
    hdr.head = 1;
    emu::launch(emu::Config(1, 64), [&] {
      if (threadIdx.x >= 32) return;
      bool want = wants_task(a.q);
      for (int i = 0; i < 200 && want; ++i) {
        const int pushed = push(i);
        if (lane_id() == 0) accepted += pushed != Q_KEPT;
        want = pushed == Q_PUSHED || wants_task(a.q);
      }
    });
    printf("%llu %u\n", accepted, hdr.tail);
  } else if (mode == "laps") {
    emu::launch(emu::Config(1, 128), [&] {
      if (lane_id() == 0) atomicAdd(&hdr.work, 1u);
      if (threadIdx.x < 64)
        for (unsigned long long i = 0, want = 0; i < 1000;) {
          if (!want && !wants_task(a.q)) {
            __nanosleep(1);
            continue;
          }
          const int pushed = push(3 * (1000 * (threadIdx.x >> 5) + i));
          if (pushed == Q_KEPT) return;
          want = pushed == Q_PUSHED;
          ++i;
          if (lane_id() == 0) ++accepted;
        }
      root_phase_done(a.q);
      unsigned long long w = 0;
      idle_phase(
          a, [&](uint32_t, unsigned long long x) { w = x; },
          [&] {
            if (lane_id() < words) taken += w;
          });
    });
    printf("%llu %llu %u\n", accepted, taken, err);
  } else if (mode == "stale") {
    seq[0] = 1;  // the task of position 0, never taken
    hdr.head = hdr.tail = cap;
    emu::launch(emu::Config(1, 32), [&] { idle_phase(a, [](uint32_t, unsigned long long) {}, [] {}); });
    printf("%u\n", err);
  } else if (mode == "held") {
    seq[0] = 1;
    hdr.head = hdr.tail = cap;
    emu::launch(emu::Config(1, 32), [&] {
      const int pushed = push(7);
      if (lane_id() == 0) accepted += pushed != Q_KEPT;
    });
    printf("%llu %u\n", accepted, err);
  } else {
    return 2;
  }
  return 0;
}
