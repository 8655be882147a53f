// wide DCAP W PX DONATE_AFTER: the row pass and one launch of the wide engine
// over a graph whose roots (row offsets, split points, lists, wide roots on
// standard input) are the whole class, with tasks sized for a widest root of
// DCAP.  Writes the cliques and the tree nodes of every vertex, the histogram
// and {status bits, tasks pushed}, 64-bit words.
#include "enc.cu"
#include "wide.cu"

namespace mce {
__global__ void queue_init_kernel(QueueView q) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < q.cap; i += gridDim.x * blockDim.x)
    q.seq[i] = i;
}
}  // namespace mce

using namespace mce;
typedef unsigned long long ull;

static std::vector<int> read() {
  int64_t n = 0;
  if (fread(&n, 8, 1, stdin) != 1) exit(2);
  std::vector<int> v(n);
  if (n && fread(v.data(), 4, n, stdin) != (size_t)n) exit(2);
  return v;
}

int main(int argc, char **argv) {
  if (argc != 5) return 2;
  const int dcap = atoi(argv[1]), W = atoi(argv[2]), xp = atoi(argv[3]);
  const std::vector<int> rp = read(), split = read(), cs = read(), roots = read();
  const int n = (int)rp.size() - 1, R = (int)roots.size();
  ShapeInfo sh{};
  for (int c = 0; c < 9; ++c) sh.cls_off[c] = c > CLS_MEM ? R : 0;
  std::vector<ull> woff(R);
  ull words = 0;
  int widest = 1, xcap = 1;
  for (int i = 0; i < R; ++i) {
    const int v = roots[i], d = rp[v + 1] - split[v];
    woff[i] = words;
    words += (ull)(rp[v + 1] - rp[v]) * ((d + 63) / 64);
    widest = max(widest, d);
    xcap = max(xcap, split[v] - rp[v]);
  }
  std::vector<uint32_t> enc(cs.size());
  std::vector<ull *> wptr(n, nullptr);
  std::vector<ull> rows(words);
  std::vector<int> nx(n);
  uint32_t next = 0;
  EncArgs e{n, rp.data(), split.data(), cs.data(), roots.data(), &sh, enc.data(), wptr.data(),
            nx.data(), &next};
  if (enc_launch(e, roots.data(), R, woff.data(), rows.data(), words, 0, widest, 0, cs.size(), 0, n,
                 1, nullptr, nullptr))
    return 1;
  std::vector<ull> hist(MCE_HIST_MAX), count(n), nodes(n), slab;
  ull all_nodes[4] = {0};
  uint32_t err[4] = {0}, fetch[8] = {0};
  QueueHdr qh;
  const uint32_t cap = 1024, task = 1 + 4 * ((dcap + 63) / 64), slot = max(task, WIDE_TASK_WORDS);
  std::vector<uint32_t> seq(cap);
  std::vector<ull> pay((size_t)cap * slot + 1, 0xA5);
  BKArgs a;
  memset(&a, 0, sizeof a);
  a.rp = rp.data();
  a.split = split.data();
  a.cs = cs.data();
  a.roots = roots.data();
  a.shape = &sh;
  a.fetch = fetch;
  a.hist = hist.data();
  a.nodes = all_nodes;
  a.root_nodes = nodes.data();
  a.root_count = count.data();
  a.err = err;
  a.dcap = dcap;
  a.xcap = xcap;
  a.enc = enc.data();
  a.wptr = wptr.data();
  a.nx = nx.data();
  a.parts = 1;
  a.donate_min = 4;
  a.donate_after = (uint32_t)atoi(argv[4]);
  a.wait_limit_ns = 1ull << 40;
  a.q.hdr = &qh;
  a.q.seq = seq.data();
  a.q.pay = pay.data();
  a.q.cap = cap;
  a.q.words = task;
  a.q.slot = slot;
  int grid = 0;
  if (wide_plan(W, xp, 1, xcap, &grid, &a.slab_words)) return 1;
  slab.resize((size_t)grid * 4 * a.slab_words);
  a.slab = slab.data();
  memset(&qh, 0, sizeof qh);
  emu::launch(emu::Config(1, 256), [&] { queue_init_kernel(a.q); });
  if (wide_launch(W, xp, a, W == 4 ? 128 : 64, 5, grid, nullptr, nullptr)) return 1;
  if (pay.back() != 0xA5) return 1;
  const ull tail[2] = {err[0], qh.pushed};
  fwrite(count.data(), 8, n, stdout);
  fwrite(nodes.data(), 8, n, stdout);
  fwrite(hist.data(), 8, MCE_HIST_MAX, stdout);
  fwrite(tail, 8, 2, stdout);
  return 0;
}
