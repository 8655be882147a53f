// peel: the one-block peel over any CSR (row offsets and lists on standard
// input), symmetric or not.  Writes every vertex's priority and core number;
// the emulation ends with status 4 when shared memory past the launch's own is
// written.
#include "peel.cu"

using namespace mce;

static std::vector<int> read() {
  int64_t n = 0;
  if (fread(&n, 8, 1, stdin) != 1) exit(2);
  std::vector<int> v(n);
  if (n && fread(v.data(), 4, n, stdin) != (size_t)n) exit(2);
  return v;
}

int main() {
  emu::max_rounds = 2000000;
  const std::vector<int> rp = read(), col = read();
  const int n = (int)rp.size() - 1;
  std::vector<char> ctl(peel_ctl_bytes());
  std::vector<uint32_t> prio(n);
  std::vector<int> core(n);
  PeelArgs a;
  memset(&a, 0, sizeof a);
  a.n = n;
  a.m = (int64_t)col.size();
  a.rp = rp.data();
  a.col = col.data();
  a.core = core.data();
  a.prio = prio.data();
  a.ctl = ctl.data();
  if (peel_launch(a, nullptr, nullptr)) return 1;
  fwrite(prio.data(), 4, n, stdout);
  fwrite(core.data(), 4, n, stdout);
  return 0;
}
