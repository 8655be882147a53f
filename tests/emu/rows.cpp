// rows: the row pass over any CSR (row offsets, split points, lists, narrow
// roots, wide roots on standard input), symmetric or not, between guard words.
// Prints the guard words that changed.
#include "enc.cu"

using namespace mce;
typedef unsigned long long ull;

static std::vector<int> read() {
  int64_t n = 0;
  if (fread(&n, 8, 1, stdin) != 1) exit(2);
  std::vector<int> v(n);
  if (n && fread(v.data(), 4, n, stdin) != (size_t)n) exit(2);
  return v;
}

int main() {
  const std::vector<int> rp = read(), split = read(), cs = read(), narrow = read(), wide = read();
  const int n = (int)rp.size() - 1, R = (int)wide.size();
  std::vector<int> roots(narrow);
  roots.insert(roots.end(), wide.begin(), wide.end());
  ShapeInfo sh{};
  for (int c = CLS_R32 + 1; c < 9; ++c) sh.cls_off[c] = c > CLS_R64 ? (uint32_t)roots.size() : (uint32_t)narrow.size();
  // guard words after each region
  constexpr ull G = 64;
  std::vector<ull> woff(R);
  ull words = 0;
  int widest = 1;
  for (int i = 0; i < R; ++i) {
    const int v = wide[i], d = rp[v + 1] - split[v];
    woff[i] = words;
    words += (ull)(rp[v + 1] - rp[v]) * ((d + 63) / 64) + G;
    widest = max(widest, d);
  }
  std::vector<uint32_t> enc(cs.size() + G);
  std::vector<ull *> wptr(n, nullptr);
  std::vector<ull> rows(words);
  std::vector<int> nx(n);
  uint32_t next = 0;
  EncArgs e{n, rp.data(), split.data(), cs.data(), roots.data(), &sh, enc.data(), wptr.data(),
            nx.data(), &next};
  if (enc_launch(e, wide.data(), R, woff.data(), rows.data(), words, (uint32_t)narrow.size(), widest, 0,
                 cs.size(), 0, n, 1, nullptr, nullptr))
    return 1;
  int bad = 0;
  for (ull k = 0; k < G; ++k) bad += enc[cs.size() + k] != 0;
  for (int i = 0; i < R; ++i) {
    const ull end = i + 1 < R ? woff[i + 1] : words;
    for (ull k = 1; k <= G; ++k) bad += rows[end - k] != 0;
  }
  printf("%d\n", bad);
  return 0;
}
