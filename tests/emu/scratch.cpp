// scratch grant WANT HELD OTHERS FREE NEEDED: what wide_grant gives.
// scratch run LIMIT HELD NEED...: a device of LIMIT bytes on which a handle
// holds rows of HELD bytes; reserve_or_drop of buffers of NEED bytes.  Prints
// {status, times reserved, bytes still held as rows, bytes allocated}.
#include "scratch.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

int main(int argc, char **argv) {
  auto num = [&](int i) { return (uint64_t)strtoull(argv[i], nullptr, 10); };
  if (argc == 7 && !strcmp(argv[1], "grant")) {
    printf("%llu\n", (unsigned long long)mce::wide_grant(num(2), num(3), num(4), num(5), num(6)));
    return 0;
  }
  if (argc < 4 || strcmp(argv[1], "run")) return 2;
  const uint64_t limit = num(2);
  uint64_t held = num(3), used = held;
  std::vector<uint64_t> have(argc, 0);
  int times = 0;
  const int rc = mce::reserve_or_drop(
      12,
      [&] {
        ++times;
        for (int i = 4; i < argc; ++i) {
          if (have[i]) continue;  // allocated before the device was full
          if (used + num(i) > limit) return 12;
          used += have[i] = num(i);
        }
        return 0;
      },
      [&] {
        const bool any = held > 0;
        used -= held;
        held = 0;
        return any;
      });
  printf("%d %d %llu %llu\n", rc, times, (unsigned long long)held, (unsigned long long)(used - held));
  return 0;
}
