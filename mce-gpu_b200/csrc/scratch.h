// Device memory of a call: what it cannot do without, and the wide roots' rows
// that it can.  Host arithmetic only.
#pragma once

#include <stdint.h>

#include <algorithm>

namespace mce {

// A handle's rows of wide roots, all regions together, and what an allocation
// of rows leaves free on the device (for this call's other buffers that come
// later, other handles, the caller).
constexpr uint64_t WIDE_BYTES = 32ull << 30;
constexpr uint64_t WIDE_RESERVE = 1ull << 30;
// Rows up to this size are allocated without asking the device what is free: a
// query takes 69 us, the first count of ER n = 40,000 1.38 ms with it and 1.26
// without.
constexpr uint64_t WIDE_UNASKED = 64ull << 20;

// Bytes that a region of rows may have: `want` for every root of the call,
// `held` in it now (given back before it grows), `others` in the handle's other
// regions, `free_now` on the device, `needed` by what the call allocates next.
// Never less than held: a region that does not grow stays as it is.
inline uint64_t wide_grant(uint64_t want, uint64_t held, uint64_t others, uint64_t free_now,
                           uint64_t needed) {
  const uint64_t bound = others < WIDE_BYTES ? WIDE_BYTES - others : 0;
  const uint64_t keep = needed + WIDE_RESERVE;
  const uint64_t room = free_now + held > keep ? free_now + held - keep : 0;
  return std::max(held, std::min(want, std::min(bound, room)));
}

// Runs reserve(), which allocates and may be run again; if the device is full
// (code `full`), once more after drop() has given the rows back (false: there
// were none).
template <typename Reserve, typename Drop>
int reserve_or_drop(int full, Reserve reserve, Drop drop) {
  const int rc = reserve();
  if (rc != full || !drop()) return rc;
  return reserve();
}

}  // namespace mce
