// The offsets a dot's run of the mid list starts at (mid_row), around 2^31
// coefficients (addresses compared as integers, nothing is read but the two
// list bounds), and the pair counts whose lists the library builds
// (mid_list_fits).  Exit status 1 on any mismatch.
#include <cstdint>
#include <cstdio>

#include "../../quest_b200/csrc/qg_internal.h"

int main()
{
  int bad = 0;
  const int ends[] = {5, (1 << 28) - 1, 1 << 28, (1 << 28) + 3, 357913942, 1 << 30, 2147483647};
  for(int q = 1; q <= qg::kMaxOrder; ++q)
    for(int last : ends) {
      const int ptr[2] = {last - 5, last};  // a dot with five entries
      qg::StepArgs a{};
      a.q = q;
      a.mid_ptr = ptr;
      a.mid_idx = reinterpret_cast<const int *>(std::uintptr_t(1) << 40);
      a.mid_delay = reinterpret_cast<const int *>(std::uintptr_t(1) << 41);
      a.mid_coef = reinterpret_cast<const double2 *>(std::uintptr_t(1) << 42);
      const qg::MidRow r = qg::mid_row(a, 0);
      const std::uint64_t e0 = std::uint64_t(last) - 5;
      const bool ok = reinterpret_cast<std::uintptr_t>(r.idx) == (std::uint64_t(1) << 40) + 4 * e0 &&
                      reinterpret_cast<std::uintptr_t>(r.delay) == (std::uint64_t(1) << 41) + 4 * e0 &&
                      reinterpret_cast<std::uintptr_t>(r.coef) == (std::uint64_t(1) << 42) + 16 * e0 * (q + 1) &&
                      r.taps == 5 * (q + 1);
      if(!ok) std::printf("mismatch: q %d, entries up to %d\n", q, last), ++bad;
    }
  // 2^30 - 1 pairs are 2^31 - 2 entries, one pair more is past an int; a count
  // whose double wraps in 32 or 64 bits is refused like any other
  const unsigned long long p30 = 1ULL << 30;
  if(!qg::mid_list_fits(0) || !qg::mid_list_fits(p30 - 1)) std::printf("mismatch: refused a list that fits\n"), ++bad;
  const unsigned long long many[] = {p30, 2 * p30, 2 * p30 + 5, 4 * p30, 1ULL << 63};
  for(unsigned long long p : many)
    if(qg::mid_list_fits(p)) std::printf("mismatch: accepted %llu pairs\n", p), ++bad;
  std::printf("mismatches %d\n", bad);
  return bad != 0;
}
