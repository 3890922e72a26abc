// How a batch of lattices is cut into sets that go through all steps of a call
// one after another.  Host code, free of CUDA types: the tests compile it with a
// host compiler.
#ifndef SLBC_SETS_CUH
#define SLBC_SETS_CUH

#include <algorithm>
#include <numeric>
#include <vector>

namespace slbc {

// The lattices of a batch are independent, so they need not take each step
// together: a set of them small enough to stay in L2 goes through all the steps
// of the call before the next set starts, and only a set's first step reads it
// from memory.  A batch that fits the L2 as a whole (up to kBatchWhole) is one
// set, whose steps are replayed from a graph; a larger one is cut into equal sets
// of at most kBatchSet.  Measured, FP32, per step: 64 lattices of 48^3 (419 MB)
// 161 us in one set, 134 in sets of 96 MB, 115 in sets of 64 MB; 16 of 45^3 (86
// MB) 29.0 in one set, 25.5 in two (before launches overlapped 16 lattices of 92
// MB took 33 in one and 36 in two, where the line comes from).
constexpr long long kBatchWhole = 112LL << 20, kBatchSet = 64LL << 20;

// The members of each set from the bytes of state per member and the member's
// launch class (a step of a set is one launch per class in it).  Members go class
// by class, so a set has few launches: 64 lattices of 48^3 in 8 classes took 278
// us per step in sets that each had all of them, 221 in one set, 166 so.  A
// member beyond kBatchSet is a set of its own, so that it does not shift the
// shares of the others; members that would be left as a small set (below half of
// kBatchSet), whose launches are shorter than the gaps between them, join the
// set before, or a member that does not fit the L2 anyway.
inline std::vector<std::vector<int>> batch_sets(const std::vector<long long> &bytes,
                                                const std::vector<int> &launch_class) {
  const int n = (int)bytes.size();
  std::vector<std::vector<int>> sets;
  std::vector<int> rest;
  long long left = 0, large = 0;  // bytes of `rest`, of the largest own set
  size_t largest = 0;
  if (std::accumulate(bytes.begin(), bytes.end(), 0LL) <= kBatchWhole) {
    rest.resize((size_t)n);
    std::iota(rest.begin(), rest.end(), 0);
    if (n > 0) sets.push_back(rest);
    return sets;
  }
  for (int d = 0; d < n; d++) {
    if (bytes[d] <= kBatchSet) {
      rest.push_back(d);
      left += bytes[d];
      continue;
    }
    if (bytes[d] > large) {
      large = bytes[d];
      largest = sets.size();
    }
    sets.push_back({d});
  }
  if (left < kBatchSet / 2 && (large > kBatchWhole || (large > 0 && large + left <= kBatchWhole))) {
    sets[largest].insert(sets[largest].end(), rest.begin(), rest.end());
    return sets;
  }
  std::stable_sort(rest.begin(), rest.end(), [&](int a, int b) { return launch_class[a] < launch_class[b]; });
  long long planned = (left + kBatchSet - 1) / kBatchSet;
  for (size_t r = 0; r < rest.size(); planned--) {
    // members whose middle lies in this set's share of what is left
    const long long share = left / std::max({1LL, std::min(planned, (left + kBatchSet - 1) / kBatchSet),
                                             (left + kBatchWhole - 1) / kBatchWhole});
    std::vector<int> set;
    long long b = 0;
    for (; r < rest.size() && (b < kBatchSet / 2 || b + bytes[rest[r]] / 2 < share); r++) {
      set.push_back(rest[r]);
      b += bytes[rest[r]];
    }
    left -= b;
    if (left < kBatchSet / 2 && b + left <= kBatchWhole)
      for (; r < rest.size(); r++) set.push_back(rest[r]);
    sets.push_back(set);
  }
  return sets;
}

}  // namespace slbc

#endif
