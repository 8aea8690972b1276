// Host entry point to place_samples (measure.cpp) -- TEST INFRASTRUCTURE ONLY.
#include "internal.h"

// items: {first, s0, ns} each, bases apart; returns their number
extern "C" int place(const double* mass, int nchunks, int chunk_bits, const double* u, int n,
                     uint32_t most, uint64_t* items, double* bases, uint32_t* placed) {
  const auto v = hisv::place_samples({mass, mass + nchunks}, chunk_bits, {u, u + n}, most, placed);
  for (size_t i = 0; i < v.size(); ++i) {
    items[3 * i] = v[i].first;
    items[3 * i + 1] = v[i].s0;
    items[3 * i + 2] = v[i].ns;
    bases[i] = v[i].base;
  }
  return int(v.size());
}
extern "C" uint32_t samples_per_block() { return hisv::kSamplesPerBlock; }
