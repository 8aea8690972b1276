// Host part of hs_measure: which chunk each sample point falls into, and the work
// items of the device search (k3_sample).
#include "internal.h"

namespace hisv {

std::vector<MeasureChunk> place_samples(const std::vector<double>& mass, int chunk_bits,
                                        const std::vector<double>& u, uint32_t most,
                                        uint32_t* placed) {
  std::vector<MeasureChunk> out;
  const uint32_t n = uint32_t(u.size());
  uint32_t k = 0;
  double cum = 0;
  for (size_t c = 0; c < mass.size() && k < n; ++c) {
    const double end = cum + mass[c];
    while (k < n && u[k] < end) {
      const uint32_t s0 = k;
      while (k < n && k - s0 < most && u[k] < end) ++k;
      out.push_back({uint64_t(c) << chunk_bits, cum, s0, k - s0});
    }
    cum = end;
  }
  *placed = k;
  return out;
}

}  // namespace hisv
