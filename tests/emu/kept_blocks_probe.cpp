// Host entry points to kept_blocks.h -- TEST INFRASTRUCTURE ONLY.
#include "kept_blocks.h"

using Pool = hisv::KeptBlocks<1000>;

extern "C" {
void* pool_new() { return new Pool; }
long pool_take(void* q, uint64_t ctx, size_t bytes) {
  return long(reinterpret_cast<intptr_t>(static_cast<Pool*>(q)->take(ctx, bytes)));
}
static int give(const std::vector<void*>& v, long* out) {
  for (size_t i = 0; i < v.size(); ++i) out[i] = long(reinterpret_cast<intptr_t>(v[i]));
  return int(v.size());
}
int pool_put(void* q, uint64_t ctx, long p, size_t bytes, long* out) {
  return give(static_cast<Pool*>(q)->put(ctx, reinterpret_cast<void*>(p), bytes), out);
}
int pool_drain(void* q, uint64_t ctx, long* out) {
  return give(static_cast<Pool*>(q)->drain(ctx), out);
}
// an allocation whose tries end in errors[0], errors[1]; 2 = out of memory.
// Returns the last error, *tries = tries made
int alloc_tries(const int* errors, int kept, int* tries) {
  *tries = 0;
  return hisv::alloc_releasing(
      2, [&] { return errors[(*tries)++]; }, [&] { return kept != 0; });
}
}
