// Tile counters of the states.
#include <mutex>
#include <vector>

#include "internal.h"

namespace hisv {

// One 32-byte sector each of a fixed array, so that a launch of k1_wide needs no
// memory of its own and none is reset between launches.  (Calls on one state are
// ordered among themselves; states share no counter.)  The array has a module of
// its own: kernels of a module with writable variables took 0.3 us more per launch
// (43 passes on 22 qubits, complex64: 603 against 590 us).
namespace {
constexpr int kTickets = 4096, kTicketStride = 8;
__device__ uint32_t g_tickets[kTickets * kTicketStride];
std::mutex g_ticket_mu;
std::vector<int> g_ticket_free;
int g_ticket_next = 0;
}  // namespace

int ticket_take() {
  std::lock_guard<std::mutex> lk(g_ticket_mu);
  if (!g_ticket_free.empty()) {
    const int i = g_ticket_free.back();
    g_ticket_free.pop_back();
    return i;
  }
  return g_ticket_next < kTickets ? g_ticket_next++ : -1;
}

void ticket_give(int i) {
  if (i < 0) return;
  std::lock_guard<std::mutex> lk(g_ticket_mu);
  g_ticket_free.push_back(i);
}

uint32_t* ticket_address(int i) {
  void* p = nullptr;
  if (i < 0 || cudaGetSymbolAddress(&p, g_tickets) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return static_cast<uint32_t*>(p) + size_t(i) * kTicketStride;
}

}  // namespace hisv
