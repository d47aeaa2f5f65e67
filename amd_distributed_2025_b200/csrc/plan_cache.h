// Plans of the problem sizes that a thread has seen: a program comes back with the same few, and a search (1.5 to 2.6 us
// for the bf16 GEMM) takes as long as a short kernel.  Each thread keeps one plan to a slot of the hash; sizes that share a
// slot are searched anew whenever they alternate.
#pragma once
#include <cstdint>

namespace b200 {

template <typename Plan>
class PlanCache {
 public:
  // make(M, N, K, sms) on a miss.  The reference is good until the thread's next call.
  template <typename F>
  const Plan& get(int M, int N, int K, int sms, int device, F&& make) {
    Entry& e = entries_[slot(M, N, K)];
    if (e.M != M || e.N != N || e.K != K || e.sms != sms || e.device != device)
      e = Entry{M, N, K, sms, device, make(M, N, K, sms)};
    return e.plan;
  }
  static constexpr int kSlots = 256;
  // Every bit of the three sizes reaches the slot: layers that differ in one of them only, and batch sizes in a row, do not
  // meet.  (An odd factor each, then the high half folded in: multiplicative hashing.)
  static uint32_t slot(int M, int N, int K) {
    uint64_t h = (uint64_t)(uint32_t)M * 0x9E3779B97F4A7C15ull;
    h = (h ^ (h >> 32) ^ (uint32_t)N) * 0x9E3779B97F4A7C15ull;
    h = (h ^ (h >> 32) ^ (uint32_t)K) * 0x9E3779B97F4A7C15ull;
    return (uint32_t)(h >> 56);
  }

 private:
  struct Entry {
    int M = 0, N = 0, K = 0, sms = 0, device = -1;
    Plan plan;
  };
  Entry entries_[kSlots];
};

}  // namespace b200
