// Which phase of each mbarrier was asked for last (a copy requested, a product committed), for draining after a give-up: a
// wait on the parity of a phase that was never asked for, or on an older one, returns at once and proves nothing.
// Plain C++, so that a host program can follow it through a kernel's order of requests.
#pragma once
#include <stdint.h>

namespace rewy {

struct PhaseLog {
  uint32_t asked = 0, odd = 0;  // bit b: barrier b was asked for at all; parity of its last phase asked for
#ifdef __CUDACC__
  __host__ __device__ __forceinline__
#endif
  void request(int b) {  // phase 0, 1, 2, .. of barrier b
    odd ^= asked & (1u << b);
    asked |= 1u << b;
  }
};

}  // namespace rewy
