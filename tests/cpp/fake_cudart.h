// Controls of the CUDA runtime's stand-in (fake_cudart.cpp).
#pragma once
#include <cstddef>
#include <map>
#include <set>

namespace fake {
extern long fail_at;       // which allocation from now on fails (0: the next); < 0: none
extern long failed;        // allocations failed so far
extern long device_syncs;  // device-wide waits so far
extern long launches;      // kernels launched so far
std::multiset<size_t> sizes();  // bytes of the live allocations
}  // namespace fake
