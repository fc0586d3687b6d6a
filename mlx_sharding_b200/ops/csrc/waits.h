// Bounds of the waits inside kernels (ptx.cuh::mbar_wait_bounded), shared by kernels and bindings.
#pragma once
#include <cstdint>

namespace b200 {

constexpr uint32_t kWaitSpins = 1u << 20;      // failed looks at a barrier before a wait gives up (a look itself blocks for some time)

}  // namespace b200
