// Bounds of the waits inside kernels (ptx.cuh::mbar_wait_bounded) and how one that runs out is reported, shared by kernels and bindings.
#pragma once
#include <cstdint>

namespace b200 {

constexpr uint32_t kWaitSpins = 1u << 20;      // failed looks at a barrier before a wait gives up (a look itself blocks for some time)

struct WaitBound {
  uint32_t spins = kWaitSpins;
  uint32_t* error = nullptr;                   // mapped host memory: receives the kernel's code below; the host looks before later launches and where it reads results
};

enum : uint32_t { kWaitPromptAttention = 1, kWaitPairGemm = 2 };

}  // namespace b200
