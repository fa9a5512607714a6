// Which of a caller's device pointers a kernel may dereference itself (host only, no CUDA header, so
// the rule can be checked without a GPU).
#pragma once
#include <cstdint>

namespace trisk {

// A state of doubles on the model's device or in managed memory, at a double's alignment. A copy
// engine takes any other device pointer too (another device's memory, peer access or not, and any byte
// address); a load faults on those.
inline bool kernel_can_access(const void* p, bool managed, int pointer_device, int model_device) {
  return reinterpret_cast<uintptr_t>(p) % sizeof(double) == 0 && (managed || pointer_device == model_device);
}

}  // namespace trisk
