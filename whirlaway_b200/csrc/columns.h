// Where a caller's device columns lie, and whether kernels may read them there.
#pragma once
#include <cstddef>
#include <cstdint>

namespace wl {

// What CUDA reports of an address: ordinary memory of a device, which one, and the allocation.
struct ColumnMemory {
  bool device_memory = false;
  int device = -1;
  uintptr_t base = 0;
  size_t size = 0;
};
// Kernels of device `dev` read `bytes` at p in place when they are whole words of an allocation of
// that device. Anything else (another device's memory, mapped host or managed memory, an odd
// address, a range that CUDA does not vouch for) takes a copy, which accepts all of it that can be
// read and refuses the rest with an error, where a kernel would end the context.
inline bool read_in_place(const ColumnMemory& m, int dev, uintptr_t p, size_t bytes) {
  return m.device_memory && m.device == dev && p % 4 == 0 && m.base && p >= m.base && bytes <= m.size &&
         p - m.base <= m.size - bytes;
}

}  // namespace wl
