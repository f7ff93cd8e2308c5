// Whether a kernel may write a caller's buffer itself, or has to leave it to a copy (which the
// driver checks and refuses where the buffer cannot take it).
#pragma once
#include <cstddef>
#include <cstdint>

namespace psl {

// What the driver reports about an address.  All zero for memory it does not know.
struct PointerFacts {
  bool device_memory = false;  // ordinary device memory, of `device`
  int device = 0;
  uint64_t mapped = 0;         // the address at which the current device reaches it, 0: it does not
  uint64_t range_start = 0;    // the allocation or registered range around the address
  size_t range_size = 0;
  unsigned int access = 0;     // of the current device: bit 0 read, bit 1 write
};

// True when all `bytes` at `address` lie in one range that `device` can write, and the address
// is aligned.  A range that ends too early or is registered read-only (cudaHostRegisterReadOnly)
// is left to the copy: a kernel that wrote there would fault.
inline bool kernel_may_write(const PointerFacts& f, uint64_t address, size_t bytes, size_t align, int device) {
  if (!f.mapped || f.mapped % align != 0) return false;
  if (f.device_memory && f.device != device) return false;
  if ((f.access & 2u) == 0) return false;
  return address >= f.range_start && f.range_size >= bytes && address - f.range_start <= f.range_size - bytes;
}

}  // namespace psl
