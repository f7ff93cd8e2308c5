// Host build of the rule that lets a kernel write a caller's buffer itself
// (psl_destination.h), for the CPU tests.
#include "psl_destination.h"

extern "C" int kernel_may_write_host(int device_memory, int memory_device, uint64_t mapped, uint64_t start, uint64_t size,
                                     unsigned int access, uint64_t address, uint64_t bytes, int device) {
  psl::PointerFacts f;
  f.device_memory = device_memory != 0;
  f.device = memory_device;
  f.mapped = mapped;
  f.range_start = start;
  f.range_size = size;
  f.access = access;
  return psl::kernel_may_write(f, address, bytes, 8, device);
}
