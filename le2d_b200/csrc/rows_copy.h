// Which way le2d_rows_out / le2d_rows_in copy (host logic without CUDA calls).
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace le2d {

// The caller's buffer as the CUDA runtime and driver describe it.
struct RowsBuffer {
  bool device_memory = false;  // plain device memory (not page-locked, managed or unregistered)
  int device = -1;
  uintptr_t at = 0;             // the buffer's address
  uintptr_t base = 0;           // the allocation around it
  size_t extent = 0;            // and its bytes
};

// One kernel copies where nothing is lost by dereferencing both sides from the current device:
// the state and the buffer are that device's own memory, the buffer is aligned to an element,
// and the whole copy (`bytes`, > 0) lies within the buffer's allocation.  Copy calls do the
// rest: they reach another device's memory without a peer mapping and refuse what they cannot.
inline bool rows_by_kernel(const RowsBuffer& b, size_t bytes, size_t elem, int task_device, int current_device) {
  return b.device_memory && b.device == task_device && task_device == current_device && b.at % elem == 0 &&
         b.at >= b.base && b.at - b.base <= b.extent && bytes <= b.extent - (b.at - b.base);
}

}  // namespace le2d
