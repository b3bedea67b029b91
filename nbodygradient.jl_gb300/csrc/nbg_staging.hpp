// nbg_staging.hpp -- host memory that one call's small arrays are gathered in,
// so that they are copied to or from the device as one block (host only).
//
// Page-locked memory is kept between the calls of a context, grow-only up to
// `limit` bytes.  A larger block, or one that the system does not grant, is not
// an error: get() returns null and the caller takes pageable memory instead.
#pragma once
#include <algorithm>
#include <cstddef>

namespace nbg {

struct StagingBlock {
  void* (*alloc)(size_t);  // null where it fails
  void (*release)(void*);
  size_t limit;
  unsigned char* p = nullptr;
  size_t bytes = 0;

  // Room for n bytes, or null.
  unsigned char* get(size_t n) {
    if (n > limit) return nullptr;
    if (bytes < n) {
      free();
      const size_t want = std::min(limit, std::max<size_t>(n, 64 * 1024));
      p = (unsigned char*)alloc(want);
      bytes = p ? want : 0;
    }
    return p;
  }
  void free() {
    if (p) release(p);
    p = nullptr;
    bytes = 0;
  }
};

}  // namespace nbg
