// mcx_alloc.h -- buffers that are allocated together: all of them or none.
#pragma once
#include <stddef.h>

#include <initializer_list>

namespace mcx {

struct Buffer {
  void **at;
  size_t bytes;
};

// Allocates every buffer with `alloc` (cudaMalloc's form; 0 is success).  On the
// first failure it releases those before it, leaves every pointer null and
// returns the failure, so that one pointer tells whether the set exists.
template <class Alloc, class Release>
inline int alloc_together(std::initializer_list<Buffer> bufs, Alloc alloc, Release release) {
  for (const Buffer &b : bufs) *b.at = nullptr;
  for (const Buffer &b : bufs) {
    const int r = (int)alloc(b.at, b.bytes);
    if (r == 0) continue;
    *b.at = nullptr;
    for (const Buffer &d : bufs) {
      if (*d.at) release(*d.at);
      *d.at = nullptr;
    }
    return r;
  }
  return 0;
}

}  // namespace mcx
