// vls_devlist.h -- a device list that grows with what it has to hold.
#pragma once
#include <cstddef>

namespace vls {

// Room for n entries: the outgrown list is given back before the longer one
// is allocated, and after a failed allocation the list holds nothing and says
// so (a capacity that ran ahead of the allocation would let the next caller
// write past the old list).  alloc(P **, n) and release(P *, n) return 0 or
// an error code, which reserve passes on.
template <typename P>
struct DeviceList {
  P *p = nullptr;
  size_t cap = 0;
  template <class Alloc, class Release>
  int reserve(size_t n, Alloc &&alloc, Release &&release) {
    if (p && n <= cap) return 0;
    P *const old = p;
    const size_t had = cap;
    p = nullptr;
    cap = 0;
    if (old)
      if (const int e = release(old, had)) return e;
    P *q = nullptr;
    if (const int e = alloc(&q, n)) return e;
    p = q;
    cap = n;
    return 0;
  }
};

}  // namespace vls
