// Several buffers that are only of use together: all of them or none.
#pragma once
#include <cstddef>
#include <vector>

namespace ua {

struct BufferNeed {
  void** p;  // receives the buffer
  size_t bytes;
};

// Allocates every buffer; where one fails, releases those before it and leaves every pointer null, so that a
// later call cannot take half of them for the whole.
template <class Alloc, class Release>
bool alloc_all(const std::vector<BufferNeed>& need, Alloc alloc, Release release) {
  for (const BufferNeed& n : need) *n.p = nullptr;
  for (const BufferNeed& n : need)
    if (!(*n.p = alloc(n.bytes))) {
      for (const BufferNeed& q : need) {
        if (*q.p) release(*q.p);
        *q.p = nullptr;
      }
      return false;
    }
  return true;
}

// Replaces the buffers by ones for `key` unless they are there for it already.  `have` is the key of the
// buffers (0: none) and is set after the last allocation.
template <class Alloc, class Release>
bool alloc_for(int& have, int key, const std::vector<BufferNeed>& need, Alloc alloc, Release release) {
  if (have == key) return true;
  if (have)
    for (const BufferNeed& n : need) release(*n.p);
  have = 0;
  if (!alloc_all(need, alloc, release)) return false;
  have = key;
  return true;
}

}  // namespace ua
