// An allocation that is tried again after memory kept for later has gone back.
#pragma once

namespace hobak {

// alloc() returns 0 on success; release() gives back what is only kept.
template <typename Alloc, typename Release>
int alloc_or_release(Alloc alloc, Release release) {
  if (alloc() == 0) return 0;
  release();
  return alloc();
}

}  // namespace hobak
