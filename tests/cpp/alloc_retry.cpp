// An allocation fails only when memory that is merely kept does not make room for it.
#include "alloc_retry.h"

#include <cstdio>

int main() {
  int room = 100, kept = 64, released = 0;
  auto release = [&] { room += kept, kept = 0, released++; };
  auto take = [&](int n) {
    return hobak::alloc_or_release([&] { return n > room ? 2 : (room -= n, 0); }, release);
  };
  bool ok = take(60) == 0 && released == 0 && room == 40;  // fits: what is kept stays
  ok = ok && take(100) == 0 && released == 1 && room == 4;  // fits with it
  ok = ok && take(5) == 2 && room == 4;                      // does not fit
  std::puts(ok ? "ok" : "wrong");
  return ok ? 0 : 1;
}
