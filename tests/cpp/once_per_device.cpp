// A set-up kept per device runs once on each of them, and again after a failure.
#include "once_per_device.h"

#include <cstdio>

int main() {
  static hobak::OncePerDevice once;
  int runs[80] = {};
  int result = 0;
  auto at = [&](int device) { return once(device, [&] { return runs[device]++, result; }); };
  bool ok = at(0) == 0 && at(0) == 0 && runs[0] == 1;
  ok = ok && at(1) == 0 && runs[1] == 1 && at(1) == 0 && at(0) == 0 && runs[1] == 1 && runs[0] == 1;
  result = 2;
  ok = ok && at(2) == 2 && at(2) == 2 && runs[2] == 2 && at(1) == 0 && runs[1] == 1;
  result = 0;
  ok = ok && at(2) == 0 && at(2) == 0 && runs[2] == 3;
  ok = ok && at(63) == 0 && at(63) == 0 && runs[63] == 1;
  ok = ok && at(64) == 0 && at(64) == 0 && runs[64] == 2;  // past the table: each time
  std::puts(ok ? "ok" : "wrong");
  return ok ? 0 : 1;
}
