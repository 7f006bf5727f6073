// Two handles (of two devices, say) each raise a function's limit once; a raise
// that fails is tried again.
#include "../../fem_b200/csrc/smem_limits.hpp"

#include <cstdio>

#define CHECK(x) \
  if (!(x)) { std::printf("failed: %s\n", #x); return 1; }

int main() {
  int f = 0, g = 0, calls = 0;
  auto count = [&] { ++calls; };
  SmemLimits a, b;
  a.raise(&f, count);
  a.raise(&f, count);
  CHECK(calls == 1);
  b.raise(&f, count);   // another handle: the function may live on another device
  CHECK(calls == 2);
  a.raise(&g, count);
  CHECK(calls == 3);
  SmemLimits c;
  bool thrown = false;
  try {
    c.raise(&f, [] { throw 1; });
  } catch (int) {
    thrown = true;
  }
  CHECK(thrown);
  c.raise(&f, count);
  CHECK(calls == 4);
  std::puts("ok");
  return 0;
}
