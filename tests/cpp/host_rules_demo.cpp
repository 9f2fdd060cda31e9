// The host-side rules of csrc/host_rules.h, checked without a device: exits
// with the number of failed checks.
#include <cstdio>

#include "host_rules.h"

static int failed = 0;
static void expect(bool ok, const char* what) {
  if (ok) return;
  failed++;
  std::printf("failed: %s\n", what);
}

static void shrinking() {
  using dda::shrink_to_fit;
  int calls = 0;
  auto room = [&](size_t have) {
    calls = 0;
    return [&calls, have](size_t bytes) { calls++; return bytes <= have; };
  };
  expect(shrink_to_fit(1000, 10, room(1000)) == 1000 && calls == 1, "what is wanted, at once");
  expect(shrink_to_fit(1000, 10, room(999)) == 500 && calls == 2, "half");
  expect(shrink_to_fit(1000, 10, room(70)) == 62 && calls == 5, "halves down to what fits");
  expect(shrink_to_fit(1000, 300, room(300)) == 300 && calls == 3, "the least instead of less");
  expect(shrink_to_fit(1000, 300, room(299)) == 0 && calls == 3, "nothing below the least");
  expect(shrink_to_fit(64, 64, room(0)) == 0 && calls == 1, "one try where want is least");
}

int main() {
  shrinking();
  return failed;
}
