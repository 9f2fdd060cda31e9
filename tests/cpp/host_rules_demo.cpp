// The host-side rules of csrc/host_rules.h, checked without a device: exits
// with the number of failed checks.
#include <cmath>
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

// Rounds of at most eight iterations; |r|^2 to fall below 1e-10.
struct State {
  double inprodR, epsB;
  int done;
};
static void rounds() {
  State st[2] = {{1.0, 1e-10, 0}, {1.0, 1e-10, 1}};
  auto one = [&](double r0, long long nr0, double r1, long long nr1) {
    st[0].inprodR = r0;
    dda::RoundLength<State> next(st, 1);
    next.update(st, nr0, 8);
    st[0].inprodR = r1;
    return next.update(st, nr1, 8);
  };
  expect(one(1.0, 8, 1e-4, 16) == 8, "twelve iterations to go: a full round");
  expect(one(1.0, 8, 1e-8, 16) == 2, "two to go");
  expect(one(1.0, 8, 1e-7, 16) == 4, "three and a half: an even number");
  expect(one(1.0, 8, 0.999, 16) == 8, "a plateau: a full round");
  expect(one(1.0, 8, 1.5, 16) == 8, "growing: a full round");
  expect(one(1.0, 8, 0.0, 16) == 2, "zero, not yet seen as done");
  const double nan = std::nan("");
  expect(one(1.0, 8, nan, 16) == 8 && one(nan, 8, 1e-8, 16) == 8, "no number: a full round");
  // a plateau, then a fast fall: the look after the fall cuts the next round,
  // and what it leaves of eight comes after it
  st[0].inprodR = 1.0;
  dda::RoundLength<State> next(st, 1);
  long long nr = 8;
  auto look = [&](double r) {
    st[0].inprodR = r;
    const int n = next.update(st, nr, 8);
    nr += n;
    return n;
  };
  expect(look(0.9) == 8 && look(0.89) == 8, "plateau");
  expect(look(1e-7) == 4 && nr == 28, "the fall seen");
  expect(look(0.99e-7) == 4 && nr == 32, "a plateau again: up to the next multiple of eight");
  expect(look(0.9e-7) == 8 && nr == 40, "and whole rounds from there");
  // two right-hand sides: the slower one decides, a done one has no say
  State two[2] = {{1.0, 1e-10, 0}, {1.0, 1e-10, 0}};
  dda::RoundLength<State> both(two, 2);
  two[0].inprodR = 1e-8;
  two[1].inprodR = 1e-4;
  expect(both.update(two, 8, 8) == 8, "the slower decides");
  two[0].inprodR = 1e-9;
  two[1].done = 1;
  expect(both.update(two, 16, 8) == 8, "ten to go at the last rate");
  two[0].inprodR = 2e-10;
  two[1].inprodR = nan;
  expect(both.update(two, 24, 8) == 4, "the done one does not count");
}

int main() {
  shrinking();
  rounds();
  return failed;
}
