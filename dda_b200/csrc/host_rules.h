// host_rules.h -- rules of the host side that need no device: how many
// iterations a solver's next round takes, and what an allocation shrinks to.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

namespace dda {

// Iterations of the next round: `poll`, or fewer when every running right-hand
// side is expected to converge within them.  A kernel whose right-hand sides
// are all done still costs its launch (a BiCGStab iteration of the two-rhs box
// 43 us of about 240), a look at the flags some 20 us.  The expectation is the
// mean rate of the residual since the last look; a round is an even number of
// iterations (RoundGraph), and rounds end on multiples of `poll` wherever they
// are not cut short, so that what is done every so many iterations is done at
// the same ones.
template <typename State> struct RoundLength {
  std::vector<double> last;
  long long last_nr = 0;
  RoundLength(const State* st, int nrhs) : last(nrhs, 0.0) {
    for (int r = 0; r < nrhs; r++) last[r] = st[r].inprodR;
  }
  int update(const State* st, long long nr, int poll) {
    const int full = poll - (int)(nr % poll);
    double need = 0;
    for (size_t r = 0; r < last.size(); r++) {
      const State& k = st[r];
      const double now = k.inprodR;
      if (!k.done) {
        const double rate = nr > last_nr && last[r] > now ? std::log(last[r] / now) / (double)(nr - last_nr) : 0.0;
        need = std::max(need, rate > 0 && k.epsB > 0 ? std::log(now / k.epsB) / rate : (double)full);
      }
      last[r] = now;
    }
    last_nr = nr;
    if (!(need < full)) return full;
    return std::max(2, std::min(full, 2 * (int)std::ceil(need / 2)));
  }
};

// The first of want, want / 2, want / 4, ..., least that alloc(bytes) takes;
// 0 when it refuses the least too.
template <typename F> size_t shrink_to_fit(size_t want, size_t least, F&& alloc) {
  for (size_t bytes = want;; bytes = std::max(least, bytes / 2)) {
    if (alloc(bytes)) return bytes;
    if (bytes <= least) return 0;
  }
}

}  // namespace dda
