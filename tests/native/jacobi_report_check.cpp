// Host check of jacobi_report: the largest report of a cluster is the sweep count when
// no CTA's wait ran out, and kEigTimedOut when any CTA's did, whichever it is.
#include <algorithm>
#include <cstdio>

#include "jacobi_sched.h"

using namespace tsvd;

int main() {
  int bad = 0, cases = 0;
  for (int C = 1; C <= 8; C *= 2)
    for (unsigned dead = 0; dead < (1u << C); ++dead)
      for (int sweeps = 1; sweeps <= 30; ++sweeps, ++cases) {
        int32_t most = 0;
        for (int c = 0; c < C; ++c)
          most = std::max(most, jacobi_report(c, (dead >> c) & 1, sweeps));
        bad += most != (dead ? kEigTimedOut : sweeps);
      }
  std::printf("cases %d mismatches %d\n", cases, bad);
  return bad != 0;
}
