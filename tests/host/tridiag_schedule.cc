// Plays the steps of k_tridiag through for every matrix size with the functions the kernel takes
// its decisions from (trl_b200/csrc/tridiag_schedule.h) and prints a line per disagreement: each
// pair sent to a CTA has to be one that the CTA's barrier counts and waits for in that step.
#include "tridiag_schedule.h"

#include <cstdio>

using namespace trl_detail;

int main()
{
  long steps = 0;
  for (int N = 3; N <= 1024; ++N) {
    int last[kTriC], owned[kTriC] = {};
    for (int c = 0; c < kTriC; ++c) last[c] = -1;
    for (int g = 0; g < N; ++g) { // by the ownership rule alone
      last[g % kTriC] = g;
      ++owned[g % kTriC];
    }
    for (int c = 0; c < kTriC; ++c)
      if (tri_last_row(N, c) != last[c]) std::printf("N %d cta %d: last row %d, not %d\n", N, c, tri_last_row(N, c), last[c]);
    if (tri_last_row(N, kTriC) != -1 || tri_last_row(N, 31) != -1) std::printf("N %d: a lane without a CTA sends\n", N);
    for (int s = 0; s < N - 1; ++s, ++steps)
      for (int c = 0; c < kTriC; ++c) {
        // a warp leaves when its last row is sent: the CTA is awaiting step s iff it has a row beyond s
        const bool awaits = owned[c] > 0 && last[c] > s;
        int sent = 0;
        for (int g = 0; g < N; ++g) sent += tri_sends(N, g, c, s);
        if (tri_waits(N, c, s) != awaits || sent != (awaits ? N - s : 0))
          std::printf("N %d step %d cta %d: awaits %d, expects %d, gets %d pairs\n", N, s, c, awaits, awaits ? N - s : 0, sent);
      }
  }
  std::printf("steps %ld\n", steps);
}
