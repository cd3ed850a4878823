// What the host makes of the words that the CTAs of a resident solve leave
// (rwig_b200/csrc/resident_words.h).  Exits 0 when all holds.
#include <cstdio>

#include "../../rwig_b200/csrc/resident_words.h"

using namespace rwig::skres;

// The outcome when CTAs leave in the given order, the one numbered `failed`
// with a wait that ran out (-1: none).
static int leave(const int* order, int n, int failed, bool done, bool grad_bad = false) {
  double res[kResWords];
  for (double& x : res) x = 1.0;  // of an earlier launch
  words_clear(res);
  for (int k = 0; k < n; ++k) {
    if (grad_bad && order[k] == 2) res[kResGradBad] = 1.0;
    words_leave(res, order[k], order[k] != failed, done && order[k] != failed);
  }
  return words_outcome(res);
}

int main() {
  const int orders[3][4] = {{0, 1, 2, 3}, {3, 2, 1, 0}, {1, 0, 3, 2}};
  int bad = 0;
  for (const auto& o : orders) {
    bad += leave(o, 4, -1, true) != 1;
    bad += leave(o, 4, -1, false) != 0;
    bad += leave(o, 4, -1, true, true) != 0;
    for (int f = 0; f < 4; ++f) {
      bad += leave(o, 4, f, true) != -1;
      bad += leave(o, 4, f, false) != -1;
    }
  }
  double res[kResWords] = {};
  words_clear(res);
  bad += words_outcome(res) != 0;  // nobody reported
  std::printf("%d wrong\n", bad);
  return bad != 0;
}
