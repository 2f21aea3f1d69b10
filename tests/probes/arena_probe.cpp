// Checks the bitmap tier's scratch arithmetic (no device needed): an arena
// sized for C candidates holds any child of n <= C candidates, while its list
// is built and while it runs, and a root's.  Prints the tightest case of each:
// words left over, C, n, K.
#include <cstdio>
#include <initializer_list>
#include <climits>

#include "cls_sizes.h"

using namespace gmbe;

struct Tight {
  long long left = LLONG_MAX, C = 0, n = 0;
  int K = 0;
  void take(long long l, long long c, long long m, int k) {
    if (l < left) left = l, C = c, n = m, K = k;
  }
};

int main() {
  Tight build, run, root;
  auto look = [&](long long C, long long n) {
    for (int K : {1, 2, 4}) {
      const int levels = cls_levels(32 * K, (int)n);
      const long long sub = cls_sub_words(C);
      // below a counts-tier push: the candidates' C indices at its end;
      // mpos lies in the counts tier's tcls (C words)
      build.take(sub - cls_list_words(n, K) - cls_build_words(n, K, false) - cls_stride(C), C, n, K);
      run.take(sub - cls_need(n, K, levels), C, n, K);
      // a root's arena also has bound, coff, fill, sidx, tcls, tlist and ckey
      root.take(sub + 8 * C - cls_key_words(K) - cls_need(n, K, levels) -
                    cls_build_words(n, K, true), C, n, K);
    }
  };
  for (long long C = 1; C <= 3000; ++C)
    for (long long n = 1; n <= C; n += 1 + C / 64) look(C, n), look(C, C);
  for (long long C = 3001; C < (1 << 24); C += 1 + C / 50)
    for (long long d = 0; d < 70; ++d) look(C, C - d), look(C, 1 + (C - 1) * d / 70);
  for (const Tight* t : {&build, &run, &root})
    printf("%lld %lld %lld %d\n", t->left, t->C, t->n, t->K);
  return 0;
}
