// The one-walk limiter of the face slopes against the reference's loop
// (src/Cell/cell_plm.c:81-113) on the host: lists of two to five slopes whose
// sizes are mixed from 1e-310 to 1e100, every order and sign, several PLM.
// Prints the number of lists that the walk decides, that it leaves to the loop,
// and that it answers otherwise; exit status 1 if there are any of the last.
#include <math.h>
#include <stdio.h>

#include "../../disco2_b200/csrc/dgpu_device.cuh"

static unsigned long long rng_state = 0x9e3779b97f4a7c15ull;
static unsigned int urand(unsigned int n) {  // splitmix64, below n
  unsigned long long z = (rng_state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  return (unsigned int)((z >> 33) % n);
}

static double loop(const double *S, int n, double m, double plm) {
  for (int k = 0; k < n; ++k) {
    if (S[k] * m < 0.0) m = 0.0;
    else if (fabs(plm * S[k]) < fabs(m)) m = plm * S[k];
  }
  return m;
}

int main() {
  const int ex[] = {-310, -300, -200, -170, -160, -150, -145, -140, -100, -17, 0, 100};
  const double plms[] = {1.0, 1.5, 2.0, 1e-3, 0.0, -0.7};
  long decided = 0, left = 0, wrong = 0;
  for (int t = 0; t < 4000000; ++t) {
    double S[5], m = 0.0;
    const int n = 2 + urand(4);
    const double plm = plms[urand(6)];
    const int lo = urand(12), hi = urand(12);
    for (int k = 0; k < n; ++k) {
      S[k] = urand(16) == 0 ? 0.0 : (1 + urand(9)) * pow(10.0, ex[urand(2) ? lo : hi]);
      if (urand(2)) S[k] = -S[k];
      m += S[k];
    }
    m /= n;
    // the kernels' walk
    double lim = HUGE_VAL;
    bool neg = plm < 0.0, pos = neg;
    for (int k = 0; k < n; ++k) {
      const double ps = plm * S[k];
      if (fabs(ps) < fabs(lim)) lim = ps;
      neg |= S[k] < 0.0;
      pos |= S[k] > 0.0;
    }
    double got = m;
    if (limit_left(got, lim, (m < 0.0 && pos) || (m > 0.0 && neg), limit_floor(plm))) {
      ++left;
      if (got != m) ++wrong;
      continue;
    }
    ++decided;
    if (got != loop(S, n, m, plm)) ++wrong;
  }
  printf("decided %ld left %ld wrong %ld\n", decided, left, wrong);
  return wrong != 0;
}
