// Host-side FFT planning: radix factorisation and twiddle tables.
#include <cmath>

#include "internal.h"

namespace rdcu {

bool make_line_plan(int L, LinePlan* p) {
  if (L < 1 || L > kMaxLine) return false;
  p->L = L;
  const RadixSeq q = radix_seq(L);
  if (q.n == 0 && L > 1) return false;
  p->nstages = q.n;
  for (int st = 0; st < q.n; ++st) p->radix[st] = q.r[st];
  int Ns = 1;
  for (int st = 0; st < p->nstages; ++st) {
    p->div_m[st] = make_fastdiv((unsigned)(L / p->radix[st]));
    p->div_ns[st] = make_fastdiv((unsigned)Ns);
    Ns *= p->radix[st];
  }
  return true;
}

void make_twiddles(int L, std::vector<double2>& tw) {
  tw.resize(L);
  const long double two_pi = 6.283185307179586476925286766559005768L;
  for (int t = 0; t < L; ++t) {
    // reduce the angle to the first octant for accuracy, using exact symmetries
    // of the L-th roots of unity
    long long num = t;  // angle = -2 pi num / L
    long double c, s;
    if (4LL * num == L) {
      c = 0.0L; s = 1.0L;
    } else if (2LL * num == L) {
      c = -1.0L; s = 0.0L;
    } else if (4LL * num == 3LL * L) {
      c = 0.0L; s = -1.0L;
    } else {
      long double ang = two_pi * (long double)num / (long double)L;
      c = cosl(ang);
      s = sinl(ang);
    }
    if (num == 0) { c = 1.0L; s = 0.0L; }
    tw[t] = make_double2((double)c, (double)(-s));
  }
}

void set_lin_ops(const std::vector<LinEntry>& lin, LinTable* t) {
  t->nops = 0;
  t->real = 1;
  for (const LinEntry& e : lin) {
    if (e.nax == 1) t->real = 0;
    int g = 0;
    while (g < t->nops && !(t->op[g].nax == e.nax && (e.nax < 1 || t->op[g].ax0 == e.ax0) &&
                            (e.nax < 2 || t->op[g].ax1 == e.ax1)))
      ++g;
    if (g == t->nops) {  // at most 1 + 3 + 9 operators exist
      t->op[g].nax = e.nax;
      t->op[g].ax0 = e.nax >= 1 ? e.ax0 : 0;
      t->op[g].ax1 = e.nax >= 2 ? e.ax1 : 0;
      for (auto& row : t->coef[g])
        for (double& c : row) c = 0.0;
      ++t->nops;
    }
    t->coef[g][e.row][e.src] += e.coef;
  }
}

}  // namespace rdcu
