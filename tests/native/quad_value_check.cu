// Host build of a pair's four values (boss_quad.cuh: quad_values, and quad_small below
// kQuadLeast) for seeded random factors, with the factors, for
// tests/test_quad_values_host.py, which checks them against exact integers.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../../theboss_gb300/csrc/boss_quad.cuh"

using namespace boss;

int main(int argc, char** argv) {
  std::mt19937_64 g(argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1);
  const int cases = argc > 2 ? std::atoi(argv[2]) : 50;
  for (int t = 0; t < cases; ++t) {
    const int nd = 2 + (int)(g() % 31), mode = t % 7, weak = 1 + (int)(g() % 50);
    // modes: full size; random widths; two digits that cancel (weakly coupled by 2^-weak) in
    // both factors, in one; exact zeros; tiny factors; a constant second factor.  Every |sum| < 2^62.
    std::vector<Cx64> u(2 * nd);
    auto draw = [&](int bits) {
      const long long x = bits > 0 ? (long long)(g() >> (64 - bits)) : 0;
      return (g() & 1) ? -x : x;
    };
    for (int f = 0; f < 2; ++f)
      for (int a = 0; a < nd; ++a) {
        int bits = 56;
        if (mode == 1) bits = (int)(g() % 57);
        if ((mode == 2 || (mode == 3 && f == 0)) && a > 1) bits = std::max(0, 56 - weak);
        if (mode == 5) bits = 6;
        Cx64 v{draw(bits), draw(bits)};
        if ((mode == 4 && (g() & 3)) || (mode == 6 && f == 1)) v = cx(0, 0);
        u[2 * a + f] = v;
      }
    if (mode == 2 || mode == 3)
      for (int f = 0; f < (mode == 2 ? 2 : 1); ++f) {
        u[f] = cx(draw(60), draw(60));
        u[2 + f] = (g() & 1) ? u[f] : cx(-u[f].re, -u[f].im);
      }
    Cx64 of = cx(0, 0), og = mode == 6 ? cx(kQuadOne, 0) : of, ep = of, em = of;
    if (mode == 6) quad_row(of, og, u[0], u[2], u[1], u[3], ep, em);
    std::vector<int> d(nd, 1);
    for (int a = 2; a < nd; ++a) {
      Cx64 rp, rm;
      quad_row(u[2 * a], u[2 * a + 1], u[0], u[2], u[1], u[3], rp, rm);
      d[a] = (g() & 1) ? -1 : 1;
      of = cx_add(of, cx_times(u[2 * a], d[a]));
      og = cx_add(og, cx_times(u[2 * a + 1], d[a]));
      ep = cx_add(ep, cx_times(rp, d[a]));
      em = cx_add(em, cx_times(rm, d[a]));
    }
    longlong2 con[kQuadConst];
    quad_constants(u[0], u[2], u[1], u[3], con);
    auto low = [&](unsigned long long x) { return (int)(unsigned)x; };
    Cx64 q[4];
    int l[4];
    quad_values(of, og, ep, em, Cx64{con[0].x, con[0].y, low(con[2].x), low((unsigned long long)con[2].x >> 32)},
                Cx64{con[1].x, con[1].y, low(con[2].y), low((unsigned long long)con[2].y >> 32)}, q, l);
    const bool direct = (g() & 1) != 0;  // all four from the factors
    std::printf("%d %lld", nd, mode == 6 ? kQuadOne : 0ll);
    for (int k = 0; k < 4; ++k) {
      const bool small = l[k] < kQuadLeast || direct;
      const longlong2 f = con[3 + (k >> 1)], g = con[5 + (k >> 1)];
      Cx64 r[2];
      int lr[2];
      quad_small(of, og, cx(f.x, f.y), cx(g.x, g.y), r, lr);
      if (small) {
        q[k] = r[k & 1];
        l[k] = lr[k & 1];
      }
      std::printf(" %lld %lld %d %d", q[k].re, q[k].im, l[k], (int)small);
    }
    for (int a = 0; a < nd; ++a)
      std::printf(" %d %lld %lld %lld %lld", d[a], u[2 * a].re, u[2 * a].im, u[2 * a + 1].re, u[2 * a + 1].im);
    std::printf("\n");
  }
  return 0;
}
