// Host build of the quad sweep's arithmetic (boss_quad.cuh): for seeded random
// factors, the four products of every outer code, formed as the kernel forms them
// (rows walked from the base, pairs, chains, alignment), and the inputs, for
// tests/test_quad_host.py, which checks them against exact integer arithmetic.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../../theboss_gb300/csrc/boss_quad.cuh"

using namespace boss;

static long long bounded(std::mt19937_64& g, int bits) {
  const long long x = bits > 0 ? (long long)(g() >> (64 - bits)) : 0;
  return (g() & 1) ? -x : x;
}

int main(int argc, char** argv) {
  std::mt19937_64 g(argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1);
  const int cases = argc > 2 ? std::atoi(argv[2]) : 50;
  for (int t = 0; t < cases; ++t) {
    const int nf = 2 + t % 9, nd = 2 + (int)(g() % 3), mode = t % 5;
    
    // |sum over the digits| < 2^62: nd <= 4 digits of at most 60 bits; modes: full size, a
    // small factor, random widths, exact zeros, one dominating digit
    std::vector<Cx64> u((size_t)nd * nf);
    for (int a = 0; a < nd; ++a)
      for (int f = 0; f < nf; ++f) {
        int bits = 59;
        if (mode == 1 && f == 0) bits = 20;
        if (mode == 2) bits = (int)(g() % 60);
        if (mode == 4 && a > 0) bits = 25;
        Cx64 v{bounded(g, bits), bounded(g, bits)};
        if (mode == 3 && (g() & 3) == 0) v = Cx64{0, 0};
        u[(size_t)a * nf + f] = v;
      }
    for (int f = 0; f < nf; ++f) {  // every factor in its own scale, as the planners choose it
      long long most = 0;
      for (int a = 0; a < nd; ++a) most += std::max(std::llabs(u[(size_t)a * nf + f].re), std::llabs(u[(size_t)a * nf + f].im));
      int up = 0;
      while (most && (most << (up + 1)) < (1ll << 62)) ++up;
      for (int a = 0; a < nd; ++a) {
        u[(size_t)a * nf + f].re *= 1ll << up;
        u[(size_t)a * nf + f].im *= 1ll << up;
      }
    }
    for (int outer = 0; outer < (1 << (nd - 2)); ++outer) {
      long long re[4], im[4];
      int e[4] = {0, 0, 0, 0}, ls = 0;
      for (int p = 0; p < quad_slots(nf); ++p) {
        const bool unit = 2 * p + 1 >= nf;  // an odd last factor is paired with the constant 1
        const Cx64 zero{0, 0};
        auto U = [&](int a, int k) { return k && unit ? zero : u[(size_t)a * nf + 2 * p + k]; };
        Cx64 of = zero, og = zero, ep = zero, em = zero, q[4], cp, cm;
        if (unit) {
          og = Cx64{kQuadOne, 0};
          quad_row(zero, og, U(0, 0), U(1, 0), zero, zero, ep, em);
        }
        for (int a = 2; a < nd; ++a) {
          Cx64 rp, rm;
          quad_row(U(a, 0), U(a, 1), U(0, 0), U(1, 0), U(0, 1), U(1, 1), rp, rm);
          const bool neg = (outer >> (a - 2)) & 1;
          of = neg ? cx_sub(of, U(a, 0)) : cx_add(of, U(a, 0));
          og = neg ? cx_sub(og, U(a, 1)) : cx_add(og, U(a, 1));
          ep = neg ? cx_sub(ep, rp) : cx_add(ep, rp);
          em = neg ? cx_sub(em, rm) : cx_add(em, rm);
        }
        quad_const(U(0, 0), U(1, 0), U(0, 1), U(1, 1), cp, cm);
        ls += quad_pair(of, og, ep, em, cp, cm, q);
        for (int k = 0; k < 4; ++k)
          e[k] += p == 0 ? quad_chain_first(re[k], im[k], q[k].re, q[k].im) : quad_chain(re[k], im[k], q[k].re, q[k].im);
      }
      std::printf("%d %d %d %d", nf, nd, outer, quad_exponent((nf & 1) ? -62 : 0, ls, quad_slots(nf)));
      for (int k = 0; k < 4; ++k) std::printf(" %lld %lld %d", re[k], im[k], e[k]);
      for (const Cx64& v : u) std::printf(" %lld %lld", v.re, v.im);
      std::printf("\n");
    }
  }
  return 0;
}
