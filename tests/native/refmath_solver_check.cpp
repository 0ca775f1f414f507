// Host check of refmath.h's solver expressions against the reference's double
// ones (src/solver.cpp:18-41,141-180): random values, smooth fields whose
// stencil cancels, exact ties, zeros, tiny and huge values.
#include "../../flip3d_gb300/csrc/refmath.h"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

using namespace refmath;

static bool same(float a, float b) {
  return (std::isnan(a) && std::isnan(b)) || (bits_of(a) == bits_of(b));
}

int main(int argc, char **argv) {
  const long N = argc > 1 ? atol(argv[1]) : 1000000;
  std::mt19937_64 rng(99);
  std::uniform_real_distribution<float> U(-1.0f, 1.0f);
  auto special = [&](long i, float x) -> float {
    switch (i % 41) {
    case 0: return 0.0f;
    case 1: return -0.0f;
    case 2: return x * 1e-30f;
    case 3: return x * 1e-44f;
    case 4: return x * 1e33f;
    case 5: return std::ldexp(1.0f, (int)(x * 20));
    case 6: return INFINITY;
    case 7: return NAN;
    }
    return x;
  };
  long bad_s = 0, bad_g = 0, bad_p = 0;
  const int ns[5] = {3, 32, 48, 75, 200};
  for (int t = 0; t < 5; t++) {
    const int n = ns[t], pow2 = (n & (n - 1)) == 0;
    const double h2 = (double)(float)(1.0 / ((double)n * n)), inv = 1.0 / h2;
    const float ih = (float)inv, il = (float)(inv - (double)ih);
    for (long i = 0; i < N; i++) {
      const float s = U(rng) * std::pow(10.0f, 4 * U(rng));
      float x[6];
      const float eps = std::pow(10.0f, -7 * std::fabs(U(rng)));
      for (float &v : x) v = i % 3 == 0 ? U(rng) : s * (1.0f + U(rng) * eps);
      float sv = s;
      if (i % 5 == 0) {
        const int k = (int)(rng() % 7);
        if (k == 6) sv = special((long)(rng() % 41), s);
        else x[k] = special((long)(rng() % 41), x[k]);
      }
      double v = 6.0 * (double)sv;
      for (float q : x) v -= (double)q;
      const float want = pow2 ? (float)(v * inv) : (float)(v / h2);
      if (!same(want, stencil_ref(sv, x[0], x[1], x[2], x[3], x[4], x[5], ih, il, h2, inv, pow2)))
        bad_s++;
      const float lc = i % 7 == 0 ? special((long)(rng() % 41), U(rng)) : -std::fabs(U(rng)) * 8;
      const float lq = i % 11 == 0 ? special((long)(rng() % 41), U(rng)) : std::fabs(U(rng)) * 2;
      if (!same((float)((double)lq / std::fmin(1.0e-6, (double)lc) * (double)sv),
                ghost_ref(lq, lc, sv)))
        bad_g++;
      const double p = 1.0 / (double)sqrtf(i % 9 == 0 ? std::ldexp(1.0f, (int)(rng() % 20))
                                                      : 1.0f + 9.0f * std::fabs(U(rng)));
      const float ph = (float)p, pl = (float)(p - (double)ph);
      if (!same((float)((double)sv * p * p), scale2_ref(sv, ph, pl, p))) bad_p++;
    }
  }
  printf("stencil %ld ghost %ld scale %ld of %ld\n", bad_s, bad_g, bad_p, 5 * N);
  return 0;
}
