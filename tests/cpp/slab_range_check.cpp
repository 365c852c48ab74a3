// The range of n . v that a slab's bounds are taken from holds the exact value and is as tight as that value rounded
// outwards to float, the form it had when it was computed in FP64, for meshes at the origin and far from it.
#include "../../thea_gb300/csrc/slab_range.cuh"

#include <cstdio>
#include <random>

static float down(long double x) {
  float f = (float)x;
  return (long double)f > x ? nextafterf(f, -INFINITY) : f;
}

int main() {
  std::mt19937_64 rng(5);
  std::normal_distribution<double> g;
  std::uniform_real_distribution<double> u(-1, 1);
  long wider = 0, total = 0;
  for (double far : {0.0, 1.0, 100.0, 1e6, 1e-30, 1e-42, 1e30}) {
    for (int i = 0; i < 200000; ++i) {
      float n[3], v[3];
      double l = 0;
      for (int a = 0; a < 3; ++a) n[a] = (float)g(rng), l += (double)n[a] * n[a];
      for (int a = 0; a < 3; ++a) n[a] = (float)(n[a] / std::sqrt(l));
      double size = far < 1e-20 && far > 0 ? far : 1.0;
      for (int a = 0; a < 3; ++a) v[a] = (float)(size * u(rng) + (size == 1.0 ? far : 0.0) * (a == 1 ? -1 : 1));
      // 80-bit sums of exact products where the compiler has them; the check allows for their rounding
      long double x = 0, m = 0;
      for (int a = 0; a < 3; ++a) x += (long double)n[a] * v[a], m += std::fabs((long double)n[a] * v[a]);
      float lo, hi;
      thea::slab_project(n[0], n[1], n[2], v[0], v[1], v[2], lo, hi);
      long double tiny = m * 0x1p-52L;
      if ((long double)lo > x + tiny || (long double)hi < x - tiny) {
        std::printf("far %g: [%.9g, %.9g] does not hold %.12Lg\n", far, lo, hi, x);
        return 1;
      }
      // as tight: within a step of the value rounded outwards, and equal to it but rarely
      float rl = down(x), rh = -down(-x);
      ++total;
      if (lo != rl || hi != rh) ++wider;
      float wl = nextafterf(down(x - m * 0x1p-43L - 3e-44L), -INFINITY), wh = nextafterf(-down(-x - m * 0x1p-43L - 3e-44L), INFINITY);
      if (lo < wl || hi > wh) {
        std::printf("far %g: [%.9g, %.9g] is wider than [%.9g, %.9g]\n", far, lo, hi, rl, rh);
        return 1;
      }
    }
  }
  float lo, hi;
  thea::slab_project(1.f, 0.f, 0.f, INFINITY, 0.f, 0.f, lo, hi);
  bool inf = lo == -INFINITY && hi == INFINITY;
  thea::slab_project(1.f, 0.f, 0.f, NAN, 0.f, 0.f, lo, hi);
  if (!inf || lo != -INFINITY || hi != INFINITY) {
    std::printf("a product that is not finite bounds nothing\n");
    return 1;
  }
  std::printf("%ld of %ld wider by a step\nranges hold and are tight\n", wider, total);
  return 0;
}
