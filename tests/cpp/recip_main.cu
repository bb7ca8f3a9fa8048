// Largest error of quot1(x, recip(d)) (csrc/ts_common.cuh, run on the host) over random x and d, in
// units of the last place of the quotient; FP32 against double, FP64 against long double.
#include <cstdio>
#include <random>

#include "ts_common.cuh"

template <typename S, typename W> double worst(int digits, double span) {
  std::mt19937_64 gen(5);
  std::uniform_real_distribution<double> m(1.0, 2.0), e(-span, span);
  double bad = 0;
  for (int i = 0; i < 2000000; ++i) {
    const S d = (S)std::ldexp(m(gen), (int)e(gen)), x = (S)std::ldexp(m(gen), (int)e(gen));
    const W q = (W)x / (W)d;
    const double err = (double)((W)ts::quot1(x, ts::recip(d)) - q);
    bad = std::fmax(bad, std::fabs(err) / std::ldexp(1.0, std::ilogb((double)q) - digits + 1));
  }
  return bad;
}

int main() {
  const ts::Recip<float> z = ts::recip(0.0f), i = ts::recip(INFINITY);
  printf("%.9f %.9f %g %g\n", worst<float, double>(24, 20), worst<double, long double>(53, 200), ts::quot1(3.0f, z),
         ts::quot1(3.0f, i));
  return 0;
}
