// Relative error of the sine of csrc/bfp.cuh for angles that its callers leave to it, against long
// double; then which angles are called small.
#include <cmath>
#include <cstdio>
#include <random>
using std::fma;
using std::sqrt;
#include "bfp.cuh"
using namespace sgdyn;

int main() {
  std::mt19937_64 g(3);
  long double s = 0;
  for (int i = 0; i < 400000; i++) {
    const double u = double(g() >> 11) * 0x1p-53, e = -bfp::kSmall * u;
    const double x = (g() & 1 ? 1 : -1) * std::exp2(i % 4 ? e : e * 1e-3 - bfp::kSmall * 0.999);
    bfp::i64 a, b;
    bfp::sincos60(x, &a, &b);
    s = fmaxl(s, fabsl(ldexpl((long double)(a), -60) / sinl(x) - 1));
  }
  const double edge = std::exp2(-bfp::kSmall), below = std::nextafter(edge, 0.0);
  const bool ok = !bfp::bfp_small(0.0) && !bfp::bfp_small(-0.0) && bfp::bfp_small(1e-300) && bfp::bfp_small(-1e-20) &&
                  bfp::bfp_small(below) && bfp::bfp_small(-below) && !bfp::bfp_small(edge) && !bfp::bfp_small(-edge) &&
                  !bfp::bfp_small(3.0);
  std::printf("relative %.3Lg\npredicate %d\n", s, int(ok));
}
