// Errors of block-floating-point operations (csrc/bfp.cuh) and of the same operations in FP64
// against long double, over seeded operands of many magnitudes. Prints "name bfp fp64" (root mean
// square, relative to the operands' norms), and for functions "name bfp" (largest error).
#include <cmath>
#include <cstdio>
#include <random>
using std::fma;
using std::sqrt;
#include "bfp.cuh"
using namespace sgdyn;
typedef long double L;

static std::mt19937_64 g(7);
static double U(double a, double b) { return a + (b - a) * double(g() >> 11) * 0x1p-53; }
static double N() { return U(-1, 1) + U(-1, 1) + U(-1, 1); }
static L val(long long m, int e) { return ldexpl(L(m), e); }

struct Sum {
  L a = 0, b = 0;
  int n = 0;
  void add(const bfp::Vec& q, V3 d, const L* w, L scale) {
    const L x[3] = {val(q.x, q.e), val(q.y, q.e), val(q.z, q.e)}, y[3] = {d.x, d.y, d.z};
    for (int k = 0; k < 3; k++) {
      a += (x[k] - w[k]) * (x[k] - w[k]) / scale / scale;
      b += (y[k] - w[k]) * (y[k] - w[k]) / scale / scale;
    }
    n++;
  }
  void print(const char* name) { std::printf("%s %.3Lg %.3Lg\n", name, sqrtl(a / n), sqrtl(b / n)); }
};

int main() {
  L s = 0, c = 0, r = 0, q = 0, out = 0;
  for (int i = 0; i < 300000; i++) {
    const double x = i % 3 ? U(-30, 30) : U(-1e-3, 1e-3);
    bfp::i64 a, b;
    bfp::sincos60(x, &a, &b);
    s = fmaxl(s, fabsl(val(a, -60) - sinl(x)));
    c = fmaxl(c, fabsl(val(b, -60) - cosl(x)));
    const long long m = (long long)(U(0.25, 1) * 0x1p60);
    r = fmaxl(r, fabsl(val(bfp::rcp60(m), -58) * val(m, -60) - 1));
    q = fmaxl(q, fabsl(val(bfp::rsqrt60(m), -59) * sqrtl(val(m, -60)) - 1));
    const long long any = (long long)(g()) >> (g() % 63);
    if (any) out = fmaxl(out, fabsl(L(bfp::to_double(any, -9)) / val(any, -9) - 1));
    const double y = N() * std::exp(U(-100, 100));
    if (bfp::to_double(bfp::from_double(y)) != y || bfp::to_double(bfp::from_double(-y)) != -y) return 1;
  }
  std::printf("sin %.3Lg\ncos %.3Lg\nreciprocal %.3Lg\nrsqrt %.3Lg\nrounding %.3Lg\n", s, c, r, q, out);
  // mantissas whose halves are the extreme ones: largest error of a cross product, relative to the norms
  L edge = 0;
  const unsigned lows[6] = {0x80000000u, 0x7fffffffu, 0xffffffffu, 0u, 1u, 0x80000001u};
  auto mantissa = [&] { return (long long)((((unsigned long long)(U(-0x1p28, 0x1p28))) << 32) | lows[g() % 6]); };
  for (int i = 0; i < 100000; i++) {
    const bfp::Vec a{mantissa(), mantissa(), mantissa(), 0}, b{mantissa(), mantissa(), mantissa(), 0};
    const bfp::Vec k = bfp::cross(a, b);
    const L A[3] = {L(a.x), L(a.y), L(a.z)}, B[3] = {L(b.x), L(b.y), L(b.z)};
    const L w[3] = {A[1] * B[2] - A[2] * B[1], A[2] * B[0] - A[0] * B[2], A[0] * B[1] - A[1] * B[0]};
    const L x[3] = {val(k.x, k.e), val(k.y, k.e), val(k.z, k.e)};
    for (int j = 0; j < 3; j++) edge = fmaxl(edge, fabsl(x[j] - w[j]) * 0x1p-120L);
    const bfp::Half4 h = bfp::split4(mantissa()), n = bfp::neg(h);
    edge = fmaxl(edge, fabsl(val(n.h, 32) + n.l + val(h.h, 32) + h.l) * 0x1p-60L);
  }
  std::printf("edges %.3Lg\n", edge);
  Sum cr, rv, sm, ax;
  for (int i = 0; i < 100000; i++) {
    const double fa = std::exp(U(-20, 20)), fb = std::exp(U(-20, 20));
    const V3 a = fa * mk(N(), N(), N()), b = fb * mk(N(), N(), N());
    const L A[3] = {a.x, a.y, a.z}, B[3] = {b.x, b.y, b.z};
    const L na = sqrtl(A[0] * A[0] + A[1] * A[1] + A[2] * A[2]), nb = sqrtl(B[0] * B[0] + B[1] * B[1] + B[2] * B[2]);
    const bfp::Vec qa = bfp::from_doubles(a.x, a.y, a.z), qb = bfp::from_doubles(b.x, b.y, b.z);
    const L w[3] = {A[1] * B[2] - A[2] * B[1], A[2] * B[0] - A[0] * B[2], A[0] * B[1] - A[1] * B[0]};
    cr.add(bfp::norm(bfp::cross(qa, qb)), cross(a, b), w, na * nb);
    const L t[3] = {A[0] + B[0], A[1] + B[1], A[2] + B[2]};
    sm.add(bfp::norm(bfp::add(qa, qb)), a + b, t, na + nb);
    const double th = U(-3, 3);
    V3 u = mk(N(), N(), N());
    u = (1 / sqrt(dot(u, u))) * u;
    const M3 R = rodrigues(u, std::sin(th), std::cos(th));
    bfp::Rot Q;
    for (int k = 0; k < 9; k++) Q.a[k] = bfp::q60(R.a[k]);
    L v[3];
    for (int k = 0; k < 3; k++) v[k] = R.a[3 * k] * A[0] + R.a[3 * k + 1] * A[1] + R.a[3 * k + 2] * A[2];
    rv.add(bfp::norm(bfp::mul(Q, qa)), mul(R, a), v, na);
    const double f = N();
    const L p[3] = {f * A[0], f * A[1], f * A[2]};
    ax.add(bfp::norm(bfp::mul(bfp::from_double(f), qa)), f * a, p, fabsl(f) * na);
  }
  cr.print("cross");
  rv.print("rotate");
  sm.print("add");
  ax.print("scale");
}
