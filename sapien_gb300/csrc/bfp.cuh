// Block floating point: spatial algebra on 64-bit integer mantissas, for a GPU whose FP64 unit
// is 64 times slower than its integer and FP32 units.
//
// Measured on GB300 (2.07 GHz, cycles per warp instruction and scheduler): DFMA 68, 32 x 32 + 64
// bit integer multiply-add (IMAD.WIDE) 4, other 32-bit integer instructions 1 to 2. One FP64
// product thus costs as much as ~17 wide integer products. Here a 3-vector holds three signed
// mantissas |m| <= 2^61 and one exponent (value m 2^e), a rotation nine mantissas of fixed
// exponent -60. A product of two mantissas takes 3 wide multiply-adds: with balanced halves
// a = ah 2^32 + al, |al| <= 2^31, ab = ah bh 2^64 + (ah bl + al bh) 2^32 + al bl, of which the
// last term is below the result's last place and is left out. The cross terms and the high
// terms of a whole dot product are summed in 64-bit accumulators with a single shift between
// them, so a 3 x 3 product costs ~450 cycles a warp against ~2150 in FP64 (probe, two warps
// per scheduler and more). Up to three products fit the accumulators.
//
// Precision: all bounds are relative to the largest component of a vector, matrix or rotation. A
// mantissa keeps 60 bits below it and a product or dot product is off by about 2^-57 of |a| |b|,
// against 2^-53 for one rounded FP64 operation. A number on its own converts exactly; beside a
// larger one it is cut off 60 bits below that, as are the terms of a sum, where FP64 keeps 53
// bits of each: a component more than 2^7 below the largest holds less here than there. Rotations
// and sines are in steps of 2^-60 at any size. So callers keep configurations with small angles
// (bfp_small) away from these routines, and results that are small against their terms. Results
// are rounded to nearest once, on their way out.
//
// Range: exponents are 32-bit integers, so nothing overflows between inputs and outputs. Callers
// keep inputs that are not finite or beyond 2^+-200 away from these routines (bfp_fits).
#pragma once
#include "spatial.cuh"

namespace sgdyn {
namespace bfp {

typedef long long i64;
typedef unsigned long long u64;

struct Half {  // balanced halves: value h 2^32 + l
  int h, l;
};
struct Sc {  // scalar m 2^e
  i64 m;
  int e;
};
struct Vec {  // 3-vector with a shared exponent
  i64 x, y, z;
  int e;
};
struct Rot {  // rotation matrix, row-major, exponent -60
  i64 a[9];
};
struct Tw {  // motion (v, w) or force (f, n), each half with its own exponent
  Vec v, w;
};
struct Rbi {  // rigid-body inertia about the frame origin: mass, first moment, xx xy xz yy yz zz
  Sc m;
  Vec h;
  i64 I[6];
  int e;
};

constexpr i64 kOne = 1LL << 60;  // 1.0 as a mantissa of exponent -60

SG_HD Half split(i64 m) {
  Half r;
  r.l = int(unsigned(u64(m)));
  r.h = int(m >> 32) + int(unsigned(r.l) >> 31);
  return r;
}
// arithmetic shift right, any shift >= 0
SG_HD i64 shr(i64 m, int s) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(s));
  return r;
#else
  return m >> (s < 63 ? s : 63);
#endif
}
SG_HD i64 shl(i64 m, int s) { return i64(u64(m) << s); }
// a b + c as one wide multiply-add (from 64-bit operands the compiler makes a 64 x 64 product)
SG_HD i64 wide(int a, int b, i64 c) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return i64(a) * i64(b) + c;
#endif
}
SG_HD int clz32(unsigned v) {
#ifdef __CUDA_ARCH__
  return __clz(int(v));
#else
  return v ? __builtin_clz(v) : 32;
#endif
}
SG_HD int hi32(i64 m) { return int(m >> 32); }
SG_HD unsigned abs_hi(i64 m) {
  const int h = hi32(m);
  return unsigned(h < 0 ? -h : h);
}
SG_HD int imax(int a, int b) { return a > b ? a : b; }

// Dot products of one to three pairs: cross terms first, their high word carried into the sum of
// the high terms. The result is in units of 2^64 times the operands' units.
SG_HD i64 cross_terms(Half a, Half b, i64 c) { return wide(a.l, b.h, wide(a.h, b.l, c)); }
constexpr i64 kRound = 1LL << 31;
SG_HD i64 prod(Half a, Half b) { return wide(a.h, b.h, cross_terms(a, b, kRound) >> 32); }
SG_HD i64 prod(Half a, Half b, Half c, Half d) {
  return wide(c.h, d.h, wide(a.h, b.h, cross_terms(c, d, cross_terms(a, b, kRound)) >> 32));
}
SG_HD i64 prod(Half a, Half b, Half c, Half d, Half f, Half g) {
  return wide(f.h, g.h,
              wide(c.h, d.h, wide(a.h, b.h, cross_terms(f, g, cross_terms(c, d, cross_terms(a, b, kRound))) >> 32)));
}
// (the low half -2^31, of which there is no opposite, becomes 2^31 - 1: one unit of the mantissa)
SG_HD int neg_low(int l) { return -imax(l, -2147483647); }
SG_HD Half neg(Half a) { return Half{-a.h, neg_low(a.l)}; }

// Operands of at most 2^60 with the high half also held times 4, for products in units of 2^60:
// numbers of exponent -60 stay in that exponent.
struct Half4 {
  int h, l, h4;
};
SG_HD Half4 split4(i64 m) {
  const Half a = split(m);
  return Half4{a.h, a.l, int(unsigned(a.h) << 2)};
}
SG_HD Half4 neg(Half4 a) { return Half4{-a.h, neg_low(a.l), -a.h4}; }
SG_HD i64 cross_terms(Half4 a, Half4 b, i64 c) { return wide(a.l, b.h, wide(a.h, b.l, c)); }
constexpr i64 kRound4 = 1LL << 27;
SG_HD i64 mul60(Half4 a, Half4 b) { return wide(a.h4, b.h4, cross_terms(a, b, kRound4) >> 28); }
SG_HD i64 mul60(i64 a, i64 b) { return mul60(split4(a), split4(b)); }
SG_HD i64 mul60(Half4 a, Half4 b, Half4 c, Half4 d) {
  return wide(c.h4, d.h4, wide(a.h4, b.h4, cross_terms(c, d, cross_terms(a, b, kRound4)) >> 28));
}
SG_HD i64 mul60(Half4 a, Half4 b, Half4 c, Half4 d, Half4 f, Half4 g) {
  return wide(f.h4, g.h4,
              wide(c.h4, d.h4,
                   wide(a.h4, b.h4, cross_terms(f, g, cross_terms(c, d, cross_terms(a, b, kRound4))) >> 28)));
}

struct H3 {
  Half x, y, z;
};
SG_HD H3 split(const Vec& v) { return H3{split(v.x), split(v.y), split(v.z)}; }
SG_HD H3 neg(H3 a) { return H3{neg(a.x), neg(a.y), neg(a.z)}; }

// ---- conversions ---------------------------------------------------------------------
SG_HD u64 dbits(double x) {
#ifdef __CUDA_ARCH__
  return u64(__double_as_longlong(x));
#else
  u64 b;
  __builtin_memcpy(&b, &x, 8);
  return b;
#endif
}
SG_HD double from_bits(u64 b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(i64(b));
#else
  double x;
  __builtin_memcpy(&x, &b, 8);
  return x;
#endif
}
// zero, or finite with 2^-200 < |x| < 2^200
SG_HD bool bfp_fits(double x) {
  const u64 b = dbits(x);
  const unsigned E = unsigned(b >> 52) & 0x7ffu;
  return (b << 1) == 0 || (E - 823u) < 400u;
}
// Not 0, but below 2^-kSmall. The sine of an angle at that edge is held to 2^-44 of itself, a
// product with it to 2^-41. An environment with such an angle may have to go through FP64, which
// takes as long again: with kSmall = 12 a fifth longer for 16384 9-DoF arms with random angles,
// with 16 no longer (three batches in four have no angle below 2^-14, eleven in twelve below 2^-16).
constexpr int kSmall = 16;
SG_HD bool bfp_small(double x) {
  const u64 b = dbits(x) << 1;
  return b != 0 && unsigned(b >> 53) < unsigned(1023 - kSmall);
}
// x = m 2^e with 2^60 <= |m| < 2^61 (0: m = 0); exact
SG_HD Sc from_double(double x) {
  const u64 b = dbits(x);
  const int E = int(b >> 52) & 0x7ff;
  i64 m = i64(((b & 0xfffffffffffffULL) | (E ? 0x10000000000000ULL : 0ULL)) << 8);
  if (i64(b) < 0) m = -m;
  return Sc{m, E - 1083};
}
// |x| < 2 as a mantissa of exponent -60
SG_HD i64 q60(double x) {
  const Sc s = from_double(x);
  return shr(s.m, imax(0, -60 - s.e));
}
SG_HD Vec from_doubles(double x, double y, double z) {
  const Sc a = from_double(x), b = from_double(y), c = from_double(z);
  const int e = imax(a.e, imax(b.e, c.e));
  return Vec{shr(a.m, e - a.e), shr(b.m, e - b.e), shr(c.m, e - c.e), e};
}
// m 2^e rounded to nearest (halves up in magnitude)
SG_HD double to_double(i64 m, int e) {
  const u64 a = u64(m < 0 ? -m : m);
  const unsigned h = unsigned(a >> 32);
  const int lz = h ? clz32(h) : 32 + clz32(unsigned(a));
  const u64 n = a << (lz & 63);
  u64 r = (n >> 11) + ((n >> 10) & 1);  // 2^52 <= r <= 2^53
  const int E = e + 1085 - lz;          // exponent field, less the leading bit that r brings
  r += u64(unsigned(E)) << 52;
  if (m < 0) r |= 0x8000000000000000ULL;
  // results beyond the double range become 0 or infinity
  if (E < 0) r = 0;
  if (E > 2045) r = (m < 0 ? 0xfff0000000000000ULL : 0x7ff0000000000000ULL);
  return from_bits(a == 0 ? 0 : r);
}
SG_HD double to_double(Sc s) { return to_double(s.m, s.e); }

// ---- scalars -------------------------------------------------------------------------
// shifted so that 2^60 <= |m| < 2^61 (or up to 2^32 less where the high half is 0)
SG_HD Sc norm(Sc a) {
  const int s = imax(0, clz32(abs_hi(a.m)) - 3);
  return Sc{shl(a.m, s), a.e - s};
}
SG_HD Sc mul(Sc a, Sc b) { return Sc{prod(split(a.m), split(b.m)), a.e + b.e + 64}; }
SG_HD Sc neg(Sc a) { return Sc{-a.m, a.e}; }
SG_HD Sc add(Sc a, Sc b) {
  const int e = imax(a.e, b.e) + 1;
  return Sc{shr(a.m, e - a.e) + shr(b.m, e - b.e), e};
}
// 1 / d for 2^58 <= d <= 2^60 (exponent -60), result in exponent -58: a 23-bit estimate y0
// and r = y0 (1 + t + t^2), t = 1 - d y0 (|t| < 2^-20)
SG_HD i64 rcp60(i64 d) {
  // d in [1/4, 1]
  const float f = 1.0f / (float(hi32(d)) * 3.7252902984619140625e-09f);  // hi / 2^28; in [1, 4]
  const int y = int(f * 67108864.0f);                                    // exponent -26, at most 2^28
  const Half dh = split(d);
  // d y0 in exponent -60 - 26 + 26 (the product's low 26 bits dropped)
  const i64 t = kOne - (shl(wide(dh.h, y, 0), 6) + (wide(dh.l, y, 0) >> 26));
  const i64 tt = t + mul60(t, t);
  // y0 tt: exponent -26 - 60 -> -58
  const Half th = split(tt);
  return shl(i64(y), 32) + shl(wide(th.h, y, 0), 4) + (wide(th.l, y, 0) >> 28);
}
// 1 / sqrt(v) for v in [1/4, 1] (exponent -60), result in exponent -59: y0 (1 + t/2 + 3/8 t^2),
// t = 1 - v y0^2
SG_HD i64 rsqrt60(i64 v) {
#ifdef __CUDA_ARCH__
  const float f = rsqrtf(float(hi32(v)) * 3.7252902984619140625e-09f);  // in [1, 2]
#else
  const float f = 1.0f / sqrtf(float(hi32(v)) * 3.7252902984619140625e-09f);
#endif
  const int y = int(f * 134217728.0f);                                  // exponent -27, at most 2^28
  const i64 yy = wide(y, y, 0);                                         // exponent -54, at most 2^56
  const i64 vy = shl(mul60(v, shl(yy, 4)), 2);                          // exponent -58 -> -60
  const i64 t = kOne - vy;
  const i64 c = (t >> 1) + 3 * (mul60(t, t) >> 3);
  const Half ch = split(c);
  return shl(i64(y), 32) + shl(wide(ch.h, y, 0), 4) + (wide(ch.l, y, 0) >> 28);
}

// Sine and cosine of x as mantissas of exponent -60: x in fixed point 2^-60, reduced by
// multiples of pi/2 (constant in two parts), Taylor polynomials on [-pi/4, pi/4]. The terms
// that weigh less than 2^-28 are summed in 32-bit products. |x| >= 24 goes through the library.
// Off by 2^-56; a sine of a small angle by 2^-60.
SG_HD void sincos60(double x, i64* s, i64* c) {
  if (!(x > -24.0 && x < 24.0)) {
    double ds, dc;
    sincos(x, &ds, &dc);
    *s = q60(ds);
    *c = q60(dc);
    return;
  }
  const Sc xs = from_double(x);
  const int sh = xs.e + 58;  // at most 2
  const i64 h = sh > 0 ? shl(xs.m, sh) : shr(xs.m, -sh);
  const int n = int((wide(hi32(h), 1367130551, 0) + (1LL << 56)) >> 57);  // x 2/pi rounded (2/pi in 2^-31)
  // x in units of 2^-60 rounded to nearest, and x - n pi/2 (pi/2 = 1811004864519280711 -
  // 1734816687 2^-32 in these units); what goes beyond 64 bits on the way cancels
  const i64 q = sh >= -2 ? shl(xs.m, sh + 2) : shr(shr(xs.m, -sh - 3) + 1, 1);
  const i64 r = i64(u64(q) - u64(n) * 1811004864519280711ULL) + (wide(n, 1734816687, 0) >> 32);
  const i64 z = mul60(r, r);
  const int zh = int(z >> 29);
  auto m31 = [](int a, int b) { return int(wide(a, b, 0) >> 31); };
  int st = m31(zh, 203) - 55104;  // units 2^-56: z / 17! - 1 / 15!
  st = m31(zh, st) + 11571761;    // 1 / 13!
  st = m31(zh, st) - 1805194656;  // 1 / 11!
  int ct = 27552 - m31(zh, 90);   // units 2^-59: 1 / 16! - z / 18!
  ct = m31(zh, ct) - 6612435;     // 1 / 14!
  ct = m31(zh, ct) + 1203463104;  // 1 / 12!
  const Half4 zs = split4(z);
  auto step = [&](i64 a) { return mul60(split4(a), zs); };
  i64 S = shl(i64(st), 4);
  S = step(S) + 3177142594265LL;      // 1 / 9!
  S = step(S) - 228754266787073LL;    // 1 / 7!
  S = step(S) + 9607679205057058LL;   // 1 / 5!
  S = step(S) - 192153584101141163LL;  // 1 / 3!
  i64 C = shl(i64(ct), 1);
  C = step(C) - 317714259426LL;        // 1 / 10!
  C = step(C) + 28594283348384LL;      // 1 / 8!
  C = step(C) - 1601279867509510LL;    // 1 / 6!
  C = step(C) + 48038396025285291LL;   // 1 / 4!
  C = step(C) - 576460752303423488LL;  // 1 / 2!
  // r S with the low product, which weighs up to 2^-58: a small sine is kept to 2^-59
  const Half4 rs = split4(r), ss = split4(step(S));
  const i64 sn = r + wide(rs.h4, ss.h4, (cross_terms(rs, ss, kRound4) + (wide(rs.l, ss.l, 0) >> 32)) >> 28);
  const i64 cs = kOne + step(C);
  const i64 a = (n & 1) ? cs : sn, b = (n & 1) ? sn : cs;
  *s = (n & 2) ? -a : a;
  *c = ((n + 1) & 2) ? -b : b;
}

// ---- 3-vectors -----------------------------------------------------------------------
// Products and sums of normalised vectors may leave up to a few leading zero bits; norm()
// brings the largest component back to 2^60 <= |m| < 2^61.
SG_HD Vec vec0() { return Vec{0, 0, 0, -4000}; }
SG_HD Vec norm(Vec a) {
  const int s = imax(0, clz32(abs_hi(a.x) | abs_hi(a.y) | abs_hi(a.z)) - 3);
  return Vec{shl(a.x, s), shl(a.y, s), shl(a.z, s), a.e - s};
}
SG_HD Vec neg(Vec a) { return Vec{-a.x, -a.y, -a.z, a.e}; }
SG_HD Vec at_exp(Vec a, int e) { return Vec{shr(a.x, e - a.e), shr(a.y, e - a.e), shr(a.z, e - a.e), e}; }
SG_HD Vec add(Vec a, Vec b) {
  const int e = imax(a.e, b.e) + 1, s = e - a.e, t = e - b.e;
  return Vec{shr(a.x, s) + shr(b.x, t), shr(a.y, s) + shr(b.y, t), shr(a.z, s) + shr(b.z, t), e};
}
// of two products (each at most 2^60)
SG_HD Vec addp(Vec a, Vec b) {
  const int e = imax(a.e, b.e), s = e - a.e, t = e - b.e;
  return Vec{shr(a.x, s) + shr(b.x, t), shr(a.y, s) + shr(b.y, t), shr(a.z, s) + shr(b.z, t), e};
}
SG_HD Vec mul(Sc s, Vec a) {
  const Half h = split(s.m);
  const H3 v = split(a);
  return Vec{prod(h, v.x), prod(h, v.y), prod(h, v.z), s.e + a.e + 64};
}
SG_HD Vec cross(H3 a, int ae, H3 b, int be) {
  const H3 n = neg(b);
  return Vec{prod(a.y, b.z, a.z, n.y), prod(a.z, b.x, a.x, n.z), prod(a.x, b.y, a.y, n.x), ae + be + 64};
}
SG_HD Vec cross(Vec a, Vec b) { return cross(split(a), a.e, split(b), b.e); }
SG_HD i64 dot(H3 a, H3 b) { return prod(a.x, b.x, a.y, b.y, a.z, b.z); }
SG_HD Sc dot(Vec a, Vec b) { return Sc{dot(split(a), split(b)), a.e + b.e + 64}; }

// ---- rotations -----------------------------------------------------------------------
struct Q3 {
  Half4 x, y, z;
};
SG_HD Q3 split4(i64 x, i64 y, i64 z) { return Q3{split4(x), split4(y), split4(z)}; }
SG_HD i64 dot60(Q3 a, Q3 b) { return mul60(a.x, b.x, a.y, b.y, a.z, b.z); }
SG_HD H3 row(const Rot& R, int i) { return H3{split(R.a[3 * i]), split(R.a[3 * i + 1]), split(R.a[3 * i + 2])}; }
SG_HD Q3 row4(const Rot& R, int i) { return split4(R.a[3 * i], R.a[3 * i + 1], R.a[3 * i + 2]); }
SG_HD Q3 col4(const Rot& R, int j) { return split4(R.a[j], R.a[3 + j], R.a[6 + j]); }
SG_HD Vec col_vec(const Rot& R, int j) { return Vec{R.a[j], R.a[3 + j], R.a[6 + j], -60}; }
SG_HD Vec mul(const Rot& R, Vec v) {
  const H3 h = split(v);
  return Vec{dot(row(R, 0), h), dot(row(R, 1), h), dot(row(R, 2), h), v.e + 4};
}
SG_HD Rot mul(const Rot& A, const Rot& B) {
  Rot C;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const Q3 r = row4(A, i);
#pragma unroll
    for (int j = 0; j < 3; j++) C.a[3 * i + j] = dot60(r, col4(B, j));
  }
  return C;
}
SG_HD Rot rot_of(const i64* R) {
  Rot r;
#pragma unroll
  for (int k = 0; k < 9; k++) r.a[k] = R[k];
  return r;
}
SG_HD Rot identity() { return Rot{{kOne, 0, 0, 0, kOne, 0, 0, 0, kOne}}; }
// rotation about the unit axis a (exponent -60 mantissas): c 1 + s [a]x + (1 - c) a a^T
SG_HD Rot rodrigues(i64 ax, i64 ay, i64 az, i64 s, i64 c) {
  // 1 - c reaches 2: halved, the products doubled
  const Half4 t = split4((kOne - c) >> 1), hs = split4(s), x = split4(ax), y = split4(ay), z = split4(az);
  const Half4 tx = split4(mul60(t, x)), ty = split4(mul60(t, y)), tz = split4(mul60(t, z));
  auto p2 = [](Half4 a, Half4 b) { return shl(mul60(a, b), 1); };
  const i64 xy = p2(tx, y), xz = p2(tx, z), yz = p2(ty, z), sx = mul60(hs, x), sy = mul60(hs, y), sz = mul60(hs, z);
  return Rot{{p2(tx, x) + c, xy - sz, xz + sy, xy + sz, p2(ty, y) + c, yz - sx, xz - sy, yz + sx, p2(tz, z) + c}};
}
// quaternion x y z w of norm 1 to within 2^-9 -> rotation, the formula of quat_to_R
SG_HD Rot quat_rot(double dx, double dy, double dz, double dw) {
  const Half4 x = split4(q60(dx)), y = split4(q60(dy)), z = split4(q60(dz)), w = split4(q60(dw));
  auto p = [](Half4 a, Half4 b) { return shl(mul60(a, b), 1); };
  const i64 xx = p(x, x), yy = p(y, y), zz = p(z, z), xy = p(x, y), xz = p(x, z), yz = p(y, z), wx = p(w, x),
            wy = p(w, y), wz = p(w, z);
  return Rot{{kOne - (yy + zz), xy - wz, xz + wy, xy + wz, kOne - (xx + zz), yz - wx, xz - wy, yz + wx,
              kOne - (xx + yy)}};
}
// Rotation -> unit quaternion w x y z (Shepperd), the case rule of R_to_quat
SG_HD void rot_quat(const Rot& R, double* q) {
  const i64* a = R.a;
  const i64 t = a[0] + a[4] + a[8];
  int c = 0;
  if (!(t > 0)) {
    const bool i1 = a[4] > a[0];
    c = a[8] > (i1 ? a[4] : a[0]) ? 3 : (i1 ? 2 : 1);
  }
  const i64 di = c <= 1 ? a[0] : (c == 2 ? a[4] : a[8]);
  const i64 dj = c <= 1 ? a[4] : (c == 2 ? a[8] : a[0]);
  const i64 dk = c <= 1 ? a[8] : (c == 2 ? a[0] : a[4]);
  const i64 v = (c == 0 ? t : di - dj - dk) + kOne;  // 1 to 4: four times the component squared
  const i64 y = rsqrt60(v >> 2);                     // 2 / sqrt(v), exponent -59
  const Half4 yh = split4(y);
  const i64 d1 = a[7] - a[5], d2 = a[2] - a[6], d3 = a[3] - a[1];
  const i64 s01 = a[1] + a[3], s02 = a[2] + a[6], s12 = a[5] + a[7];
  const i64 n0 = c == 1 ? d1 : c == 2 ? d2 : d3;
  const i64 n1 = c == 0 ? d1 : c == 2 ? s01 : s02;
  const i64 n2 = c == 0 ? d2 : c == 1 ? s01 : s12;
  const i64 n3 = c == 0 ? d3 : c == 1 ? s02 : s12;
  // n / (2 sqrt v) = n y / 4 and sqrt(v) / 2 = (v / 4) y; n up to 2, halved
  auto p = [&](i64 n) { return to_double(mul60(split4(n >> 1), yh), -60); };
  const double big = to_double(mul60(split4(v >> 2), yh), -59);
  q[0] = c == 0 ? big : p(n0);
  q[1] = c == 1 ? big : p(n1);
  q[2] = c == 2 ? big : p(n2);
  q[3] = c == 3 ? big : p(n3);
}

// ---- spatial vectors and inertias ------------------------------------------------------
SG_HD Tw norm(Tw a) { return Tw{norm(a.v), norm(a.w)}; }
SG_HD Tw add(Tw a, Tw b) { return Tw{add(a.v, b.v), add(a.w, b.w)}; }
SG_HD Tw neg(Tw a) { return Tw{neg(a.v), neg(a.w)}; }
SG_HD Tw mul(Sc s, Tw a) { return Tw{mul(s, a.v), mul(s, a.w)}; }
SG_HD Sc dot(Tw a, Tw b) { return add(dot(a.v, b.v), dot(a.w, b.w)); }
// motion x motion and motion x* force
SG_HD Tw crossm(Tw a, Tw b) {
  const H3 aw = split(a.w), bw = split(b.w);
  return Tw{addp(cross(aw, a.w.e, split(b.v), b.v.e), cross(split(a.v), a.v.e, bw, b.w.e)),
            cross(aw, a.w.e, bw, b.w.e)};
}
SG_HD Tw crossf(Tw a, Tw f) {
  const H3 aw = split(a.w), fv = split(f.v);
  return Tw{cross(aw, a.w.e, fv, f.v.e),
            addp(cross(aw, a.w.e, split(f.w), f.w.e), cross(split(a.v), a.v.e, fv, f.v.e))};
}
// I w with I = xx xy xz yy yz zz of exponent e
SG_HD Vec sym_mul(const i64* I, int e, H3 w, int we) {
  const Half xx = split(I[0]), xy = split(I[1]), xz = split(I[2]), yy = split(I[3]), yz = split(I[4]), zz = split(I[5]);
  return Vec{dot(H3{xx, xy, xz}, w), dot(H3{xy, yy, yz}, w), dot(H3{xz, yz, zz}, w), e + we + 64};
}
// Y v = (m v - h x w, I w + h x v)
SG_HD Tw mul(const Rbi& Y, Tw a) {
  const H3 w = split(a.w), h = split(Y.h), v = split(a.v);
  return Tw{addp(mul(Y.m, a.v), cross(w, a.w.e, h, Y.h.e)),
            addp(sym_mul(Y.I, Y.e, w, a.w.e), cross(h, Y.h.e, v, a.v.e))};
}
SG_HD void norm_I(Rbi& Y) {
  unsigned o = 0;
#pragma unroll
  for (int k = 0; k < 6; k++) o |= abs_hi(Y.I[k]);
  const int s = imax(0, clz32(o) - 3);
#pragma unroll
  for (int k = 0; k < 6; k++) Y.I[k] = shl(Y.I[k], s);
  Y.e -= s;
}
SG_HD Rbi add(const Rbi& a, const Rbi& b) {
  Rbi r;
  r.m = norm(add(a.m, b.m));
  r.h = norm(add(a.h, b.h));
  r.e = imax(a.e, b.e) + 1;
  const int s = r.e - a.e, t = r.e - b.e;
#pragma unroll
  for (int k = 0; k < 6; k++) r.I[k] = shr(a.I[k], s) + shr(b.I[k], t);
  norm_I(r);
  return r;
}
// The world inertia of a body: mass m, centre of mass p + R c, rotational inertia I about it.
// With s = m c_world: I' = R I R^T + (s . c) 1 - s c^T.
SG_HD Rbi transport(const BJoint& B, const Rot& R, Vec p) {
  Rbi O;
  O.m = Sc{B.m, B.me};
  const Vec c = norm(add(mul(R, Vec{B.c[0], B.c[1], B.c[2], B.ce}), p));
  O.h = norm(mul(O.m, c));
  const H3 ch = split(c), sh = split(O.h);
  const Half nx = neg(sh.x), ny = neg(sh.y);
  // T = R I, then R I R^T by rows of T and R
  const H3 i0{split(B.I[0]), split(B.I[1]), split(B.I[2])}, i1{split(B.I[1]), split(B.I[3]), split(B.I[4])},
      i2{split(B.I[2]), split(B.I[4]), split(B.I[5])};
  auto trow = [&](int i) {
    const H3 r = row(R, i);
    return split4(dot(r, i0), dot(r, i1), dot(r, i2));
  };
  const Q3 r0 = row4(R, 0), r1 = row4(R, 1), r2 = row4(R, 2), t0 = trow(0), t1 = trow(1), t2 = trow(2);
  const int ea = B.Ie + 4, eb = c.e + O.h.e + 64, e = imax(ea, eb), da = e - ea, db = e - eb;
  O.I[0] = shr(dot60(t0, r0), da) + shr(prod(sh.y, ch.y, sh.z, ch.z), db);
  O.I[1] = shr(dot60(t0, r1), da) + shr(prod(nx, ch.y), db);
  O.I[2] = shr(dot60(t0, r2), da) + shr(prod(nx, ch.z), db);
  O.I[3] = shr(dot60(t1, r1), da) + shr(prod(sh.x, ch.x, sh.z, ch.z), db);
  O.I[4] = shr(dot60(t1, r2), da) + shr(prod(ny, ch.z), db);
  O.I[5] = shr(dot60(t2, r2), da) + shr(prod(sh.x, ch.x, sh.y, ch.y), db);
  O.e = e;
  norm_I(O);
  return O;
}

}  // namespace bfp
}  // namespace sgdyn
