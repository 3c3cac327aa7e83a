// CLIK (aux_kernels.cuh: ik_env) with its linear algebra in block floating point (bfp.cuh) and the
// logarithm, its Jacobian's coefficients and the 6x6 Cholesky in FP64, one environment per thread.
//
// The FP64 kernel issues 1957 FP64 instructions per iteration and is bound by that unit (0.92 of
// its measured rate). Here the chain's kinematics, the Jacobian, the products with Jlog6 and the
// normal matrix run on the integer pipes beside the ~370 FP64 instructions that remain.
// Measured, 65536 9-DoF arms following targets, at most 100 iterations: 19.1 -> 8.5 ms; 16 of
// them, 30 iterations: 2.3 -> 1.1 ms. Bound by the latency of its ~18000 instructions per
// iteration (4.4 cycles each with under two warps per scheduler) and, with three, by their issue.
//
// Along the path to the link, u and p are each joint's world axis and position; with the link's
// joint at (Ro, po) a revolute column in its frame is Ro^T (u x (po - p), u), so with
// K1 = Jinv Ro^T, K2 = TR Ro^T and c = u x (po - p) the product with Jlog6 is (K1 c - K2 u, K1 u)
// (prismatic: (K1 u, 0)).
#pragma once
#include "aux_kernels.cuh"
#include "bfp.cuh"

namespace sgdyn {
namespace bfp {

struct Mat {  // 3x3 with a shared exponent, |m| <= 2^61
  i64 a[9];
  int e;
};
__device__ __forceinline__ Mat mat_from(const double* m) {
  Mat r;
  Sc s[9];
  int e = -4000;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    s[k] = from_double(m[k]);
    e = imax(e, s[k].e);
  }
#pragma unroll
  for (int k = 0; k < 9; k++) r.a[k] = shr(s[k].m, e - s[k].e);
  r.e = e;
  return r;
}
__device__ __forceinline__ void norm_mat(Mat& m) {
  unsigned o = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) o |= abs_hi(m.a[k]);
  const int s = imax(0, clz32(o) - 3);
#pragma unroll
  for (int k = 0; k < 9; k++) m.a[k] = shl(m.a[k], s);
  m.e -= s;
}
// X Y, or X Y^T
template <bool TRANSPOSED>
__device__ __forceinline__ Mat mul_mat(const i64* X, int xe, const i64* Y, int ye) {
  Mat r;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const H3 x{split(X[3 * i]), split(X[3 * i + 1]), split(X[3 * i + 2])};
#pragma unroll
    for (int j = 0; j < 3; j++)
      r.a[3 * i + j] = TRANSPOSED ? dot(x, H3{split(Y[3 * j]), split(Y[3 * j + 1]), split(Y[3 * j + 2])})
                                  : dot(x, H3{split(Y[j]), split(Y[3 + j]), split(Y[6 + j])});
  }
  r.e = xe + ye + 64;
  norm_mat(r);
  return r;
}
__device__ __forceinline__ Vec mul(const Mat& m, H3 v, int ve) {
  return Vec{dot(H3{split(m.a[0]), split(m.a[1]), split(m.a[2])}, v),
             dot(H3{split(m.a[3]), split(m.a[4]), split(m.a[5])}, v),
             dot(H3{split(m.a[6]), split(m.a[7]), split(m.a[8])}, v), m.e + ve + 64};
}
// 1 / sqrt(d), d > 0 finite and normal: exponent made even, then the fixed-point root
__device__ __forceinline__ double inverse_sqrt(double d) {
  const Sc s = from_double(d);        // m 2^e, 2^60 <= m < 2^61
  const int e = s.e + 62, h = e >> 1;  // d = (m 2^-62) 2^e, m 2^-62 in [1/4, 1/2)
  return to_double(rsqrt60((e & 1) ? s.m >> 1 : s.m >> 2), -59 - h);
}

// One environment; false where it needs the FP64 kernel (an input out of range, a mask entry
// that is not 0 or 1, a free flyer on the path, a normal matrix that is not positive definite; and
// one whose steps or result are small as a whole: rotations are in steps of 2^-60 here, so a first
// error of 1e-9 would be off by 1e-9 of itself, and the joints with it, where FP64 keeps it to its
// last bits along the frames' axes. A first error below kIkSmall is below the usual tolerances and
// then ends at once in FP64 too.)
constexpr double kIkSmall = 1.0 / (1 << kSmall);
template <int MAXJ>
__device__ __forceinline__ bool ik_env(const DModel* __restrict__ model, const IkArgs& a, const int64_t e) {
  const DJoint* __restrict__ JT = model_joints(model);
  const BJoint* __restrict__ BT = model_bjoints(model);
  const DLink& L = model_links(model)[a.link];
  const int nj = model->nj;
  double qs[MAXJ], qc[MAXJ], best[MAXJ], bestc[MAXJ];  // angle or slide; (cos, sin) of a continuous joint
  bool ok = true;
#pragma unroll 1
  for (int i = 1; i < nj; i++) {
    const DJoint& J = JT[i];
    ok = ok && J.kind != JK_FREEFLYER;
    double v = a.has_q0 && J.kind != JK_FREEFLYER ? ldv(a.q0, e, J.qcol) : 0.0;
    ok = ok && bfp_fits(v);
    qc[i] = 0.0;
    if (J.kind == JK_CONTINUOUS) {
      double s = 0.0, c = 1.0;
      if (a.has_q0) sincos(v, &s, &c);
      v = s;
      qc[i] = c;
    }
    qs[i] = best[i] = v;
    bestc[i] = qc[i];
  }
  short chain[MAXJ];
  int depth = 0;
#pragma unroll 1
  for (int j = L.joint; j > 0; j = JT[j].parent) chain[depth++] = short(j);
  // the target in the joint's frame, FP64 once per environment
  const V3 pt = mk(ldv(a.target, e, 0), ldv(a.target, e, 1), ldv(a.target, e, 2));
  const double w = ldv(a.target, e, 3), x = ldv(a.target, e, 4), y = ldv(a.target, e, 5), z = ldv(a.target, e, 6);
  const double n2 = w * w + x * x + y * y + z * z;
  ok = ok && n2 > 0.999 && n2 < 1.001 && bfp_fits(pt.x) && bfp_fits(pt.y) && bfp_fits(pt.z);
  M3 Rl;
  for (int k = 0; k < 9; k++) Rl.a[k] = L.R[k];
  const M3 Rd = sgdyn::mul(quat_to_R(x, y, z, w), transpose(Rl));
  const V3 pd = pt - sgdyn::mul(Rd, mk(L.p[0], L.p[1], L.p[2]));
  Rot Rdes;
#pragma unroll
  for (int k = 0; k < 9; k++) Rdes.a[k] = q60(Rd.a[k]);
  const Vec pdes = from_doubles(pd.x, pd.y, pd.z);
  unsigned long long active = 0;  // by place on the path from the root
#pragma unroll 1
  for (int d = 0; d < depth; d++) {
    const int m = a.has_mask ? a.mask[JT[chain[depth - 1 - d]].vcol] : 1;
    ok = ok && (m == 0 || m == 1);
    if (m) active |= 1ull << d;
  }
  if (!ok) return false;
  // headroom for sums over the columns: 2 |h| |l| depth < 2^63
  const int room = depth > 3 ? 30 - clz32(unsigned(depth)) : 0;
  double minErr = 1e10;
  Mot bestErr{mk(0, 0, 0), mk(0, 0, 0)};
  bool done = false;
  Vec u[MAXJ], p[MAXJ];  // by place on the path; then the columns (linear, angular) of J2
#pragma unroll 1
  for (int it = 0;; it++) {
    Rot R = identity();
    Vec o = vec0();
#pragma unroll 1
    for (int d = 0; d < depth; d++) {
      const int i = chain[depth - 1 - d];
      const DJoint& J = JT[i];
      const BJoint& B = BT[i];
      o = norm(add(norm(mul(R, Vec{B.p[0], B.p[1], B.p[2], B.pe})), o));
      if (!(J.flags & JF_ROT_IDENTITY)) R = mul(R, rot_of(B.R));
      const Vec ax = J.axis_kind == AX_Z ? col_vec(R, 2)
                                         : norm(mul(R, Vec{B.axis[0], B.axis[1], B.axis[2], -60}));
      u[d] = ax;
      if (J.kind == JK_PRISMATIC) {
        o = norm(add(norm(mul(from_double(qs[i]), ax)), o));
      } else {
        i64 s, c;
        if (J.kind == JK_CONTINUOUS) {
          s = q60(qs[i]);
          c = q60(qc[i]);
        } else {
          sincos60(qs[i], &s, &c);
        }
        if (J.axis_kind == AX_Z) {
          const Half4 hs = split4(s), hc = split4(c), ns = neg(hs);
#pragma unroll
          for (int r = 0; r < 3; r++) {
            const Half4 b0 = split4(R.a[3 * r]), b1 = split4(R.a[3 * r + 1]);
            R.a[3 * r] = mul60(hc, b0, hs, b1);
            R.a[3 * r + 1] = mul60(hc, b1, ns, b0);
          }
        } else {
          R = mul(R, rodrigues(B.axis[0], B.axis[1], B.axis[2], s, c));
        }
      }
      p[d] = o;
    }
    // err = log6(Ro^T Rdes, Ro^T (pdes - po))
    Mot err;
    double th;
    {
      Rot Rt, Re;
#pragma unroll
      for (int k = 0; k < 9; k++) Rt.a[k] = R.a[(k % 3) * 3 + k / 3];
      Re = mul(Rt, Rdes);
      const Vec pe = norm(mul(Rt, norm(add(pdes, neg(o)))));
      const V3 pv = mk(to_double(pe.x, pe.e), to_double(pe.y, pe.e), to_double(pe.z, pe.e));
      double q[4];
      rot_quat(Re, q);
      if (q[0] < 0) {
#pragma unroll
        for (int k = 0; k < 4; k++) q[k] = -q[k];
      }
      const double nn = q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
      V3 om = mk(0, 0, 0);
      th = 0;
      if (nn > 1e-100) {
        const double in = inverse_sqrt(nn), n = nn * in;
        th = 2 * atan2(n, q[0]);
        const double k = th * in;
        om = mk(k * q[1], k * q[2], k * q[3]);
      }
      const double beta = se3_f_g(th), alpha = 1 - th * th * beta;
      const V3 wxp = sgdyn::cross(om, pv);
      const double wp = beta * sgdyn::dot(om, pv);
      err.v = mk(alpha * pv.x - 0.5 * wxp.x + wp * om.x, alpha * pv.y - 0.5 * wxp.y + wp * om.y,
                 alpha * pv.z - 0.5 * wxp.z + wp * om.z);
      err.w = om;
    }
    const double nrm = sqrt(dot6(err, err));
    if (!(nrm < 1e60) || (it == 0 && nrm < kIkSmall)) return false;
    if (nrm < minErr) {
      minErr = nrm;
      bestErr = err;
#pragma unroll 1
      for (int i = 1; i < nj; i++) {
        best[i] = qs[i];
        bestc[i] = qc[i];
      }
    }
    if (nrm < a.eps) {
      done = true;
      break;
    }
    if (it >= a.max_iter) break;
    // K1 = Jinv Ro^T, K2 = Jinv Q Jinv Ro^T for Jlog6 at -err (jlog6_blocks)
    Mat K1, K2;
    {
      const V3 rho = -err.v, phi = -err.w;
      const double t2 = th * th, dd = sgdyn::dot(phi, rho);
      const double g = se3_f_g(th), fa = se3_f_tms(th), fb = se3_f_c4(th), fc = se3_f_c5(th);
      const double f[3] = {phi.x, phi.y, phi.z}, r[3] = {rho.x, rho.y, rho.z};
      const V3 fxr = sgdyn::cross(phi, rho);
      const double uu[3] = {fxr.x, fxr.y, fxr.z};
      const double Kf[9] = {0, -phi.z, phi.y, phi.z, 0, -phi.x, -phi.y, phi.x, 0};
      const double Kr[9] = {0, -rho.z, rho.y, rho.z, 0, -rho.x, -rho.y, rho.x, 0};
      const double kf = dd * (fa - fb), cc = 2 * fc * dd;
      double Ji[9], Q[9];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const double id = i == k ? 1.0 : 0.0;
          const double pp = f[i] * f[k] - t2 * id;
          Ji[i * 3 + k] = id + 0.5 * Kf[i * 3 + k] + g * pp;
          Q[i * 3 + k] = -0.5 * Kr[i * 3 + k] + fa * (r[i] * f[k] + f[i] * r[k] - 2 * dd * id) + kf * Kf[i * 3 + k] +
                         fb * (f[i] * uu[k] - uu[i] * f[k]) - cc * pp;
        }
      const Mat mj = mat_from(Ji), mq = mat_from(Q);
      K1 = mul_mat<true>(mj.a, mj.e, R.a, -60);
      const Mat jq = mul_mat<false>(mj.a, mj.e, mq.a, mq.e);
      K2 = mul_mat<false>(jq.a, jq.e, K1.a, K1.e);
    }
    // columns of J2, and the largest exponents
    int et = -4000, eb = -4000;
#pragma unroll 1
    for (int d = 0; d < depth; d++) {
      Vec top = vec0(), bot = vec0();
      if (active >> d & 1) {
        const H3 hu = split(u[d]);
        if (JT[chain[depth - 1 - d]].kind == JK_PRISMATIC) {
          top = norm(mul(K1, hu, u[d].e));
        } else {
          const Vec c = norm(cross(u[d], norm(add(o, neg(p[d])))));
          top = norm(addp(mul(K1, split(c), c.e), neg(mul(K2, hu, u[d].e))));
          bot = norm(mul(K1, hu, u[d].e));
        }
      }
      u[d] = neg(top);
      p[d] = neg(bot);
      et = imax(et, top.e);
      eb = imax(eb, bot.e);
    }
    // J2 J2^T: cross and high terms of the 21 entries, rows (top, bottom)
    et += room;
    eb += room;
    i64 cs[21], hs[21];
#pragma unroll
    for (int k = 0; k < 21; k++) {
      cs[k] = kRound;
      hs[k] = 0;
    }
#pragma unroll 1
    for (int d = 0; d < depth; d++) {
      const H3 t = split(at_exp(u[d], et)), b = split(at_exp(p[d], eb));
      const Half r[6] = {t.x, t.y, t.z, b.x, b.y, b.z};
#pragma unroll
      for (int i = 0; i < 6; i++)
#pragma unroll
        for (int k = 0; k <= i; k++) {
          const int s = i * (i + 1) / 2 + k;
          cs[s] = cross_terms(r[i], r[k], cs[s]);
          hs[s] = wide(r[i].h, r[k].h, hs[s]);
        }
    }
    double A[21];
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
      for (int k = 0; k <= i; k++) {
        const int s = i * (i + 1) / 2 + k;
        A[s] = to_double(hs[s] + (cs[s] >> 32), (i < 3 ? et : eb) + (k < 3 ? et : eb) + 64) + (i == k ? a.damp : 0.0);
      }
    // (J2 J2^T + damp) x = err, Cholesky with reciprocal diagonals
#pragma unroll
    for (int j = 0; j < 6; j++) {
      double d = A[j * (j + 1) / 2 + j];
#pragma unroll
      for (int k = 0; k < j; k++) d = fma(-A[j * (j + 1) / 2 + k], A[j * (j + 1) / 2 + k], d);
      if (!(d > 1e-60 && d < 1e60)) return false;
      const double inv = inverse_sqrt(d);
      A[j * (j + 1) / 2 + j] = inv;
#pragma unroll
      for (int i = j + 1; i < 6; i++) {
        double s = A[i * (i + 1) / 2 + j];
#pragma unroll
        for (int k = 0; k < j; k++) s = fma(-A[i * (i + 1) / 2 + k], A[j * (j + 1) / 2 + k], s);
        A[i * (i + 1) / 2 + j] = s * inv;
      }
    }
    double xs[6] = {err.v.x, err.v.y, err.v.z, err.w.x, err.w.y, err.w.z};
#pragma unroll
    for (int i = 0; i < 6; i++) {
#pragma unroll
      for (int k = 0; k < i; k++) xs[i] = fma(-A[i * (i + 1) / 2 + k], xs[k], xs[i]);
      xs[i] *= A[i * (i + 1) / 2 + i];
    }
#pragma unroll
    for (int i = 5; i >= 0; i--) {
#pragma unroll
      for (int k = i + 1; k < 6; k++) xs[i] = fma(-A[k * (k + 1) / 2 + i], xs[k], xs[i]);
      xs[i] *= A[i * (i + 1) / 2 + i];
    }
    // v = -J2^T x, joints by v dt
    const Tw X{from_doubles(xs[0], xs[1], xs[2]), from_doubles(xs[3], xs[4], xs[5])};
#pragma unroll 1
    for (int d = 0; d < depth; d++) {
      const int i = chain[depth - 1 - d];
      const double v = -to_double(dot(Tw{u[d], p[d]}, X)) * a.dt;
      if (JT[i].kind == JK_CONTINUOUS) {
        double sw, cw;
        sincos(v, &sw, &cw);
        const double nc = cw * qc[i] - sw * qs[i], ns = sw * qc[i] + cw * qs[i];
        const double k = (3 - (nc * nc + ns * ns)) / 2;
        qc[i] = nc * k;
        qs[i] = ns * k;
      } else {
        qs[i] += v;
        if (!bfp_fits(qs[i])) return false;
      }
    }
  }
  double moved = 0.0;
#pragma unroll 1
  for (int i = 1; i < nj; i++) moved = fmax(moved, fabs(best[i]));
  if (moved != 0.0 && moved < kIkSmall) return false;
#pragma unroll 1
  for (int i = 1; i < nj; i++)
    stv(a.q_out, e, JT[i].qcol, JT[i].kind == JK_CONTINUOUS ? atan2(best[i], bestc[i]) : best[i]);
  a.success[e] = done ? 1 : 0;
  if (L.joint > 0) {  // reported in the model's joint frame
    M3 C;
    for (int k = 0; k < 9; k++) C.a[k] = model_frames(model)[L.joint].C[k];
    bestErr.v = sgdyn::mul(C, bestErr.v);
    bestErr.w = sgdyn::mul(C, bestErr.w);
  }
  const double o6[6] = {bestErr.v.x, bestErr.v.y, bestErr.v.z, bestErr.w.x, bestErr.w.y, bestErr.w.z};
#pragma unroll
  for (int k = 0; k < 6; k++) stv(a.err, e, k, o6[k]);
  return true;
}

}  // namespace bfp

template <int MAXJ>
static __device__ __noinline__ void ik_env_fp64(const DModel* __restrict__ model, const IkArgs& a, int64_t e) {
  ik_env<MAXJ>(model, a, e);
}

template <int MAXJ, int BLOCKS>
__global__ void __launch_bounds__(32, BLOCKS) bfp_ik_kernel(const DModel* __restrict__ model, const IkArgs a) {
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < a.n; e += int64_t(gridDim.x) * blockDim.x)
    if (!bfp::ik_env<MAXJ>(model, a, e)) ik_env_fp64<MAXJ>(model, a, e);
}

// 168 registers hold all of an iteration, 12 warps per multiprocessor; batches beyond those take
// the kernel of 144 registers and 14 warps, which costs a few spills and saves rounds (9-DoF
// arms, 100 iterations: 65536 environments 10.1 -> 8.5 ms, but 30000: 4.8 -> 5.1 ms).
template <int MAXJ>
cudaError_t launch_bfp_ik(const DModel* dm, const IkArgs& a, cudaStream_t s) {
  const bool all_resident = (a.n + 31) / 32 <= 12 * int64_t(multiprocessors());
  return launch_ik_kernel(all_resident ? bfp_ik_kernel<MAXJ, 12> : bfp_ik_kernel<MAXJ, 14>, dm, a, s);
}

}  // namespace sgdyn
