// Differentiable dynamics with a block of threads per group of environments (bfp_block.cuh):
// rollouts, their reverse pass, and the vector-Jacobian products of RNEA and forward dynamics.
//
// The recursions are those of diff_core.cuh (world-frame RNEA adjoint; lambda = M^-1 qdd_bar and
// the RNEA adjoint at lambda for forward dynamics) in block floating point, with FP64 as the
// second algebra for environments out of its range. The adjoint's subtree sums reduce to two
// wrenches per joint, P = sum Y w and X = sum (v x* Y w - w x* Y v - Y (v x w)):
//   qbar_c  = S_c . (v_p x* (v_p x* P - X) - a_p x* P - w_p x* F)
//   qdbar_c = S_c . (X - (v_p + v_j) x* P),   qddbar_c = S_c . P       (p: the joint's parent).
//
// A rollout keeps its state in shared memory for all steps. Its reverse pass takes from a replay
// of every checkpoint segment, all segments side by side, only q, qd, qdd and the factor of M per
// step (72 doubles for a 9-DoF arm, where the FP64 reverse sweep reads 493) and rebuilds the
// rest, which costs less than the memory traffic and the serial loads did.
//
// Measured (before: the FP64 kernels, specialised per model): values and gradients of inverse and
// forward dynamics, 16384 9-DoF arms, 720 -> 605 us; a rollout of 4096 of them over 200 steps with
// a checkpoint every 20 and its reverse pass, 29.9 -> 19.4 ms (6.3 forward, of the rest two
// thirds the reverse pass). What bounds them: instruction issue between barriers, the reverse
// pass besides by its 4096 environments, one block and a bit per multiprocessor.
#pragma once
#include "bfp_block.cuh"
#include "diff_kernels.cuh"

namespace sgdyn {
namespace bfp {

// Doubles per environment and step that the reverse pass reads: q, qd, qdd (external order), then
// the factor of M by pairs, 1 / D on the diagonal. [field][environment].
SG_HD int64_t blk_record_doubles(int nv, int nq, int npairs) { return nq + 2 * int64_t(nv) + npairs; }

#ifdef __CUDACC__
// (a call of its own: rare, long FP64 code whose registers the sweeps should not carry)
static __device__ __noinline__ void ff_integrate_adjoint(const double* d, double dt, double* g, double* vb) {
  Mot v{mk(vb[0], vb[1], vb[2]), mk(vb[3], vb[4], vb[5])};
  const Mot q = free_flyer_integrate_adjoint(Mot{mk(d[0], d[1], d[2]), mk(d[3], d[4], d[5])},
                                             Mot{mk(g[0], g[1], g[2]), mk(g[3], g[4], g[5])}, dt, v);
  g[0] = q.v.x; g[1] = q.v.y; g[2] = q.v.z; g[3] = q.w.x; g[4] = q.w.y; g[5] = q.w.z;
  vb[0] = v.v.x; vb[1] = v.v.y; vb[2] = v.v.z; vb[3] = v.w.x; vb[4] = v.w.y; vb[5] = v.w.z;
}

// 1 / D of column c after blk_solve.
template <class A, int E, int EI>
__device__ __forceinline__ double blk_inverse_pivot(const Blk<A, E, EI>& b, int c) {
  const int i = b.L.A + b.row_start[c] + b.depth[c];
  if constexpr (A::kFixed) return to_double(b.W(i), 2 * b.X(b.L.xs + b.nv + c) - 58 - 2 * b.X(b.L.xs + c));
  else return b.D(i);
}
// Semi-implicit Euler on the inputs in shared memory with qdd at b + nv, in two parts with a
// barrier between: velocities, then coordinates.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_integrate_velocity(const Blk<A, E, EI>& b, double dt) {
  if (b.col < 0) return;
  const int x = b.ext[b.col];
  b.set_in(b.nq + x, fma(dt, b.D(b.L.b + b.nv + b.col), b.qd(x)));
}
template <class A, int E, int EI>
__device__ __forceinline__ void blk_integrate_position(const Blk<A, E, EI>& b, double dt) {
  if (!b.j) return;
  const DJoint& J = b.J[b.j];
  if (J.kind == JK_FREEFLYER) {
    double q[7], d[6];
    for (int k = 0; k < 7; k++) q[k] = b.q(J.qcol + k);
    for (int k = 0; k < 6; k++) d[k] = b.qd(J.vcol + k);
    free_flyer_step(q, d, dt);
    for (int k = 0; k < 7; k++) b.set_in(J.qcol + k, q[k]);
  } else {
    b.set_in(J.qcol, fma(dt, b.qd(J.vcol), b.q(J.qcol)));
  }
}
// A row of an env-major state into the inputs.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_load_row(const Blk<A, E, EI>& b, int at, const double* row, int cols) {
#pragma unroll 1
  for (int c = b.slot; c < cols; c += b.slots) b.set_in(at + c, row[c]);
}

// The environments of the block that refused, from every thread of it.
template <int E>
__device__ __forceinline__ unsigned blk_refused_set(Blk<BfpAlg, E>& b) {
  unsigned which = 0;
  const int el = b.el;
  for (int k = 0; k < b.count; k++) {
    b.el = k;
    which |= unsigned(b.refused()) << k;
  }
  b.el = el;
  return which;
}
// Steps t0 to t1 - 1 of the block's environments, whose q and qd are among the inputs; per step
// record(block state, t) before it and after(block state, t) when qdd is at b + nv. A step in FP64
// for the environments that refuse it alone: the next one is asked again.
template <int E, class R, class F>
__device__ __forceinline__ void blk_steps(Blk<BfpAlg, E>& b, const DModel* model, long long* smem, const RolloutArgs& a,
                                          int64_t e, int t0, int t1, const R& record, const F& after) {
  const int nq = b.nq, nv = b.nv;
  __syncthreads();
#pragma unroll 1
  for (int t = t0; t < t1; t++) {
    record(b, t);
    const double* tau = a.tau + (int64_t(t) * a.n + e) * nv;
#pragma unroll 1
    for (int c = b.slot; c < nv; c += b.slots) {
      blk_in(b, nq + 2 * nv + c, tau[c]);
      if (!bfp_fits(b.qd(c))) b.refuse();
    }
#pragma unroll 1
    for (int c = b.slot; c < nq; c += b.slots)
      if (!bfp_fits(b.q(c))) b.refuse();
    __syncthreads();
    b.clear_notes(b.set ^ 1);
    blk_poses(b);
    const bool none = __syncthreads_and(b.note_at(b.set, NOTE_REFUSED));
    if (!none) {
      blk_forward_dynamics(b);
      after(b, t);
      if (!b.refused()) blk_integrate_velocity(b, a.dt);
    }
    const bool some = __syncthreads_or(none || b.refused());
    if (!none && !b.refused()) blk_integrate_position(b, a.dt);
    if (some) {
      const unsigned which = blk_refused_set(b);
      if (which) {
        Blk<FpAlg, 0, E> f;
        f.init_some(model, smem, which, b.set);
        blk_poses(f);
        blk_forward_dynamics(f);
        after(f, t);
        if (f.valid) blk_integrate_velocity(f, a.dt);
        __syncthreads();
        if (f.valid) blk_integrate_position(f, a.dt);
      }
    }
    b.set ^= 1;
    __syncthreads();
  }
}

template <int E>
__device__ __forceinline__ void blk_rollout(Blk<BfpAlg, E>& b, const DModel* model, long long* smem,
                                            const RolloutArgs& a, int64_t e) {
  const int64_t n = a.n;
  const int nq = b.nq, nv = b.nv;
  blk_load_row(b, 0, a.q0 + e * nq, nq);
  blk_load_row(b, nq, a.qd0 + e * nv, nv);
  auto put = [&](double* q, double* qd) SG_INLINE {
    if (!b.valid) return;
#pragma unroll 1
    for (int c = b.slot; c < nq; c += b.slots) q[e * nq + c] = b.q(c);
#pragma unroll 1
    for (int c = b.slot; c < nv; c += b.slots) qd[e * nv + c] = b.qd(c);
  };
  blk_steps(
      b, model, smem, a, e, 0, a.T,
      [&](const auto&, int t) SG_INLINE {
        if (a.q_ckpt && t % a.K == 0) put(a.q_ckpt + int64_t(t / a.K) * n * nq, a.qd_ckpt + int64_t(t / a.K) * n * nv);
      },
      [](const auto&, int) {});
  put(a.qT, a.qdT);
}

// One segment: its steps' records into the scratch ([segment of group][step][field][env]).
template <int E>
__device__ __forceinline__ void blk_replay(Blk<BfpAlg, E>& b, const DModel* model, long long* smem,
                                           const RolloutArgs& a, int g, int64_t e0, int64_t e) {
  const int64_t n = a.n;
  const int nq = b.nq, nv = b.nv, s = a.s_lo + g;
  const int64_t rec = blk_record_doubles(nv, nq, b.npairs);
  blk_load_row(b, 0, a.q_ckpt + (int64_t(s) * n + e) * nq, nq);
  blk_load_row(b, nq, a.qd_ckpt + (int64_t(s) * n + e) * nv, nv);
  const int t0 = s * a.K, t1 = min(a.T, t0 + a.K);
  auto base = [&](const auto& c, int t) SG_INLINE {
    return a.scratch + (int64_t(g) * a.K + (t - t0)) * rec * n + e0 + c.el;
  };
  blk_steps(
      b, model, smem, a, e, t0, t1,
      [&](const auto& b, int t) SG_INLINE {
        if (!b.valid) return;
        double* o = base(b, t);
#pragma unroll 1
        for (int c = b.slot; c < nq + nv; c += b.slots) o[c * n] = b.in(c);
      },
      [&](const auto& b, int t) SG_INLINE {
        if (!b.valid) return;
        double* o = base(b, t) + (nq + nv) * n;
        if (b.col >= 0) {
          o[b.ext[b.col] * n] = b.D(b.L.b + nv + b.col);
          o[int64_t(nv + b.row_start[b.col] + b.depth[b.col]) * n] = blk_inverse_pivot(b, b.col);
        }
#pragma unroll 1
        for (int i = b.slot; i < b.npairs; i += b.slots)
          if (b.pair_row[i] != b.pair_col[i]) o[int64_t(nv + i) * n] = b.D(b.L.S + i);
      });
}

// x = M^-1 b for the factor in Y's items (1 / D on the diagonal), b at L.b, x after it.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_factor_solve(const Blk<A, E, EI>& b) {
  const int nv = b.nv, c = b.col;
  const int dc = c >= 0 ? b.depth[c] : 0, rc = c >= 0 ? b.row_start[c] : 0;
  double y = c >= 0 ? b.D(b.L.b + c) : 0.0;  // L^T y = b, deepest columns first
#pragma unroll 1
  for (int d = b.col_levels - 1; d >= 1; d--) {
    // columns of depth d are final; their ancestors take them, a column's descendants in order
    const int lo = b.col_level_start[d], hi = b.col_level_start[d + 1];
    if (c >= 0 && dc < d) {
#pragma unroll 1
      for (int k = lo; k < hi; k++) {
        const int a = b.col_order[k], i = b.row_start[a] + dc;
        if (b.pair_col[i] == c) y = fma(-b.D(b.L.Y + i), b.D(b.L.b + a), y);
      }
      if (dc == d - 1) b.setD(b.L.b + c, y);
    }
    __syncthreads();
  }
  double x = c >= 0 ? y * b.D(b.L.Y + rc + dc) : 0.0;
  if (c >= 0) b.setD(b.L.b + nv + c, x);
  __syncthreads();
#pragma unroll 1
  for (int d = 0; d + 1 < b.col_levels; d++) {
    if (c >= 0 && dc > d) {
      x = fma(-b.D(b.L.Y + rc + d), b.D(b.L.b + nv + b.pair_col[rc + d]), x);
      if (dc == d + 1) b.setD(b.L.b + nv + c, x);
    }
    __syncthreads();
  }
}

// RNEA adjoint at the inputs q, qd, qdd in shared memory and the poses, for the adjoint lam (tree
// columns) at b + nv: out(column, qbar, qdbar, qddbar), unscaled.
template <class A, int E, int EI, class F>
__device__ __forceinline__ void blk_rnea_adjoint(const Blk<A, E, EI>& b, const F& out) {
  typedef typename A::Tw Tw;
  blk_columns(b, true);
  blk_motion_forces(b, true, false);
  blk_subtrees(b, true, false);
  // w = sum of lam S from the root, into u
  Tw w{};
  if (b.j) w = joint_motion(b, [&](int c, int) SG_INLINE { return b.D(b.L.b + b.nv + c); });
  blk_from_root(b, w, [&](int j) SG_INLINE { return b.L.u + 6 * (j - 1); },
                [&](int j) SG_INLINE { return b.L.xu + 2 * (j - 1); });
  // P and X, in the place of the inertias
  const int iY = b.L.Y + 12 * (b.j - 1), xY = b.L.xu + 2 * (b.nj - 1) + 4 * (b.j - 1);
  Tw P{}, X{}, v{};
  if (b.j) {
    v = b.V(b.j - 1);
    const typename A::Rbi Y = b.rbi(b.j);
    P = norm(mul(Y, w));
    X = norm(add(crossf(w, norm(mul(Y, v))), mul(Y, norm(crossm(v, w)))));
    X = norm(add(norm(crossf(v, P)), neg(X)));
  }
  __syncthreads();  // every inertia has been read
  if (b.j) {
    b.put(iY, xY, P);
    b.put(iY + 6, xY + 2, X);
  }
  __syncthreads();
  // sums over subtrees
  const int end = b.end[b.j];
#pragma unroll 1
  for (int d = b.levels - 1; d >= 1; d--) {
    if (b.j && end > b.j + 1 && b.lv == d) {
#pragma unroll 1
      for (int k = b.j + 1; k < end; k = b.end[k]) {
        const int i = b.L.Y + 12 * (k - 1), x = b.L.xu + 2 * (b.nj - 1) + 4 * (k - 1);
        P = norm(add(P, b.tw(i, x)));
        X = norm(add(X, b.tw(i + 6, x + 2)));
      }
      b.put(iY, xY, P);
      b.put(iY + 6, xY + 2, X);
    }
    __syncthreads();
  }
  if (b.j) {
    const DJoint& J = b.J[b.j];
    Tw G{}, terms{};
    const bool root = b.p == 0;
    if (root) {  // G = v_p x* (v_p x* P - X) - a_p x* P - w_p x* F
      Tw a{};
      a.v = A::vec(-b.g[0], -b.g[1], -b.g[2]);
      a.w = A::vec(0, 0, 0);
      const Tw t = crossf(a, P);
      if constexpr (A::kFixed) terms = t;
      G = norm(neg(t));
    } else {
      const Tw vp = b.V(b.p - 1), wp = b.tw(b.L.u + 6 * (b.p - 1), b.L.xu + 2 * (b.p - 1));
      const Tw t = crossf(b.acc(b.p), P), u = crossf(wp, b.frc(b.j));
      G = norm(add(norm(crossf(vp, P)), neg(X)));
      G = norm(add(norm(crossf(vp, G)), neg(norm(t))));
      G = norm(add(G, neg(norm(u))));
      if constexpr (A::kFixed) terms = add(t, u);
      v = norm(add(vp, v));
    }
    if constexpr (A::kFixed) b.note(NOTE_GSCALE, 57 + (turns(J) ? terms.w.e : terms.v.e));
    const Tw Gd = norm(add(X, neg(norm(crossf(v, P)))));
#pragma unroll 1
    for (int k = 0; k < J.nv; k++) {
      const Tw S = b.S(J.ivx + k);
      const double gq = A::get(dot(S, G));
      b.note(NOTE_GRAD, gq);
      out(J.ivx + k, 0, gq);
      out(J.ivx + k, 1, A::get(dot(S, Gd)));
      out(J.ivx + k, 2, A::get(dot(S, P)));
    }
  }
  __syncthreads();
}

// One step of the reverse pass, record r of it (field stride n) and the state's adjoint (tangent
// layout, tree columns: q's then qd's) in the place of tau and on, replaced by that before the step.
// refused(): whether to leave it to another pass.
template <class A, int E, int EI, class P>
__device__ __forceinline__ void blk_reverse_step(const Blk<A, E, EI>& b, const RolloutArgs& a, const double* r,
                                                 double* tau_bar, const P& refused) {
  const int64_t n = a.n;
  const int nq = b.nq, nv = b.nv, c = b.col;
  const int jc = c >= 0 ? b.col_joint[c] : 1, x = c >= 0 ? b.ext[c] : 0;
  const bool ff = c >= 0 && b.J[jc].kind == JK_FREEFLYER;
  const int at = nq + 2 * nv + c;
  double qb = c >= 0 ? b.in(at) : 0.0, qdb = c >= 0 ? b.in(at + nv) : 0.0;
#pragma unroll 1
  for (int k = b.slot; k < nq + 2 * nv; k += b.slots) blk_in(b, k, r[k * n]);
#pragma unroll 1
  for (int k = b.slot; k < b.npairs; k += b.slots) b.setD(b.L.Y + k, r[(nq + 2 * nv + int64_t(k)) * n]);
  // q' = q (+) dt qd', qd' = qd + dt qdd, reversed
  if (c >= 0 && !ff) qdb = fma(a.dt, qb, qdb);
  if (ff) {  // the block of six at once: through b
    b.setD(b.L.b + c, qb);
    b.setD(b.L.b + nv + c, qdb);
  }
  __syncthreads();
  if (ff && b.col_dof[c] == 0) {
    double d[6], g[6], vb[6];
    for (int k = 0; k < 6; k++) {
      d[k] = a.dt * fma(a.dt, b.qdd(x + k), b.qd(x + k));  // the step's displacement
      g[k] = b.D(b.L.b + c + k);
      vb[k] = b.D(b.L.b + nv + c + k);
    }
    ff_integrate_adjoint(d, a.dt, g, vb);
    for (int k = 0; k < 6; k++) {
      b.setD(b.L.b + c + k, g[k]);
      b.setD(b.L.b + nv + c + k, vb[k]);
    }
  }
  __syncthreads();
  if (ff) {
    qb = b.D(b.L.b + c);
    qdb = b.D(b.L.b + nv + c);
  }
  if (c >= 0) b.setD(b.L.b + c, a.dt * qdb);
  __syncthreads();
  blk_factor_solve(b);  // lam at b + nv
  if (c >= 0) {
    const double lam = b.D(b.L.b + nv + c);
    if (!bfp_fits(lam)) b.refuse();
    if (b.valid) tau_bar[x] = lam;
  }
  blk_poses(b);
  blk_rnea_adjoint(b, [&](int col, int which, double v) SG_INLINE {
    if (which < 2) b.setD(b.L.b + (which == 0 ? 0 : nv) + col, v);
  });
  if (c >= 0 && !refused()) {
    b.set_in(at, qb - b.D(b.L.b + c));
    b.set_in(at + nv, qdb - b.D(b.L.b + nv + c));
  }
}

// In FP64 for the environments in `which` (a call of its own: inlined, its registers cost the
// reverse pass 330 more bytes of spills).
template <int E>
__device__ __noinline__ void blk_reverse_step_fp64(const DModel* model, long long* smem, unsigned which, int set,
                                                   const RolloutArgs a, const double* r, double* tau_bar) {
  Blk<FpAlg, 0, E> f;
  f.init_some(model, smem, which, set, true);
  blk_reverse_step(f, a, r + f.el, tau_bar + int64_t(f.el) * f.nv, [&]() SG_INLINE { return !f.valid; });
}
// Reverse pass of a group of segments, latest step first; a step in FP64 for the environments
// that refuse it.
template <int E>
__device__ __forceinline__ void blk_reverse(Blk<BfpAlg, E>& b, const DModel* model, long long* smem,
                                            const RolloutArgs& a, int64_t e0, int64_t e) {
  const int64_t n = a.n;
  const int nq = b.nq, nv = b.nv;
  const int64_t rec = blk_record_doubles(nv, nq, b.npairs);
  const int nseg = (a.T + a.K - 1) / a.K;
  const bool last = a.s_lo + a.s_cnt == nseg;
  const double* qin = last ? a.qT_bar : a.q0_bar;
  const double* qdin = last ? a.qdT_bar : a.qd0_bar;
  // this slot's column: q column of its coordinate in the adjoint's layout
  const int c = b.col;
  const int jc = c >= 0 ? b.col_joint[c] : 1, x = c >= 0 ? b.ext[c] : 0;
  const int qx = c >= 0 ? b.J[jc].qcol + b.col_dof[c] : 0;
  if (c >= 0) {
    b.set_in(nq + 2 * nv + c, qin ? qin[e * nq + qx] : 0.0);
    b.set_in(nq + 3 * nv + c, qdin ? qdin[e * nv + x] : 0.0);
  }
  __syncthreads();
#pragma unroll 1
  for (int s = a.s_lo + a.s_cnt - 1; s >= a.s_lo; s--) {
    const int t0 = s * a.K, t1 = min(a.T, t0 + a.K);
#pragma unroll 1
    for (int t = t1 - 1; t >= t0; t--) {
      const double* r = a.scratch + (int64_t(s - a.s_lo) * a.K + (t - t0)) * rec * n;
      double* tau_bar = a.tau_bar + int64_t(t) * n * nv;
      b.clear_notes(b.set ^ 1);
      blk_reverse_step(b, a, r + e, tau_bar + e * nv, [&]() SG_INLINE { return b.refused(); });
      if (__syncthreads_or(b.refused())) {
        if (const unsigned which = blk_refused_set(b))
          blk_reverse_step_fp64<E>(model, smem, which, b.set, a, r + e0, tau_bar + e0 * nv);
      }
      b.set ^= 1;
      __syncthreads();
    }
  }
  if (c >= 0 && b.valid) {
    a.q0_bar[e * nq + qx] = b.in(nq + 2 * nv + c);
    a.qd0_bar[e * nv + x] = b.in(nq + 3 * nv + c);
    if (b.J[jc].kind == JK_FREEFLYER && b.col_dof[c] == 0) a.q0_bar[e * nq + qx + 6] = 0.0;
  }
}
#endif  // __CUDACC__

}  // namespace bfp

#ifdef __CUDACC__
template <int E>
__global__ void __launch_bounds__(bfp::kBlkDiffThreads) bfp_rollout_kernel(const DModel* __restrict__ model,
                                                                         const RolloutArgs a) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  bfp::Blk<bfp::BfpAlg, E> b;
  b.init(model, smem, envs);
  bfp::blk_rollout(b, model, smem, a, e0 + min(b.el, envs - 1));
}
template <int E>
__global__ void __launch_bounds__(bfp::kBlkDiffThreads) bfp_replay_kernel(const DModel* __restrict__ model,
                                                                        const RolloutArgs a) {
  extern __shared__ __align__(16) long long smem[];
  // segment after segment in one grid dimension: there may be more of them than the others hold
  const unsigned per_segment = unsigned((a.n + E - 1) / E), g = blockIdx.x / per_segment;
  const int64_t e0 = int64_t(blockIdx.x - g * per_segment) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  bfp::Blk<bfp::BfpAlg, E> b;
  b.init(model, smem, envs);
  bfp::blk_replay(b, model, smem, a, int(g), e0, e0 + min(b.el, envs - 1));
}
template <int E>
__global__ void __launch_bounds__(bfp::kBlkDiffThreads) bfp_reverse_kernel(const DModel* __restrict__ model,
                                                                         const RolloutArgs a) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  bfp::Blk<bfp::BfpAlg, E> b;
  b.init(model, smem, envs, true);
  bfp::blk_reverse(b, model, smem, a, e0, e0 + min(b.el, envs - 1));
}

// The inputs of a vector-Jacobian product, the third among them at item x and the adjoint at item
// bar: all of them, as results may lie where the arguments do.
template <int E>
__device__ __forceinline__ void vjp_load(const bfp::Blk<bfp::BfpAlg, E>& b, const VjpArgs& a, int x, int bar,
                                         int64_t e) {
#pragma unroll 1
  for (int c = b.slot; c < b.nq; c += b.slots) bfp::blk_in(b, c, ldv(a.q, e, c));
#pragma unroll 1
  for (int c = b.slot; c < b.nv; c += b.slots) {
    bfp::blk_in(b, b.nq + c, ldv(a.qd, e, c));
    bfp::blk_in(b, x + c, ldv(a.x, e, c));
    b.set_in(bar + c, ldv(a.bar, e, c));
  }
  __syncthreads();
}
// Vector-Jacobian product of RNEA.
template <int E>
__global__ void __launch_bounds__(bfp::kBlkDiffThreads) bfp_rnea_vjp_kernel(const DModel* __restrict__ model,
                                                                          const VjpArgs a) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  blk_run<E>(
      model, smem, true, envs, bfp::kLost,
      [&](const auto& b) SG_INLINE { vjp_load(b, a, b.nq + b.nv, b.nq + 2 * b.nv, e0 + min(b.el, envs - 1)); },
      [&](const auto& b) SG_INLINE {
        const int64_t e = e0 + b.el;
        if (b.col >= 0) {
          const double v = b.tau(b.ext[b.col]);  // the adjoint
          if (!bfp::bfp_fits(v)) b.refuse();
          b.setD(b.L.b + b.nv + b.col, v);
        }
        __syncthreads();
        bfp::blk_rnea_adjoint(b, [&](int c, int which, double v) SG_INLINE {
          const Arr& o = which == 0 ? a.o1 : which == 1 ? a.o2 : a.o3;
          if (b.valid && o.p) stv(o, e, b.ext[c], v);
        });
      });
}
// Vector-Jacobian product of forward dynamics.
template <int E>
__global__ void __launch_bounds__(bfp::kBlkDiffThreads) bfp_aba_vjp_kernel(const DModel* __restrict__ model,
                                                                         const VjpArgs a) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  blk_run<E>(
      model, smem, true, envs, bfp::kLost,
      [&](const auto& b) SG_INLINE { vjp_load(b, a, b.nq + 2 * b.nv, b.nq + 3 * b.nv, e0 + min(b.el, envs - 1)); },
      [&](const auto& b) SG_INLINE {
        const int64_t e = e0 + b.el;
        const int nv = b.nv;
        bfp::blk_forward_dynamics(b);
        const int c = b.col, x = c >= 0 ? b.ext[c] : 0;
        // qdd joins the inputs; the factor moves to Y's items; the right-hand side becomes the adjoint
        if (c >= 0) {
          const int i = b.row_start[c] + b.depth[c];
          bfp::blk_in(b, b.nq + nv + x, b.D(b.L.b + nv + c));
          b.setD(b.L.Y + i, bfp::blk_inverse_pivot(b, c));
        }
#pragma unroll 1
        for (int i = b.slot; i < b.npairs; i += b.slots)
          if (b.pair_row[i] != b.pair_col[i]) b.setD(b.L.Y + i, b.D(b.L.S + i));
        if (c >= 0) b.setD(b.L.b + c, b.in(b.nq + 3 * nv + x));
        __syncthreads();
        bfp::blk_factor_solve(b);
        const double lam = c >= 0 ? b.D(b.L.b + nv + c) : 0.0;
        if (!bfp::bfp_fits(lam)) b.refuse();
        bfp::blk_poses(b);
        bfp::blk_rnea_adjoint(b, [&](int col, int which, double v) SG_INLINE {
          const Arr& o = which == 0 ? a.o1 : a.o2;
          if (which < 2 && b.valid && o.p) stv(o, e, b.ext[col], -v);
        });
        if (c >= 0 && b.valid && a.o3.p) stv(a.o3, e, x, lam);
      });
}
#endif

}  // namespace sgdyn
