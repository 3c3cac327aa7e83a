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
// a checkpoint every 20 and its reverse pass, 29.9 -> 19.05 ms (6.2 forward, of the rest two
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

// Whether the environment is left to the FP64 pass that follows: its results are not written,
// they may lie where that pass reads its inputs.
template <class A, int E>
__device__ __forceinline__ bool blk_refused(const Blk<A, E>& b) {
  return A::kFixed && b.X(b.L.ints - 1) != 0;
}
// 1 / D of column c after blk_solve.
template <class A, int E>
__device__ __forceinline__ double blk_inverse_pivot(const Blk<A, E>& b, int c) {
  const int i = b.L.A + b.row_start[c] + b.depth[c];
  if constexpr (A::kFixed) return to_double(b.W(i), 2 * b.X(b.L.xs + b.nv + c) - 58 - 2 * b.X(b.L.xs + c));
  else return b.D(i);
}
// Semi-implicit Euler on the inputs in shared memory with qdd at b + nv.
template <class A, int E>
__device__ __forceinline__ void blk_integrate(const Blk<A, E>& b, double dt) {
  if (b.col >= 0) {
    const int x = b.ext[b.col];
    blk_in(b, b.nq + x, fma(dt, b.D(b.L.b + b.nv + b.col), b.qd(x)));
  }
  __syncthreads();
  if (b.j) {
    const DJoint& J = b.J[b.j];
    if (J.kind == JK_FREEFLYER) {
      double q[7], d[6];
      for (int k = 0; k < 7; k++) q[k] = b.q(J.qcol + k);
      for (int k = 0; k < 6; k++) d[k] = b.qd(J.vcol + k);
      free_flyer_step(q, d, dt);
      for (int k = 0; k < 7; k++) blk_in(b, J.qcol + k, q[k]);
    } else {
      blk_in(b, J.qcol, fma(dt, b.qd(J.vcol), b.q(J.qcol)));
    }
  }
  __syncthreads();
}
// A row of an env-major state into the inputs.
template <class A, int E>
__device__ __forceinline__ void blk_load_row(const Blk<A, E>& b, int at, const double* row, int cols) {
#pragma unroll 1
  for (int c = b.slot; c < cols; c += b.slots) blk_in(b, at + c, row[c]);
}

// T steps (from step t0 on) for the block's environments; per step record(t) before it and
// after(t) when qdd is at b + nv.
template <class A, int E, class R, class F>
__device__ __forceinline__ void blk_steps(const Blk<A, E>& b, const RolloutArgs& a, int64_t e, int t0, int t1,
                                          const R& record, const F& after) {
  const int at = b.nq + 2 * b.nv;
#pragma unroll 1
  for (int t = t0; t < t1; t++) {
    record(t);
    blk_load_row(b, at, a.tau + (int64_t(t) * a.n + e) * b.nv, b.nv);
    __syncthreads();
    blk_forward_dynamics(b);
    after(t);
    blk_integrate(b, a.dt);
  }
}

template <class A, int E>
__device__ __forceinline__ void blk_rollout(const Blk<A, E>& b, const RolloutArgs& a, int64_t e, bool valid) {
  const int64_t n = a.n;
  const int nq = b.nq, nv = b.nv;
  blk_load_row(b, 0, a.q0 + e * nq, nq);
  blk_load_row(b, nq, a.qd0 + e * nv, nv);
  __syncthreads();
  blk_check_quaternion(b);
  auto put = [&](double* q, double* qd) SG_INLINE {
    if (!valid) return;
#pragma unroll 1
    for (int c = b.slot; c < nq; c += b.slots) q[e * nq + c] = b.q(c);
#pragma unroll 1
    for (int c = b.slot; c < nv; c += b.slots) qd[e * nv + c] = b.qd(c);
  };
  blk_steps(
      b, a, e, 0, a.T,
      [&](int t) SG_INLINE {
        if (a.q_ckpt && t % a.K == 0) put(a.q_ckpt + int64_t(t / a.K) * n * nq, a.qd_ckpt + int64_t(t / a.K) * n * nv);
      },
      [](int) {});
  if (!blk_refused(b)) put(a.qT, a.qdT);
}

// One segment: its steps' records into the scratch ([segment of group][step][field][env]).
template <class A, int E>
__device__ __forceinline__ void blk_replay(const Blk<A, E>& b, const RolloutArgs& a, int g, int64_t e, bool valid) {
  const int64_t n = a.n;
  const int nq = b.nq, nv = b.nv, s = a.s_lo + g;
  const int64_t rec = blk_record_doubles(nv, nq, b.npairs);
  blk_load_row(b, 0, a.q_ckpt + (int64_t(s) * n + e) * nq, nq);
  blk_load_row(b, nq, a.qd_ckpt + (int64_t(s) * n + e) * nv, nv);
  __syncthreads();
  blk_check_quaternion(b);
  const int t0 = s * a.K, t1 = min(a.T, t0 + a.K);
  auto base = [&](int t) SG_INLINE { return a.scratch + (int64_t(g) * a.K + (t - t0)) * rec * n + e; };
  blk_steps(
      b, a, e, t0, t1,
      [&](int t) SG_INLINE {
        if (!valid) return;
        double* o = base(t);
#pragma unroll 1
        for (int c = b.slot; c < nq + nv; c += b.slots) o[c * n] = b.D(b.L.in + c);
      },
      [&](int t) SG_INLINE {
        if (!valid) return;
        double* o = base(t) + (nq + nv) * n;
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
template <class A, int E>
__device__ __forceinline__ void blk_factor_solve(const Blk<A, E>& b) {
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

// RNEA adjoint at the inputs q, qd, qdd in shared memory for the adjoint lam (tree columns) at
// b + nv: out(column, qbar, qdbar, qddbar), unscaled.
template <class A, int E, class F>
__device__ __forceinline__ void blk_rnea_adjoint(const Blk<A, E>& b, const F& out) {
  typedef typename A::Tw Tw;
  blk_poses(b);
  blk_columns(b, true);
  blk_motion_forces(b, true);
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
    Tw G{};
    const bool root = b.p == 0;
    if (root) {  // G = v_p x* (v_p x* P - X) - a_p x* P - w_p x* F
      Tw a{};
      a.v = A::vec(-b.g[0], -b.g[1], -b.g[2]);
      a.w = A::vec(0, 0, 0);
      G = norm(neg(crossf(a, P)));
    } else {
      const Tw vp = b.V(b.p - 1), wp = b.tw(b.L.u + 6 * (b.p - 1), b.L.xu + 2 * (b.p - 1));
      G = norm(add(norm(crossf(vp, P)), neg(X)));
      G = norm(add(norm(crossf(vp, G)), neg(norm(crossf(b.acc(b.p), P)))));
      G = norm(add(G, neg(norm(crossf(wp, b.frc(b.j))))));
      v = norm(add(vp, v));
    }
    const Tw Gd = norm(add(X, neg(norm(crossf(v, P)))));
#pragma unroll 1
    for (int k = 0; k < J.nv; k++) {
      const Tw S = b.S(J.ivx + k);
      out(J.ivx + k, 0, A::get(dot(S, G)));
      out(J.ivx + k, 1, A::get(dot(S, Gd)));
      out(J.ivx + k, 2, A::get(dot(S, P)));
    }
  }
  __syncthreads();
}

// Reverse pass of a group of segments, latest step first. Each slot keeps its column's entries of
// the state's adjoint in registers (a free flyer's tangent block: six slots).
template <class A, int E>
__device__ __forceinline__ void blk_reverse(const Blk<A, E>& b, const RolloutArgs& a, int64_t e, bool valid) {
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
  const bool ff = c >= 0 && b.J[jc].kind == JK_FREEFLYER;
  double qb = c >= 0 && qin ? qin[e * nq + qx] : 0.0, qdb = c >= 0 && qdin ? qdin[e * nv + x] : 0.0;
  auto check = [&](double v) SG_INLINE {
    if (!bfp_fits(v)) b.refuse();
  };
#pragma unroll 1
  for (int s = a.s_lo + a.s_cnt - 1; s >= a.s_lo; s--) {
    const int t0 = s * a.K, t1 = min(a.T, t0 + a.K);
#pragma unroll 1
    for (int t = t1 - 1; t >= t0; t--) {
      const double* r = a.scratch + (int64_t(s - a.s_lo) * a.K + (t - t0)) * rec * n + e;
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
        check(lam);
        if (valid) a.tau_bar[(int64_t(t) * n + e) * nv + x] = lam;
      }
      blk_rnea_adjoint(b, [&](int col, int which, double v) SG_INLINE {
        if (which < 2) b.setD(b.L.b + (which == 0 ? 0 : nv) + col, v);
      });
      if (c >= 0) {
        qb -= b.D(b.L.b + c);
        qdb -= b.D(b.L.b + nv + c);
        check(qb);
        check(qdb);
      }
      __syncthreads();
    }
  }
  if (c >= 0 && valid && !blk_refused(b)) {
    a.q0_bar[e * nq + qx] = qb;
    a.qd0_bar[e * nv + x] = qdb;
    if (ff && b.col_dof[c] == 0) a.q0_bar[e * nq + qx + 6] = 0.0;
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
  blk_run<E>(model, smem, false, envs, [&](const auto& b, bool valid) SG_INLINE {
    bfp::blk_rollout(b, a, e0 + min(b.lane, envs - 1), valid);
  });
}
template <int E>
__global__ void __launch_bounds__(bfp::kBlkDiffThreads) bfp_replay_kernel(const DModel* __restrict__ model,
                                                                        const RolloutArgs a) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  blk_run<E>(model, smem, false, envs, [&](const auto& b, bool valid) SG_INLINE {
    bfp::blk_replay(b, a, int(blockIdx.y), e0 + min(b.lane, envs - 1), valid);
  });
}
template <int E>
__global__ void __launch_bounds__(bfp::kBlkDiffThreads) bfp_reverse_kernel(const DModel* __restrict__ model,
                                                                         const RolloutArgs a) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  blk_run<E>(model, smem, true, envs, [&](const auto& b, bool valid) SG_INLINE {
    bfp::blk_reverse(b, a, e0 + min(b.lane, envs - 1), valid);
  });
}

// Vector-Jacobian product of RNEA.
template <int E>
__global__ void __launch_bounds__(bfp::kBlkDiffThreads) bfp_rnea_vjp_kernel(const DModel* __restrict__ model,
                                                                          const VjpArgs a) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  blk_run<E>(model, smem, true, envs, [&](const auto& b, bool valid) SG_INLINE {
    const int64_t e = e0 + min(b.lane, envs - 1);
#pragma unroll 1
    for (int c = b.slot; c < b.nq; c += b.slots) bfp::blk_in(b, c, ldv(a.q, e, c));
#pragma unroll 1
    for (int c = b.slot; c < b.nv; c += b.slots) {
      bfp::blk_in(b, b.nq + c, ldv(a.qd, e, c));
      bfp::blk_in(b, b.nq + b.nv + c, ldv(a.x, e, c));
    }
    __syncthreads();
    bfp::blk_check_quaternion(b);
    if (b.col >= 0) {
      const double v = ldv(a.bar, e, b.ext[b.col]);
      if (!bfp::bfp_fits(v)) b.refuse();
      b.setD(b.L.b + b.nv + b.col, v);
    }
    __syncthreads();
    bfp::blk_rnea_adjoint(b, [&](int c, int which, double v) SG_INLINE {
      const Arr& o = which == 0 ? a.o1 : which == 1 ? a.o2 : a.o3;
      if (valid && o.p && !bfp::blk_refused(b)) stv(o, e, b.ext[c], v);
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
  blk_run<E>(model, smem, true, envs, [&](const auto& b, bool valid) SG_INLINE {
    const int64_t e = e0 + min(b.lane, envs - 1);
    const int nv = b.nv;
#pragma unroll 1
    for (int c = b.slot; c < b.nq; c += b.slots) bfp::blk_in(b, c, ldv(a.q, e, c));
#pragma unroll 1
    for (int c = b.slot; c < nv; c += b.slots) {
      bfp::blk_in(b, b.nq + c, ldv(a.qd, e, c));
      bfp::blk_in(b, b.nq + 2 * nv + c, ldv(a.x, e, c));
    }
    __syncthreads();
    bfp::blk_check_quaternion(b);
    bfp::blk_forward_dynamics(b);
    const int c = b.col, x = c >= 0 ? b.ext[c] : 0;
    // qdd joins the inputs; the factor moves to Y's items; the right-hand side becomes the adjoint
    double bar = 0.0;
    if (c >= 0) {
      const int i = b.row_start[c] + b.depth[c];
      bfp::blk_in(b, b.nq + nv + x, b.D(b.L.b + nv + c));
      bar = ldv(a.bar, e, x);
      b.setD(b.L.Y + i, bfp::blk_inverse_pivot(b, c));
    }
#pragma unroll 1
    for (int i = b.slot; i < b.npairs; i += b.slots)
      if (b.pair_row[i] != b.pair_col[i]) b.setD(b.L.Y + i, b.D(b.L.S + i));
    if (c >= 0) b.setD(b.L.b + c, bar);
    __syncthreads();
    bfp::blk_factor_solve(b);
    const double lam = c >= 0 ? b.D(b.L.b + nv + c) : 0.0;
    if (!bfp::bfp_fits(lam)) b.refuse();
    bfp::blk_rnea_adjoint(b, [&](int col, int which, double v) SG_INLINE {
      const Arr& o = which == 0 ? a.o1 : a.o2;
      if (which < 2 && valid && o.p && !bfp::blk_refused(b)) stv(o, e, b.ext[col], -v);
    });
    if (c >= 0 && valid && a.o3.p && !bfp::blk_refused(b)) stv(a.o3, e, x, lam);
  });
}
#endif

}  // namespace sgdyn
