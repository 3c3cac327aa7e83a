// The fused sweep (FK, WORLD Jacobian, CRBA, RNEA, forward dynamics) in block floating point
// (bfp.cuh) with a whole block of threads per group of environments.
//
// The world-frame recursions and joint tables are those of step_kernel.cuh. Forward dynamics is
// taken from the mass matrix: M = L^T D L with the tree's sparsity (Featherstone, "Rigid Body
// Dynamics Algorithms", 2008, sec. 6.5) on the matrix scaled to a diagonal of at most 1.
//
// Why a block: one thread per environment leaves most of the GPU idle below ~100 k environments
// (16384 of them are 512 warps for 608 schedulers, each walking its tree joint by joint with
// hardly more than one instruction in flight, 5 to 6 cycles per instruction). But only sums run
// along the tree; joint rotations, world inertias, momenta, forces, column forces, mass-matrix
// entries and the rows of an elimination step are independent per joint, column or pair. So a
// block holds E environments and G slots per environment: thread t serves environment t % E,
// and slot t / E takes one joint, one column, some pairs. Running sums go level by level, all
// joints of a level side by side. State is in shared memory ([item][environment], lanes free of
// bank conflicts), phases are separated by block barriers, and a phase's code exists once (the
// same sweep unrolled per model was bound by instruction fetch: 9 of 15 cycles per instruction).
//
// Measured (GB300, device time per call; before: the FP64 sweeps, specialised per model or in
// teams of lanes, that still serve forced settings and models out of range). All five ops: 7-DoF
// arm, 16 environments 143 -> 33 us, 1000: 145 -> 36 us; 9-DoF arm, 16384: 156 -> 98 us. CRBA +
// RNEA + forward dynamics: 9-DoF arm, 131071: 792 -> 563 us; 35-DoF humanoid, 1024: 422 -> 71 us.
// Forward dynamics alone, 18-DoF quadruped, 3001: 84 -> 43 us. What bounds it at 16384 9-DoF
// arms: 2482 warp instructions per environment (170 of its thread instructions in FP64, before
// 4215) issued at 33 % of the schedulers' rate, waiting at barriers and for instruction fetch.
#pragma once
#include "bfp.cuh"
#include "se3.cuh"
#include "step_kernel.cuh"

// on lambdas: inlined even where they are called more than once, so that the block state they
// refer to stays in registers
#define SG_INLINE __attribute__((always_inline))

namespace sgdyn {
namespace bfp {

// Shared-memory items per environment: 64-bit words and exponents of a model's state.
//   in: q, qd, qdd, tau; for adjoint sweeps one more per column, for adjoints that go in
//   A: per joint, rotation (9) + position (3), later acceleration (6) + force (6); then the
//      scaled factor's entries
//   Y: per joint, first the joint's own rotation (9), then mass, first moment, inertia (10);
//      then M's entries in FP64
//   S, V: per column 6 (V: per joint velocity, then column forces); then L in FP64
//   b: per column, right-hand side and solution
//   u: for adjoint sweeps (bfp_diff.cuh), per joint 6; there Y has 12 per joint for two wrenches
// After them the tree's ints (BTree), once per block, and the environments' notes, twice.
struct BlkLayout {
  int in, A, Y, S, V, b, u, words;    // word items
  int xA, xY, xS, xV, xs, xu, ints;   // exponent items
};
SG_HD BlkLayout blk_layout(int nj, int nv, int nq, int npairs, bool adjoint = false) {
  const int m = nj - 1;
  BlkLayout L;
  L.in = 0;
  L.A = nq + (adjoint ? 4 : 3) * nv;
  L.Y = L.A + imax(12 * m, npairs);
  L.S = L.Y + imax((adjoint ? 12 : 10) * m, npairs);
  L.V = L.S + 6 * nv;
  L.b = L.V + imax(6 * nv, npairs - 6 * nv);
  L.u = L.b + 2 * nv;
  L.words = L.u + (adjoint ? 6 * m : 0);
  L.xA = 0;             // 4 per joint: position, then acceleration (2) and force (2)
  L.xY = 4 * m;         // 3 per joint
  L.xS = L.xY + 3 * m;  // 2 per column
  L.xV = L.xS + 2 * nv;
  L.xs = L.xV + 2 * nv;  // scale and pivot shift of each column
  L.xu = L.xs + 2 * nv;  // u (2 per joint), and Y as two wrenches (4 per joint)
  L.ints = L.xu + (adjoint ? 6 * m : 0);
  return L;
}
// What a sweep notes of an environment on its way, for the question whether its results have to
// come from the FP64 algebra (Blk::refused). All after the first two are the largest binary exponent
// of something, kNoNote where there was nothing.
enum Note : int {
  NOTE_REFUSED,  // an input, a pivot or an adjoint out of range
  NOTE_ALIGNED,  // a joint's rotation maps an axis of its frame on one of the world's, or nearly
  NOTE_SCALE,    // products that the bodies' forces are summed from
  NOTE_BIAS,     // generalised bias forces (inverse dynamics)
  NOTE_DRIVE,    // applied generalised forces
  NOTE_TORQUE,   // inverse dynamics out of M qdd + bias
  NOTE_GSCALE,   // products that the gradient with respect to q is summed from
  NOTE_GRAD,     // that gradient
  kNotes
};
constexpr int kNoNote = -4000;
// binary digits of a row that may be lost, see Blk::refused: of forces, of gradients, of float32
constexpr int kLost = 7, kLostGrad = 12, kLostFloat = 24;
constexpr int kBlkMaxThreads = 640, kBlkDiffThreads = 512;
SG_HD size_t blk_bytes(const BlkLayout& L, int tree_ints, int E) {
  return size_t(E) * (8 * size_t(L.words) + 4 * size_t(L.ints) + 2 * 4 * size_t(kNotes)) + 4 * size_t(tree_ints);
}

// World motion subspace column k of joint J at pose (Ro, po).
SG_HD Tw joint_S(const DJoint& J, const BJoint& B, const Rot& Ro, Vec po, int k) {
  if (J.kind == JK_FREEFLYER) {
    const Vec r = k % 3 == 0 ? col_vec(Ro, 0) : k % 3 == 1 ? col_vec(Ro, 1) : col_vec(Ro, 2);
    return k < 3 ? Tw{r, vec0()} : Tw{norm(cross(po, r)), r};
  }
  const Vec u = J.axis_kind == AX_Z ? col_vec(Ro, 2)
                                    : norm(mul(Ro, Vec{B.axis[0], B.axis[1], B.axis[2], -60}));
  return J.kind == JK_PRISMATIC ? Tw{u, vec0()} : Tw{norm(cross(po, u)), u};
}

#ifdef __CUDACC__
// The two algebras a block sweep runs in. BfpAlg: block floating point. FpAlg: plain FP64 on
// the same phases and shared-memory items (mantissa words hold doubles), for environments that
// BfpAlg turns away (Blk::refused). Calls on their types are found in the types' namespaces
// (bfp.cuh; below for the FP64 ones).
struct BfpAlg {
  static constexpr bool kFixed = true;
  typedef bfp::Sc Sc;
  typedef bfp::Vec Vec;
  typedef bfp::Rot Rot;
  typedef bfp::Tw Tw;
  typedef bfp::Rbi Rbi;
  static __device__ __forceinline__ Sc sc(double v) { return from_double(v); }
  static __device__ __forceinline__ Vec vec(double x, double y, double z) { return from_doubles(x, y, z); }
  static __device__ __forceinline__ Vec offset(const DJoint&, const BJoint& B) { return Vec{B.p[0], B.p[1], B.p[2], B.pe}; }
  static __device__ __forceinline__ Vec axis(const DJoint&, const BJoint& B) { return Vec{B.axis[0], B.axis[1], B.axis[2], -60}; }
  static __device__ __forceinline__ Rot placement(const DJoint&, const BJoint& B) { return rot_of(B.R); }
  static __device__ __forceinline__ Vec offset(const DLink&, const BLink& B) { return Vec{B.p[0], B.p[1], B.p[2], B.pe}; }
  static __device__ __forceinline__ Rot placement(const DLink&, const BLink& B) { return rot_of(B.R); }
  static __device__ __forceinline__ Rot quaternion(double x, double y, double z, double w) { return quat_rot(x, y, z, w); }
  // Rodrigues and B Rz(q)
  static __device__ __forceinline__ Rot rotation(const DJoint&, const BJoint& B, double q) {
    i64 s, c;
    sincos60(q, &s, &c);
    return rodrigues(B.axis[0], B.axis[1], B.axis[2], s, c);
  }
  static __device__ __forceinline__ Rot placed_rz(const DJoint&, const BJoint& B, double q) {
    i64 s, c;
    sincos60(q, &s, &c);
    const Half4 hs = split4(s), hc = split4(c), ns = neg(hs);
    Rot r;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const Half4 b0 = split4(B.R[3 * k]), b1 = split4(B.R[3 * k + 1]);
      r.a[3 * k] = mul60(hc, b0, hs, b1);
      r.a[3 * k + 1] = mul60(hc, b1, ns, b0);
      r.a[3 * k + 2] = B.R[3 * k + 2];
    }
    return r;
  }
  static __device__ __forceinline__ Rbi inertia(const DJoint&, const BJoint& B, const Rot& R, Vec p) { return transport(B, R, p); }
  // one row of a rotation product, on stored words
  static __device__ __forceinline__ i64 row_dot(i64 a0, i64 a1, i64 a2, i64 b0, i64 b1, i64 b2) {
    return dot60(split4(a0, a1, a2), split4(b0, b1, b2));
  }
  static __device__ __forceinline__ void get(const Vec& v, double* o) {
    o[0] = to_double(v.x, v.e);
    o[1] = to_double(v.y, v.e);
    o[2] = to_double(v.z, v.e);
  }
  static __device__ __forceinline__ double get(Sc v) { return to_double(v); }
  static __device__ __forceinline__ void quaternion_of(const Rot& R, double* q) { rot_quat(R, q); }
};

struct FpAlg {
  static constexpr bool kFixed = false;
  typedef double Sc;
  typedef V3 Vec;
  typedef M3 Rot;
  typedef Mot Tw;
  typedef RBI Rbi;
  static __device__ __forceinline__ Sc sc(double v) { return v; }
  static __device__ __forceinline__ Vec vec(double x, double y, double z) { return mk(x, y, z); }
  static __device__ __forceinline__ M3 mat(const double* a) { return M3{{a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8]}}; }
  static __device__ __forceinline__ Vec offset(const DJoint& J, const BJoint&) { return mk(J.p[0], J.p[1], J.p[2]); }
  static __device__ __forceinline__ Vec axis(const DJoint& J, const BJoint&) { return mk(J.axis[0], J.axis[1], J.axis[2]); }
  static __device__ __forceinline__ Rot placement(const DJoint& J, const BJoint&) { return mat(J.R); }
  static __device__ __forceinline__ Vec offset(const DLink& L, const BLink&) { return mk(L.p[0], L.p[1], L.p[2]); }
  static __device__ __forceinline__ Rot placement(const DLink& L, const BLink&) { return mat(L.R); }
  static __device__ __forceinline__ Rot quaternion(double x, double y, double z, double w) { return quat_to_R(x, y, z, w); }
  static __device__ __forceinline__ Rot rotation(const DJoint& J, const BJoint& B, double q) {
    double s, c;
    sincos(q, &s, &c);
    return sgdyn::rodrigues(axis(J, B), s, c);
  }
  static __device__ __forceinline__ Rot placed_rz(const DJoint& J, const BJoint&, double q) {
    double s, c;
    sincos(q, &s, &c);
    return sgdyn::mul(mat(J.R), rot_z(s, c));
  }
  static __device__ __forceinline__ Rbi inertia(const DJoint& J, const BJoint&, const Rot& R, Vec p) {
    RBI Y{J.m, mk(J.h[0], J.h[1], J.h[2]), {J.I[0], J.I[1], J.I[2], J.I[3], J.I[4], J.I[5]}};
    return rbi_transport(Y, R, p);
  }
  static __device__ __forceinline__ i64 row_dot(i64 a0, i64 a1, i64 a2, i64 b0, i64 b1, i64 b2) {
    auto d = [](i64 v) { return __longlong_as_double(v); };
    return __double_as_longlong(fma(d(a2), d(b2), fma(d(a1), d(b1), d(a0) * d(b0))));
  }
  static __device__ __forceinline__ void get(const Vec& v, double* o) { o[0] = v.x; o[1] = v.y; o[2] = v.z; }
  static __device__ __forceinline__ double get(double v) { return v; }
  static __device__ __forceinline__ void quaternion_of(const Rot& R, double* q) { R_to_quat(R, q); }
};
}  // namespace bfp

// FP64 counterparts of the calls on block-floating-point types.
__device__ __forceinline__ V3 norm(V3 a) { return a; }
__device__ __forceinline__ Mot norm(Mot a) { return a; }
__device__ __forceinline__ V3 add(V3 a, V3 b) { return a + b; }
__device__ __forceinline__ Mot add(Mot a, Mot b) { return add6(a, b); }
__device__ __forceinline__ RBI add(const RBI& a, const RBI& b) { return rbi_add(a, b); }
__device__ __forceinline__ V3 mul(double s, V3 a) { return s * a; }
__device__ __forceinline__ Mot mul(double s, Mot a) { return scale6(s, a); }
__device__ __forceinline__ Mot mul(const RBI& Y, Mot v) { return rbi_mul(Y, v); }
__device__ __forceinline__ Mot crossm(Mot a, Mot b) { return add_crossm(Mot{mk(0, 0, 0), mk(0, 0, 0)}, a, b); }
__device__ __forceinline__ Mot crossf(Mot a, Mot f) { return add_crossf(Mot{mk(0, 0, 0), mk(0, 0, 0)}, a, f); }
__device__ __forceinline__ double dot(Mot a, Mot b) { return dot6(a, b); }
__device__ __forceinline__ double norm(double a) { return a; }
__device__ __forceinline__ Mot neg(Mot a) { return Mot{-a.v, -a.w}; }
__device__ __forceinline__ V3 col_vec(const M3& R, int j) { return mk(R.a[j], R.a[3 + j], R.a[6 + j]); }

namespace bfp {

// The block's state as algebra A sees it, E environments side by side (0: as many as a pass
// needs). EI: environments of the block, the stride of the inputs and notes, which keep their
// place when the algebra changes.
template <class A, int E, int EI = E>
struct Blk {
  typedef typename A::Vec Vec;
  typedef typename A::Rot Rot;
  typedef typename A::Tw Tw;
  typedef typename A::Rbi Rbi;
  const DModel* m;
  const DJoint* J;
  const BJoint* B;
  const int* pair_of;  // in global memory
  int nj, nv, nq, levels, npairs, col_levels;
  BlkLayout L;
  i64 *w, *win;
  int *x, *note_base;
  // the tree's arrays, in shared memory
  const int *parent, *end, *level, *order, *level_start, *col_joint, *col_dof, *depth, *ext, *row_start, *col_order,
      *col_level_start, *pair_row, *pair_col;
  int width;               // environments side by side, where E is 0
  int lane, slot, slots;   // this thread's place among them, its slot, slots per environment
  int el;                  // this thread's environment in the block
  int count;               // environments whose results are written (the first lanes)
  unsigned mask;           // which ones they are, where E is 0
  bool valid;              // whether this thread's is one of them
  int set;                 // which of the two sets of notes is in use
  int col;       // the slot's column (-1: none)
  int j, p, lv;  // the slot's joint (0: none), its parent and level
  double g[3];   // gravity

  __device__ __forceinline__ int stride() const { return E ? E : width; }
  // Copies the tree too, unless `again`: another pass over a block that is set up.
  __device__ __forceinline__ void setup(const DModel* model, long long* smem, bool adjoint, bool again) {
    m = model;
    const BTree t = *model_btree(model);
    const int* ti = reinterpret_cast<const int*>(model_btree(model) + 1);
    J = model_joints(model);
    B = model_bjoints(model);
    nj = model->nj;
    nv = model->nv;
    nq = model->nq_ext;
    levels = t.levels;
    npairs = t.npairs;
    col_levels = t.col_levels;
    pair_of = ti + t.pair_of;
    L = blk_layout(nj, nv, nq, npairs, adjoint);
    win = smem;
    w = smem + L.A * (EI - stride());  // the items after the inputs begin where the inputs end
    x = reinterpret_cast<int*>(smem + L.words * EI);
    int* s = x + L.ints * EI;
    if (!again) {
#pragma unroll 1
      for (int k = threadIdx.x; k < t.nints; k += blockDim.x) s[k] = ti[k];
    }
    note_base = s + t.nints;
    parent = s + t.parent;
    end = s + t.end;
    level = s + t.level;
    order = s + t.order;
    level_start = s + t.level_start;
    col_joint = s + t.col_joint;
    col_dof = s + t.col_dof;
    depth = s + t.col_depth;
    ext = s + t.col_ext;
    row_start = s + t.row_start;
    col_order = s + t.col_order;
    col_level_start = s + t.col_level_start;
    pair_row = s + t.pair_row;
    pair_col = s + t.pair_col;
    lane = int(threadIdx.x % unsigned(stride()));
    slot = int(threadIdx.x / unsigned(stride()));
    slots = int(blockDim.x / unsigned(stride()));
    col = slot < nv ? slot : -1;
    j = slot < nj - 1 ? slot + 1 : 0;
    for (int k = 0; k < 3; k++) g[k] = model->gravity[k];
    p = ti[t.parent + j];
    lv = ti[t.level + j];
  }
  // The first `envs` of the block's environments; the tree and the first notes are there after it.
  __device__ __forceinline__ void init(const DModel* model, long long* smem, int envs, bool adjoint = false) {
    setup(model, smem, adjoint, false);
    el = lane;
    count = envs;
    valid = lane < envs;
    set = 0;
    clear_notes(0);
    __syncthreads();
  }
  // Those in `which` (E = 0), packed side by side so that a few of them take a few warps' issue.
  // Lanes beyond them repeat the last one and share its inputs: only valid ones may change these.
  __device__ __forceinline__ void init_some(const DModel* model, long long* smem, unsigned which, int note_set,
                                            bool adjoint = false) {
    mask = which;
    count = __popc(which);
    width = count <= 1 ? 1 : 1 << (32 - __clz(count - 1));
    setup(model, smem, adjoint, true);
    valid = lane < count;
    el = env_at(min(lane, count - 1));
    set = note_set;
  }
  // the environment in the block of a lane below `count`
  __device__ __forceinline__ int env_at(int l) const {
    if constexpr (E) return l;
    unsigned r = mask;
    for (int k = 0; k < l; k++) r &= r - 1;
    return __ffs(int(r)) - 1;
  }
  __device__ __forceinline__ i64& W(int item) const { return w[item * stride() + lane]; }
  __device__ __forceinline__ int& X(int item) const { return x[item * stride() + lane]; }
  __device__ __forceinline__ double D(int item) const { return __longlong_as_double(w[item * stride() + lane]); }
  __device__ __forceinline__ double D(int item, int l) const { return __longlong_as_double(w[item * stride() + l]); }
  __device__ __forceinline__ void setD(int item, double v) const { w[item * stride() + lane] = __double_as_longlong(v); }
  __device__ __forceinline__ double in(int c) const { return __longlong_as_double(win[c * EI + el]); }
  __device__ __forceinline__ void set_in(int c, double v) const { win[c * EI + el] = __double_as_longlong(v); }
  __device__ __forceinline__ Vec vec(int item, int xi) const {
    if constexpr (A::kFixed) return Vec{W(item), W(item + 1), W(item + 2), X(xi)};
    else return Vec{D(item), D(item + 1), D(item + 2)};
  }
  __device__ __forceinline__ void put(int item, int xi, const Vec& v) const {
    if constexpr (A::kFixed) {
      W(item) = v.x;
      W(item + 1) = v.y;
      W(item + 2) = v.z;
      X(xi) = v.e;
    } else {
      setD(item, v.x);
      setD(item + 1, v.y);
      setD(item + 2, v.z);
    }
  }
  __device__ __forceinline__ Tw tw(int item, int xi) const { return Tw{vec(item, xi), vec(item + 3, xi + 1)}; }
  __device__ __forceinline__ void put(int item, int xi, const Tw& v) const {
    put(item, xi, v.v);
    put(item + 3, xi + 1, v.w);
  }
  __device__ __forceinline__ Rot rot(int item) const {
    Rot r;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      if constexpr (A::kFixed) r.a[k] = W(item + k);
      else r.a[k] = D(item + k);
    }
    return r;
  }
  __device__ __forceinline__ void put(int item, const Rot& r) const {
#pragma unroll
    for (int k = 0; k < 9; k++) {
      if constexpr (A::kFixed) W(item + k) = r.a[k];
      else setD(item + k, r.a[k]);
    }
  }
  // per joint (j >= 1) and per column
  __device__ __forceinline__ int iR(int j) const { return L.A + 9 * (j - 1); }
  __device__ __forceinline__ int iP(int j) const { return L.A + 9 * (nj - 1) + 3 * (j - 1); }
  __device__ __forceinline__ int xP(int j) const { return L.xA + j - 1; }
  __device__ __forceinline__ int iA(int j) const { return L.A + 12 * (j - 1); }
  __device__ __forceinline__ int xA(int j) const { return L.xA + 4 * (j - 1); }
  __device__ __forceinline__ int iM(int j) const { return L.Y + 9 * (j - 1); }  // joint rotation
  __device__ __forceinline__ Rbi rbi(int j) const {
    const int i = L.Y + 10 * (j - 1), xi = L.xY + 3 * (j - 1);
    Rbi r;
    r.h = vec(i + 1, xi + 1);
    if constexpr (A::kFixed) {
      r.m = Sc{W(i), X(xi)};
#pragma unroll
      for (int k = 0; k < 6; k++) r.I[k] = W(i + 4 + k);
      r.e = X(xi + 2);
    } else {
      r.m = D(i);
#pragma unroll
      for (int k = 0; k < 6; k++) r.I[k] = D(i + 4 + k);
    }
    return r;
  }
  __device__ __forceinline__ void put_rbi(int j, const Rbi& r) const {
    const int i = L.Y + 10 * (j - 1), xi = L.xY + 3 * (j - 1);
    put(i + 1, xi + 1, r.h);
    if constexpr (A::kFixed) {
      W(i) = r.m.m;
      X(xi) = r.m.e;
#pragma unroll
      for (int k = 0; k < 6; k++) W(i + 4 + k) = r.I[k];
      X(xi + 2) = r.e;
    } else {
      setD(i, r.m);
#pragma unroll
      for (int k = 0; k < 6; k++) setD(i + 4 + k, r.I[k]);
    }
  }
  __device__ __forceinline__ Tw S(int c) const { return tw(L.S + 6 * c, L.xS + 2 * c); }
  __device__ __forceinline__ Tw V(int c) const { return tw(L.V + 6 * c, L.xV + 2 * c); }
  __device__ __forceinline__ void putV(int c, Tw v) const { put(L.V + 6 * c, L.xV + 2 * c, v); }
  __device__ __forceinline__ Tw acc(int j) const { return tw(iA(j), xA(j)); }
  __device__ __forceinline__ void put_acc(int j, Tw v) const { put(iA(j), xA(j), v); }
  __device__ __forceinline__ Tw frc(int j) const { return tw(iA(j) + 6, xA(j) + 2); }
  __device__ __forceinline__ void put_frc(int j, Tw v) const { put(iA(j) + 6, xA(j) + 2, v); }

  __device__ __forceinline__ double q(int c) const { return in(c); }
  __device__ __forceinline__ double qd(int c) const { return in(nq + c); }
  __device__ __forceinline__ double qdd(int c) const { return in(nq + nv + c); }
  __device__ __forceinline__ double tau(int c) const { return in(nq + 2 * nv + c); }

  // Notes; the FP64 algebra keeps none.
  __device__ __forceinline__ int& note_at(int s, int note) const { return note_base[(s * kNotes + note) * EI + el]; }
  __device__ __forceinline__ void clear_notes(int s) const {
    if (slot == 0) {
      for (int k = 0; k < kNotes; k++) note_at(s, k) = k <= NOTE_ALIGNED ? 0 : kNoNote;
    }
  }
  __device__ __forceinline__ void refuse() const {
    if constexpr (A::kFixed) note_at(set, NOTE_REFUSED) = 1;
  }
  __device__ __forceinline__ void note(Note k, int exponent) const {
    if constexpr (A::kFixed) atomicMax(&note_at(set, k), exponent);
  }
  __device__ __forceinline__ void note(Note k, double v) const {
    note(k, (__double2hiint(v) >> 20 & 0x7ff) - 1023);
  }
  // Whether the environment has to come from the FP64 algebra: refused on its way; or bits were
  // lost that FP64 may keep. A vector here holds all its components to 2^-57 of the largest,
  // FP64 each to 2^-53 of itself, so a whole row of results that is the small remainder of large
  // terms (gravity torques next to an equilibrium, slow motion across gravity) may be exact in
  // FP64 only. lost = kLost: where a row is below 2^-7 of its terms, so that an error of 2^-57 of
  // the terms is at most 2^-50 of the row. Gradients (kLostGrad) are often that much smaller
  // than their terms about the world's origin, where FP64 loses as much: 2^-45 of the row, about
  // FP64's own error for 9-DoF arms. Results that cancel against applied forces cancel in FP64 too,
  // and so does everything where no rotation is aligned with the world's axes (NOTE_ALIGNED): among
  // dense rotations FP64's terms are off by 2^-53 of themselves. (6-DoF arms that spin fast about
  // dense axes have such rows: of 4096, some in most steps of a rollout, 26 -> 27 to 53 us a step
  // without this.)
  __device__ __forceinline__ bool refused(int lost = kLost) const {
    if constexpr (!A::kFixed) return false;
    const int scale = note_at(set, NOTE_SCALE), least = scale - lost, bias = note_at(set, NOTE_BIAS);
    const int drive = note_at(set, NOTE_DRIVE), torque = note_at(set, NOTE_TORQUE);
    const bool driven = (drive != kNoNote || torque != kNoNote) && (drive == kNoNote || drive >= least) &&
                        (torque == kNoNote || torque >= least);
    const int gscale = note_at(set, NOTE_GSCALE);
    return note_at(set, NOTE_REFUSED) != 0 ||
           (note_at(set, NOTE_ALIGNED) != 0 &&
            ((scale > kTiny && bias != kNoNote && bias < least && !driven) ||
             (gscale > kTiny && note_at(set, NOTE_GRAD) < gscale - kLostGrad)));
  }
  static constexpr int kTiny = -600;  // below: the terms are 0
};

__device__ __forceinline__ bool turns(const DJoint& J) { return J.kind == JK_REVOLUTE || J.kind == JK_CONTINUOUS; }

// The joint's rotation after its placement, R_placement M_J(q).
template <class A, class Q>
__device__ __forceinline__ typename A::Rot joint_rotation(const DJoint& J, const BJoint& B, const Q& q) {
  const bool rot_id = (J.flags & JF_ROT_IDENTITY) != 0;
  if (J.kind == JK_PRISMATIC) return A::placement(J, B);
  if (J.kind != JK_FREEFLYER && J.axis_kind == AX_Z) return A::placed_rz(J, B, q(0));
  const typename A::Rot r = J.kind == JK_FREEFLYER ? A::quaternion(q(3), q(4), q(5), q(6)) : A::rotation(J, B, q(0));
  return rot_id ? r : mul(A::placement(J, B), r);
}

// Refuses the environment for its configuration, given its world rotations: a free flyer's
// quaternion off unit length, and small angles that FP64 would hold to more bits. Rotations are in
// steps of 2^-60 here, so what is proportional to a small angle keeps fewer bits of it. FP64 keeps
// them only where the angle's sine is not added to something larger: where the rotation maps an
// axis of the joint's frame on one of the world's, or nearly (an entry above kAligned, so two of
// its row and column below 2^-10), as with joint axes along the frames' axes or on a root joint.
// (Of a quaternion: where two components are small.)
constexpr i64 kAligned = kOne - (kOne >> 21);
// (for NOTE_ALIGNED: the others of its row and column below 2^-7, which is kLost)
constexpr i64 kNearlyAligned = kOne - (kOne >> 15);
template <class A, int E, int EI>
__device__ __forceinline__ void blk_check_configuration(const Blk<A, E, EI>& b) {
  if constexpr (!A::kFixed) return;
  if (!b.j) return;
  const DJoint& J = b.J[b.j];
  if (J.kind == JK_FREEFLYER) {
    float n2 = 0;
    int small = 0, zeros = 0;
    for (int k = 3; k < 7; k++) {
      const double c = b.q(J.qcol + k);
      const float v = float(c);
      small += bfp_small(c);
      zeros += v == 0.0f;
      n2 += v * v;
    }
    if ((small && small + zeros > 1) || !(n2 > 0.999f && n2 < 1.001f)) b.refuse();
  } else if (turns(J) && bfp_small(b.q(J.qcol))) {
    bool aligned = false;
    for (int k = 0; k < 9; k++) {
      const i64 r = b.W(b.iR(b.j) + k);
      aligned = aligned || r > kAligned || r < -kAligned;
    }
    if (aligned) b.refuse();
  }
}
// World rotations and positions of all joints into A; refuses what blk_check_configuration does.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_poses(const Blk<A, E, EI>& b) {
  typedef typename A::Vec Vec;
  const DJoint& J = b.J[b.j];
  const BJoint& B = b.B[b.j];
  const int qc = J.qcol;
  if (b.j) b.put(b.iM(b.j), joint_rotation<A>(J, B, [&](int k) SG_INLINE { return b.q(qc + k); }));
  __syncthreads();
#pragma unroll 1
  for (int d = 0; d < b.levels; d++) {  // one row of a rotation per thread
    const int lo = b.level_start[d], n = 3 * (b.level_start[d + 1] - lo);
#pragma unroll 1
    for (int k = b.slot; k < n; k += b.slots) {
      const int j = b.order[lo + k / 3], r = k % 3, p = b.parent[j], o = b.iR(j) + 3 * r, im = b.iM(j);
      i64 v[3];
      if (p == 0) {
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = b.W(im + 3 * r + c);
      } else {
        const int pr = b.iR(p) + 3 * r;
        const i64 r0 = b.W(pr), r1 = b.W(pr + 1), r2 = b.W(pr + 2);
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = A::row_dot(r0, r1, r2, b.W(im + c), b.W(im + 3 + c), b.W(im + 6 + c));
      }
#pragma unroll
      for (int c = 0; c < 3; c++) b.W(o + c) = v[c];
      if constexpr (A::kFixed) {
        constexpr unsigned least = unsigned(kNearlyAligned >> 32);
        if (abs_hi(v[0]) >= least || abs_hi(v[1]) >= least || abs_hi(v[2]) >= least) b.note_at(b.set, NOTE_ALIGNED) = 1;
      }
    }
    __syncthreads();
  }
  blk_check_configuration(b);
  Vec o{};
  if (b.j) {  // offset from the parent's origin
    o = A::offset(J, B);
    if (b.p > 0) o = norm(mul(b.rot(b.iR(b.p)), o));
    if (J.kind == JK_PRISMATIC) {
      const typename A::Rot R = b.rot(b.iR(b.j));
      const Vec u = J.axis_kind == AX_Z ? col_vec(R, 2) : norm(mul(R, A::axis(J, B)));
      o = norm(add(o, norm(mul(A::sc(b.q(qc)), u))));
    } else if (J.kind == JK_FREEFLYER) {
      Vec t = A::vec(b.q(qc), b.q(qc + 1), b.q(qc + 2));
      if (!(J.flags & JF_ROT_IDENTITY)) t = norm(mul(A::placement(J, B), t));
      if (b.p > 0) t = norm(mul(b.rot(b.iR(b.p)), t));
      o = norm(add(o, t));
    }
    if (b.p == 0) b.put(b.iP(b.j), b.xP(b.j), o);
  }
  __syncthreads();
#pragma unroll 1
  for (int d = 2; d <= b.levels; d++) {
    if (b.lv == d) {
      o = norm(add(b.vec(b.iP(b.p), b.xP(b.p)), o));
      b.put(b.iP(b.j), b.xP(b.j), o);
    }
    __syncthreads();
  }
}

template <class A>
__device__ __forceinline__ typename A::Tw column_S(const DJoint& J, const BJoint& B, const typename A::Rot& R,
                                                   const typename A::Vec& p, int k) {
  if constexpr (A::kFixed) return joint_S(J, B, R, p, k);
  else return world_S(J, R, p, k);
}
// Motion subspace columns into S and (with_inertia) world inertias into Y, where the joints' own
// rotations are no longer needed.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_columns(const Blk<A, E, EI>& b, bool with_inertia) {
  if (b.col >= 0) {
    const int c = b.col, j = b.col_joint[c];
    b.put(b.L.S + 6 * c, b.L.xS + 2 * c,
          column_S<A>(b.J[j], b.B[j], b.rot(b.iR(j)), b.vec(b.iP(j), b.xP(j)), b.col_dof[c]));
  }
  if (with_inertia && b.j)
    b.put_rbi(b.j, A::inertia(b.J[b.j], b.B[b.j], b.rot(b.iR(b.j)), b.vec(b.iP(b.j), b.xP(b.j))));
  __syncthreads();
}
// sum over the slot's joint's columns of v(column of the joint, external column) S
template <class A, int E, int EI, class F>
__device__ __forceinline__ typename A::Tw joint_motion(const Blk<A, E, EI>& b, const F& v) {
  const DJoint& J = b.J[b.j];
  typename A::Tw r = norm(mul(A::sc(v(J.ivx, J.vcol)), b.S(J.ivx)));
#pragma unroll 1
  for (int k = 1; k < J.nv; k++) r = norm(add(r, mul(A::sc(v(J.ivx + k, J.vcol + k)), b.S(J.ivx + k))));
  return r;
}
// The slot's joint's motion m summed from the root (the joint's own on entry), kept at items
// at(joint) with exponents xat(joint).
template <class A, int E, int EI, class I, class X>
__device__ __forceinline__ void blk_from_root(const Blk<A, E, EI>& b, typename A::Tw& m, const I& at, const X& xat) {
  if (b.j && b.p == 0) b.put(at(b.j), xat(b.j), m);
  __syncthreads();
#pragma unroll 1
  for (int d = 2; d <= b.levels; d++) {
    if (b.lv == d) {
      m = norm(add(b.tw(at(b.p), xat(b.p)), m));
      b.put(at(b.j), xat(b.j), m);
    }
    __syncthreads();
  }
}
// Velocities (V, by joint), accelerations and body forces (A), with zero joint acceleration
// unless with_qdd; notes the terms of the bias forces, if those are to follow.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_motion_forces(const Blk<A, E, EI>& b, bool with_qdd, bool bias = true) {
  typedef typename A::Tw Tw;
  Tw vj{}, v{}, a{};
  if (b.j) v = vj = joint_motion(b, [&](int, int x) SG_INLINE { return b.qd(x); });
  blk_from_root(b, v, [&](int j) SG_INLINE { return b.L.V + 6 * (j - 1); },
                [&](int j) SG_INLINE { return b.L.xV + 2 * (j - 1); });
  if (b.j) {
    a = norm(crossm(v, vj));
    if (with_qdd) a = norm(add(a, joint_motion(b, [&](int, int x) SG_INLINE { return b.qdd(x); })));
    if (b.p == 0) a.v = norm(add(a.v, A::vec(-b.g[0], -b.g[1], -b.g[2])));
  }
  blk_from_root(b, a, [&](int j) SG_INLINE { return b.iA(j); }, [&](int j) SG_INLINE { return b.xA(j); });
  if (b.j) {
    const typename A::Rbi Y = b.rbi(b.j);
    const Tw f = add(mul(Y, a), crossf(v, norm(mul(Y, v))));
    if constexpr (A::kFixed)  // before norm() an exponent is that of the terms, of about 2^57 each
      if (bias) b.note(NOTE_SCALE, 57 + (turns(b.J[b.j]) ? f.w.e : f.v.e));
    b.put_frc(b.j, norm(f));
  }
  __syncthreads();
}
// Forces and (composite) inertias summed over subtrees: level by level, each joint its children.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_subtrees(const Blk<A, E, EI>& b, bool forces, bool composite) {
  const int end = b.end[b.j];
  const bool inner = b.j && end > b.j + 1;
#pragma unroll 1
  for (int d = b.levels - 1; d >= 1; d--) {
    if (inner && b.lv == d) {
      if (forces) {
        typename A::Tw f = b.frc(b.j);
#pragma unroll 1
        for (int k = b.j + 1; k < end; k = b.end[k]) f = norm(add(f, b.frc(k)));
        b.put_frc(b.j, f);
      }
      if (composite) {
        typename A::Rbi Y = b.rbi(b.j);
#pragma unroll 1
        for (int k = b.j + 1; k < end; k = b.end[k]) Y = add(Y, b.rbi(k));
        b.put_rbi(b.j, Y);
      }
    }
    __syncthreads();
  }
}
// Column forces F = Y S (composite Y) into V, M's entries S_c . F_a in FP64 into Y's items
// (for_output) and M into A as blk_solve takes it (for_solve).
template <class A, int E, int EI>
__device__ __forceinline__ void blk_mass_matrix(const Blk<A, E, EI>& b, bool for_solve, bool for_output) {
  typedef typename A::Sc Sc;
  const int c = b.col;
  Sc diag{};
  if (c >= 0) {
    const typename A::Tw S = b.S(c), F = norm(mul(b.rbi(b.col_joint[c]), S));
    b.putV(c, F);
    diag = dot(S, F);
  }
  __syncthreads();
  if (c >= 0) {  // diagonal and scales
    const int i = b.row_start[c] + b.depth[c];
    if constexpr (A::kFixed) {
      if (for_solve) {
        diag = norm(diag);
        const int s = (diag.e + 62) >> 1, k = diag.e + 60 - 2 * s;
        if (diag.m < (1LL << 59)) b.refuse();
        b.X(b.L.xs + c) = s;
        b.W(b.L.A + i) = k >= 0 ? shl(diag.m, k) : shr(diag.m, -k);
      }
    } else {
      b.setD(b.L.A + i, diag);
    }
    if (for_output) b.setD(b.L.Y + i, A::get(diag));
  }
  if (for_solve) __syncthreads();
  bool beyond = false;
#pragma unroll 1
  for (int i = b.slot; i < b.npairs; i += b.slots) {
    const int pa = b.pair_row[i], pc = b.pair_col[i];
    if (pa == pc) continue;
    const Sc v = dot(b.S(pc), b.V(pa));
    if (for_solve) {
      if constexpr (A::kFixed) {
        const int k = v.e + 60 - b.X(b.L.xs + pa) - b.X(b.L.xs + pc);
        // (more than 2 sqrt(M_aa M_cc): not positive definite, and it may not fit the word)
        beyond = beyond || (v.m != 0 && k - clz32(abs_hi(v.m)) > -3);
        b.W(b.L.A + i) = k >= 0 ? shl(v.m, k) : shr(v.m, -k);
      } else {
        b.setD(b.L.A + i, v);
      }
    }
    if (for_output) b.setD(b.L.Y + i, A::get(v));
  }
  if (beyond) b.refuse();
  __syncthreads();
}

// Pivot of column a: D 4^x in [1/4, 1] and its reciprocal, into the diagonal's word and the
// pivot shift; a scaled pivot below 2^-40 sends the environment to the FP64 sweep.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_pivot(const Blk<A, E, EI>& b, int a, int diag) {
  if constexpr (A::kFixed) {
    const i64 D = b.W(diag);
    if (D < (1LL << 20)) b.refuse();
    const unsigned dh = unsigned(hi32(D)), dl = unsigned(u64(D));
    const int xa = imax(0, (dh ? clz32(dh) : 32 + clz32(dl)) - 4) >> 1;
    b.W(diag) = rcp60(shl(D, 2 * xa));
    b.X(b.L.xs + b.nv + a) = xa;
  } else {
    b.setD(diag, 1.0 / b.D(diag));
  }
}
template <class A, int E, int EI>
__device__ __forceinline__ void blk_back(const Blk<A, E, EI>& b);
// M = L^T D L with the right-hand side in b carried along, then x = M^-1 b (after b). By levels
// from the deepest columns, all columns of a level between two barriers (column by column, with
// nv of them, 8192 35-DoF humanoids took 366 us instead of 297): slot c updates row c for every
// column a of the level that it is an ancestor of, f = h / D, then h_cd -= f h_ad along the row;
// the slots one level up then leave their pivots. L's entries go to S / V in FP64.
// Then L x = D^-1 y by levels, one product per column and level. M is in A: scaled fixed point
// (M_ac = h_ac 2^(s_a + s_c - 60) with |h| <= 2^60, the scales from the diagonal: a positive
// definite matrix has |M_ac| <= sqrt(M_aa M_cc), and so have the matrices that elimination
// leaves; with D 4^x in [1/4, 1] every h_ac 2^x and f = h_ac 2^x / (D 4^x) stay below 1 and 4,
// L_ac = f 2^(x_a + s_c - s_a)), or FP64. Inertias that no body has can give another matrix: the
// environment refuses with the first h_ac 2^x above 1.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_solve(const Blk<A, E, EI>& b) {
  const int nv = b.nv, col = b.col;
  const int row = col >= 0 ? b.L.A + b.row_start[col] : 0, dr = col >= 0 ? b.depth[col] : nv;
  bool beyond = false;
  if (dr == b.col_levels - 1) blk_pivot(b, col, row + dr);
  __syncthreads();
#pragma unroll 1
  for (int da = b.col_levels - 1; da >= 0; da--) {
    if (dr < da) {  // columns of depth da are final: their ancestors take them
      const int hi = b.col_level_start[da + 1];
#pragma unroll 1
      for (int k = b.col_level_start[da]; k < hi; k++) {
        const int a = b.col_order[k], ra = b.row_start[a], h0 = b.L.A + ra;
        if (b.pair_col[ra + dr] != col) continue;
        const double ba = b.D(b.L.b + a);
        if constexpr (A::kFixed) {
          const int xa = b.X(b.L.xs + nv + a);
          const i64 h = b.W(h0 + dr);
          beyond = beyond || abs_hi(h) > (1u << 28 >> xa) + 1;
          const Half4 f = split4(mul60(split4(shl(h, xa)), split4(b.W(h0 + da))));
#pragma unroll 1
          for (int d = 0; d <= dr; d++) b.W(row + d) -= shl(mul60(f, split4(shl(b.W(h0 + d), xa))), 2);
          const double l = to_double(shl(i64(f.h), 32) + f.l, xa - 58 + b.X(b.L.xs + col) - b.X(b.L.xs + a));
          b.setD(b.L.S + ra + dr, l);
          b.setD(b.L.b + col, fma(-l, ba, b.D(b.L.b + col)));
        } else {
          const double f = b.D(h0 + dr) * b.D(h0 + da);
#pragma unroll 1
          for (int d = 0; d <= dr; d++) b.setD(row + d, fma(-f, b.D(h0 + d), b.D(row + d)));
          b.setD(b.L.S + ra + dr, f);
          b.setD(b.L.b + col, fma(-f, ba, b.D(b.L.b + col)));
        }
      }
      if (dr == da - 1) blk_pivot(b, col, row + dr);
    } else if (dr == da) {
      double dinv;
      if constexpr (A::kFixed) dinv = to_double(b.W(row + dr), 2 * b.X(b.L.xs + nv + col) - 58 - 2 * b.X(b.L.xs + col));
      else dinv = b.D(row + dr);
      b.setD(b.L.b + nv + col, b.D(b.L.b + col) * dinv);
    }
    if (da == 0 && beyond) b.refuse();
    __syncthreads();
  }
  blk_back(b);
}
// x = L^-1 x (after b) for L in S / V and D^-1 applied already.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_back(const Blk<A, E, EI>& b) {
  const int nv = b.nv;
  const int c = b.slot, dc = c < nv ? b.depth[c] : 0, rc = c < nv ? b.row_start[c] : 0;
  double x = c < nv ? b.D(b.L.b + nv + c) : 0.0;
#pragma unroll 1
  for (int d = 0; d + 1 < b.col_levels; d++) {
    if (dc > d) {
      x = fma(-b.D(b.L.S + rc + d), b.D(b.L.b + nv + b.pair_col[rc + d]), x);
      if (dc == d + 1) b.setD(b.L.b + nv + c, x);
    }
    __syncthreads();
  }
}

// S_c . (subtree force of the column's joint)
template <class A, int E, int EI>
__device__ __forceinline__ double blk_torque(const Blk<A, E, EI>& b, int c) {
  return A::get(dot(b.S(c), b.frc(b.col_joint[c])));
}

// qdd (tree columns, at b + nv) = M^-1 (tau - bias) from the inputs in shared memory and the poses.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_forward_dynamics(const Blk<A, E, EI>& b) {
  blk_columns(b, true);
  blk_motion_forces(b, false);
  blk_subtrees(b, true, true);
  if (b.col >= 0) {
    const double h = blk_torque(b, b.col), tau = b.tau(b.ext[b.col]);
    b.note(NOTE_BIAS, h);
    b.note(NOTE_DRIVE, tau);
    b.setD(b.L.b + b.col, tau - h);
  }
  blk_mass_matrix(b, true, false);
  blk_solve(b);
}

// Stores an input, with its effect on the environment's notes.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_in(const Blk<A, E, EI>& b, int at, double v) {
  b.set_in(at, v);
  if (!bfp_fits(v)) b.refuse();
}
// Reads the environment's inputs; whether they suit BfpAlg goes to its notes.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_load(const Blk<A, E, EI>& b, int ops, const StepArgs& args, int64_t e) {
#pragma unroll 1
  for (int c = b.slot; c < b.nq; c += b.slots) blk_in(b, c, ldv(args.q, e, c));
#pragma unroll 1
  for (int c = b.slot; c < b.nv; c += b.slots) {
    if (ops & (OP_RNEA | OP_ABA)) blk_in(b, b.nq + c, ldv(args.qd, e, c));
    if (ops & OP_RNEA) blk_in(b, b.nq + b.nv + c, ldv(args.qdd, e, c));
    if (ops & OP_ABA) blk_in(b, b.nq + 2 * b.nv + c, ldv(args.tau, e, c));
  }
  __syncthreads();
}

// Semi-implicit Euler in place on the environment's rows of q and qd (args.q, args.qd) from the
// inputs in shared memory and qdd at b + nv, as hetero_integrate_kernel does it.
template <class A, int E, int EI>
__device__ __forceinline__ void blk_euler_rows(const Blk<A, E, EI>& b, const StepArgs& args, int64_t e, double dt) {
  if (!b.j) return;
  const DJoint& J = b.J[b.j];
  double v[6], q[7];
  const int w = J.kind == JK_FREEFLYER ? 6 : 1;
#pragma unroll 1
  for (int k = 0; k < w; k++) {
    v[k] = fma(dt, b.D(b.L.b + b.nv + J.ivx + k), b.qd(J.vcol + k));
    stv(args.qd, e, J.vcol + k, v[k]);
  }
  if (J.kind == JK_FREEFLYER) {
    for (int k = 0; k < 7; k++) q[k] = b.q(J.qcol + k);
    free_flyer_step(q, v, dt);
    for (int k = 0; k < 7; k++) stv(args.q, e, J.qcol + k, q[k]);
  } else {
    stv(args.q, e, J.qcol, fma(dt, v[0], b.q(J.qcol)));
  }
}

// One sweep over the block's environments, whose poses are there; row(environment in block): its row of the arrays,
// this thread's e.
template <class A, int E, int EI, class Row>
__device__ __forceinline__ void blk_step(const Blk<A, E, EI>& b, int ops, const StepArgs& args, int64_t e,
                                         const Row& row) {
  typedef typename A::Sc Sc;
  typedef typename A::Vec Vec;
  typedef typename A::Rot Rot;
  const bool valid = b.valid;
  // (run-time flags, uniform in the grid: one kernel per E serves every op set)
  const bool kFK = ops & OP_FK, kJAC = ops & OP_JAC, kCRBA = ops & OP_CRBA, kRNEA = ops & OP_RNEA,
             kABA = ops & OP_ABA;
  const bool kVel = kRNEA || kABA, kComposite = kCRBA || kABA, kInertia = kVel || kCRBA;
  const int nv = b.nv;
  if (kFK) {
    const DLink* LT = model_links(b.m);
    const BLink* BL = model_blinks(b.m);
#pragma unroll 1
    for (int l = b.slot; l < b.m->nlinks; l += b.slots) {
      const int j = LT[l].joint;
      const Vec pl = A::offset(LT[l], BL[l]);
      Rot R = A::placement(LT[l], BL[l]);
      Vec pp = pl;
      if (j > 0) {
        const Rot Rj = b.rot(b.iR(j));
        R = (LT[l].flags & JF_ROT_IDENTITY) ? Rj : mul(Rj, R);
        pp = norm(add(mul(Rj, pl), b.vec(b.iP(j), b.xP(j))));
      }
      double o[7];
      A::get(pp, o);
      A::quaternion_of(R, o + 3);
      if (valid) {
#pragma unroll
        for (int k = 0; k < 7; k++) stv(args.poses, e, l * 7 + k, o[k]);
      }
    }
  }
  if (!kJAC && !kInertia) return;
  blk_columns(b, kInertia);
  const int c = b.col, xc = c >= 0 ? b.ext[c] : 0;
  if (kJAC && c >= 0) {
    const typename A::Tw S = b.S(c);
    double o[6];
    A::get(S.v, o);
    A::get(S.w, o + 3);
    if (valid) {
#pragma unroll
      for (int k = 0; k < 6; k++) stv(args.J, e, k * nv + xc, o[k]);
    }
  }
  if (!kInertia) return;
  if (kVel) blk_motion_forces(b, kRNEA && !kABA);
  blk_subtrees(b, kVel, kComposite);
  if (kVel && c >= 0) {
    const double f = blk_torque(b, c);
    b.note(NOTE_BIAS, f);
    if (kABA) b.setD(b.L.b + c, f);
    else if (valid) stv(args.tau_out, e, xc, f);
  }
  if (!kComposite) return;
  blk_mass_matrix(b, kABA, kCRBA || kRNEA);
  if (kCRBA && args.M.cs != 1) {  // structure of arrays: lanes are environments
#pragma unroll 1
    for (int rc = b.slot; rc < nv * nv; rc += b.slots) {
      const int i = b.pair_of[rc];
      if (valid) stv(args.M, e, rc, i < 0 ? 0.0 : b.D(b.L.Y + i));
    }
  } else if (kCRBA) {  // entries of a row side by side, environments of the block in turn
#pragma unroll 1
    for (int rc = threadIdx.x; rc < nv * nv; rc += blockDim.x) {
      const int i = b.pair_of[rc];
#pragma unroll 1
      for (int l = 0; l < b.count; l++) stv(args.M, row(b.env_at(l)), rc, i < 0 ? 0.0 : b.D(b.L.Y + i, l));
    }
  }
  if (!kABA) return;
  if (c >= 0) {
    const double h = b.D(b.L.b + c);
    if (kRNEA) {  // tau = b + M qdd
      double t = h;
      const int* of = b.pair_of + xc * nv;
#pragma unroll 4
      for (int k = 0; k < nv; k++) {
        const int i = of[k];
        if (i >= 0) t = fma(b.D(b.L.Y + i), b.qdd(k), t);
      }
      b.note(NOTE_TORQUE, t);
      if (valid) stv(args.tau_out, e, xc, t);
    }
    b.note(NOTE_DRIVE, b.tau(xc));
    b.setD(b.L.b + c, b.tau(xc) - h);
  }
  __syncthreads();
  blk_solve(b);
  if (c >= 0 && valid) stv(args.qdd_out, e, xc, b.D(b.L.b + nv + c));
}
#endif  // __CUDACC__

}  // namespace bfp

#ifdef __CUDACC__
// Runs body(block state) in block floating point on the block's `envs` environments, whose inputs
// load(block state) has read and whose poses are there, and in FP64 for those that refused (lost:
// see Blk::refused). Only these are repeated, packed side by side, and block floating point goes
// no further than the poses where all refuse. CRBA + RNEA + forward dynamics of 16384 9-DoF arms,
// with the call: 112 us with none refused, 150 with 8, 192 with 1 in 20, 203 with all (131072: 584,
// 584, 1178, 1166); before, with the whole block repeated, 158, 251 and 257 (585, 1484, 1509).
template <int E, class Ld, class F>
__device__ __forceinline__ void blk_run(const DModel* model, long long* smem, bool adjoint, int envs, int lost,
                                        const Ld& load, const F& body) {
  bfp::Blk<bfp::BfpAlg, E> b;
  b.init(model, smem, envs, adjoint);
  load(b);
  bfp::blk_poses(b);
  const bool none = __syncthreads_and(b.note_at(0, bfp::NOTE_REFUSED));
  if (!none) body(b);
  __syncthreads();  // all notes are in
  if (__syncthreads_or(none || b.refused(lost))) {
    unsigned which = 0;
    for (int k = 0; k < envs; k++) {
      b.el = k;
      which |= unsigned(none || b.refused(lost)) << k;
    }
    if (which == 0) return;  // (a lane beyond the batch repeats the last environment)
    bfp::Blk<bfp::FpAlg, 0, E> f;
    f.init_some(model, smem, which, 0, adjoint);
    bfp::blk_poses(f);
    body(f);
  }
}

// ROWS: the environments are rows of the arrays by a list, and may take an Euler step (an
// instantiation of its own: the plain sweep is 4 % slower with it). At most 640 threads, so that
// a thread may hold 96 registers.
template <int E, bool ROWS>
__global__ void __launch_bounds__(bfp::kBlkMaxThreads) bfp_block_kernel(const DModel* __restrict__ model, int ops,
                                                                        const StepArgs args, const BfpRows r) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = args.n - e0 < E ? int(args.n - e0) : E;
  auto row = [&](int el) SG_INLINE {
    const int64_t e = e0 + min(el, envs - 1);
    return ROWS ? int64_t(r.rows[e]) : e;
  };
  blk_run<E>(
      model, smem, false, envs, bfp::kLost, [&](auto& b) SG_INLINE { bfp::blk_load(b, ops, args, row(b.el)); },
      [&](auto& b) SG_INLINE {
        const int64_t e = row(b.el);
        bfp::blk_step(b, ops, args, e, row);
        if (ROWS && r.integrate && b.valid && !b.refused()) bfp::blk_euler_rows(b, args, e, r.dt);
      });
}

// PhysxArticulation::computePassiveForce on float32 state rows (physx_interop.cu): RNEA at zero
// acceleration with the gravity and / or velocity terms.
template <int E>
__global__ void __launch_bounds__(bfp::kBlkMaxThreads) bfp_passive_kernel(const DModel* __restrict__ model,
                                                                          const PassiveArgs a) {
  extern __shared__ __align__(16) long long smem[];
  const int64_t e0 = int64_t(blockIdx.x) * E;
  const int envs = a.n - e0 < E ? int(a.n - e0) : E;
  blk_run<E>(
      model, smem, false, envs, bfp::kLostFloat,
      [&](auto& b) SG_INLINE {
        const int64_t e = e0 + min(b.el, envs - 1);
        if (b.col >= 0) {  // one-DoF joints only: as many coordinates as columns
          bfp::blk_in(b, b.col, double(a.qpos[e * a.in_stride + b.col]));
          bfp::blk_in(b, b.nq + b.col, a.coriolis ? double(a.qvel[e * a.in_stride + b.col]) : 0.0);
        }
        __syncthreads();
      },
      [&](auto& b) SG_INLINE {
        if (!a.gravity) b.g[0] = b.g[1] = b.g[2] = 0.0;
        bfp::blk_columns(b, true);
        bfp::blk_motion_forces(b, false);
        bfp::blk_subtrees(b, true, false);
        if (b.col >= 0) {
          const double f = bfp::blk_torque(b, b.col);
          b.note(bfp::NOTE_BIAS, f);
          if (b.valid) a.qf[(e0 + b.el) * a.out_stride + b.ext[b.col]] = float(f);
        }
      });
}
#endif

}  // namespace sgdyn
