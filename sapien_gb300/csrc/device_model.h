// Flat, depth-first joint table read by the kernels. One contiguous buffer:
//   DModel header | DJoint[nj] (joint 0 = universe, unused) | DLink[nlinks] | DFrame[nj]
// Every environment of a batch reads the same table, so all lanes of a warp load the
// same address (a broadcast through L1).
//
// Canonical joint frames. Each revolute / continuous / prismatic joint's frame is rotated
// by a constant C (DFrame) so that its axis is +z: the model's joint frame F and the
// table's frame F' = F C. Placements, axes, body inertias and link offsets are stored in
// the F' frames, so a joint rotation is Rz(q) and a motion subspace is a column of the
// world rotation (no axis products). World-frame results and link frames are unchanged;
// only a quantity reported in a joint frame (the CLIK error) is rotated back by C.
#pragma once
#ifdef __CUDACC_RTC__
// run-time compilation: no standard headers
typedef long long int64_t;
typedef unsigned long size_t;
#else
#include <cstddef>
#include <cstdint>
#endif

#ifdef __CUDACC__
#define SG_HD __host__ __device__ __forceinline__
#else
#define SG_HD inline
#endif

namespace sgdyn {

// Constants of a joint and of a link as block-floating-point mantissas (bfp.cuh): rotations and
// the axis of exponent -60, the others with the exponents pe, me, ce, Ie. The body inertia is
// kept as mass, centre of mass and rotational inertia about it.
struct alignas(16) BJoint {
  long long R[9], p[3], axis[3], m, c[3], I[6];
  int pe, me, ce, Ie;
  long long pad_;
};
static_assert(sizeof(BJoint) == 224, "BJoint layout");
struct alignas(16) BLink {
  long long R[9], p[3];
  int pe, pad_[3];
};
static_assert(sizeof(BLink) == 112, "BLink layout");

// The tree as the block sweeps (bfp_block.cuh) walk it: `off` entries index the int array that
// follows. Tree columns are velocity indices in depth-first order; a column's depth counts the
// columns above it; a pair is a column with itself or one of its ancestor columns, pairs of a
// column in order of depth, so that pair (a, c) is number row_start[a] + depth(c).
struct alignas(16) BTree {
  int levels;      // joint levels
  int npairs;
  int col_levels;  // column depths
  int nints;       // without pair_of
  int parent, end, level;  // [nj] each: DJoint::parent, subtree_end, level from 1
  int order;       // [nj - 1] joints by level
  int level_start; // [levels + 1]
  int col_joint, col_dof, col_depth, col_ext, row_start;  // [nv] each
  int col_order;   // [nv] columns by depth
  int col_level_start;  // [col_levels + 1]
  int pair_row, pair_col;  // [npairs] each
  int pair_of;     // [nv * nv], after the others: pair of an external row and column, -1 where M is 0
  int pad_;
};
static_assert(sizeof(BTree) == 80, "BTree layout");

enum JointKind : int { JK_NONE = 0, JK_REVOLUTE = 1, JK_PRISMATIC = 2, JK_CONTINUOUS = 3, JK_FREEFLYER = 4 };
enum AxisKind : int { AX_X = 0, AX_Y = 1, AX_Z = 2, AX_GENERAL = 3 };
enum JointFlags : int { JF_ROT_IDENTITY = 1 };

struct alignas(16) DJoint {
  double R[9];   // placement rotation (parent joint frame <- this joint frame at q = 0), row-major
  double p[3];   // placement translation
  double axis[3];  // +z for revolute / continuous / prismatic (canonical frame), else 0
  double m;      // body inertia carried by this joint, about the joint origin:
  double h[3];   //   first moment m*c
  double I[6];   //   rotational inertia about the origin: xx xy xz yy yz zz
  int parent;    // parent joint (0 = universe)
  int kind;      // JointKind
  int axis_kind; // AxisKind
  int flags;     // JointFlags
  int qcol;      // external q column of the first coordinate
  int vcol;      // external v column of the first velocity
  int nv;        // 1, or 6 for a free flyer
  int depth;     // 1 for children of the universe
  int ivx;       // first velocity index in depth-first (tree) order
  int subtree_end;  // one past the last joint of this joint's subtree (depth-first order)
  int pad_[4];
};
static_assert(sizeof(DJoint) == 256, "DJoint layout");

struct alignas(16) DLink {
  double R[9];  // link frame in its joint frame
  double p[3];
  int joint;
  int flags;    // JF_ROT_IDENTITY when the placement rotation is exactly identity
  int pad_[2];
};
static_assert(sizeof(DLink) == 112, "DLink layout");

struct alignas(16) DFrame {
  double C[9];  // model joint frame <- table joint frame, row-major (identity for free flyers)
  double pad_;
};
static_assert(sizeof(DFrame) == 80, "DFrame layout");

struct alignas(16) DModel {
  int nj;       // joints incl. universe
  int nv;
  int nq_ext;
  int nlinks;
  int max_depth;
  int n_free_flyer;
  int pad_[2];
  double gravity[3];
  double pad2_;
};
static_assert(sizeof(DModel) == 64, "DModel layout");

SG_HD const DJoint* model_joints(const DModel* m) {
  return reinterpret_cast<const DJoint*>(reinterpret_cast<const char*>(m) + sizeof(DModel));
}
SG_HD const DLink* model_links(const DModel* m) {
  return reinterpret_cast<const DLink*>(reinterpret_cast<const char*>(m) + sizeof(DModel) +
                                        sizeof(DJoint) * size_t(m->nj));
}
SG_HD const DFrame* model_frames(const DModel* m) {
  return reinterpret_cast<const DFrame*>(reinterpret_cast<const char*>(model_links(m)) +
                                         sizeof(DLink) * size_t(m->nlinks));
}
SG_HD size_t model_table_bytes(int nj, int nlinks) {
  return sizeof(DModel) + sizeof(DJoint) * size_t(nj) + sizeof(DLink) * size_t(nlinks) +
         sizeof(DFrame) * size_t(nj);
}
// The block-floating-point constants follow the frames in a model's device copy.
SG_HD const BJoint* model_bjoints(const DModel* m) {
  return reinterpret_cast<const BJoint*>(reinterpret_cast<const char*>(m) + model_table_bytes(m->nj, m->nlinks));
}
SG_HD const BLink* model_blinks(const DModel* m) { return reinterpret_cast<const BLink*>(model_bjoints(m) + m->nj); }
SG_HD const BTree* model_btree(const DModel* m) {
  return reinterpret_cast<const BTree*>(model_blinks(m) + m->nlinks);
}
SG_HD size_t model_bfp_bytes(int nj, int nlinks) {
  return sizeof(BJoint) * size_t(nj) + sizeof(BLink) * size_t(nlinks);
}

}  // namespace sgdyn
