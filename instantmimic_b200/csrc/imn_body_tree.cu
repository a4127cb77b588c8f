// imn_body_tree.cu -- bottom-up body-tree reductions and the smooth-dynamics stages
// built on them (reference: src/instantmimic/utils/mjw_kernels/tree_fusion.py,
// velocity_fusion.py):
//
//   imn_body_tree_accumulate   accumulate()      tree_fusion.py:52-170  (also
//                              subtree_com_accumulate, :173-183, with 3 components)
//   imn_crb                    crb()             tree_fusion.py:186-206 (composite
//                              inertias, then the joint-space inertia M)
//   imn_rne                    rne()             tree_fusion.py:209-222 (bias forces)
//   imn_com_vel                com_vel()         velocity_fusion.py:15-126
//
// The reference walks m.body_tree inside one cooperative block per world, one level
// after the other with a block barrier in between.  Here a world is a team of 8, 16 or 32
// lanes of a warp: its per-body values sit in the team's slice of shared memory, a level
// is a strided loop over (body, component) entries, and __syncwarp() separates levels.  Inputs arrive
// and results leave as contiguous per-world runs (coalesced); nothing is read twice
// from HBM.
//
// Summation order.  A parent receives its children in the order in which they stand
// in the level list, one writer per (parent, component): the reference's
// deterministic kernels (tree_fusion.py:80-135), which its own test pins bit for bit
// against a sequential depth-ordered sum.  The unordered (atomic) mode of the
// reference has no order to reproduce; the ordered result satisfies its tolerance.
//
// RESTATED: the per-body arithmetic of crb / rne (spatial inertia times motion vector,
// force cross product, the ancestor walk of M, the bias projection) lives in
// mujoco-warp's smooth.py and math.py, whose source is not available; what follows is
// MuJoCo's published mj_crb / mj_rne / mj_comVel arithmetic with sums written as
// left-to-right fused multiply-add chains.  velocity_fusion.py spells its joint
// branches out, and those are followed statement by statement.
#include "imn_common.cuh"

namespace imn {

static const int kTreeWarps = 4, kVelWarps = 2;

struct Sp6 {
  float v[6];
};

__device__ __forceinline__ Sp6 ld6(const float* p) {
  Sp6 r;
#pragma unroll
  for (int k = 0; k < 6; ++k) r.v[k] = p[k];
  return r;
}
__device__ __forceinline__ void st6(float* p, const Sp6& a) {
#pragma unroll
  for (int k = 0; k < 6; ++k) p[k] = a.v[k];
}
// a + b * s, component by component
__device__ __forceinline__ Sp6 axpy6(const Sp6& a, const Sp6& b, float s) {
  Sp6 r;
#pragma unroll
  for (int k = 0; k < 6; ++k) r.v[k] = fmaf(b.v[k], s, a.v[k]);
  return r;
}
__device__ __forceinline__ float dot6(const Sp6& a, const Sp6& b) {
  float acc = a.v[0] * b.v[0];
#pragma unroll
  for (int k = 1; k < 6; ++k) acc = fmaf(a.v[k], b.v[k], acc);
  return acc;
}
// x y' - y x'
__device__ __forceinline__ float det2(float x, float yp, float y, float xp) { return fmaf(x, yp, -(y * xp)); }
__device__ __forceinline__ void cross3(const float* a, const float* b, float* r) {
  r[0] = det2(a[1], b[2], a[2], b[1]);
  r[1] = det2(a[2], b[0], a[0], b[2]);
  r[2] = det2(a[0], b[1], a[1], b[0]);
}
// Spatial motion cross product (MuJoCo mju_crossMotion): angular = w x a_ang,
// linear = w x a_lin + v x a_ang, for vel = (w, v).
__device__ __forceinline__ Sp6 motion_cross(const Sp6& vel, const Sp6& a) {
  Sp6 r;
  float t[3], u[3];
  cross3(vel.v, a.v, r.v);
  cross3(vel.v, a.v + 3, t);
  cross3(vel.v + 3, a.v, u);
#pragma unroll
  for (int k = 0; k < 3; ++k) r.v[3 + k] = t[k] + u[k];
  return r;
}
// Spatial force cross product (MuJoCo mju_crossForce): angular = w x f_ang + v x f_lin,
// linear = w x f_lin.
__device__ __forceinline__ Sp6 motion_cross_force(const Sp6& vel, const Sp6& f) {
  Sp6 r;
  float t[3], u[3];
  cross3(vel.v, f.v, t);
  cross3(vel.v + 3, f.v + 3, u);
#pragma unroll
  for (int k = 0; k < 3; ++k) r.v[k] = t[k] + u[k];
  cross3(vel.v, f.v + 3, r.v + 3);
  return r;
}
// 10-number spatial inertia (Ixx Iyy Izz Ixy Ixz Iyz, m*cx m*cy m*cz, m) times a motion
// vector (MuJoCo mju_mulInertVec), each sum a left-to-right chain contracted the way
// nvcc contracts "a*b + c*d + ..." (the first sum or difference of two products fuses
// its LEFT product and rounds the right one; every later product is fused into the
// running value) -- the rule the reference's generated tree L'DL code follows when run.
__device__ __forceinline__ Sp6 inert_vec(const float* i, const Sp6& a) {
  const float* v = a.v;
  Sp6 r;
  r.v[0] = fmaf(i[7], v[5], fmaf(-i[8], v[4], fmaf(i[4], v[2], fmaf(i[0], v[0], i[3] * v[1]))));
  r.v[1] = fmaf(-i[6], v[5], fmaf(i[8], v[3], fmaf(i[5], v[2], fmaf(i[3], v[0], i[1] * v[1]))));
  r.v[2] = fmaf(i[6], v[4], fmaf(-i[7], v[3], fmaf(i[2], v[2], fmaf(i[4], v[0], i[5] * v[1]))));
  r.v[3] = fmaf(i[9], v[3], fmaf(i[8], v[1], -(i[7] * v[2])));
  r.v[4] = fmaf(i[9], v[4], fmaf(i[6], v[2], -(i[8] * v[0])));
  r.v[5] = fmaf(i[9], v[5], fmaf(i[7], v[0], -(i[6] * v[1])));
  return r;
}

// A world is worked on by a team of GW lanes (8, 16 or 32): the levels of a body tree are a
// few bodies wide, so a whole warp per world would leave most lanes idle through the
// per-body arithmetic (measured: 8 of 32 lanes active per instruction, the kernels bound by
// instruction issue).  A warp therefore takes 32 / GW consecutive worlds; control flow is the
// same for all of them (one model), so __syncwarp() separates levels for every team at once.
// The last warp's surplus teams run on the last world and store nothing.
template <int GW>
struct Team {
  int sl;      // lane within the team
  int w;       // the team's world (clamped to the batch)
  int slot;    // the team's slice of the CTA's shared memory
  bool live;   // false: surplus team, no stores
  bool none;   // the whole warp is surplus
};
template <int GW>
__device__ __forceinline__ Team<GW> make_team(int nworld) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per = 32 / GW;
  const int first = (blockIdx.x * (blockDim.x >> 5) + warp) * per, sub = lane / GW;
  Team<GW> t;
  t.sl = lane - sub * GW;
  t.live = first + sub < nworld;
  t.w = t.live ? first + sub : nworld - 1;
  t.slot = warp * per + sub;
  t.none = first >= nworld;
  return t;
}

// ---- everything on its way at once ----------------------------------------------------
//
// A stage is a few levels of short arithmetic; what took the time was reads that waited for one another: the
// level's tables (position -> body -> parent, dofs, joints), one dependent read from global memory after the other in
// every level, qvel inside them, and inputs fetched where they are needed.  A warp now sends for all of
// its worlds' inputs and for the tables of the tree that the stage reads (four to six words per body, in its own shared
// memory: no block barrier) with asynchronous copies, waits once, and walks the levels in
// shared memory.  Five smooth stages in a graph, us: 34 dofs 64 worlds 37.0 -> 28.6, 1000 worlds 40.6 -> 31.3, 8192 worlds
// 52.0 -> 46.5; 56 dofs 500 worlds 83.9 -> 66.9, 4096 worlds 86.9 -> 72.0; 35 dofs 16384 worlds 148.1 -> 133.0.  (com_vel with a
// lane per world, 32 worlds per block, was ahead of the teams from 4096 worlds on and is not any more: 65536 worlds of 34
// dofs 53.4 us against 45.1, 56 dofs 97.0 against 75.0, 35 dofs 93.2 against 76.4.)
__device__ __forceinline__ void async_word(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}
// A world's run of n floats by the lanes of its team: 16 bytes a piece where the runs are whole pieces on 16-byte
// boundaries (`dst` always is), four bytes elsewhere.
template <int GW>
__device__ __forceinline__ void async_run(float* dst, const float* src, int n, int sl) {
  if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll 2
    for (int i = 4 * sl; i < n; i += 4 * GW)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + i)), "l"(src + i)
                   : "memory");
  } else {
#pragma unroll 4
    for (int i = sl; i < n; i += GW) async_word(dst + i, src + i);
  }
}
// The warp's copies of the tables; a stage lays out those that it reads.
struct WarpTables {
  int *bodies, *child_ptr, *child_ids, *parent, *dofadr, *dofnum, *offsets, *dof_body;
};
// behind the worlds of the CTA (32 / GW per warp, `per_world` floats each), a warp's `words` of tables after the other's
template <int GW>
__device__ __forceinline__ int* table_space(float* smem, int per_world, int words) {
  return reinterpret_cast<int*>(smem + (size_t)(blockDim.x >> 5) * (32 / GW) * per_world) + (threadIdx.x >> 5) * words;
}
__host__ __device__ inline int sweep_words(int nbody, int nlevels) { return 3 * nbody + 1 + nlevels + 1; }
// of the tree alone, without a look at its dofs: what a sweep up reads
__device__ __forceinline__ WarpTables sweep_tables(const ImnBodyTree& T, int* at) {
  WarpTables t = {};
  t.bodies = at, t.child_ids = t.bodies + T.nbody, t.child_ptr = t.child_ids + T.nbody, t.offsets = t.child_ptr + T.nbody + 1;
  return t;
}
// the same where it is in global memory
__device__ __forceinline__ WarpTables sweep_tables(const ImnBodyTree& T) {
  WarpTables t = {};
  t.bodies = const_cast<int*>(T.level_bodies), t.child_ids = const_cast<int*>(T.child_ids);
  t.child_ptr = const_cast<int*>(T.child_ptr), t.offsets = const_cast<int*>(T.level_offsets);
  return t;
}
__device__ __forceinline__ void send_words(int* dst, const int* src, int n) {
#pragma unroll 1
  for (int i = threadIdx.x & 31; i < n; i += 32) async_word(dst + i, src + i);
}
// what a sweep up reads (child_ptr has an entry per position and one behind; the leaves' children take one pointer each)
__device__ __forceinline__ void send_sweep(const ImnBodyTree& T, const WarpTables& t) {
  send_words(t.offsets, T.level_offsets, T.nlevels + 1);
  send_words(t.bodies, T.level_bodies, T.nbody);
  send_words(t.child_ptr, T.child_ptr, T.nbody + 1);
  send_words(t.child_ids, T.child_ids, T.nbody - 1);
}
__device__ __forceinline__ void send_levels(const ImnBodyTree& T, const WarpTables& t) {
  send_words(t.parent, T.body_parentid, T.nbody);
  send_words(t.dofadr, T.body_dofadr, T.nbody);
  send_words(t.dofnum, T.body_dofnum, T.nbody);
}

// Bottom-up sweep over the team's values (nbody x C floats in shared memory): the
// parents of a level take their children of the next level, in level-list order
// (tree_fusion.py:94-112).  child_ptr is indexed by the parent's position in the level
// list.  FIXED: the number of components where it is known (a division by it otherwise).
template <int GW, int FIXED>
__device__ __forceinline__ void sweep_up(const WarpTables& t, int nlevels, float* v, int components, bool skip_root_parent, int sl) {
  const int C = FIXED ? FIXED : components;
#pragma unroll 1
  for (int level = nlevels - 1; level > 0; --level) {
    const int pstart = t.offsets[level - 1];
    const int pcount = t.offsets[level] - pstart;
#pragma unroll 1
    for (int entry = sl; entry < pcount * C; entry += GW) {
      const int pos = pstart + entry / C, comp = entry - (entry / C) * C;
      const int parent = t.bodies[pos];
      if (skip_root_parent && parent == 0) continue;
      float value = v[parent * C + comp];
      const int cend = t.child_ptr[pos + 1];
#pragma unroll 1
      for (int k = t.child_ptr[pos]; k < cend; ++k) value = value + v[t.child_ids[k] * C + comp];
      v[parent * C + comp] = value;
    }
    __syncwarp();
  }
}

template <int GW>
__device__ __forceinline__ void copy_out(float* __restrict__ dst, const float* src, int n, int sl, bool live) {
  if (!live) return;
  if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll 2
    for (int i = 4 * sl; i < n; i += 4 * GW) *reinterpret_cast<float4*>(dst + i) = *reinterpret_cast<const float4*>(src + i);
    return;
  }
#pragma unroll 4
  for (int i = sl; i < n; i += GW) dst[i] = src[i];
}

template <int GW>
__global__ void __launch_bounds__(32 * kTreeWarps)
    tree_accumulate_kernel(const ImnBodyTree T, float* __restrict__ values, const int64_t world_ld, const int C,
                           const int skip_root_parent, const int staged, const int nworld) {
  extern __shared__ __align__(16) float tree_smem[];
  chain_wait();
  const Team<GW> t = make_team<GW>(nworld);
  if (t.none) return;
  const int n = T.nbody * C, per_world = (n + 3) & ~3;
  float* v = tree_smem + (size_t)t.slot * per_world;
  const WarpTables tab = sweep_tables(T, table_space<GW>(tree_smem, per_world, sweep_words(T.nbody, T.nlevels)));
  float* g = values + (size_t)t.w * world_ld;
  async_run<GW>(v, g, n, t.sl);
  if (staged) send_sweep(T, tab);
  async_wait();
  if (!staged)
    sweep_up<GW, 0>(sweep_tables(T), T.nlevels, v, C, skip_root_parent != 0, t.sl);
  else if (C == 3)
    sweep_up<GW, 3>(tab, T.nlevels, v, C, skip_root_parent != 0, t.sl);
  else
    sweep_up<GW, 0>(tab, T.nlevels, v, C, skip_root_parent != 0, t.sl);
  copy_out<GW>(g, v, n, t.sl, t.live);
}

// crb: composite inertias (cinert summed up the tree, the world body's children kept
// out of it: tree_fusion.py:190-191), then M (tree_fusion.py:192-206): row i of M holds
// i's ancestors in ascending order with the diagonal last; entry (i, j) is
// cdof_j . (crb[body_i] cdof_i), the diagonal on top of the armature.
// One world per warp (GW = 32).
__host__ __device__ inline bool sweep_in_bufs(int nbody, int nlevels, int nv) { return sweep_words(nbody, nlevels) <= 6 * nv; }
__host__ __device__ inline int crb_words(int nbody, int nlevels, int nv) {
  return nv + (sweep_in_bufs(nbody, nlevels, nv) ? 0 : sweep_words(nbody, nlevels));
}
template <int GW>
__global__ void __launch_bounds__(32 * kTreeWarps)
    crb_kernel(const ImnBodyTree T, const float* __restrict__ cinert, const float* __restrict__ cdof,
               float* __restrict__ crb, float* __restrict__ M, const int64_t M_ld, const int nworld) {
  extern __shared__ __align__(16) float tree_smem[];
  chain_wait();
  const Team<GW> t = make_team<GW>(nworld);
  if (t.none) return;
  const int sl = t.sl, w = t.w;
  const int nb10 = T.nbody * 10, nv6 = T.nv * 6, per_world = ((nb10 + 3) & ~3) + 2 * ((nv6 + 3) & ~3);
  float* c = tree_smem + (size_t)t.slot * per_world;
  float* dof = c + ((nb10 + 3) & ~3);
  float* bufs = dof + ((nv6 + 3) & ~3);
  // the sweep's tables lie where `bufs` of the warp's world will, or behind the worlds where they take more
  int* const behind = table_space<GW>(tree_smem, per_world, crb_words(T.nbody, T.nlevels, T.nv));
  WarpTables tab = sweep_tables(T, sweep_in_bufs(T.nbody, T.nlevels, T.nv) ? reinterpret_cast<int*>(bufs) : behind + T.nv);
  tab.dof_body = behind;
  async_run<GW>(c, cinert + (size_t)w * nb10, nb10, sl);
  async_run<GW>(dof, cdof + (size_t)w * nv6, nv6, sl);
  send_sweep(T, tab);
  send_words(tab.dof_body, T.dof_bodyid, T.nv);
  async_wait();
  sweep_up<GW, 10>(tab, T.nlevels, c, 10, true, sl);
  copy_out<GW>(crb + (size_t)w * nb10, c, nb10, sl, t.live);
  const float* arm = T.dof_armature + (size_t)(w % T.n_armature) * T.nv;
  float* Mw = M + (size_t)w * M_ld;
  // crb[body_i] cdof_i per dof, then one stored entry of M per lane: entry e = (i, j) is
  // cdof_j . buf_i -- the ancestor walk of the reference flattened over M's CSR, so that
  // every lane is busy and consecutive lanes store consecutive entries
#pragma unroll 1
  for (int i = sl; i < T.nv; i += GW) st6(bufs + 6 * i, inert_vec(c + 10 * tab.dof_body[i], ld6(dof + 6 * i)));
  __syncwarp();
  constexpr int B = 2;  // entries whose indices are read together (four: 8192 34-dof worlds 13.5 -> 15.8 us, others equal)
#pragma unroll 1
  for (int e0 = sl; e0 < T.nM; e0 += B * GW) {
    int i[B], j[B];
#pragma unroll
    for (int k = 0; k < B; ++k) {
      const int e = min(e0 + k * GW, T.nM - 1);
      i[k] = __ldg(T.M_rowidx + e), j[k] = __ldg(T.M_colind + e);
    }
#pragma unroll
    for (int k = 0; k < B; ++k) {
      const int e = e0 + k * GW;
      if (e >= T.nM) break;
      float v = dot6(ld6(dof + 6 * j[k]), ld6(bufs + 6 * i[k]));
      if (i[k] == j[k]) v = arm[i[k]] + v;
      if (t.live) Mw[e] = v;
    }
  }
}

__host__ __device__ inline int rne_floats(int nbody, int nv) {
  return 2 * ((nbody * 6 + 3) & ~3) + ((nv * 6 + 3) & ~3) + ((nbody * 10 + 3) & ~3) + ((nv + 3) & ~3);
}
__host__ __device__ inline int rne_words(int nbody, int nlevels) { return 4 * nbody + nlevels + 1; }
// rne without accelerations (tree_fusion.py:209-222): cacc down the tree from
// -gravity, per-body forces cinert cacc + cvel x* (cinert cvel), summed up the tree,
// projected on the dofs.
template <int GW>
__global__ void __launch_bounds__(32 * kTreeWarps)
    rne_kernel(const ImnBodyTree T, const float* __restrict__ cinert, const float* __restrict__ cvel,
               const float* __restrict__ cdof, const float* __restrict__ cdof_dot, const float* __restrict__ qvel,
               const int64_t qvel_ld, float* __restrict__ cacc_out, float* __restrict__ cfrc_out,
               float* __restrict__ qfrc_bias, const int64_t bias_ld, const int nworld) {
  extern __shared__ __align__(16) float tree_smem[];
  chain_wait();
  const Team<GW> t = make_team<GW>(nworld);
  if (t.none) return;
  const int sl = t.sl, w = t.w;
  const int nb6 = T.nbody * 6, nv6 = T.nv * 6, nb6p = (nb6 + 3) & ~3, nv6p = (nv6 + 3) & ~3;
  const int nb10 = T.nbody * 10, nb10p = (nb10 + 3) & ~3, per_world = rne_floats(T.nbody, T.nv);
  float* cacc = tree_smem + (size_t)t.slot * per_world;
  float* cfrc = cacc + nb6p;  // cvel until the body's force replaces it
  float* dd = cfrc + nb6p;    // cdof_dot, then cdof
  float* inert = dd + nv6p;
  float* qv = inert + nb10p;
  // the walk down's tables; those of the sweep up take their place, the dofs' bodies that of the warp's first qvel
  WarpTables tab = {};
  tab.bodies = table_space<GW>(tree_smem, per_world, rne_words(T.nbody, T.nlevels)), tab.offsets = tab.bodies + T.nbody;
  tab.parent = tab.offsets + T.nlevels + 1, tab.dofadr = tab.parent + T.nbody, tab.dofnum = tab.dofadr + T.nbody;
  tab.child_ptr = tab.parent, tab.child_ids = tab.child_ptr + T.nbody + 1;
  tab.dof_body = reinterpret_cast<int*>(qv - (size_t)(t.slot % (32 / GW)) * per_world);
  async_run<GW>(dd, cdof_dot + (size_t)w * nv6, nv6, sl);
  async_run<GW>(qv, qvel + (size_t)w * qvel_ld, T.nv, sl);
  async_run<GW>(inert, cinert + (size_t)w * nb10, nb10, sl);
  async_run<GW>(cfrc, cvel + (size_t)w * nb6, nb6, sl);
  send_words(tab.offsets, T.level_offsets, T.nlevels + 1);
  send_words(tab.bodies, T.level_bodies, T.nbody);
  send_levels(T, tab);
  if (sl < 6) {
    const float* g = T.gravity + 3 * (size_t)(w % T.n_gravity);
    cacc[sl] = (sl < 3 || !T.gravity_enabled) ? 0.0f : -g[sl - 3];
  }
  async_wait();
#pragma unroll 1
  for (int level = 1; level < T.nlevels; ++level) {
    const int end = tab.offsets[level + 1];
#pragma unroll 1
    for (int pos = tab.offsets[level] + sl; pos < end; pos += GW) {
      const int b = tab.bodies[pos];
      Sp6 a = ld6(cacc + 6 * tab.parent[b]);
      const int d0 = tab.dofadr[b], d1 = d0 + tab.dofnum[b];
#pragma unroll 1
      for (int dofid = d0; dofid < d1; ++dofid) a = axpy6(a, ld6(dd + 6 * dofid), qv[dofid]);
      st6(cacc + 6 * b, a);
    }
    __syncwarp();
  }
  // what comes next arrives during the forces (64 to 512 worlds, where space does not count: 5.5 -> 5.8 us)
  send_words(tab.child_ptr, T.child_ptr, T.nbody + 1);
  send_words(tab.child_ids, T.child_ids, T.nbody - 1);
  send_words(tab.dof_body, T.dof_bodyid, T.nv);
  async_run<GW>(dd, cdof + (size_t)w * nv6, nv6, sl);
  copy_out<GW>(cacc_out + (size_t)w * nb6, cacc, nb6, sl, t.live);
#pragma unroll 1
  for (int b = sl; b < T.nbody; b += GW) {
    Sp6 r;
    if (b == 0) {
#pragma unroll
      for (int k = 0; k < 6; ++k) r.v[k] = 0.0f;
    } else {
      float in[10];
#pragma unroll
      for (int k = 0; k < 10; ++k) in[k] = inert[10 * b + k];
      const Sp6 v = ld6(cfrc + 6 * b);
      const Sp6 f = inert_vec(in, ld6(cacc + 6 * b));
      const Sp6 x = motion_cross_force(v, inert_vec(in, v));
#pragma unroll
      for (int k = 0; k < 6; ++k) r.v[k] = f.v[k] + x.v[k];
    }
    st6(cfrc + 6 * b, r);
  }
  async_wait();
  sweep_up<GW, 6>(tab, T.nlevels, cfrc, 6, false, sl);
  __syncwarp();
  copy_out<GW>(cfrc_out + (size_t)w * nb6, cfrc, nb6, sl, t.live);
  float* bias = qfrc_bias + (size_t)w * bias_ld;
#pragma unroll 1
  for (int i = sl; i < T.nv; i += GW) {
    const float e = dot6(ld6(dd + 6 * i), ld6(cfrc + 6 * tab.dof_body[i]));
    if (t.live) bias[i] = e;
  }
}

__host__ __device__ inline int vel_words(int nbody, int nlevels) { return 6 * nbody + nlevels + 1; }
// Body velocities by depth (velocity_fusion.py:15-103): cvel of a body is its parent's
// plus cdof qvel of its own dofs; cdof_dot of a dof is cvel x cdof taken before that
// dof's own contribution (for a free joint: the three translations first, zero
// cdof_dot; then the rotations against the velocity that includes the translations).
template <int GW>
__global__ void __launch_bounds__(32 * kTreeWarps)
    com_vel_kernel(const ImnBodyTree T, const float* __restrict__ qvel, const int64_t qvel_ld,
                   const float* __restrict__ cdof, float* __restrict__ cvel_out, float* __restrict__ cdof_dot_out,
                   const int nworld) {
  extern __shared__ __align__(16) float tree_smem[];
  chain_wait();
  const Team<GW> t = make_team<GW>(nworld);
  if (t.none) return;
  const int sl = t.sl, w = t.w;
  const int nb6 = T.nbody * 6, nv6 = T.nv * 6, nb6p = (nb6 + 3) & ~3, nv6p = (nv6 + 3) & ~3, nvp = (T.nv + 3) & ~3;
  const int per_world = nb6p + 2 * nv6p + nvp;
  float* cvel = tree_smem + (size_t)t.slot * per_world;
  float* dof = cvel + nb6p;
  float* dot = dof + nv6p;
  float* qv = dot + nv6p;
  WarpTables tab = {};
  tab.bodies = table_space<GW>(tree_smem, per_world, vel_words(T.nbody, T.nlevels)), tab.offsets = tab.bodies + T.nbody;
  tab.parent = tab.offsets + T.nlevels + 1, tab.dofadr = tab.parent + T.nbody;
  int* const jntadr = tab.dofadr + T.nbody;
  int* const jntnum = jntadr + T.nbody;
  int* const kind = jntnum + T.nbody;  // of the body's first joint
  async_run<GW>(dof, cdof + (size_t)w * nv6, nv6, sl);
  async_run<GW>(qv, qvel + (size_t)w * qvel_ld, T.nv, sl);
  send_words(tab.offsets, T.level_offsets, T.nlevels + 1);
  send_words(tab.bodies, T.level_bodies, T.nbody);
  send_words(tab.parent, T.body_parentid, T.nbody);
  send_words(tab.dofadr, T.body_dofadr, T.nbody);
  send_words(jntnum, T.body_jntnum, T.nbody);
#pragma unroll 1
  for (int b = threadIdx.x & 31; b < T.nbody; b += 32) {
    const int adr = T.body_jntadr[b];
    jntadr[b] = adr;
    kind[b] = T.body_jntnum[b] > 0 ? T.jnt_type[adr] : 0;
  }
  async_wait();
#pragma unroll 1
  for (int level = 0; level < T.nlevels; ++level) {
    const int end = tab.offsets[level + 1];
#pragma unroll 1
    for (int pos = tab.offsets[level] + sl; pos < end; pos += GW) {
      const int b = tab.bodies[pos];
      Sp6 v;
      if (b == 0) {
#pragma unroll
        for (int k = 0; k < 6; ++k) v.v[k] = 0.0f;
      } else {
        v = ld6(cvel + 6 * tab.parent[b]);
        int dofid = tab.dofadr[b], type = kind[b];
        const int j0 = jntadr[b], j1 = j0 + jntnum[b];
#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
          if (j > j0) type = T.jnt_type[j];
          if (type == IMN_JNT_FREE) {
            Sp6 zero;
#pragma unroll
            for (int k = 0; k < 6; ++k) zero.v[k] = 0.0f;
#pragma unroll 1
            for (int k = 0; k < 3; ++k) {
              v = axpy6(v, ld6(dof + 6 * (dofid + k)), qv[dofid + k]);
              st6(dot + 6 * (dofid + k), zero);
            }
#pragma unroll 1
            for (int k = 3; k < 6; ++k) st6(dot + 6 * (dofid + k), motion_cross(v, ld6(dof + 6 * (dofid + k))));
#pragma unroll 1
            for (int k = 3; k < 6; ++k) v = axpy6(v, ld6(dof + 6 * (dofid + k)), qv[dofid + k]);
            dofid += 6;
          } else if (type == IMN_JNT_BALL) {
#pragma unroll 1
            for (int k = 0; k < 3; ++k) st6(dot + 6 * (dofid + k), motion_cross(v, ld6(dof + 6 * (dofid + k))));
#pragma unroll 1
            for (int k = 0; k < 3; ++k) v = axpy6(v, ld6(dof + 6 * (dofid + k)), qv[dofid + k]);
            dofid += 3;
          } else {
            st6(dot + 6 * dofid, motion_cross(v, ld6(dof + 6 * dofid)));
            v = axpy6(v, ld6(dof + 6 * dofid), qv[dofid]);
            dofid += 1;
          }
        }
      }
      st6(cvel + 6 * b, v);
    }
    __syncwarp();
  }
  copy_out<GW>(cvel_out + (size_t)w * nb6, cvel, nb6, sl, t.live);
  copy_out<GW>(cdof_dot_out + (size_t)w * nv6, dot, nv6, sl, t.live);
}


static int check_tree(const ImnBodyTree* T, const char* who, bool need_dofs) {
  if (!T) return set_error("%s: NULL tree", who), IMN_ERR_NULL;
  if (T->nbody <= 0 || T->nlevels <= 0) return set_error("%s: empty body tree", who), IMN_ERR_SHAPE;
  if (!T->body_parentid || !T->level_bodies || !T->level_offsets || !T->child_ptr || !T->child_ids)
    return set_error("%s: a body-tree table is NULL", who), IMN_ERR_NULL;
  if (need_dofs) {
    if (T->nv <= 0) return set_error("%s: nv must be positive", who), IMN_ERR_SHAPE;
    if (!T->dof_bodyid || !T->dof_parentid || !T->body_dofadr || !T->body_dofnum)
      return set_error("%s: a dof table is NULL", who), IMN_ERR_NULL;
  }
  return IMN_OK;
}

// Lanes per world: the tree's team_lanes when it is 8, 16 or 32 (the host mirror sets the
// smallest that covers the widest level), else a whole warp.
// Per kernel the width is raised to what was measured fastest for full batches on a B200 (65536 worlds, 34-dof
// humanoid, 56-dof SNU-like, 35-dof G1-like tree, widths 8 / 16 / 32 in us):
//   tree sum, 3 components   12 / 18 / 32     17 / 25 / 40     33 / 32 / 57    -> the tree's width
//   com_vel                  45 / 58 / 108    75 / 96 / 152    76 / 86 / 154   -> the tree's width
//   rne                      53 / 62 / 96    104 / 96 / 128   161 / 135 / 155  -> at least 16
//   crb                     115 / 85 / 84    365 / 232 / 171  245 / 153 / 133  -> 32
// A narrow team fills the lanes during the per-body arithmetic but multiplies the shared
// memory of a CTA (16 worlds instead of 4), which costs resident warps: crb keeps three
// per-world arrays on chip and its entry loop fills a whole warp anyway.
//
// What a warp's worlds and tables take decides how many warps an SM holds.  With tables for every stage in
// every stage's space, cdof beside cdof_dot and blocks of four warps throughout, us for 8192, 16384 and 65536 worlds:
// com_vel SNU 16.5, 28.5, 83; crb SNU 30.9, -, 171, G1 20.1, -, 133; rne SNU 18.9, -, 111, G1 22.4, -, 149.
// Each stage its own tables, those of one phase in the place of another's: crb SNU 25.3, 47, 168, G1 20.1, 38, 132; rne SNU
// 14.9, 28, 96, G1 18.7, 39, 135; com_vel in blocks of two warps SNU 10.8, 22.8, 75 (of four 16.9, 28.8, 84, of one 10.8,
// 22.7, 73; G1 11.9 / 12.7 / 12.0 at 8192).  The other stages lose in blocks of two (crb SNU 31.6, 50, 169).
static int team_lanes(const ImnBodyTree* T, int at_least = 8) {
  const int lanes = (T->team_lanes == 8 || T->team_lanes == 16) ? T->team_lanes : 32;
  return lanes > at_least ? lanes : at_least;
}

template <typename... Args>
static int launch_tree(const char* who, void (*kernel)(Args...), int warps, int gw, size_t floats_per_world,
                       int table_words, int nworld, void* stream, Args... args) {
  if (nworld < 0) return set_error("%s: negative world count", who), IMN_ERR_SHAPE;
  if (nworld == 0) return IMN_OK;
  // fewer warps a block for trees of hundreds of bodies, whose worlds would not fit
  const size_t warp_bytes = 4 * (floats_per_world * (32 / gw) + table_words);
  while (warps > 1 && warps * warp_bytes > 227 * 1024) warps /= 2;
  const int per_cta = warps * (32 / gw);
  const size_t bytes = warps * warp_bytes;
  if (bytes > 227 * 1024)
    return set_error("%s: %zu bytes of shared memory per block exceed the 227 KB of an SM", who, bytes), IMN_ERR_LIMIT;
  {
    const cudaError_t e = allow_shared(kernel, bytes);
    if (e != cudaSuccess) return set_error("%s: cudaFuncSetAttribute: %s", who, cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  }
  const cudaError_t e =
      launch_chained(kernel, (nworld + per_cta - 1) / per_cta, 32 * warps, bytes, (cudaStream_t)stream, args...);
  if (e != cudaSuccess) return set_error("%s: launch failed: %s", who, cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  return IMN_OK;
}

static size_t up4z(size_t n) { return (n + 3) & ~(size_t)3; }

// KERNEL<8 | 16 | 32> by the tree's team width
#define IMN_TEAM_LAUNCH(LANES, KERNEL, WARPS, FLOATS, TABLES, NWORLD, STREAM, ...)                        \
  ((LANES) == 8    ? imn::launch_tree(who, KERNEL<8>, WARPS, 8, FLOATS, TABLES, NWORLD, STREAM, __VA_ARGS__)   \
   : (LANES) == 16 ? imn::launch_tree(who, KERNEL<16>, WARPS, 16, FLOATS, TABLES, NWORLD, STREAM, __VA_ARGS__) \
                   : imn::launch_tree(who, KERNEL<32>, WARPS, 32, FLOATS, TABLES, NWORLD, STREAM, __VA_ARGS__))

}  // namespace imn

extern "C" int imn_body_tree_accumulate(const ImnBodyTree* T, float* values, int64_t world_ld, int32_t components,
                                        int32_t skip_root_parent, int32_t nworld, void* stream) {
  const char* who = "imn_body_tree_accumulate";
  int rc = imn::check_tree(T, who, false);
  if (rc) return rc;
  if (!values) return imn::set_error("%s: NULL values", who), IMN_ERR_NULL;
  if (components <= 0 || world_ld < (int64_t)T->nbody * components)
    return imn::set_error("%s: components %d / world stride %lld do not hold %d bodies", who, components,
                          (long long)world_ld, T->nbody),
           IMN_ERR_SHAPE;
  // A tree whose tables do not fit behind a warp's worlds (one component, a warp per world, from 12 to 15 thousand
  // bodies on) is walked in global memory.
  const int lanes = imn::team_lanes(T), words = imn::sweep_words(T->nbody, T->nlevels);
  const size_t floats = imn::up4z((size_t)T->nbody * components);
  const int staged = 4 * (floats * (32 / lanes) + words) <= 227 * 1024;
  return IMN_TEAM_LAUNCH(lanes, imn::tree_accumulate_kernel, imn::kTreeWarps, floats, staged ? words : 0, nworld, stream, *T, values, world_ld,
                         (int)components, (int)skip_root_parent, staged, (int)nworld);
}

extern "C" int imn_crb(const ImnBodyTree* T, const float* cinert, const float* cdof, float* crb, float* M,
                       int64_t M_ld, int32_t nworld, void* stream) {
  const char* who = "imn_crb";
  int rc = imn::check_tree(T, who, true);
  if (rc) return rc;
  if (!cinert || !cdof || !crb || !M || !T->dof_armature || !T->M_rowidx || !T->M_colind)
    return imn::set_error("%s: NULL array", who), IMN_ERR_NULL;
  if (T->n_armature <= 0 || M_ld < T->nM) return imn::set_error("%s: bad armature count or M stride", who), IMN_ERR_SHAPE;
  return imn::launch_tree(who, imn::crb_kernel<32>, imn::kTreeWarps, 32,
                         imn::up4z((size_t)T->nbody * 10) + 2 * imn::up4z((size_t)T->nv * 6),
                         imn::crb_words(T->nbody, T->nlevels, T->nv), nworld, stream, *T, cinert, cdof, crb, M, M_ld, (int)nworld);
}

extern "C" int imn_rne(const ImnBodyTree* T, const float* cinert, const float* cvel, const float* cdof,
                       const float* cdof_dot, const float* qvel, int64_t qvel_ld, float* cacc, float* cfrc_int,
                       float* qfrc_bias, int64_t bias_ld, int32_t nworld, void* stream) {
  const char* who = "imn_rne";
  int rc = imn::check_tree(T, who, true);
  if (rc) return rc;
  if (!cinert || !cvel || !cdof || !cdof_dot || !qvel || !cacc || !cfrc_int || !qfrc_bias || !T->gravity)
    return imn::set_error("%s: NULL array", who), IMN_ERR_NULL;
  if (T->n_gravity <= 0 || qvel_ld < T->nv || bias_ld < T->nv)
    return imn::set_error("%s: bad gravity count or stride", who), IMN_ERR_SHAPE;
  return IMN_TEAM_LAUNCH(imn::team_lanes(T, 16), imn::rne_kernel, imn::kTreeWarps, (size_t)imn::rne_floats(T->nbody, T->nv),
                         imn::rne_words(T->nbody, T->nlevels), nworld, stream, *T, cinert, cvel, cdof, cdof_dot, qvel, qvel_ld, cacc, cfrc_int, qfrc_bias, bias_ld,
                         (int)nworld);
}

extern "C" int imn_com_vel(const ImnBodyTree* T, const float* qvel, int64_t qvel_ld, const float* cdof, float* cvel,
                           float* cdof_dot, int32_t nworld, void* stream) {
  const char* who = "imn_com_vel";
  int rc = imn::check_tree(T, who, true);
  if (rc) return rc;
  if (!qvel || !cdof || !cvel || !cdof_dot || !T->body_jntadr || !T->body_jntnum || !T->jnt_type)
    return imn::set_error("%s: NULL array", who), IMN_ERR_NULL;
  if (qvel_ld < T->nv) return imn::set_error("%s: qvel stride < nv", who), IMN_ERR_SHAPE;
  return IMN_TEAM_LAUNCH(imn::team_lanes(T), imn::com_vel_kernel, imn::kVelWarps, imn::up4z((size_t)T->nbody * 6) + 2 * imn::up4z((size_t)T->nv * 6) + imn::up4z(T->nv),
                         imn::vel_words(T->nbody, T->nlevels), nworld, stream, *T, qvel, qvel_ld, cdof, cvel, cdof_dot, (int)nworld);
}
