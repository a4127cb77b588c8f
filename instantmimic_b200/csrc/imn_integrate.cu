// imn_integrate.cu -- the implicit-fast integrator's tail, the step right after the
// constraint solve (reference: _integrate, mjw_step_optimized.py:5209-5297):
//
//   1. A = M - h qDeriv on M's sparsity, qDeriv = d(qfrc_smooth)/d(qvel) restricted to
//      the actuator term  sum_a moment_a moment_a^T dforce_a/dvelocity_a  (the
//      actuator-centric assembly, mjw_step_optimized.py:629-669, 4172-4295) and the
//      passive joint damping  -diag(dof_damping)  (upstream _qderiv_actuator_passive);
//   2. x = A^-1 efc.Ma  -- the tree L'DL / blocked dense kernels (imn_msolve.cu,
//      imn_tree_jit.cu), launched by the host layer between the two kernels here;
//   3. the advance  qvel += h x, qpos integrated on its manifold with the new qvel,
//      time += h  (upstream _advance through _advance_with_scratch,
//      mjw_step_optimized.py:4823-4847).
//
// RESTATED: the arithmetic of steps 1 and 3 lives in mujoco-warp (derivative.py,
// forward.py), whose source is not available; what follows is MuJoCo's published
// semi-implicit update (mj_advance, mju_quatIntegrate) and the derivative terms named
// above, with a fixed summation order.  The reference adds the actuator products with
// atomics in whatever order the hardware picks; here an entry receives them in
// ascending actuator order, so results are reproducible bit for bit (and equal to the
// CPU oracle's).  Tendon damping, fluid forces and the free-body correction of
// mujoco-warp 3.16 are not part of this file.
#include "imn_common.cuh"

namespace imn {

// One warp per world.  qD is assembled in the warp's shared-memory row (nM floats),
// then A = M - h qD leaves coalesced.  Actuators are taken 32 at a time, lane = actuator, so that the
// chain row length -> row address -> dofs and moments -> entry index is walked once for 32
// actuators.  An entry takes its products in ascending actuator order; how that is kept:
//   rows of one dof (servos)   lanes that hit the same diagonal entry are ranked by lane and add one
//                              rank after the other;
//   rows of up to four dofs    every lane forms its row's nonzero products; when no entry is hit by
//                              two actuators of the batch (each pair marks its entry and looks
//                              whether the mark stayed) the order does not matter and all add at
//                              once.  Motors on the axes of a ball joint store three dofs with one
//                              nonzero moment, so their products land on three different diagonals;
//   anything else              actuator by actuator.
// Per 8192 humanoid worlds with 28 motors in three-dof rows the batch form takes 10 us where actuator
// by actuator took 44 (the chain of dependent reads, 28 times).
//
// Two variants (imn_implicit_matrix chooses), same sums for any rows:
//   ROWS   the batch form, and M fetched ahead.  64 registers a thread and a second shared-memory row for the
//          marks: 32 warps per SM.
//   !ROWS  neither: 32 registers, 64 warps per SM; rows of several dofs go actuator by actuator.
// A pass over a large batch is bound by memory in flight, so the warps count where no row needs the
// batch form; a batch of a wave or two is bound by one world's chain of reads, which the
// fetched-ahead M shortens.  Servo rows (34 dofs, 28 actuators), us with / without ROWS: 512 worlds
// 3.6 / 4.4, 4096 5.0 / 5.7, 8192 9.2 / 9.4, 16384 19.5 / 17.9, 65536 65.1 / 55.8 (199 MB: 3.6 TB/s).
static const int kMatrixWarps = 8;
static const int kRowDofs = 4;  // rows of the batch form
static const int kRowsBlocksPerSm = 4;  // of the ROWS variant: 64 registers x 256 threads

__device__ __forceinline__ void add_batch(float* qd, int e, float c, int lane) {
  const unsigned peers = __match_any_sync(IMN_FULL_MASK, e);
  const int rank = __popc(peers & ((1u << lane) - 1u));
  const int rounds = __reduce_max_sync(IMN_FULL_MASK, e >= 0 ? __popc(peers) : 0);
#pragma unroll 1
  for (int r = 0; r < rounds; ++r) {
    if (e >= 0 && rank == r) qd[e] = qd[e] + c;
    __syncwarp();
  }
}

template <bool ROWS>
__global__ void __launch_bounds__(32 * kMatrixWarps)
    implicit_matrix_kernel(const ImnImplicit P, const float* __restrict__ M, const int64_t M_ld,
                           float* __restrict__ out, const int64_t out_ld, const int nworld) {
  extern __shared__ float qd_all[];
  chain_wait();
  const int lane = threadIdx.x & 31, w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= nworld) return;
  const int row = (P.nM + 3) & ~3;
  float* qd = qd_all + (threadIdx.x >> 5) * (ROWS ? 2 : 1) * row;
  int* mark = reinterpret_cast<int*>(qd + row);  // the actuator of the batch that hit an entry last
  // M's entries are on their way while the actuators are worked on
  constexpr int kAhead = ROWS ? 12 : 0;
  const float* Mw = M + (size_t)w * M_ld;
  float m[kAhead + 1];
#pragma unroll
  for (int k = 0; k < kAhead; ++k) m[k] = lane + 32 * k < P.nM ? __ldg(Mw + lane + 32 * k) : 0.0f;
  const float h = P.timestep[w % P.n_timestep];
#pragma unroll 4
  for (int e = lane; e < P.nM; e += 32) qd[e] = 0.0f;
  __syncwarp();
  if (P.nu > 0 && P.actuation) {
    const int* rownnz = P.moment_rownnz + (size_t)w * P.nu;
    const int* rowadr = P.moment_rowadr + (size_t)w * P.nu;
    const int* colind = P.moment_colind + (size_t)w * P.moment_ld;
    const float* moment = P.actuator_moment + (size_t)w * P.moment_ld;
    const float* gain = P.actuator_velocity_gain + (size_t)w * P.nu;
#pragma unroll 1
    for (int a0 = 0; a0 < P.nu; a0 += 32) {
      const int a = a0 + lane;
      const bool mine = a < P.nu;
      const int n = mine ? rownnz[a] : 0, base = mine ? rowadr[a] : 0;
      float vel = 0.0f;
      if (mine) {
        if (P.ctrl) {
          const size_t k = (size_t)(w % P.n_coefficients) * P.nu + a;
          vel = P.ctrl[(size_t)w * P.ctrl_ld + a] * P.gain_g2[k];
          vel = vel + P.gain_b2[k];
          P.velocity_gain_out[(size_t)w * P.nu + a] = vel;
        } else {
          vel = gain[a];
        }
      }
      const int longest = __reduce_max_sync(IMN_FULL_MASK, n);
      if (longest <= 1) {
        int e = -1;
        float c = 0.0f;
        if (n == 1 && vel != 0.0f) {
          const int di = colind[base];
          c = (moment[base] * moment[base]) * vel;
          if (c != 0.0f) e = __ldg(P.M_elemid + di * P.nv + di);
        }
        add_batch(qd, e, c, lane);
        continue;
      }
      if (ROWS && longest <= kRowDofs) {
        int dof[kRowDofs];
        float mo[kRowDofs];
#pragma unroll
        for (int k = 0; k < kRowDofs; ++k) {
          const bool in = k < n;
          dof[k] = in ? colind[base + k] : 0, mo[k] = in ? moment[base + k] : 0.0f;
        }
        int e[kRowDofs * (kRowDofs + 1) / 2];
        float c[kRowDofs * (kRowDofs + 1) / 2];
#pragma unroll
        for (int i = 0, p = 0; i < kRowDofs; ++i)
#pragma unroll
          for (int j = 0; j <= i; ++j, ++p) {
            c[p] = (mo[i] * mo[j]) * vel;
            e[p] = i < n && vel != 0.0f && c[p] != 0.0f ? __ldg(P.M_elemid + dof[i] * P.nv + dof[j]) : -1;
          }
        bool clash = false;
#pragma unroll
        for (int p = 0; p < kRowDofs * (kRowDofs + 1) / 2; ++p)
          if (e[p] >= 0) mark[e[p]] = lane;
        __syncwarp();
#pragma unroll
        for (int p = 0; p < kRowDofs * (kRowDofs + 1) / 2; ++p) clash = clash || (e[p] >= 0 && mark[e[p]] != lane);
        if (!__any_sync(IMN_FULL_MASK, clash)) {
#pragma unroll
          for (int p = 0; p < kRowDofs * (kRowDofs + 1) / 2; ++p)
            if (e[p] >= 0) qd[e[p]] = qd[e[p]] + c[p];
          __syncwarp();
          continue;
        }
      }
      const int a1 = min(a0 + 32, P.nu);
#pragma unroll 1
      for (int s = a0; s < a1; ++s) {
        const float v = __shfl_sync(IMN_FULL_MASK, vel, s - a0);
        const int ns = __shfl_sync(IMN_FULL_MASK, n, s - a0), bs = __shfl_sync(IMN_FULL_MASK, base, s - a0);
        if (v == 0.0f || ns <= 0) continue;  // warp-uniform
        // pairs (ri >= rj) of the actuator's moment row; distinct pairs hit distinct
        // entries of M, so the lanes never collide within one actuator
#pragma unroll 1
        for (int p = lane; p < ns * (ns + 1) / 2; p += 32) {
          int ri = (int)((sqrtf(8.0f * (float)p + 1.0f) - 1.0f) * 0.5f);
          while ((ri + 1) * (ri + 2) / 2 <= p) ++ri;
          while (ri * (ri + 1) / 2 > p) --ri;
          const int rj = p - ri * (ri + 1) / 2;
          const int di = colind[bs + ri], dj = colind[bs + rj];
          const int e = P.M_elemid[di * P.nv + dj];
          if (e < 0) continue;
          const float c = (moment[bs + ri] * moment[bs + rj]) * v;
          if (c != 0.0f) qd[e] = qd[e] + c;
        }
        __syncwarp();
      }
    }
  }
  if (P.damper)
    for (int i = lane; i < P.nv; i += 32) {
      const int e = P.M_elemid[i * P.nv + i];
      qd[e] = qd[e] - P.dof_damping[i];
    }
  __syncwarp();
  float* ow = out + (size_t)w * out_ld;
#pragma unroll
  for (int k = 0; k < kAhead; ++k)
    if (lane + 32 * k < P.nM) ow[lane + 32 * k] = m[k] - h * qd[lane + 32 * k];
#pragma unroll 4
  for (int e = lane + 32 * kAhead; e < P.nM; e += 32) ow[e] = Mw[e] - h * qd[e];
}

__device__ __forceinline__ void quat_integrate(float q[4], const float w[3], float h) {
  // q <- normalise(q (x) [cos(a/2), axis sin(a/2)]),  a = h |w|,  axis = w / |w|
  const float norm = sqrtf(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
  float r[4] = {1.0f, 0.0f, 0.0f, 0.0f};
  if (norm >= IMN_MJ_MINVAL) {
    const float half = 0.5f * (h * norm);
    const float s = sinf(half) / norm;
    r[0] = cosf(half), r[1] = w[0] * s, r[2] = w[1] * s, r[3] = w[2] * s;
  }
  const float a = q[0], b = q[1], c = q[2], d = q[3];
  float o[4] = {a * r[0] - b * r[1] - c * r[2] - d * r[3], a * r[1] + b * r[0] + c * r[3] - d * r[2],
                a * r[2] - b * r[3] + c * r[0] + d * r[1], a * r[3] + b * r[2] - c * r[1] + d * r[0]};
  const float len = sqrtf(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3]);
  if (len < IMN_MJ_MINVAL) {
    q[0] = 1.0f, q[1] = q[2] = q[3] = 0.0f;
    return;
  }
  const float inv = 1.0f / len;
  q[0] = o[0] * inv, q[1] = o[1] * inv, q[2] = o[2] * inv, q[3] = o[3] * inv;
}

// The advance of one joint of one world: its dofs get their new velocity, then its
// coordinates move with it.  `qvel`, `qpos`, `acc` point at the joint's first entry.
__device__ __forceinline__ void advance_joint(int type, float h, float* qvel, float* qpos, const float* acc) {
  const int ndof = type == IMN_JNT_FREE ? 6 : (type == IMN_JNT_BALL ? 3 : 1);
  float v[6];
  for (int k = 0; k < ndof; ++k) {
    v[k] = qvel[k] + h * acc[k];
    qvel[k] = v[k];
  }
  if (type == IMN_JNT_FREE) {
    for (int k = 0; k < 3; ++k) qpos[k] = qpos[k] + h * v[k];
    float q[4] = {qpos[3], qpos[4], qpos[5], qpos[6]};
    quat_integrate(q, v + 3, h);
    for (int k = 0; k < 4; ++k) qpos[3 + k] = q[k];
  } else if (type == IMN_JNT_BALL) {
    float q[4] = {qpos[0], qpos[1], qpos[2], qpos[3]};
    quat_integrate(q, v, h);
    for (int k = 0; k < 4; ++k) qpos[k] = q[k];
  } else {
    qpos[0] = qpos[0] + h * v[0];
  }
}

// A block advances 32 consecutive worlds: their qpos, qvel and qacc rows come into shared
// memory with coalesced loads, lane = world, the warps share the joints (a warp works on
// one joint of 32 worlds at a time, so its lanes take the same branch: with a thread per
// (world, joint) every warp held a free joint next to hinges and ran the quaternion path
// for one lane in 29), and the rows leave with coalesced stores.
static const int kAdvanceWarps = 4;
__host__ __device__ inline int advance_stride(int n) { return (n & 3) == 0 ? (n | 1) : n; }

__global__ void __launch_bounds__(32 * kAdvanceWarps)
    advance_kernel(const ImnAdvance P, const float* __restrict__ qacc, const int64_t qacc_ld, const int nworld) {
  extern __shared__ __align__(16) float rows[];
  chain_wait();
  // row strides: the lanes of a warp read the same element of 32 rows; a row length that
  // shares a factor of 4 or more with the 32 banks is padded to an odd stride
  const int tq = advance_stride(P.nq), tv = advance_stride(P.nv);
  float* sq = rows;            // [32][tq]
  float* sv = sq + 32 * tq;    // [32][tv]
  float* sa = sv + 32 * tv;    // [32][tv]
  const int w0 = blockIdx.x * 32, nw = min(32, nworld - w0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the block's rows as one run of nw * n elements over all threads (consecutive threads,
  // consecutive addresses).  Row and column come from a multiplication by 1 / n, exact for
  // these few thousand elements ((e + 1/2) / n is at least 1 / (2 n) away from an integer),
  // so that the iterations do not depend on each other and their loads overlap.
  auto move = [&](float* tile, int stride, float* global, const float* source, int64_t ld, int n, bool store) {
    if (stride == n && ld == n) {  // rows back to back on both sides: one straight copy
      float* g = global ? global + (size_t)w0 * ld : nullptr;
      const float* src = source ? source + (size_t)w0 * ld : g;
#pragma unroll 4
      for (int e = threadIdx.x; e < nw * n; e += 32 * kAdvanceWarps)
        if (store) g[e] = tile[e];
        else tile[e] = src[e];
      return;
    }
    const float inv = 1.0f / (float)n;
#pragma unroll 4
    for (int e = threadIdx.x; e < nw * n; e += 32 * kAdvanceWarps) {
      const int r = (int)(((float)e + 0.5f) * inv), c = e - r * n;
      const size_t at = (size_t)(w0 + r) * ld + c;
      if (store) global[at] = tile[r * stride + c];
      else tile[r * stride + c] = source ? source[at] : global[at];
    }
  };
  move(sq, tq, P.qpos, nullptr, P.qpos_ld, P.nq, false);
  move(sv, tv, P.qvel, nullptr, P.qvel_ld, P.nv, false);
  move(sa, tv, nullptr, qacc, qacc_ld, P.nv, false);
  __syncthreads();
  if (lane < nw) {
    const int w = w0 + lane;
    const float h = P.timestep[w % P.n_timestep];
#pragma unroll 1
    for (int j = warp; j < P.njnt; j += kAdvanceWarps) {
      const int dof = P.jnt_dofadr[j], pos = P.jnt_qposadr[j];
      advance_joint(P.jnt_type[j], h, sv + lane * tv + dof, sq + lane * tq + pos, sa + lane * tv + dof);
    }
    if (warp == 0 && P.time) P.time[w] = P.time[w] + h;
  }
  __syncthreads();
  move(sq, tq, P.qpos, nullptr, P.qpos_ld, P.nq, true);
  move(sv, tv, P.qvel, nullptr, P.qvel_ld, P.nv, true);
}

}  // namespace imn

extern "C" int imn_implicit_matrix(const ImnImplicit* p, const float* M, int64_t M_ld, float* out, int64_t out_ld,
                                   int32_t nworld, void* stream) {
  if (!p || !M || !out || !p->M_elemid || !p->timestep)
    return imn::set_error("imn_implicit_matrix: NULL argument"), IMN_ERR_NULL;
  if (p->n_timestep <= 0) return imn::set_error("imn_implicit_matrix: empty opt.timestep"), IMN_ERR_SHAPE;
  if (p->nv <= 0 || p->nM <= 0 || p->nu < 0 || nworld < 0 || M_ld < p->nM || out_ld < p->nM)
    return imn::set_error("imn_implicit_matrix: bad extent or stride"), IMN_ERR_SHAPE;
  if (p->damper && !p->dof_damping) return imn::set_error("imn_implicit_matrix: dof_damping is NULL"), IMN_ERR_NULL;
  if (p->nu > 0 && p->actuation &&
      (!p->moment_rownnz || !p->moment_rowadr || !p->moment_colind || !p->actuator_moment ||
       !p->actuator_velocity_gain || p->moment_ld <= 0))
    return imn::set_error("imn_implicit_matrix: an actuator array is NULL"), IMN_ERR_NULL;
  if (p->nu > 0 && p->actuation && p->ctrl &&
      (!p->gain_g2 || !p->gain_b2 || !p->velocity_gain_out || p->n_coefficients <= 0 || p->ctrl_ld < p->nu))
    return imn::set_error("imn_implicit_matrix: controls without gain coefficients or with a short stride"), IMN_ERR_NULL;
  if (nworld == 0) return IMN_OK;
  // A world whose moment row storage is no longer than nu holds one dof per actuator (or none for others
  // beside a longer row): no work for the batch form.  Such batches, beyond two waves of its blocks (one of
  // the other variant's), and an M whose marks would not fit take the variant without.
  const size_t row_bytes = sizeof(float) * (size_t)((p->nM + 3) & ~3);
  const bool several = p->nu > 0 && p->actuation && p->moment_ld > p->nu;
  const bool few = (int64_t)nworld <= 2 * (int64_t)imn::sm_count() * imn::kRowsBlocksPerSm * imn::kMatrixWarps;
  const bool rows = (several || few) && 2 * row_bytes <= 227 * 1024;
  const auto kernel = rows ? imn::implicit_matrix_kernel<true> : imn::implicit_matrix_kernel<false>;
  const size_t per_warp = (rows ? 2 : 1) * row_bytes;  // qD and the marks
  int warps = imn::kMatrixWarps;
  while (warps > 1 && per_warp * warps > 227 * 1024) warps /= 2;
  const size_t bytes = per_warp * warps;
  if (bytes > 227 * 1024) return imn::set_error("imn_implicit_matrix: nM %d too large", p->nM), IMN_ERR_LIMIT;
  {
    const cudaError_t e = imn::allow_shared(kernel, bytes);
    if (e != cudaSuccess)
      return imn::set_error("imn_implicit_matrix: cudaFuncSetAttribute: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  }
  const cudaError_t e = imn::launch_chained(kernel, (nworld + warps - 1) / warps, 32 * warps, bytes, (cudaStream_t)stream,
                                            *p, M, M_ld, out, out_ld, nworld);
  if (e != cudaSuccess) return imn::set_error("imn_implicit_matrix: launch failed: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  return IMN_OK;
}

extern "C" int imn_advance(const ImnAdvance* p, const float* qacc, int64_t qacc_ld, int32_t nworld, void* stream) {
  if (!p || !qacc || !p->qvel || !p->qpos || !p->jnt_type || !p->jnt_dofadr || !p->jnt_qposadr || !p->timestep)
    return imn::set_error("imn_advance: NULL argument"), IMN_ERR_NULL;
  if (p->n_timestep <= 0) return imn::set_error("imn_advance: empty opt.timestep"), IMN_ERR_SHAPE;
  if (p->njnt <= 0 || p->nv <= 0 || p->nq < p->nv || nworld < 0 || qacc_ld < p->nv || p->qvel_ld < p->nv ||
      p->qpos_ld < p->nq)
    return imn::set_error("imn_advance: bad extent or stride"), IMN_ERR_SHAPE;
  if (nworld == 0) return IMN_OK;
  const size_t bytes = sizeof(float) * 32 * ((size_t)imn::advance_stride(p->nq) + 2 * (size_t)imn::advance_stride(p->nv));
  if (bytes > 227 * 1024) return imn::set_error("imn_advance: nq %d too large", p->nq), IMN_ERR_LIMIT;
  {
    const cudaError_t e = imn::allow_shared(imn::advance_kernel, bytes);
    if (e != cudaSuccess)
      return imn::set_error("imn_advance: cudaFuncSetAttribute: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  }
  const cudaError_t e = imn::launch_chained(imn::advance_kernel, (unsigned)((nworld + 31) / 32), 32 * imn::kAdvanceWarps, bytes,
                                            (cudaStream_t)stream, *p, qacc, qacc_ld, nworld);
  if (e != cudaSuccess) return imn::set_error("imn_advance: launch failed: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  return IMN_OK;
}
