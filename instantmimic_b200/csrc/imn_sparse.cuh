// imn_sparse.cuh -- numeric phases of the static-pattern sparse L'DL of the Newton
// Hessian, executed by one warp on shared-memory operands.
//
// The reference generates these bodies per model with the index tables baked in
// (sparse_hessian.py:410-480 level factor and backward solve, :528-544 forward
// solve, :571-637 initial assembly, :501-527 incremental update).  Here the tables
// are device arrays (ImnSparsePlan) and the code is generic.  Entries hold N = L D;
// slots are row-major, so an entry's terms are runs of contiguous slots; a level is
// one parallel sweep; levels with few long entries split each entry over a team of
// T lanes joined by a shuffle-down tree of width T.  Every entry sums its terms in
// a fixed order, so results do not depend on scheduling.
#pragma once

#include "imn_newton_dev.cuh"

namespace imn {

// The model's and the plan's tables as the fused kernel reads them.  TSM: copies in shared memory,
// one per CTA (slots: 4 a | 4 b << 9 | (entry of M + 1) << 18; orig widened); else the arrays of
// ImnModel / ImnSparsePlan in global memory, slots and orig through the plan.
struct Tables {
  const uint4 *mulm, *fstep;
  const uint2* bstep;
  const uint32_t *slots, *orig, *pmask;
};
template <bool TSM, class T>
__device__ __forceinline__ T tab_at(const T* p) {
  return TSM ? *p : __ldg(p);
}
template <bool TSM>
__device__ __forceinline__ int tab_orig(const Tables& tab, const ImnSparsePlan& P, int j) {
  return TSM ? (int)tab.orig[j] : (int)__ldg(P.orig + j);
}

// N[rhs + j] = grad[dof of elimination index j], thread `t` of `threads`; the caller's barrier follows
template <bool TSM>
__device__ __forceinline__ void sp_load_rhs(const ImnSparsePlan& P, const Tables& tab, float* N, const float* grad, int t, int threads) {
#pragma unroll 1
  for (int j = t; j < P.nv; j += threads) N[P.nfac + j] = grad[tab_orig<TSM>(tab, P, j)];
}
// N[rhs + j] = grad[dof of elimination index j]
__device__ __forceinline__ void sp_load_rhs(const ImnSparsePlan& P, float* N, const float* grad, int lane) {
#pragma unroll 1
  for (int j = lane; j < P.nv; j += 32) N[P.nfac + j] = grad[__ldg(P.orig + j)];
  __syncwarp();
}

// Left-looking numeric factor over elimination-tree levels; the right-hand side
// rides as the augmented last row (forward solve).
__device__ __forceinline__ void sp_factor_levels(const ImnSparsePlan& P, float* N, float* iD, int lane) {
#pragma unroll 1
  for (int l = 0; l < P.nlevels; ++l) {
    const int e0 = __ldg(P.lvl_ptr + l), e1 = __ldg(P.lvl_ptr + l + 1);
    const int T = __ldg(P.lvl_team + l);
    const int tl = lane & (T - 1), team = lane / T, per = 32 / T;
#pragma unroll 1
    for (int eb = e0; eb < e1; eb += per) {
      const int e = eb + team;
      float v = 0.0f;
      int sl = 0, col = -1;
      if (e < e1) {
        sl = __ldg(P.ent_slot + e);
        col = __ldg(P.ent_col + e);
        const int r1 = __ldg(P.run_ptr + e + 1);
#pragma unroll 1
        for (int r = __ldg(P.run_ptr + e); r < r1; ++r) {
          const uint32_t ab = __ldg(P.run_ab + r), kl = __ldg(P.run_kl + r);
          const float* pa = N + (ab & 0xFFFFu);
          const float* pb = N + (ab >> 16);
          const float* pd = iD + (kl & 0xFFFFu);
          const int len = (int)(kl >> 16);
#pragma unroll 2
          for (int t = tl; t < len; t += T) v = fmaf(pa[t] * pb[t], pd[t], v);
        }
      }
#pragma unroll 1
      for (int off = T >> 1; off > 0; off >>= 1) v = v + __shfl_down_sync(IMN_FULL_MASK, v, off, T);
      if (e < e1 && tl == 0) {
        const float w = N[sl] - v;
        N[sl] = w;
        if (col >= 0) iD[col] = 1.0f / w;
      }
    }
    __syncwarp();
  }
}

__device__ __forceinline__ float sp_at(const float* N, uint32_t offset) {
  return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(N) + offset);
}
// The same factorisation driven by the step records (ImnSparsePlan::fstep): one 128-bit load,
// issued a step ahead, gives a lane its run of terms and its entry as byte offsets from N[0], so
// that a term costs its three reads, two multiplications and a predicate.
//
// A factorisation is a chain of steps, most of them with few terms, so what counts is a step's own
// latency.  The records of a tree's plan begin with the sweeps of a lane per entry and one run of
// terms; these have a loop of their own that asks a record for nothing but its terms and its diagonals.
// With one loop for every kind of step, a step without any terms took 300 cycles, 100 of them in the
// test for a reduction tree that it does not have, 130 in 1 / w (which only steps with a diagonal
// need); the loop for them takes 50.  us per solve, one loop -> two: 34 dofs (16 steps) 16 worlds 125.6 -> 112.5,
// 8192 worlds 561 -> 539; 35 dofs (21 steps) 16 worlds 229 -> 207, 16384 worlds 2330 -> 2277; 56 dofs (47 steps), 4096
// worlds 1097 -> 1088.  In full batches the size of the code counts as much: with the next four terms'
// reads in flight 112.5 / 550 / 207 / 2345 / 1123, with two sweeps of a level at once on top 56 dofs at 1200.
//
// SHARE: the warps of a team take the sweeps of a level in turn, for plans whose sweeps mostly have company in
// their level (ImnSparsePlan::pairs).  56 dofs (47 steps in 22 levels): 16 worlds 272 -> 245 us, 592 worlds 356 -> 330.
// Elsewhere the barriers cost more than the few extra sweeps: 34 dofs (16 in 13) 112.4 -> 114.1, 592 worlds
// 139.9 -> 145.5; 35 dofs (21 in 16) 207.0 -> 208.0.
// Reads past a lane's last term are not added.  They stay inside the world's shared memory: a lane
// reads fewer than (terms of the step + 4) x team elements past its first one, at most 5 nv, and six
// vectors of up4(nv + 1) elements follow 1 / D.
// v plus the lane's terms of a record
__device__ __forceinline__ float sp_terms(const float* N, const uint4 rec, uint32_t stride, float v) {
  uint32_t a = rec.x & 0xFFFFu, b = rec.x >> 16, d = rec.y & 0xFFFFu;
  int count = (int)(rec.z & 0xFFFFu);
#pragma unroll 1
  for (int left = (int)((rec.w >> 8) & 0xFFu); left > 0; left -= 4, count -= 4) {
    float ab[4], q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) ab[k] = sp_at(N, a + stride * k) * sp_at(N, b + stride * k), q[k] = sp_at(N, d + stride * k);
    a += 4 * stride, b += 4 * stride, d += 4 * stride;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (count > k) v = fmaf(ab[k], q[k], v);
  }
  return v;
}
__device__ __forceinline__ void sp_store(float* N, const uint4 rec, float w) {
  char* at = reinterpret_cast<char*>(N);
  if (rec.w & 1u) *reinterpret_cast<float*>(at + (rec.y >> 16)) = w;
  if (rec.w & 64u) {
    const uint32_t diag = rec.z >> 16;
    const float inv = 1.0f / (diag ? w : 1.0f);
    if (diag) *reinterpret_cast<float*>(at + diag) = inv;
  }
}

// `part` of `parts` warps; sync() orders the team's warps.
template <bool TSM, bool SHARE, class Sync>
__device__ __forceinline__ void sp_factor_steps(const ImnSparsePlan& P, const Tables& tables, float* N, int lane, int part, int parts,
                                                Sync sync) {
  const uint4* tab = tables.fstep + lane;
  uint4 cur = tab_at<TSM>(tab);
  int s = P.nfstep;
  int turn = 0;  // the warp whose sweep it is
  // a lane per entry, one run each
#pragma unroll 1
  for (; s > 0 && (cur.w & 0x3Cu) == 32u; --s) {
    tab += 32;
    const uint4 nxt = tab_at<TSM>(tab);
    if (!SHARE || turn == part) {
      const float start = sp_at(N, cur.y >> 16);
      const float v = sp_terms(N, cur, 4u, 0.0f);
      sp_store(N, cur, start - v);
    }
    if (SHARE) {
      turn = turn + 1 < parts ? turn + 1 : 0;
      if (cur.w & 2u) sync(), turn = 0;
    } else {
      __syncwarp();
    }
    cur = nxt;
  }
  float v = 0.0f;
#pragma unroll 1
  for (; s > 0; --s) {
    tab += 32;
    const uint4 nxt = tab_at<TSM>(tab);
    if (!SHARE || turn == part) {
      const float start = sp_at(N, cur.y >> 16);
      const uint32_t log_team = __reduce_or_sync(IMN_FULL_MASK, (cur.w >> 2) & 7u);  // the same in every lane, and known to be
      v = sp_terms(N, cur, 4u << log_team, v);
      if (cur.w & 32u) {
        if (log_team > 3) {
          if (log_team > 4) v = v + __shfl_down_sync(IMN_FULL_MASK, v, 16, 32);
          v = v + __shfl_down_sync(IMN_FULL_MASK, v, 8, 16);
        }
        if (log_team > 2) v = v + __shfl_down_sync(IMN_FULL_MASK, v, 4, 8);
        if (log_team > 1) v = v + __shfl_down_sync(IMN_FULL_MASK, v, 2, 4);
        if (log_team > 0) v = v + __shfl_down_sync(IMN_FULL_MASK, v, 1, 2);
        sp_store(N, cur, start - v);
        v = 0.0f;
      }
    }
    if (SHARE) {
      if (cur.w & 32u) turn = turn + 1 < parts ? turn + 1 : 0;
      if (cur.w & 2u) sync(), turn = 0;
    } else {
      __syncwarp();
    }
    cur = nxt;
  }
}

// Forward solve with a stored factor (rows by level).
__device__ __forceinline__ void sp_forward(const ImnSparsePlan& P, float* N, const float* iD,
                                           const float* grad, int lane) {
  const int rhs = P.nfac;
#pragma unroll 1
  for (int l = 0; l < P.nlevels; ++l) {
    const int q1 = __ldg(P.f_lvl + l + 1);
#pragma unroll 1
    for (int q = __ldg(P.f_lvl + l) + lane; q < q1; q += 32) {
      const int j = __ldg(P.f_row + q);
      float v = grad[__ldg(P.orig + j)];
      const float* rowp = N + __ldg(P.row_start + j);
      const int k0 = __ldg(P.rk_ptr + j), cnt = __ldg(P.rk_ptr + j + 1) - k0;
#pragma unroll 1
      for (int t = 0; t < cnt; ++t) {
        const int k = __ldg(P.rk + k0 + t);
        v = fmaf(-(rowp[t] * iD[k]), N[rhs + k], v);
      }
      N[rhs + j] = v;
    }
    __syncwarp();
  }
}

// Backward solve (levels in reverse, each finished unknown pushes its column terms
// to its descendants), search = -x, and the sums (sum x^2, sum grad x) in the order
// of a block of `bd` threads: strided partials, a tree per warp, warps in order.
__device__ __forceinline__ void sp_backward(const ImnSparsePlan& P, float* N, const float* iD,
                                            const float* grad, float* search, int bd, int lane,
                                            float& sum0, float& sum1) {
  const int rhs = P.nfac, n = P.nv;
#pragma unroll 1
  for (int l = 0; l < P.nlevels; ++l) {
    const int p1 = __ldg(P.b_lvl + l + 1);
#pragma unroll 1
    for (int p = __ldg(P.b_lvl + l) + lane; p < p1; p += 32) {
      const int i = __ldg(P.b_src + p), j = __ldg(P.b_dst + p);
      N[rhs + j] = fmaf(-N[__ldg(P.b_slot + p)], N[rhs + i] * iD[i], N[rhs + j]);
    }
    __syncwarp();
  }
  float ra = 0.0f, rb = 0.0f;
#pragma unroll 1
  for (int w = 0; w < bd / 32; ++w) {
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 1
    for (int j = lane + 32 * w; j < n; j += bd) {
      const int d = __ldg(P.orig + j);
      const float v = N[rhs + j] * iD[j];
      search[d] = -v;
      s0 = fmaf(v, v, s0);
      s1 = fmaf(grad[d], v, s1);
    }
    ra = ra + warp_tree_sum(s0);
    rb = rb + warp_tree_sum(s1);
  }
  sum0 = ra, sum1 = rb;
  __syncwarp();
}

// sp_backward driven by the step records (ImnSparsePlan::bstep); returns the sums, grad . grad among them.
template <bool TSM>
__device__ __forceinline__ SearchSums sp_backward_steps(const ImnSparsePlan& P, const Tables& tables, float* N, const float* iD,
                                                        const float* grad, float* search, int bd, int lane) {
  const uint2* tab = tables.bstep + lane;
  uint2 cur = tab_at<TSM>(tab);
#pragma unroll 1
  for (int s = P.nbsweep; s > 0; --s) {
    tab += 32;
    const uint2 nxt = tab_at<TSM>(tab);
    const uint32_t to = cur.y >> 16;
    const float x = sp_at(N, cur.x >> 16) * sp_at(N, cur.y & 0xFFFCu);
    const float r = fmaf(-sp_at(N, cur.x & 0xFFFCu), x, sp_at(N, to));
    if (cur.x & 1u) *reinterpret_cast<float*>(reinterpret_cast<char*>(N) + to) = r;
    if (cur.y & 1u) __syncwarp();
    cur = nxt;
  }
  const SearchSums sum = search_sums(P.nv, bd, lane, [&](int j, float& x, float& gx, float& g) {
    const int d = tab_orig<TSM>(tables, P, j);
    x = N[P.nfac + j] * iD[j];
    gx = grad[d], g = grad[j];
    search[d] = -x;
  });
  __syncwarp();
  return sum;
}

// Count one pattern violation in the world's counter (last element of its hfactor);
// the first one of a world is reported (sparse_hessian.py:521-523, 619-620).
__device__ __forceinline__ void sp_violation(float* counter, int world, const char* what) {
  if (counter && atomicAdd(counter, 1.0f) == 0.0f)
    printf("sparse Hessian: world %d %s outside the declared coupling pattern\n", world, what);
}

}  // namespace imn
