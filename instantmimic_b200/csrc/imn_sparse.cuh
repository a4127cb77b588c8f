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

#include "imn_common.cuh"

namespace imn {

// The model's and the plan's tables as the fused kernel reads them.  TSM: copies in shared memory,
// one per CTA (slots: 4 a | 4 b << 9 | (entry of M + 1) << 18; orig widened); else the arrays of
// ImnModel / ImnSparsePlan in global memory, slots and orig through the plan.
struct Tables {
  const uint4 *mulm, *fstep;
  const uint2* bstep;
  const uint32_t *slots, *orig;
};
template <bool TSM, class T>
__device__ __forceinline__ T tab_at(const T* p) {
  return TSM ? *p : __ldg(p);
}
template <bool TSM>
__device__ __forceinline__ int tab_orig(const Tables& tab, const ImnSparsePlan& P, int j) {
  return TSM ? (int)tab.orig[j] : (int)__ldg(P.orig + j);
}

// N[rhs + j] = grad[dof of elimination index j]
template <bool TSM>
__device__ __forceinline__ void sp_load_rhs(const ImnSparsePlan& P, const Tables& tab, float* N, const float* grad, int lane) {
#pragma unroll 1
  for (int j = lane; j < P.nv; j += 32) N[P.nfac + j] = grad[tab_orig<TSM>(tab, P, j)];
  __syncwarp();
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

// The same factorisation driven by the step records (ImnSparsePlan::fstep): one 128-bit load,
// issued a step ahead, gives a lane its run of terms and its entry as byte offsets from N[0], so
// that a term costs its three reads, two multiplications and a predicate.  Teams of one lane, where
// most terms are, take four terms per trip with constant offsets between them; reads past a lane's
// last term stay inside the world's shared memory and are not added.  (A lane that took the terms
// of its run one by one from scaled indices spent 180 cycles per term step: 34-dof humanoid, 8192
// worlds, 15 k cycles per factorisation.)
__device__ __forceinline__ float sp_at(const float* N, uint32_t offset) {
  return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(N) + offset);
}
// Two sweeps of a level, whose chains of reads and sums run side by side (56 dofs, levels of up to
// three sweeps, 4096 worlds: 1187 -> 1090 us per solve; four terms per trip instead of two: 1125).
__device__ __forceinline__ void sp_two_sweeps(float* N, const uint4 e, const uint4 g) {
  uint32_t a = e.x & 0xFFFFu, b = e.x >> 16, d = e.y & 0xFFFFu, A = g.x & 0xFFFFu, B = g.x >> 16, D = g.y & 0xFFFFu;
  int n = (int)(e.z & 0xFFFFu), m = (int)(g.z & 0xFFFFu);
  const uint32_t slot = e.y >> 16, Slot = g.y >> 16, stride = 4u << ((e.w >> 2) & 7u);
  const float start = sp_at(N, slot), Start = sp_at(N, Slot);
  float v = 0.0f, V = 0.0f;
#pragma unroll 1
  for (int left = (int)((e.w >> 8) & 0xFFu); left > 0; left -= 2, n -= 2, m -= 2) {
    const float p0 = sp_at(N, a) * sp_at(N, b), q0 = sp_at(N, d), P0 = sp_at(N, A) * sp_at(N, B), Q0 = sp_at(N, D);
    a += stride, b += stride, d += stride, A += stride, B += stride, D += stride;
    const float p1 = sp_at(N, a) * sp_at(N, b), q1 = sp_at(N, d), P1 = sp_at(N, A) * sp_at(N, B), Q1 = sp_at(N, D);
    a += stride, b += stride, d += stride, A += stride, B += stride, D += stride;
    if (n > 0) v = fmaf(p0, q0, v);
    if (m > 0) V = fmaf(P0, Q0, V);
    if (n > 1) v = fmaf(p1, q1, v);
    if (m > 1) V = fmaf(P1, Q1, V);
  }
  const int T = 1 << ((e.w >> 2) & 7u);
#pragma unroll 1
  for (int off = T >> 1; off > 0; off >>= 1) {
    const float x = __shfl_down_sync(IMN_FULL_MASK, v, off, T), X = __shfl_down_sync(IMN_FULL_MASK, V, off, T);
    v = v + x, V = V + X;
  }
  const float w = start - v, W = Start - V;
  char* at = reinterpret_cast<char*>(N);
  if (e.w & 1u) *reinterpret_cast<float*>(at + slot) = w;
  if (g.w & 1u) *reinterpret_cast<float*>(at + Slot) = W;
  if ((e.w | g.w) & 64u) {
    const uint32_t di = e.z >> 16, Di = g.z >> 16;
    const float inv = 1.0f / (di ? w : 1.0f), Inv = 1.0f / (Di ? W : 1.0f);
    if (di) *reinterpret_cast<float*>(at + di) = inv;
    if (Di) *reinterpret_cast<float*>(at + Di) = Inv;
  }
}

template <bool TSM, bool PAIR>
__device__ __forceinline__ void sp_factor_steps(const ImnSparsePlan& P, const Tables& tables, float* N, int lane) {
  const uint4* tab = tables.fstep + lane;
  uint4 cur = tab_at<TSM>(tab);
  float v = 0.0f;
#pragma unroll 1
  for (int s = P.nfstep; s > 0; --s) {
    tab += 32;
    const uint4 nxt = tab_at<TSM>(tab);
    const uint32_t fl = cur.w, slot = cur.y >> 16;
    if (PAIR && (fl & 128u)) {  // two sweeps of the level at once
      tab += 32;
      const uint4 then = tab_at<TSM>(tab);
      sp_two_sweeps(N, cur, nxt);
      if (nxt.w & 2u) __syncwarp();
      cur = then;
      --s;
      continue;
    }
    uint32_t a = cur.x & 0xFFFFu, b = cur.x >> 16, d = cur.y & 0xFFFFu;
    int cnt = (int)(cur.z & 0xFFFFu);
    const float start = sp_at(N, slot);
    int left = (int)((fl >> 8) & 0xFFu);
    if ((fl & 0x1Cu) == 0u) {
#pragma unroll 1
      for (; left > 0; left -= 4, cnt -= 4, a += 16, b += 16, d += 16) {
        float p[4], q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) p[k] = sp_at(N, a + 4 * k) * sp_at(N, b + 4 * k), q[k] = sp_at(N, d + 4 * k);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (cnt > k) v = fmaf(p[k], q[k], v);
      }
    } else {
      const uint32_t stride = 4u << ((fl >> 2) & 7u);
#pragma unroll 1
      for (; left > 0; left -= 2, cnt -= 2) {
        const float p0 = sp_at(N, a) * sp_at(N, b), q0 = sp_at(N, d);
        a += stride, b += stride, d += stride;
        const float p1 = sp_at(N, a) * sp_at(N, b), q1 = sp_at(N, d);
        a += stride, b += stride, d += stride;
        if (cnt > 0) v = fmaf(p0, q0, v);
        if (cnt > 1) v = fmaf(p1, q1, v);
      }
    }
    if (fl & 32u) {
      const int T = 1 << ((fl >> 2) & 7u);
#pragma unroll 1
      for (int off = T >> 1; off > 0; off >>= 1) v = v + __shfl_down_sync(IMN_FULL_MASK, v, off, T);
      const float w = start - v;
      if (fl & 1u) *reinterpret_cast<float*>(reinterpret_cast<char*>(N) + slot) = w;
      if (fl & 64u) {
        const uint32_t diag = cur.z >> 16;
        const float inv = 1.0f / (diag ? w : 1.0f);
        if (diag) *reinterpret_cast<float*>(reinterpret_cast<char*>(N) + diag) = inv;
      }
      v = 0.0f;
    }
    if (fl & 2u) __syncwarp();
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

// sp_backward driven by the step records (ImnSparsePlan::bstep).
template <bool TSM>
__device__ __forceinline__ void sp_backward_steps(const ImnSparsePlan& P, const Tables& tables, float* N, const float* iD,
                                                  const float* grad, float* search, int bd, int lane,
                                                  float& sum0, float& sum1) {
  const int rhs = P.nfac, n = P.nv;
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
  float ra = 0.0f, rb = 0.0f;
#pragma unroll 1
  for (int w = 0; w < bd / 32; ++w) {
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 1
    for (int j = lane + 32 * w; j < n; j += bd) {
      const int d = tab_orig<TSM>(tables, P, j);
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

// Count one pattern violation in the world's counter (last element of its hfactor);
// the first one of a world is reported (sparse_hessian.py:521-523, 619-620).
__device__ __forceinline__ void sp_violation(float* counter, int world, const char* what) {
  if (counter && atomicAdd(counter, 1.0f) == 0.0f)
    printf("sparse Hessian: world %d %s outside the declared coupling pattern\n", world, what);
}

}  // namespace imn
