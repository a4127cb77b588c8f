// imn_newton_dev.cuh -- device helpers of the fused Newton kernel: TMA bulk copy
// and mbarrier wrappers, the piecewise row costs of the line search, and the
// reductions that reproduce the reference's summation orders.
#pragma once

#include "imn_common.cuh"

namespace imn {

// ---- TMA bulk copy + mbarrier (sm_90+ PTX) -----------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(void* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// a barrier whose phase is unknown (its copies did not arrive) starts anew
__device__ __forceinline__ void mbar_restart(void* bar, int count) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
  mbar_init(bar, count);
}
__device__ __forceinline__ void mbar_expect_tx(void* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, void* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// 16 bytes by one lane, and the lane's arrival at a barrier once all its copies so far have landed
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void mbar_arrive_copies(void* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(void* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// ---- pairs of floats: one instruction for two fused multiply-adds, each rounded as fmaf rounds it ----------
typedef unsigned long long Pair;
__device__ __forceinline__ Pair make_pair(float x, float y) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float pair_x(Pair a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x;
}
__device__ __forceinline__ float pair_y(Pair a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return y;
}
__device__ __forceinline__ Pair pair_fma(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
struct alignas(16) Pair2 {
  Pair a, b;
};
__device__ __forceinline__ Pair2 ld_pair2(const float* p) { return *reinterpret_cast<const Pair2*>(p); }

// ---- row cost pieces (the statement is in oracle/newton_oracle.c) -------------
__device__ __forceinline__ int row_zone(float x, bool fr, float rf) {
  if (fr) return x <= -rf ? IMN_STATE_LINEARNEG : (x >= rf ? IMN_STATE_LINEARPOS : IMN_STATE_QUADRATIC);
  return x >= 0.0f ? IMN_STATE_SATISFIED : IMN_STATE_QUADRATIC;
}
__device__ __forceinline__ float zone_cost(int z, float x, float D, float f, float rf) {
  if (z == IMN_STATE_QUADRATIC) return ((0.5f * D) * x) * x;
  if (z == IMN_STATE_LINEARNEG) return f * (-0.5f * rf - x);
  if (z == IMN_STATE_LINEARPOS) return f * (-0.5f * rf + x);
  return 0.0f;
}
// One constraint row prepared for repeated evaluation along the search direction.
struct Row {
  float D, ja, j, f, rf, jvD, h, q1r, cost0;
  int z0;  // -1: no row
};
__device__ __forceinline__ Row make_row(bool valid, bool fr, float f, float D, float ja, float j) {
  Row r;
  r.f = fr ? f : 0.0f, r.D = D, r.ja = ja, r.j = j;
  r.rf = fr ? safe_div(f, D) : -1.0f;  // rf < 0 marks an inequality row
  r.z0 = valid ? row_zone(ja, fr, r.rf) : -1;
  r.jvD = j * D;
  r.h = j * r.jvD;
  r.q1r = r.jvD * ja;
  r.cost0 = zone_cost(r.z0, ja, D, r.f, r.rf);
  return r;
}
// (cost(alpha) - cost(0), slope, curvature) at alpha; with `absolute` the first
// component is the cost itself (used at alpha = 0 only).
__device__ __forceinline__ Vec3 row_at(const Row& r, float alpha, bool absolute) {
  if (r.z0 < 0) return v3(0.0f, 0.0f, 0.0f);
  const float x = fmaf(alpha, r.j, r.ja);
  Vec3 o = v3(0.0f, 0.0f, 0.0f);
  int z;
  if (r.rf < 0.0f) {
    z = x < 0.0f ? IMN_STATE_QUADRATIC : IMN_STATE_SATISFIED;
  } else {
    z = row_zone(x, true, r.rf);
    if (z == IMN_STATE_LINEARNEG) o.c1 = -r.f * r.j;
    if (z == IMN_STATE_LINEARPOS) o.c1 = r.f * r.j;
  }
  if (z == IMN_STATE_QUADRATIC) o.c1 = r.jvD * x, o.c2 = r.h;
  if (absolute)
    o.c0 = r.cost0;
  else if (z != r.z0)
    o.c0 = zone_cost(z, x, r.D, r.f, r.rf) - r.cost0;
  else if (z == IMN_STATE_QUADRATIC)
    o.c0 = alpha * fmaf(0.5f * alpha, r.h, r.q1r);
  else if (z == IMN_STATE_LINEARNEG)
    o.c0 = -r.f * (alpha * r.j);
  else if (z == IMN_STATE_LINEARPOS)
    o.c0 = r.f * (alpha * r.j);
  return o;
}
// A plain inequality row (limit or pyramidal contact edge: cost 0.5 D x^2 while x < 0, else
// nothing) prepared for evaluation at several step sizes.  The values equal row_at's.  A lane
// without a row takes D = 0, ja = 1, j = 0, which contributes exact zeros everywhere.
struct IneqRow {
  float ja, j, jvD, h, q1r, hD, neg_cost0;
  bool on0;
};
__device__ __forceinline__ IneqRow ineq_row(float D, float ja, float j) {
  IneqRow r;
  r.ja = ja, r.j = j;
  r.jvD = j * D;
  r.h = j * r.jvD;
  r.q1r = r.jvD * ja;
  r.hD = 0.5f * D;
  r.on0 = ja < 0.0f;
  r.neg_cost0 = r.on0 ? -((r.hD * ja) * ja) : 0.0f;
  return r;
}
// acc += (cost(alpha) - cost(0), slope, curvature)
__device__ __forceinline__ void ineq_add(const IneqRow& r, float alpha, float half_alpha, Vec3& acc) {
  const float x = fmaf(alpha, r.j, r.ja);
  const bool on = x < 0.0f;
  const float same = alpha * fmaf(half_alpha, r.h, r.q1r), enter = (r.hD * x) * x;
  acc.c0 = acc.c0 + (on ? (r.on0 ? same : enter) : r.neg_cost0);
  const float slope = r.jvD * x;
  if (on) acc.c1 = acc.c1 + slope, acc.c2 = acc.c2 + r.h;
}
__device__ __forceinline__ Vec3 eval_quad(float q1, float q2, float alpha) {
  return v3(fmaf(alpha, q1, (alpha * alpha) * q2) + 0.0f, fmaf(2.0f * alpha, q2, q1), 2.0f * q2);
}
__device__ __forceinline__ bool in_bracket(Vec3 x, Vec3 y) {
  return (x.c1 < y.c1 && y.c1 < 0.0f) || (x.c1 > y.c1 && y.c1 > 0.0f);
}
// A friction-loss row's force and state.
__device__ __forceinline__ void eval_friction(float jaref, float D, float floss, float& force, int& state) {
  const float rf = safe_div(floss, D);
  force = -D * jaref, state = IMN_STATE_QUADRATIC;
  if (jaref <= -rf)
    force = floss, state = IMN_STATE_LINEARNEG;
  else if (jaref >= rf)
    force = -floss, state = IMN_STATE_LINEARPOS;
}

// The sums behind a search direction x over the dofs: x . x, grad . x and grad . grad, in the reference's order: one
// value per thread of its logical block (bd = 32 or 64 threads), each thread summing its strided elements, then
// Warp's block reduction, a tree per warp and the later warp added to the first (newton_stages.py:34-38).  The
// physical warp plays both logical warps.  at(j, x, gx, g): x_j, the gradient's entry that goes with it, and the
// j-th entry of the gradient.  A lane's elements (at most 80 dofs: three) are read at once and the trees of the three
// sums run side by side; with a loop and a tree for every sum, a row update with a branch per kind of row and a
// division per convergence measure, a pass took 700 cycles more (us per solve: 34 dofs, 16 worlds 107.9 -> 104.3, 8192 worlds 522
// -> 511; 27 dofs x 32 rows, dense factor, 16384 worlds 808 -> 767; 64 x 512, 4096 worlds 4112 -> 4024).
struct SearchSums {
  float xx, gx, gg;
};
template <class At>
__device__ __forceinline__ SearchSums search_sums(int nv, int bd, int lane, At at) {
  float x[3], h[3], g[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    x[k] = h[k] = g[k] = 0.0f;
    if (lane + 32 * k < nv) at(lane + 32 * k, x[k], h[k], g[k]);
  }
  SearchSums sum = {0.0f, 0.0f, 0.0f};
  const bool two = bd == 64;
#pragma unroll 1
  for (int w = 0; w < (two ? 2 : 1); ++w) {
    SearchSums a = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (!two || (k & 1) == w) a.xx = fmaf(x[k], x[k], a.xx), a.gx = fmaf(h[k], x[k], a.gx), a.gg = fmaf(g[k], g[k], a.gg);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float u = __shfl_down_sync(IMN_FULL_MASK, a.xx, off), v = __shfl_down_sync(IMN_FULL_MASK, a.gx, off),
                  t = __shfl_down_sync(IMN_FULL_MASK, a.gg, off);
      a.xx = a.xx + u, a.gx = a.gx + v, a.gg = a.gg + t;
    }
    sum.xx = sum.xx + a.xx, sum.gx = sum.gx + a.gx, sum.gg = sum.gg + a.gg;
  }
  sum.xx = __shfl_sync(IMN_FULL_MASK, sum.xx, 0);
  sum.gx = __shfl_sync(IMN_FULL_MASK, sum.gx, 0);
  sum.gg = __shfl_sync(IMN_FULL_MASK, sum.gg, 0);
  return sum;
}

// Lane sums of N values at once in the order of N shuffle-down trees, broadcast, then "+0" per
// later logical warp of the line search (newton_stages.py:39-49).  A tree's steps only ever need
// half, a quarter, ... of the lanes, so two values share each step: one half of the lanes goes on
// with the first value, the other half with the second (an addition's operands may come in
// either order), and after five steps value k sits in lanes of its own.  Nine values take 16
// shuffles and additions plus the broadcasts instead of 45.
template <int N>
__device__ __forceinline__ void ls_sum(float (&v)[N], int bd, int lane) {
  constexpr int N1 = (N + 1) / 2, N2 = (N1 + 1) / 2, N3 = (N2 + 1) / 2, N4 = (N3 + 1) / 2;
  static_assert(N4 == 1, "at most 16 values");
  float a[N1], b[N2], c[N3], d[N4];
  auto fold = [&](auto& out, auto& in, int n, int off) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int k = 0; k < n; k += 2) {
      if (k + 1 < n) {
        const float keep = up ? in[k + 1] : in[k], send = up ? in[k] : in[k + 1];
        out[k / 2] = keep + __shfl_xor_sync(IMN_FULL_MASK, send, off);
      } else {
        out[k / 2] = in[k] + __shfl_xor_sync(IMN_FULL_MASK, in[k], off);
      }
    }
  };
  const float zero = bd == 64 ? 0.0f : -0.0f;  // x + -0 is x
  fold(a, v, N, 16);
  fold(b, a, N1, 8);
  fold(c, b, N2, 4);
  fold(d, c, N3, 2);
  const float e = d[0] + __shfl_xor_sync(IMN_FULL_MASK, d[0], 1);
#pragma unroll
  for (int k = 0; k < N; ++k) {
    // value k went up at step s when its index at that step was odd
    const int src = ((k & 1) ? 16 : 0) | ((k & 2) ? 8 : 0) | ((k & 4) ? 4 : 0) | ((k & 8) ? 2 : 0);
    v[k] = __shfl_sync(IMN_FULL_MASK, e, src);
    v[k] = v[k] + zero;
  }
}

// advance an upper-triangle pair (i <= j), enumerated column by column, by `step`
__device__ __forceinline__ void pair_advance(int& i, int& j, int step) {
  i += step;
  while (i > j) i -= j + 1, ++j;
}

// The same enumeration as a table: entry e holds i | j << 8 of the e-th pair (i <= j),
// for every pair of up to 80 indices.  One coalesced load replaces the stepping loop.
struct PairTable {
  uint16_t v[80 * 81 / 2];
  constexpr PairTable() : v() {
    int e = 0;
    for (int j = 0; j < 80; ++j)
      for (int i = 0; i <= j; ++i) v[e++] = (uint16_t)(i | (j << 8));
  }
};
__device__ const PairTable g_pairs = PairTable();
__device__ __forceinline__ void pair_lookup(int e, int& i, int& j) {
  const int p = g_pairs.v[e];
  i = p & 0xFF, j = p >> 8;
}

}  // namespace imn
