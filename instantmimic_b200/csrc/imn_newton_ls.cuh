// imn_newton_ls.cuh -- exact line search on the piecewise-quadratic cost along the
// search direction (reference: newton_stages.py:182-367), one warp, rows over lanes.
//
// The search is a sequence of evaluation passes over the inequality / friction rows:
// pass 0 at alpha = 0 (absolute costs), pass 1 at the first Newton step, then one pass per
// bracket iteration at three step sizes.  A lane keeps its first two rows prepared in
// registers and prepares further rows (more than 64 inequality rows) from shared memory once
// per pass, for all step sizes of the pass; each lane adds its rows in ascending order, as a
// strided loop would.
#pragma once

#include "imn_newton_linalg.cuh"

namespace imn {

// Sums of one lane's friction-loss rows (ne+lane, ne+lane+32, ... below nef, ascending) at NA step
// sizes, each row prepared from shared memory once.  Kept out of line: models without friction-loss
// rows never run it, and the line search's resident code stays small (the kernel is bound by instruction
// fetch).  Friction rows come before a lane's inequality rows, so these are added to its sums by the
// common path.  (Every row of a lane in this general form, prepared for each step size: 35-dof
// chains with 5 friction rows, 1000 worlds, 399 us against 339.)
template <int NA>
struct Sums {
  Vec3 v[NA];
};
template <int NA>
__device__ __noinline__ Sums<NA> ls_friction_rows(const float* floss, const float* D, const float* Jaref, const float* jv, int ne,
                                                  int nef, int lane, float a0, float a1, float a2, bool absolute) {
  const float al[3] = {a0, a1, a2};
  Sums<NA> acc;
#pragma unroll
  for (int k = 0; k < NA; ++k) acc.v[k] = v3(0.0f, 0.0f, 0.0f);
#pragma unroll 1
  for (int r = ne + lane; r < nef; r += 32) {
    const Row row = make_row(true, true, floss[r], D[r], Jaref[r], jv[r]);
#pragma unroll
    for (int k = 0; k < NA; ++k) acc.v[k] = acc.v[k] + row_at(row, al[k], absolute);
  }
  return acc;
}

struct LineSearchResult {
  float alpha, improvement, noise_floor;
  bool converged;
  int passes;  // row-evaluation passes made
};

// Row sums of the warp at NA step sizes (each lane's own part).
template <int NA>
__device__ __forceinline__ void ls_rows(const World& s, const IneqRow& rowa, const IneqRow& rowb, bool fric, int more,
                                        const float (&al)[NA], Vec3 (&acc)[NA]) {
#pragma unroll
  for (int k = 0; k < NA; ++k) acc[k] = v3(0.0f, 0.0f, 0.0f);
  if (fric) {  // warp-uniform, rare
    const Sums<NA> f =
        ls_friction_rows<NA>(s.floss, s.Dsm, s.Jaref, s.jv, s.ne, s.nef, s.lane, al[0], al[NA / 2], al[NA - 1], false);
#pragma unroll
    for (int k = 0; k < NA; ++k) acc[k] = f.v[k];
  }
#pragma unroll
  for (int k = 0; k < NA; ++k) {
    ineq_add(rowa, al[k], 0.5f * al[k], acc[k]);
    ineq_add(rowb, al[k], 0.5f * al[k], acc[k]);
  }
#pragma unroll 1
  for (int r = more; r < s.nefc; r += 32) {
    const IneqRow row = ineq_row(s.Dsm[r], s.Jaref[r], s.jv[r]);
#pragma unroll
    for (int k = 0; k < NA; ++k) ineq_add(row, al[k], 0.5f * al[k], acc[k]);
  }
}

__device__ __forceinline__ LineSearchResult line_search(const World& s, float search_dot, float tolerance,
                                                        float ls_tolerance, float scale, float eps,
                                                        int ls_iterations) {
  const int lane = s.lane, nv = s.nv, ne = s.ne, nef = s.nef, nefc = s.nefc, bd = s.bd;
  float q[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
  for (int i = lane; i < nv; i += 32) {
    const float si = s.search[i];
    q[0] = fmaf(si, s.Ma[i] - s.qfs[i], q[0]);
    q[1] = fmaf(0.5f * si, s.mv[i], q[1]);
  }
#pragma unroll 1
  for (int r = lane; r < ne; r += 32) {
    const float j = s.jv[r], jvD = j * s.Dsm[r];
    q[0] = fmaf(jvD, s.Jaref[r], q[0]);
    q[1] = fmaf(0.5f * j, jvD, q[1]);
  }
  const int ra = ne + lane, rb = ra + 32;
  const bool va = ra >= nef && ra < nefc, vb = rb >= nef && rb < nefc;
  const bool fric = nef > ne;
  int more = rb + 32;  // the lane's first inequality row that is not held in registers
  if (fric)
    while (more < nef) more += 32;
  const IneqRow rowa = ineq_row(va ? s.Dsm[ra] : 0.0f, va ? s.Jaref[ra] : 1.0f, va ? s.jv[ra] : 0.0f);
  const IneqRow rowb = ineq_row(vb ? s.Dsm[rb] : 0.0f, vb ? s.Jaref[rb] : 1.0f, vb ? s.jv[rb] : 0.0f);

  // pass 0: absolute costs at alpha = 0
  LineSearchResult out;
  out.alpha = 0.0f, out.improvement = 0.0f, out.converged = false, out.passes = 1;
  if (fric) {
    const Vec3 z = ls_friction_rows<1>(s.floss, s.Dsm, s.Jaref, s.jv, ne, nef, lane, 0.0f, 0.0f, 0.0f, true).v[0];
    q[2] = z.c0, q[3] = z.c1, q[4] = z.c2;
  }
  {
    auto at_zero = [&](const IneqRow& r) {
      if (r.on0) q[2] = q[2] - r.neg_cost0, q[3] = q[3] + r.q1r, q[4] = q[4] + r.h;
    };
    at_zero(rowa);
    at_zero(rowb);
#pragma unroll 1
    for (int r = more; r < nefc; r += 32) at_zero(ineq_row(s.Dsm[r], s.Jaref[r], s.jv[r]));
  }
  ls_sum(q, bd, lane);
  const float q1 = q[0], q2 = q[1];
  const Vec3 p0 = v3(0.0f, q1, 2.0f * q2) + v3(q[2], q[3], q[4]);
  // Roots and quotients take 110 cycles each and come in pairs: one for the lower half of the warp, one for the upper.
  const bool up = lane >= 16;
  const float root = sqrtf(up ? 2.0f * fmaxf(q[2], 0.0f) * fmaxf(q[4], 0.0f) : search_dot);
  const float snorm = __shfl_sync(IMN_FULL_MASK, root, 0);
  const float gtol = fmaxf(tolerance * ls_tolerance * snorm * scale, 1e-06f);
  const float q1_abs = __shfl_sync(IMN_FULL_MASK, root, 16) + fabsf(q1);
  const float gtol_accept = fmaxf(gtol, eps * q1_abs);
  const float quotient = safe_div(up ? q1_abs : p0.c1, p0.c2);
  const float a_in = -__shfl_sync(IMN_FULL_MASK, quotient, 0);
  out.noise_floor = eps * fmaxf(1.0f, __shfl_sync(IMN_FULL_MASK, quotient, 16));
  if (fabsf(p0.c1) < eps * q1_abs) {
    out.converged = true;
    return out;
  }

  // pass 1: the first Newton step
  Vec3 lo, hi;
  float lo_alpha, hi_alpha;
  {
    const float al[1] = {a_in};
    Vec3 acc[1];
    ls_rows<1>(s, rowa, rowb, fric, more, al, acc);
    float r3[3] = {acc[0].c0, acc[0].c1, acc[0].c2};
    ls_sum(r3, bd, lane);
    const Vec3 lo_in = eval_quad(q1, q2, a_in) + v3(r3[0], r3[1], r3[2]);
    out.passes = 2;
    if (fabsf(lo_in.c1) < gtol_accept && lo_in.c0 < 0.0f) {
      out.converged = true;
      out.alpha = a_in;
      out.improvement = -lo_in.c0;
      return out;
    }
    const Vec3 p0_delta = v3(0.0f, p0.c1, p0.c2);
    const bool lo_less = lo_in.c1 < p0.c1;
    lo = lo_less ? lo_in : p0_delta;
    lo_alpha = lo_less ? a_in : 0.0f;
    hi = lo_less ? p0_delta : lo_in;
    hi_alpha = lo_less ? 0.0f : a_in;
  }

  // bracket passes
#pragma unroll 1
  for (int pass = 0; pass < ls_iterations; ++pass) {
    const float step = safe_div(up ? hi.c1 : lo.c1, up ? hi.c2 : lo.c2);
    const float al[3] = {lo_alpha - __shfl_sync(IMN_FULL_MASK, step, 0), hi_alpha - __shfl_sync(IMN_FULL_MASK, step, 16),
                         0.5f * (lo_alpha + hi_alpha)};
    Vec3 acc[3];
    ls_rows<3>(s, rowa, rowb, fric, more, al, acc);
    float r9[9] = {acc[0].c0, acc[0].c1, acc[0].c2, acc[1].c0, acc[1].c1, acc[1].c2, acc[2].c0, acc[2].c1, acc[2].c2};
    ls_sum(r9, bd, lane);
    out.passes = pass + 3;
    const Vec3 lo_next = eval_quad(q1, q2, al[0]) + v3(r9[0], r9[1], r9[2]);
    const Vec3 hi_next = eval_quad(q1, q2, al[1]) + v3(r9[3], r9[4], r9[5]);
    const Vec3 mid = eval_quad(q1, q2, al[2]) + v3(r9[6], r9[7], r9[8]);
    const bool conv_lo = fabsf(lo_next.c1) < gtol_accept && lo_next.c0 < 0.0f;
    const bool conv_hi = fabsf(hi_next.c1) < gtol_accept && hi_next.c0 < 0.0f;
    const bool conv_mid = fabsf(mid.c1) < gtol_accept && mid.c0 < 0.0f;
    const bool converged = conv_lo || conv_hi || conv_mid;
    bool swap_lo = false, swap_hi = false;
    if (converged) {
      Vec3 best = v3(IMN_MJ_MAXVAL, 0.0f, 0.0f);
      float best_alpha = 0.0f;
      if (conv_lo && lo_next.c0 < best.c0) best = lo_next, best_alpha = al[0];
      if (conv_hi && hi_next.c0 < best.c0) best = hi_next, best_alpha = al[1];
      if (conv_mid && mid.c0 < best.c0) best = mid, best_alpha = al[2];
      lo = hi = best;
      lo_alpha = hi_alpha = best_alpha;
    } else {
      // candidates in the order lo_next, mid, hi_next for the low end and
      // hi_next, mid, lo_next for the high end, each against the end as moved
      bool t;
      t = in_bracket(lo, lo_next);
      if (t) lo = lo_next, lo_alpha = al[0];
      swap_lo |= t;
      t = in_bracket(lo, mid);
      if (t) lo = mid, lo_alpha = al[2];
      swap_lo |= t;
      t = in_bracket(lo, hi_next);
      if (t) lo = hi_next, lo_alpha = al[1];
      swap_lo |= t;
      t = in_bracket(hi, hi_next) || (hi.c1 < 0.0f && hi_next.c1 > 0.0f);
      if (t) hi = hi_next, hi_alpha = al[1];
      swap_hi |= t;
      t = in_bracket(hi, mid);
      if (t) hi = mid, hi_alpha = al[2];
      swap_hi |= t;
      t = in_bracket(hi, lo_next);
      if (t) hi = lo_next, hi_alpha = al[0];
      swap_hi |= t;
    }
    const bool ls_done = converged || (!swap_lo && !swap_hi) ||
                         (lo.c0 < 0.0f && lo.c1 < 0.0f && lo.c1 > -gtol) ||
                         (hi.c0 < 0.0f && hi.c1 > 0.0f && hi.c1 < gtol);
    if (lo.c0 < 0.0f || hi.c0 < 0.0f) {
      const bool lo_better = lo.c0 < hi.c0;
      out.alpha = lo_better ? lo_alpha : hi_alpha;
      out.improvement = -(lo_better ? lo.c0 : hi.c0);
    }
    if (ls_done) {
      out.converged = true;
      break;
    }
  }
  return out;
}

}  // namespace imn
