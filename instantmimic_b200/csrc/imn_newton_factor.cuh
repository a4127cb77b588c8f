// imn_newton_factor.cuh -- upper Cholesky H = U^T U of one world with the
// right-hand side carried as one more column (forward solve), then the back
// substitution (reference: newton_stages.py:546-609).
//
// Storage: A is (nv+1) x ldu in shared memory.  U[r][c] (r <= c <= nv; column nv
// is the carried right-hand side) lives at A[r*ldu + c]; H[r][c] (r <= c < nv)
// at A[(c+1)*ldu + r], so H survives the factorisation for the next incremental
// update.  dinv[r] = 1 / U[r][r].
//
// Order of operations (identical to the CPU oracle): every entry starts from H
// (or grad) and subtracts U[t][r] * U[t][c] for t = 0, 1, ... with fused
// multiply-adds; the pivot is sqrtf; the row is scaled by the reciprocal pivot.
//
// Mapping: 16 rows at a time.  A lane owns K columns c = b0 + lane + 32k (K = 1 or 2 by the
// columns that are left; columns past the 64th follow when the block's rows are done) and keeps the block's 16 running
// sums of each in registers, two rows to a pair, so that one instruction does two of the fused multiply-adds (a
// register and an instruction per row instead: 48 dofs x 96 rows, 4096 worlds 1140 us against 1067, 32 x 128, 8192 worlds 1784
// against 1775, others equal).  Phase 1 adds the terms of all earlier rows (one shared-memory read of U[t][c] per
// column and four 128-bit broadcast reads of U[t][b0..b0+15] feed 8 K pairs).  Phase 2 eliminates the block's
// rows.  Its chain per row is scale -> own square -> shuffle -> root -> reciprocal: the pivot of row
// r + 1 is its lane's own sum after row r, which that lane has at once, so it travels while the
// other sums wait for row r to come back from shared memory as four broadcast reads (the block's
// entries of a row sit in 16 lanes; fetched by 15 shuffles each row cost 700 cycles).  Four rows per
// trip, so that every sum has a fixed register and the reads start on 16-byte boundaries.
#pragma once

#include "imn_newton_linalg.cuh"

namespace imn {

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

template <int K>
__device__ __forceinline__ void factor_block(const World& s, int b0) {
  const int lane = s.lane, nv = s.nv, ldu = s.ldu, nr = min(16, nv - b0);
  float* A = s.A;
  Pair acc[K][8];  // rows 2h and 2h + 1
  int cc[K];
  bool valid[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int c = b0 + lane + 32 * k;
    valid[k] = c <= nv;
    cc[k] = valid[k] ? c : nv;
    // H column cc (rows b0..), or grad for the carried column; rows below the diagonal and past the
    // last hold values that are never stored or read by another lane
    const float* src = (cc[k] < nv ? A + (cc[k] + 1) * ldu : s.grad) + b0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      Pair2 h = {0ull, 0ull};
      if (4 * g < nr) h = ld_pair2(src + 4 * g);
      acc[k][2 * g] = h.a, acc[k][2 * g + 1] = h.b;
    }
  }
  // phase 1: terms of rows t < b0
#pragma unroll 2
  for (int t = 0; t < b0; ++t) {
    const float* Ut = A + t * ldu;
    Pair uc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) uc[k] = make_pair(-Ut[cc[k]], -Ut[cc[k]]);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const Pair2 u = ld_pair2(Ut + b0 + 4 * g);  // past the last row: values of the next rows, never stored
#pragma unroll
      for (int k = 0; k < K; ++k)
        acc[k][2 * g] = pair_fma(u.a, uc[k], acc[k][2 * g]), acc[k][2 * g + 1] = pair_fma(u.b, uc[k], acc[k][2 * g + 1]);
    }
  }
  IMN_MARK(s, 12);
  // phase 2: acc[k][q / 2] belongs to row g + q
  const auto row = [&](int k, int q) { return q & 1 ? pair_y(acc[k][q >> 1]) : pair_x(acc[k][q >> 1]); };
  float pv = __shfl_sync(IMN_FULL_MASK, row(0, 0), 0);
#pragma unroll 1
  for (int g = 0; g < nr; g += 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = g + q;
      if (r >= nr) break;  // warp-uniform
      const float dg = sqrtf(pv), rinv = 1.0f / dg;
      float* Ur = A + (b0 + r) * ldu;
      float u[K];
#pragma unroll
      for (int k = 0; k < K; ++k) u[k] = row(k, q) * rinv;
      pv = __shfl_sync(IMN_FULL_MASK, fmaf(-u[0], u[0], row(0, q + 1)), r + 1);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (valid[k] && cc[k] >= b0 + r) Ur[cc[k]] = k == 0 && lane == r ? dg : u[k];
      if (lane == 0) s.dinv[b0 + r] = rinv;
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const Pair2 m = ld_pair2(Ur + b0 + g + 4 * h);
#pragma unroll
        for (int k = 0; k < K; ++k) {  // sums of finished rows go on as pairs of others
          const Pair nu = make_pair(-u[k], -u[k]);
          if (4 * h + 1 > q) acc[k][2 * h] = pair_fma(m.a, nu, acc[k][2 * h]);
          if (4 * h + 3 > q) acc[k][2 * h + 1] = pair_fma(m.b, nu, acc[k][2 * h + 1]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int h = 0; h < 8; ++h) acc[k][h] = h < 6 ? acc[k][h + 2] : 0ull;
  }
  __syncwarp();
  IMN_MARK(s, 13);
}

// The block's rows at one column c0 + lane behind the 64 of factor_block: the same sums, scaled with the
// stored reciprocals.
__device__ __forceinline__ void factor_follow(const World& s, int b0, int c0) {
  const int nv = s.nv, ldu = s.ldu, nr = min(16, nv - b0), c = c0 + s.lane, cc = min(c, nv);
  float* A = s.A;
  float acc[16];
  const float* src = (cc < nv ? A + (cc + 1) * ldu : s.grad) + b0;
#pragma unroll
  for (int g = 0; g < 16; ++g) acc[g] = g < nr ? src[g] : 0.0f;
#pragma unroll 1
  for (int t = 0; t < b0; ++t) {
    const float uc = A[t * ldu + cc];
#pragma unroll
    for (int g = 0; g < 16; ++g) acc[g] = fmaf(-A[t * ldu + b0 + g], uc, acc[g]);
  }
#pragma unroll 1
  for (int r = 0; r < nr; ++r) {
    float* Ur = A + (b0 + r) * ldu;
    const float u = acc[0] * s.dinv[b0 + r];
    if (c <= nv) Ur[c] = u;
#pragma unroll
    for (int h = 1; h < 16; ++h) acc[h - 1] = fmaf(-Ur[min(b0 + r + h, nv)], u, acc[h]);
  }
  __syncwarp();
}

__device__ __forceinline__ SearchSums factor_solve(const World& s, bool factor) {
  const int lane = s.lane, nv = s.nv, ldu = s.ldu;
  float* A = s.A;
  if (factor) {
#pragma unroll 1
    for (int b0 = 0; b0 < nv; b0 += 16) {
      const int columns = nv + 1 - b0;
      if (columns <= 32)
        factor_block<1>(s, b0);
      else
        factor_block<2>(s, b0);
      if (columns > 64) factor_follow(s, b0, b0 + 64);
    }
  } else {
    // forward substitution with the stored factor: unknown r receives its terms
    // in ascending order, exactly as the carried column of the factorisation
#pragma unroll 1
    for (int i = lane; i < nv; i += 32) s.xsm[i] = s.grad[i];
    __syncwarp();
#pragma unroll 1
    for (int t = 0; t < nv; ++t) {
      const float yt = s.xsm[t] * s.dinv[t];
      const float* Ut = A + t * ldu;
      __syncwarp();
#pragma unroll 1
      for (int r = t + 1 + lane; r < nv; r += 32) s.xsm[r] = fmaf(-Ut[r], yt, s.xsm[r]);
      if (lane == 0) A[t * ldu + nv] = yt;
      __syncwarp();
    }
  }
  // back substitution, 16-row blocks from the last: later blocks' columns in
  // ascending order first, then the block's own columns from its last inwards.  A lane reads its row
  // four columns at a time and ahead, so that a column costs a product, a shuffle and a sum
  // (us per solve, a column at a time -> four: 27 dofs x 32 rows, 16384 worlds 768 -> 759, 35 dofs, 1000 worlds 348 -> 341, 40 x
  // 100, 300 worlds 212 -> 204, 64 x 512, 4096 worlds 4022 -> 3947; all sixteen unrolled, code that full batches pay for,
  // 27 dofs 784, 48 dofs 1143 -> 1169).
#pragma unroll 1
  for (int b0 = ((nv - 1) / 16) * 16; b0 >= 0; b0 -= 16) {
    const int nr = min(16, nv - b0);
    const int r = b0 + (lane < nr ? lane : 0);  // the other lanes repeat the first row and store nothing
    const float* Ur = A + r * ldu;
    float acc = Ur[nv];
    const float di = s.dinv[r];
    int g = (nr - 1) & ~3;
    float4 u = ld4(Ur + b0 + g);  // past the last row: values of the next rows, never used
#pragma unroll 1
    for (int c = b0 + 16; c < nv; c += 4) {
      const float4 q = ld4(Ur + c), x = ld4(s.xsm + c);
      acc = fmaf(-q.x, x.x, acc);
      if (c + 1 < nv) acc = fmaf(-q.y, x.y, acc);
      if (c + 2 < nv) acc = fmaf(-q.z, x.z, acc);
      if (c + 3 < nv) acc = fmaf(-q.w, x.w, acc);
    }
    const auto column = [&](int k, float uk) {
      const float xk = __shfl_sync(IMN_FULL_MASK, acc * di, k);
      if (lane < k) acc = fmaf(-uk, xk, acc);
    };
#pragma unroll 1
    for (; g >= 0; g -= 4) {
      const float4 next = ld4(Ur + b0 + max(g - 4, 0));
      if (g + 3 < nr) column(g + 3, u.w);  // warp-uniform, as all of these
      if (g + 2 < nr) column(g + 2, u.z);
      if (g + 1 < nr) column(g + 1, u.y);
      column(g, u.x);
      u = next;
    }
    if (lane < nr) s.xsm[r] = acc * di;
    __syncwarp();
  }
  IMN_MARK(s, 14);
  const SearchSums sum = search_sums(nv, s.bd, lane, [&](int i, float& x, float& gx, float& g) {
    x = s.xsm[i];
    gx = g = s.grad[i];
    s.search[i] = -x;
  });
  __syncwarp();
  IMN_MARK(s, 15);
  return sum;
}

}  // namespace imn
