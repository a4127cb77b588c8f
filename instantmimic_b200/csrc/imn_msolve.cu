// imn_msolve.cu -- factor + solve of inertia-like matrices (M and M - h qDeriv):
// the tree-structured L'DL and the blocked dense Cholesky.
//
// Tree L'DL (reference: tree_ldl.py:196-359, 419-433).  The reference generates
// straight-line source per model; imn_tree_jit.cu does the same with NVRTC.  The
// kernel here interprets the plan's instruction list instead (the fallback when no
// run-time compiler is installed, and the statement the generated code must match).  A block serves 32 worlds with one warp per group; lane l of
// every warp works on world 32*block + l, all operands of a world live in column
// l of a [slot][32] shared-memory array (bank = lane, so no conflicts), every
// lane of a warp executes the same instruction on its own world, and the only
// synchronisation is the pair of block barriers around the trunk.
//
// Blocked dense Cholesky (reference: indexed_factor.py:15-173, 217-493).  One warp
// per world gathers M through the plan's block-major index table into shared
// memory, factors it (same entry formula as the Newton Hessian factor), carries
// `rhs_count` right-hand sides through the forward and backward substitution and
// stores U (pad x pad, upper) in the caller's workspace.
#include <atomic>

#include "imn_common.cuh"

namespace imn {

enum { OP_LOAD_M, OP_LOAD_Y, OP_ZERO, OP_INV, OP_UPD, OP_SCALE, OP_SUBMUL, OP_MUL, OP_ADD, OP_STORE_X, OP_MULSUB, OP_MULADD };

__device__ __forceinline__ void tree_run(const int4* __restrict__ prog, int lo, int hi, float* col,
                                         const float* __restrict__ Mr, const float* __restrict__ yr,
                                         float* __restrict__ xr, bool live) {
#pragma unroll 1
  for (int pc = lo; pc < hi; ++pc) {
    const int4 ins = __ldg(prog + pc);
    const int dst = ins.y, a = ins.z & 0xFFFF, b = (ins.z >> 16) & 0xFFFF, c = ins.w;
    switch (ins.x) {
      case OP_LOAD_M: col[dst * 32] = Mr[a]; break;
      case OP_LOAD_Y: col[dst * 32] = yr[a]; break;
      case OP_ZERO: col[dst * 32] = 0.0f; break;
      case OP_INV: col[dst * 32] = 1.0f / col[a * 32]; break;
      case OP_UPD: col[dst * 32] = fmaf(-(col[a * 32] * col[b * 32]), col[c * 32], col[dst * 32]); break;
      case OP_SCALE: col[dst * 32] = col[dst * 32] * col[a * 32]; break;
      case OP_SUBMUL: col[dst * 32] = fmaf(-col[a * 32], col[b * 32], col[dst * 32]); break;
      case OP_MUL: col[dst * 32] = col[a * 32] * col[b * 32]; break;
      case OP_ADD: col[dst * 32] = col[dst * 32] + col[a * 32]; break;
      case OP_MULSUB: col[dst * 32] = fmaf(col[a * 32], col[b * 32], -col[dst * 32]); break;
      case OP_MULADD: col[dst * 32] = fmaf(col[a * 32], col[b * 32], col[dst * 32]); break;
      case OP_STORE_X:
        if (live) xr[dst] = col[a * 32];
        break;
      default: break;
    }
  }
}

__global__ void tree_ldl_kernel(const int4* __restrict__ prog, const int* __restrict__ ptr, int groups,
                                int owner, const float* __restrict__ M, int64_t M_ld,
                                const float* __restrict__ y, int64_t y_ld, float* __restrict__ x,
                                int64_t x_ld, int nworld) {
  extern __shared__ float slots[];  // [nslot][32]
  const int lw = threadIdx.x & 31, part = threadIdx.x >> 5;
  const int world = blockIdx.x * 32 + lw;
  const bool live = world < nworld;
  const int src = live ? world : nworld - 1;
  const float* Mr = M + (size_t)src * M_ld;
  const float* yr = y + (size_t)src * y_ld;
  float* xr = x + (size_t)src * x_ld;
  float* col = slots + lw;
  // streams: forward_0..forward_{G-1}, trunk, backward_0..backward_{G-1}
  tree_run(prog, ptr[part], ptr[part + 1], col, Mr, yr, xr, live);
  __syncthreads();
  if (part == owner) tree_run(prog, ptr[groups], ptr[groups + 1], col, Mr, yr, xr, live);
  __syncthreads();
  tree_run(prog, ptr[groups + 1 + part], ptr[groups + 2 + part], col, Mr, yr, xr, live);
}

// ---- blocked dense Cholesky ------------------------------------------------------
// One warp per world (or two worlds per warp, see dense_factor_carry), four warps per
// CTA.  Shared memory of a world:
//   A    (n + carry + 1) x ldu.  U[r][c] (r <= c) at A[r*ldu + c]; the value column c
//        starts from (M's column c above the diagonal, or right-hand side c - n) is
//        kept transposed at A[(c+1)*ldu + r], so a lane reads the 16 rows of its
//        column with four 128-bit loads.
//   dinv n, X n x rhs (right-hand sides, then solutions).
// The factorisation works on the nv x nv part only: with zero padding and a unit
// diagonal the padded rows of U are exactly the identity, which is what is stored.
// Up to `carry` right-hand sides ride through the factorisation as extra columns
// (that is the forward substitution); further ones, and mode 1, take the
// substitution with the stored factor.  Every value receives its terms in the same
// order as the plain row-by-row statement of the algorithm (ascending t).
static const int kDenseWarps = 4;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// A warp per world, `l` its lane.  What bounds the kernel is the chain of a world's rows and the warps
// an SM holds to cover it: registers for 28 warps per SM (models up to 64 columns), so that 4096 worlds are
// in flight at once.  4096 humanoid worlds, three right-hand sides, then one with the stored factor:
// 104 us with two worlds per warp, three column groups throughout and 15 shuffles per row; 95 at 24
// warps per SM; 67 at 28 (47 with what the comments below say).  Two worlds per warp halve the warps and take
// three column groups for one or two: slower at every batch size.
//
// Rows b0 .. b0 + 15 at the K column groups that are left.  As in the Newton factor
// (imn_newton_factor.cuh): the pivot of row r + 1 is its own lane's sum after row r and travels at
// once, the row's block entries come back from shared memory as broadcast reads, four rows per trip.
template <int K, int R>
__device__ __forceinline__ void dense_block(float* A, float* dinv, const int b0, const int n, const int nc, const int ldu,
                                            const int l) {
  const int nr = min(16, n - b0);
  float acc[K][R];
  int cc[K];
  bool valid[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int c = b0 + l + 32 * k;
    valid[k] = c < nc;
    cc[k] = valid[k] ? c : nc - 1;
    const float* src = A + (cc[k] + 1) * ldu + b0;
#pragma unroll
    for (int g = 0; g < R; g += 4) {
      const float4 h = g < nr ? ld4(src + g) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      acc[k][g] = h.x, acc[k][g + 1] = h.y, acc[k][g + 2] = h.z, acc[k][g + 3] = h.w;
    }
  }
  // terms of the rows above the block
#pragma unroll 2
  for (int t = 0; t < b0; ++t) {
    const float* Ut = A + t * ldu;
    float uc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) uc[k] = Ut[cc[k]];
#pragma unroll
    for (int g = 0; g < R; g += 4) {
      const float4 u = ld4(Ut + b0 + g);  // past the last row: values that end in sums nobody stores
#pragma unroll
      for (int k = 0; k < K; ++k) {
        acc[k][g] = fmaf(-u.x, uc[k], acc[k][g]), acc[k][g + 1] = fmaf(-u.y, uc[k], acc[k][g + 1]);
        acc[k][g + 2] = fmaf(-u.z, uc[k], acc[k][g + 2]), acc[k][g + 3] = fmaf(-u.w, uc[k], acc[k][g + 3]);
      }
    }
  }
  __syncwarp();  // row b0 of U goes where column b0 - 1 stood
  float pv = __shfl_sync(IMN_FULL_MASK, acc[0][0], 0);
#pragma unroll 1
  for (int g = 0; g < nr; g += 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = g + q;
      if (r >= nr) break;  // uniform: one model
      const float dg = sqrtf(pv), rinv = 1.0f / dg;
      float* Ur = A + (b0 + r) * ldu;
      float u[K];
#pragma unroll
      for (int k = 0; k < K; ++k) u[k] = acc[k][q] * rinv;
      pv = __shfl_sync(IMN_FULL_MASK, fmaf(-u[0], u[0], q + 1 < R ? acc[0][q + 1] : 0.0f), r + 1);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (valid[k] && cc[k] >= b0 + r) Ur[cc[k]] = k == 0 && l == r ? dg : u[k];
      if (l == 0) dinv[b0 + r] = rinv;
      __syncwarp();
#pragma unroll
      for (int h = 0; h < R; h += 4) {
        const float4 m = ld4(Ur + b0 + g + h);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (h > q) acc[k][h] = fmaf(-m.x, u[k], acc[k][h]);
          if (h + 1 > q) acc[k][h + 1] = fmaf(-m.y, u[k], acc[k][h + 1]);
          if (h + 2 > q) acc[k][h + 2] = fmaf(-m.z, u[k], acc[k][h + 2]);
          if (h + 3 > q) acc[k][h + 3] = fmaf(-m.w, u[k], acc[k][h + 3]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int h = 0; h < R; ++h) acc[k][h] = h + 4 < R ? acc[k][h + 4] : 0.0f;
  }
  __syncwarp();
}

template <int KM>
__device__ __forceinline__ void dense_factor_carry(float* A, float* dinv, const int n, const int nc, const int ldu, const int l) {
#pragma unroll 1
  for (int b0 = 0; b0 < n; b0 += 16) {
    // a last block of up to four rows (33 to 36 dofs) keeps no sums of the twelve it does not have
    // (4096 34-dof worlds 49.8 -> 47.4 us).  The same for up to eight rows is not worth its code: 8192 56-dof worlds 228.0 ->
    // 226.7, 512 32.8 -> 33.1, and 4096 34-dof worlds 45.8 -> 47.0.
    if (n - b0 <= 4 && nc - b0 <= 32)
      dense_block<1, 4>(A, dinv, b0, n, nc, ldu, l);
    else if (nc - b0 <= 32)
      dense_block<1, 16>(A, dinv, b0, n, nc, ldu, l);
    else if (KM == 2 || nc - b0 <= 64)
      dense_block<2, 16>(A, dinv, b0, n, nc, ldu, l);
    else
      dense_block<KM, 16>(A, dinv, b0, n, nc, ldu, l);
  }
}

// Forward substitution with the stored factor for right-hand sides [q0, q0 + RQ): a lane keeps rows
// l, l + 32, l + 64 of each in registers, so that a column of U is read once for all of them
// and the only traffic between lanes is the finished unknown.  Unknown r receives its terms in
// ascending order.
template <int KM, int RQ>
__device__ __forceinline__ void dense_forward(const float* A, const float* dinv, float* X, const int n, const int ldu,
                                              const int rhs, const int q0, const int l) {
  float x[RQ][KM];
#pragma unroll
  for (int k = 0; k < KM; ++k)
#pragma unroll
    for (int j = 0; j < RQ; ++j) x[j][k] = l + 32 * k < n && q0 + j < rhs ? X[(l + 32 * k) * rhs + q0 + j] : 0.0f;
#pragma unroll
  for (int kb = 0; kb < KM; ++kb) {
    const int tn = min(32, n - 32 * kb);
#pragma unroll 2
    for (int tl = 0; tl < tn; ++tl) {
      const int t = 32 * kb + tl;
      const float di = dinv[t];
      float a[KM];
#pragma unroll
      for (int k = kb; k < KM; ++k) {
        const int r = l + 32 * k;
        a[k] = r > t && r < n ? A[t * ldu + r] : 0.0f;
      }
#pragma unroll
      for (int j = 0; j < RQ; ++j) {
        const float yt = __shfl_sync(IMN_FULL_MASK, x[j][kb], tl) * di;
#pragma unroll
        for (int k = kb; k < KM; ++k) x[j][k] = fmaf(-a[k], yt, x[j][k]);
        if (l == tl) x[j][kb] = yt;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KM; ++k)
#pragma unroll
    for (int j = 0; j < RQ; ++j)
      if (l + 32 * k < n && q0 + j < rhs) X[(l + 32 * k) * rhs + q0 + j] = x[j][k];
  __syncwarp();
}

// Back substitution of the same right-hand sides in 16-row blocks from the last: later blocks'
// columns first (ascending), then the block's own columns from its last inwards.  The upper half of
// the warp takes the next RQ right-hand sides.
template <int RQ>
__device__ __forceinline__ void dense_back(const float* A, const float* dinv, float* X, const int n, const int ldu, const int rhs,
                                           int q0, const int l) {
  q0 += (l >> 4) * RQ;
  const int l16 = l & 15;
#pragma unroll 1
  for (int b0 = ((n - 1) / 16) * 16; b0 >= 0; b0 -= 16) {
    const int b1 = min(b0 + 16, n), r = min(b0 + l16, n - 1);
    const bool mine = b0 + l16 < b1;
    const float* Ur = A + r * ldu;
    const float di = dinv[r];
    float acc[RQ];
#pragma unroll
    for (int j = 0; j < RQ; ++j) acc[j] = mine && q0 + j < rhs ? X[r * rhs + q0 + j] : 0.0f;
    int c = b1;
#pragma unroll 2
    for (; c + 4 <= n; c += 4) {
      const float4 u = ld4(Ur + c);
      const float uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < RQ; ++j) acc[j] = fmaf(-uu[i], X[(c + i) * rhs + min(q0 + j, rhs - 1)], acc[j]);
    }
#pragma unroll 1
    for (; c < n; ++c)
#pragma unroll
      for (int j = 0; j < RQ; ++j) acc[j] = fmaf(-Ur[c], X[c * rhs + min(q0 + j, rhs - 1)], acc[j]);
#pragma unroll 2
    for (int c = b1 - 1; c >= b0; --c) {
      const float u = Ur[c];
#pragma unroll
      for (int j = 0; j < RQ; ++j) {
        const float xc = __shfl_sync(IMN_FULL_MASK, acc[j] * di, (l & ~15) | (c - b0));
        if (b0 + l16 < c) acc[j] = fmaf(-u, xc, acc[j]);
      }
    }
    // row b0 + l16 is final: its unknown is its sum scaled
#pragma unroll
    for (int j = 0; j < RQ; ++j)
      if (mine && q0 + j < rhs) X[r * rhs + q0 + j] = acc[j] * di;
    __syncwarp();
  }
}

template <int KM, int RQ>
__device__ __forceinline__ void dense_substitute(const float* A, const float* dinv, float* X, const int n, const int ldu,
                                                 const int rhs, const int carried, const int l) {
#pragma unroll 1
  for (int q = carried; q < rhs; q += RQ) dense_forward<KM, RQ>(A, dinv, X, n, ldu, rhs, q, l);
#pragma unroll 1
  for (int q = 0; q < rhs; q += 2 * RQ) dense_back<RQ>(A, dinv, X, n, ldu, rhs, q, l);
}

// an entry of M whose position belongs to a later one (ImnBlockedPlan::places)
constexpr int kNoPlace = 0xFFFF;

template <int KM>
__global__ void __launch_bounds__(32 * kDenseWarps, KM == 2 ? 7 : 4)
    blocked_dense_kernel(const int nv, const int pad, const int nM, const int* __restrict__ indices,
                         const uint16_t* __restrict__ places,
                         const float* __restrict__ identity, const float* __restrict__ M, const int64_t M_ld,
                         const float* __restrict__ y, float* __restrict__ Ug, float* __restrict__ x,
                         const int* __restrict__ active, const int rhs, const int mode, const int carry,
                         const int ldu, const int per_world, const int vec, const int nworld) {
  extern __shared__ __align__(16) float sm[];
  chain_wait();
  const int l = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int w = blockIdx.x * kDenseWarps + warp;
  if (w >= nworld || (active && active[w] == 0)) return;
  const int n = nv, nc = n + carry;
  float* A = sm + warp * per_world;
  float* dinv = A + (nc + 1) * ldu;
  float* X = dinv + ((n + 3) & ~3);
  float* Uw = Ug + (size_t)w * pad * pad;
  const int nblk = pad >> 4;
  // four columns per lane of a row of U, several rows at a time (pad <= 80)
  const int quads = pad >> 2, vrows = 32 / quads;
  const int vr = l / quads < vrows ? l / quads : n, c = 4 * (l % quads);
  const float* yw = y + (size_t)w * n * rhs;
  for (int q = l; q < n * rhs; q += 32) X[q] = yw[q];
  if (mode == 0) {
    // the padded diagonal's roots, a lane each
    const float root = n + l < pad ? sqrtf(__ldg(identity + (((n + l) & 15) << 4 | ((n + l) & 15)))) : 0.0f;
    const float* Mw = M + (size_t)w * M_ld;
    if (places) {
      // M's entries in storage order, coalesced, each to its place; the positions between them are zero.  Looked up
      // position by position (a read of the table, a branch, a read of M for every position of a block) this was 25 k
      // of the 78 k cycles of a 34-dof world.  us, 4096 34-dof worlds, three right-hand sides and a second solve 61 -> 50,
      // 256 worlds 29 -> 24; 8192 56-dof worlds 271 -> 220.
      constexpr int B = 8;
      for (int q = l; 4 * q < (n + 1) * ldu; q += 32) *reinterpret_cast<float4*>(A + 4 * q) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      __syncwarp();
#pragma unroll 1
      for (int e0 = l; e0 < nM; e0 += 32 * B) {
        float v[B];
        int at[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
          const int e = min(e0 + 32 * j, nM - 1);
          v[j] = __ldg(Mw + e), at[j] = __ldg(places + e);
        }
#pragma unroll
        for (int j = 0; j < B; ++j)
          if (e0 + 32 * j < nM && at[j] != kNoPlace) A[((at[j] >> 8) + 1) * ldu + (at[j] & 255)] = v[j];
      }
    } else {
      // gather the blocks on and above the diagonal: table entry
      // ((kb*nblk + ib)*16 + r)*16 + c addresses M's value of (16 kb + r, 16 ib + c);
      // index nM is the extra zero slot
      for (int kb = 0; kb < nblk; ++kb)
        for (int ib = kb; ib < nblk; ++ib) {
          const int* tab = indices + ((kb * nblk + ib) << 8);
#pragma unroll 4
          for (int q = l; q < 256; q += 32) {
            const int row = 16 * kb + (q >> 4), colm = 16 * ib + (q & 15);
            const int idx = __ldg(tab + q);
            if (row <= colm && colm < n) A[(colm + 1) * ldu + row] = idx < nM ? __ldg(Mw + idx) : 0.0f;
          }
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int q = 0; q < carry; ++q)
      for (int r = l; r < n; r += 32) A[(n + q + 1) * ldu + r] = X[r * rhs + q];
    __syncwarp();
    dense_factor_carry<KM>(A, dinv, n, nc, ldu, l);
    // the factor, padded: zeros below the diagonal, the padded diagonal's own root; four columns
    // per store where the workspace allows it
    if (vec) {
#pragma unroll 4
      for (int r = vr; r < n; r += vrows) {
        const float4 a = c < ldu ? ld4(A + r * ldu + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float4 o;
        o.x = c >= r && c < n ? a.x : 0.0f, o.y = c + 1 >= r && c + 1 < n ? a.y : 0.0f;
        o.z = c + 2 >= r && c + 2 < n ? a.z : 0.0f, o.w = c + 3 >= r && c + 3 < n ? a.w : 0.0f;
        *reinterpret_cast<float4*>(Uw + r * pad + c) = o;
      }
    } else {
      for (int r = 0; r < n; ++r) {
        const float* Ar = A + r * ldu;
        float* Ur = Uw + r * pad;
#pragma unroll 3
        for (int c = l; c < pad; c += 32) Ur[c] = (c >= r && c < n) ? Ar[c] : 0.0f;
      }
    }
#pragma unroll 1
    for (int r = n; r < pad; ++r) {
      const float dg = __shfl_sync(IMN_FULL_MASK, root, r - n);
#pragma unroll 3
      for (int cl = l; cl < pad; cl += 32) Uw[r * pad + cl] = cl == r ? dg : 0.0f;
    }
#pragma unroll 1
    for (int q = 0; q < carry; ++q)
      for (int r = l; r < n; r += 32) X[r * rhs + q] = A[r * ldu + n + q];
  } else {
    if (vec) {
      // six reads in flight, then their stores (one after the other: 10 k of the 20 k cycles of a second solve of 34-dof worlds)
      constexpr int B = 6;
#pragma unroll 1
      for (int r0 = vr; r0 < n; r0 += B * vrows) {
        float4 v[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
          const int r = min(r0 + j * vrows, n - 1);
          v[j] = *reinterpret_cast<const float4*>(Uw + r * pad + c);
        }
#pragma unroll
        for (int j = 0; j < B; ++j) {
          const int r = r0 + j * vrows;
          if (r < n && c + 3 >= r && c < n) *reinterpret_cast<float4*>(A + r * ldu + c) = v[j];
        }
      }
    } else {
      for (int r = 0; r < n; ++r)
        for (int c = r + l; c < n; c += 32) A[r * ldu + c] = Uw[r * pad + c];
    }
    __syncwarp();
    for (int r = l; r < n; r += 32) dinv[r] = 1.0f / A[r * ldu + r];
  }
  __syncwarp();
  // right-hand sides one, two or four at a time
  const int carried = mode == 0 ? carry : 0;
  if (rhs == 1)
    dense_substitute<KM, 1>(A, dinv, X, n, ldu, rhs, carried, l);
  else if (rhs == 2)
    dense_substitute<KM, 2>(A, dinv, X, n, ldu, rhs, carried, l);
  else
    dense_substitute<KM, 4>(A, dinv, X, n, ldu, rhs, carried, l);
  float* xw = x + (size_t)w * n * rhs;
  for (int q = l; q < n * rhs; q += 32) xw[q] = X[q];
}

}  // namespace imn

extern "C" int imn_tree_ldl_solve(const ImnTreePlan* plan, const float* M, int64_t M_ld, const float* y,
                                  int64_t y_ld, float* x, int64_t x_ld, int32_t nworld, void* stream) {
  if (!plan || !M || !y || !x || !plan->prog || !plan->prog_ptr)
    return imn::set_error("imn_tree_ldl_solve: NULL argument"), IMN_ERR_NULL;
  if (plan->nv <= 0 || plan->groups < 1 || plan->groups > 4 || plan->owner < 0 || plan->owner >= plan->groups ||
      plan->nslot <= 0)
    return imn::set_error("imn_tree_ldl_solve: malformed plan"), IMN_ERR_SHAPE;
  if (nworld < 0 || M_ld < plan->nM || y_ld < plan->nv || x_ld < plan->nv)
    return imn::set_error("imn_tree_ldl_solve: a stride is smaller than its extent"), IMN_ERR_SHAPE;
  if (nworld == 0) return IMN_OK;
  const size_t bytes = (size_t)plan->nslot * 32 * sizeof(float);
  if (bytes > 227 * 1024)
    return imn::set_error("imn_tree_ldl_solve: plan needs %zu bytes of shared memory per block (max %d)", bytes,
                          227 * 1024),
           IMN_ERR_LIMIT;
  {
    const cudaError_t e = imn::allow_shared(imn::tree_ldl_kernel, bytes);
    if (e != cudaSuccess)
      return imn::set_error("imn_tree_ldl_solve: cudaFuncSetAttribute: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  }
  imn::tree_ldl_kernel<<<(nworld + 31) / 32, 32 * plan->groups, bytes, (cudaStream_t)stream>>>(
      reinterpret_cast<const int4*>(plan->prog), plan->prog_ptr, plan->groups, plan->owner, M, M_ld, y, y_ld, x,
      x_ld, nworld);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return imn::set_error("imn_tree_ldl_solve: launch failed: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  return IMN_OK;
}

extern "C" int imn_blocked_dense_factor_solve(const ImnBlockedPlan* plan, const float* M, int64_t M_ld,
                                              const float* y, float* U, float* x, const int32_t* active,
                                              int32_t nworld, int32_t rhs_count, int32_t mode, void* stream) {
  if (!plan || !y || !U || !x || (mode == 0 && (!M || !plan->indices || !plan->identity)))
    return imn::set_error("imn_blocked_dense_factor_solve: NULL argument"), IMN_ERR_NULL;
  if (plan->nv <= 0 || plan->pad % 16 != 0 || plan->pad < plan->nv || plan->pad >= plan->nv + 16)
    return imn::set_error("imn_blocked_dense_factor_solve: pad %d is not nv %d rounded up to 16", plan->pad,
                          plan->nv),
           IMN_ERR_SHAPE;
  if (mode != 0 && mode != 1) return imn::set_error("imn_blocked_dense_factor_solve: mode must be 0 or 1"), IMN_ERR_SHAPE;
  if (nworld < 0 || rhs_count < 1 || (mode == 0 && M_ld < plan->nM))
    return imn::set_error("imn_blocked_dense_factor_solve: bad extent or stride"), IMN_ERR_SHAPE;
  if (nworld == 0) return IMN_OK;
  const int n = plan->nv;
  if (n > 80) return imn::set_error("imn_blocked_dense_factor_solve: nv %d above 80", n), IMN_ERR_UNSUPPORTED;
  // right-hand sides that ride through the factorisation as extra columns
  const int carry = mode == 0 ? (rhs_count < 96 - n ? rhs_count : 96 - n) : 0;
  // rows of an odd number of quads: 128-bit reads of one quad from consecutive rows meet no bank twice
  // (the largest models with many right-hand sides only fit without)
  auto floats = [&](int ld) { return (n + carry + 1) * ld + ((n + 3) & ~3) + ((n * rhs_count + 3) & ~3); };
  int ldu = 4 * (((n + carry + 3) >> 2) | 1);
  if (sizeof(float) * (size_t)floats(ldu) * imn::kDenseWarps > 227 * 1024) ldu = (n + carry + 3) & ~3;
  const int per_world = floats(ldu);
  const int per_cta = imn::kDenseWarps;
  const size_t bytes = sizeof(float) * (size_t)per_world * per_cta;
  auto kernel = n + carry <= 64 ? imn::blocked_dense_kernel<2> : imn::blocked_dense_kernel<3>;
  if (bytes > 227 * 1024)
    return imn::set_error("imn_blocked_dense_factor_solve: %zu bytes of shared memory needed (max %d)", bytes,
                          227 * 1024),
           IMN_ERR_LIMIT;
  {
    const cudaError_t e = imn::allow_shared(kernel, bytes, true);
    if (e != cudaSuccess)
      return imn::set_error("imn_blocked_dense_factor_solve: cudaFuncSetAttribute: %s", cudaGetErrorString(e)),
             IMN_ERR_LAUNCH;
  }
  const int vec = (reinterpret_cast<uintptr_t>(U) & 15) == 0;  // pad is a multiple of 16 floats
  const cudaError_t e = imn::launch_chained(kernel, (nworld + per_cta - 1) / per_cta, 32 * imn::kDenseWarps, bytes,
                                            (cudaStream_t)stream, plan->nv, plan->pad, plan->nM, plan->indices, plan->places, plan->identity,
                                            M, M_ld, y, U, x, active, rhs_count, mode, carry, ldu, per_world, vec, nworld);
  if (e != cudaSuccess)
    return imn::set_error("imn_blocked_dense_factor_solve: launch failed: %s", cudaGetErrorString(e)),
           IMN_ERR_LAUNCH;
  return IMN_OK;
}

// ---- factor + solve without any caller- or library-side allocation ---------------
//
// Some hosts of this library may not allocate device memory at the point where they
// need a factor + solve: a simulation step that is being recorded into a CUDA graph,
// a control loop that has handed all device memory to another framework's pool at
// start-up, or a plug-in whose host forbids cudaMalloc after initialisation (the call
// synchronises the device).  imn_blocked_dense_factor_solve needs a (W, pad, pad)
// workspace for the factor; this variant keeps that workspace inside the library, in
// a fixed-size array in device memory that every GPU loading the library holds until
// the process exits.
namespace imn {

static __device__ __align__(256) float g_static_factor[IMN_STATIC_FACTOR_FLOATS];

// Device address of g_static_factor per CUDA device.  In host code the array's name is
// only a handle; the address a kernel can use comes from cudaGetSymbolAddress, asked
// once per device with that device current.  The slots are atomics: two host threads
// that make the first call on a device at the same time both look the address up and
// store the same value.  A cached address belongs to the device's primary context; it
// does not survive cudaDeviceReset (after a reset, reload the library).
static std::atomic<float*> g_static_factor_ptr[64];

static int static_factor_workspace(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return set_error("static workspace: cudaGetDevice: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  if (dev < 0 || dev >= 64) return set_error("static workspace: device index %d out of range", dev), IMN_ERR_LIMIT;
  float* ptr = g_static_factor_ptr[dev].load(std::memory_order_acquire);
  if (!ptr) {
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_factor);
    if (e != cudaSuccess || !ptr)
      return set_error("static workspace: cudaGetSymbolAddress: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
    g_static_factor_ptr[dev].store(ptr, std::memory_order_release);
  }
  *out = ptr;
  return IMN_OK;
}

}  // namespace imn

extern "C" int imn_blocked_dense_factor_solve_static(const ImnBlockedPlan* plan, const float* M, int64_t M_ld,
                                                     const float* y, float* x, const int32_t* active,
                                                     int32_t nworld, int32_t rhs_count, void* stream) {
  if (!plan) return imn::set_error("imn_blocked_dense_factor_solve_static: NULL plan"), IMN_ERR_NULL;
  if (nworld < 0 || plan->pad <= 0)
    return imn::set_error("imn_blocked_dense_factor_solve_static: bad extent"), IMN_ERR_SHAPE;
  const int64_t need = (int64_t)nworld * plan->pad * plan->pad;
  if (need > (int64_t)IMN_STATIC_FACTOR_FLOATS)
    return imn::set_error("imn_blocked_dense_factor_solve_static: %d worlds x pad %d^2 = %lld floats exceed the "
                          "built-in workspace of %lld floats; use imn_blocked_dense_factor_solve with your own",
                          nworld, plan->pad, (long long)need, (long long)IMN_STATIC_FACTOR_FLOATS),
           IMN_ERR_LIMIT;
  float* U = nullptr;
  const int rc = imn::static_factor_workspace(&U);
  if (rc) return rc;
  // The factor kernel writes every entry of an active world's U before the solve
  // reads it, so nothing in the shared workspace has to start at zero.
  return imn_blocked_dense_factor_solve(plan, M, M_ld, y, U, x, active, nworld, rhs_count, 0, stream);
}
