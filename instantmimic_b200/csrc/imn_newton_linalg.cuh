// imn_newton_linalg.cuh -- per-world linear algebra of the fused Newton kernel,
// executed by one warp on shared-memory operands.  Every function is called from
// exactly one place in the kernel so that the machine code stays small (the
// kernel is bound by instruction fetch and latency, not by arithmetic).
#pragma once

#include <stdio.h>

#include "imn_newton_dev.cuh"
#include "imn_sparse.cuh"

namespace imn {

// Shared-memory view of one world plus the per-world constants.
struct World {
  int nv, ldj, ldp, ldu, bd, nefc, ne, nef, lane, nM;
  // a team of `parts` warps may share the world (the TEAM kernels), each with a row tile, a copy barrier
  // and its words of its own; `box` carries single values from part 0 to the others
  int part, parts, team_bar, tile_words, mulm_part;  // mulm_part: the warp that forms M v
  int* box;
  float* tile;
  float *Jsm, *A, *qacc, *Ma, *search, *mv, *grad, *qfs, *xsm, *dinv;
  // the world's M stays in global memory: its nM values are read once per iteration by
  // `products` (independent loads, issued together) and once by the Hessian assembly, and
  // the shared memory they would take holds more worlds per SM instead (when a CTA held one world:
  // humanoid 0.792 -> 0.785 ms per 8192 worlds, SNU-like 1.820 -> 1.736 ms per 4096)
  const float* M;
  float *Jaref, *jv, *Dsm, *force;
  const float* floss;  // global memory: only friction-loss rows read it
  // row states and the two row lists are 16-bit (njmax < 32768: bit 15 is a flag in ids): shared memory per
  // world decides how many worlds an SM holds
  uint16_t *state, *ids, *frows;
  int* uni;
  uint32_t* masks;  // the dofs each row touches (store_mask)
  int mwords, r4;
  const float* Jg;    // this world's J in global memory
  const float *Jbeg, *Jend;  // first element and one past the last row of the whole J array
  // streamed J: the copy barrier of the row tile, the parity of its next phase and the
  // flag a timed-out copy raises (all in shared memory); wait limit in polls and the
  // failure-path test switch that withholds the copies
  void* jbar;
  int* jphase;
  int* jfail;
  int wait_polls, withhold_copies;
  Tables tab;
  int mulm_batches;
  const int *M_rowadr, *M_rownnz, *M_colind;
  // sparse plan only: packed H, N = L D with the carried row, 1/D, the world's
  // violation counter in global memory, the world index (for messages)
  float *Hp, *N, *iD, *viol;
  int world;
#ifdef IMN_PROFILE
  long long* prof_acc;
  long long* prof_t;
#endif
};

// The warps of a world's team wait for one another, on the team's own barrier; a team of one warp has
// its lanes to order.
template <bool TEAM>
__device__ __forceinline__ void team_sync(const World& s) {
  if (TEAM)
    asm volatile("bar.sync %0, %1;" ::"r"(s.team_bar), "r"(32 * s.parts) : "memory");
  else
    __syncwarp();
}
template <bool TEAM>
__device__ __forceinline__ int team_part(const World& s) { return TEAM ? s.part : 0; }
template <bool TEAM>
__device__ __forceinline__ int team_parts(const World& s) { return TEAM ? s.parts : 1; }

#ifdef IMN_PROFILE
#define IMN_MARK(s, k) do { const long long t_ = clock64(); (s).prof_acc[k] += t_ - *(s).prof_t; *(s).prof_t = t_; } while (0)
#else
#define IMN_MARK(s, k)
#endif

// J16: the elements of up to 32 rows in pieces of 16 bytes, consecutive lanes on consecutive pieces,
// nv / 4 pieces per row; f(row, piece) copies one.
template <typename F>
__device__ __forceinline__ void each_piece(const World& s, int rows, F f) {
  const int n = s.nv >> 2, dr = 32 / n, dc = 32 - dr * n;
  int row = s.lane / n, c = s.lane - row * n;
#pragma unroll 4
  while (row < rows) {
    f(row, c);
    row += dr, c += dc;
    if (c >= n) c -= n, ++row;
  }
}

// Rows [base, base+32) of J: resident rows are addressed in place, otherwise they are staged
// through the 32-row tile; the wait for the copies is bounded.
// J16 (streamed only; nv, the row stride and every row multiples of four floats): 16-byte copies to a
// row stride of ldp floats, a multiple of four with ldp / 4 odd.  With lane = row the 128-bit reads of
// eight consecutive lanes then hit eight different groups of four banks; at their own stride the rows
// of such models (56, 64 floats) put 4 or all 32 lanes on one bank.  (64 dofs x 512 rows, 4096
// worlds: 7326 -> 4816 us per solve with a bulk copy per row; 4621 with the pieces.)
// Otherwise rows keep their own stride and the tile is one contiguous TMA bulk copy.
template <bool JRES, bool J16>
__device__ __forceinline__ const float* j_tile(const World& s, int base) {
  if (JRES) return s.Jsm + base * s.ldj;
  IMN_MARK(s, 23);
  __syncwarp();  // every lane is done with the previous tile
  const int rows = min(32, s.nefc - base), n = rows * s.ldj;
  const float* src = s.Jg + (size_t)base * s.ldj;
  // A bulk copy wants 16-byte aligned ends, so the smallest aligned range around a run of rows is
  // copied (up to three floats of the neighbouring rows on either side, still inside the J
  // array) and the tile starts `head` floats into the buffer.
  const int head = J16 ? 0 : (int)((reinterpret_cast<uintptr_t>(src) & 15) >> 2);
  const uint32_t bytes = (uint32_t)((head + n + 3) & ~3) * 4u;
  // after a copy that timed out the barrier's phase is unknown: the world is lost (the
  // caller checks jfail at the end of the pass) and the rest of the pass uses plain loads
  if ((J16 || (src - head >= s.Jbeg && src - head + (bytes >> 2) <= s.Jend)) && !*s.jfail) {
    const uint32_t parity = (uint32_t)*s.jphase;
    __syncwarp();
    if (J16) {
      if (s.lane == 0) *s.jphase = (int)(parity ^ 1u);
      if (!(s.withhold_copies & 2)) {
        each_piece(s, rows, [&](int row, int c) { copy16(s.tile + row * s.ldp + 4 * c, src + (size_t)row * s.ldj + 4 * c); });
        mbar_arrive_copies(s.jbar);
      }
    } else if (s.lane == 0) {
      mbar_expect_tx(s.jbar, bytes);
      if (!(s.withhold_copies & 2)) bulk_g2s(s.tile, src - head, bytes, s.jbar);
      *s.jphase = (int)(parity ^ 1u);
    }
    bool arrived = false;
#pragma unroll 1
    for (int tries = 0; tries < s.wait_polls && !arrived; ++tries) arrived = mbar_try_wait(s.jbar, parity);
    if (!arrived && s.lane == 0) *s.jfail = 1;
    __syncwarp();
    IMN_MARK(s, 17);
    return s.tile + head;
  }
  if (J16) return s.tile;  // a lost world: its results are never written
#pragma unroll 4
  for (int i = s.lane; i < n; i += 32) s.tile[i] = src[i];
  // the next tile may arrive through the async proxy into the same buffer
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  return s.tile;
}

// Rows of the list s.ids (bit 15: the row leaves the QUADRATIC set, its D counts negative) as the
// Hessian stages read them.  A resident J is read in place.  Streamed rows are gathered into the
// tile, up to 32 listed rows at a time and up4(nv) floats apart: the stages read a row many times
// over, and taking its elements from global memory each time was a half of the whole solve at
// 64 dofs x 512 rows.
// place of the at-th gathered row (a team has a tile of 32 per warp)
template <bool TEAM>
__device__ __forceinline__ float* gathered(const World& s, int at, int ld) {
  return TEAM ? s.Jsm + (at >> 5) * s.tile_words + (at & 31) * ld : s.Jsm + at * ld;
}
struct ListRow {
  const float* J;
  float D;
};
template <bool JRES, bool TEAM>
__device__ __forceinline__ ListRow list_row(const World& s, int t, int t0) {
  const int id = s.ids[t], r = id & 0x7FFF;
  ListRow o;
  const int at = t - t0, ld = (s.nv + 3) & ~3;
  o.J = JRES ? s.Jsm + r * s.ldj : gathered<TEAM>(s, at, ld);
  o.D = __int_as_float(__float_as_int(s.Dsm[r]) ^ ((id & 0x8000) << 16));
  return o;
}
template <bool JRES, bool J16, bool TEAM>
__device__ __forceinline__ void gather_rows(const World& s, int t0, int t1) {
  if (JRES) return;
  team_sync<TEAM>(s);  // every lane is done with the tile's previous contents
  int at = 0;  // a team's warps gather a share of the rows each
  if (TEAM) {
    const int share = (t1 - t0 + s.parts - 1) / s.parts;
    at = share * s.part, t1 = min(t1, t0 + at + share), t0 += at;
  }
  const int ld = (s.nv + 3) & ~3, lane = s.lane;
  if (J16) {
    each_piece(s, t1 - t0, [&](int row, int c) {
      copy16(gathered<TEAM>(s, at + row, ld) + 4 * c, s.Jg + (size_t)(s.ids[t0 + row] & 0x7FFF) * s.ldj + 4 * c);
    });
    asm volatile("cp.async.wait_all;" ::: "memory");
    team_sync<TEAM>(s);
    return;
  }
  const int ids = t0 + lane < t1 ? s.ids[t0 + lane] & 0x7FFF : 0;
#pragma unroll 4
  for (int t = t0; t < t1; ++t) {
    const uint32_t dst = smem_u32(gathered<TEAM>(s, at + t - t0, ld) + lane);
    const float* src = s.Jg + (size_t)__shfl_sync(IMN_FULL_MASK, ids, t - t0) * s.ldj + lane;
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (32 * q + lane < s.nv)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 128u * q), "l"(src + 32 * q) : "memory");
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // a later tile may arrive through the async proxy into the same buffer
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  team_sync<TEAM>(s);
}

// The dofs each row touches, as s.mwords 32-bit words per row in shared memory (word q of row r at
// s.masks[q * r4 + r]), formed once per world while the first pass has the row in hand (lane = row).
// The Hessian stages need them at every change of the active set: for the dofs the flipped rows
// touch, and to know that no row leaves the sparse plan's pattern.
__device__ __forceinline__ void store_mask(const World& s, const float* Jr, int r) {
#pragma unroll 1
  for (int q = 0; q < s.mwords; ++q) {
    unsigned m = 0u;
    const int n = min(32, s.nv - 32 * q);
#pragma unroll 4
    for (int i = 0; i < n; ++i) m |= (unsigned)(Jr[32 * q + i] != 0.0f) << i;
    s.masks[q * s.r4 + r] = m;
  }
}
// Whether row r's dofs are not all coupled in the plan's pattern: every dof's couplings must hold the whole row.
// (One branch per dof and word of the masks, each read from global memory, was a twentieth of a 34-dof solve: without
// the branches and from the staged tables 16 worlds 112.1 -> 108.0 us, 8192 worlds 535 -> 521; 56 dofs x 128 rows, 16 worlds
// 245 -> 233, 4096 worlds 1094 -> 1079; 35 dofs x 250 rows, 16384 worlds 2281 -> 2243.)
template <bool TSM>
__device__ __forceinline__ bool row_outside(const uint32_t* masks, int r4, int mwords, int r, const uint32_t* pmask) {
  uint32_t all[3] = {~0u, ~0u, ~0u};  // dofs that every dof of the row is coupled with (at most 80)
#pragma unroll 1
  for (int q = 0; q < mwords; ++q)
#pragma unroll 1
    for (unsigned left = masks[q * r4 + r]; left; left &= left - 1u) {
      const uint32_t* with = pmask + (32 * q + __ffs(left) - 1) * mwords;
#pragma unroll
      for (int p = 0; p < 3; ++p)
        if (p < mwords) all[p] &= tab_at<TSM>(with + p);
    }
  uint32_t out = 0u;
#pragma unroll
  for (int p = 0; p < 3; ++p)
    if (p < mwords) out |= masks[p * r4 + r] & ~all[p];
  return out != 0u;
}
// The dofs of the flipped rows, ascending, and their count (ctx.newton_dof_union).
__device__ __forceinline__ void write_union(const World& s, int count) {
  int n = 0;
#pragma unroll 1
  for (int q = 0; q < s.mwords; ++q) {
    unsigned m = 0u;
#pragma unroll 1
    for (int t = s.lane; t < count; t += 32) m |= s.masks[q * s.r4 + (s.ids[t] & 0x7FFF)];
    m = __reduce_or_sync(IMN_FULL_MASK, m);
    if ((m >> s.lane) & 1u) s.uni[n + __popc(m & ((1u << s.lane) - 1u))] = 32 * q + s.lane;
    n += __popc(m);
  }
  if (s.lane == 0) s.uni[s.nv] = n;
}

// outM = M v over the symmetric rows (newton_fusion.py:171-176) and
// outJ[r] = J[r,:] v (- minus[r]): one running sum per row; above 50 dofs in
// 20-dof partials joined by plain adds (newton_stages.py:157-174).
template <bool JRES, bool J16, bool TSM, bool TEAM>
__device__ __forceinline__ void products(const World& s, const float* v, float* outM, float* outJ,
                                         const float* minus) {
  const int lane = s.lane, nv = s.nv;
  // a team deals the tiles of 32 rows to its warps, M v to the warp that is next
  const int part = team_part<TEAM>(s), stride = 32 * team_parts<TEAM>(s);
  // M v by the lane program: a lane owns whole rows and forms each row's sum in table order,
  // four entries per batch.  The program is read coalesced and a batch ahead, so that the reads
  // of M (global, L1) and v of a batch are issued together.  With a lane per dof and the row table
  // itself, the table reads touched up to 18 cache lines per instruction, stood in front of the
  // reads of M, and dofs past 32 took a second round (34-dof model, 8192 worlds: 7000 -> 5900 cycles
  // of the world's warp per product; 56-dof model, 4096 worlds: 1745 -> 1669 us per solve).
  if (!TEAM || s.mulm_part == part) {
    const uint4* prog = s.tab.mulm + lane;
    uint4 p = tab_at<TSM>(prog);
    float acc = 0.0f;
    const auto M = [&](uint32_t w) { return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(s.M) + (w >> 16))); };
    const auto V = [&](uint32_t w) { return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(v) + (w & 0x1FCu)); };
#pragma unroll 1
    for (int b = s.mulm_batches; b > 0; --b) {
      prog += 32;
      const uint4 nxt = tab_at<TSM>(prog);
      const float m0 = M(p.x), m1 = M(p.y), m2 = M(p.z), m3 = M(p.w);
      acc = fmaf(m3, V(p.w), fmaf(m2, V(p.z), fmaf(m1, V(p.y), fmaf(m0, V(p.x), acc))));
      outM[(p.y >> 9) & 0x7F] = acc;  // stored with every batch of the row: no branch, and the last one stays
      if (p.x & 0x200u) acc = 0.0f;
      p = nxt;
    }
  }
  IMN_MARK(s, 16);
  const int chunk = nv > 50 ? 20 : nv;
#pragma unroll 1
  for (int base = 32 * part; base < s.nefc; base += stride) {
    const float* Jt = j_tile<JRES, J16>(s, base);
    const int r = base + lane;
    if (r < s.nefc) {
      const float* Jr = Jt + lane * (J16 ? s.ldp : s.ldj);
      const float sub = minus ? minus[r] : 0.0f;
      float total = 0.0f;
#pragma unroll 1
      for (int s0 = 0; s0 < nv; s0 += chunk) {
        float p = 0.0f;
        const int e = min(s0 + chunk, nv);
        if (J16) {
#pragma unroll 5
          for (int i = s0; i < e; i += 4) {
            const float4 a = *reinterpret_cast<const float4*>(Jr + i), x = *reinterpret_cast<const float4*>(v + i);
            p = fmaf(a.w, x.w, fmaf(a.z, x.z, fmaf(a.y, x.y, fmaf(a.x, x.x, p))));
          }
        } else {
#pragma unroll 4
          for (int i = s0; i < e; ++i) p = fmaf(Jr[i], v[i], p);
        }
        if (s0 == 0)
          total = minus ? p - sub : (nv > 50 ? 0.0f + p : p);
        else
          total = total + p;
      }
      outJ[r] = total;
      if (minus) store_mask(s, Jr, r);  // the first pass
    }
    if (!JRES) __syncwarp();
  }
}

// grad = Ma - qfrc_smooth - J^T force over the rows with a nonzero force (a zero
// force leaves the running sums unchanged; newton_stages.py:785-795).  Lane = dof.  Every element of J is used once, so a streamed J is read
// straight from global memory (coalesced), without the detour through the tile; the listed rows go
// several at a time so that their reads overlap.
template <bool JRES, bool TEAM>
__device__ __forceinline__ void full_gradient(const World& s, int nfr) {
  const int lane = s.lane, nv = s.nv;
  float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f;
  const int i0 = lane, i1 = lane + 32, i2 = lane + 64;
  const int part = team_part<TEAM>(s), parts = team_parts<TEAM>(s);  // 32 dofs per warp of a team, in turn
  const bool h0 = i0 < nv && (!TEAM || part == 0), h1 = i1 < nv && (!TEAM || part == 1),
             h2 = i2 < nv && (!TEAM || part == (parts > 2 ? 2 : 0));
  if (TEAM && 32 * part >= nv) nfr = 0;
  // rows in flight: reads of a streamed J come from L2, which a team alone on its warps has to cover itself; where the
  // other worlds do, the shorter code counts (eight -> four: 56 dofs, 4096 worlds 1057 -> 1048 us, 35 dofs x 250 rows,
  // 16384 worlds 2152 -> 2112; in teams 64 dofs x 512 rows 3711 -> 3933, 16 worlds of 56 dofs 226 -> 236)
  constexpr int B = !JRES && TEAM ? 8 : 4;
  const float* J = (JRES ? s.Jsm : s.Jg) + lane;
#pragma unroll 1
  for (int a = 0; a < nfr; a += B) {
    float f[B], j0[B], j1[B], j2[B];
#pragma unroll
    for (int k = 0; k < B; ++k) {
      const int r = s.frows[min(a + k, nfr - 1)];
      f[k] = a + k < nfr ? s.force[r] : 0.0f;  // past the end the last row again, without a force
      const float* Jr = J + (size_t)r * s.ldj;
      j0[k] = h0 ? Jr[0] : 0.0f, j1[k] = h1 ? Jr[32] : 0.0f, j2[k] = h2 ? Jr[64] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < B; ++k) s0 = fmaf(j0[k], f[k], s0), s1 = fmaf(j1[k], f[k], s1), s2 = fmaf(j2[k], f[k], s2);
  }
  if (h0) s.grad[i0] = (s.Ma[i0] - s.qfs[i0]) - s0;
  if (h1) s.grad[i1] = (s.Ma[i1] - s.qfs[i1]) - s1;
  if (h2) s.grad[i2] = (s.Ma[i2] - s.qfs[i2]) - s2;
  team_sync<TEAM>(s);
}

// The Hessian from the listed rows, dense form.  First call: H = M + sum D J^T J over the
// QUADRATIC rows, every entry starting from M and summing its rows in ascending order.  Later:
// every entry's change is summed over the flipped rows in list order (newton_stages.py:651-701)
// and added to H.  H[r][c] (r <= c) lives at A[(c+1)*ldu + r]; the sums of a list that does not fit
// one tile wait in the factor's half of the array (U[r][c] at A[r*ldu + c]), which is dead until
// the factorisation that follows.
// A lane owns 4 x 4 blocks of the upper triangle: eight values of a row feed 16 fused
// multiply-adds, so the stage is bound by arithmetic instead of by shared-memory reads (an entry
// per lane reads two values and looks its row up for every multiply-add).
template <bool JRES, bool J16, bool TEAM>
__device__ __forceinline__ void hessian_dense(const World& s, int count, bool first) {
  const int at = 32 * team_part<TEAM>(s), stride = 32 * team_parts<TEAM>(s);  // a team's warps take turns
  const int lane = s.lane, nv = s.nv, ldu = s.ldu;
  float* A = s.A;
  if (first) {
#pragma unroll 4
    for (int e = at + lane; e < (nv + 1) * ldu; e += stride) A[e] = 0.0f;
    team_sync<TEAM>(s);
#pragma unroll 1
    for (int i = at + lane; i < nv; i += stride) {
      const int e0 = __ldg(s.M_rowadr + i), n = __ldg(s.M_rownnz + i);
#pragma unroll 4
      for (int k = 0; k < n; ++k) A[(i + 1) * ldu + __ldg(s.M_colind + e0 + k)] = __ldg(s.M + e0 + k);
    }
  }
  const int nb = (nv + 3) >> 2, nblock = nb * (nb + 1) / 2;
  const int step = JRES ? max(count, 1) : stride;
#pragma unroll 1
  for (int t0 = 0; t0 < count; t0 += step) {
    const int t1 = min(t0 + step, count);
    gather_rows<JRES, J16, TEAM>(s, t0, t1);
    if (JRES || !TEAM) team_sync<TEAM>(s);
    IMN_MARK(s, 22);
    const bool keep = t0 > 0 || first, last = t1 == count;
#pragma unroll 1
    for (int b0 = at; b0 < nblock; b0 += stride) {
      const bool live = b0 + lane < nblock;
      int bi, bj;
      pair_lookup(min(b0 + lane, nblock - 1), bi, bj);
      const int i0 = 4 * bi, j0 = 4 * bj;
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool in = i0 + i <= j0 + j && j0 + j < nv;
          acc[i][j] = !(keep && in) ? 0.0f : t0 > 0 ? A[(i0 + i) * ldu + j0 + j] : A[(j0 + j + 1) * ldu + i0 + i];
        }
#pragma unroll 2
      for (int t = t0; t < t1; ++t) {
        const ListRow row = list_row<JRES, TEAM>(s, t, t0);
        float a[4], b[4];
        if (JRES) {  // rows lie at their own stride, on any boundary
#pragma unroll
          for (int k = 0; k < 4; ++k) a[k] = row.J[i0 + k], b[k] = row.J[j0 + k];
        } else {
          const float4 fa = *reinterpret_cast<const float4*>(row.J + i0), fb = *reinterpret_cast<const float4*>(row.J + j0);
          a[0] = fa.x, a[1] = fa.y, a[2] = fa.z, a[3] = fa.w, b[0] = fb.x, b[1] = fb.y, b[2] = fb.z, b[3] = fb.w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float ad = a[i] * row.D;
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ad, b[j], acc[i][j]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (live && i0 + i <= j0 + j && j0 + j < nv) {
            float* h = A + (j0 + j + 1) * ldu + i0 + i;
            if (!last)
              A[(i0 + i) * ldu + j0 + j] = acc[i][j];
            else
              *h = first ? acc[i][j] : *h + acc[i][j];
          }
    }
  }
  if (!first && at == 0) write_union(s, count);
  team_sync<TEAM>(s);
  IMN_MARK(s, 18);
}

// Pattern violations, for a world that has a row outside the pattern: at the first call one per
// QUADRATIC row with D != 0, later one per pair of touched dofs without a slot whose H entry the
// flipped rows change (sparse_hessian.py:501-527, 619-620).
__device__ __noinline__ void count_violations(bool first, const float* Jw, int ld, int nv, const float* Dsm, const uint32_t* masks,
                                              int r4, int mwords, const uint16_t* ids, int count, const uint32_t* pmask,
                                              const int* pair, float* viol, int world, int lane) {
  if (first) {
    for (int t = lane; t < count; t += 32)
      if (Dsm[ids[t]] != 0.0f && row_outside<false>(masks, r4, mwords, ids[t], pmask)) sp_violation(viol, world, "has a constraint row");
    return;
  }
  for (int e = lane; e < nv * (nv + 1) / 2; e += 32) {
    int i, j;
    pair_lookup(e, i, j);
    if (__ldg(pair + i * nv + j) >= 0) continue;
    float delta = 0.0f;
    for (int t = 0; t < count; ++t) {
      const int id = ids[t], r = id & 0x7FFF;
      const float* J = Jw + (size_t)r * ld;
      const float D = (id & 0x8000) ? -Dsm[r] : Dsm[r];
      if (J[i] != 0.0f && J[j] != 0.0f) delta = fmaf(D * J[i], J[j], delta);
    }
    if (delta != 0.0f) sp_violation(viol, world, "updates an H entry");
  }
}

// The same on the pattern slots of a sparse plan (sparse_hessian.py:501-527, 571-637): first call
// M + sum D J^T J, later H plus the flipped rows' change; the result goes to the packed H and to N,
// where the factorisation starts.  Every slot is summed, whether the rows touch it or not: slot
// tables are read coalesced once per call, a slot costs four instructions per row, and no pair list
// of touched dofs has to be formed and looked up.  `outside`: the world has a row whose dofs do not
// all lie in the pattern.  Sums of a list that does not fit one tile wait in N.
template <bool JRES, bool J16, bool TSM, bool TEAM>
__device__ __forceinline__ void hessian_sparse(const World& s, int count, bool first, bool outside, const ImnSparsePlan& SP) {
  const int lane = s.lane, nv = s.nv, nfac = SP.nfac;
  // slots a lane sums at a time: few in a team, whose warps take turns at the slots, and beside a streamed J, where the
  // shorter code counts for more than the second look at a row (twelve -> six: 56 dofs, 4096 worlds 1067 -> 1057 us, 35
  // dofs x 250 rows, 16384 worlds 2183 -> 2152; ten -> five with J resident: 34 dofs, 8192 worlds 511 -> 517)
  constexpr int Q = TEAM ? 5 : JRES ? 10 : 6;
  const int part = team_part<TEAM>(s), parts = team_parts<TEAM>(s);
  const int step = JRES ? max(count, 1) : 32 * parts;
  // a list without rows still has to place M (first call)
  int t0 = 0;
  do {
    const int t1 = min(t0 + step, count);
    gather_rows<JRES, J16, TEAM>(s, t0, t1);
    IMN_MARK(s, 22);
    const bool last = t1 == count;
#pragma unroll 1
    for (int base = 32 * Q * part; base < nfac; base += 32 * Q * parts) {
      float acc[Q];
      int a[Q], b[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int sl = min(base + 32 * q + lane, nfac - 1);
        int e;
        if (TSM) {
          const uint32_t w = s.tab.slots[sl];
          a[q] = w & 0x1FC, b[q] = (w >> 9) & 0x1FC, e = (int)(w >> 18) - 1;
        } else {
          a[q] = 4 * __ldg(SP.s_a + sl), b[q] = 4 * __ldg(SP.s_b + sl), e = first ? __ldg(SP.s_m + sl) : -1;
        }
        acc[q] = t0 > 0 ? s.N[sl] : first && e >= 0 ? __ldg(s.M + e) : 0.0f;
      }
#pragma unroll 1
      for (int t = t0; t < t1; ++t) {
        const ListRow row = list_row<JRES, TEAM>(s, t, t0);
#pragma unroll
        for (int q = 0; q < Q; ++q) acc[q] = fmaf(sp_at(row.J, a[q]) * row.D, sp_at(row.J, b[q]), acc[q]);
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int sl = base + 32 * q + lane;
        if (sl < nfac) {
          if (last) {
            if (!first) acc[q] = s.Hp[sl] + acc[q];
            s.Hp[sl] = acc[q];
          }
          s.N[sl] = acc[q];
        }
      }
    }
    t0 = t1;
  } while (t0 < count);
  if (!first && part == 0) write_union(s, count);
  if (outside && part == 0)
    count_violations(first, JRES ? s.Jsm : s.Jg, s.ldj, nv, s.Dsm, s.masks, s.r4, s.mwords, s.ids, count, SP.pmask, SP.pair, s.viol,
                     s.world, lane);
  team_sync<TEAM>(s);
  IMN_MARK(s, 18);
}

}  // namespace imn
