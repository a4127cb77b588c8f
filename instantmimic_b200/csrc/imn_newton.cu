// imn_newton.cu -- the fused Newton constraint solve, a warp or a small team of warps per world.
//
// One launch replaces the reference's whole solve pipeline
// (mjw_step_optimized.py:2588-2680): _solve_init_dof, the init of
// newton_fusion.py:431-472 (Jaref, Ma = M qacc, constraint update, gradient,
// Hessian, factor, first search direction), the persistent iteration loop of
// newton_fusion.py:170-296 and the final qfrc_constraint_from_grad.
//
// B200 mapping.  The solve is latency-bound small dense algebra (nv <= 79), not a
// tensor-core contraction, so the design goal is to touch HBM exactly once: a warp owns a world, one
// CTA per SM holds as many worlds as fit.  A world's J and row data arrive in shared memory
// through TMA bulk copies (cp.async.bulk, one mbarrier; M, read once per iteration,
// stays in global memory and comes through L1), the Hessian, its
// Cholesky factor and every vector stay on chip for all iterations, and the
// results are written once.  A warp needs no block barrier (only __syncwarp) and
// lane reductions are shuffle trees; a warp that has finished a world takes the next from a
// counter, worlds with many rows first, so that iteration counts that differ leave no SM waiting.
// Models whose J would leave room for few worlds per SM stream it through a 32-row tile (TMA bulk
// copies or 16-byte pieces from L2) instead.  Where the worlds in hand leave warps of an SM unused (small
// batches, very large worlds) a team of two to four warps shares each world (plan_launch).
// The initialisation runs through the same code as an iteration (as "iteration 0"
// without a line search): the kernel is bound by instruction fetch and latency, so
// every stage exists once.
//
// Arithmetic contract.  Every value that decides an active set or an iteration
// count is formed by the same float32 operations in the same order as the CPU
// oracle used by the tests: explicit fmaf chains in ascending index order,
// shuffle-down trees for lane sums, IEEE sqrt and division.  Blocking, register
// tiling and the lane mapping never change the order in which one value
// receives its terms.
#include <stdio.h>

#include "imn_newton_factor.cuh"
#include "imn_newton_ls.cuh"

namespace imn {

// Phase timers, compiled only into the profiling build (-DIMN_PROFILE).
#ifdef IMN_PROFILE
__device__ unsigned long long g_prof[24];
#define PROF_DECL long long prof_t = clock64(); long long prof_acc[24] = {0}; s.prof_acc = prof_acc; s.prof_t = &prof_t
#define PROF(k) do { const long long t_ = clock64(); prof_acc[k] += t_ - prof_t; prof_t = t_; } while (0)
#define PROF_FLUSH do { if (tid == 0) for (int k_ = 0; k_ < 24; ++k_) atomicAdd(&g_prof[k_], (unsigned long long)prof_acc[k_]); } while (0)
#else
#define PROF_DECL
#define PROF(k)
#define PROF_FLUSH
#endif

// Internal error bit OR-ed into `overflow` when the input copies of a world do not
// complete within the wait limit (the world is left unsolved).
#define IMN_OVERFLOW_COPY_TIMEOUT (1 << 30)

struct Geom {
  int nv, njmax, ldj, ldp, ldu, nM, bd;
  bool j16;  // a streamed J is copied row by row and read 16 bytes at a time (j_tile)
  int jrows;  // rows of J held in shared memory (njmax when resident, else 32)
  // offsets in 4-byte words; every region starts on a 16-byte boundary
  int oBar, oJ, oA, oVec, nv4, oRowF, oRowI, oMask, mwords, r4, oUni, total;
  // tables in shared memory (Tables), in words from its start; the worlds' slices (`total` words
  // each, offsets above) follow at `tab` words.  warps: worlds in hand per CTA
  bool tsm;
  int tM, tF, tB, tS, tO, tP, tab, warps;
  // warps per world (make_geom); the tiles of a streamed J are `tile` words apart
  int parts, tile, oBox;
  bool early;  // the launch before this one is its own counter kernel, which writes no table
  // polls a copy wait may take before the world gives up, and the failure-path test
  // switch: when set no bulk copy is issued (plain loads bring the data) while the
  // barrier is told to expect bytes, so the wait runs out with nothing in flight
  int wait_polls, withhold_copies;
};

// Set by imn_set_copy_wait_limit; read when a launch is planned.
static int g_wait_polls = 1 << 22;
static int g_withhold_copies = 0;


// Most warps (worlds in hand) of a CTA: bounds the registers at 128 with a resident J, 168 with a
// streamed one, whose worlds take more shared memory and are fewer.
static const int kResidentWarps = 16, kStreamedWarps = 12;

static inline int up4(int n) { return (n + 3) & ~3; }

static Geom make_geom(const ImnModel& m, const ImnData& d, bool resident, const ImnSparsePlan* sp, int parts) {
  Geom g;
  g.nv = m.nv;
  g.njmax = d.njmax;
  g.ldj = (int)d.J_ld_row;
  g.ldu = up4(m.nv + 1);
  g.nM = m.nM;
  g.bd = m.nv_pad >= 64 ? 64 : 32;
  g.jrows = resident ? d.njmax : 32;
  g.nv4 = up4(m.nv + 1);  // M_mulm_lanes reads a zero behind a vector
  g.r4 = up4(d.njmax);
  int o = 0;
  g.parts = parts;
  g.oBar = o, o += 8 * parts;  // per warp: load barrier, its phase, jfail; tile barrier (J16), its phase
  g.oBox = o, o += parts > 1 ? 12 : 0;  // single values for the team
  // a streamed tile may start up to three floats into its buffer and end on a 16-byte boundary
  // a dense block reads up to three floats past a row; the gathered rows are up4(nv) floats apart
  g.ldp = 4 * ((m.nv / 4) | 1);
  g.j16 = !resident && m.nv % 4 == 0 && d.J_ld_row % 4 == 0 && !d.J_world_offset && d.J_ld_world % 4 == 0 &&
          (reinterpret_cast<uintptr_t>(d.efc_J) & 15) == 0;
  g.tile = resident ? up4(g.jrows * g.ldj + 3) : g.j16 ? 32 * g.ldp : max(up4(32 * g.ldj) + 8, 32 * up4(m.nv));
  g.oJ = o, o += resident ? g.tile : parts * g.tile;
  // dense: H and its factor share one (nv+1) x ldu array; sparse plan: packed H | N | 1/D
  g.oA = o, o += sp ? up4(sp->nfac) + up4(sp->nslots) + up4(m.nv) : (m.nv + 1) * g.ldu;
  // dof vectors; the dense factor needs two more (forward-solve scratch, 1 / pivot)
  g.oVec = o, o += (sp ? 6 : 8) * g.nv4;
  g.oRowF = o, o += 4 * g.r4;
  g.oRowI = o, o += up4(3 * g.r4 / 2);  // three 16-bit row lists
  g.mwords = (m.nv + 31) / 32;
  g.oMask = o, o += g.mwords * g.r4;
  g.oUni = o, o += up4(m.nv + 1);
  g.total = o;
  int t = 0;
  g.tM = t, t += (m.n_mulm_batches + 1) * 128;
  g.tF = t, t += sp ? (sp->nfstep + 1) * 128 : 0;
  g.tB = t, t += sp ? (sp->nbsweep + 1) * 64 : 0;
  g.tS = t, t += sp ? up4(sp->nfac) : 0;
  g.tO = t, t += sp ? up4(m.nv) : 0;
  g.tP = t;
  const int masks = sp ? up4(m.nv * g.mwords) : 0;
  // A plan's tables stay in global memory when they would take more than a third of an SM's shared memory;
  // without a plan there is the M v program only, at most 31 KB for 79 dofs.  us per solve, tables in shared /
  // global memory: 34 dofs (19 KB) 592 worlds 155 / 171, 8192 worlds 562 / 547 (14 worlds per SM against 16);
  // 56 dofs (43 KB) 4096 worlds 1114 / 1193 (9 against 11); 79 dofs (57 KB) 1401 / 1940.  Beyond the
  // third: 64 dofs with coupled limbs (81 KB) 592 worlds 472 / 688, 4096 worlds 1803 / 1955; 79 dofs
  // (106 KB) 661 / 869, 3186 / 3312; (137 KB) 1437 / 1112, 7720 / 4234.  The third keeps the tables of every
  // tree alone on chip and errs on the side of more worlds; the crossing lies near half an SM.
  g.tsm = !sp || 4 * t <= kMaxSmem / 3;
  // The pattern's masks (up to 960 bytes) came to the staged tables last: a world of thousands of rows that leaves no
  // room for them reads all tables from global memory rather than being refused (79 dofs: row limits 4457 to 4484).
  if (parts == 1 && 4 * (t + g.total) <= kMaxSmem && 4 * (t + masks + g.total) > kMaxSmem) g.tsm = false;
  g.tab = g.tsm ? t + masks : 0;
  g.wait_polls = g_wait_polls;
  g.withhold_copies = g_withhold_copies;
  return g;
}

// The two overflow warnings of the reference (newton_stages.py:430-436, newton_fusion.py:283-289),
// kept out of line (measured 0.6 % faster than inline).
__device__ __noinline__ void warn_limit(int which, unsigned limit) {
  if (which == 0)
    printf("linesearch iterations limit reached - please increase ls_iterations to %u\n", limit);
  else
    printf("solver iterations limit reached - please increase iterations to %u\n", limit);
}

// A CTA holds `warps` worlds in hand, a warp (or a team of `parts` warps) each, and as many CTAs as there
// are SMs share the batch: every table of the model and the plan then exists once per SM in shared
// memory.  Read from global memory by one-world CTAs the tables cost about 210 cycles per trip of the
// loops they drive, whatever the distance of the prefetch.  The worlds of a CTA never wait for one another
// after the tables have arrived.  A slot's first world is number slot * grid + CTA of the launch order,
// further ones come from a counter.
// A team (TEAM) runs the same statements: every warp takes the same decisions from values in shared
// memory, part 0 does the stages that are one chain and passes its results on in `box`, every stage that
// others read from ends in team_sync.
// The solve is written as one loop whose trip is "take a world if none is in hand, else run one
// pass of it" rather than as a load followed by a pass loop: the same statements, but the compiler
// lays the single loop out better (when a CTA held one world: 0.836 -> 0.796 ms per 8192 humanoid worlds at
// the same occupancy).
template <bool JRES, bool J16, int SPARSE, bool STATS, bool TSM, bool TEAM>
__device__ __forceinline__ void newton_worlds(const ImnModel& m, const ImnData& d, const ImnCtx& cx, const Geom& g,
                                              const ImnSparsePlan& sp) {
  extern __shared__ __align__(16) float smem_all[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the first warps of the teams come first, so that they are spread over the SM's four schedulers
  const int part = TEAM ? warp / g.warps : 0, slot = TEAM ? warp - part * g.warps : warp;
  const int tid = lane + 32 * part, threads = TEAM ? 32 * g.parts : 32;  // of the world's team
  float* smem = smem_all + g.tab + slot * g.total;
  const int nv = g.nv, R = g.njmax, nv4 = g.nv4, r4 = g.r4;

  void* bar = smem + g.oBar + 8 * part;  // copy barriers per warp
  World s;
  s.nv = nv, s.ldj = g.ldj, s.ldp = g.ldp, s.ldu = g.ldu, s.bd = g.bd, s.lane = lane, s.nM = g.nM;
  s.part = part, s.parts = g.parts, s.team_bar = 1 + slot, s.tile_words = g.tile;
  s.box = reinterpret_cast<int*>(smem + g.oBox);
  s.Jsm = smem + g.oJ;
  s.tile = s.Jsm + (JRES ? 0 : part * g.tile);
  s.A = smem + g.oA;
  s.qacc = smem + g.oVec;
  s.Ma = s.qacc + nv4;
  s.search = s.Ma + nv4;
  s.mv = s.search + nv4;
  s.grad = s.mv + nv4;
  s.qfs = s.grad + nv4;
  s.xsm = SPARSE ? nullptr : s.qfs + nv4;
  s.dinv = SPARSE ? nullptr : s.xsm + nv4;
  s.Jaref = smem + g.oRowF;
  s.jv = s.Jaref + r4;
  s.Dsm = s.jv + r4;
  s.force = s.Dsm + r4;
  s.masks = reinterpret_cast<uint32_t*>(smem + g.oMask);
  s.mwords = g.mwords, s.r4 = r4;
  s.state = reinterpret_cast<uint16_t*>(smem + g.oRowI);
  s.ids = s.state + r4;
  s.frows = s.ids + r4;  // rows with a nonzero force, ascending
  s.uni = reinterpret_cast<int*>(smem + g.oUni);
  s.mulm_batches = m.n_mulm_batches;
  if (TSM) {
    s.tab.mulm = reinterpret_cast<const uint4*>(smem_all + g.tM);
    s.tab.fstep = reinterpret_cast<const uint4*>(smem_all + g.tF);
    s.tab.bstep = reinterpret_cast<const uint2*>(smem_all + g.tB);
    s.tab.slots = reinterpret_cast<const uint32_t*>(smem_all + g.tS);
    s.tab.orig = reinterpret_cast<const uint32_t*>(smem_all + g.tO);
    s.tab.pmask = reinterpret_cast<const uint32_t*>(smem_all + g.tP);
  } else {
    s.tab.mulm = reinterpret_cast<const uint4*>(m.M_mulm_lanes);
    s.tab.fstep = reinterpret_cast<const uint4*>(sp.fstep);
    s.tab.bstep = reinterpret_cast<const uint2*>(sp.bstep);
    s.tab.pmask = sp.pmask;
  }
  s.M_rowadr = m.M_rowadr, s.M_rownnz = m.M_rownnz, s.M_colind = m.M_colind;
  int* const load_phase_at = static_cast<int*>(bar) + 2;  // the barrier itself takes two words
  s.jbar = J16 ? static_cast<float*>(bar) + 4 : bar;  // J16: every lane arrives at the tiles' own barrier
  s.jphase = load_phase_at + (J16 ? 4 : 0);
  s.jfail = load_phase_at + 1;
  s.wait_polls = g.wait_polls, s.withhold_copies = g.withhold_copies;
  s.Hp = s.A;
  s.N = s.A + (SPARSE ? ((sp.nfac + 3) & ~3) : 0);
  s.iD = s.N + (SPARSE ? ((sp.nslots + 3) & ~3) : 0);
  s.Jbeg = d.efc_J;
  s.Jend = d.efc_J + (d.J_world_offset ? (size_t)d.J_elems
                                       : (size_t)(d.nworld - 1) * d.J_ld_world + (size_t)d.njmax * d.J_ld_row);
  if (lane == 0) {
    mbar_init(bar, 1), *load_phase_at = 0;
    if (J16) mbar_init(s.jbar, 32), *s.jphase = 0;
  }
  __syncwarp();
  if (!g.early) chain_wait();
  if (TSM) {
    auto stage = [&](int at, const void* src, int words) {
#pragma unroll 1
      for (int i = threadIdx.x; i < words / 4; i += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_all + at + 4 * i)),
                     "l"(static_cast<const uint4*>(src) + i)
                     : "memory");
    };
    stage(g.tM, m.M_mulm_lanes, (m.n_mulm_batches + 1) * 128);
    if (SPARSE) {
      stage(g.tF, sp.fstep, (sp.nfstep + 1) * 128);
      stage(g.tB, sp.bstep, (sp.nbsweep + 1) * 64);
#pragma unroll 4
      for (int i = threadIdx.x; i < sp.nfac; i += blockDim.x)
        reinterpret_cast<uint32_t*>(smem_all + g.tS)[i] =
            4u * __ldg(sp.s_a + i) | (4u * __ldg(sp.s_b + i)) << 9 | (uint32_t)(__ldg(sp.s_m + i) + 1) << 18;
      for (int i = threadIdx.x; i < nv; i += blockDim.x) reinterpret_cast<uint32_t*>(smem_all + g.tO)[i] = __ldg(sp.orig + i);
      for (int i = threadIdx.x; i < nv * g.mwords; i += blockDim.x) reinterpret_cast<uint32_t*>(smem_all + g.tP)[i] = __ldg(sp.pmask + i);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  }
  if (g.early) chain_wait();
  // The release itself gains nothing (imn_common.cuh).  The dense kernels keep the branch because the compiler lays
  // their loop out better with it, the sparse ones better without: 64 dofs x 512 rows 4148 us without, 4116
  // with; 56-dof plan, 4096 worlds, 1091 without, 1111 with.
  if (SPARSE == 0 && gridDim.x <= 64) chain_release();

  PROF_DECL;
  // the world in hand
  int w = 0, nefc = 0, ne = 0, nef = 0;
  bool rowless = false;
  size_t dofo = 0, efco = 0;
  float tolerance = 0.0f, ls_tolerance = 0.0f, scale = 1.0f;
  float search_dot = 0.0f, grad_dot = 0.0f, grad_scale = 1.0f, decrement = 0.0f;
  float improvement = 0.0f, alpha = 0.0f;
  int quad_count = 0, state_count = 0, niter = 0, overflow = 0;
  bool search_unchanged = false, ls_exhausted = false;
  int st_passes = 0, st_flips = 0, st_factor = 0, st_grad = 0;  // work counters (ctx.stats)
  bool have = false, first = true;
  bool outside = false;  // a row of the world leaves the sparse plan's pattern
  int idx = slot * (int)gridDim.x + (int)blockIdx.x;  // the next world's place in the launch order
  bool turn = false;  // the first world was taken

#pragma unroll 1
  for (;;) {
    if (!have) {
      // ---- take a world --------------------------------------------------------------
      if (turn && cx.work_counter) {
        if (tid == 0) idx = (int)gridDim.x * g.warps + atomicAdd(cx.work_counter, 1);
        idx = __shfl_sync(IMN_FULL_MASK, idx, 0);
      } else if (turn) {
        idx += (int)gridDim.x * g.warps;
      }
      turn = true;
      if (TEAM) {  // part 0 takes the world; past the barrier every warp has left the previous one
        if (tid == 0) s.box[0] = idx;
        team_sync<TEAM>(s);
        idx = s.box[0];
      }
      if (idx >= d.nworld) break;
      {
        w = cx.world_order ? cx.world_order[idx] : idx;
        s.world = w;
        s.viol = (SPARSE && cx.hfactor) ? cx.hfactor + ((size_t)w + 1) * m.nv_pad * m.nv_pad - 1 : nullptr;
        const int nefc_in = d.nefc[w];
        nefc = min(R, nefc_in);
        ne = d.ne[w], nef = ne + d.nf[w];
        s.nefc = nefc, s.ne = ne, s.nef = nef;
        if (TEAM) s.mulm_part = ((nefc + 31) >> 5) % g.parts;  // the one behind those that take a tile of rows
        rowless = nefc_in == 0;
        dofo = (size_t)w * d.dof_ld, efco = (size_t)w * d.efc_ld;
        s.Jg = d.efc_J + (d.J_world_offset ? (size_t)d.J_world_offset[w] : (size_t)w * d.J_ld_world);
        s.M = d.M + (size_t)w * d.M_ld;
        s.floss = d.efc_frictionloss + efco;

        // ---- load: TMA bulk copies for the 16-byte-aligned bulk of every array, plain
        // loads for the ragged ends ---------------------------------------------------
        const float* q0 = (m.warmstart && !rowless) ? d.qacc_warmstart : d.qacc_smooth;
        struct Src {
          float* dst;
          const float* src;
          int n;
        };
        const Src srcs[5] = {
            {s.Jsm, s.Jg, JRES ? nefc * s.ldj : 0},
            {s.Dsm, d.efc_D + efco, nefc},
            {s.jv, d.efc_aref + efco, nefc},  // aref is parked in jv until Jaref is formed
            {s.qacc, q0 + dofo, nv},
            {s.qfs, d.qfrc_smooth + dofo, nv},
        };
        __syncwarp();  // every lane has left the previous world
        bool arrived = false;
        if (TEAM && lane == 0) *s.jfail = 0;
        if (!TEAM || part == 0) {
          const uint32_t load_phase = (uint32_t)*load_phase_at;
          // the previous world's values were written through the generic proxy
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            *load_phase_at = (int)(load_phase ^ 1u);
            *s.jfail = 0;
          }
          __syncwarp();
          const bool bulk = !(g.withhold_copies & 1);
          uint32_t tx = 0;
#pragma unroll
          for (int k = 0; k < 5; ++k)
            if (bulk && (reinterpret_cast<uintptr_t>(srcs[k].src) & 15) == 0) tx += (uint32_t)(srcs[k].n & ~3) * 4u;
          if (lane == 0) {
            mbar_expect_tx(bar, bulk ? tx : 16u);
#pragma unroll
            for (int k = 0; k < 5; ++k) {
              const uint32_t bytes =
                  bulk && (reinterpret_cast<uintptr_t>(srcs[k].src) & 15) == 0 ? (uint32_t)(srcs[k].n & ~3) * 4u : 0u;
              if (bytes) bulk_g2s(srcs[k].dst, srcs[k].src, bytes, bar);
            }
          }
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            const int done_n = bulk && (reinterpret_cast<uintptr_t>(srcs[k].src) & 15) == 0 ? (srcs[k].n & ~3) : 0;
#pragma unroll 1
            for (int i = done_n + lane; i < srcs[k].n; i += 32) srcs[k].dst[i] = srcs[k].src[i];
          }
#pragma unroll 1
          for (int i = lane; i < nv; i += 32) s.search[i] = 0.0f, s.mv[i] = 0.0f, s.grad[i] = 0.0f;
          if (lane == 0) s.search[nv] = 0.0f, s.qacc[nv] = 0.0f;
#pragma unroll 1
          for (int i = lane; i <= nv; i += 32) s.uni[i] = 0;
          // bounded wait for the copies; when it runs out the copies get one more bounded wait
          // (they write shared memory that the warp's next world takes over), then the world is left
          // unsolved with the time-out bit set and the barrier starts anew
#pragma unroll 1
          for (int tries = 0; tries < g.wait_polls && !arrived; ++tries) arrived = mbar_try_wait(bar, load_phase);
          if (!arrived) {
            bool late = false;
#pragma unroll 1
            for (int tries = 0; tries < g.wait_polls && !late; ++tries) late = mbar_try_wait(bar, load_phase);
            if (lane == 0) {
              d.overflow[w] |= IMN_OVERFLOW_COPY_TIMEOUT;
              mbar_restart(bar, 1);
              *load_phase_at = 0;
            }
          }
        }
        if (TEAM) {
          if (tid == 0) s.box[1] = arrived;
          team_sync<TEAM>(s);
          arrived = s.box[1] != 0;
        }
        if (arrived) {
          have = true, first = true;
          search_dot = 0.0f, grad_dot = 0.0f, grad_scale = 1.0f, decrement = 0.0f;
          improvement = 0.0f, alpha = 0.0f;
          quad_count = 0, state_count = 0, niter = 0, overflow = 0;
          search_unchanged = false, ls_exhausted = false;
          if (STATS) st_passes = 0, st_flips = 0, st_factor = 0, st_grad = 0;
          tolerance = m.opt_tolerance[w % m.n_tolerance];
          ls_tolerance = m.opt_ls_tolerance[w % m.n_ls_tolerance];
          scale = m.stat_meaninertia[w % m.n_meaninertia] * (float)nv;
        }
        __syncwarp();
        PROF(0);
      }
    }
    if (!have) continue;

    // Pass 0 is the initialisation (newton_fusion.py:431-472): Jaref = J qacc - aref,
    // Ma = M qacc, row states, gradient, full Hessian, factor, first search direction.
    // Every later pass is one Newton iteration (newton_fusion.py:170-296).
    bool finished = false, failed = false;
    do {
      // one call site: Ma = M qacc, Jaref = J qacc - aref on pass 0; mv = M search,
      // jv = J search afterwards
      if (first || !search_unchanged)
        products<JRES, J16, TSM, TEAM>(s, first ? s.qacc : s.search, first ? s.Ma : s.mv, first ? s.Jaref : s.jv,
                       first ? s.jv : nullptr);
      team_sync<TEAM>(s);
      PROF(5);
      if (rowless) {
        finished = true;
        break;
      }
      float noise_floor = 0.0f;
      bool ls_converged = true;
      if (!first && part == 0) {  // the search and the row lists are part 0's
        const LineSearchResult ls =
            line_search(s, search_dot, tolerance, ls_tolerance, scale, m.alpha_noise_eps, m.ls_iterations);
        alpha = ls.alpha, improvement = ls.improvement, noise_floor = ls.noise_floor;
        ls_converged = ls.converged;
        if (STATS) st_passes += ls.passes;
#pragma unroll 1
        for (int i = lane; i < nv; i += 32) {
          s.qacc[i] = fmaf(alpha, s.search[i], s.qacc[i]);
          s.Ma[i] = fmaf(alpha, s.mv[i], s.Ma[i]);
        }
      }
      PROF(6);
      // ---- move along the search direction, re-evaluate rows, list QUADRATIC flips
      // (newton_stages.py:373-426); on pass 0 this is upstream's constraint update
      quad_count = 0;
      state_count = 0;
      int nfr = 0;
#pragma unroll 1
      for (int base = part == 0 ? 0 : nefc; base < nefc; base += 32) {
        const int r = base + lane;
        bool flip = false, changed = false, leaves = false;
        float f = 0.0f;
        if (r < nefc) {
          const float nj = first ? s.Jaref[r] : rounded_step(s.Jaref[r], alpha, s.jv[r]);
          s.Jaref[r] = nj;
          // an equality or an inequality row without a branch; friction-loss rows are few and come first
          const float D = s.Dsm[r];
          const bool quad = r < ne || !(nj >= 0.0f);
          f = quad ? -D * nj : 0.0f;
          int ns = quad ? IMN_STATE_QUADRATIC : IMN_STATE_SATISFIED;
          if (r >= ne && r < nef) eval_friction(nj, D, s.floss[r], f, ns);
          const int old = first ? -1 : s.state[r];
          s.force[r] = f;
          s.state[r] = ns;
          if (first) s.jv[r] = 0.0f;  // aref no longer needed
          // pass 0 lists every QUADRATIC row (the rows of the full Hessian, whatever their
          // force: a row at Jaref == 0 has no force but still carries D J^T J); later
          // passes list the rows whose QUADRATIC membership flipped
          flip = first ? ns == IMN_STATE_QUADRATIC
                       : (old == IMN_STATE_QUADRATIC) != (ns == IMN_STATE_QUADRATIC);
          changed = old != ns;
          leaves = ns != IMN_STATE_QUADRATIC;
        }
        const unsigned below = (1u << lane) - 1u;
        const unsigned fm = __ballot_sync(IMN_FULL_MASK, flip);
        if (flip) s.ids[quad_count + __popc(fm & below)] = r | (leaves ? 0x8000 : 0);
        quad_count += __popc(fm);
        state_count += __popc(__ballot_sync(IMN_FULL_MASK, changed));
        const unsigned nz = __ballot_sync(IMN_FULL_MASK, f != 0.0f);
        if (f != 0.0f) s.frows[nfr + __popc(nz & below)] = r;
        nfr += __popc(nz);
      }
      if (TEAM) {
        if (tid == 0) {
          s.box[2] = quad_count, s.box[3] = state_count, s.box[4] = nfr, s.box[7] = ls_converged;
          s.box[8] = __float_as_int(alpha), s.box[9] = __float_as_int(improvement), s.box[10] = __float_as_int(noise_floor);
        }
        team_sync<TEAM>(s);
        quad_count = s.box[2], state_count = s.box[3], nfr = s.box[4], ls_converged = s.box[7] != 0;
        alpha = __int_as_float(s.box[8]), improvement = __int_as_float(s.box[9]), noise_floor = __int_as_float(s.box[10]);
      }
      if (!first) {
        ls_exhausted = fabsf(alpha) < noise_floor;
        if (ls_exhausted) state_count += 1;
        if (!ls_converged) {
          if ((m.warn_overflow & m.overflow_ls_iterations) && tid == 0) warn_limit(0, (unsigned)m.ls_iterations);
          overflow |= m.overflow_ls_iterations;
        }
      }
      __syncwarp();
      PROF(7);
      // ---- gradient (newton_stages.py:745-798), Hessian, factor (newton_stages.py:629-740)
      const bool changed = first || state_count != 0;
      search_unchanged = !changed;
      if (!changed) {
        const float sigma = grad_scale, ns = sigma - alpha;
        const float ratio = sigma != 0.0f ? ns / sigma : 0.0f;
        const float rsq = ratio * ratio;
        grad_dot *= rsq;
        decrement *= rsq;
        grad_scale = ns;
      } else {
        full_gradient<JRES, TEAM>(s, nfr);
        if (STATS) {
          ++st_grad;
          if (!first) st_flips += quad_count;
          if (first || quad_count > 0) ++st_factor;
        }
        PROF(8);
        grad_scale = 1.0f;
        if (first || quad_count > 0) {
          if (SPARSE && first) {
            bool bad = false;
#pragma unroll 1
            for (int r = lane; r < nefc; r += 32) bad = bad || row_outside<TSM>(s.masks, r4, g.mwords, r, s.tab.pmask);
            outside = __any_sync(IMN_FULL_MASK, bad);
          }
          if (SPARSE)
            hessian_sparse<JRES, J16, TSM, TEAM>(s, quad_count, first, outside, sp);
          else
            hessian_dense<JRES, J16, TEAM>(s, quad_count, first);
        }
        PROF(9);
        // the sweeps of a sparse factor's levels can be shared by the team; the solves and the dense factor are chains: part 0's
        if (SPARSE && (first || quad_count > 0)) {
          // refactor the packed H, or solve with the resident factor
          // (sparse_hessian.py:490-547)
          sp_load_rhs<TSM>(sp, s.tab, s.N, s.grad, tid, threads);
          team_sync<TEAM>(s);
          IMN_MARK(s, 1);
          if (SPARSE == 2 || part == 0)
            sp_factor_steps<TSM, SPARSE == 2>(sp, s.tab, s.N, lane, part, g.parts, [&] { team_sync<SPARSE == 2>(s); });
          IMN_MARK(s, 2);
        }
        SearchSums sum = {0.0f, 0.0f, 0.0f};
        if (TEAM && part != 0) {
        } else if (SPARSE) {
          if (!(first || quad_count > 0)) {
            sp_forward(sp, s.N, s.iD, s.grad, lane);
            IMN_MARK(s, 3);
          }
          sum = sp_backward_steps<TSM>(sp, s.tab, s.N, s.iD, s.grad, s.search, s.bd, lane);
          IMN_MARK(s, 4);
        } else {
          sum = factor_solve(s, first || quad_count > 0);
        }
        if (TEAM) {
          if (tid == 0) s.box[5] = __float_as_int(sum.xx), s.box[6] = __float_as_int(sum.gx), s.box[11] = __float_as_int(sum.gg);
          team_sync<TEAM>(s);
          sum = {__int_as_float(s.box[5]), __int_as_float(s.box[6]), __int_as_float(s.box[11])};
        }
        search_dot = sum.xx, decrement = sum.gx, grad_dot = sum.gg;
        PROF(10);
      }
      bool lost = !JRES && *s.jfail;
      if (TEAM && !JRES) {  // the flags are raised by `products`, a barrier or more ago
        const int* flags = reinterpret_cast<const int*>(smem + g.oBar) + 3;  // jfail of each warp
#pragma unroll 1
        for (int p = 0; p < g.parts; ++p) lost = lost || flags[8 * p] != 0;
      }
      if (lost) {
        // a tile copy of this pass did not complete within its wait limit, so the pass
        // worked on stale rows: give the copy one more bounded wait (it writes this
        // CTA's shared memory), then leave the world unsolved, results unwritten
        const uint32_t parity = (uint32_t)*s.jphase ^ 1u;
        bool arrived = TEAM && !*s.jfail;  // a team: each warp its own copy
        const bool restart = !arrived;
#pragma unroll 1
        for (int tries = 0; tries < g.wait_polls && !arrived; ++tries) arrived = mbar_try_wait(s.jbar, parity);
        if (tid == 0) d.overflow[w] |= IMN_OVERFLOW_COPY_TIMEOUT;
        if (restart && lane == 0) {
          mbar_restart(s.jbar, J16 ? 32 : 1);
          *s.jphase = 0;
        }
        finished = true, failed = true;
        break;
      }
      if (first) {
        quad_count = 0, state_count = 0;
        break;
      }
      // ---- convergence (newton_fusion.py:267-295) -------------------------------
      ++niter;
      // the three measures over the lanes, one division for all of them, and no branch between them
      float measure = lane == 0 ? improvement : lane == 1 ? sqrtf(grad_dot) : 0.5f * decrement;
      measure = measure / scale;
      const bool converged =
          __any_sync(IMN_FULL_MASK, alpha == 0.0f || (measure < tolerance && (lane != 0 || improvement > 0.0f)));
      if (converged || niter == m.iterations) {
        if (!converged) {
          if ((m.warn_overflow & m.overflow_iterations) && tid == 0) warn_limit(1, (unsigned)m.iterations);
          overflow |= m.overflow_iterations;
        }
        if (tid == 0 && cx.nsolving) atomicAdd(cx.nsolving, -1);
        finished = true;
      }
    } while (false);
    first = false;
    if (!finished) continue;
    have = false;
    if (failed) continue;

    // ---- results (once) ---------------------------------------------------------
#pragma unroll 1
    for (int i = tid; i < nv; i += threads) {
      d.qacc[dofo + i] = s.qacc[i];
      d.efc_Ma[dofo + i] = s.Ma[i];
      d.qfrc_constraint[dofo + i] = rowless ? 0.0f : fmaf(-grad_scale, s.grad[i], s.Ma[i] - s.qfs[i]);
      if (cx.search) cx.search[dofo + i] = s.search[i];
      if (cx.mv) cx.mv[dofo + i] = s.mv[i];
      if (cx.grad) cx.grad[(size_t)w * cx.grad_ld + i] = s.grad[i];
    }
#pragma unroll 1
    for (int r = tid; r < nefc; r += threads) {
      d.efc_force[efco + r] = s.force[r];
      d.efc_state[efco + r] = s.state[r];
      if (cx.Jaref) cx.Jaref[efco + r] = s.Jaref[r];
      if (cx.jv) cx.jv[efco + r] = s.jv[r];
      if (cx.quad_changed_ids && r < quad_count) cx.quad_changed_ids[efco + r] = s.ids[r] & 0x7FFF;
    }
    if (cx.dof_union && !rowless)
#pragma unroll 1
      for (int i = tid; i <= nv; i += threads) cx.dof_union[(size_t)w * (nv + 1) + i] = s.uni[i];
    if (SPARSE && !rowless && cx.hfactor && cx.h) {
      // packed H | N | 1/D, the reference's hfactor layout (sparse_hessian.py:488-489).
      // The factor never leaves the chip here, so it is written only for callers that
      // inspect the context (those that also pass ctx.h); the violation counter in the
      // last element is always live.
      float* Uf = cx.hfactor + (size_t)w * m.nv_pad * m.nv_pad;
#pragma unroll 1
      for (int q = tid; q < sp.nfac; q += threads) Uf[q] = s.Hp[q], Uf[sp.nfac + q] = s.N[q];
#pragma unroll 1
      for (int q = tid; q < nv; q += threads) Uf[2 * sp.nfac + q] = s.iD[q];
    }
    if (!SPARSE && !rowless) {
      const size_t ho = (size_t)w * m.nv_pad * m.nv_pad;
      if (cx.h)
#pragma unroll 1
        for (int r = 0; r < nv; ++r)
#pragma unroll 1
          for (int c = r + tid; c < nv; c += threads) cx.h[ho + (size_t)r * m.nv_pad + c] = s.A[(c + 1) * s.ldu + r];
      if (cx.hfactor)
#pragma unroll 1
        for (int r = 0; r < nv; ++r)
#pragma unroll 1
          for (int c = r + tid; c < nv; c += threads) cx.hfactor[ho + (size_t)r * m.nv_pad + c] = s.A[r * s.ldu + c];
    }
    PROF(11);
    if (tid == 0) {
      d.solver_niter[w] = niter;
      if (overflow) d.overflow[w] |= overflow;
      if (cx.search_dot) cx.search_dot[w] = search_dot;
      if (cx.done) cx.done[w] = 1;
      if (STATS && cx.stats) {
        int4 st = make_int4(st_passes, st_flips, st_factor, st_grad);
        *reinterpret_cast<int4*>(cx.stats + 4 * (size_t)w) = st;
      }
      if (!rowless) {
        if (cx.grad_dot) cx.grad_dot[w] = grad_dot;
        if (cx.grad_scale) cx.grad_scale[w] = grad_scale;
        if (cx.newton_decrement) cx.newton_decrement[w] = decrement;
        if (cx.improvement) cx.improvement[w] = improvement;
        if (cx.alpha) cx.alpha[w] = alpha;
        if (cx.search_unchanged) cx.search_unchanged[w] = search_unchanged;
        if (cx.ls_exhausted) cx.ls_exhausted[w] = ls_exhausted;
        if (cx.quad_changed_count) cx.quad_changed_count[w] = quad_count;
        if (cx.state_changed_count) cx.state_changed_count[w] = state_count;
      }
    }
    __syncwarp();
  }
  PROF_FLUSH;
}

// Two entry points over the same body, with the register bounds that follow from the most worlds
// in hand (kResidentWarps, kStreamedWarps).
// SPARSE: 0 the dense factor, 1 a sparse plan, 2 a sparse plan whose sweeps a team shares (sp_factor_steps).
// STATS compiles the work counters of ImnCtx.stats in: four more live values in a kernel that is
// short of registers cost 9 % of its speed (measured), so the counting variants run only for
// callers that pass the stats array.
template <int SPARSE, bool STATS, bool TSM, bool TEAM>
__global__ void __launch_bounds__(32 * kResidentWarps, 1)
    newton_kernel_resident(const ImnModel m, const ImnData d, const ImnCtx cx, const Geom g, const ImnSparsePlan sp) {
  newton_worlds<true, false, SPARSE, STATS, TSM, TEAM>(m, d, cx, g, sp);
}
template <bool J16, int SPARSE, bool STATS, bool TSM, bool TEAM>
__global__ void __launch_bounds__(32 * kStreamedWarps, 1)
    newton_kernel_streamed(const ImnModel m, const ImnData d, const ImnCtx cx, const Geom g, const ImnSparsePlan sp) {
  newton_worlds<false, J16, SPARSE, STATS, TSM, TEAM>(m, d, cx, g, sp);
}
using Kernel = void (*)(ImnModel, ImnData, ImnCtx, Geom, ImnSparsePlan);
template <int SPARSE, bool STATS, bool TSM, bool TEAM>
static Kernel newton_kernel(bool resident, bool j16) {
  return resident ? (Kernel)newton_kernel_resident<SPARSE, STATS, TSM, TEAM>
         : j16    ? (Kernel)newton_kernel_streamed<true, SPARSE, STATS, TSM, TEAM>
                  : (Kernel)newton_kernel_streamed<false, SPARSE, STATS, TSM, TEAM>;
}
template <int SPARSE, bool STATS, bool TSM>
static Kernel newton_kernel(bool resident, const Geom& g, bool share) {
  if constexpr (!STATS)
    if (g.parts > 1) {
      if constexpr (SPARSE != 0)
        if (share) return newton_kernel<2, STATS, TSM, true>(resident, g.j16);
      return newton_kernel<SPARSE, STATS, TSM, true>(resident, g.j16);
    }
  return newton_kernel<SPARSE, STATS, TSM, false>(resident, g.j16);
}
template <int SPARSE, bool STATS>
static Kernel newton_kernel(bool resident, const Geom& g, bool share) {
  if constexpr (SPARSE != 0)
    if (!g.tsm) return newton_kernel<SPARSE, STATS, false>(resident, g, share);
  return newton_kernel<SPARSE, STATS, true>(resident, g, share);
}

__global__ void start_counters(int* nsolving, int* work_counter, int nworld) {
  chain_wait();
  chain_release();
  if (nsolving) *nsolving = nworld;
  if (work_counter) *work_counter = 0;
}

// A world's solve time grows with its row count, so worlds are taken by descending row
// count: the long solves start first and the launch ends with short ones instead of a few
// stragglers.  One CTA sorts the worlds into 64 classes of row count (counting sort through
// shared memory); the order inside a class depends on atomics and is irrelevant: every
// world is solved independently of which warp takes it.
#define IMN_ORDER_CLASSES 64
__global__ void __launch_bounds__(1024) order_worlds_kernel(const int* __restrict__ nefc, int njmax, int nworld,
                                                            int* __restrict__ order, int* nsolving, int* work_counter) {
  __shared__ int count[IMN_ORDER_CLASSES], start[IMN_ORDER_CLASSES];
  const int tid = threadIdx.x;
  if (tid < IMN_ORDER_CLASSES) count[tid] = 0;
  chain_wait();
  chain_release();
  if (tid == 0 && nsolving) *nsolving = nworld;
  if (tid == 0 && work_counter) *work_counter = 0;
  __syncthreads();
  // class 0 holds the largest row counts
  auto cls = [&](int n) {
    n = min(max(n, 0), njmax);
    return (int)(((long long)(njmax - n) * IMN_ORDER_CLASSES) / (njmax + 1));
  };
  for (int w = tid; w < nworld; w += blockDim.x) atomicAdd(&count[cls(nefc[w])], 1);
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    for (int c = 0; c < IMN_ORDER_CLASSES; ++c) start[c] = run, run += count[c];
  }
  __syncthreads();
  for (int w = tid; w < nworld; w += blockDim.x) order[atomicAdd(&start[cls(nefc[w])], 1)] = w;
}

// Resident-J budget per world: keep at least 4 worlds per SM.
static const int kResidentBudget = kMaxSmem / 4;

static int validate(const ImnModel* m, const ImnData* d, const ImnCtx* cx) {
  if (!m || !d || !cx) return set_error("imn_solve: NULL struct"), IMN_ERR_NULL;
  if (d->nworld < 0 || d->njmax < 0) return set_error("imn_solve: negative extent"), IMN_ERR_SHAPE;
  if (d->njmax >= (1 << 15)) return set_error("imn_solve: njmax %d exceeds 15-bit row indices", d->njmax), IMN_ERR_LIMIT;
  if (m->nv <= 0 || m->nv > 79 || m->nv_pad % 16 != 0 || m->nv_pad > 80 || m->nv_pad <= m->nv)
    return set_error("imn_solve: nv %d / nv_pad %d outside the fused path (0 < nv <= 79, nv_pad %% 16 == 0, nv < nv_pad <= 80)",
                     m->nv, m->nv_pad),
           IMN_ERR_UNSUPPORTED;
  if (m->iterations <= 0) return set_error("imn_solve: iterations must be positive"), IMN_ERR_UNSUPPORTED;
  if (m->n_tolerance <= 0 || m->n_ls_tolerance <= 0 || m->n_meaninertia <= 0)
    return set_error("imn_solve: empty option array"), IMN_ERR_SHAPE;
  const void* need[] = {m->opt_tolerance, m->opt_ls_tolerance, m->stat_meaninertia, m->M_rowadr,
                        m->M_rownnz, m->M_colind, m->M_mulm_lanes, d->nefc, d->ne, d->nf, d->qacc_smooth, d->qacc_warmstart,
                        d->qfrc_smooth, d->efc_J, d->efc_D, d->efc_aref, d->efc_frictionloss, d->M, d->qacc,
                        d->qfrc_constraint, d->efc_Ma, d->efc_force, d->efc_state, d->solver_niter,
                        d->overflow};
  for (const void* p : need)
    if (!p) return set_error("imn_solve: a required Model/Data pointer is NULL"), IMN_ERR_NULL;
  if (d->dof_ld < m->nv || d->J_ld_row < m->nv || d->efc_ld < d->njmax || d->M_ld < m->nM ||
      (!d->J_world_offset && d->J_ld_world < (int64_t)d->njmax * d->J_ld_row) ||
      (d->J_world_offset && d->J_elems < 0))
    return set_error("imn_solve: a stride is smaller than its extent"), IMN_ERR_SHAPE;
  if (d->J_ld_row > 4 * (int64_t)m->nv + 64)
    return set_error("imn_solve: efc.J row stride %lld is far larger than nv %d", (long long)d->J_ld_row, m->nv),
           IMN_ERR_SHAPE;
  if (m->n_mulm_batches <= 0) return set_error("imn_solve: empty M_mulm_lanes program"), IMN_ERR_SHAPE;
  if (m->nM >= (1 << 16)) return set_error("imn_solve: nM exceeds 16-bit indices"), IMN_ERR_LIMIT;
  if (cx->grad && cx->grad_ld < m->nv) return set_error("imn_solve: ctx.grad stride < nv"), IMN_ERR_SHAPE;
  if (cx->sparse_plan) {
    const ImnSparsePlan* sp = cx->sparse_plan;
    if (sp->nv != m->nv || sp->nv_pad != m->nv_pad || sp->nfac <= 0 || sp->nslots != sp->nfac + sp->nv ||
        2 * sp->nfac + sp->nv >= sp->nv_pad * sp->nv_pad - 1 || sp->nlevels <= 0)
      return set_error("imn_solve: sparse plan does not match the model"), IMN_ERR_SHAPE;
    if (!cx->hfactor) return set_error("imn_solve: the sparse path needs ctx.hfactor (violation counter)"), IMN_ERR_NULL;
    if (!sp->lvl_ptr || !sp->lvl_team || !sp->ent_slot || !sp->ent_col || !sp->run_ptr || !sp->run_ab ||
        !sp->run_kl || !sp->orig || !sp->b_lvl || !sp->b_slot || !sp->b_src || !sp->b_dst || !sp->pair ||
        !sp->f_lvl || !sp->f_row || !sp->row_start || !sp->rk_ptr || !sp->rk || !sp->pmask || !sp->s_a ||
        !sp->s_b || !sp->s_m || !sp->fstep || !sp->bstep || sp->nfstep <= 0 || sp->nbsweep < 0)
      return set_error("imn_solve: a sparse plan table is NULL"), IMN_ERR_NULL;
  }
  return IMN_OK;
}

// Worlds one SM can have in hand.
static int worlds_per_sm(const Geom& g, int most) {
  const int n = (kMaxSmem - 4 * g.tab) / (4 * g.total);
  return n < most ? n : most;
}

// J resident in shared memory or streamed through the 32-row tile.  Resident J is
// read once from HBM; a streamed J is re-read from L2 in every stage but leaves room
// for more worlds per SM.  Stream when it holds at least 1.6x the worlds.  us per solve of a batch that
// fills the GPU, resident / streamed (worlds per SM): 34 dofs x 64 rows 563 / 709 (14 / 12), dense factor 940 /
// 1007 (13 / 12); 27 x 128 dense 476 / 536 (8 / 12); 35 x 128 dense 750 / 829 (8 / 12: 1.5x); 64 x 64
// dense 1831 / 1779 (5 / 5); 48 x 96 dense 1381 / 1201 (5 / 10); 56 x 128 rows 1423 / 1115 (4 / 9); 64 x 128
// dense 3650 / 2487 (3 / 5: 1.7x); 35 x 250 4600 / 2334 (4 / 12).  The ratio is that of full SMs; batches of up to 4
// worlds per SM fit either way and differ by a few per cent: 56 x 128, 16 worlds 250 / 263, 592 worlds
// 317 / 340; 35 x 250 240 / 232, 249 / 254.
//
// Warps per world: a world's rows, dofs and Hessian entries can be dealt to several warps; the line
// search, the row lists and most factors cannot, and each stage costs a barrier.  How much of a solve can be dealt
// follows J: streamed, its rows come from L2, and more warps hide that (one world per SM, one to four warps, us: 56 dofs
// 414 / 314 / 289 / 276, 35 x 250 264 / 223 / 193 / 187, 64 x 512 879 / 594 / 519 / 494); resident, the chains are most of
// it (34 dofs 135 / 126 / 120 / 120, 40 x 100 dense 248 / 211 / 203 / 204, 60 x 64 dense 444 / 384 / 371 / 355).
// With n worlds in hand a solve takes kTeamTime + n kCrowded of one warp's time alone.  A launch lasts as many solves as
// its SMs take worlds one after the other: share / n if worlds filled in for one another, `rounds` if a started round
// took as long as a full one.  Worlds go by falling row counts, so a last round is short: a tenth of `rounds`, nothing
// where J is resident.  The choice is the least product.  Over 289 batches (17 models, 1 to 28 worlds per SM) the mean distance from the best
// of the four is 0.4 %, 2.1 % by the largest (worlds in hand) x sqrt(team), and none is more than 3.3 % behind
// that; 1.2 % with one column of times for every J and half of `rounds` (56 dofs, 7 worlds per SM, 473 us where two warps
// take 429; 35 x 512, 28 per SM 1758 / 1566).  What is left are batches of one world more than teams of two
// hold: where worlds differ in rows two warps are ahead (35 x 96 dense, 9 per SM 308 against 345 us), where all have
// the same count one is (27 x 32 dense 131 against 150), and the rule takes two.
static const float kTeamTime[2][5] = {{0.0f, 1.0f, 0.72f, 0.58f, 0.55f}, {0.0f, 1.0f, 0.84f, 0.81f, 0.74f}};  // [J resident]
static const float kCrowded[2] = {0.03f, 0.01f}, kRounds[2] = {0.1f, 0.0f};
static const int kMaxParts = 4;

static int plan_launch(const ImnModel* m, const ImnData* d, const ImnSparsePlan* sp, bool stats, Geom* g, bool* resident,
                       int* grid) {
  const Geom gr = make_geom(*m, *d, true, sp, 1);
  const Geom gs = make_geom(*m, *d, false, sp, 1);
  const int nr = worlds_per_sm(gr, kResidentWarps), ns = worlds_per_sm(gs, kStreamedWarps);
  const bool fits = gr.total * 4 <= kResidentBudget && nr >= 1;
  *resident = fits && 10 * ns < 16 * nr;
  *g = *resident ? gr : gs;
  if (!*resident && ns < 1)
    return set_error("imn_solve: njmax %d needs %d bytes of shared memory per world (max %d)", d->njmax, 4 * (gs.total + gs.tab),
                     kMaxSmem),
           IMN_ERR_LIMIT;
  // one CTA per SM; a batch that does not fill the GPU is spread over all SMs
  const int sms = sm_count(), share = max((d->nworld + sms - 1) / sms, 1);
  g->warps = min(share, *resident ? nr : ns);
  const auto time = [&](const Geom& q) {
    const float n = (float)q.warps, rounds = (float)((share + q.warps - 1) / q.warps);
    const float turns = (float)share / n;
    return (turns + kRounds[*resident] * (rounds - turns)) * (kTeamTime[*resident][q.parts] + n * kCrowded[*resident]);
  };
  for (int parts = 2; parts <= kMaxParts && !stats; ++parts) {  // the counting kernels know no teams
    Geom team = make_geom(*m, *d, *resident, sp, parts);
    team.warps = min(share, worlds_per_sm(team, (*resident ? kResidentWarps : kStreamedWarps) / parts));
    if (team.warps > 0 && time(team) < time(*g)) *g = team;
  }
  const int need = (d->nworld + g->warps - 1) / g->warps;
  *grid = need < sms ? need : sms;
  return IMN_OK;
}

}  // namespace imn

#ifdef IMN_PROFILE
extern "C" int imn_debug_profile(unsigned long long* out, int reset) {
  cudaMemcpyFromSymbol(out, imn::g_prof, sizeof(unsigned long long) * 24);
  if (reset) {
    unsigned long long z[24] = {0};
    cudaMemcpyToSymbol(imn::g_prof, z, sizeof z);
  }
  return 0;
}
#endif

extern "C" int imn_set_copy_wait_limit(int32_t polls, int32_t withhold_copies) {
  if (polls <= 0) return imn::set_error("imn_set_copy_wait_limit: polls must be positive"), IMN_ERR_SHAPE;
  imn::g_wait_polls = polls;
  imn::g_withhold_copies = withhold_copies & 3;
  return IMN_OK;
}

extern "C" int imn_launch_info(const ImnModel* m, const ImnData* d, const ImnCtx* cx, ImnLaunchInfo* out) {
  if (!out) return imn::set_error("imn_launch_info: NULL out"), IMN_ERR_NULL;
  int rc = imn::validate(m, d, cx);
  if (rc) return rc;
  imn::Geom g;
  bool res;
  int grid = 0;
  rc = imn::plan_launch(m, d, cx->sparse_plan, cx->stats != nullptr, &g, &res, &grid);
  if (rc) return rc;
  out->world_threads = g.bd;
  out->worlds_per_cta = g.warps;
  out->smem_bytes = 4 * (g.tab + g.warps * g.total);
  out->j_resident = res ? 1 : 0;
  out->grid = grid;
  return IMN_OK;
}

extern "C" int imn_solve(const ImnModel* m, const ImnData* d, const ImnCtx* cx, void* stream_) {
  int rc = imn::validate(m, d, cx);
  if (rc) return rc;
  cudaStream_t stream = (cudaStream_t)stream_;
  if (d->nworld == 0) return IMN_OK;
  imn::Geom g;
  bool res;
  int grid = 0;
  rc = imn::plan_launch(m, d, cx->sparse_plan, cx->stats != nullptr, &g, &res, &grid);
  if (rc) return rc;
  const int bytes = 4 * (g.tab + g.warps * g.total);
  const bool sparse = cx->sparse_plan != nullptr, stats = cx->stats != nullptr, share = sparse && cx->sparse_plan->pairs;
  const ImnSparsePlan sp = sparse ? *cx->sparse_plan : ImnSparsePlan{};
  const imn::Kernel kern = sparse ? (stats ? imn::newton_kernel<1, true>(res, g, share) : imn::newton_kernel<1, false>(res, g, share))
                                  : (stats ? imn::newton_kernel<0, true>(res, g, share) : imn::newton_kernel<0, false>(res, g, share));
  {
    const cudaError_t e = imn::allow_shared(kern, bytes, true);
    if (e != cudaSuccess)
      return imn::set_error("imn_solve: cudaFuncSetAttribute: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  }
  cudaError_t e = cudaSuccess;
  if (cx->world_order)
    e = imn::launch_chained(imn::order_worlds_kernel, 1, 1024, 0, stream, d->nefc, d->njmax, d->nworld, cx->world_order,
                            cx->nsolving, cx->work_counter);
  else if (cx->nsolving || cx->work_counter)
    e = imn::launch_chained(imn::start_counters, 1, 1, 0, stream, cx->nsolving, cx->work_counter, d->nworld);
  g.early = cx->world_order || cx->nsolving || cx->work_counter;
  if (e == cudaSuccess) e = imn::launch_chained(kern, grid, 32 * g.warps * g.parts, bytes, stream, *m, *d, *cx, g, sp);
  if (e != cudaSuccess) return imn::set_error("imn_solve: launch failed: %s", cudaGetErrorString(e)), IMN_ERR_LAUNCH;
  return IMN_OK;
}
