"""The performance cases of the framework: what its users have it do, over the sizes and
options they have it do it with.

A case is a dict of plain values.  ``listed`` names the fixed cases, ``draw`` gives further
ones of the same ranges, ``prepare`` builds what a program holds before the call (inputs from
the seed, model, plans, scratch), ``run`` is one pass through the public entry points,
``work`` the bytes and operations the pass cannot do without and ``tolerance`` how far
another correct implementation may be off.

Kinds of work:

* ``solve``      one constraint solve of a batch (``solve_with_scratch``);
* ``substep``    every stage of a substep that the framework covers, one call after the other:
                 body velocities, subtree centres of mass, M, bias forces, smooth acceleration,
                 constraint solve, implicit-fast integration;
* ``smooth``     the stages before the solve only;
* ``integrate``  the implicit-fast tail after the solve;
* ``retained``   M factored once with a few right-hand sides, then solved again with the
                 factor that was kept;
* ``host``       batches in pinned host memory through ``HostBatchPipeline``.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from instantmimic_b200 import host_batch, mjw_model, synthetic, types
from instantmimic_b200 import mjw_step_optimized as runtime
from instantmimic_b200.mjw_kernels import indexed_factor, tree_fusion, tree_ldl, velocity_fusion

DEVICE = "cuda"


def listed():
    return [
        # one person watching a policy in the viewer: a handful of worlds, the model's authored
        # budget of 4 iterations, every stage called eagerly -- launches and latency only
        dict(name="substep_humanoid_16", kind="substep", model="humanoid", worlds=16, njmax=64, lo=16, hi=64,
             iterations=4, ls=4, sparse=True, rowless=0.1),
        # evaluation batch of the humanoid (1024 worlds, the benchmark's configuration 1)
        _solve("solve_humanoid_1024", "humanoid", 1024, 64, 16, 64),
        # the headline benchmark: one training GPU's worth of humanoids
        _solve("solve_humanoid_8192", "humanoid", 8192, 64, 16, 64),
        # muscle humanoid at its training size (streamed Jacobian, 64-wide logical blocks)
        _solve("solve_snu_4096", "snu", 4096, 128, 24, 128),
        # contact-heavy G1-like robot with that task's own budget; many worlds, many padded rows
        _solve("solve_g1_16384", "g1", 16384, 250, 16, 200, iterations=10, ls=20),
        # odd sizes: one chain with equality and friction-loss rows, airborne worlds, dense factor
        _solve("solve_chain35_rows_1000", "chain35", 1000, 96, 20, 90, sparse=False, ne=6, nf=5, rowless=0.1),
        # the isolated sweep's small and large ends: rows that couple two chains (dense factor)
        _solve("solve_limb27_32_16384", "limb27", 16384, 32, 32, 32, sparse=False, rows="generic"),
        _solve("solve_limb64_512_4096", "limb64", 4096, 512, 512, 512, sparse=False, rows="generic"),
        # the stages before the solve at training size
        dict(name="smooth_humanoid_8192", kind="smooth", model="humanoid", worlds=8192),
        # the integrator's tail; motors on ball joints carry three-entry moment rows
        dict(name="integrate_humanoid_8192", kind="integrate", model="humanoid", worlds=8192, ball_rows=True),
        # factor kept between solves (several right-hand sides, some worlds switched off)
        dict(name="retained_humanoid_4096", kind="retained", model="humanoid", worlds=4096, rhs=3, again=1),
        # replay of recorded solver states from host memory, byte column indices
        dict(name="host_humanoid_4096", kind="host", model="humanoid", worlds=4096, njmax=64, lo=16, hi=64,
             iterations=50, ls=50, sparse=True, rowless=0.0, mode="sparse8"),
    ]


def _solve(name, model, worlds, njmax, lo, hi, *, iterations=50, ls=50, sparse=True, rows="contacts", ne=0, nf=0,
           rowless=0.0):
    return dict(name=name, kind="solve", model=model, worlds=worlds, njmax=njmax, lo=lo, hi=hi, iterations=iterations,
                ls=ls, sparse=sparse, rows=rows, ne=ne, nf=nf, rowless=rowless)


# Row storage of the three named models: njmax, fewest and most live rows of a world.
_ROWS = {"humanoid": (64, 16, 64), "snu": (128, 24, 128), "g1": (250, 16, 200)}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["solve", "substep", "smooth", "integrate", "retained", "host"], [6, 1, 2, 1, 1, 1])[0]
    model = rng.choice(["humanoid", "snu", "g1"])
    budget = dict(zip(("iterations", "ls"), rng.choice([(4, 4), (10, 20), (50, 50)])))
    if kind == "smooth":
        return dict(kind=kind, model=model, worlds=_log(rng, 16, 32768))
    if kind == "integrate":
        return dict(kind=kind, model=model, worlds=_log(rng, 16, 32768), ball_rows=rng.random() < 0.5)
    if kind == "retained":
        return dict(kind=kind, model=model, worlds=_log(rng, 16, 8192), rhs=rng.randint(1, 6), again=rng.randint(1, 4))
    if kind in ("substep", "host"):
        njmax, lo, hi = _ROWS[model]
        top = 8192 if kind == "substep" else 4096
        case = dict(kind=kind, model=model, worlds=_log(rng, 16, top), njmax=njmax, lo=lo, hi=hi, **budget, sparse=True,
                    rowless=rng.choice([0.0, 0.1]))
        if kind == "host":
            case["mode"] = rng.choice(["sparse8", "sparse", "compact", "whole"])
        return case
    if rng.random() < 0.5:  # a named model
        njmax, lo, hi = _ROWS[model]
        case = _solve(None, model, _log(rng, 16, 16384), njmax, lo, hi, **budget, rowless=rng.choice([0.0, 0.1]))
    elif rng.random() < 0.4:  # one chain with equality and friction-loss rows
        nv, njmax = rng.randint(13, 79), rng.randint(24, 160)
        lo = rng.randint(16, njmax)
        case = _solve(None, "chain%d" % nv, _log(rng, 16, 8192), njmax, lo, rng.randint(lo, njmax), **budget, sparse=False,
                      ne=rng.randint(0, 8), nf=rng.randint(0, 8), rowless=rng.choice([0.0, 0.1]))
    else:  # a point of the sweep
        nv, nefc = rng.randint(27, 64), _log(rng, 32, 512)
        coupled = rng.random() < 0.7
        case = _solve(None, "limb%d" % nv, _log(rng, 256, 16384), nefc, nefc, nefc, **budget, sparse=not coupled,
                      rows="generic" if coupled else "contacts")
    del case["name"]
    # no dearer than the largest listed case
    nv = _tree(case["model"])[0].size
    per_world = nv * nv * (case["njmax"] + 100)
    case["worlds"] = max(16, min(case["worlds"], 4096 * 64 * 64 * 612 // per_world))
    return case


# ---- models --------------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _tree(name):
    named = {"humanoid": synthetic.humanoid_tree, "snu": synthetic.snu_tree, "g1": synthetic.g1_like_tree}
    if name in named:
        return named[name]()
    return {"limb": synthetic.limb_tree, "chain": synthetic.chain_tree}[name.rstrip("0123456789")](int(name.lstrip("limbchan")))


@functools.lru_cache(maxsize=None)
def _model(name, iterations=50, ls=50):
    """(host, device) model: a program has one for as long as it runs."""
    parent, body = _tree(name)
    m = mjw_model.put_model(parent, body_of_dof=body, iterations=iterations, ls_iterations=ls, tolerance=1e-8)
    rng = np.random.default_rng(7)
    m.dof_armature = rng.uniform(0.1, 0.5, (1, m.nv)).astype(np.float32)
    m.dof_damping = rng.uniform(0.0, 1.0, m.nv).astype(np.float32)
    # one position servo per dof behind the free joint
    m.nu = max(m.nv - 6, 1)
    m.actuator_gaintype = np.zeros(m.nu, np.int32)
    m.actuator_biastype = np.full(m.nu, int(types.BiasType.AFFINE), np.int32)
    m.actuator_dyntype = np.zeros(m.nu, np.int32)
    m.actuator_gainprm = np.zeros((m.nu, 10), np.float32)
    m.actuator_biasprm = np.zeros((m.nu, 10), np.float32)
    m.actuator_biasprm[:, 2] = -rng.uniform(1.0, 20.0, m.nu)
    return m, mjw_model.to_device(m, DEVICE)


@functools.lru_cache(maxsize=None)
def _plans(name):
    """The per-model plans of the stages around the solve, made once per program."""
    _, md = _model(name)
    return tree_ldl.create_tree_factor_solve_scratch(md, DEVICE), tree_fusion.create_tree_reduction_scratch(md)


# ---- inputs --------------------------------------------------------------------------------


class _Draws:
    """Random device tensors from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(shape, device=DEVICE, generator=self.g)

    def uniform(self, lo, hi, *shape):
        return torch.rand(shape, device=DEVICE, generator=self.g) * (hi - lo) + lo

    def integers(self, lo, hi, *shape):  # hi included
        return torch.randint(lo, hi + 1, shape, device=DEVICE, generator=self.g)


def _masses(m, W, r):
    """(W, nM) stored entries and the dense (W, nv, nv) of M = L^T D L on the tree's pattern."""
    rows = torch.from_numpy(np.asarray(m.M_hinit_i)).long().to(DEVICE)
    cols = torch.from_numpy(np.asarray(m.M_colind)).long().to(DEVICE)
    L = torch.zeros(W, m.nv, m.nv, device=DEVICE)
    L[:, rows, cols] = 0.3 * r.normal(W, m.nM)
    L.diagonal(dim1=1, dim2=2).fill_(1.0)
    scaled = L * r.uniform(0.5, 2.0, W, m.nv, 1).sqrt()
    dense = scaled.transpose(1, 2) @ scaled
    return dense[:, rows, cols].contiguous(), dense


def _data(m, W, njmax):
    """Empty device-side Data."""
    f = lambda *s: torch.zeros(s, device=DEVICE)  # noqa: E731
    i = lambda *s: torch.zeros(s, dtype=torch.int32, device=DEVICE)  # noqa: E731
    return mjw_model.Data(
        nworld=W, njmax=njmax, nefc=i(W), ne=i(W), nf=i(W), qacc_smooth=f(W, m.nv), qacc_warmstart=f(W, m.nv),
        qfrc_smooth=f(W, m.nv), M=f(W, m.nM), qacc=f(W, m.nv), qfrc_constraint=f(W, m.nv), solver_niter=i(W), overflow=i(W),
        efc=mjw_model.Constraint(J=f(W, njmax, m.nv), D=f(W, njmax), aref=f(W, njmax), frictionloss=f(W, njmax),
                                 force=f(W, njmax), state=i(W, njmax), Ma=f(W, m.nv)))


def _rows(m, d, case, r):
    """Constraint rows: pyramidal contact quadruples on one ancestor chain with joint limits at the
    end of a world's rows, or rows on one or two chains; equality and friction-loss rows first."""
    W, R, nv = d.nworld, d.njmax, m.nv
    ne, nf = case.get("ne", 0), case.get("nf", 0)
    nefc = r.integers(max(case["lo"], ne + nf), max(case["hi"], ne + nf), W)
    nefc = torch.where(r.uniform(0, 1, W) < case["rowless"], torch.zeros_like(nefc), nefc)
    chains = torch.from_numpy(synthetic.ancestor_masks(np.asarray(m.dof_parentid)).astype(np.float32)).to(DEVICE)
    J, worlds = d.efc.J, torch.arange(W, device=DEVICE)
    if case.get("rows") == "generic":
        mask = chains[r.integers(0, nv - 1, W, R)]
        two = (r.uniform(0, 1, W, R, 1) < 0.5).float()
        mask = torch.maximum(mask, chains[r.integers(0, nv - 1, W, R)] * two)
        torch.mul(r.normal(W, R, nv), mask, out=J)
    else:
        n = (R + 3) // 4
        mask = chains[r.integers(0, nv - 1, W, n)]
        jn, jt1, jt2 = (r.normal(W, n, nv) * mask for _ in range(3))
        mu = r.uniform(0.5, 1.0, W, n, 1)
        J.copy_(torch.stack([jn + mu * jt1, jn - mu * jt1, jn + mu * jt2, jn - mu * jt2], 2).view(W, 4 * n, nv)[:, :R])
        limits = r.integers(0, 6, W)
        for k in range(6):
            at = nefc - 1 - k
            w = worlds[(k < limits) & (at >= ne + nf)]
            J[w, at[w]] = 0.0
            J[w, at[w], r.integers(min(6, nv - 1), nv - 1, W)[w]] = (2 * r.integers(0, 1, W)[w] - 1).float()
    if ne:
        J[:, :ne] = r.normal(W, ne, nv) * chains[r.integers(0, nv - 1, W, ne)]
    if nf:
        J[:, ne:ne + nf] = torch.nn.functional.one_hot(r.integers(0, nv - 1, W, nf), nv).float()
        d.efc.frictionloss[:, ne:ne + nf] = r.uniform(0.1, 1.0, W, nf)
    d.efc.D.copy_(r.uniform(0.1, 10.0, W, R))
    d.efc.aref.copy_(r.normal(W, R))
    d.nefc.copy_(nefc)
    d.ne.copy_((nefc > 0) * ne)
    d.nf.copy_((nefc > 0) * nf)


def _solver_state(m, case, r):
    W = case["worlds"]
    d = _data(m, W, case["njmax"])
    _rows(m, d, case, r)
    M, dense = _masses(m, W, r)
    d.M.copy_(M)
    d.qacc_smooth.copy_(r.normal(W, m.nv))
    d.qfrc_smooth.copy_((dense @ d.qacc_smooth[:, :, None])[:, :, 0])
    d.qacc_warmstart.copy_(d.qacc_smooth + 0.1 * r.normal(W, m.nv))
    return d


def _smooth_state(m, d, r):
    """Physical per-body inertias about a common origin, unit-scale motion axes, velocities."""
    W, nv, nb = d.nworld, m.nv, int(np.asarray(m.body_parentid).size)
    mass, com = r.uniform(0.5, 5.0, W, nb, 1), r.uniform(-0.3, 0.3, W, nb, 3)
    a = 0.1 * r.normal(W, nb, 3, 3)
    eye = torch.eye(3, device=DEVICE)
    c2 = (com * com).sum(-1)[..., None, None] * eye - com[..., :, None] * com[..., None, :]
    full = a @ a.transpose(-1, -2) + 0.02 * eye + mass[..., None] * c2
    six = torch.stack([full[..., i, j] for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))], -1)
    d.cinert = torch.cat([six, mass * com, mass], -1).contiguous()
    d.cinert[:, 0] = 0.0
    d.cdof, d.qvel = 0.6 * r.normal(W, nv, 6), 0.5 * r.normal(W, nv)
    z = lambda *s: torch.zeros(s, device=DEVICE)  # noqa: E731
    d.crb, d.cvel, d.cacc, d.cfrc_int = z(W, nb, 10), z(W, nb, 6), z(W, nb, 6), z(W, nb, 6)
    d.cdof_dot, d.qfrc_bias = z(W, nv, 6), z(W, nv)
    d.body_moments, d.subtree_com = r.uniform(0.1, 1.0, W, nb, 3), z(W, nb, 3)
    d.qfrc_smooth.copy_(10.0 * r.normal(W, nv))


def _actuated_state(m, d, r, ball_rows):
    """Joint coordinates, controls and the actuators' moment rows.  A motor on one axis of a ball
    joint has a row over the joint's three dofs (MuJoCo's transmission stores all three) when
    ``ball_rows``, else every row holds one dof."""
    W, nu, first = d.nworld, m.nu, m.nv - m.nu
    ball = np.zeros(m.nv, bool)
    for t, a in zip(np.asarray(m.jnt_type), np.asarray(m.jnt_dofadr)):
        if ball_rows and t == int(types.JointType.BALL):
            ball[a:a + 3] = True
    nnz, cols, vals, start = [], [], [], {}
    for dof in range(first, m.nv):
        if ball[dof] and dof - 1 in start and dof - start[dof - 1] < 3:
            start[dof] = start[dof - 1]
        else:
            start[dof] = dof
        row = range(start[dof], start[dof] + 3) if ball[dof] else [dof]
        nnz.append(len(row))
        cols += row
        vals += [float(c == dof) for c in row]
    put = lambda v, t: torch.tensor(v, dtype=t, device=DEVICE).repeat(W, 1)  # noqa: E731
    d.moment_rownnz = put(nnz, torch.int32)
    d.moment_rowadr = put(np.concatenate(([0], np.cumsum(nnz)[:-1])).tolist(), torch.int32)
    d.moment_colind, d.actuator_moment = put(cols, torch.int32), put(vals, torch.float32)
    d.ctrl = r.uniform(-1, 1, W, nu)
    d.qpos = 0.1 * r.normal(W, m.nq)
    for t, p in zip(np.asarray(m.jnt_type), np.asarray(m.jnt_qposadr)):
        p = int(p) + (3 if t == int(types.JointType.FREE) else 0)
        if t in (int(types.JointType.FREE), int(types.JointType.BALL)):
            d.qpos[:, p] = 1.0
            d.qpos[:, p:p + 4] /= d.qpos[:, p:p + 4].norm(dim=1, keepdim=True)
    d.qvel = 0.5 * r.normal(W, m.nv)
    d.time = torch.zeros(W, device=DEVICE)


def _scratch(m, md, d, case):
    sc = runtime.make_optimized_fwd_position_scratch(md, d, DEVICE, include_optimized_kernel_scratch=False)
    if case.get("sparse"):
        groups = [[b] for b in range(1, len(np.asarray(m.body_dofadr)))]
        runtime.refresh_sparse_hessian(md, d, sc, groups, DEVICE)
    return sc


@functools.lru_cache(maxsize=1)
def _pipeline(model, worlds, njmax, iterations, ls, mode):
    """The host pipeline of a program that replays batches of one shape."""
    m, md = _model(model, iterations, ls)
    groups = [[b] for b in range(1, len(np.asarray(m.body_dofadr)))]
    return host_batch.HostBatchPipeline(md, mjw_model.make_data(m, worlds, njmax), DEVICE, slots=3, sparse_groups=groups,
                                        mode=mode)


def prepare(case, seed):
    r = _Draws(seed)
    m, md = _model(case["model"], case.get("iterations", 50), case.get("ls", 50))
    W, kind = case["worlds"], case["kind"]
    if kind == "host":
        batches = []
        for k in range(3):
            d = mjw_model.to_host(_solver_state(m, case, r))
            batches.append(host_batch.pin_batch(d, chunk=128))
        pipe = _pipeline(case["model"], W, case["njmax"], case["iterations"], case["ls"], case["mode"])
        for slot in pipe.slots:  # rows at and beyond a world's count keep what was there before
            slot["dd"].efc.force.zero_()
            slot["dd"].efc.state.zero_()
        return dict(kind=kind, pipe=pipe, batches=batches)
    if kind == "retained":
        d = _data(m, W, 1)
        d.M.copy_(_masses(m, W, r)[0])
        plan = indexed_factor.create_blocked_dense_factor_solve_scratch(md, d, DEVICE)
        y, y2 = r.normal(W, m.nv, case["rhs"]), r.normal(W, m.nv, case["again"])
        return dict(kind=kind, plan=plan, M=d.M, y=y, y2=y2, x=torch.zeros_like(y), x2=torch.zeros_like(y2),
                    active=(r.uniform(0, 1, W) < 0.9).int(), rhs=case["rhs"], again=case["again"])
    if kind == "solve":
        d = _solver_state(m, case, r)
        return dict(kind=kind, m=md, d=d, sc=_scratch(m, md, d, case))
    d = _solver_state(m, case, r) if kind == "substep" else _data(m, W, 1)
    if kind in ("substep", "smooth"):
        _smooth_state(m, d, r)
    if kind in ("substep", "integrate"):
        _actuated_state(m, d, r, case.get("ball_rows", True))
    if kind == "integrate":
        d.M.copy_(_masses(m, W, r)[0])
        d.efc.Ma.copy_(r.normal(W, m.nv))
    sc = _scratch(m, md, d, case)
    sc.tree_factor_solve, sc.tree_reduction = _plans(case["model"])
    runtime.attach_implicit_scratch(md, d, sc, DEVICE)
    return dict(kind=kind, m=md, d=d, sc=sc)


# ---- one pass ------------------------------------------------------------------------------


def _smooth(m, d, sc):
    tree = sc.tree_reduction
    velocity_fusion.com_vel(m, d, tree)
    d.subtree_com.copy_(d.body_moments)  # the position stage writes the bodies' own moments every step
    tree_fusion.subtree_com_accumulate(m, d, tree)
    tree_fusion.crb(m, d, tree)
    tree_fusion.rne(m, d, tree)
    runtime.fwd_acceleration_solve(m, d, sc)
    return dict(cvel=d.cvel, cdof_dot=d.cdof_dot, subtree_com=d.subtree_com, crb=d.crb, M=d.M, cacc=d.cacc,
                cfrc_int=d.cfrc_int, qfrc_bias=d.qfrc_bias, qacc_smooth=d.qacc_smooth)


def _constraints(m, d, sc):
    runtime.solve_with_scratch(m, d, sc, use_optimized_kernel=True)
    return dict(qacc=d.qacc, qfrc_constraint=d.qfrc_constraint, Ma=d.efc.Ma, force=d.efc.force, state=d.efc.state,
                niter=d.solver_niter, overflow=d.overflow)


def _integrate(m, d, sc):
    runtime.implicitfast_integrate(m, d, sc)
    return dict(A=sc.implicit_qderiv, x=sc.implicit_qacc, qvel=d.qvel, qpos=d.qpos, time=d.time)


def run(s):
    kind = s["kind"]
    if kind == "host":
        for k, batch in enumerate(s["batches"]):
            s["pipe"].submit(k, batch)
        return [dict(s["pipe"].result(k)) for k in range(3)]
    if kind == "retained":
        plan = s["plan"]
        indexed_factor.factor_multi_solve(plan, s["M"], s["y"], s["active"], plan.U, s["x"], s["rhs"])
        indexed_factor.multi_solve(plan, plan.U, s["y2"], s["active"], s["x2"], s["again"])
        return dict(x=s["x"], x2=s["x2"], U=plan.U)
    args = s["m"], s["d"], s["sc"]
    out = {}
    if kind in ("substep", "smooth"):
        out.update(_smooth(*args))
    if kind in ("substep", "solve"):
        out.update(_constraints(*args))
    if kind in ("substep", "integrate"):
        out.update(_integrate(*args))
    return out


# ---- what a pass cannot do without ---------------------------------------------------------


def work(case):
    m = _model(case["model"], case.get("iterations", 50), case.get("ls", 50))[0]
    W, nv, nM, kind = case["worlds"], m.nv, m.nM, case["kind"]
    nb, nu = int(np.asarray(m.body_parentid).size), m.nu
    floats = flops = 0.0
    if kind in ("solve", "substep", "host"):
        rows = 0.5 * (case["lo"] + case["hi"]) * (1.0 - case["rowless"])
        # J, three row vectors, M, three dof vectors, counts; acceleration, forces, row states
        one = rows * nv + 3 * rows + nM + 3 * nv + 3 + 3 * nv + 2 * rows + 2
        # first residual, gradient and Hessian over half of the rows, one factor, one iteration
        ops = 2 * rows * nv * 3 + 4 * nM * 2 + 0.5 * rows * nv * (nv + 1) + nv**3 / 3 + 2 * nv * nv + 60 * rows
        floats += one * (3 if kind == "host" else 1)
        flops += ops * (3 if kind == "host" else 1)
    if kind in ("smooth", "substep"):
        # com_vel, subtree sums, crb with M, rne, acceleration: inputs once, results once
        floats += (nv + 6 * nv) + 10 * nb + 3 * nb + nv + (6 * nb + 6 * nv) + 3 * nb + 10 * nb + nM + 12 * nb + nv + nv
        flops += 60 * nv + 6 * nb + 20 * nb + 11 * nM + 200 * nb + 3 * nM * 6
    if kind in ("integrate", "substep"):
        nq, nnz = m.nq, nu * (3 if case.get("ball_rows", True) and case["model"] != "g1" else 1)
        floats += nM + nv + nu * 3 + 2 * nnz + nv + nq + 1 + nM + nv + nv + nq + 1
        flops += 2 * nM + 6 * nnz + 3 * nM * 6 + 40 * nq
    if kind == "retained":
        pad = (nv + 15) // 16 * 16
        k = case["rhs"] + case["again"]
        floats += 0.9 * (nM + nv * k + pad * pad + nv * k)
        flops += 0.9 * (nv**3 / 3 + 2 * nv * nv * k)
    return {"bytes": 4.0 * W * floats, "flops": float(W * flops)}


def tolerance(case):
    """The solve is 32-bit arithmetic inside an iteration that stops at a threshold: a world may stop
    one step apart and a row at its switching point may take either state.  The other stages are
    short 32-bit sums; solutions with M pick up its condition number."""
    if case["kind"] in ("solve", "substep", "host"):
        return {"rel": 1e-4, "max": 0.02, "differ": 2e-3}
    return {"rel": 1e-5, "max": 1e-3}
