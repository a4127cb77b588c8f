"""The implicit-fast integrator's tail: A = M - h qDeriv (joint damping + actuator-centric
actuation term), (A) x = efc.Ma, advance.  CPU: the oracle against float64 numpy
(dense algebra, rotation by the axis-angle formula).  GPU: the CUDA kernels against the
oracle -- A bit for bit, the advanced state within 2e-6 (sinf / cosf differ in the last
place between libm and the GPU), the solved acceleration against a float64 dense solve
with the tolerance the reference uses for its M-side solves (2e-4 relative)."""

import copy

import numpy as np
import pytest

from instantmimic_b200 import mjw_model, synthetic, types

ADVANCE_TOL = 2e-6
SOLVE_RTOL = 2e-4


def _problem(worlds=70, nu=20, seed=3, damping=True, single=False):
    rng = np.random.default_rng(seed)
    m, d, Mdense = synthetic.make_workload("humanoid", worlds, seed=seed)
    m.dof_damping = rng.uniform(0.0, 2.0, m.nv).astype(np.float32) if damping else np.zeros(m.nv, np.float32)
    m.nu = nu
    # moment rows: most actuators act on one dof, some span a dof and a few of its ancestors
    parent = np.asarray(m.dof_parentid)
    chains = [[[] for _ in range(nu)] for _ in range(worlds)]
    for w in range(worlds):
        for a in range(nu):
            want = 1 if single or rng.random() < 0.7 else int(rng.integers(2, 5))
            chain = [int(rng.integers(6, m.nv))]
            while len(chain) < want and parent[chain[-1]] >= 0:
                chain.append(int(parent[chain[-1]]))
            chains[w][a] = sorted(chain)
    nnz = np.array([[len(c) for c in row] for row in chains], np.int32)
    adr = np.zeros((worlds, nu), np.int32)
    if nu:
        adr[:, 1:] = np.cumsum(nnz, axis=1)[:, :-1]
    ld = max(int(nnz.sum(axis=1).max()) if nu else 1, 1)
    colind = np.zeros((worlds, ld), np.int32)
    moment = np.zeros((worlds, ld), np.float32)
    for w in range(worlds):
        for a in range(nu):
            c = chains[w][a]
            colind[w, adr[w, a] : adr[w, a] + len(c)] = c
            moment[w, adr[w, a] : adr[w, a] + len(c)] = rng.normal(size=len(c))
    d.moment_rownnz, d.moment_rowadr, d.moment_colind, d.actuator_moment = nnz, adr, colind, moment
    gain = (-rng.uniform(0.0, 30.0, (worlds, nu)) * (rng.random((worlds, nu)) < 0.8)).astype(np.float32)
    d.qpos = np.zeros((worlds, m.nq), np.float32)
    for j in range(m.njnt):
        p = int(m.jnt_qposadr[j])
        if m.jnt_type[j] == types.JointType.FREE:
            d.qpos[:, p : p + 3] = rng.normal(size=(worlds, 3))
            p += 3
        if m.jnt_type[j] in (types.JointType.FREE, types.JointType.BALL):
            q = rng.normal(size=(worlds, 4))
            d.qpos[:, p : p + 4] = q / np.linalg.norm(q, axis=1, keepdims=True)
        else:
            d.qpos[:, p] = rng.normal(size=worlds)
    d.qvel = rng.normal(0.0, 2.0, (worlds, m.nv)).astype(np.float32)
    d.time = rng.uniform(0, 5, worlds).astype(np.float32)
    d.efc.Ma[:] = rng.normal(size=(worlds, m.nv)).astype(np.float32)
    return m, d, Mdense, gain


def _dense_a(m, d, Mdense, gain):
    """float64 A = M - h (sum_a gain_a mom_a mom_a^T - diag(damping)) restricted to M's pattern."""
    h = float(m.opt.timestep[0])
    W, nv = d.nworld, m.nv
    pattern = np.asarray(m.M_elemid) >= 0
    pattern = pattern | pattern.T
    A = Mdense.astype(np.float64).copy()
    for w in range(W):
        qd = -np.diag(m.dof_damping.astype(np.float64))
        for a in range(m.nu):
            n, s = int(d.moment_rownnz[w, a]), int(d.moment_rowadr[w, a])
            mom = np.zeros(nv)
            mom[d.moment_colind[w, s : s + n]] = d.actuator_moment[w, s : s + n]
            qd += float(gain[w, a]) * np.outer(mom, mom)
        A[w] -= h * qd * pattern
    return A


def _quat_rotate_reference(q, w, h):
    """float64 q (x) exp(h w / 2), normalised."""
    out = np.empty_like(q, dtype=np.float64)
    for k in range(q.shape[0]):
        a = np.linalg.norm(w[k])
        r = np.array([1.0, 0, 0, 0]) if a < 1e-15 else np.concatenate(([np.cos(0.5 * h * a)], np.sin(0.5 * h * a) * w[k] / a))
        p = q[k].astype(np.float64)
        o = np.array([p[0] * r[0] - p[1:] @ r[1:], *(p[0] * r[1:] + r[0] * p[1:] + np.cross(p[1:], r[1:]))])
        out[k] = o / np.linalg.norm(o)
    return out


def test_oracle_matrix_and_advance_against_float64(oracle):
    m, d, Mdense, gain = _problem()
    A = oracle.implicit_matrix(m, d, gain)
    want = _dense_a(m, d, Mdense, gain)
    rows, cols = np.nonzero(np.asarray(m.M_elemid) >= 0)
    got_dense = np.zeros_like(want)
    got_dense[:, rows, cols] = A[:, np.asarray(m.M_elemid)[rows, cols]]
    got_dense[:, cols, rows] = got_dense[:, rows, cols]
    assert np.abs(got_dense - want).max() <= 1e-5 * np.abs(want).max()
    # without actuators and damping A is M itself, bit for bit
    m0, d0, _, _ = _problem(nu=0, damping=False)
    np.testing.assert_array_equal(oracle.implicit_matrix(m0, d0, None), d0.M)
    # advance
    h = float(m.opt.timestep[0])
    d1 = copy.deepcopy(d)
    qacc = np.random.default_rng(9).normal(0, 5, (d.nworld, m.nv)).astype(np.float32)
    oracle.advance(m, d1, qacc)
    v = d.qvel.astype(np.float64) + h * qacc
    assert np.abs(d1.qvel - v).max() < 1e-5
    np.testing.assert_allclose(d1.time, d.time + np.float32(h), rtol=0, atol=1e-6)
    for j in range(m.njnt):
        p, k = int(m.jnt_qposadr[j]), int(m.jnt_dofadr[j])
        if m.jnt_type[j] == types.JointType.FREE:
            assert np.abs(d1.qpos[:, p : p + 3] - (d.qpos[:, p : p + 3] + h * v[:, k : k + 3])).max() < 1e-5
            p, k = p + 3, k + 3
        if m.jnt_type[j] in (types.JointType.FREE, types.JointType.BALL):
            ref = _quat_rotate_reference(d.qpos[:, p : p + 4], v[:, k : k + 3], h)
            assert np.abs(d1.qpos[:, p : p + 4] - ref).max() < 1e-5
            assert np.abs(np.linalg.norm(d1.qpos[:, p : p + 4], axis=1) - 1).max() < 1e-5
        else:
            assert np.abs(d1.qpos[:, p] - (d.qpos[:, p] + h * v[:, k])).max() < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [33, 70])
def test_cuda_single_dof_actuators_add_in_actuator_order(oracle, cuda_device, nu):
    """Batches of single-dof actuators take the ranked one-step path; several actuators on
    one dof (70 actuators on 28 dofs) must still add in ascending actuator order."""
    import torch

    from instantmimic_b200 import mjw_step_optimized as runtime

    m, d, _, gain = _problem(nu=nu, single=True, seed=9)
    assert (d.moment_rownnz == 1).all()
    md, dd = mjw_model.to_device(m, cuda_device), mjw_model.to_device(copy.deepcopy(d), cuda_device)
    scratch = runtime.make_optimized_fwd_position_scratch(md, dd, cuda_device)
    runtime.attach_implicit_scratch(md, dd, scratch, cuda_device)
    scratch.implicit_actuator_vel.copy_(torch.from_numpy(gain))
    runtime.deriv_smooth_vel_dense_actuator_centric(md, dd, scratch.implicit_qderiv, scratch)
    torch.cuda.synchronize()
    A = oracle.implicit_matrix(m, d, gain)
    np.testing.assert_array_equal(scratch.implicit_qderiv.cpu().numpy().view(np.uint32), A.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [0, 20])
def test_cuda_implicitfast_tail_matches_oracle(oracle, cuda_device, nu):
    import torch

    from instantmimic_b200 import mjw_step_optimized as runtime

    m, d, Mdense, gain = _problem(nu=nu)
    md, dd = mjw_model.to_device(m, cuda_device), mjw_model.to_device(copy.deepcopy(d), cuda_device)
    scratch = runtime.make_optimized_fwd_position_scratch(md, dd, cuda_device)
    runtime.attach_implicit_scratch(md, dd, scratch, cuda_device)
    if nu:
        scratch.implicit_actuator_vel.copy_(torch.from_numpy(gain))
    # 1. the matrix, bit for bit
    runtime.deriv_smooth_vel_dense_actuator_centric(md, dd, scratch.implicit_qderiv, scratch)
    torch.cuda.synchronize()
    A = oracle.implicit_matrix(m, d, gain if nu else None)
    np.testing.assert_array_equal(scratch.implicit_qderiv.cpu().numpy().view(np.uint32), A.view(np.uint32))
    # 2. solve + advance through the tree L'DL kernel
    runtime._factor_solve_i_dense(md, dd, scratch.implicit_qderiv, scratch.implicit_qacc, dd.efc.Ma,
                                  scratch.dense_factor_solve, tree_factor_solve=scratch.tree_factor_solve)
    runtime._advance_with_scratch(md, dd, scratch.implicit_qacc, scratch)
    torch.cuda.synchronize()
    x = scratch.implicit_qacc.cpu().numpy()
    exact = np.linalg.solve(_dense_a(m, d, Mdense, gain), d.efc.Ma.astype(np.float64)[..., None])[..., 0]
    np.testing.assert_allclose(x, exact, rtol=SOLVE_RTOL, atol=SOLVE_RTOL * np.abs(exact).max())
    want = copy.deepcopy(d)
    oracle.advance(m, want, x)  # same acceleration in: compares the advance alone
    got = mjw_model.to_host(dd)
    np.testing.assert_array_equal(got.qvel.view(np.uint32), want.qvel.view(np.uint32))
    assert np.abs(got.qpos - want.qpos).max() <= ADVANCE_TOL
    np.testing.assert_array_equal(got.time, want.time)


@pytest.mark.gpu
def test_implicitfast_integrate_entry(oracle, cuda_device):
    """The whole tail through one call, on a model with affine (position-servo) actuators:
    the velocity gains come from the actuator parameters."""
    import torch

    from instantmimic_b200 import mjw_step_optimized as runtime

    m, d, Mdense, _ = _problem(nu=20)
    rng = np.random.default_rng(4)
    m.actuator_gaintype = np.zeros(m.nu, np.int32)
    m.actuator_biastype = np.full(m.nu, int(types.BiasType.AFFINE), np.int32)
    m.actuator_dyntype = np.zeros(m.nu, np.int32)
    m.actuator_gainprm = np.zeros((m.nu, 10), np.float32)
    m.actuator_biasprm = np.zeros((m.nu, 10), np.float32)
    m.actuator_biasprm[:, 2] = -rng.uniform(1.0, 20.0, m.nu)  # -kd
    d.ctrl = rng.uniform(-1, 1, (d.nworld, m.nu)).astype(np.float32)
    gain = np.broadcast_to(m.actuator_biasprm[:, 2], (d.nworld, m.nu)).astype(np.float32)
    md, dd = mjw_model.to_device(m, cuda_device), mjw_model.to_device(copy.deepcopy(d), cuda_device)
    scratch = runtime.make_optimized_fwd_position_scratch(md, dd, cuda_device)
    runtime.attach_implicit_scratch(md, dd, scratch, cuda_device)
    runtime.implicitfast_integrate(md, dd, scratch)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(scratch.implicit_actuator_vel.cpu().numpy(), gain)
    exact = np.linalg.solve(_dense_a(m, d, Mdense, gain), d.efc.Ma.astype(np.float64)[..., None])[..., 0]
    h = float(m.opt.timestep[0])
    got = mjw_model.to_host(dd)
    assert np.abs(got.qvel - (d.qvel + h * exact)).max() <= 1e-4 * (np.abs(exact).max() + 1)


@pytest.mark.gpu
@pytest.mark.parametrize("nu,shape", [(28, "ball"), (33, "ball"), (70, "ball"), (1, "hinge"), (32, "hinge"), (5, "clash")])
def test_gains_formed_in_the_assembly_and_batches_of_moment_rows(oracle, cuda_device, nu, shape):
    """The assembly that forms the velocity gains itself equals gain call + assembly bit for bit, and
    the oracle: three-dof rows with one nonzero moment (ball-joint motors), rows of one dof, and
    three-dof rows whose actuators meet on the same entries."""
    import torch

    from instantmimic_b200 import mjw_step_optimized as runtime

    m, d = _problem(worlds=37, nu=nu, seed=nu, single=True)[:2]
    rng = np.random.default_rng(nu)
    W, n = d.nworld, (1 if shape == "hinge" else 3)
    first = rng.integers(6, m.nv - 3, (W, nu)) if shape != "clash" else np.full((W, nu), 6)
    d.moment_rownnz = np.full((W, nu), n, np.int32)
    d.moment_rowadr = np.tile(np.arange(nu, dtype=np.int32) * n, (W, 1))
    d.moment_colind = (first[..., None] + np.arange(n)).reshape(W, -1).astype(np.int32)
    moment = rng.normal(size=(W, nu, n)).astype(np.float32)
    if shape == "ball":
        moment *= np.eye(3, dtype=np.float32)[rng.integers(0, 3, (W, nu))]
    d.actuator_moment = moment.reshape(W, -1).copy()
    d.ctrl = rng.uniform(-1, 1, (W, nu)).astype(np.float32)
    m.actuator_gaintype = np.full(nu, int(types.GainType.AFFINE), np.int32)
    m.actuator_biastype = np.full(nu, int(types.BiasType.AFFINE), np.int32)
    m.actuator_dyntype = np.zeros(nu, np.int32)
    m.actuator_gainprm = rng.normal(size=(nu, 10)).astype(np.float32)
    m.actuator_biasprm = -rng.uniform(1, 20, (nu, 10)).astype(np.float32)
    md, dd = mjw_model.to_device(m, cuda_device), mjw_model.to_device(d, cuda_device)
    scratch = runtime.make_optimized_fwd_position_scratch(md, dd, cuda_device)
    runtime.attach_implicit_scratch(md, dd, scratch, cuda_device)
    runtime.actuator_velocity_gain(md, dd, scratch.implicit_actuator_vel, scratch)
    runtime.deriv_smooth_vel_dense_actuator_centric(md, dd, scratch.implicit_qderiv, scratch)
    A, gains = scratch.implicit_qderiv.clone(), scratch.implicit_actuator_vel.clone()
    scratch.implicit_qderiv.zero_(), scratch.implicit_actuator_vel.zero_()
    runtime._implicit_matrix(md, dd, scratch.implicit_qderiv, scratch, runtime._fused_gain_coefficients(md, dd, scratch), None)
    torch.cuda.synchronize()
    assert torch.equal(gains, scratch.implicit_actuator_vel) and torch.equal(A, scratch.implicit_qderiv)
    np.testing.assert_array_equal(A.cpu().numpy(), oracle.implicit_matrix(m, d, gains.cpu().numpy()))


def _controls(ctrl, form):
    """The controls (W, nu) of all-equal rows in another form with the same values."""
    import torch

    return {"one row": lambda: ctrl[:1].clone(), "expanded": lambda: ctrl[:1].expand(ctrl.shape),
            "row of its own": lambda: ctrl[0].clone(), "every other": lambda: ctrl.repeat_interleave(2, 1)[:, ::2],
            "transposed": lambda: ctrl.t().contiguous().t(), "float64": lambda: ctrl.double(),
            "other device": lambda: ctrl.to("meta" if ctrl.device.type == "cpu" else "cpu"),
            "padded rows": lambda: torch.cat((ctrl, ctrl), 1)[:, :ctrl.shape[1]]}[form]()


CONTROL_FORMS = ("one row", "expanded", "row of its own", "every other", "transposed", "float64", "other device")


@pytest.mark.parametrize("form", CONTROL_FORMS + ("padded rows",))
def test_gains_are_formed_in_the_assembly_for_float_rows_of_controls_only(form):
    """The assembly reads a float row of controls per world; any other form would be read out of
    range or as other numbers and has to go through torch."""
    from types import SimpleNamespace

    import torch

    from instantmimic_b200 import mjw_step_optimized as runtime

    W, nu = 3, 4
    d = SimpleNamespace(nworld=W, ctrl=_controls(torch.ones(W, nu), form))
    pair = (torch.ones(nu), torch.ones(nu))
    scratch = SimpleNamespace(implicit_gain_coefficients=pair, implicit_actuator_vel=torch.zeros(W, nu))
    got = runtime._fused_gain_coefficients(SimpleNamespace(nu=nu), d, scratch)
    assert got is (pair if form == "padded rows" else None)
    d.ctrl = torch.ones(W, nu)
    scratch.implicit_gain_coefficients = tuple(t.to("meta") for t in pair)
    assert runtime._fused_gain_coefficients(SimpleNamespace(nu=nu), d, scratch) is None


@pytest.mark.gpu
@pytest.mark.parametrize("form", CONTROL_FORMS + ("padded rows",))
def test_implicitfast_integrate_takes_controls_of_every_form(cuda_device, form):
    import torch

    from instantmimic_b200 import mjw_step_optimized as runtime

    m, d = _problem(worlds=37, nu=20)[:2]
    rng = np.random.default_rng(5)
    m.actuator_gaintype = np.full(m.nu, int(types.GainType.AFFINE), np.int32)
    m.actuator_biastype = np.full(m.nu, int(types.BiasType.AFFINE), np.int32)
    m.actuator_dyntype = np.zeros(m.nu, np.int32)
    m.actuator_gainprm = rng.normal(size=(m.nu, 10)).astype(np.float32)
    m.actuator_biasprm = -rng.uniform(1, 20, (m.nu, 10)).astype(np.float32)
    d.ctrl = np.tile(rng.uniform(-1, 1, m.nu).astype(np.float32), (d.nworld, 1))
    results = []
    for f in (None, form):
        md, dd = mjw_model.to_device(m, cuda_device), mjw_model.to_device(copy.deepcopy(d), cuda_device)
        if f:
            dd.ctrl = _controls(dd.ctrl, f)
        scratch = runtime.make_optimized_fwd_position_scratch(md, dd, cuda_device)
        runtime.attach_implicit_scratch(md, dd, scratch, cuda_device)
        runtime.implicitfast_integrate(md, dd, scratch)
        torch.cuda.synchronize()
        results.append((scratch.implicit_actuator_vel, scratch.implicit_qderiv, dd.qvel, dd.qpos))
    assert all(torch.equal(a, b) for a, b in zip(*results))


def test_one_dof_assembly_leaves_room_for_every_warp(tmp_path):
    """The assembly variant of large batches of one-dof rows is bound by memory in flight: 64 warps per SM
    (65536 registers), so 32 registers a thread; carrying the several-dof form's products and marks
    costs half of the warps and a seventh of the speed."""
    import re
    import subprocess

    from instantmimic_b200 import build

    flags = [f for f in build.NVCC_FLAGS if f not in ("-shared", "-ldl")]
    cmd = [build.nvcc(), *flags, "-Xptxas", "-v", "-c", str(build.CSRC / "imn_integrate.cu"), "-o", str(tmp_path / "x.o")]
    log = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    used = [int(n) for n in re.findall(r"implicit_matrix_kernel.*?Used (\d+) registers", log, flags=re.S)]
    assert used and min(used) <= 32, used


@pytest.mark.gpu
@pytest.mark.parametrize("worlds", [9472, 9473])
@pytest.mark.parametrize("shape", ["servo", "padded", "mixed", "none"])
def test_both_assembly_variants(oracle, cuda_device, worlds, shape):
    """Either side of the batch size at which one-dof rows change variant: rows of one dof, the same in
    wider storage, storage of one dof per actuator that holds rows of three beside empty ones, and no
    actuators."""
    import torch

    from instantmimic_b200 import mjw_step_optimized as runtime

    nu = 0 if shape == "none" else 21
    m, d = _problem(worlds=4, nu=nu, seed=11, single=True)[:2]
    rng = np.random.default_rng(11)
    if shape != "none":
        n = np.tile([3, 0, 0], (4, nu // 3)) if shape == "mixed" else np.ones((4, nu), int)
        width = nu + 5 if shape == "padded" else nu
        d.moment_rownnz = n.astype(np.int32)
        d.moment_rowadr = (np.cumsum(n, 1) - n).astype(np.int32)
        d.moment_colind = np.zeros((4, width), np.int32)
        d.moment_colind[:, :nu] = np.arange(nu) + 6
        d.actuator_moment = rng.normal(size=(4, width)).astype(np.float32)
    gain = -rng.uniform(1, 20, (4, nu)).astype(np.float32) if nu else None
    md, dd = mjw_model.to_device(m, cuda_device), mjw_model.to_device(d, cuda_device)
    dd.nworld = worlds
    rep = lambda t: t.repeat(worlds // 4 + 1, 1)[:worlds].contiguous()  # noqa: E731
    dd.M = rep(dd.M)
    if nu:
        for name in ("moment_rownnz", "moment_rowadr", "moment_colind", "actuator_moment"):
            setattr(dd, name, rep(getattr(dd, name)))
    from types import SimpleNamespace

    scratch = SimpleNamespace(implicit_actuator_vel=rep(torch.from_numpy(gain).to(cuda_device)) if nu else None)
    out = torch.empty_like(dd.M)
    runtime.deriv_smooth_vel_dense_actuator_centric(md, dd, out, scratch)
    torch.cuda.synchronize()
    want = oracle.implicit_matrix(m, d, gain)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), np.resize(want, out.shape).view(np.uint32))
