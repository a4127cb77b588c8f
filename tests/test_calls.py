"""C-ABI calls (instantmimic_b200/calls.py) see the buffers as they are at the call: nothing of an earlier
one is kept, and no buffer is kept alive."""

import copy
import ctypes as C
import gc
import weakref

import pytest
import torch

from instantmimic_b200 import _lib, abi, mjw_model, synthetic
from instantmimic_b200 import mjw_step_optimized as runtime
from instantmimic_b200.mjw_kernels import indexed_factor, newton_fusion, tree_fusion, tree_ldl, velocity_fusion


@pytest.fixture
def seen(monkeypatch):
    """(function, its arguments) of every call, in place of the library."""
    calls = []

    class Library:
        def __getattr__(self, name):
            return lambda *args: calls.append((name, args)) or 0

    monkeypatch.setattr(_lib, "lib", Library)
    monkeypatch.setattr(_lib, "packed", lambda name: getattr(Library(), name), raising=False)
    monkeypatch.setattr(_lib, "current_stream_handle", lambda stream=None: 7)
    monkeypatch.setattr(newton_fusion, "_on_cuda", lambda m: True)
    return calls


def _struct(cls, arg):
    return cls.from_buffer_copy(arg) if isinstance(arg, bytes) else arg._obj


def _workload(worlds=5):
    m, d, _ = synthetic.make_workload("humanoid", worlds, seed=1)
    synthetic.add_smooth_state(m, d, seed=1)
    return mjw_model.to_device(m, "cpu"), mjw_model.to_device(d, "cpu")


def _padded(t, extra=4):
    """The same values at the same first address, rows further apart."""
    wide = torch.zeros(*t.shape[:-1], t.shape[-1] + extra, dtype=t.dtype)
    wide[..., :t.shape[-1]] = t
    return wide[..., :t.shape[-1]]


def test_strides_changed_in_place_are_seen(seen):
    """The same objects at the same addresses, with rows further apart than at the call before."""
    m, d = _workload()
    plan = tree_ldl.create_tree_factor_solve_scratch(m, "cpu", generate=False)
    M, x, y = _padded(d.M), _padded(d.qacc_smooth), _padded(d.qfrc_smooth)
    wide = [t.stride(0) for t in (M, y, x)]
    for t in (M, x, y):
        t.as_strided_(t.shape, (t.shape[1], 1))
    tree_ldl.tree_factor_solve(plan, M, x, y)
    for t, ld in zip((M, y, x), wide):
        t.as_strided_(t.shape, (ld, 1))
    tree_ldl.tree_factor_solve(plan, M, x, y)
    lds = [[args[k] for k in (2, 4, 6)] for _, args in seen]
    assert lds == [[M.shape[1], y.shape[1], x.shape[1]], wide]
    y.as_strided_(y.shape, (1, y.shape[0]))
    with pytest.raises(ValueError, match="contiguous"):
        tree_ldl.tree_factor_solve(plan, M, x, y)


def test_a_layout_that_is_refused_stays_refused(seen):
    m, d = _workload()
    tree = tree_fusion.create_tree_reduction_scratch(m)
    for stage in (tree_fusion.crb, tree_fusion.rne, velocity_fusion.com_vel):
        stage(m, d, tree)
    cdof = d.cdof
    cdof.as_strided_(cdof.shape, (1, 6, cdof.shape[1]))
    for stage in (tree_fusion.crb, tree_fusion.rne, velocity_fusion.com_vel):
        with pytest.raises(ValueError, match="d.cdof"):
            stage(m, d, tree)
    blocked = indexed_factor.create_blocked_dense_factor_solve_scratch(m, d, "cpu")
    x = torch.zeros_like(d.qfrc_smooth)
    indexed_factor.blocked_dense_factor_solve(d, d.M, x, d.qfrc_smooth, blocked)
    x.as_strided_(x.shape, (1, x.shape[0]))
    with pytest.raises(ValueError, match="contiguous x"):
        indexed_factor.blocked_dense_factor_solve(d, d.M, x, d.qfrc_smooth, blocked)


def test_the_solve_sees_options_tables_strides_and_context_as_they_are(seen):
    m, d = _workload()
    scratch = runtime.make_optimized_fwd_position_scratch(m, d, "cpu", include_optimized_kernel_scratch=False)

    def solve():
        runtime.solve_with_scratch(m, d, scratch, use_optimized_kernel=True)
        name, args = seen[-1]
        assert name == "imn_solve"
        return (_struct(abi.ImnModel, args[0]), _struct(abi.ImnData, args[1]), _struct(abi.ImnCtx, args[2]))

    solve()
    # J rows further apart, at the same first address
    J = _padded(d.efc.J)
    d.efc.J = J.as_strided(J.shape, (J.shape[1] * J.shape[2], J.shape[2], 1))
    assert solve()[1].J_ld_row == J.shape[2]
    d.efc.J = J
    assert solve()[1].J_ld_row == J.stride(1)
    # a table of the model in another place
    m.M_colind = m.M_colind.clone()
    assert solve()[0].M_colind == m.M_colind.data_ptr()
    # per-world options in storage that starts where the single one did
    wide = torch.full((d.nworld,), 1e-6)
    m.opt.tolerance = wide[:1]
    assert solve()[0].n_tolerance == 1
    m.opt.tolerance = wide
    assert solve()[0].n_tolerance == d.nworld
    # another plan struct behind the same plan
    groups = [[b] for b in range(1, len(m.body_dofadr))]
    assert runtime.refresh_sparse_hessian(m, d, scratch, groups, "cpu") == "enabled"
    plan = scratch.solver_context.sparse_hessian_plan
    assert C.addressof(solve()[2].sparse_plan.contents) == C.addressof(plan.struct)
    plan.struct = abi.ImnSparsePlan.from_buffer_copy(plan.struct)
    assert C.addressof(solve()[2].sparse_plan.contents) == C.addressof(plan.struct)
    # a context that is outside the path from now on
    scratch.solver_context.sparse_compact = True
    with pytest.raises(RuntimeError, match="sparse-compact"):
        solve()


def test_nothing_is_kept_on_the_callers_objects(seen):
    m, d = _workload()
    scratch = runtime.make_optimized_fwd_position_scratch(m, d, "cpu", include_optimized_kernel_scratch=False)
    tree = tree_fusion.create_tree_reduction_scratch(m)
    plan = tree_ldl.create_tree_factor_solve_scratch(m, "cpu", generate=False)
    blocked = indexed_factor.create_blocked_dense_factor_solve_scratch(m, d, "cpu")
    owners = (m, d, d.efc, scratch, scratch.solver_context, tree, plan, blocked)
    before = [dict(vars(o)) for o in owners]

    def step():
        velocity_fusion.com_vel(m, d, tree)
        tree_fusion.crb(m, d, tree)
        tree_fusion.rne(m, d, tree)
        tree_fusion.accumulate(m, d, d.cfrc_int, 6, True, tree)
        runtime._factor_solve_i_dense(m, d, d.M, d.qacc_smooth, d.qfrc_smooth, None, tree_factor_solve=plan)
        indexed_factor.blocked_dense_factor_solve(d, d.M, d.qacc_smooth, d.qfrc_smooth, blocked)
        runtime.solve_with_scratch(m, d, scratch, use_optimized_kernel=True)

    step()
    assert [set(vars(o)) for o in owners] == [set(b) for b in before]
    first = list(seen)
    d2, watched = copy.deepcopy(d), [weakref.ref(t) for t in (d.cdof, d.M, d.qfrc_smooth, d.efc.J)]
    d = d2  # other buffers: the same calls, and the old ones can go
    del before, owners, d2
    seen.clear()
    step()
    gc.collect()
    assert [name for name, _ in seen] == [name for name, _ in first]
    assert all(ref() is None for ref in watched)
