"""Batches that give an SM a few worlds (several warps per world), as many as it holds, and more
(a warp takes further worlds): J resident, streamed by rows of whole quads (snu, nv 64) and by
contiguous tiles (g1), dense and sparse factor, against the oracle bit for bit."""

import copy

import numpy as np
import pytest

from instantmimic_b200 import mjw_model, synthetic
from instantmimic_b200 import mjw_step_optimized as runtime
from instantmimic_b200.mjw_kernels import sparse_hessian

from helpers import host_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm", [2, 5, 18])
@pytest.mark.parametrize("name,sparse", [("humanoid", False), ("humanoid", True), ("snu", True), ("g1", False), ("nv64", False)])
def test_worlds_per_sm(oracle, cuda_device, name, sparse, per_sm):
    import torch

    worlds = per_sm * torch.cuda.get_device_properties(cuda_device).multi_processor_count - 3
    if name == "nv64":
        m, d, _ = synthetic.make_sweep_point(64, 96, worlds, seed=3, iterations=4, ls_iterations=6)
    else:
        m, d, _ = synthetic.make_workload(name, worlds, seed=3, iterations=6, ls_iterations=6, rowless_fraction=0.1)
    md, dd = mjw_model.to_device(m, cuda_device), mjw_model.to_device(copy.deepcopy(d), cuda_device)
    scratch = runtime.make_optimized_fwd_position_scratch(md, dd, cuda_device)
    plan = None
    if sparse:
        groups = [[b] for b in range(1, len(m.body_dofadr))]
        assert runtime.refresh_sparse_hessian(md, dd, scratch, groups, cuda_device) == "enabled"
        plan = sparse_hessian.host_struct(scratch.solver_context.sparse_hessian_plan)
    runtime.solve_with_scratch(md, dd, scratch, use_optimized_kernel=True)
    got = mjw_model.to_host(dd)
    want = copy.deepcopy(d)
    oracle.solve(m, want, host_ctx(m, want), np.zeros(1, np.int32), sparse_plan_struct=plan)
    np.testing.assert_array_equal(got.solver_niter, want.solver_niter)
    np.testing.assert_array_equal(got.overflow, want.overflow)
    live = np.arange(want.njmax)[None, :] < np.minimum(want.nefc, want.njmax)[:, None]
    np.testing.assert_array_equal(got.efc.state[live], want.efc.state[live])
    for a, b in ((got.qacc, want.qacc), (got.efc.Ma, want.efc.Ma), (got.qfrc_constraint, want.qfrc_constraint),
                 (got.efc.force[live], want.efc.force[live])):
        np.testing.assert_array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


def test_worlds_that_leave_the_staged_masks_no_room(oracle, cuda_device):
    """The largest row limit of the humanoid's plan: a world that fits beside the plan's tables and not beside the masks
    as well, whose tables stay in global memory."""
    m, d, _ = synthetic.make_workload("humanoid", 3, seed=3, iterations=6, ls_iterations=6)
    rows, most = d.njmax, 6840
    for name, a in vars(d.efc).items():
        if isinstance(a, np.ndarray) and a.ndim >= 2 and a.shape[1] == rows:
            setattr(d.efc, name, np.concatenate([a, np.zeros((3, most - rows, *a.shape[2:]), a.dtype)], 1))
    d.njmax = most
    md, dd = mjw_model.to_device(m, cuda_device), mjw_model.to_device(copy.deepcopy(d), cuda_device)
    scratch = runtime.make_optimized_fwd_position_scratch(md, dd, cuda_device)
    groups = [[b] for b in range(1, len(m.body_dofadr))]
    assert runtime.refresh_sparse_hessian(md, dd, scratch, groups, cuda_device) == "enabled"
    plan = sparse_hessian.host_struct(scratch.solver_context.sparse_hessian_plan)
    runtime.solve_with_scratch(md, dd, scratch, use_optimized_kernel=True)
    got, want = mjw_model.to_host(dd), copy.deepcopy(d)
    oracle.solve(m, want, host_ctx(m, want), np.zeros(1, np.int32), sparse_plan_struct=plan)
    np.testing.assert_array_equal(got.solver_niter, want.solver_niter)
    for a, b in ((got.qacc, want.qacc), (got.efc.Ma, want.efc.Ma), (got.qfrc_constraint, want.qfrc_constraint)):
        np.testing.assert_array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))
