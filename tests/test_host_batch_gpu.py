"""Batches in pinned host memory (instantmimic_b200/host_batch.py): only rows below each
chunk's largest nefc cross PCIe, in either world order, and the results equal the
oracle's bit for bit."""

import numpy as np
import pytest

from instantmimic_b200 import host_batch, mjw_model, synthetic

from helpers import run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,grouped", [("compact", False), ("rows", False), ("rows", True), ("whole", False),
                                          ("sparse", False), ("sparse8", False)])
def test_host_batch_pipeline_matches_oracle(oracle, cuda_device, mode, grouped):
    import torch

    m, d, _ = synthetic.make_workload("humanoid", 700, seed=5, rowless_fraction=0.05)
    if grouped:
        d, _ = host_batch.group_by_row_count(d)
        assert (np.diff(d.nefc) <= 0).all()
    want, _, _ = run_oracle(oracle, m, d)
    md = mjw_model.to_device(m, cuda_device)
    pipe = host_batch.HostBatchPipeline(md, d, cuda_device, slots=2, mode=mode)
    batch = host_batch.pin_batch(d, chunk=128)
    full = d.nworld * 4 * (3 + 3 * m.nv + m.nM + d.njmax * (m.nv + 3))
    moved = batch.h2d_bytes(m.nv, m.nv, m.nM, d.njmax, mode)
    assert moved <= full + 8 * d.nworld and batch.h2d_bytes(m.nv, m.nv, m.nM, d.njmax, "whole") == full
    if grouped or mode == "compact":
        assert moved < 0.8 * full  # no dead rows (compact) or few (rows of grouped worlds)
    if mode in ("sparse", "sparse8"):
        assert moved < (0.65 if mode == "sparse" else 0.5) * full  # only the nonzeros of the live rows, with their indices
        d.efc.J[0, 0, 3] = -0.0  # a stored negative zero survives the round trip
        batch = host_batch.pin_batch(d, chunk=128)
        want, _, _ = run_oracle(oracle, m, d)
    for k in range(3):  # both slots, one reused
        pipe.submit(k, batch)
    for k in range(3):
        out = pipe.result(k)
        np.testing.assert_array_equal(out["solver_niter"].numpy(), want.solver_niter)
        np.testing.assert_array_equal(out["qacc"].numpy().view(np.uint32), want.qacc.view(np.uint32))
        live = np.arange(d.njmax)[None, :] < d.nefc[:, None]
        np.testing.assert_array_equal(out["state"].numpy()[live], want.efc.state[live])
        np.testing.assert_array_equal(out["force"].numpy()[live].view(np.uint32), want.efc.force[live].view(np.uint32))
    torch.cuda.synchronize()


@pytest.mark.parametrize("worlds", [1129, 1130, 2300])
def test_results_that_go_back_in_pieces(oracle, cuda_device, worlds):
    """Either side of one piece, and several pieces with a remainder."""
    m, d, _ = synthetic.make_workload("humanoid", worlds, seed=6, iterations=4)
    want, _, _ = run_oracle(oracle, m, d, matrices=False)
    pipe = host_batch.HostBatchPipeline(mjw_model.to_device(m, cuda_device), d, cuda_device, slots=2, mode="sparse8")
    sizes = [p.numel() for p, _ in pipe.slots[0]["sparse"]["pieces"]]
    total = host_batch.result_layout(worlds, d.njmax, m.nv)[1]
    assert sum(sizes) == total and max(sizes) <= 1 << 20 and len(sizes) == -(-total // (1 << 20))
    pipe.submit(0, host_batch.pin_batch(d))
    out = pipe.result(0)
    live = np.arange(d.njmax)[None, :] < d.nefc[:, None]
    for name, ref in (("qacc", want.qacc), ("qfrc_constraint", want.qfrc_constraint), ("Ma", want.efc.Ma),
                      ("solver_niter", want.solver_niter), ("overflow", want.overflow)):
        np.testing.assert_array_equal(out[name].numpy().view(np.uint32), ref.view(np.uint32), err_msg=name)
    for name in ("force", "state"):
        np.testing.assert_array_equal(out[name].numpy()[live], getattr(want.efc, name)[live], err_msg=name)
