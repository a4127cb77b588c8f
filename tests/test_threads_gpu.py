"""Solves of several threads at once, each with a context and a stream of its own."""

import copy
import threading

import pytest

from instantmimic_b200 import mjw_model, synthetic
from instantmimic_b200 import mjw_step_optimized as runtime
from instantmimic_b200.mjw_kernels import newton_fusion


@pytest.mark.gpu
def test_batches_of_different_size_from_two_threads(cuda_device):
    """Batches of 12 and 13 worlds per SM run the same kernel with 204 and 221 KB of shared memory per CTA:
    a call's limit must not be lowered by the other thread's before its launch."""
    import torch

    m, d, _ = synthetic.make_workload("humanoid", 64, seed=3)
    md = mjw_model.to_device(m, cuda_device)
    jobs, errors = [], []
    for worlds in (12 * 148, 13 * 148):
        dd = mjw_model.to_device(copy.deepcopy(d), cuda_device)

        def rep(t):
            return t.repeat((worlds // 64 + 1,) + (1,) * (t.dim() - 1))[:worlds].contiguous()

        for o in (dd, dd.efc):
            for name, t in list(vars(o).items()):
                if isinstance(t, torch.Tensor):
                    setattr(o, name, rep(t))
        dd.nworld = worlds
        scratch = runtime.make_optimized_fwd_position_scratch(md, dd, cuda_device, include_optimized_kernel_scratch=False)
        runtime.solve_with_scratch(md, dd, scratch, use_optimized_kernel=True)
        jobs.append((dd, scratch, torch.cuda.Stream(), dd.qacc.clone()))
    torch.cuda.synchronize()

    def run(dd, scratch, stream):
        try:
            with torch.cuda.stream(stream):
                call = newton_fusion.solve_call(md, dd, scratch.solver_context, scratch.solver_nsolving, cache_on=scratch)
                for _ in range(3000):  # the library call alone, so that the two overlap often
                    call()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=job[:3]) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for dd, _, _, want in jobs:
        assert torch.equal(dd.qacc, want)
