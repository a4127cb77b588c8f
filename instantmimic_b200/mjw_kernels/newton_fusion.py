"""Fused per-world Newton iteration: eligibility, launch geometry and the launch.

Mirrors the interface of the reference's
``src/instantmimic/utils/mjw_kernels/newton_fusion.py``; the kernels themselves
are ``csrc/imn_newton.cu`` behind ``imn_solve``.
"""

from __future__ import annotations

import ctypes as C
from typing import Any

from .. import _lib, abi, binding, calls, types
from ..arrays import is_device

# CTAs per SM requested from the compiler for the reference's Warp kernel
# (newton_fusion.py:27-33).  The CUDA kernel here is one warp per world and is
# limited by shared memory, not registers; the function is kept because callers
# and tests of the reference use it.
_NEWTON_MAX_BLOCKS_PER_SM = 12


def newton_min_blocks_per_sm(nworld: int, sm_count: int) -> int:
    """CTAs per SM worth demanding for a grid of ``nworld`` worlds, 0 for none
    (newton_fusion.py:36-49)."""
    if nworld <= 0 or sm_count <= 0:
        return 0
    return max(1, min(nworld // sm_count, _NEWTON_MAX_BLOCKS_PER_SM))


def _use_incremental(m: Any) -> bool:
    """Upstream ``solver._use_incremental``: the Newton solver keeps H between
    iterations."""
    return int(m.opt.solver) == binding.upstream_constants()["solver_newton"]


def _sparse_compact(ctx: Any) -> bool:
    return bool(getattr(ctx, "sparse_compact", False))


def _on_cuda(m: Any) -> bool:
    ref = getattr(m, "body_parentid", None)
    device = getattr(ref, "device", None)
    if device is not None and hasattr(device, "is_cuda"):
        return bool(device.is_cuda)
    if device is not None and hasattr(device, "type"):
        return device.type == "cuda"
    return ref is not None and is_device(ref)


def eligible(m: Any, ctx: Any, *, compact: bool = False) -> bool:
    """Structural gates of the fused path (newton_fusion.py:307-322)."""
    return bool(
        not compact
        and _on_cuda(m)
        and 0 < m.nv <= 79
        and m.nv_pad % 16 == 0
        and m.nv_pad <= 80
        and _use_incremental(m)
        and int(m.opt.integrator) != binding.upstream_constants()["integrator_discrete"]
        and int(m.opt.cone) == binding.upstream_constants()["cone_pyramidal"]
        and not m.is_sparse
        and not _sparse_compact(ctx)
        and m.opt.iterations > 0
        and m.block_dim.linesearch_iterative == 32
    )


def ineligible_reasons(m: Any, ctx: Any, *, compact: bool = False) -> list[str]:
    """The gates of ``eligible`` that this model fails, in words."""
    checks = [
        (not compact, "compact (sleeping-island) solve"),
        (_on_cuda(m), "model buffers are not on a CUDA device"),
        (0 < m.nv <= 79, f"nv {m.nv} outside 1..79"),
        (m.nv_pad % 16 == 0 and m.nv_pad <= 80, f"nv_pad {m.nv_pad} is not a multiple of 16 up to 80"),
        (_use_incremental(m), "solver is not Newton"),
        (int(m.opt.integrator) != binding.upstream_constants()["integrator_discrete"], "DISCRETE integrator"),
        (int(m.opt.cone) == binding.upstream_constants()["cone_pyramidal"], "elliptic friction cones"),
        (not m.is_sparse, "sparse constraint Jacobian"),
        (not _sparse_compact(ctx), "sparse-compact solver context"),
        (m.opt.iterations > 0, "opt.iterations is 0"),
        (m.block_dim.linesearch_iterative == 32, "line-search block width is not 32"),
    ]
    return [why for ok, why in checks if not ok]


def newton_block_dim(m: Any) -> int:
    """Logical block width of one world (newton_fusion.py:325-327).  It fixes the
    order of the per-thread partial sums; the CUDA kernel reproduces that order
    inside one physical warp."""
    return 64 if m.nv_pad >= 64 else m.block_dim.linesearch_iterative


def attach_scratch(m: Any, d: Any, ctx: Any, device: Any) -> None:
    """``ctx.newton_dof_union``: the dofs the changed rows touch and their count
    (newton_fusion.py:301-304)."""
    import torch

    ctx.newton_dof_union = torch.zeros((d.nworld, m.nv + 1), dtype=torch.int32, device=device)


class SolveCall:
    """The packed structs of one (Model, Data, context) triple as its buffers are now.  Every solve
    packs its own: a call is for one use (or for ``launch_info``) and is not kept."""

    def __init__(self, m: Any, d: Any, ctx: Any, nsolving: Any):
        plan = getattr(ctx, "sparse_hessian_plan", None)
        # the plan's struct has to outlive the call
        self.plan_struct = getattr(plan, "struct", None) if plan is not None and plan.path == "fused" else None
        data, dof_ld, efc_ld = binding.pack_data(m, d)
        address = C.addressof(self.plan_struct) if self.plan_struct is not None else 0
        self.args = (binding.pack_model(m), data, binding.pack_ctx(int(d.nworld), dof_ld, efc_ld, ctx, nsolving, address))

    def launch_info(self) -> abi.ImnLaunchInfo:
        info = abi.ImnLaunchInfo()
        _lib.check(_lib.packed("imn_launch_info")(*self.args, C.byref(info)), "imn_launch_info")
        return info

    def __call__(self, stream=None) -> None:
        calls.call("imn_solve", self.args, stream)


def solve_call(m: Any, d: Any, ctx: Any, nsolving: Any, cache_on: Any = None) -> SolveCall:
    """``cache_on`` is accepted for callers that name the scratch; nothing is kept on it."""
    del cache_on
    return SolveCall(m, d, ctx, nsolving)


def run(m: Any, d: Any, ctx: Any, nsolving: Any, stream=None) -> None:
    """Init, every Newton iteration and the final force of all worlds: one launch
    (reference: init_context + run + qfrc_constraint_from_grad,
    newton_fusion.py:330-409, 431-472, 522-539)."""
    SolveCall(m, d, ctx, nsolving)(stream)
