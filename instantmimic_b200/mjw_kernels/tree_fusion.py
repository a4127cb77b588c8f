"""Bottom-up rigid-body reductions: the subtree centres of mass, the composite inertias
with the joint-space inertia M, and the bias forces.

Host side of the reference's ``src/instantmimic/utils/mjw_kernels/tree_fusion.py``
(``TreeReductionScratch`` :27-33, ``create_tree_reduction_scratch`` :36-50, ``accumulate``
:138-170, ``subtree_com_accumulate`` :173-183, ``crb`` :186-206, ``rne`` :209-222).  The
kernels are in ``csrc/imn_body_tree.cu`` behind ``imn_body_tree_accumulate``, ``imn_crb``
and ``imn_rne``: a world is one warp that walks the levels of ``m.body_tree`` in its slice
of shared memory.

The reference's scratch selects between atomic and ordered ("deterministic") sums and
between one cooperative launch and one launch per level.  Here there is one kernel, it is
ordered (children join their parent in level-list order, one writer per parent) and it is
one launch; the two flags are kept on the scratch because callers read them
(``_select_tree_reduction``, mjw_step_optimized.py:2887-2894).  Without a scratch the
reference runs upstream mujoco-warp's per-level launches; this package has no second
path, so a missing scratch is an error.
"""

from __future__ import annotations

from dataclasses import dataclass, field
from typing import Any

import numpy as np

from .. import abi, binding, calls
from ..arrays import addr, addrs, dense, device_of, elem_strides, is_contiguous, is_device, length, to_host


@dataclass(frozen=True)
class TreeReductionScratch:
    bodies: Any
    offsets: Any
    levels: int
    deterministic: bool = False
    cooperative: bool = True
    # per parent (by position in ``bodies``) its children in level-list order; no
    # counterpart in the reference, which scans the whole next level for every parent
    child_ptr: Any = None
    child_ids: Any = None
    # lanes of a warp per world: the smallest of 8, 16, 32 that covers the widest level
    team_lanes: int = 32
    keep: tuple = field(default=(), repr=False, compare=False)


def level_tables(body_tree, body_parentid) -> dict[str, np.ndarray]:
    """Level list, level offsets and the per-parent child lists of a body tree."""
    levels = [np.asarray(to_host(level), dtype=np.int32).reshape(-1) for level in body_tree]
    parent = np.asarray(to_host(body_parentid), dtype=np.int32).reshape(-1)
    bodies = np.concatenate(levels).astype(np.int32)
    offsets = np.cumsum([0] + [len(level) for level in levels]).astype(np.int32)
    if sorted(bodies.tolist()) != list(range(len(parent))):
        raise ValueError("m.body_tree must list every body exactly once")
    position = np.empty(len(parent), dtype=np.int64)
    position[bodies] = np.arange(len(bodies))
    depth = np.searchsorted(offsets, position, side="right") - 1
    for body in range(1, len(parent)):
        if depth[body] != depth[parent[body]] + 1:
            raise ValueError(f"body {body} is not one level below its parent {parent[body]}")
    children: list[list[int]] = [[] for _ in bodies]
    for body in bodies.tolist():  # level-list order
        if body != 0:
            children[position[parent[body]]].append(body)
    child_ptr = np.cumsum([0] + [len(c) for c in children]).astype(np.int32)
    child_ids = np.asarray([b for c in children for b in c] or [0], dtype=np.int32)
    widest = max(len(level) for level in levels)
    team = 8 if widest <= 8 else (16 if widest <= 16 else 32)
    return {"bodies": bodies, "offsets": offsets, "child_ptr": child_ptr, "child_ids": child_ids, "team_lanes": team}


def _place(table: np.ndarray, like: Any):
    """A table next to ``like``: a torch tensor on its device, or the numpy array itself."""
    if is_device(like):
        import torch

        return torch.from_numpy(table).to(device_of(like))
    return table


def create_tree_reduction_scratch(m: Any, *, deterministic: bool = False, cooperative: bool = True):
    if not getattr(m, "body_tree", None):
        return None
    t = level_tables(m.body_tree, m.body_parentid)
    return TreeReductionScratch(
        _place(t["bodies"], m.body_parentid),
        _place(t["offsets"], m.body_parentid),
        len(m.body_tree),
        deterministic,
        cooperative,
        _place(t["child_ptr"], m.body_parentid),
        _place(t["child_ids"], m.body_parentid),
        int(t["team_lanes"]),
    )


def _need(scratch: Any, who: str) -> None:
    if scratch is None:
        raise RuntimeError(
            f"{who}: this library has no per-level upstream path; pass the scratch of create_tree_reduction_scratch")


_TREE = calls.getter("bodies", "offsets", "child_ptr", "child_ids")
_DOFS = ("body_parentid", "body_dofadr", "body_dofnum", "dof_bodyid", "dof_parentid")
_JOINT_TABLES = calls.getter(*_DOFS, "body_jntnum", "body_jntadr", "jnt_type")
_INERTIA_TABLES = calls.getter(*_DOFS, "dof_armature", "M_hinit_i", "M_colind")
_GRAVITY_TABLES = calls.getter(*_DOFS, "opt.gravity")
_pack_tree = abi.packer(abi.ImnBodyTree)


def _rows_of(a: Any, width: int, name: str, extent: str) -> int:
    """Rows of a contiguous (n, width) or (width) option array."""
    dims = a.shape
    if dims[-1] != width or not is_contiguous(a):
        raise ValueError(f"m.{name} must be a contiguous (n, {extent}) or ({extent}) array")
    return dims[0] if len(dims) == 2 else 1


# The C struct over the model's tables, one function per set of tables that a call reads.

def pack_tree(m: Any, t: TreeReductionScratch) -> bytes:
    """The tree alone."""
    parent = m.body_parentid
    at = addrs((parent, *_TREE(t)))
    return _pack_tree(parent.shape[0], 0, 0, t.levels, *at, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, getattr(t, "team_lanes", 32))


def pack_tree_joints(m: Any, t: TreeReductionScratch) -> bytes:
    tables = _JOINT_TABLES(m)
    parent, dofadr, dofnum, body, dof_parent, jntnum, jntadr, kind, *tree = addrs(tables + _TREE(t))
    return _pack_tree(tables[0].shape[0], m.nv, 0, t.levels, parent, *tree, jntnum, jntadr, dofadr, dofnum, kind, body, dof_parent,
                      0, 0, 0, 0, 0, 0, 0, getattr(t, "team_lanes", 32))


def pack_tree_inertia(m: Any, t: TreeReductionScratch) -> bytes:
    tables, nv = _INERTIA_TABLES(m), m.nv
    parent, dofadr, dofnum, body, dof_parent, armature, rows, cols, *tree = addrs(tables + _TREE(t))
    return _pack_tree(tables[0].shape[0], nv, tables[7].shape[0], t.levels, parent, *tree, 0, 0, dofadr, dofnum, 0, body, dof_parent,
                      armature, _rows_of(tables[5], nv, "dof_armature", "nv"), rows, cols, 0, 0, 0, getattr(t, "team_lanes", 32))


def pack_tree_gravity(m: Any, t: TreeReductionScratch) -> bytes:
    tables = _GRAVITY_TABLES(m)
    parent, dofadr, dofnum, body, dof_parent, gravity, *tree = addrs(tables + _TREE(t))
    enabled = 0 if int(m.opt.disableflags) & binding.upstream_constants()["disable_gravity"] else 1
    return _pack_tree(tables[0].shape[0], m.nv, 0, t.levels, parent, *tree, 0, 0, dofadr, dofnum, 0, body, dof_parent, 0, 0, 0, 0,
                      gravity, _rows_of(tables[5], 3, "opt.gravity", "3"), enabled, getattr(t, "team_lanes", 32))


def tree_struct(m: Any, scratch: TreeReductionScratch, *, dofs: bool = False, joints: bool = False,
                inertia: bool = False, gravity: bool = False) -> abi.ImnBodyTree:
    """The struct for a call that reads the named tables (each set includes the dofs')."""
    pack = pack_tree_inertia if inertia else pack_tree_gravity if gravity else pack_tree_joints if joints else pack_tree
    return abi.ImnBodyTree.from_buffer_copy(pack(m, scratch))


def _per_body(a: Any, nworld: int, nbody: int, width: int, name: str) -> int:
    """Address of a contiguous (nworld, nbody, width) float array (a Warp vector array has
    the same bytes with the last extent folded into its dtype)."""
    if tuple(a.shape) not in ((nworld, nbody, width), (nworld, nbody)) or not is_contiguous(a):
        raise ValueError(f"{name} must be a contiguous ({nworld}, {nbody}, {width}) float array")
    return addr(a)


def _all_per_body(arrays: tuple, shapes: list, names: tuple) -> tuple:
    """The same for several arrays of the given shapes."""
    if dense(arrays, shapes):
        return addrs(arrays)
    return tuple([_per_body(a, *dims, "d." + name) for a, dims, name in zip(arrays, shapes, names)])


def _row_ld(a: Any) -> int:
    return elem_strides(a)[0]


def accumulate(m: Any, d: Any, values: Any, components: int, skip_root_parent: bool, scratch: TreeReductionScratch,
               stream=None) -> None:
    """values[:, parent] += values[:, body], deepest level first (tree_fusion.py:138-170)."""
    _need(scratch, "accumulate")
    nbody = length(m.body_parentid)
    calls.call("imn_body_tree_accumulate", (
        pack_tree(m, scratch), _per_body(values, d.nworld, nbody, components, "values"), nbody * components, int(components),
        int(bool(skip_root_parent)), int(d.nworld)), stream)


def subtree_com_accumulate(m: Any, d: Any, scratch: TreeReductionScratch | None = None, stream=None) -> None:
    _need(scratch, "subtree_com_accumulate")
    accumulate(m, d, d.subtree_com, 3, False, scratch, stream)


def crb(m: Any, d: Any, scratch: TreeReductionScratch | None = None, stream=None) -> None:
    """d.crb and d.M from d.cinert and d.cdof (tree_fusion.py:186-206)."""
    _need(scratch, "crb")

    nb, nv, W, M = length(m.body_parentid), m.nv, int(d.nworld), d.M
    cinert, cdof, crb = _all_per_body((d.cinert, d.cdof, d.crb), [(W, nb, 10), (W, nv, 6), (W, nb, 10)],
                                      ("cinert", "cdof", "crb"))
    calls.call("imn_crb", (pack_tree_inertia(m, scratch), cinert, cdof, crb, addr(M), _row_ld(M), W), stream)


def rne(m: Any, d: Any, scratch: TreeReductionScratch | None = None, stream=None) -> None:
    """d.cacc, d.cfrc_int and d.qfrc_bias (tree_fusion.py:209-222)."""
    _need(scratch, "rne")

    nb, nv, W = length(m.body_parentid), m.nv, int(d.nworld)
    per_body, per_dof = (W, nb, 6), (W, nv, 6)
    cinert, cvel, cdof, cdof_dot, cacc, cfrc_int = _all_per_body(
        (d.cinert, d.cvel, d.cdof, d.cdof_dot, d.cacc, d.cfrc_int),
        [(W, nb, 10), per_body, per_dof, per_dof, per_body, per_body],
        ("cinert", "cvel", "cdof", "cdof_dot", "cacc", "cfrc_int"))
    qvel, qfrc_bias = d.qvel, d.qfrc_bias
    calls.call("imn_rne", (pack_tree_gravity(m, scratch), cinert, cvel, cdof, cdof_dot, addr(qvel), _row_ld(qvel), cacc, cfrc_int,
                           addr(qfrc_bias), _row_ld(qfrc_bias), W), stream)
