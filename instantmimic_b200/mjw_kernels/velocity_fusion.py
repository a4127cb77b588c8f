"""Depth-ordered body velocities.

Host side of the reference's ``src/instantmimic/utils/mjw_kernels/velocity_fusion.py``
(``com_vel`` :105-126, kernel :15-103); the kernel is ``com_vel_kernel`` in
``csrc/imn_body_tree.cu`` behind ``imn_com_vel``.  Without a tree scratch the reference
runs upstream mujoco-warp's per-level launches; this package has no second path.
"""

from __future__ import annotations

import ctypes as C
from typing import Any

from .. import calls
from ..arrays import addr, length
from . import tree_fusion


_MODEL = calls.getter("body_parentid", "body_dofadr", "body_dofnum", "dof_bodyid", "dof_parentid", "body_jntadr",
                      "body_jntnum", "jnt_type")
_DATA = calls.getter("qvel", "cdof", "cvel", "cdof_dot")


def com_vel(m: Any, d: Any, tree: Any, stream=None) -> None:
    """d.cvel and d.cdof_dot from d.qvel and d.cdof."""
    tree_fusion._need(tree, "com_vel")

    def build():
        nbody = length(m.body_parentid)
        t = tree_fusion.tree_struct(m, tree, dofs=True, joints=True)
        return (C.byref(t), addr(d.qvel), tree_fusion._row_ld(d.qvel),
                tree_fusion._per_body(d.cdof, d.nworld, m.nv, 6, "d.cdof"),
                tree_fusion._per_body(d.cvel, d.nworld, nbody, 6, "d.cvel"),
                tree_fusion._per_body(d.cdof_dot, d.nworld, m.nv, 6, "d.cdof_dot"), int(d.nworld)), t

    calls.call(d, "imn_com_vel", _MODEL(m) + tree_fusion._TREE(tree) + _DATA(d), (m.nv, d.nworld, tree.levels), build, stream)
