"""Depth-ordered body velocities.

Host side of the reference's ``src/instantmimic/utils/mjw_kernels/velocity_fusion.py``
(``com_vel`` :105-126, kernel :15-103); the kernel is ``com_vel_kernel`` in
``csrc/imn_body_tree.cu`` behind ``imn_com_vel``.  Without a tree scratch the reference
runs upstream mujoco-warp's per-level launches; this package has no second path.
"""

from __future__ import annotations

from typing import Any

from .. import calls
from ..arrays import addr, length
from . import tree_fusion


def com_vel(m: Any, d: Any, tree: Any, stream=None) -> None:
    """d.cvel and d.cdof_dot from d.qvel and d.cdof."""
    tree_fusion._need(tree, "com_vel")
    nb, nv, W, qvel = length(m.body_parentid), m.nv, int(d.nworld), d.qvel
    per_dof = (W, nv, 6)
    cdof, cvel, cdof_dot = tree_fusion._all_per_body((d.cdof, d.cvel, d.cdof_dot), [per_dof, (W, nb, 6), per_dof],
                                                     ("cdof", "cvel", "cdof_dot"))
    calls.call("imn_com_vel", (tree_fusion.pack_tree_joints(m, tree), addr(qvel), tree_fusion._row_ld(qvel), cdof, cvel, cdof_dot,
                               W), stream)
