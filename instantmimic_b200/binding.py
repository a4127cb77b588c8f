"""Builds the C-ABI structs of ``include/imnewton.h`` from Model / Data / context
objects.  Works on any array type ``arrays.addr`` understands, so the same code
describes device buffers for the CUDA library and host buffers for the oracle
used by the tests."""

from __future__ import annotations

import ctypes as C
from typing import Any

from . import abi, calls, types
from .arrays import addr, addrs, all_strides, dense, elem_strides, is_contiguous, itemsize, length, shape


_UPSTREAM: dict | None = None


def upstream_constants(module_types: Any = None, module_solver: Any = None) -> dict:
    """Every constant this package shares with mujoco-warp, from the live upstream
    modules when they import (``mujoco_warp._src.types`` / ``.solver``; the arguments
    let a test pass stand-ins), else this package's defaults (``types``).

    MuJoCo has moved ``mjDSBL_*`` bits and enum members between releases, so nothing
    that is compared with a value stored in a caller's ``Model`` / ``Data`` is taken
    from this package when the real definition is at hand.  ``MJ_MINVAL`` /
    ``MJ_MAXVAL`` are compiled into the kernels: a live module that disagrees with
    them is an error, not an override."""
    global _UPSTREAM
    injected = module_types is not None or module_solver is not None
    if _UPSTREAM is not None and not injected:
        return _UPSTREAM
    if not injected:
        try:  # pragma: no cover - mujoco_warp is not installed in the build image
            from mujoco_warp._src import solver as module_solver
            from mujoco_warp._src import types as module_types
        except Exception:
            module_solver = module_types = None

    def member(enum_name: str, name: str, default: int) -> int:
        enum_cls = getattr(module_types, enum_name, None) if module_types is not None else None
        value = getattr(enum_cls, name, None)
        return int(default if value is None else value)

    out = {
        "source": "mujoco_warp" if module_types is not None else "package defaults",
        "alpha_noise_eps": float(getattr(module_solver, "_ALPHA_NOISE_EPS", types.ALPHA_NOISE_EPS)),
        "overflow_iterations": member("OverflowType", "ITERATIONS", types.OverflowType.ITERATIONS),
        "overflow_ls_iterations": member("OverflowType", "LS_ITERATIONS", types.OverflowType.LS_ITERATIONS),
        "disable_warmstart": member("DisableBit", "WARMSTART", types.DisableBit.WARMSTART),
        "disable_damper": member("DisableBit", "DAMPER", types.DisableBit.DAMPER),
        "disable_gravity": member("DisableBit", "GRAVITY", types.DisableBit.GRAVITY),
        "disable_actuation": member("DisableBit", "ACTUATION", types.DisableBit.ACTUATION),
        "disable_refsafe": member("DisableBit", "REFSAFE", types.DisableBit.REFSAFE),
        "constraint_limit_joint": member("ConstraintType", "LIMIT_JOINT", types.ConstraintType.LIMIT_JOINT),
        "solver_newton": member("SolverType", "NEWTON", types.SolverType.NEWTON),
        "cone_pyramidal": member("ConeType", "PYRAMIDAL", types.ConeType.PYRAMIDAL),
        "integrator_discrete": member("IntegratorType", "DISCRETE", types.IntegratorType.DISCRETE),
    }
    for name in ("SATISFIED", "QUADRATIC", "LINEARNEG", "LINEARPOS"):
        live = member("ConstraintState", name, getattr(types.ConstraintState, name))
        if live != int(getattr(types.ConstraintState, name)):
            raise RuntimeError(
                f"mujoco_warp ConstraintState.{name} = {live} differs from the value compiled into the kernels "
                f"({int(getattr(types.ConstraintState, name))})")
    for name in ("MJ_MINVAL", "MJ_MAXVAL"):
        live = getattr(module_types, name, None) if module_types is not None else None
        if live is not None and float(live) != float(getattr(types, name)):
            raise RuntimeError(
                f"mujoco_warp {name} = {live} differs from the value compiled into the kernels "
                f"({getattr(types, name)})")
    if not injected:
        _UPSTREAM = out
    return out


def _mulm_lanes(m: Any):
    """The lane program of a model's M_mulm rows; built once (and cached on the model) for
    Model objects that come from mujoco-warp and do not carry it."""
    lanes = getattr(m, "M_mulm_lanes", None)
    if lanes is None:
        lanes = getattr(m, "_imn_mulm_lanes", None)
    if lanes is None:
        import numpy as np

        from .arrays import device_of, to_host
        from .mjw_model import mulm_lane_program

        col, madr = m.M_mulm_col, m.M_mulm_madr
        host = mulm_lane_program(to_host(m.M_mulm_rowadr), to_host(col), to_host(madr), int(m.nv))
        if isinstance(col, np.ndarray):
            lanes = host
        else:
            import torch

            # on the device that holds the model's tables, not torch's current one
            lanes = torch.from_numpy(host).to(device_of(col))
        try:
            m._imn_mulm_lanes = lanes
        except AttributeError:
            pass
    return lanes


_MODEL = calls.getter("opt.tolerance", "opt.ls_tolerance", "stat.meaninertia", "M_rowadr", "M_rownnz", "M_colind",
                      "M_mulm_rowadr", "M_mulm_col", "M_mulm_madr")
_pack_model = abi.packer(abi.ImnModel)


def pack_model(m: Any) -> bytes:
    c, opt = upstream_constants(), m.opt
    arrays = (*_MODEL(m), _mulm_lanes(m))
    tolerance, ls_tolerance, meaninertia, _, _, colind, _, _, _, lanes = arrays
    return _pack_model(
        m.nv, m.nv_pad, colind.shape[0], int(opt.iterations), int(opt.ls_iterations),
        0 if int(opt.disableflags) & c["disable_warmstart"] else 1,
        tolerance.shape[0], ls_tolerance.shape[0], meaninertia.shape[0], *addrs(arrays),
        c["alpha_noise_eps"], c["overflow_iterations"], c["overflow_ls_iterations"],
        int(getattr(opt, "warn_overflow", 0) or 0), lanes.shape[0] - 1)


def model_struct(m: Any) -> abi.ImnModel:
    return abi.ImnModel.from_buffer_copy(pack_model(m))


def _row_ld(a: Any) -> int:
    st = elem_strides(a)
    if st[-1] != 1:
        raise ValueError("solver buffers need a unit innermost stride")
    return st[0]


def _same_ld(name: str, strides: tuple) -> int:
    first = strides[0]
    if first is not None and strides == (first,) * len(strides) and len(first) == 2 and first[1] == 1:
        return first[0]
    present = [st for st in strides if st is not None]
    if any([st[-1] != 1 for st in present]):
        raise ValueError("solver buffers need a unit innermost stride")
    lds = {st[0] for st in present}
    if len(lds) != 1:
        raise ValueError(f"{name} arrays must share one world stride, got {sorted(lds)}")
    return lds.pop()


_DATA = calls.getter("nefc", "ne", "nf", "qacc_smooth", "qacc_warmstart", "qfrc_smooth", "efc.J", "efc.D", "efc.aref",
                     "efc.frictionloss", "M", "qacc", "qfrc_constraint", "efc.Ma", "efc.force", "efc.state", "solver_niter",
                     "overflow")
_pack_data = abi.packer(abi.ImnData)


def pack_data(m: Any, d: Any) -> tuple[bytes, int, int]:
    """(ImnData, world stride of the dof arrays, of the row arrays)."""
    nworld, njmax = int(d.nworld), int(d.njmax)
    arrays = _DATA(d)
    J, strides = arrays[6], all_strides(arrays[3:6] + arrays[10:14])
    M_ld, inner = strides[3]
    if inner != 1:
        raise ValueError("solver buffers need a unit innermost stride")
    dof_ld = _same_ld("dof", strides[:3] + strides[4:])
    offsets = getattr(d.efc, "J_world_offset", None)
    ld_world = ld_row = efc_ld = offset_addr = elems = 0
    if offsets is not None:
        # compact J: (total rows, >= nv) with one int64 element offset per world
        if itemsize(offsets) != 8 or length(offsets) < nworld:
            raise ValueError("efc.J_world_offset must hold one int64 per world")
        js = elem_strides(J)
        if len(js) != 2 or js[1] != 1:
            raise ValueError("a compact efc.J is a (rows, nv) array with a unit innermost stride")
        offset_addr = addr(offsets) or 0
        ld_row = js[0]
        elems = length(J) * js[0]
    elif njmax > 0:
        js = elem_strides(J)
        if js[2] != 1:
            raise ValueError("efc.J needs a unit innermost stride")
        ld_world, ld_row = js[0], js[1]
    if njmax > 0:
        efc_ld = _same_ld("efc", all_strides(arrays[7:10] + arrays[14:16]))
    # else: a model without constraint storage: the row arrays are empty, their strides carry no
    # information, and only the rowless hand-off may be called
    (a_nefc, a_ne, a_nf, a_smooth, a_warm, a_qfs, a_J, a_D, a_aref, a_loss, a_M, a_qacc, a_qfrc, a_Ma, a_force, a_state,
     a_niter, a_overflow) = addrs(arrays)
    packed = _pack_data(nworld, njmax, a_nefc, a_ne, a_nf, a_smooth, a_warm, a_qfs, dof_ld, a_J, ld_world, ld_row, a_D, a_aref,
                        a_loss, efc_ld, a_M, M_ld, a_qacc, a_qfrc, a_Ma, a_force, a_state, a_niter, a_overflow,
                        offset_addr, elems)
    return packed, dof_ld, efc_ld


def data_struct(m: Any, d: Any) -> abi.ImnData:
    return abi.ImnData.from_buffer_copy(pack_data(m, d)[0])


_CTX_ARRAYS = ("Jaref", "jv", "search", "mv", "grad", "h", "hfactor", "search_dot", "grad_dot", "grad_scale",
               "newton_decrement", "improvement", "alpha", "done", "search_unchanged", "ls_exhausted", "quad_changed_ids",
               "quad_changed_count", "state_changed_count", "newton_dof_union", "world_order", "stats", "work_counter")
_CTX_ROWS = ("Jaref", "jv", "search", "mv", "quad_changed_ids")
_CTX = calls.getter(*_CTX_ARRAYS)
_pack_ctx = abi.packer(abi.ImnCtx)


def pack_ctx(nworld: int, dof_ld: int, efc_ld: int, ctx: Any, nsolving: Any, plan_address: int = 0) -> bytes:
    """``ctx`` may omit any array (attribute missing or None): the kernel then skips
    writing it back."""
    try:
        arrays = _CTX(ctx)
    except AttributeError:
        arrays = tuple([getattr(ctx, name, None) for name in _CTX_ARRAYS])
    # grad, which has a stride of its own, and the arrays that share one with the row or dof arrays
    grad_stride, *strides = all_strides((arrays[4], *arrays[:4], arrays[16]))
    if grad_stride is not None and grad_stride[-1] != 1:
        raise ValueError("solver buffers need a unit innermost stride")
    rows, dofs = (efc_ld, 1), (dof_ld, 1)
    if strides != [rows, rows, dofs, dofs, rows]:
        for name, st, want in zip(_CTX_ROWS, strides, (rows, rows, dofs, dofs, rows)):
            if st is not None and st[-1] != 1:
                raise ValueError("solver buffers need a unit innermost stride")
            if st is not None and st[0] != want[0]:
                raise ValueError(f"ctx.{name} must share the world stride of the {'efc' if want is rows else 'dof'} arrays")
    order, stats = arrays[20], arrays[21]
    if order is not None and length(order) < nworld:
        raise ValueError("ctx.world_order must hold one int32 per world")
    if stats is not None and (tuple(stats.shape) != (nworld, 4) or elem_strides(stats) != (4, 1)):
        raise ValueError("ctx.stats must be a contiguous (nworld, 4) int32 array")
    try:
        at = [0 if a is None else a.data_ptr() for a in arrays]
    except AttributeError:
        at = addrs(arrays)
    return _pack_ctx(*at[:5], grad_stride[0] if grad_stride is not None else 0, *at[5:20], addr(nsolving) or 0, plan_address,
                     *at[20:])


def ctx_struct(d_struct: abi.ImnData, ctx: Any, nsolving: Any, sparse_plan_struct=None) -> abi.ImnCtx:
    s = abi.ImnCtx.from_buffer_copy(pack_ctx(d_struct.nworld, d_struct.dof_ld, d_struct.efc_ld, ctx, nsolving))
    if sparse_plan_struct is not None:
        s.sparse_plan = C.pointer(sparse_plan_struct)
    return s


def _timestep(m: Any) -> tuple[int, int]:
    """Address and length of opt.timestep, mujoco-warp's per-world float array (world w
    reads element w % n, in the kernels, like every other per-world option)."""
    h = m.opt.timestep
    if isinstance(h, (int, float)) or h is None:
        raise ValueError("m.opt.timestep must be a float array of length 1 or nworld, next to the other arrays")
    n = h.shape[0]
    if n <= 0 or not is_contiguous(h):
        raise ValueError("m.opt.timestep must be a contiguous, non-empty float array")
    return addr(h), n


_pack_implicit, _pack_advance = abi.packer(abi.ImnImplicit), abi.packer(abi.ImnAdvance)


def pack_implicit(m: Any, d: Any, velocity_gain: Any, coefficients: Any = None) -> bytes:
    """``velocity_gain``: (nworld, nu) d(actuator force)/d(actuator velocity), or None.  With
    ``coefficients`` (g2, b2 per actuator) the kernel forms it from ``d.ctrl`` and stores it there."""
    c, flags, nu, W = upstream_constants(), int(m.opt.disableflags), int(getattr(m, "nu", 0) or 0), int(d.nworld)
    actuation = 0 if flags & c["disable_actuation"] else 1
    timestep, n_timestep = _timestep(m)
    tables = m.dof_damping, m.M_elemid
    nnz = adr = col = moment = gain = moment_ld = ctrl = ctrl_ld = g2 = b2 = n_coefficients = 0
    if nu and actuation:
        if velocity_gain is None:
            raise ValueError("an actuated model needs the actuators' velocity gains")
        per_actuator = d.moment_rownnz, d.moment_rowadr, velocity_gain
        if not dense(per_actuator, [(W, nu)] * 3):
            for name, a in zip(("d.moment_rownnz", "d.moment_rowadr", "velocity gains"), per_actuator):
                if tuple(a.shape) != (W, nu) or not is_contiguous(a):
                    raise ValueError(f"{name} must be a contiguous (nworld, nu) array")
        entries = d.moment_colind, d.actuator_moment
        strides = all_strides(entries)
        moment_ld, inner = strides[1]
        if strides[0] != strides[1] or inner != 1:
            raise ValueError("d.moment_colind and d.actuator_moment must share one layout")
        if coefficients is None:
            damping, elemid, nnz, adr, gain, col, moment = addrs(tables + per_actuator + entries)
        else:
            dims = coefficients[0].shape
            n_coefficients, ctrl_ld = dims[0] if len(dims) == 2 else 1, _row_ld(d.ctrl)
            damping, elemid, nnz, adr, gain, col, moment, ctrl, g2, b2 = addrs(
                tables + per_actuator + entries + (d.ctrl, *coefficients))
    else:
        damping, elemid = addrs(tables)
    return _pack_implicit(m.nv, length(m.M_colind), nu, actuation, 0 if flags & c["disable_damper"] else 1, timestep, n_timestep,
                          damping, elemid, nnz, adr, col, moment, moment_ld, gain, ctrl, ctrl_ld, g2, b2, n_coefficients,
                          gain if ctrl else 0)


def implicit_struct(m: Any, d: Any, velocity_gain: Any, coefficients: Any = None) -> abi.ImnImplicit:
    return abi.ImnImplicit.from_buffer_copy(pack_implicit(m, d, velocity_gain, coefficients))


def pack_advance(m: Any, d: Any) -> bytes:
    timestep, n_timestep = _timestep(m)
    state = d.qvel, d.qpos
    (qvel_ld, qvel_in), (qpos_ld, qpos_in) = all_strides(state)
    if qvel_in != 1 or qpos_in != 1:
        raise ValueError("solver buffers need a unit innermost stride")
    kind, dofadr, qposadr, qvel, qpos = addrs((m.jnt_type, m.jnt_dofadr, m.jnt_qposadr, *state))
    return _pack_advance(m.nv, m.nq, m.njnt, timestep, n_timestep, kind, dofadr, qposadr, qvel, qvel_ld, qpos, qpos_ld,
                         addr(getattr(d, "time", None)) or 0)


def advance_struct(m: Any, d: Any) -> abi.ImnAdvance:
    return abi.ImnAdvance.from_buffer_copy(pack_advance(m, d))
