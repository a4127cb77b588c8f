"""The C-ABI library loads without a GPU, exports every symbol the header declares,
its ctypes mirror has the compiler's struct sizes, and host-side validation rejects
bad calls without launching anything."""

import ctypes as C
import re
import subprocess
import sys
from pathlib import Path

import pytest

from instantmimic_b200 import _lib, abi

ROOT = Path(__file__).resolve().parents[1]
HEADER = ROOT / "include" / "imnewton.h"


def _declared_functions():
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return sorted(set(re.findall(r"\b(imn_[a-z_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    lib = _lib.lib()
    names = _declared_functions()
    assert "imn_solve" in names and "imn_tree_ldl_solve" in names and len(names) >= 10
    for name in names:
        assert hasattr(lib, name), name
    assert sorted(abi.SYMBOLS) == names
    assert lib.imn_abi_version() == abi.IMN_ABI_VERSION


def test_ctypes_structs_match_the_compiler(tmp_path):
    structs = ["ImnModel", "ImnData", "ImnCtx", "ImnSparsePlan", "ImnTreePlan", "ImnBlockedPlan", "ImnLaunchInfo",
               "ImnImplicit", "ImnAdvance", "ImnBallLimits"]
    src = tmp_path / "sizes.c"
    body = "".join(f'  printf("{s} %zu\\n", sizeof({s}));\n' for s in structs)
    src.write_text(f'#include <stdio.h>\n#include "{HEADER}"\nint main(void) {{\n{body}  return 0;\n}}\n')
    exe = tmp_path / "sizes"
    subprocess.run(["/usr/bin/gcc", "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    sizes = dict(line.split() for line in out.strip().splitlines())
    for s in structs:
        assert C.sizeof(getattr(abi, s)) == int(sizes[s]), s


# sizeof every struct of a layout version: a struct that changes takes the next number
_LAYOUTS = {
    6: dict(ImnAdvance=96, ImnBallLimits=304, ImnBlockedPlan=32, ImnBodyTree=168, ImnCtx=208, ImnData=208, ImnImplicit=152,
            ImnLaunchInfo=20, ImnModel=144, ImnSparsePlan=256, ImnTreePlan=48),
    7: dict(ImnAdvance=96, ImnBallLimits=304, ImnBlockedPlan=40, ImnBodyTree=168, ImnCtx=208, ImnData=208, ImnImplicit=152,
            ImnLaunchInfo=20, ImnModel=144, ImnSparsePlan=256, ImnTreePlan=48),
}


def test_struct_sizes_are_those_of_the_layout_version():
    """A host built against another version's header is refused by the number, so a layout has one number."""
    sizes = {name: C.sizeof(getattr(abi, name)) for name in dir(abi) if name.startswith("Imn")}
    assert sizes == _LAYOUTS[_lib.lib().imn_abi_version()]
    assert int(re.search(r"#define IMN_ABI_VERSION (\d+)", HEADER.read_text())[1]) == abi.IMN_ABI_VERSION


def test_validation_rejects_bad_calls_before_any_launch():
    lib = _lib.lib()
    m, d, c = abi.ImnModel(), abi.ImnData(), abi.ImnCtx()
    assert lib.imn_solve(None, C.byref(d), C.byref(c), None) == abi.IMN_ERR_NULL
    m.nv, m.nv_pad, m.iterations = 80, 96, 4  # beyond the fused path
    assert lib.imn_solve(C.byref(m), C.byref(d), C.byref(c), None) == abi.IMN_ERR_UNSUPPORTED
    assert b"nv 80" in lib.imn_last_error()
    m.nv, m.nv_pad = 34, 40  # nv_pad not a multiple of 16
    assert lib.imn_solve(C.byref(m), C.byref(d), C.byref(c), None) == abi.IMN_ERR_UNSUPPORTED
    m.nv, m.nv_pad, m.iterations = 34, 48, 0
    assert lib.imn_solve(C.byref(m), C.byref(d), C.byref(c), None) == abi.IMN_ERR_UNSUPPORTED
    m.iterations = 4
    m.n_tolerance = m.n_ls_tolerance = m.n_meaninertia = 1
    assert lib.imn_solve(C.byref(m), C.byref(d), C.byref(c), None) == abi.IMN_ERR_NULL  # no buffers
    plan = abi.ImnTreePlan()
    assert lib.imn_tree_ldl_solve(C.byref(plan), None, 0, None, 0, None, 0, 1, None) == abi.IMN_ERR_NULL
    bp = abi.ImnBlockedPlan()
    bp.nv, bp.pad = 35, 40
    one = C.c_float(0)
    p = C.addressof(one)
    assert lib.imn_blocked_dense_factor_solve(C.byref(bp), p, 0, p, p, p, None, 1, 1, 1, None) == abi.IMN_ERR_SHAPE


def test_copy_wait_limit_is_validated():
    lib = _lib.lib()
    assert lib.imn_set_copy_wait_limit(0, 0) == abi.IMN_ERR_SHAPE
    assert b"positive" in lib.imn_last_error()
    assert lib.imn_set_copy_wait_limit(1 << 22, 0) == 0


def test_launch_info_reports_geometry_without_a_gpu():
    """Host-only: which kernel variant and how much shared memory a model gets."""
    import numpy as np

    from instantmimic_b200 import binding, synthetic
    from helpers import host_ctx

    lib = _lib.lib()
    # humanoid: J stays in shared memory; the SNU-like model streams it (the 128-row J would
    # leave room for 4 worlds per SM, the row tile for 7)
    for name, resident, threads in (("humanoid", 1, 32), ("snu", 0, 64)):
        m, d, _ = synthetic.make_workload(name, 4, seed=0)
        ms, ds = binding.model_struct(m), binding.data_struct(m, d)
        cs = binding.ctx_struct(ds, host_ctx(m, d), np.zeros(1, np.int32))
        info = abi.ImnLaunchInfo()
        assert lib.imn_launch_info(C.byref(ms), C.byref(ds), C.byref(cs), C.byref(info)) == 0
        assert (info.j_resident, info.world_threads, info.grid) == (resident, threads, 4)
        assert 0 < info.smem_bytes <= 227 * 1024
    m, d, _ = synthetic.make_sweep_point(64, 512, 2, seed=0)
    ms, ds = binding.model_struct(m), binding.data_struct(m, d)
    cs = binding.ctx_struct(ds, None, None)
    info = abi.ImnLaunchInfo()
    assert lib.imn_launch_info(C.byref(ms), C.byref(ds), C.byref(cs), C.byref(info)) == 0
    assert info.j_resident == 0  # 512 rows x 64 dofs stream through the staging tile


@pytest.mark.parametrize("name,per_sm,worlds", [
    # one world more than teams of two hold: they are ahead where worlds differ in rows (473 us against 429, 336 / 306)
    ("snu", 7, 6), ("g1", 7, 6),
    # the same with the dense factor (345 / 308), and its full batches (323 / 278 us, 3502 / 2773, 1758 / 1566)
    ("chain35x96", 9, 8), ("humanoid dense", 14, 13), ("limb64x512", 20, 4), ("limb35x512", 28, 6), ("chain60x64", 7, 6),
    # few worlds: all in hand, with as many warps as there is room for; full batches: a warp each
    ("snu", 1, 1), ("limb64x512", 3, 3), ("humanoid", 6, 6), ("humanoid", 28, 14), ("snu", 28, 9), ("g1", 28, 12)])
def test_worlds_in_hand_follow_the_measured_best(name, per_sm, worlds):
    """Host-only: worlds an SM takes at once, by worlds per SM."""
    import numpy as np

    from instantmimic_b200 import binding, synthetic
    from instantmimic_b200.mjw_kernels import sparse_hessian
    from instantmimic_b200.mjw_model import make_data, put_model
    from helpers import host_ctx

    kind, _, rows = name.partition("x")
    if kind[:5] in ("chain", "limb6", "limb3"):
        parent, body = (synthetic.chain_tree if kind[:5] == "chain" else synthetic.limb_tree)(int(kind.lstrip("chainlimb")))
        m = put_model(parent, body_of_dof=body)
        d, plan = make_data(m, 4, int(rows)), None
    else:
        kind, _, dense = name.partition(" ")
        m, d, _ = synthetic.make_workload(kind, 4, seed=0)
        groups = [[b] for b in range(1, len(m.body_dofadr))]
        plan = None if dense else sparse_hessian.build_plan(m, groups, 32 if m.nv_pad < 64 else 64, "fused")
    ms, ds = binding.model_struct(m), binding.data_struct(m, d)
    cs = binding.ctx_struct(ds, host_ctx(m, d), np.zeros(1, np.int32))
    cs.stats = None
    ds.nworld = 148 * per_sm
    if plan is not None:
        host = sparse_hessian.host_struct(plan)
        cs.sparse_plan = C.pointer(host)
    info = abi.ImnLaunchInfo()
    assert _lib.lib().imn_launch_info(C.byref(ms), C.byref(ds), C.byref(cs), C.byref(info)) == 0, _lib.lib().imn_last_error()
    assert info.worlds_per_cta == worlds


@pytest.mark.parametrize("nv,most", [(35, 6752), (64, 5688), (79, 4484)])
def test_the_largest_worlds_of_a_plan_stay_accepted(nv, most):
    """Host-only: what is staged beside the tables does not lower the row limit of a world."""
    import numpy as np

    from instantmimic_b200 import binding, synthetic
    from instantmimic_b200.mjw_kernels import sparse_hessian
    from instantmimic_b200.mjw_model import make_data, put_model
    from helpers import host_ctx

    parent, body = synthetic.limb_tree(nv)
    m = put_model(parent, body_of_dof=body)
    groups = [[b] for b in range(1, len(m.body_dofadr))]
    host = sparse_hessian.host_struct(sparse_hessian.build_plan(m, groups, 32 if m.nv_pad < 64 else 64, "fused"))
    for njmax, status in ((most, 0), (most + 1, abi.IMN_ERR_LIMIT)):
        d = make_data(m, 2, njmax)
        ms, ds = binding.model_struct(m), binding.data_struct(m, d)
        cs = binding.ctx_struct(ds, host_ctx(m, d), np.zeros(1, np.int32))
        cs.stats, cs.sparse_plan = None, C.pointer(host)
        info = abi.ImnLaunchInfo()
        assert _lib.lib().imn_launch_info(C.byref(ms), C.byref(ds), C.byref(cs), C.byref(info)) == status
        assert status or info.smem_bytes <= 227 * 1024


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_LIB", None)
    monkeypatch.setattr(_lib, "_PATH", tmp_path / "absent.so")
    with pytest.raises(_lib.ImnError, match="no CPU or PyTorch fallback"):
        _lib.lib()
