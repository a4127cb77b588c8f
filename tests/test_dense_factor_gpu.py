"""Blocked dense factor + solve around the edges of its launch rules: the column counts where the
two-group kernel ends (64), right-hand sides around the groups they are solved in, and a workspace that
does not lie on a 16-byte boundary."""

import numpy as np
import pytest

from instantmimic_b200 import mjw_model
from instantmimic_b200.mjw_kernels import indexed_factor

from test_msolve import _blocked_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv,rhs,offset", [(63, 1, 0), (64, 1, 0), (60, 4, 1), (33, 5, 1), (34, 9, 0), (48, 18, 3)])
def test_dense_factor_edges(oracle, cuda_device, nv, rhs, offset):
    import torch

    worlds = 10
    m, Mv, _, pad, layout, ident, y = _blocked_case(nv, worlds, rhs)
    md = mjw_model.to_device(m, cuda_device)
    dd = mjw_model.to_device(mjw_model.make_data(m, worlds, 4), cuda_device)
    scratch = indexed_factor.create_blocked_dense_factor_solve_scratch(md, dd, cuda_device)
    Mt, yt = torch.from_numpy(Mv).to(cuda_device), torch.from_numpy(y).to(cuda_device)
    active = torch.ones(worlds, dtype=torch.int32, device=cuda_device)
    x, x2 = torch.zeros_like(yt), torch.zeros_like(yt)
    U = torch.zeros(worlds * pad * pad + 4, device=cuda_device)[offset:offset + worlds * pad * pad].view(worlds, pad, pad)
    indexed_factor.factor_multi_solve(scratch, Mt, yt, active, U, x, rhs)
    indexed_factor.multi_solve(scratch, U, yt, active, x2, rhs)
    want_x, want_U = oracle.blocked_dense_factor_solve(nv, pad, layout, ident, Mv, y)
    np.testing.assert_array_equal(x.cpu().numpy(), want_x)
    np.testing.assert_array_equal(x2.cpu().numpy(), want_x)
    np.testing.assert_array_equal(U.cpu().numpy(), want_U)


@pytest.mark.parametrize("places", [True, False])
@pytest.mark.parametrize("nv,rhs", [(33, 1), (36, 28), (36, 29), (37, 3), (52, 2), (80, 1)])
def test_last_block_and_entry_places(oracle, cuda_device, nv, rhs, places):
    """Last blocks of one, four and five rows, with as many columns as the narrow form takes and one more; M's entries
    laid out by their places and looked up position by position."""
    import torch

    worlds = 7
    m, Mv, _, pad, layout, ident, y = _blocked_case(nv, worlds, rhs)
    md = mjw_model.to_device(m, cuda_device)
    dd = mjw_model.to_device(mjw_model.make_data(m, worlds, 4), cuda_device)
    scratch = indexed_factor.create_blocked_dense_factor_solve_scratch(md, dd, cuda_device)
    if not places:
        scratch.struct.places = None
    Mt, yt = torch.from_numpy(Mv).to(cuda_device), torch.from_numpy(y).to(cuda_device)
    active = torch.ones(worlds, dtype=torch.int32, device=cuda_device)
    active[3] = 0
    x, x2, U = torch.zeros_like(yt), torch.zeros_like(yt), torch.full((worlds, pad, pad), 7.0, device=cuda_device)
    indexed_factor.factor_multi_solve(scratch, Mt, yt, active, U, x, rhs)
    indexed_factor.multi_solve(scratch, U, yt, active, x2, rhs)
    want_x, want_U = oracle.blocked_dense_factor_solve(nv, pad, layout, ident, Mv, y)
    want_x[3], want_U[3] = 0.0, 7.0
    np.testing.assert_array_equal(x.cpu().numpy(), want_x)
    np.testing.assert_array_equal(x2.cpu().numpy(), want_x)
    np.testing.assert_array_equal(U.cpu().numpy(), want_U)


@pytest.mark.parametrize("filler", [0.0, 9.0])
@pytest.mark.parametrize("places", [True, False])
def test_rows_of_m_wider_than_their_entries(oracle, cuda_device, places, filler):
    import torch

    nv, rhs, worlds = 34, 2, 5
    m, Mv, _, pad, layout, ident, y = _blocked_case(nv, worlds, rhs)
    md = mjw_model.to_device(m, cuda_device)
    d = mjw_model.make_data(m, worlds, 4)
    d.M = np.concatenate([Mv, np.full((worlds, 2), filler, np.float32)], 1)
    dd = mjw_model.to_device(d, cuda_device)
    scratch = indexed_factor.create_blocked_dense_factor_solve_scratch(md, dd, cuda_device)
    if not places:
        scratch.struct.places = None
    yt = torch.from_numpy(y).to(cuda_device)
    x, x2 = torch.zeros_like(yt), torch.zeros_like(yt)
    indexed_factor.factor_multi_solve(scratch, dd.M, yt, None, scratch.U, x, rhs)
    indexed_factor.multi_solve(scratch, scratch.U, yt, None, x2, rhs)
    want_x, want_U = oracle.blocked_dense_factor_solve(nv, pad, layout, ident, Mv, y)
    np.testing.assert_array_equal(x.cpu().numpy(), want_x)
    np.testing.assert_array_equal(x2.cpu().numpy(), want_x)
    np.testing.assert_array_equal(scratch.U.cpu().numpy(), want_U)


def test_entry_places_are_the_index_table_the_other_way_round():
    m = _blocked_case(35, 1, 1)[0]
    table = indexed_factor.dense_index_table(m)
    places = indexed_factor.entry_places(table, int(m.nM))
    rows, cols = places & 0xFF, places >> 8
    assert (rows <= cols).all() and np.array_equal(table[rows, cols], np.arange(m.nM))
