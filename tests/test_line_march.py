"""The line-marching executor of 2-D five-point operators (csrc/line_march.cu): bit for bit the CSR products in order."""
import numpy as np
import pytest

from tests.test_gather import _scipy
from tests import common
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


def _csr(t):
    n = len(t[0]) - 1
    return api.CSRMatrix(n, n, *t)


# lines around the 28 points that a warp completes, two lines, a column of one tile, several segments along y
@pytest.mark.parametrize("dims", [(3, 2), (27, 5), (28, 9), (29, 40), (57, 33), (200, 150), (8, 700)])
@pytest.mark.parametrize("n_cols", [1, 4, 16, 20, 47, 64, 100])
def test_line_march(built_lib, dims, n_cols):
    import torch
    a = synth.laplacian(dims)
    n = len(a[0]) - 1
    rows = np.repeat(np.arange(n), np.diff(a[0]))
    b = (a[0], a[1], (a[2] * (1.0 + (rows % 2)) * np.where(a[1] > rows, 0.5, 1.0)).astype(np.float32))
    c = synth.uniform(3, (n, n_cols))
    cd = torch.from_numpy(c).cuda()
    for first, B in ((a, None), (b, _csr(b))):
        plan = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols)
        assert plan.info()["threads"] == 128, plan.info()
        d = torch.full((n, n_cols), float("nan"), device="cuda")
        for _ in range(2):
            plan.spmm_spmm(cd, d)
        plan.status()
        common.assert_close(d.cpu().numpy(), _scipy(a, n) @ (_scipy(first, n) @ c.astype(np.float64)), f"{dims} {n_cols}")
        ref = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols, mode=api.MODE_UNFUSED, tile_slots=-1, lattice_march=-1)
        d0 = torch.empty_like(d)
        ref.spmm_spmm(cd, d0)
        ref.status()
        assert torch.equal(d, d0)
        dh = np.full((n, n_cols), np.nan, np.float32)
        plan.spmm_spmm_host(c, dh)
        np.testing.assert_array_equal(dh, d.cpu().numpy())
        if n_cols % 4:  # operands off the 16-byte grid are taken where rows are read value by value
            cu = torch.empty(n * n_cols + 1, device="cuda")[1:].view(n, n_cols).copy_(cd)
            du = torch.full((n * n_cols + 1,), float("nan"), device="cuda")[1:].view(n, n_cols)
            plan.spmm_spmm(cu, du)
            plan.status()
            assert torch.equal(du, d)
        plan.close()
        ref.close()


# grids whose segments are long enough that warps ask L2 for lines ahead: to the grid's last line, a ragged last chunk of columns
@pytest.mark.parametrize("dims,n_cols", [((611, 280), 100), ((1023, 331), 64), ((300, 701), 128)])
def test_segments_that_read_ahead(built_lib, dims, n_cols):
    import torch
    a = synth.laplacian(dims)
    n = len(a[0]) - 1
    rows = np.repeat(np.arange(n), np.diff(a[0]))
    b = (a[0], a[1], (a[2] * (1.0 + (rows % 2))).astype(np.float32))
    c = torch.from_numpy(synth.uniform(3, (n, n_cols))).cuda()
    for B in (None, _csr(b)):
        out = []
        for kw in ({}, dict(mode=api.MODE_UNFUSED, tile_slots=-1, lattice_march=-1)):
            plan = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols, **kw)
            d = torch.full((n, n_cols), float("nan"), device="cuda")
            plan.spmm_spmm(c, d)
            plan.status()
            out.append(d)
            plan.close()
        assert torch.equal(*out)


def test_infinities_stay_where_they_are(built_lib):
    """Rows beyond the grid are zero and not multiplied by it: infinities on the rim reach their neighbours only."""
    import torch
    dims, n_cols = (57, 30), 64
    t = synth.laplacian(dims)
    n = len(t[0]) - 1
    t = (t[0], t[1], np.abs(t[2]))
    c = np.abs(synth.uniform(3, (n, n_cols)))
    c[[0, 20, 56, 57 * 10, 57 * 11 - 1, n - 57, n - 1]] = np.inf
    plan = api.Plan("spmm_spmm", _csr(t), n_cols=n_cols)
    d = torch.empty((n, n_cols), device="cuda")
    plan.spmm_spmm(torch.from_numpy(c).cuda(), d)
    plan.status()
    A = _scipy(t, n)
    want = A @ (A @ c.astype(np.float64))
    got = d.cpu().numpy()
    np.testing.assert_array_equal(np.isinf(got), np.isinf(want))
    assert not np.isnan(got).any()
    plan.close()


def test_other_operators_are_declined(built_lib):
    """A neighbour missing inside the grid, a column that is none, too many coefficient vectors: the general paths."""
    base = synth.laplacian((40, 20))
    n = 800
    S = _scipy(base, n).tolil()
    for edit in ("missing", "extra", "values"):
        T = S.copy()
        if edit == "missing":
            T[100, 101] = 0
        elif edit == "extra":
            T[100, 103] = 1
        T = T.tocsr()
        T.eliminate_zeros()
        T.sort_indices()
        data = T.data.astype(np.float32)
        if edit == "values":
            data = data * (1 + np.arange(len(data)) % 97).astype(np.float32)
        plan = api.Plan("spmm_spmm", api.CSRMatrix(n, n, T.indptr.astype(np.int32), T.indices.astype(np.int32), data), n_cols=32)
        assert plan.info()["threads"] != 128
        plan.close()


@pytest.mark.parametrize("dims,taken", [((1000, 2), True), ((511, 2), True), ((400, 2), False), ((1000, 3), False)])
def test_two_long_lines_off_the_16_byte_grid(built_lib, dims, taken):
    """Two long lines have no reuse that a gather tile could hold, and the executor that takes such operators reads rows wherever
    they lie: so does this one.  Where tiles would be taken, operands off the 16-byte grid are refused as they ask."""
    import torch
    from tile_fusion_b200 import _lib
    t = synth.laplacian(dims)
    n, w = len(t[0]) - 1, 32
    plan = api.Plan("spmm_spmm", _csr(t), n_cols=w)
    old = api.Plan("spmm_spmm", _csr(t), n_cols=w, lattice_march=-1)
    assert plan.info()["threads"] == 128
    c = torch.from_numpy(synth.uniform(3, (n, w))).cuda()
    d = torch.empty((n, w), device="cuda")
    plan.spmm_spmm(c, d)
    cu = torch.empty(n * w + 1, device="cuda")[1:].view(n, w).copy_(c)
    du = torch.full((n * w + 1,), float("nan"), device="cuda")[1:].view(n, w)
    for p in (plan, old):
        if taken:
            p.spmm_spmm(cu, du)
            p.status()
            assert torch.equal(du, d)
            du.fill_(float("nan"))
        else:
            with pytest.raises(_lib.TileFusionError) as e:
                p.spmm_spmm(cu, du)
            assert e.value.code == _lib.TF_ERR_ARG
        p.close()
