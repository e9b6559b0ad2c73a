"""The plane-marching kernel on 3-D grids with an odd x extent and on widths off the multiples of four: the points with even and with odd x come
through maps of their own, and rows of T that do not exist are zero.  Bit for bit the CSR products."""
import numpy as np
import pytest

from tests import common
from tests.test_gather import _scipy
from tests.test_line_march import _csr
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


# the odd column at every place a 16-wide tile with two points of rim can have it, the last line likewise (tiles of 8)
@pytest.mark.parametrize("dims", [(9, 8, 7), (15, 9, 3), (17, 10, 5), (19, 16, 3), (31, 7, 20), (33, 17, 9), (101, 66, 5)])
@pytest.mark.parametrize("n_cols", [4, 48, 100])
def test_odd_extent(built_lib, dims, n_cols):
    import torch
    a = synth.laplacian(dims)
    n = len(a[0]) - 1
    rows = np.repeat(np.arange(n), np.diff(a[0]))
    b = (a[0], a[1], (a[2] * (1.0 + (rows % 2)) * np.where(a[1] > rows, 0.5, 1.0)).astype(np.float32))
    c = synth.uniform(3, (n, n_cols))
    # the operand ends with its allocation's last row; rows behind it would be seen as what they are
    big = torch.full((n + 64, n_cols), float("nan"), device="cuda")
    cd = big[:n].copy_(torch.from_numpy(c))
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
        plan.close()
        ref.close()


@pytest.mark.parametrize("dims", [(17, 10, 9), (33, 9, 6)])
def test_infinities_stay_where_they_are(built_lib, dims):
    """Rows of the intermediate beyond the grid are zero and not multiplied by it."""
    import torch
    n_cols = 32
    t = synth.laplacian(dims)
    n = len(t[0]) - 1
    t = (t[0], t[1], np.abs(t[2]))
    plane = dims[0] * dims[1]
    c = np.abs(synth.uniform(3, (n, n_cols)))
    c[[0, dims[0] - 1, plane - 1, 3 * plane, 4 * plane + 5 * dims[0] - 1, n - plane, n - 1]] = np.inf
    plan = api.Plan("spmm_spmm", _csr(t), n_cols=n_cols)
    assert plan.info()["threads"] == 128
    d = torch.empty((n, n_cols), device="cuda")
    plan.spmm_spmm(torch.from_numpy(c).cuda(), d)
    plan.status()
    A = _scipy(t, n)
    want = A @ (A @ c.astype(np.float64))
    got = d.cpu().numpy()
    np.testing.assert_array_equal(np.isinf(got), np.isinf(want))
    assert not np.isnan(got).any()
    plan.close()


# widths off the multiples of four march from a padded copy: either parity of x, the narrowest taken and the one below it, a last
# chunk of one column, operands off the 16-byte grid, infinities on the rim
@pytest.mark.parametrize("dims", [(16, 8, 7), (33, 17, 9), (18, 11, 4)])
@pytest.mark.parametrize("n_cols", [3, 5, 33, 47])
def test_widths_off_the_multiples_of_four(built_lib, dims, n_cols):
    import torch
    a = synth.laplacian(dims)
    n = len(a[0]) - 1
    rows = np.repeat(np.arange(n), np.diff(a[0]))
    b = (a[0], a[1], (a[2] * (1.0 + (rows % 2)) * np.where(a[1] > rows, 0.5, 1.0)).astype(np.float32))
    c = torch.from_numpy(synth.uniform(3, (n, n_cols))).cuda()
    ci = c.clone()
    ci[[0, dims[0] - 1, dims[0] * dims[1] - 1, n - 1]] = float("inf")
    for B in (None, _csr(b)):
        plan = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols)
        assert (plan.info()["threads"] == 128) == (n_cols >= 5)
        ref = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols, mode=api.MODE_UNFUSED, tile_slots=-1, lattice_march=-1)
        for x in (c, ci):
            xu = torch.empty(n * n_cols + 1, device="cuda")[1:].view(n, n_cols).copy_(x)
            du = torch.full((n * n_cols + 3,), float("nan"), device="cuda")
            d = du[1:-2].view(n, n_cols)
            plan.spmm_spmm(xu, d)
            plan.status()
            d0 = torch.empty((n, n_cols), device="cuda")
            ref.spmm_spmm(x, d0)
            ref.status()
            assert torch.equal(torch.nan_to_num(d, nan=7.0), torch.nan_to_num(d0, nan=7.0))
            assert torch.isnan(du[[0, -2, -1]]).all()
        dh = np.full((n, n_cols), np.nan, np.float32)
        plan.spmm_spmm_host(c.cpu().numpy(), dh)
        plan.spmm_spmm(c, d)
        np.testing.assert_array_equal(dh, d.cpu().numpy())
        plan.close()
        ref.close()


# cross-sections of which the tiles find little, and widths of which the chunks do: the gather, and the same bits
@pytest.mark.parametrize("dims,n_cols,marches", [((2, 2, 9000), 33, False), ((2, 2, 9000), 5, False), ((10, 10, 400), 47, False), ((4, 4, 500), 33, False),
                                                 ((12, 6, 500), 18, False), ((12, 6, 500), 99, True), ((12, 6, 500), 13, True), ((20, 12, 90), 7, True),
                                                 ((24, 24, 60), 18, True), ((9, 9, 250), 7, False), ((40, 33, 20), 35, True),
                                                 ((20, 20, 20), 47, False), ((17, 17, 17), 33, False), ((40, 4, 9), 33, True)])
def test_ragged_widths_on_thin_grids(built_lib, dims, n_cols, marches):
    import torch
    a = _csr(synth.laplacian(dims))
    c = torch.from_numpy(synth.uniform(3, (int(np.prod(dims)), n_cols))).cuda()
    out = []
    for kw in ({}, dict(mode=api.MODE_UNFUSED, tile_slots=-1, lattice_march=-1)):
        plan = api.Plan("spmm_spmm", a, n_cols=n_cols, **kw)
        if not kw:
            assert (plan.info()["threads"] == 128) == marches
        out.append(torch.full_like(c, float("nan")))
        plan.spmm_spmm(c, out[-1])
        plan.status()
        plan.close()
    assert torch.equal(*out)
