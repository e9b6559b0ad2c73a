"""The balanced gather of operators without row reuse (csrc/gather.cu, gather_plan.cpp) against an fp64 product.

An fp32 sum of k products in order has a relative error below k * 2^-24 of the sum of the magnitudes; the rows here have
at most 5 000 nonzeros and random signs, for which the tolerance of tests/common.py leaves an order of magnitude."""
import numpy as np
import pytest

from tests import common
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


def _graph(n, seed, empty=(), hubs=()):
    """Random rows of 0 .. 9 nonzeros, some rows emptied, some with most columns."""
    rng = np.random.default_rng(seed)
    rows = []
    for r in range(n):
        k = 0 if r in empty else int(rng.integers(0, 10))
        rows.append(np.sort(rng.choice(n, size=min(n, k), replace=False)))
    for r, k in hubs:
        rows[r] = np.sort(rng.choice(n, size=k, replace=False))
    ap = np.zeros(n + 1, np.int32)
    ap[1:] = np.cumsum([len(r) for r in rows])
    ai = np.concatenate(rows).astype(np.int32)
    return ap, ai, rng.uniform(-1, 1, len(ai)).astype(np.float32)


def _scipy(t, n):
    import scipy.sparse as sp
    return sp.csr_matrix((t[2].astype(np.float64), t[1], t[0]), shape=(n, n))


# widths: each group size (8, 16, 32 lanes), a second panel, widths that are no multiple of four, one column
@pytest.mark.parametrize("n_cols", [1, 4, 31, 32, 33, 64, 68, 128, 132, 300])
def test_gather_chain(built_lib, n_cols):
    import torch
    n = 5000
    # hubs around the lengths at which a row is cut (a multiple of the unit size) and far above
    t = _graph(n, 3, empty={0, 1, 2, n - 1}, hubs=((5, 5000), (17, 63), (18, 64), (19, 65), (4000, 256), (4001, 513)))
    f = _graph(n, 4, hubs=((n - 1, 700),))
    A, F = api.CSRMatrix(n, n, *t), api.CSRMatrix(n, n, *f)
    c = synth.uniform(3, (n, n_cols))
    cd = torch.from_numpy(c).cuda()
    for first, B in ((t, None), (f, F)):
        want = _scipy(t, n) @ (_scipy(first, n) @ c.astype(np.float64))
        plan = api.Plan("spmm_spmm", A, B=B, n_cols=n_cols)
        assert plan.info()["launches"] == 0 and plan.info()["items"] == 0  # no ticket list: the gather was chosen
        d = torch.full((n, n_cols), float("nan"), device="cuda")
        plan.spmm_spmm(cd, d)
        first_bits = d.clone()
        d.fill_(float("nan"))
        plan.spmm_spmm(cd, d)  # the counters of cut rows must be back at zero
        plan.status()
        assert torch.equal(d, first_bits)  # pieces of a row are added in order: same bits every time
        common.assert_close(d.cpu().numpy(), want, f"gather N={n_cols}")
        # operands off the 16-byte grid
        cu = torch.empty(n * n_cols + 1, device="cuda")[1:].view(n, n_cols).copy_(cd)
        du = torch.full((n * n_cols + 1,), float("nan"), device="cuda")[1:].view(n, n_cols)
        plan.spmm_spmm(cu, du)
        plan.status()
        assert torch.equal(du, first_bits)
        dh = np.full((n, n_cols), np.nan, np.float32)
        plan.spmm_spmm_host(c, dh)
        assert np.array_equal(dh, d.cpu().numpy())
        plan.close()


def test_infinities_stay_where_they_are(built_lib):
    """The entries that fill up a unit have value 0 and name the unit's last column again: where that column holds an
    infinity, their product is no number and must not reach a row, long ones (cut into pieces) included."""
    import torch
    n, w = 5000, 32
    t = _graph(n, 8, hubs=((5, 5000), (40, 333), (41, 65)))
    ap, ai, ax = t
    ax = np.abs(ax) + 0.5
    c = np.abs(synth.uniform(3, (n, w)))
    c[ai[ap[1:] - 1][::7]] = np.inf  # the last column of every seventh row
    plan = api.Plan("spmm_spmm", api.CSRMatrix(n, n, ap, ai, ax), n_cols=w)
    d = torch.empty((n, w), device="cuda")
    plan.spmm_spmm(torch.from_numpy(c).cuda(), d)
    plan.status()
    A = _scipy((ap, ai, ax), n)
    want = A @ (A @ c.astype(np.float64))
    got = d.cpu().numpy()
    np.testing.assert_array_equal(np.isinf(got), np.isinf(want))
    assert not np.isnan(got).any()
    plan.close()


@pytest.mark.parametrize("kind,n_cols", [("grid", 33), ("grid", 47), ("band", 47), ("two", 30), ("gaps", 41)])
def test_host_call_in_pieces(built_lib, kind, n_cols):
    """Host pointers on operators that name rows near their own, at widths that no march takes: the call runs in pieces, so that
    copies and products overlap, and gives the bits of the device call.  Two operators of different reach; rows without nonzeros."""
    import torch
    n = 30_000
    if kind == "grid":
        t = synth.laplacian((32, 30, 31))
        n = len(t[0]) - 1
    else:
        rng = np.random.default_rng(2)

        def band(reach, per_row, empty=0):
            r = np.repeat(np.arange(n), per_row)
            c = np.clip(r + rng.integers(-reach, reach + 1, len(r)), 0, n - 1)
            key = np.unique(r.astype(np.int64) * n + c)
            key = key[(key // n) % 11 >= empty]
            ap = np.concatenate([[0], np.cumsum(np.bincount(key // n, minlength=n))]).astype(np.int32)
            return ap, (key % n).astype(np.int32), rng.uniform(-1, 1, len(key)).astype(np.float32)
        t = band(40, 12, empty=3 if kind == "gaps" else 0)
    A = api.CSRMatrix(n, n, *t)
    F = api.CSRMatrix(n, n, *band(300, 5, empty=2)) if kind == "two" else None
    c = synth.uniform(3, (n, n_cols))
    plan = api.Plan("spmm_spmm", A, B=F, n_cols=n_cols)
    d = torch.full((n, n_cols), float("nan"), device="cuda")
    plan.spmm_spmm(torch.from_numpy(c).cuda(), d)
    plan.status()
    for _ in range(2):
        dh = np.full((n, n_cols), np.nan, np.float32)
        plan.spmm_spmm_host(c, dh)
        assert plan.info()["launches"] > 16
        np.testing.assert_array_equal(dh, d.cpu().numpy())
    first = _scipy(t if F is None else (F.Ap, F.Ai, F.Ax), n)
    common.assert_close(dh, _scipy(t, n) @ (first @ c.astype(np.float64)), kind)
    plan.close()
