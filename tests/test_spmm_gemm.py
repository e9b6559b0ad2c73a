"""GeMM-SpMM in one launch on star stencils (csrc/spmm_gemm.cu).

Bound on the relative error: as in test_row_gemm.py for the shapes of the tensor-core tile, K / 8 * 3 sums cut off at 2^-23, 2e-6 up to
K = 256."""
import ctypes as C

import numpy as np
import pytest

from tests import common
from tests.test_gather import _scipy
from tile_fusion_b200 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _varying(t, seed=5):
    return t[0], t[1], np.random.default_rng(seed).uniform(-2, 2, len(t[2])).astype(np.float32)


def _run(plan, b, w, relu=False, wt=False):
    import torch
    d = torch.full((len(b), w.shape[1]), float("nan"), device="cuda")
    plan.gemm_spmm(torch.from_numpy(b).cuda(), torch.from_numpy(np.ascontiguousarray(w.T) if wt else w).cuda(), d, w_transposed=wt, relu=relu)
    plan.status()
    return d.cpu().numpy()


# bricks that fill the grid and that it cuts off on every side, lines shorter than a brick, an odd number of bricks, more bricks than
# CTAs; the last slice full, cut off and of four columns, every number of accumulators, the weight in shared memory and streamed
@pytest.mark.parametrize("dims", [(64, 64), (97, 83), (1030, 4), (5, 820), (203, 311), (32, 32, 32), (33, 37, 29), (5, 6, 1100), (900, 7, 6)])
@pytest.mark.parametrize("k,n_cols", [(4, 16), (32, 48), (68, 64), (100, 128), (36, 240), (160, 112), (256, 256)])
def test_grids(built_lib, dims, k, n_cols):
    t = synth.laplacian(dims)
    n = len(t[0]) - 1
    b, w = synth.uniform(3, (n, k)), synth.uniform(4, (k, n_cols))
    for relu, tr in ((False, t), (True, _varying(t))):
        want = _scipy(tr, n) @ (b.astype(np.float64) @ w.astype(np.float64))
        plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *tr), k=k, n_cols=n_cols)
        assert (plan.info()["threads"] == 480) == (len(dims) == 2 or 2 * k <= 3 * n_cols)
        got = _run(plan, b, w, relu, wt=relu)
        rel, _ = common.assert_close(got, np.maximum(want, 0) if relu else want, f"{dims} {k} {n_cols}")
        assert rel < 2e-6, rel
        dh = np.full((n, n_cols), np.nan, np.float32)
        plan.gemm_spmm_host(b, np.ascontiguousarray(w.T) if relu else w, dh, relu, relu)
        np.testing.assert_array_equal(dh, got)
        plan.close()


def test_operators_it_leaves(built_lib):
    """A neighbour left out, a nonzero too many, small grids: other executors, the same product."""
    t = synth.laplacian((80, 70))
    n = len(t[0]) - 1
    rows = np.repeat(np.arange(n), np.diff(t[0]))
    keep = ~((rows == 2000) & (t[1] == 2001))
    left_out = (np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=n))]).astype(np.int32), t[1][keep], t[2][keep])
    b, w = synth.uniform(3, (n, 32)), synth.uniform(4, (32, 64))
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *left_out), k=32, n_cols=64)
    assert plan.info()["threads"] != 480
    b[2001, 5] = np.inf
    assert np.isfinite(_run(plan, b, w)[2000]).all()
    plan.close()
    for dims in ((63, 65), (31, 32, 33)):
        m = int(np.prod(dims))
        plan = api.Plan("gemm_spmm", api.CSRMatrix(m, m, *synth.laplacian(dims)), k=32, n_cols=64)
        assert plan.info()["threads"] != 480
        plan.close()


@pytest.mark.parametrize("bits", [0x7FFFFFFF, 0x7F800001, 0x7F800000])
def test_numbers_that_are_none_stay_where_they_belong(built_lib, bits):
    """A NaN or an infinity in B makes a NaN (or an infinity) of the rows that name it and of no other; one in the weight, of its column."""
    t = _varying(synth.laplacian((70, 60)))
    n = len(t[0]) - 1
    A = _scipy(t, n)
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=40, n_cols=32)
    assert plan.info()["threads"] == 480
    b, w = synth.uniform(3, (n, 40)), synth.uniform(4, (40, 32))
    odd = np.array([bits], np.uint32).view(np.float32)[0]
    bn, wn = b.copy(), w.copy()
    bn[69, 39], bn[1717, 0], wn[3, 31] = odd, odd, odd
    hit = np.asarray((A[:, [69, 1717]] != 0).sum(1)).ravel() > 0
    np.testing.assert_array_equal(~np.isfinite(_run(plan, bn, w)), np.broadcast_to(hit[:, None], (n, 32)))
    got = ~np.isfinite(_run(plan, b, wn))
    assert got[:, 31].all() and not got[:, :31].any()
    plan.close()


def test_intermediate(built_lib):
    """Asked for T = B W, a plan leaves it from then on."""
    t = synth.laplacian((80, 70))
    n = len(t[0]) - 1
    b, w = synth.uniform(3, (n, 32)), synth.uniform(4, (32, 64))
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=32, n_cols=64)
    first = _run(plan, b, w)
    p, rows, cols = C.c_void_p(), C.c_longlong(), C.c_int()
    _lib.check(_lib.lib().tf_plan_intermediate(plan._h, C.byref(p), C.byref(rows), C.byref(cols)))
    assert p.value and rows.value == n and cols.value == 64 and plan.info()["threads"] != 480
    common.assert_close(_run(plan, b, w), first.astype(np.float64), "with T")
    import torch
    one = [torch.arange(n + 1, dtype=torch.int32, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda"), torch.ones(n, device="cuda")]
    out = torch.empty((n, 64), device="cuda")
    _lib.check(_lib.lib().tf_spmm_dev(*(q.data_ptr() for q in one[:3]), n, p.value, 64, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    common.assert_close(out.cpu().numpy(), b.astype(np.float64) @ w.astype(np.float64), "T")
    plan.close()


# thin grids, bricks of which much lies outside: an operator whose coefficients differ is left to the gather earlier
@pytest.mark.parametrize("dims,k,n_cols,uniform,varying", [((5, 60_000), 256, 32, True, False), ((5, 60_000), 64, 64, True, True), ((9, 40_000), 256, 32, True, True),
                                                           ((5, 4000), 256, 32, True, True), ((5, 2, 30_000), 256, 256, True, False),
                                                           ((5, 5, 12_000), 80, 64, True, False), ((5, 6, 10_000), 64, 64, True, True),
                                                           ((5, 5, 12_000), 24, 16, True, True), ((40, 40, 40), 96, 64, True, True)])
def test_thin_grids(built_lib, dims, k, n_cols, uniform, varying):
    t = synth.laplacian(dims)
    n = len(t[0]) - 1
    b, w = synth.uniform(3, (n, k)), synth.uniform(4, (k, n_cols))
    for tr, one in ((t, uniform), (_varying(t), varying)):
        plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *tr), k=k, n_cols=n_cols)
        assert (plan.info()["threads"] == 480) == one
        rel, _ = common.assert_close(_run(plan, b, w), _scipy(tr, n) @ (b.astype(np.float64) @ w.astype(np.float64)), f"{dims} {k} {n_cols}")
        assert rel < 2e-6, rel
        plan.close()


def test_rows_of_the_intermediate(built_lib):
    """A plan that keeps no intermediate says so."""
    t = synth.laplacian((80, 70))
    n = len(t[0]) - 1
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=32, n_cols=64)
    assert plan.info()["intermediate_rows"] == 0
    _lib.check(_lib.lib().tf_plan_intermediate(plan._h, None, None, None))
    assert plan.info()["intermediate_rows"] == n
    plan.close()
