"""GeMM-SpMM on the dense product of its own launch (csrc/row_gemm.cu) and the balanced gather, in either order.

Bounds on the relative error, beside the tolerance of tests/common.py: shapes of the tensor-core tile (K a multiple of 4, N
of 16) add K / 8 * 3 sums that are cut off at 2^-23: 2e-6 up to K = 256, as in test_gpu_tc.py.  All others are fp32
FMAs up to 31 terms and as exact as those beyond: per eight terms one sum cut off at 2^-23, then K / 8 rounded sums, each of random sign against the rest, and the
dropped lo * lo terms at 2^-22 of a product: below 2^-22 + 2^-24 * sqrt(K / 8) < 6e-7 up to K = 300."""
import numpy as np
import pytest

from tests import common
from tests.test_gather import _graph, _scipy
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


def _check(t, n, k, n_cols, seed, off=0, wt=False, relu=False, plan=None):
    import torch
    b, w = synth.uniform(seed, (n, k)), synth.uniform(seed + 1, (k, n_cols))
    want = _scipy(t, n) @ (b.astype(np.float64) @ w.astype(np.float64))
    if relu:
        want = np.maximum(want, 0)
    plan = plan or api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=k, n_cols=n_cols)
    bd = torch.empty(n * k + off, device="cuda")[off:].view(n, k).copy_(torch.from_numpy(b))
    wd = torch.from_numpy(np.ascontiguousarray(w.T) if wt else w).cuda()
    d = torch.full((n * n_cols + off,), float("nan"), device="cuda")[off:].view(n, n_cols)
    plan.gemm_spmm(bd, wd, d, w_transposed=wt, relu=relu)
    plan.status()
    rel, _ = common.assert_close(d.cpu().numpy(), want, f"{n}x{k}x{n_cols} off={off}")
    assert rel < (2e-6 if k % 4 == 0 and n_cols % 16 == 0 else 6e-7), rel
    return plan, b, w, d


# rows around a CTA's half tile, a pair's tile and a whole wave of pairs; K and N around the 32-column slices
@pytest.mark.parametrize("m", [1, 127, 129, 255, 257, 74 * 256 + 1])
@pytest.mark.parametrize("k,n_cols", [(4, 1), (32, 256), (36, 33), (256, 47), (17, 64), (300, 225)])
def test_dense_product_sizes(built_lib, m, k, n_cols):
    """The operator is a scaled permutation, so that D is the dense product."""
    rng = np.random.default_rng(m + k)
    t = (np.arange(m + 1, dtype=np.int32), rng.permutation(m).astype(np.int32), rng.uniform(1, 2, m).astype(np.float32))
    _check(t, m, k, n_cols, 3, wt=(m + k) % 2 == 1, relu=m % 2 == 0)[0].close()


@pytest.mark.parametrize("k,n_cols", [(64, 40), (40, 64), (100, 256), (256, 47), (33, 128), (8, 7)])
def test_graph_in_either_order(built_lib, k, n_cols):
    n = 3000
    t = _graph(n, 5, empty={0, 7, n - 1}, hubs=((9, 3000), (11, 257)))
    plan, b, w, d = _check(t, n, k, n_cols, 3)
    dh = np.full((n, n_cols), np.nan, np.float32)
    plan.gemm_spmm_host(b, w, dh)
    np.testing.assert_array_equal(dh, d.cpu().numpy())
    if k % 4 or n_cols % 16:  # operands off the 16-byte grid: taken where the shape does not ask for vectors
        _check(t, n, k, n_cols, 3, off=1, plan=plan)
    plan.close()


@pytest.mark.parametrize("dims,k,n_cols", [((90, 70), 64, 64), ((90, 70), 20, 47), ((31, 30, 12), 100, 32), ((32, 30, 12), 36, 48)])
def test_grid_host_call_in_pieces(built_lib, dims, k, n_cols):
    """Host pointers on operators that name rows near their own: the call runs in pieces and gives the same bits."""
    t = synth.laplacian(dims)
    n = len(t[0]) - 1
    plan, b, w, d = _check(t, n, k, n_cols, 3)
    dh = np.full((n, n_cols), np.nan, np.float32)
    for _ in range(2):
        plan.gemm_spmm_host(b, w, dh)
        np.testing.assert_array_equal(dh, d.cpu().numpy())
    plan.close()
    _check(t, n, k, n_cols, 3, relu=True)[0].close()


@pytest.mark.parametrize("dims", [(16, 8, 2), (18, 9, 5), (17, 10, 9), (33, 17, 6), (101, 66, 3)])
@pytest.mark.parametrize("k,n_cols", [(64, 64), (20, 100), (17, 4), (128, 256)])
def test_grid_one_product_march(built_lib, dims, k, n_cols):
    """3-D grids: the sparse product on the one-product march.  Bit for bit the balanced gather (the same dense product in
    front of either), even and odd x extents, with and without the ReLU, tiles and chunks cut off by the grid and the width."""
    import torch
    t = synth.laplacian(dims)
    n = len(t[0]) - 1
    A = api.CSRMatrix(n, n, *t)
    b, w = torch.from_numpy(synth.uniform(5, (n, k))).cuda(), torch.from_numpy(synth.uniform(6, (k, n_cols))).cuda()
    plans = [api.Plan("gemm_spmm", A, k=k, n_cols=n_cols, lattice_march=lm) for lm in (0, -1)]
    assert plans[0].info()["threads"] == 128 and plans[1].info()["threads"] != 128
    for relu in (False, True):
        out = []
        for p in plans:
            d = torch.full((n, n_cols), float("nan"), device="cuda")
            for _ in range(2):
                p.gemm_spmm(b, w, d, relu=relu)
            p.status()
            out.append(d)
        assert torch.equal(*out)
        want = _scipy(t, n) @ (b.double() @ w.double()).cpu().numpy()
        common.assert_close(out[0].cpu().numpy(), np.maximum(want, 0) if relu else want, f"{dims} {k} {n_cols}")
    for p in plans:
        p.close()


# both forms of the dense product, the sparse product in front of it, and the ticket executor's tile
@pytest.mark.parametrize("k,n_cols,opts", [(64, 64, {}), (128, 256, {}), (64, 47, {}), (33, 64, {}), (32, 64, {}), (64, 64, {"ctas_per_sm": 1})])
@pytest.mark.parametrize("bits", [0x7FFFFFFF, 0xFFFFFFFF, 0x7FC00000, 0x7F800001])
def test_nan_stays_nan(built_lib, k, n_cols, opts, bits):
    """A NaN of any payload -- 0x7FFFFFFF is the one that arithmetic on the GPU gives -- in B, in the weight, or made by the
    gather in front of the dense product (0 * infinity) makes a NaN of every result that it enters, and of no other."""
    import torch
    n = 700
    ap, ai, ax = _graph(n, 5, empty={0, n - 1}, hubs=((9, 600),))
    hole = int(ai[ap[20]])  # row 20 multiplies the row of B that holds infinities by a zero
    ax[ap[20]] = 0.0
    A = _scipy((ap, ai, ax), n)
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, ap, ai, ax), k=k, n_cols=n_cols, **opts)
    b, w = torch.from_numpy(synth.uniform(3, (n, k))).cuda(), torch.from_numpy(synth.uniform(4, (k, n_cols))).cuda()
    nan = torch.tensor([bits - (1 << 32) if bits >> 31 else bits], dtype=torch.int32, device="cuda").view(torch.float32)

    def run(b, w):
        d = torch.zeros((n, n_cols), device="cuda")
        plan.gemm_spmm(b, w, d)
        plan.status()
        return d.cpu().numpy()

    bn = b.clone()
    bn[5, k - 1:], bn[300, 3:4] = nan, nan
    hit = np.zeros(n, bool)
    for r in (5, 300):
        hit |= np.asarray((A[:, [r]] != 0).todense()).ravel()
    hit |= np.isin(np.arange(n), [20]) & (hole in (5, 300))
    got = run(bn, w)
    np.testing.assert_array_equal(np.isnan(got), np.broadcast_to(hit[:, None], got.shape))
    wn = w.clone()
    wn[2, n_cols - 1:] = nan
    got = run(b, wn)
    want = np.zeros(got.shape, bool)
    want[np.diff(ap) > 0, n_cols - 1] = True
    np.testing.assert_array_equal(np.isnan(got), want)
    bi = b.clone()
    bi[hole, 1] = float("inf")
    assert np.isnan(run(bi, w)[20]).all()
    plan.close()


# fewer terms than the precise form is taken for, and shapes the tensor-core tile does not take: FMAs in the order of the terms
@pytest.mark.parametrize("k,n_cols", [(1, 1), (3, 64), (17, 16), (17, 256), (31, 225), (28, 20), (8, 7)])
@pytest.mark.parametrize("m", [1, 127, 130, 80_011])
def test_few_terms_are_fmas(built_lib, m, k, n_cols):
    """Bit for bit the ticket executor's CUDA-core tile (n_cols <= k or k off the multiples of four: no sparse product in front),
    infinities included, on rows and results off the 16-byte grid too."""
    import torch
    rng = np.random.default_rng(m + k)
    t = (np.arange(m + 1, dtype=np.int32), rng.permutation(m).astype(np.int32), rng.uniform(1, 2, m).astype(np.float32))
    b, w = synth.uniform(3, (m, k)), synth.uniform(4, (k, n_cols))
    b[m // 2, k - 1], w[0, 0] = np.inf, -np.inf
    A = api.CSRMatrix(m, m, *t)
    for off, wt, relu in ((0, False, False), (1, True, True)):
        bd = torch.empty(m * k + off, device="cuda")[off:].view(m, k).copy_(torch.from_numpy(b))
        wd = torch.from_numpy(np.ascontiguousarray(w.T) if wt else w).cuda()
        out = []
        for opts in ({"tile_slots": -1}, {"tile_slots": -1, "tensor_cores": -1}):
            plan = api.Plan("gemm_spmm", A, k=k, n_cols=n_cols, **opts)
            out.append(torch.full((m * n_cols + off,), 7.0, device="cuda")[off:].view(m, n_cols))
            plan.gemm_spmm(bd, wd, out[-1], w_transposed=wt, relu=relu)
            plan.status()
            plan.close()
        assert torch.equal(torch.isnan(out[0]), torch.isnan(out[1]))
        assert torch.equal(out[0].nan_to_num(), out[1].nan_to_num())


@pytest.mark.parametrize("m,k,n_cols,off", [(700, 33, 128, 0), (700, 64, 47, 0), (129, 36, 33, 1), (300, 300, 225, 0), (1, 50, 70, 1)])
def test_infinities_of_the_precise_form(built_lib, m, k, n_cols, off):
    """Shapes that FMAs always took: an infinity in B or in the weight, and a number that rounds to one in TF32, give what FMAs
    give -- the infinity, the finite sum, no number only where infinities meet their negatives or a zero."""
    import torch
    rng = np.random.default_rng(m + k)
    t = (np.arange(m + 1, dtype=np.int32), rng.permutation(m).astype(np.int32), np.ones(m, np.float32))
    b, w = synth.uniform(3, (m, k)), synth.uniform(4, (k, n_cols))
    big = np.float32(3.4027e38)  # finite; its nearest TF32 number is not
    b[0, 1], b[m // 2, k - 1], b[m // 3, 0], b[m // 3, 2] = np.inf, -np.inf, np.inf, np.inf
    b[m // 5, 3] = big
    w[1, 4], w[k - 1, 5], w[:, n_cols - 1] = 0.0, np.inf, np.abs(w[:, n_cols - 1]) + 1e-3
    w[3] *= 1e-3
    plan = api.Plan("gemm_spmm", api.CSRMatrix(m, m, *t), k=k, n_cols=n_cols)
    bd = torch.empty(m * k + off, device="cuda")[off:].view(m, k).copy_(torch.from_numpy(b))
    for wt in (False, True):
        d = torch.zeros(m * n_cols + off, device="cuda")[off:].view(m, n_cols)
        plan.gemm_spmm(bd, torch.from_numpy(np.ascontiguousarray(w.T) if wt else w).cuda(), d, w_transposed=wt)
        plan.status()
        with np.errstate(invalid="ignore"):
            want = (b.astype(np.float64) @ w.astype(np.float64))[t[1]]
        got = d.cpu().numpy()
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
        np.testing.assert_array_equal(np.where(np.isinf(got), got, 0), np.where(np.isinf(want), want, 0))
        fin = np.isfinite(want)
        scale = np.where(fin, np.abs(want), 0).max(1, keepdims=True)  # (a row of sums of up to 300 terms, each sum within 6e-7 of it)
        assert (np.where(fin, np.abs(got - want), 0) <= 1e-6 * scale).all()
    plan.close()


@pytest.mark.parametrize("dims", [(16, 8, 6), (17, 10, 5)])
@pytest.mark.parametrize("k,n_cols", [(64, 64), (33, 48), (17, 20)])
def test_grid_with_missing_couplings(built_lib, dims, k, n_cols):
    """A 3-D grid some of whose rows do not name a neighbour: nothing is multiplied that is not stored, so what is no finite
    number in a row of B reaches the rows that name it and no others."""
    import torch
    ap, ai, ax = synth.laplacian(dims)
    n = len(ap) - 1
    rows = np.repeat(np.arange(n), np.diff(ap))
    keep = (rows == ai) | (np.random.default_rng(1).uniform(size=len(ai)) > 0.1)
    ap = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=n))]).astype(np.int32)
    ai, ax = ai[keep], ax[keep]
    b, w = synth.uniform(5, (n, k)), synth.uniform(6, (k, n_cols))
    b[np.arange(5, n, 50), 1] = np.inf
    A = _scipy((ap, ai, ax), n)
    hit = np.asarray(A.astype(bool)[:, 5::50].sum(1)).ravel() > 0
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, ap, ai, ax), k=k, n_cols=n_cols)
    for relu in (False, True):
        d = torch.zeros((n, n_cols), device="cuda")
        plan.gemm_spmm(torch.from_numpy(b).cuda(), torch.from_numpy(w).cuda(), d, relu=relu)
        plan.status()
        got = d.cpu().numpy()
        assert np.isfinite(got[~hit]).all()
        if not relu:
            assert not np.isfinite(got[hit]).any()
        want = A[~hit] @ np.where(np.isfinite(b), b, 0).astype(np.float64) @ w.astype(np.float64)
        common.assert_close(got[~hit], np.maximum(want, 0) if relu else want, "rows without an infinity")
    plan.close()


@pytest.mark.parametrize("chain,n_cols", [("gemm_spmm", 96), ("spmm_spmm", 65)])
def test_large_intermediate_stays_a_ring(built_lib, chain, n_cols):
    """A plan on a grid (of one dimension here) keeps no more of T than the ring that the operator allows where all of it (and the padded rows of C of a
    width that is no multiple of four) would take more than a 48th of the device's memory."""
    import torch
    free, mem = torch.cuda.mem_get_info()
    t = synth.laplacian((int(1.05 * mem / 48 / (4 * n_cols * (1 if chain == "gemm_spmm" else 2))),))
    n = len(t[0]) - 1
    plan = api.Plan(chain, api.CSRMatrix(n, n, *t), k=17, n_cols=n_cols)
    assert plan.info()["ring_rows"] > 0
    assert free - torch.cuda.mem_get_info()[0] < 2 << 30  # operator and tiles, ring, weight
    plan.close()


@pytest.mark.parametrize("k,n_cols", [(64, 64), (64, 47)])
@pytest.mark.parametrize("bits", [0x7FFFFFFF, 0x7F800001])
def test_nan_stays_nan_in_the_sums_of_the_ticket_executor(built_lib, k, n_cols, bits):
    test_nan_stays_nan(None, k, n_cols, {"tensor_cores": 1}, bits)
