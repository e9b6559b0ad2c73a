"""tf_plan_intermediate: T = F C (T = B W) of a chain, local rows first, whichever executor the plan runs on."""
import ctypes as C

import numpy as np
import pytest

from tests import common
from tests.test_gather import _graph, _scipy
from tile_fusion_b200 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _read(plan, n):
    """The first n rows of the plan's intermediate, as an identity's product with them."""
    import torch
    L = _lib.lib()
    p, rows, cols = C.c_void_p(), C.c_longlong(), C.c_int()
    _lib.check(L.tf_plan_intermediate(plan._h, C.byref(p), C.byref(rows), C.byref(cols)))
    assert p.value and rows.value == n
    ap, ai, ax = torch.arange(n + 1, dtype=torch.int32, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda"), torch.ones(n, device="cuda")
    out = torch.empty((n, cols.value), device="cuda")
    _lib.check(L.tf_spmm_dev(ap.data_ptr(), ai.data_ptr(), ax.data_ptr(), n, p.value, cols.value, out.data_ptr(),
                             torch.cuda.current_stream().cuda_stream))
    return out.cpu().numpy()


def _band(n, reach, per_row):
    rng = np.random.default_rng(reach)
    r = np.repeat(np.arange(n), per_row)
    key = np.unique(r.astype(np.int64) * n + np.clip(r + rng.integers(-reach, reach + 1, len(r)), 0, n - 1))
    ap = np.concatenate([[0], np.cumsum(np.bincount(key // n, minlength=n))]).astype(np.int32)
    return ap, (key % n).astype(np.int32), rng.uniform(-1, 1, len(key)).astype(np.float32)


@pytest.mark.parametrize("kind,n_cols", [("lines", 64), ("lines", 33), ("two lines", 32), ("band", 96), ("two bands", 32), ("odd", 32), ("graph", 64)])
def test_spmm_spmm(built_lib, kind, n_cols):
    import torch
    two = None
    if "lines" in kind:
        t = synth.laplacian((90, 70))
        two = (t[0], t[1], t[2] * np.where(np.arange(len(t[2])) % 3 == 0, np.float32(0.5), np.float32(1))) if kind[:3] == "two" else None
    elif "band" in kind:
        t = _band(9001, 40, 12)
        two = _band(9001, 100, 11) if kind[:3] == "two" else None
    else:
        t = synth.laplacian((17, 10, 9)) if kind == "odd" else _graph(3000, 4)
    n = len(t[0]) - 1
    c = synth.uniform(3, (n, n_cols))
    plan = api.Plan("spmm_spmm", api.CSRMatrix(n, n, *t), B=api.CSRMatrix(n, n, *two) if two else None, n_cols=n_cols)
    cd = torch.from_numpy(c).cuda()
    d = [torch.full((n, n_cols), float("nan"), device="cuda") for _ in range(2)]
    plan.spmm_spmm(cd, d[0])
    if kind in ("odd", "graph"):
        _read(plan, n)
    else:
        _lib.check(_lib.lib().tf_plan_intermediate(plan._h, None, None, None))
    plan.spmm_spmm(cd, d[1])
    plan.status()
    assert torch.equal(*d)
    want = _scipy(two or t, n) @ c.astype(np.float64)
    common.assert_close(_read(plan, n)[:, :n_cols], want, kind)
    c2 = synth.uniform(4, (n, n_cols))
    plan.spmm_spmm_host(c2, np.empty((n, n_cols), np.float32))
    common.assert_close(_read(plan, n)[:, :n_cols], _scipy(two or t, n) @ c2.astype(np.float64), kind + ", host call")
    plan.close()


@pytest.mark.parametrize("kind", ["graph", "grid"])
@pytest.mark.parametrize("k,n_cols", [(32, 64), (64, 40)])
def test_gemm_spmm(built_lib, kind, k, n_cols):
    import torch
    t = _graph(3000, 4, hubs=((5, 900),)) if kind == "graph" else synth.laplacian((18, 10, 9))
    n = len(t[0]) - 1
    b, w = synth.uniform(3, (n, k)), synth.uniform(4, (k, n_cols))
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=k, n_cols=n_cols)
    d = torch.empty((n, n_cols), device="cuda")
    for _ in range(2):
        plan.gemm_spmm(torch.from_numpy(b).cuda(), torch.from_numpy(w).cuda(), d)
        plan.status()
        tm = _read(plan, n)
    tw = b.astype(np.float64) @ w.astype(np.float64)
    common.assert_close(tm[:, :n_cols], tw, kind)
    common.assert_close(d.cpu().numpy(), _scipy(t, n) @ tw, kind)
    plan.close()
