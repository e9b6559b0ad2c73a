"""The gather on rows that are read value by value (a width that is no multiple of four, or operands off the 16-byte grid): the
lanes and columns that it takes for a width, and panels beyond 128 columns.  fp32 sums of up to a few hundred products: the tolerance of
tests/common.py."""
import numpy as np
import pytest

from tests import common
from tests.test_gather import _graph, _scipy
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols", [1, 7, 8, 9, 16, 17, 24, 25, 31, 33, 47, 48, 49, 64, 65, 96, 97, 127, 129, 130])
@pytest.mark.parametrize("off", [0, 1])
def test_widths(built_lib, n_cols, off):
    import torch
    n = 3000
    t = _graph(n, 5, empty={0, 7, n - 1}, hubs=((9, 3000), (11, 700)))
    plan = api.Plan("spmm_spmm", api.CSRMatrix(n, n, *t), n_cols=n_cols)
    x = synth.uniform(3, (n, n_cols))
    xd = torch.empty(n * n_cols + off, device="cuda")[off:].view(n, n_cols).copy_(torch.from_numpy(x))
    out = torch.full((n * n_cols + off,), float("nan"), device="cuda")[off:].view(n, n_cols)
    for _ in range(2):
        plan.spmm(xd, out)
    plan.status()
    common.assert_close(out.cpu().numpy(), _scipy(t, n) @ x.astype(np.float64), f"{n_cols} off={off}")
    plan.close()


@pytest.mark.parametrize("kq,nv", [(32, 32), (64, 64), (64, 128), (128, 64), (128, 128), (36, 20), (60, 100), (33, 64), (64, 47), (100, 4), (4, 3)])
def test_sddmm_widths(built_lib, kq, nv):
    """Every lane with all its columns of K or not, rows of V that end inside a lane's columns, values read one by one."""
    import torch
    n = 2000
    t = _graph(n, 5, empty={0, n - 1}, hubs=((9, 1500), (11, 300)))
    q, k, v = (synth.uniform(s, (n, w)) for s, w in ((3, kq), (4, kq), (5, nv)))
    plan = api.Plan("sddmm_spmm", api.CSRMatrix(n, n, *t), k=kq, n_cols=nv)
    d = torch.full((n, nv), float("nan"), device="cuda")
    for _ in range(2):
        plan.sddmm_spmm(*(torch.from_numpy(a).cuda() for a in (q, k, v)), d)
    plan.status()
    A = _scipy(t, n).tocoo()
    s = A.copy()
    s.data = A.data * (q.astype(np.float64)[A.row] * k.astype(np.float64)[A.col]).sum(1)
    common.assert_close(d.cpu().numpy(), s.tocsr() @ v.astype(np.float64), f"{kq} {nv}")
    plan.close()
