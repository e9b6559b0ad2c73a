"""SDDMM-SpMM over the balanced gather's units (csrc/sddmm_gather.cu) against fp64, with the tolerance of tests/common.py:
a dot product of up to 128 terms in front of each product keeps errors of a few 1e-7 of the sum of the magnitudes."""
import numpy as np
import pytest

from tests import common
from tests.test_gather import _graph, _scipy
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


# one, two and four columns per lane on either side, read as vectors and one by one
@pytest.mark.parametrize("kq,nv", [(1, 1), (32, 32), (31, 47), (33, 64), (64, 128), (62, 126), (100, 128), (97, 33), (128, 100), (100, 2)])
def test_sddmm_gather(built_lib, kq, nv):
    import torch
    n = 3000
    # (n - 1 has entries: the last unit is filled up behind the last row)
    t = _graph(n, 6, empty={0, 1, 5}, hubs=((7, 3000), (17, 63), (18, 64), (19, 65), (2000, 700), (n - 1, 3)))
    q, k, v = (synth.normal(s, (n, w), 0.125) for s, w in ((2, kq), (3, kq), (4, nv)))
    A = _scipy(t, n)
    S = A.copy()
    rows = np.repeat(np.arange(n), np.diff(A.indptr))
    S.data = A.data * np.einsum("ij,ij->i", q[rows].astype(np.float64), k[A.indices].astype(np.float64))
    want = S @ v.astype(np.float64)
    plan = api.Plan("sddmm_spmm", api.CSRMatrix(n, n, *t), k=kq, n_cols=nv)
    assert plan.info()["items"] == 0  # no ticket list: the gather was chosen
    first = None
    for off in (0, 0, 1, 2):
        qd, kd, vd = (torch.empty(x.size + off, device="cuda")[off:].view(x.shape).copy_(torch.from_numpy(x)) for x in (q, k, v))
        d = torch.full((n * nv + off,), float("nan"), device="cuda")[off:].view(n, nv)
        plan.sddmm_spmm(qd, kd, vd, d)
        plan.status()
        common.assert_close(d.cpu().numpy(), want, f"SDDMM {kq} {nv} off={off}")
        if first is None:
            first = d.clone()
        elif off == 0:
            assert torch.equal(d, first)  # pieces of a row are added in order, and the counters are back at zero
    plan.close()
