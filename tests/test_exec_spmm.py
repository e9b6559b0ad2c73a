"""tf_exec_spmm: out = A X with the operator of any plan, whichever executor it is for and whatever the width."""
import numpy as np
import pytest

from tests import common
from tests.test_gather import _graph, _scipy
from tests.test_intermediate import _band
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu

_HUBS = ((5, 900), (17, 64))
_PLANS = [("spmm_spmm", "graph", dict(n_cols=32)), ("spmm_spmm", "graph", dict(n_cols=33)), ("spmm_spmm", "lines", dict(n_cols=32)),
          ("spmm_spmm", "band", dict(n_cols=32)), ("spmm_spmm", "grid", dict(n_cols=32)), ("spmm_spmm", "odd", dict(n_cols=32)),
          ("gemm_spmm", "graph", dict(k=16, n_cols=32)), ("gemm_spmm", "grid", dict(k=16, n_cols=32)),
          ("gemm_spmm", "graph", dict(k=16, n_cols=32, ctas_per_sm=1)), ("sddmm_spmm", "graph", dict(k=16, n_cols=32))]


@pytest.mark.parametrize("chain,kind,opts", _PLANS)
def test_any_plan_any_width(built_lib, chain, kind, opts):
    import torch
    t = {"graph": lambda: _graph(3000, 4, empty={0, 7, 2999}, hubs=_HUBS), "lines": lambda: synth.laplacian((50, 40)),
         "band": lambda: _band(5003, 40, 12), "grid": lambda: synth.laplacian((18, 10, 9)), "odd": lambda: synth.laplacian((17, 10, 9))}[kind]()
    n = len(t[0]) - 1
    plan = api.Plan(chain, api.CSRMatrix(n, n, *t), **opts)
    for width, off in ((1, 0), (32, 0), (32, 1), (36, 0), (47, 0), (100, 0), (131, 1)):
        x = synth.uniform(width, (n, width))
        xd = torch.empty(n * width + off, device="cuda")[off:].view(n, width).copy_(torch.from_numpy(x))
        buf = torch.full((n * width + off + 64,), float("nan"), device="cuda")
        out = buf[off:off + n * width].view(n, width)
        for _ in range(2):
            plan.spmm(xd, out)
        common.assert_close(out.cpu().numpy(), _scipy(t, n) @ x.astype(np.float64), f"{chain} {kind} {width}")
        assert torch.isnan(buf[off + n * width:]).all()
    plan.close()
