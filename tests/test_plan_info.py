"""Plan.info()["threads"]: the CTA size of the kernel that a plan of default options runs on."""
import pytest

from tests.test_gather import _graph
from tests.test_intermediate import _band
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chain,kind,threads", [("spmm_spmm", "grid", 128), ("spmm_spmm", "lines", 128), ("spmm_spmm", "band", 512),
                                                ("spmm_spmm", "graph", 256), ("gemm_spmm", "grid", 128), ("gemm_spmm", "lines", 256),
                                                ("gemm_spmm", "graph", 256), ("sddmm_spmm", "graph", 256)])
def test_threads(built_lib, chain, kind, threads):
    t = {"grid": lambda: synth.laplacian((18, 10, 9)), "lines": lambda: synth.laplacian((50, 40)), "band": lambda: _band(5003, 40, 12),
         "graph": lambda: _graph(3000, 4)}[kind]()
    n = len(t[0]) - 1
    plan = api.Plan(chain, api.CSRMatrix(n, n, *t), k=64, n_cols=64)
    assert plan.info()["threads"] == threads
    plan.close()
