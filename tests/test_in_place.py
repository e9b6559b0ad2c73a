"""GeMM-SpMM whose result lies over an operand, on the star stencils that otherwise run in one launch: as the two products in turn give it."""
import numpy as np
import pytest

from tests import common
from tests.test_gather import _scipy
from tests.test_spmm_gemm import _varying
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


def _setup(dims, k, n_cols):
    import torch
    t = _varying(synth.laplacian(dims))
    n = len(t[0]) - 1
    A = api.CSRMatrix(n, n, *t)
    b, w = synth.uniform(3, (n, k)), synth.uniform(4, (k, n_cols))
    plan, two = (api.Plan("gemm_spmm", A, k=k, n_cols=n_cols, lattice_march=lm) for lm in (0, -1))
    assert plan.info()["threads"] == 480
    b, w = torch.from_numpy(b).cuda(), torch.from_numpy(w).cuda()
    want = torch.full((n, n_cols), float("nan"), device="cuda")
    two.gemm_spmm(b, w, want)
    two.status()
    two.close()
    common.assert_close(want.cpu().numpy(), _scipy(t, n) @ (b.double() @ w.double()).cpu().numpy(), f"{dims} {k} {n_cols}")
    return plan, b, w, want


@pytest.mark.parametrize("dims", [(640, 500), (64, 50, 40)])
@pytest.mark.parametrize("k", [32, 128, 256])
def test_result_over_b(built_lib, dims, k):
    plan, b, w, want = _setup(dims, k, k)
    for _ in range(2):
        d = b.clone()
        plan.gemm_spmm(d, w, d)
        plan.status()
        assert (d == want).all()
    plan.close()


@pytest.mark.parametrize("shift", [1, 700])  # rows by which the result starts behind (in front of) B
@pytest.mark.parametrize("k,n_cols", [(64, 64), (64, 32), (32, 64)])
def test_result_over_part_of_b(built_lib, shift, k, n_cols):
    import torch
    plan, b, w, want = _setup((203, 311), k, n_cols)
    n, off = len(b), shift * max(k, n_cols)
    for at_b, at_d in ((0, off), (off, 0)):
        buf = torch.empty(off + n * max(k, n_cols), device="cuda")
        x, d = buf[at_b:at_b + n * k].view(n, k), buf[at_d:at_d + n * n_cols].view(n, n_cols)
        x.copy_(b)
        plan.gemm_spmm(x, w, d)
        plan.status()
        assert (d == want).all()
    plan.close()


def test_result_over_the_weight(built_lib):
    plan, b, w, want = _setup((203, 311), 64, 128)
    d = want.clone().fill_(float("nan"))
    x = d.view(-1)[-w.numel():].view(w.shape)
    x.copy_(w)
    plan.gemm_spmm(b, x, d)
    plan.status()
    assert (d == want).all()
    plan.close()


def test_captured(built_lib):
    """The call may be part of a graph, as one whose operands lie apart."""
    import torch
    plan, b, w, want = _setup((203, 311), 64, 64)
    d = b.clone()
    plan.gemm_spmm(d, w, d)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.gemm_spmm(d, w, d)
    for _ in range(3):
        d.copy_(b)
        g.replay()
        torch.cuda.synchronize()
        assert (d == want).all()
    plan.status()
    plan.close()
