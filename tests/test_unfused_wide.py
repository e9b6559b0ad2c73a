"""The unfused mode above 128 columns on star stencils, where it takes the sums of the one launch in two passes: bit for bit the default mode,
and both against executors that share no sums with them."""
import ctypes as C

import numpy as np
import pytest

from tests import common
from tests.test_gather import _scipy
from tests.test_spmm_gemm import _run, _varying
from tile_fusion_b200 import _lib, api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(97, 83), (33, 37, 29)])
@pytest.mark.parametrize("k,n_cols", [(36, 144), (128, 240), (256, 256)])
def test_modes(built_lib, dims, k, n_cols):
    """Error bound as in test_spmm_gemm.py, 2e-6 in every executor, so 4e-6 between two of them."""
    t = _varying(synth.laplacian(dims))
    n = len(t[0]) - 1
    A = api.CSRMatrix(n, n, *t)
    b, w = synth.uniform(3, (n, k)), synth.uniform(4, (k, n_cols))
    want = _scipy(t, n) @ (b.astype(np.float64) @ w.astype(np.float64))
    out = []
    for kw in ({}, dict(mode=api.MODE_UNFUSED), dict(mode=api.MODE_UNFUSED, lattice_march=-1), dict(lattice_march=-1)):
        plan = api.Plan("gemm_spmm", A, k=k, n_cols=n_cols, **kw)
        out.append(_run(plan, b, w))
        rel, _ = common.assert_close(out[-1], want, f"{dims} {k} {n_cols} {kw}")
        assert rel < 2e-6, rel
        plan.close()
    np.testing.assert_array_equal(out[0], out[1])
    for other in out[2:]:
        assert np.linalg.norm(out[0] - other) < 4e-6 * np.linalg.norm(want)


def test_memory(built_lib):
    """Two passes need no coefficients of the one launch: an operator whose coefficients differ takes no more than one whose don't."""
    import torch
    t = synth.laplacian((100, 100, 100))
    n = len(t[0]) - 1
    used = []
    for tr in (t, t, _varying(t)):  # (the first plan of a process pays for more than itself)
        before = torch.cuda.mem_get_info()[0]
        plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *tr), k=32, n_cols=144, mode=api.MODE_UNFUSED)
        used.append(before - torch.cuda.mem_get_info()[0])
        plan.close()
    assert abs(used[2] - used[1]) <= 4 << 20  # (allocations come in units of 2 MB)


def test_intermediate(built_lib):
    import torch
    t = synth.laplacian((80, 70))
    n = len(t[0]) - 1
    b, w = synth.uniform(3, (n, 32)), synth.uniform(4, (32, 144))
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=32, n_cols=144, mode=api.MODE_UNFUSED)
    _run(plan, b, w)
    p, rows, cols = C.c_void_p(), C.c_longlong(), C.c_int()
    _lib.check(_lib.lib().tf_plan_intermediate(plan._h, C.byref(p), C.byref(rows), C.byref(cols)))
    assert p.value and rows.value == n and cols.value == 144
    common.assert_close(_run(plan, b, w), _scipy(t, n) @ (b.astype(np.float64) @ w.astype(np.float64)), "with T")
    one = [torch.arange(n + 1, dtype=torch.int32, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda"), torch.ones(n, device="cuda")]
    out = torch.empty((n, 144), device="cuda")
    _lib.check(_lib.lib().tf_spmm_dev(*(q.data_ptr() for q in one), n, p.value, 144, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    common.assert_close(out.cpu().numpy(), b.astype(np.float64) @ w.astype(np.float64), "T")
    plan.close()
