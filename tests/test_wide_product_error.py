"""Error of dense products above 128 columns on operands with few nonzero terms, on a weight that selects, and on operands constant along K.

With the operator the identity (a star stencil whose neighbours are stored as zeros) D is the dense product alone.  x = hi + lo to 11
bits each: half a unit of hi is 2^-11 of x at most and 2.0e-4 in the mean square (uniform over half a unit, mantissas uniform).  So what
three TF32 products leave out of a term, lo * lo and the rounding of either lo, is 4.1e-8 of it each in the mean square, 7.1e-8
together; every sum that is not with zero is cut off by up to 2^-23, 4.3e-8 in the mean, three times for a single term.
* one term, or a handful of equal ones: 7.1e-8 and at most three cuts of a like sign, 1.3e-7, within 3e-7
* the weight a selection of columns: the rounding of lo alone, 4.1e-8, within 1e-7
* constant operands: K / 8 * 3 sums of one sign, 2e-6 as in test_spmm_gemm.py; what is left out of a term is the same for all and at
  most 3 * 2^-22 of it, 7.2e-7, inside that
"""
import numpy as np
import pytest

from tests.test_spmm_gemm import _run
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu

ROUTES = {"default": {}, "two_launches": dict(lattice_march=-1), "two_passes": dict(mode=api.MODE_UNFUSED), "ticket_sums": dict(tensor_cores=1)}


def _identity(dims):
    t = synth.laplacian(dims)
    rows = np.repeat(np.arange(len(t[0]) - 1), np.diff(t[0]))
    return t[0], t[1], (t[1] == rows).astype(np.float32)


def _operands(kind, n, k, n_cols):
    rng = np.random.default_rng(7)
    w = rng.standard_normal((k, n_cols)).astype(np.float32)
    b = np.zeros((n, k), np.float32)
    if kind == "one_term":
        b[np.arange(n), rng.integers(0, k, n)] = rng.uniform(-1, 1, n).astype(np.float32)
    elif kind == "bag_of_words":  # binary rows, normalised
        hit = rng.random((n, k)) < 0.01
        b = (hit / np.maximum(hit.sum(1, keepdims=True), 1)).astype(np.float32)
    elif kind == "selection":
        b = rng.uniform(-1, 1, (n, k)).astype(np.float32)
        w = np.eye(k, n_cols, dtype=np.float32)
    else:
        b[:], w[:] = np.float32(1.01206494), np.float32(1.00432873)
    return b, w


BOUND = {"one_term": 3e-7, "bag_of_words": 3e-7, "selection": 1e-7, "constant": 2e-6}


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("kind", BOUND)
@pytest.mark.parametrize("k,n_cols", [(128, 144), (128, 256), (256, 256)])
def test_terms(built_lib, route, kind, k, n_cols):
    dims = (70, 60)
    n = dims[0] * dims[1]
    b, w = _operands(kind, n, k, n_cols)
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *_identity(dims)), k=k, n_cols=n_cols, **ROUTES[route])
    want = b.astype(np.float64) @ w.astype(np.float64)
    rel = np.linalg.norm(_run(plan, b, w) - want) / np.linalg.norm(want)
    assert rel < BOUND[kind], rel
    plan.close()


def _tf32(x):
    return ((x.view(np.uint32) + np.uint32(0x1000)) & np.uint32(0xFFFFE000)).view(np.float32)


# (up to 128 columns the two passes are the ticket executor's tile, which cuts the low halves off)
@pytest.mark.parametrize("route,k", [(r, k) for r in ("default", "two_launches") for k in (64, 128, 256)] + [("two_passes", 256)])
def test_low_halves_are_rounded(built_lib, route, k):
    """Identity operator and weight: D is hi + lo with lo rounded to eleven bits, which fp32 holds exactly."""
    dims = (70, 60)
    n = dims[0] * dims[1]
    b = np.random.default_rng(3).standard_normal((n, k)).astype(np.float32)  # (synth.uniform's values end a bit before the last)
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *_identity(dims)), k=k, n_cols=k, **ROUTES[route])
    hi = _tf32(b)
    np.testing.assert_array_equal(_run(plan, b, np.eye(k, dtype=np.float32)), hi + _tf32(b - hi))
    plan.close()
