"""The band-marching executor (csrc/band_march.cu) against the CSR products, bit for bit."""
import numpy as np
import pytest

from tests import common
from tests.test_gather import _scipy
from tests.test_line_march import _csr
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


def _band(n, per_row, reach, seed):
    """Rows of up to per_row nonzeros within `reach` of the diagonal, some rows empty, the reach itself taken."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), per_row)
    cols = np.clip(rows + rng.integers(-reach, reach + 1, size=rows.size), 0, n - 1)
    far = np.arange(n - reach)
    rows, cols = np.concatenate([rows, far, far + reach]), np.concatenate([cols, far + reach, far])
    S = sp.csr_matrix((rng.uniform(-1, 1, rows.size).astype(np.float32), (rows, cols)), shape=(n, n))
    S = sp.diags((np.arange(n) % 11 != 3).astype(np.float32)) @ S
    S = sp.csr_matrix(S, dtype=np.float32)
    S.eliminate_zeros()
    S.sort_indices()
    return S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data


# reaches up to and beyond a block of 64 and of 128 rows (129: another executor), row counts around blocks and groups of four
@pytest.mark.parametrize("n,per_row,reach", [(1026, 5, 63), (1024, 9, 64), (1300, 7, 65), (2563, 12, 128), (2500, 12, 129), (4003, 3, 40)])
@pytest.mark.parametrize("n_cols", [4, 32, 36, 96])
def test_band(built_lib, n, per_row, reach, n_cols):
    import torch
    a, b = _band(n, per_row, reach, 1), _band(n, per_row + 2, min(reach, 30), 2)
    c = synth.uniform(3, (n, n_cols))
    cd = torch.from_numpy(c).cuda()
    for first, B in ((a, None), (b, _csr(b))):
        plan = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols)
        d = torch.full((n, n_cols), float("nan"), device="cuda")
        for _ in range(2):
            plan.spmm_spmm(cd, d)
        plan.status()
        common.assert_close(d.cpu().numpy(), _scipy(a, n) @ (_scipy(first, n) @ c.astype(np.float64)), f"{n} {reach} {n_cols}")
        ref = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols, mode=api.MODE_UNFUSED, tile_slots=-1, lattice_march=-1)
        d0 = torch.empty_like(d)
        ref.spmm_spmm(cd, d0)
        ref.status()
        assert torch.equal(d, d0)
        dh = np.full((n, n_cols), np.nan, np.float32)
        plan.spmm_spmm_host(c, dh)
        np.testing.assert_array_equal(dh, d.cpu().numpy())
        plan.close()
        ref.close()


def test_band_host_call_in_slabs(built_lib):
    import torch
    n, n_cols = 60_003, 96
    a = _band(n, 6, 50, 4)
    c = synth.uniform(5, (n, n_cols))
    plan = api.Plan("spmm_spmm", _csr(a), n_cols=n_cols)
    d = torch.full((n, n_cols), float("nan"), device="cuda")
    plan.spmm_spmm(torch.from_numpy(c).cuda(), d)
    plan.status()
    dh = np.full((n, n_cols), np.nan, np.float32)
    plan.spmm_spmm_host(c, dh)
    np.testing.assert_array_equal(dh, d.cpu().numpy())
    common.assert_close(dh, _scipy(a, n) @ (_scipy(a, n) @ c.astype(np.float64)), "slabs")
    plan.close()
