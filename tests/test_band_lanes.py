"""The band march with a row to a lane (csrc/band_march.cu), which operators of more than two blocks of rows per CTA take, against the CSR
products, bit for bit."""
import numpy as np
import pytest

from tests import common
from tests.test_band_march import _band
from tests.test_gather import _scipy
from tests.test_line_march import _csr
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


# rows around blocks of 64 and 128 and groups of 32, widths that end inside a chunk of 32 columns, both block heights, two operators
@pytest.mark.parametrize("n,per_row,reach,n_cols", [(38_016, 5, 64, 4), (38_017, 3, 40, 36), (20_031, 9, 63, 100), (13_000, 14, 33, 132), (20_033, 6, 128, 96),
                                                    (19_969, 7, 65, 64)])
def test_lanes(built_lib, n, per_row, reach, n_cols):
    import torch
    a, b = _band(n, per_row, reach, 1), _band(n, 2, min(reach, 30), 2)
    c = synth.uniform(3, (n, n_cols))
    c[n // 2, 0] = np.inf
    cd = torch.from_numpy(c).cuda()
    for B in (None, _csr(b)):
        plan = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols)
        if B is None:
            assert plan.info()["threads"] == (128 if reach <= 64 else 256)
        d = torch.full((n, n_cols), float("nan"), device="cuda")
        for _ in range(2):
            plan.spmm_spmm(cd, d)
        plan.status()
        ref = api.Plan("spmm_spmm", _csr(a), B=B, n_cols=n_cols, mode=api.MODE_UNFUSED, tile_slots=-1, lattice_march=-1)
        d0 = torch.empty_like(d)
        ref.spmm_spmm(cd, d0)
        ref.status()
        assert torch.equal(torch.nan_to_num(d, 1e30), torch.nan_to_num(d0, 1e30))
        with np.errstate(invalid="ignore"):
            want = _scipy(a, n) @ (_scipy(a if B is None else b, n) @ c.astype(np.float64))
        fin = np.isfinite(want).all(1)
        common.assert_close(d.cpu().numpy()[fin], want[fin], f"{n} {reach} {n_cols}")
        dh = np.full((n, n_cols), np.nan, np.float32)
        plan.spmm_spmm_host(c, dh)
        np.testing.assert_array_equal(dh, d.cpu().numpy())
        plan.close()
        ref.close()
