"""The weight gradient's product over all rows (csrc/atb.cu) against fp64: sums of at most a few thousand fp32 products and of
at most 296 partial sums, of random signs, keep a relative error below 1e-6 (2^-24 times the root of their number)."""
import numpy as np
import pytest

from tile_fusion_b200 import _lib, synth

pytestmark = pytest.mark.gpu


# rows around the 16 that are staged and the 64 of a range; columns around the tiles of 64 and 128, rows off the 16-byte grid
@pytest.mark.parametrize("m", [1, 15, 17, 65, 5003, 120_001])
@pytest.mark.parametrize("na,nb", [(40, 128), (128, 128), (7, 33), (64, 129), (65, 4), (256, 100)])
def test_atb(built_lib, m, na, nb):
    import torch
    L = _lib.lib()
    a, b = synth.uniform(1, (m, na)), synth.uniform(2, (m, nb))
    ad, bd = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    want = (ad.double().t() @ bd.double()).cpu().numpy()
    work = torch.empty(L.tf_atb_work_floats(m, na, nb), device="cuda")
    first = None
    for _ in range(2):
        out = torch.full((na, nb), float("nan"), device="cuda")
        _lib.check(L.tf_atb_dev(ad.data_ptr(), na, bd.data_ptr(), nb, m, out.data_ptr(), work.data_ptr(), work.numel(),
                                torch.cuda.current_stream().cuda_stream))
        got = out.cpu().numpy()
        assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
        assert first is None or np.array_equal(got, first)
        first = got
    assert L.tf_atb_dev(ad.data_ptr(), na, bd.data_ptr(), nb, m, out.data_ptr(), work.data_ptr(), work.numel() - 1, None) == -1
