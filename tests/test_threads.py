"""Plans of different shapes used by host threads at the same time, each on a stream of its own."""
import threading

import numpy as np
import pytest

from tests.test_intermediate import _band
from tile_fusion_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chain", ["gemm", "precise", "band"])
def test_plans_do_not_disturb_each_other(built_lib, chain):
    """Kernels whose shared memory depends on the plan: the widest and the narrowest side by side give the bits they give alone."""
    import torch
    n = 6000
    t = _band(n, 60, 10) if chain == "band" else (np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n, np.float32))
    work = []
    for i in range(2):
        if chain == "band":
            tt = t if i == 0 else _band(n, 20, 40)
            plan = api.Plan("spmm_spmm", api.CSRMatrix(n, n, *tt), n_cols=32)
            args = [torch.from_numpy(synth.uniform(i, (n, 32))).cuda(), torch.empty(n, 32, device="cuda")]
            call = plan.spmm_spmm
        else:
            k, c = (64, (32, 256)[i]) if chain == "gemm" else (33, (7, 64)[i])
            plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=k, n_cols=c)
            args = [torch.from_numpy(synth.uniform(i, (n, k))).cuda(), torch.from_numpy(synth.uniform(i + 2, (k, c))).cuda(),
                    torch.empty(n, c, device="cuda")]
            call = plan.gemm_spmm
        call(*args)
        plan.status()
        work.append((plan, call, args, args[-1].clone(), torch.cuda.Stream()))
    errors = []

    def loop(plan, call, args, want, stream):
        try:
            for _ in range(1500):
                call(*args, stream=stream.cuda_stream)
            plan.status(stream.cuda_stream)
            if not torch.equal(args[-1], want):
                errors.append("results differ")
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=loop, args=w) for w in work]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
    for w in work:
        w[0].close()
