"""Who waits for the last products of the one-launch GeMM-SpMM (csrc/spmm_gemm.cu): its barriers replayed on the CPU under random
interleavings, and long runs of a weight that stays in shared memory."""
import random

import numpy as np
import pytest

from tests import common
from tests.test_gather import _scipy
from tests.test_spmm_gemm import _run, _varying
from tile_fusion_b200 import api, synth


class _Barrier:
    """An mbarrier: a wait of parity p passes while the phase under way has the other parity (before the first one ends, p = 1 passes)."""

    def __init__(self):
        self.phase = 0

    def passes(self, parity):
        return (self.phase & 1) != parity


def _replay(stages, slices, watcher, seed):
    """The summing warps, the tensor core and the warp that sees to the last products: 'summing' (one of the former) or 'idle' (one that
    waits for every phase without anything else to do).  True where all come to their end."""
    ready, empty = ([_Barrier() for _ in range(stages)] for _ in range(2))
    done = []

    def last(st, ph, used):
        for i in range(used):
            yield empty[i], ph if i < st else ph ^ 1
        assert all(e.phase == (slices - i + stages - 1) // stages for i, e in enumerate(empty))  # every product is done

    def summing():
        st = ph = used = 0
        for _ in range(slices):
            if used >= stages:
                yield empty[st], ph ^ 1
            used = min(stages, used + 1)
            ready[st].phase += 1
            st += 1
            if st == stages:
                st, ph = 0, ph ^ 1
        if watcher == "summing":
            yield from last(st, ph, used)

    def tensor():
        st = ph = 0
        for _ in range(slices):
            yield ready[st], ph
            empty[st].phase += 1
            st += 1
            if st == stages:
                st, ph = 0, ph ^ 1

    def idle():
        st = ph = used = 0
        for _ in range(slices):
            if used >= stages:
                yield empty[st], ph ^ 1
            used = min(stages, used + 1)
            st += 1
            if st == stages:
                st, ph = 0, ph ^ 1
        yield from last(st, ph, used)

    rng = random.Random(seed)
    roles = {"summing": summing(), "tensor": tensor()}
    if watcher == "idle":
        roles["idle"] = idle()
    weight = {r: rng.choice((1, 1, 30)) for r in roles}
    waits = {r: next(g, None) for r, g in roles.items()}
    while True:
        able = [r for r, w in waits.items() if w and w[0].passes(w[1])]
        if not able:
            return all(w is None for w in waits.values())
        r = rng.choices(able, [weight[x] for x in able])[0]
        waits[r] = next(roles[r], None)


@pytest.mark.parametrize("stages", [2, 3, 4])
def test_last_products_are_waited_for(stages):
    runs = [(slices, seed) for slices in (1, 2, 3, 4, 5, 9, 16, 33) for seed in range(60)]
    assert all(_replay(stages, slices, "summing", seed) for slices, seed in runs)
    assert not all(_replay(stages, slices, "idle", seed) for slices, seed in runs)  # what a warp that nothing paces comes to


@pytest.mark.gpu
@pytest.mark.parametrize("dims,k,n_cols", [((1200, 900), 256, 32), ((1030, 700), 256, 64), ((110, 100, 90), 128, 128), ((64, 64, 64), 32, 64)])
def test_long_runs_of_a_resident_weight(built_lib, dims, k, n_cols):
    import torch
    t = _varying(synth.laplacian(dims))
    n = len(t[0]) - 1
    b, w = synth.uniform(3, (n, k)), synth.uniform(4, (k, n_cols))
    plan = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=k, n_cols=n_cols)
    assert plan.info()["threads"] == 480
    got = _run(plan, b, w)
    bd, wd, d = torch.from_numpy(b).cuda(), torch.from_numpy(w).cuda(), torch.empty(n, n_cols, device="cuda")
    for _ in range(200):
        plan.gemm_spmm(bd, wd, d)
    plan.status()
    np.testing.assert_array_equal(d.cpu().numpy(), got)
    common.assert_close(got, _scipy(t, n) @ (b.astype(np.float64) @ w.astype(np.float64)), f"{dims} {k} {n_cols}")
    plan.close()
