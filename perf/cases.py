"""Cases by which the speed of the fused chains is measured: what a user of this library has it do.

The path is one sparse operator and dense fp32 matrices through one of the public entry points: the README-level
executors, a plan's executors, the two-layer GCN forward, the ``torch.ops.sw_gcn`` layers with their backward, and the
host-pointer call.  The operators are the three kinds that the library is used on: grid Laplacians in natural order
(2-D and 3-D, even, odd and ragged extents), banded matrices as finite elements give them, and power-law graphs (R-MAT).
Matrices and dense operands are made on the GPU from the seed; the plan is what a program keeps for an operator.
"""
import math

import numpy as np
import torch

from tile_fusion_b200 import api, synth

# Dense widths in use: the sweep's 32, 64 and 128, the GCN's 100, 256 and 47, and ones that are no multiple of anything.
_WIDTHS = (8, 16, 32, 33, 47, 64, 96, 100, 128)


def listed():
    return [
        # The README call on a small 2-D grid (the tests' 40 x 33): launches and the call itself are what counts.
        dict(name="executor_small", kind="executor", matrix="grid", nx=40, ny=33, nz=1, n_cols=64),
        # SpMM-SpMM on the benchmark's operator, the 128^3 7-point Laplacian.
        dict(name="spmm_grid3d", kind="spmm", matrix="grid", nx=128, ny=128, nz=128, n_cols=128),
        # The same chain where no extent is a multiple of anything and the width is the GCN's 100.
        dict(name="spmm_grid3d_ragged", kind="spmm", matrix="grid", nx=101, ny=67, nz=83, n_cols=100),
        # A 2-D 5-point operator, the grid of image and plane problems, at the sweep's middle width.
        dict(name="spmm_grid2d", kind="spmm", matrix="grid", nx=1023, ny=777, nz=1, n_cols=64),
        # An unstructured band: finite-element matrices after a bandwidth-reducing ordering.
        dict(name="spmm_band", kind="spmm", matrix="band", n=200_003, per_row=12, half_width=40, n_cols=96),
        # The chain on a power-law graph (two hops of message passing), the sweep's width 64.
        dict(name="spmm_graph", kind="spmm", matrix="graph", n=200_000, degree=20, n_cols=64),
        # GeMM-SpMM on the 256^2 5-point Laplacian, K = N = 64: an ordinary call of tens of microseconds.
        dict(name="gemm_grid2d", kind="gemm", matrix="grid", nx=256, ny=256, nz=1, k=64, n_cols=64),
        # GeMM-SpMM, K = N = 256, on one eighth of the 256^3 grid: what one of eight GPUs holds; the largest case.
        dict(name="gemm_grid3d", kind="gemm", matrix="grid", nx=256, ny=256, nz=32, k=256, n_cols=256),
        # Inference of a two-layer GCN with the benchmark's widths 100 -> 256 -> 47 and degree 25.
        dict(name="gcn_forward", kind="gcn", matrix="graph", n=500_009, degree=25, k=100, hidden=256, out=47),
        # One training step of a smaller two-layer GCN written on the torch operators: forward, loss, both gradients.
        dict(name="gcn_train", kind="gcn_train", matrix="graph", n=120_001, degree=14, k=128, hidden=128, out=40),
        # Attention-style SDDMM-SpMM with the benchmark's widths and degree.
        dict(name="sddmm_graph", kind="sddmm", matrix="graph", n=262_144, degree=32, k=64, n_cols=128),
        # The drop-in call of a host program: numpy arrays in pageable memory, copies both ways inside the call.
        dict(name="host_grid3d", kind="host", matrix="grid", nx=64, ny=64, nz=64, n_cols=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, rows_lo, rows_hi):
    """A 2-D or 3-D grid of rows_lo .. rows_hi points with extents that differ by up to a factor of about four."""
    rows = _log(rng, rows_lo, rows_hi)
    d = rng.choice((2, 3))
    if rows < 1000:
        d = 2
    s = rows ** (1.0 / d)
    nx = max(8, int(s * rng.uniform(0.5, 2.0)))
    if d == 2:
        return dict(matrix="grid", nx=nx, ny=max(8, rows // nx), nz=1)
    ny = max(4, int(s * rng.uniform(0.5, 2.0)))
    return dict(matrix="grid", nx=nx, ny=ny, nz=max(4, rows // (nx * ny)))


def draw(rng):
    kind = rng.choice(("executor", "spmm_grid", "spmm_grid", "spmm_band", "spmm_graph", "gemm_grid", "gemm_grid", "gcn",
                       "gcn_train", "sddmm", "host"))
    if kind == "executor":
        return dict(kind="executor", n_cols=rng.choice(_WIDTHS), **_grid(rng, 500, 40_000))
    if kind == "spmm_grid":
        return dict(kind="spmm", n_cols=rng.choice(_WIDTHS), **_grid(rng, 4_000, 2_000_000))
    if kind == "spmm_band":
        per_row = rng.randint(5, 16)
        return dict(kind="spmm", matrix="band", n=_log(rng, 4_000, 400_000), per_row=per_row,
                    half_width=rng.randint(2 * per_row, 60), n_cols=rng.choice(_WIDTHS))
    if kind == "spmm_graph":
        return dict(kind="spmm", matrix="graph", n=_log(rng, 3_000, 500_000), degree=rng.randint(5, 25),
                    n_cols=rng.choice(_WIDTHS))
    if kind == "gemm_grid":
        return dict(kind="gemm", k=rng.choice((17, 32, 64, 100, 128, 256)), n_cols=rng.choice((16, 47, 64, 100, 128, 256)),
                    **_grid(rng, 4_000, 1_500_000))
    if kind == "gcn":
        return dict(kind="gcn", matrix="graph", n=_log(rng, 3_000, 500_000), degree=rng.randint(5, 25),
                    k=rng.choice((32, 64, 100, 128)), hidden=rng.choice((64, 128, 256)), out=rng.choice((7, 40, 47, 64)))
    if kind == "gcn_train":
        return dict(kind="gcn_train", matrix="graph", n=_log(rng, 3_000, 200_000), degree=rng.randint(5, 25),
                    k=rng.choice((32, 64, 100, 128)), hidden=rng.choice((32, 64, 128)), out=rng.choice((7, 40, 47)))
    if kind == "sddmm":
        return dict(kind="sddmm", matrix="graph", n=_log(rng, 3_000, 300_000), degree=rng.randint(8, 32),
                    k=rng.choice((32, 64, 100)), n_cols=rng.choice((32, 47, 64, 128)))
    return dict(kind="host", n_cols=rng.choice(_WIDTHS), **_grid(rng, 2_000, 300_000))


# ---------------------------------------------------------------------------------------------------------------------
# Operators
# ---------------------------------------------------------------------------------------------------------------------
def _host_csr(rows, cols, vals, n):
    """CSRMatrix of sorted (row, column) pairs on the GPU; duplicates have been removed."""
    ap = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ap[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return api.CSRMatrix(n, n, ap.to(torch.int32).cpu().numpy(), cols.to(torch.int32).cpu().numpy(),
                         vals.to(torch.float32).cpu().numpy())


def _laplacian(nx, ny, nz):
    """synth.laplacian on the GPU: diagonal 2 * dimensions, off-diagonals -1, natural order."""
    dims = (nx, ny) if nz == 1 else (nx, ny, nz)
    n = nx * ny * nz
    idx = torch.arange(n, device="cuda")
    below, above, stride = [], [], 1
    for d in dims:
        x = (idx // stride) % d
        below.insert(0, (idx - stride, x > 0, -1.0))
        above.append((idx + stride, x < d - 1, -1.0))
        stride *= d
    parts = below + [(idx, idx >= 0, 2.0 * len(dims))] + above
    ok = torch.stack([p[1] for p in parts], 1)
    cols = torch.stack([p[0] for p in parts], 1)[ok]
    vals = torch.tensor([p[2] for p in parts], device="cuda").expand(n, -1)[ok]
    return _host_csr(torch.repeat_interleave(idx, ok.sum(1)), cols, vals, n)


def _band(n, per_row, half_width, gen):
    rows = torch.arange(n, device="cuda").repeat_interleave(per_row)
    cols = (rows + torch.randint(-half_width, half_width + 1, (n * per_row,), device="cuda", generator=gen)).clamp_(0, n - 1)
    key = torch.unique(rows * n + cols)
    vals = 2 * torch.rand(key.numel(), device="cuda", generator=gen) - 1
    return _host_csr(key // n, key % n, vals, n)


def _rmat(n, edges, gen):
    """R-MAT endpoints (a, b, c = 0.57, 0.19, 0.19), ids at or above n rejected."""
    src, dst, have = [], [], 0
    while have < edges:
        m = min(1 << 23, int((edges - have) * 1.4) + 1024)
        s = torch.zeros(m, dtype=torch.int64, device="cuda")
        d = torch.zeros(m, dtype=torch.int64, device="cuda")
        for _ in range(max(1, math.ceil(math.log2(n)))):
            u = torch.rand(m, device="cuda", generator=gen)
            down = u >= 0.76
            s = 2 * s + down
            d = 2 * d + (((u >= 0.57) & ~down) | (u >= 0.95))
        ok = (s < n) & (d < n)
        src.append(s[ok])
        dst.append(d[ok])
        have += int(src[-1].numel())
    return torch.cat(src)[:edges], torch.cat(dst)[:edges]


def _graph(n, degree, gen, symmetric):
    """synth.rmat_gcn (symmetrised, self loops, values D^-1/2 (A + I) D^-1/2) or synth.rmat_pattern (directed, values 1)."""
    loops = torch.arange(n, device="cuda")
    if symmetric:
        s, d = _rmat(n, degree * n // 2, gen)
        key = torch.unique(torch.cat([s * n + d, d * n + s, loops * n + loops]))
        rows, cols = key // n, key % n
        deg = torch.bincount(rows, minlength=n).double()
        vals = 1.0 / torch.sqrt(deg[rows] * deg[cols])
    else:
        s, d = _rmat(n, degree * n, gen)
        empty = loops[torch.bincount(s, minlength=n) == 0]
        key = torch.unique(torch.cat([s * n + d, empty * n + empty]))
        rows, cols = key // n, key % n
        vals = torch.ones(key.numel(), device="cuda")
    return _host_csr(rows, cols, vals, n)


def _operator(case, gen):
    if case["matrix"] == "grid":
        return _laplacian(case["nx"], case["ny"], case["nz"])
    if case["matrix"] == "band":
        return _band(case["n"], case["per_row"], case["half_width"], gen)
    return _graph(case["n"], case["degree"], gen, case["kind"] != "sddmm")


def _rows_nnz(case):
    """Rows and (for graphs and bands: before duplicates are dropped, about) nonzeros of a case's operator."""
    if case["matrix"] == "grid":
        dims = [d for d in (case["nx"], case["ny"], case["nz"]) if d > 1]
        n = int(np.prod(dims))
        return n, n + sum(2 * (d - 1) * (n // d) for d in dims)
    if case["matrix"] == "band":
        return case["n"], case["n"] * case["per_row"]
    return case["n"], case["n"] * (case["degree"] + (case["kind"] != "sddmm"))


# ---------------------------------------------------------------------------------------------------------------------
# One case
# ---------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    A = _operator(case, gen)
    kind, m = case["kind"], A.M

    def uniform(*shape):
        return 2 * torch.rand(shape, device="cuda", generator=gen) - 1

    def normal(sigma, *shape):
        return sigma * torch.randn(shape, device="cuda", generator=gen)

    def glorot(out_dim, in_dim):
        return uniform(out_dim, in_dim) * math.sqrt(6.0 / (in_dim + out_dim))

    if kind == "executor":
        return dict(kind=kind, A=A, sched=api.inspector(A, 8), C=uniform(m, case["n_cols"]),
                    D=torch.empty(m, case["n_cols"], device="cuda"))
    if kind == "host":
        c = np.ascontiguousarray(uniform(m, case["n_cols"]).cpu().numpy())
        return dict(kind=kind, A=A, sched=api.inspector(A, 8), C=c, D=np.zeros_like(c))
    if kind == "spmm":
        return dict(kind=kind, plan=api.Plan("spmm_spmm", A, n_cols=case["n_cols"]), C=uniform(m, case["n_cols"]),
                    D=torch.empty(m, case["n_cols"], device="cuda"))
    if kind == "gemm":
        return dict(kind=kind, plan=api.Plan("gemm_spmm", A, k=case["k"], n_cols=case["n_cols"]), B=uniform(m, case["k"]),
                    W=uniform(case["k"], case["n_cols"]), D=torch.empty(m, case["n_cols"], device="cuda"))
    if kind == "sddmm":
        return dict(kind=kind, plan=api.Plan("sddmm_spmm", A, k=case["k"], n_cols=case["n_cols"]),
                    Q=normal(0.125, m, case["k"]), K=normal(0.125, m, case["k"]), V=normal(0.125, m, case["n_cols"]),
                    D=torch.empty(m, case["n_cols"], device="cuda"))
    k, hid, out = case["k"], case["hidden"], case["out"]
    X, W1, W2 = normal(1.0, m, k), glorot(hid, k), glorot(out, hid)
    if kind == "gcn":
        plans = (api.Plan("gemm_spmm", A, k=k, n_cols=hid), api.Plan("gemm_spmm", A, k=hid, n_cols=out))
        return dict(kind=kind, A=A, X=X, W1=W1, W2=W2, plans=plans)
    import tile_fusion_b200.sw_gcn  # noqa: F401  (registers torch.ops.sw_gcn)
    adj = torch.sparse_csr_tensor(torch.from_numpy(A.Ap), torch.from_numpy(A.Ai), torch.from_numpy(A.Ax), size=(m, m)).cuda()
    sched = torch.ops.sw_gcn.inspect_vt_ro(adj, k, hid, 500000, 8)
    return dict(kind=kind, adj=adj, sched=sched, X=X, W1=W1.requires_grad_(True), W2=W2.requires_grad_(True),
                labels=torch.randint(0, out, (m,), device="cuda", generator=gen))


def run(state):
    kind = state["kind"]
    if kind in ("executor", "host"):
        A, C, D = state["A"], state["C"], state["D"]
        m, n = C.shape
        api.spMMSpMMExecutor(A, A, api.Matrix(m, n, C), api.Matrix(m, n, D), state["sched"], 8)
        return D
    if kind == "spmm":
        state["plan"].spmm_spmm(state["C"], state["D"])
        return state["D"]
    if kind == "gemm":
        state["plan"].gemm_spmm(state["B"], state["W"], state["D"])
        return state["D"]
    if kind == "sddmm":
        state["plan"].sddmm_spmm(state["Q"], state["K"], state["V"], state["D"])
        return state["D"]
    if kind == "gcn":
        out, _ = api.gcn_forward(state["A"], state["X"], state["W1"], state["W2"], state["plans"])
        return out
    layer = torch.ops.sw_gcn.fusedGeMMSpMM_vt_ro
    h = layer(state["adj"], state["X"], state["W1"], state["sched"], 8, 128).relu()
    o = layer(state["adj"], h, state["W2"], state["sched"], 8, 128)
    loss = torch.nn.functional.cross_entropy(o, state["labels"])
    g1, g2 = torch.autograd.grad(loss, (state["W1"], state["W2"]))
    return dict(loss=loss.detach(), logits=o.detach(), grad_w1=g1, grad_w2=g2)


def work(case):
    n, nnz = _rows_nnz(case)
    kind = case["kind"]
    if kind in ("executor", "host", "spmm"):
        return {"bytes": synth.bytes_spmm_spmm(n, nnz, case["n_cols"]), "flops": synth.flops_spmm_spmm(nnz, nnz, case["n_cols"])}
    if kind == "gemm":
        return {"bytes": synth.bytes_gemm_spmm(n, nnz, case["k"], case["n_cols"]),
                "flops": synth.flops_gemm_spmm(n, nnz, case["k"], case["n_cols"])}
    if kind == "sddmm":
        return {"bytes": synth.bytes_sddmm_spmm(n, nnz, case["k"], case["n_cols"]),
                "flops": synth.flops_sddmm_spmm(nnz, case["k"], case["n_cols"])}
    k, hid, out = case["k"], case["hidden"], case["out"]
    weights = k * hid + hid * out
    flops = synth.flops_gemm_spmm(n, nnz, k, hid) + synth.flops_gemm_spmm(n, nnz, hid, out)
    nbytes = 4 * (n * k + n * out + weights + 2 * nnz + n + 1)
    if kind == "gcn_train":  # labels in, gradients out; A dY, dW and (second layer) dX
        nbytes += 8 * n + 4 * weights
        flops += 2 * nnz * (hid + out) + 2 * n * weights + 2 * n * hid * out
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times the largest error against the same chain in fp64 over the listed cases and two dozen drawn ones."""
    kind = case["kind"]
    if kind in ("executor", "host", "spmm"):   # fp32 sums: 1e-7 and 7e-7
        return {"rel": 4e-7, "max": 3e-6}
    if kind == "sddmm":                        # a short dot product in front of each product: 2.3e-7 and 2.8e-5
        return {"rel": 1e-6, "max": 1.2e-4}
    if kind == "gcn_train":
        # logits 1e-6 and 4e-6, but the first gradient passes a ReLU: an activation within a rounding error of zero may
        # fall on either side of it, and where that row is a hub of the graph the gradient moves by 7e-5 (and 1.6e-3)
        return {"rel": 3e-4, "max": 7e-3}
    return {"rel": 8e-6, "max": 4e-5}          # fp32 accuracy through the tensor cores, K = 256: 1.9e-6 and 8e-6
