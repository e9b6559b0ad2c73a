"""torch.ops.sw_gcn on CUDA tensors: the layers of the reference's GCN scripts, written exactly as they call the
operators (binding-project/gcn-e2e-training/FusedGCNLayer.py:8-42, FusedGCNModule.py:7-18), against dense torch."""
import pytest

from tests import common
from tile_fusion_b200 import synth

pytestmark = pytest.mark.gpu


def _layers(torch):
    import tile_fusion_b200.sw_gcn  # noqa: F401  (registers torch.ops.sw_gcn)

    class FusedGCNLayer(torch.nn.Module):  # as FusedGCNLayer.py:8-42
        def __init__(self, feat_dim, embed_dim, m_tile_size, adj, schedule, num_threads):
            super().__init__()
            self.weight = torch.nn.Parameter(torch.empty(embed_dim, feat_dim, device="cuda"))
            torch.nn.init.xavier_uniform_(self.weight)
            self.adj, self.schedule, self.num_threads = adj, schedule, num_threads
            self.forward_fn = torch.ops.sw_gcn.fusedGeMMSpMM_vt_ro
            level_ptr, mix_ptr = self.schedule[0], self.schedule[1]
            self.max_tile_size = 0
            for x in range(level_ptr[0], level_ptr[1]):
                self.max_tile_size = max(self.max_tile_size, int(mix_ptr[x * 2 + 2] - mix_ptr[x * 2]))

        def forward(self, x):
            return self.forward_fn(self.adj, x, self.weight, self.schedule, self.num_threads, self.max_tile_size)

    class FusedGCN(torch.nn.Module):  # as FusedGCNModule.py:7-18
        def __init__(self, feat_dim, embed_dim, num_classes, adj, num_threads):
            super().__init__()
            schedule = torch.ops.sw_gcn.inspect_vt_ro(adj, feat_dim, embed_dim, 500000, num_threads)
            self.conv1 = FusedGCNLayer(feat_dim, embed_dim, 128, adj, schedule, num_threads)
            self.conv2 = FusedGCNLayer(embed_dim, num_classes, 128, adj, schedule, num_threads)

        def forward(self, x):
            return self.conv2(self.conv1(x).relu())
    return FusedGCN


def test_two_layer_gcn_forward_and_backward(built_lib):
    import torch
    torch.manual_seed(0)
    n, feat, hid, cls = 3000, 100, 64, 47
    g = synth.rmat_gcn(6, n, 12)
    adj = torch.sparse_csr_tensor(torch.from_numpy(g[0]), torch.from_numpy(g[1]), torch.from_numpy(g[2]), size=(n, n)).cuda()
    dense = adj.to_dense().double()
    model = _layers(torch)(feat, hid, cls, adj, 8)
    x = torch.from_numpy(synth.normal(2, (n, feat))).cuda().requires_grad_(True)
    out = model(x)
    w1, w2 = model.conv1.weight.double(), model.conv2.weight.double()
    xd = x.detach().double().requires_grad_(True)
    w1d, w2d = w1.detach().requires_grad_(True), w2.detach().requires_grad_(True)
    want = dense @ ((dense @ (xd @ w1d.t())).relu() @ w2d.t())
    common.assert_close(out.detach().cpu().numpy(), want.detach().cpu().numpy(), "sw_gcn forward")
    loss_w = torch.from_numpy(synth.uniform(9, (n, cls))).cuda()
    (out * loss_w).sum().backward()
    (want * loss_w.double()).sum().backward()
    # the adjacency of a GCN is symmetric, so multiplying the gradient by A (as the reference does) is A^T dY
    common.assert_close(model.conv1.weight.grad.cpu().numpy(), w1d.grad.cpu().numpy(), "dW1")
    common.assert_close(model.conv2.weight.grad.cpu().numpy(), w2d.grad.cpu().numpy(), "dW2")
    common.assert_close(x.grad.cpu().numpy(), xd.grad.cpu().numpy(), "dX")


def test_other_operators(built_lib):
    import torch
    import tile_fusion_b200.sw_gcn  # noqa: F401
    n = 1500
    g = synth.rmat_gcn(4, n, 8)
    adj = torch.sparse_csr_tensor(torch.from_numpy(g[0]), torch.from_numpy(g[1]), torch.from_numpy(g[2]), size=(n, n)).cuda()
    x = torch.from_numpy(synth.normal(2, (n, 32))).cuda()
    w = torch.from_numpy(synth.glorot(3, 48, 32)).cuda()
    want = (adj.to_dense().double() @ (x.double() @ w.double().t())).cpu().numpy()
    sched = torch.ops.sw_gcn.inspect(adj, 128)
    assert len(sched) == 3 and sched[0].dtype == torch.int32 and int(sched[0][2]) >= int(sched[0][1]) > 0
    for got in (torch.ops.sw_gcn.fusedGeMMSpMM(adj, x, w, sched, 4), torch.ops.sw_gcn.unfused_gcn_forward(adj, x, w, 4),
                torch.ops.sw_gcn.geMMSpMM_f_bw(adj, x, w, sched, 4)):
        common.assert_close(got.cpu().numpy(), want, "sw_gcn forward variants")
    af = torch.sparse.mm(adj, x)
    common.assert_close(torch.ops.sw_gcn.cachedSpMMGeMM(af, w, 4).cpu().numpy(), want, "cachedSpMMGeMM")


@pytest.mark.parametrize("k,n_cols", [(64, 64), (32, 128), (128, 128), (100, 256), (36, 16)])
def test_layers_keep_the_order_of_their_sums(built_lib, k, n_cols):
    """Bit for bit the ticket executor's activations, whichever of k and n_cols is the larger: one that rounding puts on the
    other side of zero is another gradient.  Rows around the 256 nonzeros that its warps share, up to the 4096 that a CTA takes."""
    import torch
    import tile_fusion_b200.sw_gcn  # noqa: F401
    from tests.test_gather import _graph
    from tile_fusion_b200 import api
    n = 5000
    t = _graph(n, 5, empty={0, 7, n - 1}, hubs=((9, 4096), (11, 255), (12, 256), (13, 257), (400, 513), (4000, 3000), (4001, 64)))
    adj = torch.sparse_csr_tensor(*(torch.from_numpy(x) for x in t), size=(n, n)).cuda()
    x, w = torch.from_numpy(synth.normal(2, (n, k))).cuda(), torch.from_numpy(synth.glorot(3, n_cols, k)).cuda()
    ticket = api.Plan("gemm_spmm", api.CSRMatrix(n, n, *t), k=k, n_cols=n_cols, rows_per_block=128)
    assert ticket.info()["items"] > 0
    want = torch.full((n, n_cols), float("nan"), device="cuda")
    ticket.gemm_spmm(x, w, want, w_transposed=True)
    ticket.status()
    with torch.no_grad():
        assert torch.equal(torch.ops.sw_gcn.fusedGeMMSpMM(adj, x, w, [], 4), want)
    ticket.close()


def test_backward_on_two_streams(built_lib):
    """Two models on one adjacency share its plan; the sparse products of their backward passes run beside one another, long rows
    (cut into pieces that are counted) included."""
    import torch
    import tile_fusion_b200.sw_gcn as sw
    from tests.test_gather import _graph
    n, k, c = 4000, 48, 64
    t = _graph(n, 5, hubs=[(r, 1500 + r) for r in range(0, 400, 10)])
    adj = torch.sparse_csr_tensor(*(torch.from_numpy(x) for x in t), size=(n, n)).cuda()
    plan = sw._plan(adj, k, c)
    assert sw._lib.lib().tf_exec_spmm_work_bytes(plan._h) > 0
    gs = [torch.from_numpy(synth.uniform(s, (n, c))).cuda() for s in (1, 2)]
    want = [sw._spmm(plan, g) for g in gs]
    streams = [torch.cuda.Stream() for _ in gs]
    torch.cuda.synchronize()
    for _ in range(20):
        got = []
        for s, g in zip(streams, gs):
            with torch.cuda.stream(s):
                got.append([sw._spmm(plan, g) for _ in range(4)])
        torch.cuda.synchronize()
        for outs, w in zip(got, want):
            assert all(torch.equal(o, w) for o in outs)
    # scratch that is too small is refused
    x, w = gs[0], torch.empty(16, dtype=torch.uint8, device="cuda")
    assert sw._lib.lib().tf_exec_spmm_work(plan._h, x.data_ptr(), c, want[0].data_ptr(), w.data_ptr(), 16, None) == sw._lib.TF_ERR_ARG


@pytest.mark.parametrize("n,k,c", [(300, 4100, 4099), (9000, 32, 7), (9000, 32, 12), (5000, 1433, 16), (2000, 602, 256), (600, 1, 40), (600, 64, 1)])
def test_weight_gradient_of_any_size(built_lib, n, k, c):
    """Layers of more than 2^24 weights, of one feature or class, of few entries and of many: dW against fp64, as before the
    library had a kernel of its own for it."""
    import torch
    import tile_fusion_b200.sw_gcn  # noqa: F401
    g = synth.rmat_gcn(6, n, 8)
    adj = torch.sparse_csr_tensor(*(torch.from_numpy(t) for t in g), size=(n, n)).cuda()
    x = torch.from_numpy(synth.normal(2, (n, k))).cuda()
    w = torch.from_numpy(synth.glorot(3, c, k)).cuda().requires_grad_(True)
    dy = torch.from_numpy(synth.uniform(4, (n, c))).cuda()
    torch.ops.sw_gcn.fusedGeMMSpMM(adj, x, w, [], 4).backward(dy)
    want = (adj.to_dense().double() @ dy.double()).t() @ x.double()
    common.assert_close(w.grad.cpu().numpy(), want.cpu().numpy(), "dW")


@pytest.mark.parametrize("index,value", [("int32", "float32"), ("int64", "float32"), ("int64", "float64")])
def test_adjacency_is_held_and_not_copied(built_lib, index, value):
    """The cache knows an adjacency by where it lies, so it holds it -- another of the same sizes is another one -- but keeps no
    second copy on the device: what a first call on an adjacency leaves allocated is its plan's and the output's."""
    import torch
    import tile_fusion_b200.sw_gcn as sw
    n = 3000
    g = synth.rmat_gcn(6, n, 12)
    x, w = torch.from_numpy(synth.normal(2, (n, 32))).cuda(), torch.from_numpy(synth.glorot(3, 48, 32)).cuda()
    for scale in (1.0, 2.0, 3.0):
        parts = [torch.from_numpy(g[0]).to(getattr(torch, index)).cuda(), torch.from_numpy(g[1]).to(getattr(torch, index)).cuda(),
                 (torch.from_numpy(g[2]) * scale).to(getattr(torch, value)).cuda()]
        adj = torch.sparse_csr_tensor(*parts, size=(n, n))
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        out = torch.ops.sw_gcn.fusedGeMMSpMM(adj, x, w, [], 4)
        assert torch.cuda.memory_allocated() - before <= out.numel() * 4 + 512
        want = adj.to_dense().double() @ (x.double() @ w.double().t())
        common.assert_close(out.cpu().numpy(), want.cpu().numpy(), f"scale {scale}")
        del adj, parts, out, want
