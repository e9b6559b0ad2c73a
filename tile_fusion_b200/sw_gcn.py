"""The reference's torch operator library ``sw_gcn`` on CUDA tensors.

Importing this module registers, under the same names and with the same argument order as
``binding-project/main.cpp:133-142`` of the reference::

    torch.ops.sw_gcn.inspect(adj, m_tile_size)                                   -> [level_ptr, mix_ptr, partition]
    torch.ops.sw_gcn.inspect_vt_ro(adj, in_dim, out_dim, cache_size, threads)    -> [level_ptr, mix_ptr, l2_ptr]
    torch.ops.sw_gcn.fusedGeMMSpMM(adj, feature, weight, schedule, threads)      -> adj @ (feature @ weight.T)
    torch.ops.sw_gcn.fusedGeMMSpMM_vt_ro(adj, feature, weight, schedule, threads, max_tile_size)
    torch.ops.sw_gcn.geMMSpMM_f_bw(adj, feature, weight, schedule, threads)
    torch.ops.sw_gcn.unfused_gcn_forward(adj, feature, weight, threads)
    torch.ops.sw_gcn.cachedSpMMGeMM(af, weight, threads)                          -> af @ weight.T

``adj`` is a torch sparse-CSR tensor (int32 indices, fp32 values), ``weight`` is stored ``[out, in]`` as the
reference's layers do (``gcn-e2e-training/FusedGCNLayer.py:10-11``), everything lives on the GPU and the results
take part in autograd: the backward is the reference's (``src/Functions.cpp:819-1043``, ``:1192-1244``),
``dX = (A dY) W`` and ``dW = (A dY)^T X`` -- like the reference it multiplies by ``A``, not ``A^T``, i.e. it
assumes the symmetric adjacency of a GCN.  The forward runs the library's fused GeMM-SpMM executor; the sparse
product of the backward runs on the same plan's operator, the weight gradient -- a sum over all rows -- on a kernel
of the library's own where that is the faster one, the other dense product is a plain library GEMM.

The schedule tensors have the reference's layout (level pointers, per-partition kernel boundaries, row ids) and
come from the library's inspector for the same cache budget; the GPU executor plans its own tiles and does not
read them back (they are accepted and ignored), so a layer written for the reference
(``FusedGCNLayer.forward``: ``forward_fn(adj, x, weight, schedule, num_threads, max_tile_size)``) runs unchanged.
"""
from __future__ import annotations

import numpy as np
import torch

from . import _lib, api

_LIB = torch.library.Library("sw_gcn", "DEF")
_plans: dict = {}


def _csr_of(adj: torch.Tensor):
    """(key, CSRMatrix on the host) of a sparse-CSR adjacency; cached per tensor storage.  The entry holds the tensors
    themselves, whatever their types, so that no other adjacency can come to lie where a cached one lay."""
    if adj.layout != torch.sparse_csr:
        raise ValueError("sw_gcn: the adjacency must be a torch sparse CSR tensor")
    crow, col, val = adj.crow_indices(), adj.col_indices(), adj.values()
    key = (crow.data_ptr(), col.data_ptr(), val.data_ptr(), adj.shape[0], int(val.numel()), val._version)
    hit = _plans.get(("csr", key))
    if hit is None:
        A = api.CSRMatrix(adj.shape[0], adj.shape[1], crow.to(torch.int32).cpu().numpy(), col.to(torch.int32).cpu().numpy(),
                          val.to(torch.float32).cpu().numpy())
        if len(_plans) > 64:
            for p in list(_plans.values()):
                if isinstance(p, api.Plan):
                    p.close()
            _plans.clear()
        hit = _plans[("csr", key)] = (A, (crow, col, val))
    return key, hit[0]


def _plan(adj, k, n, unfused=False):
    key, A = _csr_of(adj)
    pk = ("plan", key, k, n, unfused)
    p = _plans.get(pk)
    if p is None:
        # (tensor_cores=1: the sums of the ticket executor.  A hidden activation within a rounding error of zero falls on one
        # side of the ReLU or on the other, and the gradient with it, so layers keep the order of their sums.)
        p = _plans[pk] = api.Plan("gemm_spmm", A, k=k, n_cols=n, mode=api.MODE_UNFUSED if unfused else api.MODE_STREAM,
                                  tensor_cores=1)
    return p


def _spmm(plan, x):
    """A @ x with the operator of a layer's plan."""
    x = x.contiguous().float()
    out = torch.empty((x.shape[0], x.shape[1]), device=x.device, dtype=torch.float32)
    plan.spmm(x, out)
    return out


def _own_weight_grad(m, na, nb):
    """Whether the library's own kernel takes a weight gradient of na x nb over m rows.  Its tiles are 64 or 128 x 128 and
    it gains by cutting the rows into as many ranges as the device holds.  So not: one row or column (a matrix-vector product:
    120 001 rows, 1 x 256: 103 us, torch 43); so few entries that a tile is mostly padding (16 x 16: 58 and 43, 500 009 rows:
    207 and 107; 7 x 64: 58 and 154, 209 and 110); so many tiles that few ranges are left (512 x 512: 1 289 and 1 245, 12 tiles
    of 16 x 1433: 619 and 541, at 20 000 rows 115 and 179), above all of few rows (1 000 rows, 256 x 602: 29 and 21); and
    nothing beyond 2^24 entries, which it does not take at all."""
    entries, tiles = na * nb, -(-na // (64 if na <= 64 else 128)) * -(-nb // 128)
    if na == 1 or nb == 1 or entries > 1 << 24:
        return False
    if (entries <= 320 and m >= 8192) or (entries <= 512 and m >= 1 << 18):
        return False
    return tiles <= 8 or (tiles <= 10 and m >= 4096) or (tiles < 16 and 4096 <= m < 65536)


def _weight_grad(a, b):
    """a.T @ b for two tall matrices: a sum over all rows.  (With a graph to record, by the operator that records.)"""
    m, na, nb = a.shape[0], a.shape[1], b.shape[1]
    if torch.is_grad_enabled() or not _own_weight_grad(m, na, nb):
        return a.t() @ b
    L = _lib.lib()
    out = torch.empty((na, nb), device=a.device, dtype=torch.float32)
    work = torch.empty(L.tf_atb_work_floats(m, na, nb), device=a.device, dtype=torch.float32)
    _lib.check(L.tf_atb_dev(a.data_ptr(), na, b.data_ptr(), nb, m, out.data_ptr(), work.data_ptr(), work.numel(),
                            torch.cuda.current_stream().cuda_stream))
    return out


class _FusedGeMMSpMM(torch.autograd.Function):
    """Forward D = A (X W^T) on the fused executor; backward as FusedGeMMSpMMROAdj::backward
    (binding-project/src/Functions.cpp:1192-1244)."""

    @staticmethod
    def forward(ctx, adj, feature, weight, unfused):
        x = feature.contiguous().float()
        w = weight.contiguous().float()
        out = torch.empty((adj.shape[0], w.shape[0]), device=x.device, dtype=torch.float32)
        _plan(adj, x.shape[1], w.shape[0], unfused).gemm_spmm(x, w, out, w_transposed=True)
        ctx.adj, ctx.unfused = adj, unfused
        ctx.save_for_backward(x, w)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        x, w = ctx.saved_tensors
        ag = _spmm(_plan(ctx.adj, x.shape[1], w.shape[0], ctx.unfused), grad_out)  # A dY (the reference multiplies by A: symmetric adjacency)
        grad_x = ag @ w if ctx.needs_input_grad[1] else None
        grad_w = _weight_grad(ag, x) if ctx.needs_input_grad[2] else None
        return None, grad_x, grad_w, None


class _CachedSpMMGeMM(torch.autograd.Function):
    """ForwardCachingAF (binding-project/src/Functions.cpp): out = AF W^T for a first layer whose A X is cached."""

    @staticmethod
    def forward(ctx, af, weight):
        ctx.save_for_backward(af, weight)
        return af @ weight.t()

    @staticmethod
    def backward(ctx, grad_out):
        af, weight = ctx.saved_tensors
        return (grad_out @ weight if ctx.needs_input_grad[0] else None), grad_out.t() @ af


def _schedule_tensors(adj, kind, **prm):
    _, A = _csr_of(adj)
    s = api.inspector(A, prm.pop("threads"), kind=kind, **prm)
    level = torch.from_numpy(np.concatenate([s.ptr1, np.zeros(max(0, 3 - len(s.ptr1)), np.int32)])[:3].astype(np.int32))
    mix = torch.from_numpy(np.concatenate([np.zeros(2, np.int32), s.ker_begin]).astype(np.int32)) if s.ker_begin is not None \
        else torch.zeros(2, dtype=torch.int32)
    ids = torch.from_numpy(s.id[s.type == 1].astype(np.int32)) if len(s.id) else torch.zeros(0, dtype=torch.int32)
    return [level, mix, ids]


def _inspect(adj, m_tile_size):
    """Fixed tiles of m_tile_size rows (createSchedule, binding-project/src/Functions.cpp:551-627)."""
    return _schedule_tensors(adj, api.INSPECT_FIXED, threads=1, iter_per_partition=max(1, int(m_tile_size)))


def _inspect_vt(adj, in_dim, out_dim, cache_size, num_threads):
    """Variable tiles under a cache budget (inspect_vt, binding-project/main.cpp:51-88)."""
    return _schedule_tensors(adj, api.INSPECT_VT_GEMM, threads=max(1, int(num_threads)), tile_m=int(cache_size),
                             b_cols=int(in_dim), c_cols=int(out_dim))


_LIB.define("inspect(Tensor adj, int m_tile_size) -> Tensor[]")
_LIB.define("inspect_vt_ro(Tensor adj, int in_dim, int out_dim, int cache_size, int num_threads) -> Tensor[]")
_LIB.define("fusedGeMMSpMM(Tensor adj, Tensor feature, Tensor weight, Tensor[] schedule, int num_threads) -> Tensor")
_LIB.define("fusedGeMMSpMM_vt_ro(Tensor adj, Tensor feature, Tensor weight, Tensor[] schedule, int num_threads, "
            "int max_tile_size) -> Tensor")
_LIB.define("geMMSpMM_f_bw(Tensor adj, Tensor feature, Tensor weight, Tensor[] schedule, int num_threads) -> Tensor")
_LIB.define("unfused_gcn_forward(Tensor adj, Tensor feature, Tensor weight, int num_threads) -> Tensor")
_LIB.define("cachedSpMMGeMM(Tensor af, Tensor weight, int num_threads) -> Tensor")

# CompositeImplicitAutograd: the implementations call autograd Functions themselves, as the reference's ops do.
_LIB.impl("inspect", _inspect, "CompositeImplicitAutograd")
_LIB.impl("inspect_vt_ro", _inspect_vt, "CompositeImplicitAutograd")
_LIB.impl("fusedGeMMSpMM", lambda adj, f, w, sched, nt: _FusedGeMMSpMM.apply(adj, f, w, False), "CompositeImplicitAutograd")
_LIB.impl("fusedGeMMSpMM_vt_ro", lambda adj, f, w, sched, nt, mts: _FusedGeMMSpMM.apply(adj, f, w, False),
          "CompositeImplicitAutograd")
_LIB.impl("geMMSpMM_f_bw", lambda adj, f, w, sched, nt: _FusedGeMMSpMM.apply(adj, f, w, False), "CompositeImplicitAutograd")
_LIB.impl("unfused_gcn_forward", lambda adj, f, w, nt: _FusedGeMMSpMM.apply(adj, f, w, True), "CompositeImplicitAutograd")
_LIB.impl("cachedSpMMGeMM", lambda af, w, nt: _CachedSpMMGeMM.apply(af, w), "CompositeImplicitAutograd")
