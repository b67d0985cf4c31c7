"""The fast kNN kernels (a thread per query, fast_one.cuh; a warp per query for
few queries, warp.cuh) against the reference-order kernels at the sizes where it can go wrong: trees around the home subtree's size and a
partly filled last level, lists at and around each compiled capacity, cut-offs
that leave lists unfilled, records that can and cannot be read as vectors,
tie-heavy and duplicate points.  Bit-exact: the reference-order kernels are
pinned to the oracle in test_gpu_query.py.
"""
import ctypes as C
import math

import pytest
import torch

import cudakdtree_b200 as ck
from tests.helpers import make_points, make_queries

pytestmark = pytest.mark.gpu


def _check(tree, q, k, method, lay, wb, **kw):
    a = ck.knn(tree, q, k, method, layout=lay, world_bounds=wb, with_max=True, **kw)
    b = ck.knn(tree, q, k, method, layout=lay, world_bounds=wb, with_max=True,
               reference_order=True, **kw)
    for x, y in zip(a, b):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))


@pytest.mark.parametrize("k", [2, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("kind", ["uniform", "tie", "same"])
@pytest.mark.parametrize("nq", [333, 17000])
def test_tree_sizes_and_list_capacities(k, scalar, kind, nq):
    q = torch.from_numpy(make_queries(nq, 3, kind, scalar=scalar, seed=2)).cuda()
    for n in (1, 2, k - 1, k, k + 1, 2 * k, 62, 63, 64, 127, 255, 256, 300, 1023, 5000):
        tree = torch.from_numpy(make_points(n, 3, kind, scalar=scalar, seed=n)).cuda()
        wb = ck.build_tree(tree)
        _check(tree, q, k, ["stack_based", "stack_free", "cct"][n % 3], None, wb)


@pytest.mark.parametrize("D", [2, 3, 4])
@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("k,cutoff", [(2, 0.03), (16, 0.1), (40, 0.2)])
@pytest.mark.parametrize("nq", [777, 17000])
def test_cutoffs_and_record_layouts(D, scalar, k, cutoff, nq):
    n = 3001
    pts = torch.from_numpy(make_points(n, D, "uniform", scalar=scalar, seed=5)).cuda()
    q = torch.from_numpy(make_queries(nq, D, "uniform", scalar=scalar, seed=6)).cuda()
    kw = {"cutoff": cutoff} if scalar == "float32" else {"cutoff_d2": int((2000 * cutoff) ** 2)}
    for stride, poff, doff, shift in ((4 * D, 0, -1, 0), (4 * D + 4, 0, 4 * D, 0),
                                      (32, 16, -1, 0), (32, 0, 28, 4), (24, 4, 0, 0)):
        lay = ck.layout_for(scalar, D, stride=stride, point_offset=poff, dim_offset=doff,
                            dim_shift=shift, dim_bits=32 - shift)
        words = torch.zeros(n * stride // 4 + 1, dtype=torch.int32, device="cuda")
        for first in (0, 1):  # an array that starts 4 bytes off a 16-byte boundary
            tree = words[first:first + n * stride // 4]
            tree.view(n, -1)[:, poff // 4:poff // 4 + D] = pts.view(torch.int32)
            wb = ck.build_tree(tree, layout=lay)
            for method in ("stack_free", "cct"):
                _check(tree, q, k, method, lay, wb)
                _check(tree, q, k, method, lay, wb, **kw)


@pytest.mark.parametrize("scale", [1e-25, 1e-12, 1e12, 1e18])
@pytest.mark.parametrize("nq", [500, 17000])
def test_extreme_scales(scale, nq):
    """Bounds too small to scale stack entries by, and near the float range."""
    pts = torch.from_numpy(make_points(5000, 3, "gmm", seed=7)).cuda() * scale
    q = torch.from_numpy(make_queries(nq, 3, "gmm", seed=8)).cuda() * scale
    wb = ck.build_tree(pts)
    for k in (3, 16, 64):
        _check(pts, q, k, "stack_based", None, wb)
        _check(pts, q, k, "cct", None, wb, cutoff=math.inf, morton=False)


@pytest.mark.parametrize("method", ["stack_based", "stack_free", "cct"])
@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("kind", ["uniform", "tie", "same"])
def test_few_queries_fcp_and_k1(method, scalar, kind):
    """FCP and k = 1 of few queries (a warp each), trees of up to several
    treelets (5 levels) and partly filled ones; strict '<' of FCP, cut-offs."""
    q = torch.from_numpy(make_queries(400, 3, kind, scalar=scalar, seed=3)).cuda()
    for n in (1, 2, 15, 16, 31, 32, 33, 500, 1023, 1024, 1025, 40000):
        tree = torch.from_numpy(make_points(n, 3, kind, scalar=scalar, seed=n)).cuda()
        wb = ck.build_tree(tree)
        for kw in ({}, {"cutoff": 0.05} if scalar == "float32" else {"cutoff_d2": 9000}):
            a = ck.fcp(tree, q, method, world_bounds=wb, with_d2=True, **kw)
            b = ck.fcp(tree, q, method, world_bounds=wb, with_d2=True, reference_order=True, **kw)
            for x, y in zip(a, b):
                assert torch.equal(x.view(torch.int32), y.view(torch.int32))
            _check(tree, q, 1, method, None, wb, **kw)


def test_far_queries_keep_many_subtrees_pending():
    """Queries far from a shell of points: nearly every subtree is as near as
    the next, so the warp kernel's pending subtrees outgrow best-first order."""
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    v = torch.randn((300_000, 3), device="cuda", generator=g)
    tree = v / v.norm(dim=1, keepdim=True)
    wb = ck.build_tree(tree)
    q = torch.randn((300, 3), device="cuda", generator=g) * 1e-3
    for k in (1, 16, 100):
        _check(tree, q, k, "cct", None, wb)


@pytest.mark.parametrize("nq", [300, 17000])
@pytest.mark.parametrize("k", [2, 8])
def test_stack_free_eps_does_not_change_lists(nq, k):
    """eps of a stack-free kNN applies to ties only: without ties the list is
    the exact one, for few queries as for many."""
    tree = torch.from_numpy(make_points(20000, 3, "uniform", seed=9)).cuda()
    wb = ck.build_tree(tree)
    lay = ck.infer_layout(tree)
    q = torch.from_numpy(make_queries(nq, 3, "uniform", seed=10)).cuda()
    want = ck.knn(tree, q, k, "stack_free", world_bounds=wb)
    p = ck._params("stack_free", k, eps=0.5)
    ids, d2 = torch.empty_like(want[0]), torch.empty_like(want[1])
    ck._check(ck.lib().cukd_knn(ck._ptr(tree), 20000, C.byref(lay), ck._ptr(wb), ck._ptr(q), nq,
                                C.byref(p), ck._ptr(ids), ck._ptr(d2), None, ck._stream(None),
                                None), "cukd_knn")
    assert torch.equal(ids, want[0]) and torch.equal(d2, want[1])
