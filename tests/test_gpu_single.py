"""FCP and k = 1 (fcp_fast_one of fast_one.cuh for many queries, warp.cuh before
it for few) against the reference-order kernels: ties at the nearest distance,
whose outcome depends on the traversal's order, duplicated points, points at
exactly the cut-off, int distances that their float bounds round differently,
trees around the home subtree's size (7 full nodes), every record layout.
Bit-exact: the reference-order kernels are pinned to the oracle in
test_gpu_query.py.
"""
import itertools

import numpy as np
import pytest
import torch

import cudakdtree_b200 as ck
from tests.helpers import make_points, make_queries

pytestmark = pytest.mark.gpu

METHODS = ["stack_based", "stack_free", "cct"]
MANY, FEW = 17003, 401


def _check(tree, q, method, lay, wb, **kw):
    a = ck.fcp(tree, q, method, layout=lay, world_bounds=wb, with_d2=True, **kw)
    b = ck.fcp(tree, q, method, layout=lay, world_bounds=wb, with_d2=True, reference_order=True,
               **kw)
    a += ck.knn(tree, q, 1, method, layout=lay, world_bounds=wb, with_max=True, **kw)
    b += ck.knn(tree, q, 1, method, layout=lay, world_bounds=wb, with_max=True,
                reference_order=True, **kw)
    for x, y in zip(a, b):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))


def _inputs(n, nq, D, kind, scalar):
    if kind == "copies":  # every point three times, queries at points and beside them
        one = make_points(max(1, n // 3), D, "uniform", scalar=scalar, seed=n)
        pts = np.resize(np.concatenate([one] * 3), (n, D))
        q = pts[np.arange(nq) % n].copy()
        q[::2, 0] += 1
    else:
        pts = make_points(n, D, kind, scalar=scalar, seed=n)
        q = make_queries(nq, D, kind, scalar=scalar, seed=n + 1)
    return torch.from_numpy(np.ascontiguousarray(pts)).cuda(), torch.from_numpy(q).cuda()


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("D", [2, 3, 4])
@pytest.mark.parametrize("kind", ["uniform", "tie", "same", "copies"])
@pytest.mark.parametrize("nq", [FEW, MANY])
def test_tree_sizes_and_ties(method, scalar, D, kind, nq):
    for n in (1, 2, 3, 6, 7, 8, 14, 15, 16, 33, 500, 1025, 6000):
        tree, q = _inputs(n, nq, D, kind, scalar)
        wb = ck.build_tree(tree)
        _check(tree, q, method, None, wb)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("r2", [0, 1, 2, 4])
@pytest.mark.parametrize("nq", [FEW, MANY])
def test_points_at_exactly_the_cutoff(method, scalar, r2, nq):
    """Lattice points: many at exactly the radius (k = 1 takes them if its
    traversal visits them, FCP does not)."""
    kw = {"cutoff": float(np.sqrt(np.float64(r2)))} if scalar == "float32" else {"cutoff_d2": r2}
    for n in (5, 15, 100, 300):
        rng = np.random.Generator(np.random.MT19937(n + r2))
        pts = rng.integers(0, 12, size=(n, 3)).astype(scalar)
        q = rng.integers(-2, 14, size=(nq, 3)).astype(scalar)
        tree = torch.from_numpy(pts).cuda()
        wb = ck.build_tree(tree)
        _check(tree, torch.from_numpy(q).cuda(), method, None, wb, **kw)


@pytest.mark.parametrize("D", [2, 3, 4])
@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("kind", ["uniform", "tie"])
@pytest.mark.parametrize("nq", [FEW, MANY])
def test_record_layouts(D, scalar, kind, nq):
    n = 3001
    pts = torch.from_numpy(make_points(n, D, kind, scalar=scalar, seed=5)).cuda()
    q = torch.from_numpy(make_queries(nq, D, kind, scalar=scalar, seed=6)).cuda()
    kw = {"cutoff": 0.03} if scalar == "float32" else {"cutoff_d2": 3600}
    for stride, poff, doff, shift in ((4 * D, 0, -1, 0), (4 * D + 4, 0, 4 * D, 0),
                                      (32, 16, -1, 0), (32, 0, 28, 4), (24, 4, 0, 0)):
        lay = ck.layout_for(scalar, D, stride=stride, point_offset=poff, dim_offset=doff,
                            dim_shift=shift, dim_bits=32 - shift)
        words = torch.zeros(n * stride // 4 + 1, dtype=torch.int32, device="cuda")
        for first in (0, 1):  # an array that starts 4 bytes off a 16-byte boundary
            tree = words[first:first + n * stride // 4]
            tree.view(n, -1)[:, poff // 4:poff // 4 + D] = pts.view(torch.int32)
            wb = ck.build_tree(tree, layout=lay)
            for method in METHODS:
                _check(tree, q, method, lay, wb)
                _check(tree, q, method, lay, wb, **kw)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("D", [2, 3, 4])
def test_wide_distances_and_their_bounds(method, scalar, D):
    """Offsets of one large triple (or pair, or four) in every order and sign
    around the query: equal exact distances whose rounded bounds differ, next
    to neighbours one unit nearer and farther."""
    base = (268435399, 134217689, 67108859, 33554393)[:D]
    offs = np.array([[s * v for s, v in zip(signs, perm)]
                     for perm in itertools.permutations(base)
                     for signs in itertools.product((-1, 1), repeat=D)], np.int64)
    rng = np.random.Generator(np.random.MT19937(D))
    pts = np.concatenate([offs, offs + rng.integers(-1, 2, size=offs.shape), offs])
    q = rng.integers(-1, 2, size=(MANY, D))
    tree = torch.from_numpy(pts.astype(scalar)).cuda()
    wb = ck.build_tree(tree)
    for nq in (FEW, MANY):
        _check(tree, torch.from_numpy(q[:nq].astype(scalar)).cuda(), method, None, wb)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("nq", [FEW, MANY])
def test_large_groups_of_equal_points(method, nq):
    """One location, and four, holding 300,000 points: a query costs a path,
    not the group."""
    for where in (1, 4):
        rng = np.random.Generator(np.random.MT19937(where))
        pts = rng.random((where, 3), dtype=np.float32)[rng.integers(0, where, size=300_000)]
        tree = torch.from_numpy(pts).cuda()
        wb = ck.build_tree(tree)
        q = torch.from_numpy(rng.random((nq, 3), dtype=np.float32)).cuda()
        q[::2] = tree[torch.arange(0, nq, 2, device="cuda")]
        _check(tree, q, method, None, wb)


def test_cutoffs_that_are_no_radius():
    """A NaN or negative cut-off: what the traversal makes of it."""
    tree = torch.from_numpy(make_points(500, 3, "uniform", seed=1)).cuda()
    wb = ck.build_tree(tree)
    itree = torch.from_numpy(make_points(500, 3, "uniform", scalar="int32", seed=1)).cuda()
    iwb = ck.build_tree(itree)
    for nq in (FEW, MANY):
        q = torch.from_numpy(make_queries(nq, 3, "uniform", seed=2)).cuda()
        iq = torch.from_numpy(make_queries(nq, 3, "uniform", scalar="int32", seed=2)).cuda()
        for method in METHODS:
            _check(tree, q, method, None, wb, cutoff=float("nan"))
            _check(itree, iq, method, None, iwb, cutoff_d2=-5)
