"""Spatial builds whose widest extent has no centre inside it: l + h overflows,
infinities of both signs meet, or a coordinate is NaN.  Such splits alternate
the prims between the children, so every build ends with every prim in one
leaf; the GPU's tree is the oracle's."""
import numpy as np
import pytest

from oracle import pyoracle as po


def _points(n, kind, D):
    rng = np.random.Generator(np.random.MT19937(n + D))
    p = rng.random((n, D)).astype(np.float32)
    if kind == "overflow":  # finite, but l + h is not
        p[:, D - 1] = (2e38 + 1e38 * p[:, D - 1]).astype(np.float32)
    elif kind == "negative":  # the same below zero, in the first dim
        p[:, 0] = (-3e38 + 1e38 * p[:, 0]).astype(np.float32)
    elif kind == "whole":  # the whole float range
        p = ((p.astype(np.float64) - 0.5) * 6.8e38).astype(np.float32)
    elif kind == "infinities":
        p[rng.random(n) < 0.3, D - 1] = np.inf
        p[rng.random(n) < 0.3, D - 1] = -np.inf
    elif kind == "nan":
        p[rng.random(n) < 0.2, D - 1] = np.nan
    elif kind == "all_nan":
        p[:] = np.nan
    return p


KINDS = ["overflow", "negative", "whole", "infinities", "nan", "all_nan"]
SIZES = [(2, 1), (9, 0), (40, 0), (1024, 3), (1025, 0), (5000, 0), (5000, 1500)]


def _check_partition(nodes, prims, n):
    assert np.array_equal(np.sort(prims), np.arange(n, dtype=np.uint32))
    assert int(nodes["count"].astype(np.int64).sum()) == n
    leaves = nodes["count"] > 0
    assert 2 * int(leaves.sum()) == len(nodes)  # 2 l - 1 nodes and the dummy: no empty leaf


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,thr", SIZES)
def test_oracle_build_ends(kind, n, thr):
    nodes, prims, _ = po.spatial_build(_points(n, kind, 3), thr or 8)
    _check_partition(nodes, prims, n)


@pytest.mark.gpu
@pytest.mark.parametrize("D", [2, 3, 4])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,thr", SIZES)
def test_build_matches_oracle(kind, n, thr, D):
    import torch

    import cudakdtree_b200 as ck
    pts = _points(n, kind, D)
    on, op, ob = po.spatial_build(pts, thr or 8)
    t = torch.from_numpy(pts).cuda()
    tree = ck.spatial_build(t, leaf_threshold=thr)
    nodes = tree.nodes().cpu().numpy().copy().view(po.SPATIAL_NODE).reshape(-1)
    prims = tree.prim_ids().cpu().numpy().astype(np.uint32)
    _check_partition(nodes, prims, n)
    assert np.array_equal(nodes.view(np.uint8), on.view(np.uint8))
    assert np.array_equal(prims, op)
    assert np.array_equal(np.array(tree.bounds, np.float32).view(np.uint32),
                          np.asarray(ob, np.float32).view(np.uint32))
    tree.free()
