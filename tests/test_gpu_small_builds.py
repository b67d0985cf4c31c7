"""Builds of one tile (one launch, build.cu's small_kernel) and the warp-level
bottom of the subtree phase (subtree.cuh) against the oracle: sizes around a
warp, the tile and the general sequence's first size, ties, explicit dims at
any place of the record, odd strides.  Plus the visiting order of large query
batches (morton.cu's query_order): answers do not depend on it.
"""
import numpy as np
import pytest
import torch

import cudakdtree_b200 as ck
from oracle import pyoracle as po
from tests.helpers import make_points, make_queries

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 4, 15, 31, 32, 33, 47, 63, 64, 65, 96, 500, 511, 513, 1000, 1023, 1024, 1025,
         1500, 2047, 4095)


@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("kind", ["uniform", "tie", "same", "gmm"])
@pytest.mark.parametrize("D,stride,poff,doff,shift", [
    (2, 8, 0, -1, 0), (3, 12, 0, -1, 0), (4, 16, 0, -1, 0), (3, 16, 0, 12, 30), (3, 20, 4, 0, 0),
    (4, 36, 8, 28, 3), (2, 44, 0, 40, 0), (8, 36, 4, 0, 0)])
def test_small_builds_match_oracle(scalar, kind, D, stride, poff, doff, shift):
    for n in SIZES:
        pts = make_points(n, D, kind, scalar=scalar, seed=n)
        perm, dims, bounds = po.build(pts, explicit_dim=doff >= 0)
        rng = np.random.Generator(np.random.MT19937(n))
        rec = rng.integers(0, 2 ** 31, size=(n, stride // 4), dtype=np.int64).astype(np.int32)
        rec[:, poff // 4:poff // 4 + D] = pts.view(np.int32)
        bits = 32 - shift
        lay = ck.layout_for(scalar, D, stride=stride, point_offset=poff, dim_offset=doff,
                            dim_shift=shift, dim_bits=bits)
        d = torch.from_numpy(rec).cuda()
        wb = ck.build_tree(d, layout=lay)
        out = d.cpu().numpy()
        want = rec[perm].copy()
        if doff >= 0:
            word = want[:, doff // 4].view(np.uint32)
            mask = np.uint32(((1 << bits) - 1) << shift)
            word[:] = (word & ~mask) | (dims.astype(np.uint32) << np.uint32(shift))
        assert np.array_equal(out, want), n
        assert np.array_equal(wb.cpu().numpy(), bounds), n


@pytest.mark.parametrize("D", [2, 3, 4])
@pytest.mark.parametrize("scalar", ["float32", "int32"])
def test_visiting_order_of_large_batches(D, scalar):
    tree = torch.from_numpy(make_points(500, D, "uniform", scalar=scalar, seed=1)).cuda()
    wb = ck.build_tree(tree)
    for nq in (16385, 70001, (1 << 22) + 5):  # three sort passes; four
        q = torch.from_numpy(make_queries(nq, D, "uniform", scalar=scalar, seed=2)).cuda()
        for f in (lambda m: ck.fcp(tree, q, "cct", world_bounds=wb, with_d2=True, morton=m),
                  lambda m: ck.knn(tree, q, 2, "cct", world_bounds=wb, morton=m)):
            for x, y in zip(f(True), f(False)):
                assert torch.equal(x, y)
