"""Builds of up to 1024 wide records: the one-launch kernel up to a size of the
array, the general sequence beyond it (build.cu), both against the oracle."""
import numpy as np
import pytest
import torch

import cudakdtree_b200 as ck
from oracle import pyoracle as po
from tests.helpers import make_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stride,doff,shift", [(192, -1, 0), (240, 236, 0), (244, 40, 30),
                                               (480, -1, 0), (1024, 1020, 4)])
@pytest.mark.parametrize("kind", ["uniform", "tie"])
def test_wide_records_match_oracle(stride, doff, shift, kind):
    for n in (100, 511, 512, 513, 777, 1023, 1024, 1025):
        pts = make_points(n, 3, kind, seed=n)
        perm, dims, bounds = po.build(pts, explicit_dim=doff >= 0)
        rng = np.random.Generator(np.random.MT19937(n))
        rec = rng.integers(0, 2 ** 31, size=(n, stride // 4), dtype=np.int64).astype(np.int32)
        rec[:, 2:5] = pts.view(np.int32)
        lay = ck.layout_for("float32", 3, stride=stride, point_offset=8, dim_offset=doff,
                            dim_shift=shift, dim_bits=2 if shift == 30 else 32 - shift)
        d = torch.from_numpy(rec).cuda()
        before = ck.launch_count()
        wb = ck.build_tree(d, layout=lay)
        one = n <= 512 or (n <= 1024 and n * stride <= 240 * 1024)
        assert (ck.launch_count() - before == 1) == one
        want = rec[perm].copy()
        if doff >= 0:
            word = want[:, doff // 4].view(np.uint32)
            mask = np.uint32(((1 << (32 - shift)) - 1) << shift)
            word[:] = (word & ~mask) | (dims.astype(np.uint32) << np.uint32(shift))
        assert np.array_equal(d.cpu().numpy(), want), n
        assert np.array_equal(wb.cpu().numpy(), bounds), n
