"""Builds and searches with a caller's memory resource that limits the size of
its blocks: what the single arrays fit is enough."""
import ctypes as C

import pytest
import torch

import cudakdtree_b200 as ck
from tests.helpers import make_points, make_queries

pytestmark = pytest.mark.gpu


class _Limited:
    """A memory resource whose blocks have at most `limit` bytes."""

    def __init__(self, limit):
        self.blocks, self.refused = {}, 0

        def alloc(ctx, out, nbytes, stream):
            if nbytes > limit:
                self.refused += 1
                return 1
            buf = torch.empty(int(nbytes), dtype=torch.uint8, device="cuda")
            self.blocks[buf.data_ptr()] = buf
            out[0] = buf.data_ptr()
            return 0

        def release(ctx, ptr, stream):
            self.blocks.pop(ptr)
            return 0

        self.fns = ck._ALLOC_FN(alloc), ck._RELEASE_FN(release)
        self.mr = ck.MemResource(None, *(C.cast(f, C.c_void_p) for f in self.fns))


@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("stride,doff", [(12, -1), (16, 12)])
def test_build_and_search_with_limited_blocks(scalar, stride, doff):
    n, nq, k = 60000, 900_000, 8
    lay = ck.layout_for(scalar, 3, stride=stride, dim_offset=doff)
    rec = torch.zeros((n, stride // 4), dtype=torch.int32, device="cuda")
    rec[:, :3] = torch.from_numpy(make_points(n, 3, "uniform", scalar=scalar,
                                              seed=1)).cuda().view(torch.int32)
    want = rec.clone()
    wb = ck.build_tree(want, layout=lay)
    # the largest single array of the build is the record copy, of the search
    # one with a word per query
    res = _Limited(n * stride + 4096)
    got_wb = torch.empty_like(wb)
    st = ck._stream(None)
    ck._check(ck.lib().cukd_build_tree(rec.data_ptr(), n, C.byref(lay), got_wb.data_ptr(), 0, st,
                                       C.byref(res.mr)), "cukd_build_tree")
    torch.cuda.synchronize()
    assert res.refused >= 1 and not res.blocks
    assert torch.equal(rec, want) and torch.equal(got_wb, wb)
    q = torch.from_numpy(make_queries(nq, 3, "uniform", scalar=scalar, seed=2)).cuda()
    wi, wd = ck.knn(want, q, k, layout=lay, world_bounds=wb)
    res = _Limited(nq * 4 + 4096)
    p = ck._params("stack_based", k)
    ids, d2 = torch.empty_like(wi), torch.empty_like(wd)
    ck._check(ck.lib().cukd_knn(want.data_ptr(), n, C.byref(lay), wb.data_ptr(), q.data_ptr(), nq,
                                C.byref(p), ids.data_ptr(), d2.data_ptr(), None, st,
                                C.byref(res.mr)), "cukd_knn")
    torch.cuda.synchronize()
    assert res.refused >= 1 and not res.blocks
    assert torch.equal(ids, wi) and torch.equal(d2, wd)
