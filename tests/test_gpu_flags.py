"""CUKD_QUERY_WARP_PACKET and CUKD_QUERY_TREE_ORDER take effect at every number
of queries: few queries, which otherwise go to the warp-per-query kernel, run
the asked-for kernel or order, and the packet kernel's queries are sorted
(counted by the library's launches: answers are the same by construction)."""
import pytest
import torch

import cudakdtree_b200 as ck
from tests.helpers import make_points, make_queries

pytestmark = pytest.mark.gpu


def _launches(f):
    before = ck.launch_count()
    out = f()
    torch.cuda.synchronize()
    return ck.launch_count() - before, out


@pytest.mark.parametrize("nq", [101, 5003, 17003])
def test_flags_take_effect(nq):
    tree = torch.from_numpy(make_points(20000, 3, "uniform", seed=1)).cuda()
    wb = ck.build_tree(tree)
    q = torch.from_numpy(make_queries(nq, 3, "uniform", seed=2)).cuda()
    plain, want = _launches(lambda: ck.knn(tree, q, 8, world_bounds=wb))
    for kw in ({"warp_packet": True}, {"tree_order": True}):
        count, got = _launches(lambda: ck.knn(tree, q, 8, world_bounds=wb, **kw))
        bare, same = _launches(lambda: ck.knn(tree, q, 8, world_bounds=wb, morton=False,
                                              **({} if "tree_order" in kw else kw)))
        assert count > plain and count > bare  # a sort before the search
        for x, y, z in zip(got, want, same):
            assert torch.equal(x, y) and torch.equal(z, y)
    f = lambda **kw: ck.fcp(tree, q, world_bounds=wb, with_d2=True, **kw)
    few, want = _launches(f)
    count, got = _launches(lambda: f(tree_order=True))
    assert count > few
    for x, y in zip(got, want):
        assert torch.equal(x, y)
