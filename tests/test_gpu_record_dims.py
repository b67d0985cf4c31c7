"""Records whose split dim is none of the point's (an array that was not built
with this layout): the searches read such a dim as the first one and never a
word outside the record."""
import pytest
import torch

import cudakdtree_b200 as ck
from tests.helpers import make_points, make_queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,stride,doff", [(2, 16, 8), (3, 16, 12), (3, 20, 16), (4, 32, 16)])
@pytest.mark.parametrize("nq", [100, 17000])
def test_dims_beyond_the_point(D, stride, doff, nq):
    n = 3000
    tree = torch.zeros((n, stride // 4), dtype=torch.int32, device="cuda")
    tree[:, :D] = torch.from_numpy(make_points(n, D, "uniform", seed=1)).cuda().view(torch.int32)
    lay = ck.layout_for("float32", D, stride=stride, dim_offset=doff)
    wb = ck.compute_bounds(tree, layout=lay)
    q = torch.from_numpy(make_queries(nq, D, "uniform", seed=2)).cuda()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    for dims in (torch.full((n,), D, device="cuda"), torch.full((n,), -1, device="cuda"),
                 torch.randint(-2 ** 31, 2 ** 31 - 1, (n,), device="cuda", generator=gen)):
        tree[:, doff // 4] = dims.to(torch.int32)
        for method in ("stack_based", "stack_free", "cct"):
            outs = [ck.fcp(tree, q, method, layout=lay, world_bounds=wb)]
            outs += [ck.knn(tree, q, k, method, layout=lay, world_bounds=wb)[0] for k in (1, 8, 40)]
            for ids in outs:
                assert int(ids.min()) >= -1 and int(ids.max()) < n
