"""kNN lists of the stack-free traversal with eps are the exact ones unless the
k-th distance ties (where they are the traversal's), also when distances lie
so close that the search's truncated keys cannot tell them apart."""
import ctypes as C

import numpy as np
import pytest
import torch

import cudakdtree_b200 as ck

pytestmark = pytest.mark.gpu


def _shell(n, scalar, rng):
    """Points whose squared distances from the origin are 20 ulps (ints: 2^-19
    of them) apart, in random directions."""
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    r = np.sqrt(1 + np.arange(n) * 20 * 2.0 ** -23)[:, None]
    return (v * r).astype(np.float32) if scalar == "float32" else np.rint(v * r * 2 ** 24).astype(np.int32)


@pytest.mark.parametrize("scalar", ["float32", "int32"])
@pytest.mark.parametrize("k", [3, 31, 32, 100, 127])
@pytest.mark.parametrize("nq", [300, 17000])
def test_near_equal_distances(scalar, k, nq):
    rng = np.random.Generator(np.random.MT19937(k))
    tree = torch.from_numpy(_shell(20000, scalar, rng)).cuda()
    wb = ck.build_tree(tree)
    q = rng.standard_normal((nq, 3)) * 1e-4
    q = torch.from_numpy(q.astype(np.float32) if scalar == "float32"
                         else np.rint(q * 2 ** 24).astype(np.int32)).cuda()
    wi, wd = ck.knn(tree, q, k + 1, "stack_based", world_bounds=wb)
    clear = wd[:, k] > wd[:, k - 1]  # no tie at the k-th distance
    assert int(clear.sum()) > nq // 2
    p = ck._params("stack_free", k, eps=0.5)
    ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    d2 = torch.empty((nq, k), dtype=wd.dtype, device="cuda")
    lay = ck.infer_layout(tree)
    ck._check(ck.lib().cukd_knn(ck._ptr(tree), len(tree), C.byref(lay), ck._ptr(wb), ck._ptr(q), nq,
                                C.byref(p), ck._ptr(ids), ck._ptr(d2), None, ck._stream(None),
                                None), "cukd_knn")
    assert torch.equal(ids[clear], wi[clear, :k])
    assert torch.equal(d2[clear], wd[clear, :k])


@pytest.mark.parametrize("k", [3, 100])
def test_near_equal_distances_in_clouds(k):
    n, nq = 20000, 3000
    rng = np.random.Generator(np.random.MT19937(k + 1))
    pts = torch.from_numpy(np.concatenate([_shell(n, "float32", rng) for _ in range(2)])).cuda()
    q = torch.from_numpy((rng.standard_normal((2 * nq, 3)) * 1e-4).astype(np.float32)).cuda()
    plan = ck.BatchPlan([0, n, 2 * n], [0, nq, 2 * nq], num_dims=3, k=k, method="stack_free",
                        eps=0.5)
    tree = pts.clone()
    ids, d2 = plan.run(tree, q)
    for c in range(2):
        own = pts[c * n:(c + 1) * n].clone()
        wb = ck.build_tree(own)
        assert torch.equal(own, tree[c * n:(c + 1) * n])
        part = slice(c * nq, (c + 1) * nq)
        wi, wd = ck.knn(own, q[part], k + 1, "stack_based", world_bounds=wb)
        clear = wd[:, k] > wd[:, k - 1]
        assert int(clear.sum()) > nq // 2
        assert torch.equal(ids[part][clear], wi[clear, :k])
        assert torch.equal(d2[part][clear], wd[clear, :k])
