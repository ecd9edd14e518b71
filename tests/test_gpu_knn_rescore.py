"""The rescoring warps of the tensor-core search: bit-exact lists against the oracle where every column of every
tile is a candidate (their rings run full), where equal distances decide, and at the sizes of a tile."""
import numpy as np
import pytest
import torch

from nngpr_b200 import ops
from oracle import nngp_oracle as O

pytestmark = pytest.mark.gpu


def run(monkeypatch, ref, q, m, cut):
    monkeypatch.setenv('NNGP_KNN_KERNEL', 'tc')
    r = torch.from_numpy(np.ascontiguousarray(ref, dtype=np.float32)).cuda()
    qq = r if q is ref else torch.from_numpy(np.ascontiguousarray(q, dtype=np.float32)).cuda()
    flags = ops.new_flags(r.device)
    out = ops.knn(r, qq, m, cut, None, flags=flags).cpu().numpy()
    assert int(flags.item()) == 0
    return out


@pytest.mark.parametrize('d', [1, 3, 4, 8, 10, 16, 18, 24])
@pytest.mark.parametrize('m', [1, 5, 31, 32])
def test_rescoring_matches_oracle(monkeypatch, d, m):
    rng = np.random.default_rng(100 * d + m)
    # each ref nearer to the origin than the one before it: no bound excludes anything
    r = rng.normal(size=(2100, d))
    r *= np.linspace(3, 0.1, len(r))[:, None] / np.linalg.norm(r, axis=1)[:, None]
    q = rng.normal(scale=1e-3, size=(290, d))
    for n in (2100, 129, 127):
        for cut in (None, -40):
            assert np.array_equal(run(monkeypatch, r[:n], q, m, cut), O.knn(r[:n], q, m, cut, None, np.float32))
    # lattice points, and all points equal: ties at the m-th distance, the lower indices win
    x = rng.integers(0, 2, (1500, d)).astype(np.float64)
    for pts in (x, x[::-1].copy(), np.ones((700, d))):
        assert np.array_equal(run(monkeypatch, pts, pts, m, 0), O.knn(pts, pts, m, 0, None, np.float32))


@pytest.mark.parametrize('d', [2, 6, 7, 8, 9, 16, 21, 24])
def test_curves_of_one_sort_match_the_direct_search(monkeypatch, d):
    """Seeds of a prefix search and of queries (both curves and the queries in one sort; from d = 7 on some shapes
    drop a key's lowest bits for the two that tell them apart), with points on one spot and a far outlier."""
    rng = np.random.default_rng(d)
    r = rng.normal(size=(9001, d)).astype(np.float32)
    r[100:400] = r[100]
    r[8200] = 1e6
    q = rng.normal(size=(16385, d)).astype(np.float32)
    q[5] = r[100]
    rt, qt = torch.from_numpy(r).cuda(), torch.from_numpy(q).cuda()
    for a, cut in ((rt, 0), (qt, None)):
        lists = []
        for kernel in ('tc', 'direct'):
            monkeypatch.setenv('NNGP_KNN_KERNEL', kernel)
            lists.append(ops.knn(rt, a, 32, cut, None))
        assert torch.equal(lists[0], lists[1])


@pytest.mark.parametrize('d', [3, 8, 16, 20])
@pytest.mark.parametrize('n,nq', [(9001, 0), (2047, 130), (4096, 700), (20001, 0), (16600, 16500)])
def test_parts_of_an_unpruned_search_match_the_direct_search(monkeypatch, d, n, nq):
    """Groups split into parts of their tiles (several in number, down to none where a prefix is short) and merged."""
    rng = np.random.default_rng(n + d)
    rt = torch.from_numpy(rng.normal(size=(n, d)).astype(np.float32)).cuda()
    rt[n // 2] = rt[n // 3]
    q = rt if nq == 0 else torch.from_numpy(rng.normal(size=(nq, d)).astype(np.float32)).cuda()
    for m, cut in ((32, 0), (5, 0)) if nq == 0 else ((32, None), (7, -100), (32, 1000)):
        lists = []
        for kernel in ('tc', 'direct'):
            monkeypatch.setenv('NNGP_KNN_KERNEL', kernel)
            lists.append(ops.knn(rt, q, m, cut, None))
        assert torch.equal(lists[0], lists[1])
