"""Prefix search with cells (9 features, 131,072 points and more): rows grouped and refs tiled by k-means
cell, tiles excluded by the slab between two cells.  Lists stay bit-identical."""
import numpy as np
import pytest
import torch

from nngpr_b200 import ops

pytestmark = pytest.mark.gpu


def mixture(n, d, parts, seed):
    rng = np.random.default_rng(seed)
    means = rng.uniform(-3, 3, (parts, d))
    return means[rng.integers(0, parts, n)] + 0.5 * rng.normal(size=(n, d))


def search(monkeypatch, t, q, m, cut, ls, prune):
    monkeypatch.setenv('NNGP_KNN_PRUNE', '1' if prune else '0')
    flags = ops.new_flags(t.device)
    out = ops.knn(t, q, m, cut, ls, flags=flags)
    assert int(flags.item()) == 0
    return out


@pytest.mark.parametrize('n,d,parts,m', [(131072, 9, 64, 32), (140003, 12, 7, 16), (262145, 16, 200, 32),
                                         (150000, 18, 1, 32), (140001, 24, 30, 1)])
def test_lists_equal_the_unpruned_search(monkeypatch, capfd, n, d, parts, m):
    x = torch.from_numpy(mixture(n, d, parts, n % 97).astype(np.float32)).cuda()
    ls = np.linspace(0.5, 1.5, d) if d % 2 else 0.8
    monkeypatch.setenv('NNGP_KNN_DEBUG', '1')
    a = search(monkeypatch, x, x, m, 0, ls, True)
    assert 'pruned=1' in capfd.readouterr().err
    monkeypatch.setenv('NNGP_KNN_DEBUG', '0')
    assert torch.equal(a, search(monkeypatch, x, x, m, 0, ls, False))
    r0, r1 = n // 3, n // 3 + 30000  # a row shard plans its own rows over the same cells
    assert torch.equal(search(monkeypatch, x, x[r0:r1], m, r0, ls, True), a[r0:r1])


def test_duplicates_outliers_and_equal_pivots(monkeypatch):
    """Half of the points in 40 places (pivots coincide, ties by index), far outliers, sorted input."""
    rng = np.random.default_rng(8)
    x = mixture(135000, 10, 20, 4)
    x[::2] = x[rng.integers(0, 40, x[::2].shape[0])]
    x[[5, 70000, 134999]] = [[1e6] * 10, [-1e6] * 10, [3e5] * 10]
    x = x[np.lexsort(x.T[:2])]
    t = torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).cuda()
    assert torch.equal(search(monkeypatch, t, t, 32, 0, 0.7, True), search(monkeypatch, t, t, 32, 0, 0.7, False))
