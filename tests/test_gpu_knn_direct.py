"""The direct search (refs spread over a CTA's threads): bit-exact lists against the oracle at the sizes
where it can go wrong, and the dispatch between it and the other kernels."""
import numpy as np
import pytest
import torch

from nngpr_b200 import ops
from oracle import nngp_oracle as O

pytestmark = pytest.mark.gpu


def run(monkeypatch, ref, q, m, cut, ls, dtype, kernel='direct'):
    monkeypatch.setenv('NNGP_KNN_KERNEL', kernel)
    r = torch.from_numpy(np.ascontiguousarray(ref, dtype=dtype)).cuda()
    qq = r if q is ref else torch.from_numpy(np.ascontiguousarray(q, dtype=dtype)).cuda()
    flags = ops.new_flags(r.device)
    out = ops.knn(r, qq, m, cut, ls, flags=flags).cpu().numpy()
    assert int(flags.item()) == 0
    return out


@pytest.mark.parametrize('dtype', [np.float32, np.float64])
@pytest.mark.parametrize('d', [1, 4, 5, 8, 12, 16, 20, 24, 26, 32, 40])
@pytest.mark.parametrize('m', [1, 32, 33, 128])
def test_direct_prefix_and_queries_match_oracle(monkeypatch, dtype, d, m):
    """Around one thread's refs (256) and the four-queries-per-CTA line (1,184 queries)."""
    rng = np.random.default_rng(10 * d + m)
    x = rng.uniform(-1, 1, (1300, d))
    ls = rng.uniform(0.3, 2.0, d) if d % 2 else 0.4
    assert np.array_equal(run(monkeypatch, x, x, m, 0, ls, dtype), O.knn(x, x, m, 0, ls, dtype))
    for n, nq in ((1, 3), (m, 5), (255, 7), (257, 1), (1025, 2)):
        q = rng.uniform(-1.2, 1.2, (nq, d))
        assert np.array_equal(run(monkeypatch, x[:n], q, m, None, ls, dtype), O.knn(x[:n], q, m, None, ls, dtype))
    q = rng.uniform(-1, 1, (1187, d))
    for cut in (-3, 2, 5000):
        assert np.array_equal(run(monkeypatch, x[:900], q, m, cut, ls, dtype), O.knn(x[:900], q, m, cut, ls, dtype))


@pytest.mark.parametrize('dtype', [np.float32, np.float64])
def test_direct_ties_overflow_the_candidate_list(monkeypatch, dtype):
    """Lattice points and all-equal points: more refs at the m-th distance than the list holds, the lower
    indices win; and refs of one query's list that all fall to one thread (every 256th point near)."""
    rng = np.random.default_rng(5)
    x = rng.integers(0, 3, (4000, 3)).astype(np.float64)
    assert np.array_equal(run(monkeypatch, x, x, 32, 0, None, dtype), O.knn(x, x, 32, 0, None, dtype))
    same = np.ones((3000, 2))
    assert np.array_equal(run(monkeypatch, same, same[:9], 128, None, None, dtype), O.knn(same, same[:9], 128, None, None, dtype))
    y = rng.uniform(5, 6, (256 * 40, 3))
    y[7::256] = rng.uniform(0, 0.1, (40, 3))
    q = rng.uniform(0, 0.1, (11, 3))
    assert np.array_equal(run(monkeypatch, y, q, 32, None, None, dtype), O.knn(y, q, 32, None, None, dtype))


@pytest.mark.parametrize('dtype', [np.float32, np.float64])
def test_direct_skips_nan_and_infinite_distances(monkeypatch, dtype):
    """As the generic kernel: refs at a NaN or infinite distance are never listed."""
    rng = np.random.default_rng(6)
    x = rng.normal(size=(700, 3))
    x[5] = np.nan
    x[300, 1] = np.inf
    x[301, 2] = -np.inf
    x[400] = 1e200 if dtype == np.float64 else 1e30
    q = x[:600:50]
    with np.errstate(all='ignore'):
        a = run(monkeypatch, x, q, 32, None, None, dtype)
        b = run(monkeypatch, x, q, 32, None, None, dtype, 'generic')
    assert np.array_equal(a, b)


@pytest.mark.parametrize('n,nq,d,m,want', [(2000, 256, 3, 32, True), (16599, 1000, 18, 32, True), (434874, 64, 3, 32, True),
                                           (100000, 16384, 3, 32, False), (16384, 0, 8, 32, True),
                                           (16385, 0, 8, 32, False), (30000, 0, 3, 48, True), (3000, 40, 30, 16, True)])
def test_direct_dispatch(monkeypatch, capfd, n, nq, d, m, want):
    """Auto selection takes the direct search for few queries (nq 0: a prefix search of the set), with the
    screened kernels' lists."""
    gen = torch.Generator(device='cuda').manual_seed(n + d)
    x = torch.rand((n, d), generator=gen, device='cuda')
    q = torch.rand((nq, d), generator=gen, device='cuda') if nq else x
    monkeypatch.setenv('NNGP_KNN_DEBUG', '1')
    a = ops.knn(x, q, m, None if nq else 0, 0.3)
    assert ('direct path' in capfd.readouterr().err) == want
    monkeypatch.setenv('NNGP_KNN_KERNEL', 'tc' if m <= 32 and d <= 24 else 'simt')
    assert torch.equal(a, ops.knn(x, q, m, None if nq else 0, 0.3))
