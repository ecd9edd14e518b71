"""The direct search on points whose near refs lie a fixed number of places apart (grids by rows, periods) or in
the same place: the lists are the oracle's, and the time stays near that of random points.  And on
refs chosen so that the near ones all fall to one thread in spite of its hash."""
import numpy as np
import pytest
import torch

from nngpr_b200 import ops
from oracle import nngp_oracle as O

pytestmark = pytest.mark.gpu


def grid(w, h):
    y, x = np.meshgrid(np.arange(h), np.arange(w), indexing='ij')
    return np.stack([x.ravel(), y.ravel()], 1).astype(np.float64)


def places(rng, n):
    x = rng.uniform(0, 1, (n, 2))
    k = rng.permutation(n)[:n // 2]
    x[k] = rng.uniform(0, 1, (20, 2))[rng.integers(0, 20, n // 2)]
    return x


def layout(name):
    rng = np.random.default_rng(11)
    if name == 'places':
        return places(rng, 100000)
    if name == 'period':
        t = np.arange(16384.0)
        return np.stack([np.sin(2 * np.pi * t / 256), np.cos(2 * np.pi * t / 256), t / 16384], 1)
    return grid(*map(int, name.split('x')))


def cuda(x, dtype):
    return torch.from_numpy(np.ascontiguousarray(x, dtype=dtype)).cuda()


@pytest.mark.parametrize('dtype', [np.float32, np.float64])
@pytest.mark.parametrize('name', ['256x64', '128x128', '512x40', 'period', 'places'])
@pytest.mark.parametrize('nq,m', [(300, 32), (1500, 32), (300, 128), (1500, 100)])
def test_lists_match_the_oracle(monkeypatch, dtype, name, nq, m):
    monkeypatch.setenv('NNGP_KNN_KERNEL', 'direct')
    x = layout(name)
    rng = np.random.default_rng(nq + m)
    q = x[rng.choice(len(x), nq, replace=False)]
    got = ops.knn(cuda(x, dtype), cuda(q, dtype), m, None, None).cpu().numpy()
    rows = np.arange(0, nq, nq // 60)
    assert np.array_equal(got[rows], O.knn(x, q[rows], m, None, None, dtype))


@pytest.mark.parametrize('dtype', [np.float32, np.float64])
@pytest.mark.parametrize('m', [32, 128])
def test_prefix_lists_of_grid_points_match_the_oracle(monkeypatch, dtype, m):
    monkeypatch.setenv('NNGP_KNN_KERNEL', 'direct')
    x = grid(256, 20)
    t = cuda(x, dtype)
    assert np.array_equal(ops.knn(t, t, m, 0, None).cpu().numpy(), O.knn(x, x, m, 0, None, dtype))


def turn(g):
    h = (g.astype(np.uint64) * 0x9E3779B1) & 0xFFFFFFFF
    h = ((h ^ (h >> np.uint64(15))) * 0x85EBCA6B) & 0xFFFFFFFF
    return (h >> np.uint64(24)).astype(np.int64)


@pytest.mark.parametrize('dtype', [np.float32, np.float64])
@pytest.mark.parametrize('nq,blocks', [(9, 4), (1300, 1)])
def test_near_refs_in_one_thread_overflow_the_list(monkeypatch, dtype, nq, blocks):
    """1,200 near refs in one thread (blocks: blocks of 256 refs that share a hash), three of them kept."""
    monkeypatch.setenv('NNGP_KNN_KERNEL', 'direct')
    rng = np.random.default_rng(3)
    j = np.arange(256 * 1200)
    k = j // 256
    thread = (j % 256) ^ turn(k // blocks) ^ (k % blocks * 64)
    x = rng.uniform(5, 6, (len(j), 3))
    near = thread == 77
    assert near.sum() == 1200
    x[near] = rng.uniform(0, 0.1, (1200, 3))
    q = rng.uniform(0, 0.1, (nq, 3))
    got = ops.knn(cuda(x, dtype), cuda(q, dtype), 32, None, None).cpu().numpy()
    rows = np.arange(0, nq, max(1, nq // 9))
    assert np.array_equal(got[rows], O.knn(x, q[rows], 32, None, None, dtype))


def time_us(x, q, m):
    ops.knn(x, q, m, None, None)
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(True), torch.cuda.Event(True)
        a.record()
        ops.knn(x, q, m, None, None)
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 1e3)
    return sorted(times)[3]


@pytest.mark.parametrize('dtype', [np.float32, np.float64])
@pytest.mark.parametrize('name', ['256x64', '512x40', 'period', 'places'])
@pytest.mark.parametrize('nq', [1000, 4096])
def test_time_stays_near_that_of_random_points(monkeypatch, dtype, name, nq):
    """At most three times it: what two more passes over the refs would cost."""
    monkeypatch.setenv('NNGP_KNN_KERNEL', 'direct')
    x = layout(name)
    rng = np.random.default_rng(1)
    pick = rng.choice(len(x), nq, replace=False)
    y = rng.uniform(0, 1, x.shape)
    got = time_us(cuda(x, dtype), cuda(x[pick], dtype), 32)
    plain = time_us(cuda(y, dtype), cuda(y[pick], dtype), 32)
    assert got <= 3 * plain, (got, plain)
