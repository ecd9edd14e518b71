"""Local systems solved two or four to a warp: edges of the row classes (16, 32), points left over in
the last warp, odd feature counts and unaligned inputs, against the FP64 oracle.  Tolerances as in
test_gpu_loglik.py (FP64 1e-10 / 1e-9, FP32 1e-5) and test_gpu_predict.py; FP32 inputs run with every
system re-solved in FP64 where the log-likelihood of a few points cancels to near zero."""
import numpy as np
import pytest
import torch

from nngpr_b200 import _lib, ops
from nngpr_b200.kernel_params import extract
from oracle import nngp_oracle as O
from sklearn.gaussian_process import kernels as skk

from _common import oracle_params, rel

pytestmark = pytest.mark.gpu


def problem(n, d, m, ard, ydim, seed, nu=None):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 1, (n, d)).astype(np.float32).astype(np.float64)
    y = (np.sin(4 * x[:, :1]) + rng.normal(0, 0.1, (n, ydim))).astype(np.float32).astype(np.float64)
    ls = rng.uniform(0.3, 0.9, d) if ard and d > 1 else 0.5
    stat = skk.RBF(ls) if nu is None else skk.Matern(ls, nu=nu)
    p = extract(skk.ConstantKernel(0.9) * stat + skk.ConstantKernel(0.2) + skk.WhiteKernel(0.05))
    return x, y, p, O.fit_neighbours(x, m, p.length_scale, np.float32)


def unaligned(a, dtype):
    """The array on the device, one element past a 16-byte boundary."""
    buf = torch.zeros(a.size + 1, dtype=dtype, device='cuda')
    t = buf[1:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    assert t.data_ptr() % 16 != 0
    return t


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('m', [1, 8, 15, 16, 17, 31, 32])
@pytest.mark.parametrize('d,ard', [(1, False), (3, True), (4, False), (6, True), (7, False), (16, True)])
def test_loglik_row_classes_and_tails(dtype, m, d, ard):
    tol = 1e-2 if dtype == torch.float64 else 1e30
    for n, ydim in ((m + 2, 1), (67, 2)):
        x, y, p, nbr = problem(n, d, m, ard, ydim, 100 * d + m)
        want_l, want_g = O.log_marginal_likelihood(x, y, nbr, oracle_params(p), 1e-8, True)
        nt = torch.from_numpy(np.ascontiguousarray(nbr, dtype=np.int32)).cuda()
        for put in (lambda a: torch.from_numpy(a).to('cuda', dtype), lambda a: unaligned(a, dtype)):
            out = ops.loglik(put(x), put(y), nt, p, 1e-8, True, tol).cpu().numpy()
            assert abs(out[0] - want_l) < 1e-10 * abs(want_l)
            assert rel(out[1:], want_g) < 1e-9
            only = ops.loglik(put(x), put(y), nt, p, 1e-8, False, tol).cpu().numpy()
            assert abs(only[0] - want_l) < 1e-10 * abs(want_l)


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('m', [33, 47, 63, 64, 65, 80])
def test_more_than_32_neighbours(dtype, m):
    """FP64 systems whatever the inputs: one warp per point up to 64 neighbours, one CTA above."""
    for d, ard, ydim in ((3, False, 1), (6, True, 3)):
        x, y, p, nbr = problem(m + 37, d, m, ard, ydim, m + d)
        want_l, want_g = O.log_marginal_likelihood(x, y, nbr, oracle_params(p), 1e-8, True)
        nt = torch.from_numpy(np.ascontiguousarray(nbr, dtype=np.int32)).cuda()
        xt, yt = torch.from_numpy(x).to('cuda', dtype), torch.from_numpy(y).to('cuda', dtype)
        out = ops.loglik(xt, yt, nt, p, 1e-8, True).cpu().numpy()
        assert abs(out[0] - want_l) < 1e-10 * abs(want_l)
        assert rel(out[1:], want_g) < 1e-9
        only = ops.loglik(xt, yt, nt, p, 1e-8, False).cpu().numpy()
        assert abs(only[0] - want_l) < 1e-10 * abs(want_l)
        xq = np.random.default_rng(m).uniform(0, 1, (9, d)).astype(np.float32).astype(np.float64)
        nq = O.knn(x, xq, m, None, p.length_scale)
        want, std = O.predict(x, y, xq, nq, oracle_params(p), 1e-8)
        mean, var = ops.predict(xt, yt, torch.from_numpy(xq).to('cuda', dtype),
                                torch.from_numpy(np.ascontiguousarray(nq, dtype=np.int32)).cuda(), p, 1e-8)
        lim = 1e-10 if dtype == torch.float64 else 1e-6
        assert np.max(np.abs(mean.cpu().numpy() - want)) < lim * max(1.0, np.max(np.abs(want)))
        assert np.max(np.abs(np.sqrt(var.cpu().numpy().astype(np.float64)) - std)) < lim * np.max(std)


@pytest.mark.parametrize('m', [16, 32, 50])
def test_matern_groups(m):
    for nu in (0.5, 2.5):
        x, y, p, nbr = problem(131, 5, m, True, 1, m, nu)
        want_l, want_g = O.log_marginal_likelihood(x, y, nbr, oracle_params(p), 1e-8, True)
        out = ops.loglik(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(),
                         torch.from_numpy(np.ascontiguousarray(nbr, dtype=np.int32)).cuda(), p, 1e-8, True).cpu().numpy()
        assert abs(out[0] - want_l) < 1e-10 * abs(want_l)
        assert rel(out[1:], want_g) < 1e-9


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('m', [5, 16, 32])
@pytest.mark.parametrize('nq', [1, 3, 70])
def test_predict_groups(dtype, m, nq):
    """A warp may hold FP32 systems that pass and that are re-solved in FP64 (threshold between their
    pivots), which must give the same predictions."""
    x, y, p, _ = problem(300, 3, m, False, 2, 7 * m + nq)
    xq = np.random.default_rng(nq).uniform(0, 1, (nq, 3)).astype(np.float32).astype(np.float64)
    nbr = O.knn(x, xq, m, None, p.length_scale)
    want, std = O.predict(x, y, xq, nbr, oracle_params(p), 1e-8)
    put = lambda a: torch.from_numpy(a).to('cuda', dtype)
    nt = torch.from_numpy(np.ascontiguousarray(nbr, dtype=np.int32)).cuda()
    for tol in (0.0, 0.08, 1e30):
        mean, var = ops.predict(put(x), put(y), put(xq), nt, p, 1e-8, pivot_tol=tol)
        lim = 1e-10 if dtype == torch.float64 else 1e-5
        assert np.max(np.abs(mean.cpu().numpy() - want)) < lim * max(1.0, np.max(np.abs(want)))
        assert np.max(np.abs(np.sqrt(var.cpu().numpy().astype(np.float64)) - std)) < lim * np.max(std)


def test_partly_resolved_warps_count():
    """The FP64 re-solve count equals the systems below the threshold whatever warp they share."""
    x, y, p, nbr = problem(1000, 3, 32, False, 1, 3)
    xt, yt = torch.from_numpy(x).float().cuda(), torch.from_numpy(y).float().cuda()
    nt = torch.from_numpy(np.ascontiguousarray(nbr, dtype=np.int32)).cuda()
    want = ops.loglik(xt.double(), yt.double(), nt, p, 1e-8, True).cpu().numpy()
    counts = []
    for tol in (1e-6, 0.048, 0.06, 1e30):
        flags, st = ops.new_flags(xt.device), {}
        out = ops.loglik(xt, yt, nt, p, 1e-8, True, tol, flags=flags, stats=st).cpu().numpy()
        counts.append(int(st['fp64_systems'].item()))
        assert abs(out[0] - want[0]) < 1e-5 * abs(want[0]) and rel(out[1:], want[1:]) < 1e-5
        assert bool(int(flags.item()) & _lib.NNGP_FLAG_FP64_FALLBACK) == (counts[-1] > 0)
    assert counts[0] == 0 and counts[-1] == 1000 and counts == sorted(counts)
