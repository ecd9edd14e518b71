"""One or two rows of a local system per lane: both forms on either side of the lines between them (points, features),
with points left over in the last warp, against the FP64 oracle.  Tolerances as in test_gpu_local_groups.py."""
import numpy as np
import pytest
import torch

from nngpr_b200 import ops
from nngpr_b200.kernel_params import extract
from oracle import nngp_oracle as O
from sklearn.gaussian_process import kernels as skk

from _common import oracle_params, rel

pytestmark = pytest.mark.gpu


def check(n, d, m, dtype, ard=False, ydim=1, nu=None):
    rng = np.random.default_rng(1000 * m + d + n)
    x = rng.uniform(0, 1, (n, d)).astype(np.float32).astype(np.float64)
    y = (np.sin(4 * x[:, :1]) + rng.normal(0, 0.1, (n, ydim))).astype(np.float32).astype(np.float64)
    wide = max(1.0, (d / 8) ** 0.5)
    ls = rng.uniform(0.3, 0.9, d) * wide if ard else 0.5 * wide
    stat = skk.RBF(ls) if nu is None else skk.Matern(ls, nu=nu)
    p = extract(skk.ConstantKernel(0.9) * stat + skk.ConstantKernel(0.2) + skk.WhiteKernel(0.05))
    nbr = O.fit_neighbours(x, m, p.length_scale, np.float32)
    want_l, want_g = O.log_marginal_likelihood(x, y, nbr, oracle_params(p), 1e-8, True)
    xt, yt = torch.from_numpy(x).to('cuda', dtype), torch.from_numpy(y).to('cuda', dtype)
    nt = torch.from_numpy(np.ascontiguousarray(nbr, dtype=np.int32)).cuda()
    tight = dtype == torch.float64
    out = ops.loglik(xt, yt, nt, p, 1e-8, True).cpu().numpy()
    assert abs(out[0] - want_l) < (1e-10 if tight else 1e-5) * abs(want_l)
    assert rel(out[1:], want_g) < (1e-9 if tight else 1e-5)
    only = ops.loglik(xt, yt, nt, p, 1e-8, False).cpu().numpy()
    assert abs(only[0] - want_l) < (1e-10 if tight else 1e-5) * abs(want_l)
    nq = O.knn(x, x, m, None, p.length_scale)
    mean, var = ops.predict(xt, yt, xt, torch.from_numpy(nq.astype(np.int32)).cuda(), p, 1e-8)
    wm, ws = O.predict(x, y, x, nq, oracle_params(p), 1e-8)
    tol = 1e-10 if tight else 1e-5
    assert np.max(np.abs(mean.cpu().numpy().astype(np.float64) - wm)) < tol * max(1.0, np.max(np.abs(wm)))
    assert np.max(np.abs(np.sqrt(var.cpu().numpy().astype(np.float64)) - ws)) < tol * max(1.0, np.max(ws))


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('n,m', [(5, 32), (1036, 32), (1037, 32), (1039, 17), (3256, 16), (3257, 16), (3259, 9)])
@pytest.mark.parametrize('d,ard,ydim,nu', [(3, True, 1, None), (7, False, 2, None), (16, False, 1, 1.5)])
def test_both_forms_around_the_line_of_points(dtype, n, m, d, ard, ydim, nu):
    check(n, d, m, dtype, ard, ydim, nu)


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('n,m', [(1041, 32), (3261, 8)])
@pytest.mark.parametrize('d', [27, 28, 35, 36, 55, 56, 71, 72])
def test_both_forms_around_the_line_of_features(dtype, n, m, d):
    check(n, d, m, dtype)


def test_long_rows_cost_no_more_than_their_length():
    """The work per point is a constant plus a term in d, so d = 128 may take 128 / 40 times as long as d = 40; with a
    quarter for noise 4.0.  Points that share a warp cost 5.1 there: their rows leave shared memory for few warps."""
    n, m = 30000, 32
    g = torch.Generator(device='cuda').manual_seed(3)
    nbr = torch.randint(0, n, (n, m), device='cuda', generator=g).sort(1).values.int()
    nbr = torch.where(nbr < torch.arange(n, device='cuda', dtype=torch.int32)[:, None], nbr, -1).contiguous()
    y = torch.rand((n, 1), device='cuda', dtype=torch.float64, generator=g)
    took = []
    for d in (40, 128):
        x = torch.rand((n, d), device='cuda', dtype=torch.float64, generator=g)
        p = extract(skk.ConstantKernel() * skk.RBF(0.5 * d ** 0.5) + skk.WhiteKernel(1e-2))
        best = float('inf')
        for _ in range(9):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            ops.loglik(x, y, nbr, p, 1e-10, False)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        took.append(best)
    assert took[1] < 4.0 * took[0], took
