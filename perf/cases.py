"""Work that users of this framework run on one GPU, as measurable cases.

A case is one call (or the two calls that make up one operation) through the package's public entry
points: the neighbour search (``ops.knn``), the fit step's local systems (``ops.loglik``), search and
predictive systems together (``ops.knn`` + ``ops.predict``), the differentiable fit step
(``autograd.NngpLogLik``) and the estimator's ``predict``.  Sizes are those of the benchmark's
workloads (3-d 434,874 points, 8-d ARD, the 16-d mixture of a million points, the 18-d served model)
and of the test suite, and what lies between them.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from sklearn.gaussian_process import kernels as skk

from nngpr_b200 import B200Nngpr, ops
from nngpr_b200.autograd import LogLikProblem, NngpLogLik
from nngpr_b200.kernel_params import extract

ALPHA = 1e-10


def listed():
    return [
        # one log-likelihood evaluation of a small model (the CPU configuration's size): every
        # launch and host call counts, an optimiser makes hundreds of them
        {'name': 'fit_small_2k', 'kind': 'fit', 'n': 2000, 'd': 3, 'm': 16, 'data': 'uniform', 'ls': 0.3, 'ard': False,
         'noise': 0.01, 'f64': True, 'search64': False, 'ydim': 1, 'pivot_tol': 1e-2},
        # an interactive prediction through the estimator, host arrays in and out
        {'name': 'predict_call_1k', 'kind': 'predict_call', 'n': 16599, 'nq': 1000, 'd': 18, 'm': 32, 'data': 'normal',
         'ls': 0.5, 'ard': True, 'noise': 0.01},
        # one optimiser step through autograd: theta on the device, ARD, FP32 systems with FP64 re-solves
        {'name': 'fit_step_ard_8d', 'kind': 'autograd', 'n': 434874, 'd': 8, 'm': 32, 'data': 'unit', 'ls': 0.1,
         'ard': True, 'noise': 4e-4, 'f64': False, 'pivot_tol': 1e-2},
        # the fit step's search: low dimension, uniform points
        {'name': 'search_3d', 'kind': 'search', 'n': 434874, 'd': 3, 'm': 32, 'data': 'uniform', 'ls': 0.2,
         'ard': False, 'search64': False},
        # the fit step's search: a million points of a mixture in 16 dimensions
        {'name': 'search_16d', 'kind': 'search', 'n': 1000000, 'd': 16, 'm': 32, 'data': 'mixture', 'parts': 64,
         'ls': 0.8, 'ard': False, 'search64': False},
        # the FP64 search of allow_downcast_f32='no'
        {'name': 'search_f64_20k', 'kind': 'search', 'n': 20000, 'd': 3, 'm': 32, 'data': 'uniform', 'ls': 0.2,
         'ard': False, 'search64': True},
        # the fit step's local systems in FP64 (the default precision), with gradient
        {'name': 'systems_f64_3d', 'kind': 'systems', 'n': 434874, 'd': 3, 'm': 32, 'data': 'uniform', 'ls': 0.2,
         'ard': False, 'noise': 1e-3, 'f64': True, 'ydim': 1, 'pivot_tol': 1e-2, 'grad': True, 'family': 'rbf'},
        # ... in FP32 at the mixed-precision configuration's threshold
        {'name': 'systems_f32_16d', 'kind': 'systems', 'n': 1000000, 'd': 16, 'm': 32, 'data': 'mixture', 'parts': 64,
         'ls': 0.8, 'ard': False, 'noise': 1e-4, 'f64': False, 'ydim': 1, 'pivot_tol': 1e-6, 'grad': True,
         'family': 'rbf'},
        # ... with more than 32 neighbours and two outputs
        {'name': 'systems_m64', 'kind': 'systems', 'n': 20000, 'd': 4, 'm': 64, 'data': 'uniform', 'ls': 0.4,
         'ard': True, 'noise': 0.02, 'f64': True, 'ydim': 2, 'pivot_tol': 1e-2, 'grad': True, 'family': 'rbf'},
        # prediction at many points on device arrays
        {'name': 'predict_3d_100k', 'kind': 'predict', 'n': 434874, 'nq': 100000, 'd': 3, 'm': 32, 'data': 'uniform',
         'ls': 0.2, 'ard': False, 'noise': 1e-3, 'f64': True, 'ydim': 1, 'pivot_tol': 1e-2},
        # the largest batch of the served model, and its smallest
        {'name': 'predict_18d_16k', 'kind': 'predict', 'n': 16599, 'nq': 16384, 'd': 18, 'm': 32, 'data': 'normal',
         'ls': 0.5, 'ard': True, 'noise': 0.01, 'f64': False, 'ydim': 1, 'pivot_tol': 1e-2},
        {'name': 'predict_18d_256', 'kind': 'predict', 'n': 16599, 'nq': 256, 'd': 18, 'm': 32, 'data': 'normal',
         'ls': 0.5, 'ard': True, 'noise': 0.01, 'f64': False, 'ydim': 1, 'pivot_tol': 1e-2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['fit', 'predict_call', 'autograd', 'search', 'search', 'systems', 'systems', 'systems_wide',
                       'predict', 'predict', 'search64'])
    m = rng.choice([8, 13, 16, 20, 24, 30, 32, 32])
    f64 = rng.random() < 0.5
    if kind in ('search', 'systems') and rng.random() < 0.4:  # mixtures, 9 to 24 dimensions
        d = rng.randint(9, 24)
        n = _log(rng, 20000, 1e6 * min(1.0, 16 / d))
        base = {'n': n, 'd': d, 'm': m, 'data': 'mixture', 'parts': rng.choice([16, 40, 64, 100, 200]), 'ls': 0.8,
                'ard': False}
        noise = 1e-4
    elif kind in ('search', 'systems', 'fit', 'autograd'):
        d = rng.randint(1, 8)
        base = {'n': _log(rng, 1000, 434874), 'd': d, 'm': m, 'data': rng.choice(['uniform', 'unit']),
                'ls': round(0.1 * d ** 0.5, 3), 'ard': rng.random() < 0.5}
        noise = 1e-3
    elif kind == 'search64':
        return {'kind': 'search', 'n': _log(rng, 500, 20000), 'd': rng.randint(1, 12), 'm': m, 'data': 'uniform',
                'ls': 0.3, 'ard': rng.random() < 0.5, 'search64': True}
    elif kind == 'systems_wide':
        d = rng.randint(1, 8)
        return {'kind': 'systems', 'n': _log(rng, 1000, 20000), 'd': d, 'm': rng.randint(33, 64), 'data': 'uniform',
                'ls': 0.4, 'ard': rng.random() < 0.5, 'noise': 0.02, 'f64': f64, 'ydim': rng.randint(1, 3),
                'pivot_tol': 1e-2, 'grad': rng.random() < 0.8, 'family': 'rbf'}
    else:  # predict, predict_call
        d = rng.randint(2, 20)
        base = {'n': _log(rng, 2000, 434874 if d <= 4 else 50000), 'nq': _log(rng, 1, 100000 if d <= 4 else 20000),
                'd': d, 'm': m, 'data': 'normal' if d > 8 else 'uniform', 'ls': 0.5 if d > 8 else 0.3,
                'ard': rng.random() < 0.5}
        if kind == 'predict_call':
            base['n'], base['nq'] = min(base['n'], 50000), min(base['nq'], 5000)
            return dict(base, kind=kind, noise=0.01)
        return dict(base, kind=kind, noise=0.01, f64=f64, ydim=rng.randint(1, 3), pivot_tol=1e-2)
    if kind == 'search':
        return dict(base, kind='search', search64=False)
    if kind == 'autograd':
        return dict(base, kind=kind, noise=noise, f64=f64, pivot_tol=1e-2)
    if kind == 'fit':
        base['n'] = min(base['n'], 50000)
        return dict(base, kind=kind, noise=0.01, f64=f64, search64=f64 and base['n'] <= 20000 and rng.random() < 0.3,
                    ydim=rng.randint(1, 3), pivot_tol=1e-2)
    mixture = base['data'] == 'mixture'
    return dict(base, kind='systems', noise=noise, f64=f64, ydim=rng.randint(1, 2),
                pivot_tol=1e-6 if mixture else 1e-2, grad=rng.random() < 0.8,
                family=rng.choice(['rbf', 'rbf', 'rbf', 'matern32']))


# ---- inputs --------------------------------------------------------------------------------
def _points(case, n, gen, means):
    """``n`` points of the case's distribution (float64, on the GPU)."""
    d = case['d']
    if case['data'] == 'mixture':
        which = torch.randint(0, means.shape[0], (n,), generator=gen, device='cuda')
        return means[which] + 0.5 * torch.randn((n, d), generator=gen, device='cuda', dtype=torch.float64)
    if case['data'] == 'normal':
        return torch.randn((n, d), generator=gen, device='cuda', dtype=torch.float64)
    u = torch.rand((n, d), generator=gen, device='cuda', dtype=torch.float64)
    if case['data'] == 'unit':
        return u
    axis = torch.tensor([1.0, 0.7, 0.4] * 8, device='cuda', dtype=torch.float64)[:d]
    return (2 * u - 1) * axis


def _inputs(case, seed):
    """x, y (float64, on the GPU), queries (or None) and the length scale (float or numpy array)."""
    gen = torch.Generator(device='cuda').manual_seed(1000 + seed)
    d = case['d']
    means = 6 * torch.rand((case.get('parts', 1), d), generator=gen, device='cuda', dtype=torch.float64) - 3
    ls = case['ls']
    if case['ard']:  # log-uniform over a factor of ten
        ls = case['ls'] * np.exp(np.log(10.0) * np.random.default_rng(seed).uniform(size=d))
    x = _points(case, case['n'], gen, means)
    xq = _points(case, case['nq'], gen, means) if 'nq' in case else None
    # smooth outputs: random Fourier features at the length scale, plus noise
    ydim = case.get('ydim', 1)
    omega = torch.randn((128, d), generator=gen, device='cuda', dtype=torch.float64) / torch.as_tensor(
        ls, device='cuda', dtype=torch.float64)
    w = torch.randn((128, ydim), generator=gen, device='cuda', dtype=torch.float64) * (2 / 128) ** 0.5
    y = torch.cat([torch.cos(c @ omega.T) @ w for c in x.split(65536)])
    y += case.get('noise', 1e-3) ** 0.5 * torch.randn((case['n'], ydim), generator=gen, device='cuda',
                                                      dtype=torch.float64)
    return x, y, xq, ls


def _kernel(case, ls):
    part = skk.Matern(ls, nu=1.5) if case.get('family') == 'matern32' else skk.RBF(ls)
    return skk.ConstantKernel(1.0) * part + skk.WhiteKernel(case['noise'])


def _curve(x):
    """Order of the points along a Morton curve."""
    n, d = x.shape
    bits = min(10, 62 // d)
    lo, hi = x.min(0).values, x.max(0).values
    q = ((x - lo) / (hi - lo).max().clamp_min(1e-30) * (2 ** bits - 1)).to(torch.int64)
    key = torch.zeros(n, dtype=torch.int64, device=x.device)
    for b in range(bits):
        for f in range(d):
            key |= ((q[:, f] >> b) & 1) << (b * d + f)
    return torch.argsort(key, stable=True)


def _near_lists(x, m):
    """Near earlier points of every point, ``(n, m)`` int32, ascending distance, -1 padded: what a
    fit step's local systems are given.  Exact for the first 8,192 points, else the nearest among the
    512 around the point along a Morton curve of the points before it and of its own level."""
    n = x.shape[0]
    x = x.float()
    out = torch.full((n, m), -1, dtype=torch.int32, device=x.device)

    def keep(rows, cand, dist):
        w = min(m, cand.shape[1])
        v, at = torch.topk(dist, w, dim=1, largest=False, sorted=True)
        j = torch.gather(cand, 1, at)
        out[rows, :w] = torch.where(torch.isfinite(v), j, -1).to(torch.int32)

    head = min(n, 8192)
    for r0 in range(0, head, 2048):
        rows = torch.arange(r0, min(head, r0 + 2048), device=x.device)
        cand = torch.arange(head, device=x.device).expand(rows.numel(), head)
        dist = torch.zeros((rows.numel(), head), device=x.device)
        for f in range(x.shape[1]):
            dist += (x[rows, f][:, None] - x[:head, f][None]) ** 2
        keep(rows, cand, dist.masked_fill_(cand >= rows[:, None], math.inf))
    top = n
    while top > head:
        low = max(head, top // 8)
        order = _curve(x[:top])
        pos = torch.nonzero(order >= low).flatten()
        off = torch.arange(-256, 257, device=x.device)
        for p in pos.split(32768):
            rows = order[p]
            at = p[:, None] + off
            cand = order[at.clamp(0, top - 1)]
            dist = torch.zeros(cand.shape, device=x.device)
            for f in range(x.shape[1]):
                dist += (x[rows, f][:, None] - x[cand, f]) ** 2
            bad = (cand >= rows[:, None]) | (at < 0) | (at >= top)
            keep(rows, cand, dist.masked_fill_(bad, math.inf))
        top = low
    return out


def prepare(case, seed):
    x, y, xq, ls = _inputs(case, seed)
    kind = case['kind']
    sdt = torch.float64 if case.get('search64') else torch.float32
    s = {'kind': kind, 'm': case['m'], 'ls': ls, 'pivot_tol': case.get('pivot_tol')}
    if kind == 'search':
        s['x'] = x.to(sdt)
        return s
    kernel = _kernel(case, ls)
    if kind == 'predict_call':
        s['model'] = B200Nngpr(kernel=kernel, num_nn=case['m'], optimizer=None, alpha=ALPHA).fit(
            x.cpu().numpy(), y[:, 0].cpu().numpy())
        s['xq'] = xq.cpu().numpy()
        return s
    s['p'] = extract(kernel)
    dt = torch.float64 if case['f64'] else torch.float32
    s['x'], s['y'] = x.to(dt), y.to(dt)
    if kind == 'autograd':
        s['theta'] = torch.tensor(kernel.theta, dtype=torch.float64, device='cuda', requires_grad=True)
        s['problem'] = LogLikProblem(x.float(), s['x'], s['y'], s['p'], case['m'], ALPHA, pivot_tol=case['pivot_tol'])
    elif kind == 'systems':
        s['nbr'] = _near_lists(x / torch.as_tensor(ls, device='cuda', dtype=torch.float64), case['m'])
        s['grad'] = case['grad']
    elif kind == 'predict':
        s['xs'], s['xq'] = x.float(), xq.to(dt)
    else:
        s['xs'] = x.to(sdt)
    return s


def run(s):
    kind = s['kind']
    if kind == 'search':
        return ops.knn(s['x'], s['x'], s['m'], 0, s['ls'])
    if kind == 'predict_call':
        return s['model'].predict(s['xq'], return_std=True)
    if kind == 'autograd':
        s['theta'].grad = None
        lml = NngpLogLik.apply(s['theta'], s['problem'])
        lml.backward()
        return lml.detach(), s['theta'].grad
    flags = ops.new_flags(s['x'].device)
    if kind == 'predict':
        xq = s['xq']
        nbr = ops.knn(s['xs'], xq.float(), s['m'], None, s['ls'], flags=flags)
        mean, var = ops.predict(s['x'], s['y'], xq, nbr, s['p'], ALPHA, s['pivot_tol'], flags=flags)
        return nbr, mean, var
    if kind == 'systems':
        return ops.loglik(s['x'], s['y'], s['nbr'], s['p'], ALPHA, s['grad'], s['pivot_tol'], flags=flags)
    nbr = ops.knn(s['xs'], s['xs'], s['m'], 0, s['ls'], flags=flags)
    return nbr, ops.loglik(s['x'], s['y'], nbr, s['p'], ALPHA, True, s['pivot_tol'], flags=flags)


def work(case):
    n, d, m, k = case['n'], case['d'], case['m'], case['m'] + 1
    kind = case['kind']
    w = 4 if kind in ('search', 'predict', 'predict_call', 'autograd', 'fit') and not case.get('search64') else 8
    rows = case.get('nq', n)
    lists = 4 * rows * m
    # the search: the points read, the lists written, the distances of the lists' own entries
    search = {'bytes': w * d * (n + (rows if 'nq' in case else 0)) + lists, 'flops': 3 * d * rows * m}
    # the systems: fill (3 d + 1 per entry), factor, forward solves; with gradient two backward
    # solves and the weighted fill
    v = 8 if case.get('f64', True) else 4
    ydim = case.get('ydim', 1)
    n_ls = d if case['ard'] else 1
    grad = kind in ('autograd', 'fit') or case.get('grad', False)
    flops = k ** 3 / 3 + k * (k + 1) / 2 * (3 * d + 1) + m * m * (1 + ydim)
    if grad:
        flops += 2 * m * m + k * (k + 1) / 2 * (8 + (3 * d if n_ls > 1 else 2))
    systems = {'bytes': v * n * (d + ydim) + lists + (v * rows * (d + ydim + 1) if 'nq' in case else 8 * (3 + n_ls)),
               'flops': rows * flops}
    if kind == 'search':
        return search
    if kind == 'systems':
        return systems
    return {q: search[q] + systems[q] for q in search}


# ---- 64-bit results ------------------------------------------------------------------------
def _lists64(x, m, xq=None):
    """Nearest neighbours in 64 bits: among the earlier points of ``x``, or of the queries among ``x``."""
    n = x.shape[0]
    rows = n if xq is None else xq.shape[0]
    q = x if xq is None else xq
    nx = (x * x).sum(1)
    out = torch.full((rows, m), -1, dtype=torch.int64, device=x.device)
    step = max(1, min(4096, 400_000_000 // n))
    for r0 in range(0, rows, step):
        r1 = min(rows, r0 + step)
        top = n if xq is not None else max(r1 - 1, 1)
        d2 = nx[:top] - 2 * q[r0:r1] @ x[:top].T
        if xq is None:
            at = torch.arange(r0, r1, device=x.device)
            d2.masked_fill_(torch.arange(top, device=x.device) >= at[:, None], math.inf)
        w = min(m, top)
        v, j = torch.topk(d2, w, dim=1, largest=False, sorted=True)
        out[r0:r1, :w] = torch.where(torch.isfinite(v), j, -1)
    return out


def _systems64(case, x, y, nbr, theta, ard, xq=None, grad=False):
    """Log-likelihood (and gradient) or predictive mean and variance, by a batched Cholesky in 64 bits."""
    x, y = x.double(), y.double()
    theta = theta.clone().requires_grad_(grad)
    d, m = x.shape[1], nbr.shape[1]
    total, means, variances = 0.0, [], []
    eye = torch.eye(m + 1, device=x.device, dtype=torch.float64)
    for r0 in range(0, nbr.shape[0], 16384):
        idx = nbr[r0:r0 + 16384].long()
        ok = idx >= 0
        amp, ls, noise = theta[0].exp(), theta[1:-1].exp(), theta[-1].exp()
        pt = x[r0:r0 + idx.shape[0]] if xq is None else xq[r0:r0 + idx.shape[0]].double()
        pts = torch.cat([x[idx.clamp_min(0)], pt[:, None]], 1)
        d2 = 0.0
        for f in range(d):
            c = pts[:, :, f]
            d2 = d2 + (c[:, :, None] - c[:, None]) ** 2 / ls[f if ard else 0] ** 2
        if case.get('family') == 'matern32':
            r = torch.where(d2 > 0, 3 * d2, torch.ones_like(d2)).sqrt()
            s = torch.where(d2 > 0, (1 + r) * torch.exp(-r), torch.ones_like(d2))
        else:
            s = torch.exp(-0.5 * d2)
        live = torch.cat([ok, torch.ones_like(ok[:, :1])], 1)
        both = live[:, :, None] & live[:, None]
        add = torch.full((m + 1,), ALPHA, device=x.device, dtype=torch.float64)
        if xq is not None:
            add[m] = 0.0
        K = torch.where(both, amp * s + torch.diag(add) + noise * eye, eye)
        L = torch.linalg.cholesky(K)
        yn = torch.where(ok[:, :, None], y[idx.clamp_min(0)], 0.0)
        z = torch.linalg.solve_triangular(L[:, :m, :m], yn, upper=False)
        mu = (L[:, m, :m, None] * z).sum(1)
        s2 = L[:, m, m] ** 2
        if xq is not None:
            means.append(mu.detach())
            variances.append(s2.detach())
            continue
        res = y[r0:r0 + idx.shape[0]] - mu
        ll = (-0.5 * res ** 2 / s2[:, None] - 0.5 * torch.log(s2)[:, None] - 0.5 * math.log(2 * math.pi)).sum()
        if grad:
            ll.backward()
        total += ll.detach()
    if xq is not None:
        return torch.cat(means), torch.cat(variances)
    return (total, theta.grad) if grad else (total, None)


def exact(case, seed):
    kind = case['kind']
    if kind == 'search':  # whole numbers
        return None
    x, y, xq, ls = _inputs(case, seed)
    if case['n'] * case.get('nq', case['n']) > 3e11 and kind != 'systems':
        return None
    scale = torch.as_tensor(ls, device='cuda', dtype=torch.float64)
    theta = torch.tensor(_kernel(case, ls).theta, dtype=torch.float64, device='cuda')
    if kind in ('predict', 'predict_call'):
        if kind == 'predict' and not case['f64']:
            x, y, xq = x.float().double(), y.float().double(), xq.float().double()
        nbr = _lists64(x.float().double() / scale, case['m'], xq.float().double() / scale)
        mean, var = _systems64(case, x, y, nbr, theta, case['ard'], xq)
        return (mean[:, 0], var.sqrt()) if kind == 'predict_call' else (None, mean, var)
    f64 = case['f64']
    xs = x if case.get('search64') else x.float().double()
    if not f64:
        x, y = x.float().double(), y.float().double()
    nbr = _near_lists(_inputs(case, seed)[0] / scale, case['m']) if kind == 'systems' else _lists64(xs / scale, case['m'])
    lml, grad = _systems64(case, x, y, nbr, theta, case['ard'], grad=case.get('grad', True))
    if kind == 'autograd':
        return lml, grad
    out = torch.cat([lml.reshape(1), grad]) if grad is not None else lml.reshape(1)
    return out if kind == 'systems' else (None, out)
