"""The exponential of the FP64 local systems: at most 0.85 ulp off over [-708, 0], 0 below, NaN kept."""
import ctypes

import numpy as np
import pytest
import torch

from nngpr_b200 import _lib

pytestmark = pytest.mark.gpu


def exp_neg(x):
    t = torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).cuda()
    out = torch.empty_like(t)
    st = _lib.lib().nngp_exp_neg_probe(ctypes.c_void_p(t.data_ptr()), ctypes.c_void_p(out.data_ptr()), t.numel(),
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    _lib.check(st, 'nngp_exp_neg_probe')
    return out.cpu().numpy()


def ulps(x):
    """Error in units of the last place of the exact value (an 80-bit exponential, good to 2^-10 of them)."""
    assert np.finfo(np.longdouble).nmant >= 63
    want = np.exp(x.astype(np.longdouble))
    unit = np.spacing(want.astype(np.float64)).astype(np.longdouble)
    return np.abs(exp_neg(x).astype(np.longdouble) - want) / unit


def near(points, steps=3):
    out = [points]
    for direction in (-np.inf, np.inf):
        p = points
        for _ in range(steps):
            p = np.nextafter(p, direction)
            out.append(p)
    x = np.concatenate(out)
    return x[(x <= 0) & (x >= -708)]


@pytest.mark.parametrize('points', ['uniform', 'small', 'tiny', 'halves', 'ends'])
def test_error_stays_below_the_stated_bound(points):
    rng = np.random.default_rng(1)
    x = {'uniform': lambda: rng.uniform(-708, 0, 4_000_000),
         'small': lambda: rng.uniform(-2, 0, 4_000_000),
         'tiny': lambda: -10.0 ** rng.uniform(-320, 0, 1_000_000),
         # where the reduced argument changes sign or its multiple of ln 2 changes
         'halves': lambda: near(-np.arange(0, 2043) * (np.log(2) / 2)),
         'ends': lambda: near(np.array([0.0, -0.0, -1.0, -708.0, -707.5, -5e-324, -2.3e-308]))}[points]()
    assert ulps(x).max() <= 0.85


def test_exact_values_and_values_outside_the_range():
    below = np.array([np.nextafter(-708.0, -np.inf), -709.0, -745.2, -1e5, -1e300, -np.inf])
    assert np.array_equal(exp_neg(below), np.zeros(6))
    assert np.array_equal(exp_neg(np.array([0.0, -0.0, -5e-324])), np.ones(3))
    assert exp_neg(np.array([-708.0]))[0] > 3e-308
    assert np.isnan(exp_neg(np.array([np.nan]))).all()
