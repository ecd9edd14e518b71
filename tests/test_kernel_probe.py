"""The values a kernel tree would hold at another theta, read without cloning it, against the clone's."""
import numpy as np
import pytest
from sklearn.gaussian_process import kernels as K

from nngpr_b200 import kernel_params as kp

C, R, M, W = K.ConstantKernel, K.RBF, K.Matern, K.WhiteKernel
TREES = [
    C(2.0) * R(0.5) + W(0.1),
    W(0.1) + C(2.0, constant_value_bounds='fixed') * R([0.5, 1.0, 2.0]),
    R(np.array([0.7])) + C(0.3) + W(0.2, noise_level_bounds='fixed'),
    C(1.5) * (M([0.5, 1.0], nu=1.5) + W(0.1, noise_level_bounds='fixed')),
    C(1.0, 'fixed') * (C(3.0) * M(0.4, nu=np.inf)) + C(0.1),
    C(2.0) * R([1.0, 2.0], length_scale_bounds='fixed'),
    W(0.5),
    C(2.0) * C(3.0) * R(1.0),  # a product of free parameters: no map
    W(0.1) + W(0.2) + R(1.0),
]


class Doubled(R):
    """A subclass whose theta is not scikit-learn's."""

    @property
    def theta(self):
        return 2 * super().theta

    @theta.setter
    def theta(self, v):
        K.Kernel.theta.fset(self, np.asarray(v) / 2)

    def clone_with_theta(self, theta):
        return Doubled(float(np.exp(theta[0] / 2)))


@pytest.mark.parametrize('i', range(len(TREES)))
def test_probe_equals_the_clone(i):
    kernel = TREES[i]
    assert kp._plain_tree(kernel)
    theta = np.linspace(-1.3, 0.9, len(kernel.theta))
    probe = kp._Probe(theta)
    got, want = kp._values(kernel, probe), kp._values(kernel.clone_with_theta(theta))
    assert probe.used == len(kernel.theta)
    assert got.keys() == want.keys()
    for k in got:
        assert np.ndim(got[k]) == np.ndim(want[k]) and np.array_equal(got[k], want[k])


def test_other_thetas_are_probed_through_the_clone():
    assert not kp._plain_tree(C(1.0) * Doubled(1.0))
    with pytest.raises(NotImplementedError):
        kp.extract(Doubled(0.5))
    for i in (7, 8):
        with pytest.raises(NotImplementedError):
            kp.extract(TREES[i])
