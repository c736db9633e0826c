"""Lennard-Jones evaluators at the ends of their ranges.
"""
import numpy as np
import pytest

from minim_gb300 import abi, runtime
from oracle.oracle import Oracle
from tests.workloads import Rng

pytestmark = pytest.mark.gpu


def _grid(n, seed=3):
    """n points of a cubic grid of spacing 1.08 with noise of 0.05."""
    k = int(np.ceil(n ** (1.0 / 3)))
    idx = np.indices((k,) * 3).reshape(3, -1).T[:n].astype(float)
    return 1.08 * idx + 0.1 * (Rng(seed).uniform(3 * n).reshape(n, 3) - 0.5)


@pytest.mark.parametrize("n", [33, 65, 80, 96, 130, 300])
def test_padding_is_out_of_reach(n):
    """A cluster with sigma = 1e5 around (1e6 (n + 1), 0, 0): no padding particle
    of a tile may stand near it.  A coordinate split into two FP32 parts is good
    to 2^-48 of 3e8, 1.1e-11 sigma, and the energy's and the force's relative
    derivatives are below 20 / sigma: 2e-9 with the sums' own error."""
    sigma = 1e5
    p = abi.lj(sigma=sigma)
    x = (sigma * (_grid(n) - 2.0) + np.array([1e6 * (n + 1), 0.0, 0.0])).ravel()
    eo, go = Oracle(p, x).energy_gradient()
    gmax = np.max(np.abs(go))
    inst = runtime.Instance(p, x)
    e, g = inst.energy_gradient(x)
    assert abs(e - eo) <= 2e-9 * abs(eo) and np.max(np.abs(g - go)) <= 2e-9 * gmax
    e, g = inst.eval_kernel(abi.EVAL_FP64S_CTA, x)
    assert abs(e - eo) <= 2e-9 * abs(eo) and np.max(np.abs(g - go)) <= 2e-7 * gmax
