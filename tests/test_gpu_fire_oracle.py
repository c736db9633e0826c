"""FIRE without a line search (dt_max given) against the oracle's, which is the
reference's step by step: the same iterates after 1, 2, 7, 21 and 61 iterations,
over which the time step is halved and grows again, and the same minimum.  One
CTA by rows (up to 64 particles), by single and by double tiles, a cluster, the
whole GPU.

An iterate's error: gradient, velocity and step are FP32 numbers, three
roundings of 2^-24 of each step's length, and a trajectory of k + 1 steps near
a minimum covers at most some ten times its largest displacement d: 2e-6 d, and
the FP32 stage's forces add 1e-6 of theirs: 1e-5 d allows for both.  FP32
coordinates add their own rounding, 2^-24 of the largest each step.  A wrong
mixing factor, time step or reset shows at 0.01 d and more.
"""
import numpy as np
import pytest

from minim_gb300 import abi, runtime
from oracle.oracle import Oracle
from tests.workloads import Rng

pytestmark = pytest.mark.gpu


def _cluster(n, seed):
    """n points of a cubic grid of spacing 1.08 with noise of 0.05: FIRE's first steps from it are far from chaotic."""
    k = int(np.ceil(n ** (1.0 / 3)))
    idx = np.indices((k,) * 3).reshape(3, -1).T[:n].astype(float)
    return (1.08 * idx + 0.1 * (Rng(seed).uniform(3 * n).reshape(n, 3) - 0.5)).ravel()


def _close(x, xo, x0, k, precision):
    d = np.max(np.abs(xo - x0))
    tol = 1e-5 * d
    if precision == "fp32":
        tol += (k + 2) * 2.0 ** -24 * np.max(np.abs(xo))
    assert np.max(np.abs(x - xo)) <= tol, (np.max(np.abs(x - xo)), tol)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("k", [0, 1, 6, 20, 60])
def test_iterates_batch(k, precision):
    ns = [13, 40, 64, 65, 130, 256, 257, 300, 400]
    mp = abi.minimiser("fire", dt_max=0.02, tol=0.0, max_iter=k, precision=precision)
    x0 = [_cluster(n, n) for n in ns]
    insts = [runtime.Instance(abi.lj(), x) for x in x0]
    b = runtime.Batch()
    for h in insts:
        b.add(h, mp)
    b.run(256 if k % 2 else 128)
    for h, x in zip(insts, x0):
        o = Oracle(abi.lj(), x)
        o.minimise(mp)
        _close(h.coords, o.coords, x, k, precision)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [13, 96, 97, 300, 1100])
def test_iterates_single(n, precision):
    x0 = _cluster(n, n)
    inst, o = runtime.Instance(abi.lj(), x0), Oracle(abi.lj(), x0)
    for k in (0, 1, 6, 20, 60):
        if n > 1000 and k == 60:
            continue  # the oracle's time
        mp = abi.minimiser("fire", dt_max=0.02, tol=0.0, max_iter=k, precision=precision)
        inst.coords = x0
        o.coords = x0
        inst.minimise(mp)
        o.minimise(mp)
        _close(inst.coords, o.coords, x0, k, precision)


@pytest.mark.parametrize("n", [13, 64, 130, 300])
def test_minimum_across_precisions(n):
    """The mixed run crosses from the FP32 to the FP64 stage and ends in the oracle's minimum."""
    x0 = _cluster(n, n + 1)
    p = abi.lj()
    mp = abi.minimiser("fire", dt_max=0.02, tol=1e-6, max_iter=20000)
    one, many = runtime.Instance(p, x0), runtime.Instance(p, x0)
    b = runtime.Batch()
    b.add(many, mp)
    rs = [one.minimise(mp), b.run()[0]]
    o = Oracle(p, x0)
    ro = o.minimise(mp)
    assert ro.status == abi.RES_CONVERGED
    for r, h in zip(rs, (one, many)):
        assert r.status == abi.RES_CONVERGED and r.fp64_iters > 0 and r.fp64_iters < r.iter
        e, g = o.energy_gradient(h.coords)
        assert np.sqrt(np.mean(g ** 2)) < 1e-6
        assert abs(e - ro.energy) <= 1e-10 * abs(e) and abs(r.energy - e) <= 1e-10 * abs(e)
