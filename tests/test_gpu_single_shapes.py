"""Which single minimisations and evaluations run on one CTA or cluster (one
launch) and which on the whole GPU (a launch every 64 iterations), by size and
precision, and that both give minima and energies on either side of each bound.
"""
import numpy as np
import pytest

from minim_gb300 import abi, runtime
from oracle.oracle import Oracle
from tests.workloads import Rng, pf_noise, pf_simplex, sheet

pytestmark = pytest.mark.gpu


def _grid(n, seed=3):
    k = int(np.ceil(n ** (1.0 / 3)))
    idx = np.indices((k,) * 3).reshape(3, -1).T[:n].astype(float)
    return (1.08 * idx + 0.1 * (Rng(seed).uniform(3 * n).reshape(n, 3) - 0.5)).ravel()


def _lj(n, cutoff=0.0):
    return abi.lj(cutoff=cutoff), _grid(n), None


def _pf1(nx, ny):
    g = (nx, ny, 1)
    return abi.phase_field(g, interface_size=1.0, surface_tension=1.0), pf_noise(g, seed=2) + 0.1, None


def _wall(nx, ny):
    s = np.zeros((nx, ny), np.uint8)
    s[0] = s[-1] = 1
    return abi.phase_field((nx, ny, 1), interface_size=1.0, surface_tension=1.0, solid=s.ravel(),
                           contact_angle=60.0), pf_noise((nx, ny, 1), seed=3) + 0.1, None


def _pf3(nx, ny):
    g = (nx, ny, 1)
    return abi.phase_field(g, nfluid=3, volume_fixed=True), pf_simplex(g, 3, seed=4), None


def _sheet(k):
    flat, tris, pert = sheet(k, seed=k)
    return abi.bar_and_hinge(triangulation=tris, rigidity=(1, 0.01)), flat, pert


SIDES = [
    # (instance, precision, one launch)
    (_lj(512), "fp64", True), (_lj(513), "fp64", False), (_lj(640), "mixed", True), (_lj(641), "mixed", False),
    (_lj(1024), "fp32", True), (_lj(1025), "fp32", False), (_lj(512, 2.5), "mixed", True),
    (_lj(513, 2.5), "mixed", False), (_lj(768, 2.5), "fp32", True), (_lj(769, 2.5), "fp32", False),
    (_pf1(96, 96), "fp64", True), (_pf1(97, 96), "fp64", False), (_pf1(128, 128), "mixed", True),
    (_pf1(128, 129), "mixed", False), (_pf1(125, 160), "fp32", True), (_pf1(127, 158), "fp32", False),
    (_wall(64, 128), "fp64", True), (_wall(65, 128), "fp64", False), (_wall(100, 120), "mixed", True),
    (_wall(101, 120), "mixed", False), (_pf3(80, 100), "fp64", True), (_pf3(81, 100), "fp64", False),
    (_sheet(14), "fp64", True), (_sheet(15), "fp64", True), (_sheet(18), "mixed", True), (_sheet(19), "mixed", True),
    (_sheet(36), "fp64", True), (_sheet(37), "fp64", False)]


@pytest.mark.parametrize("case", range(len(SIDES)))
def test_sides(case):
    (p, x0, x), precision, one = SIDES[case]
    x = x0 if x is None else x
    inst = runtime.Instance(p, x0)
    inst.coords = x
    before = runtime.launch_count()
    r = inst.minimise(abi.minimiser("lbfgs", tol=0.0, max_iter=100, precision=precision))
    assert r.iter >= 100 and (runtime.launch_count() - before == 1) == one
    # what it returns is a point of the potential with this energy (an FP32 one
    # while the run is in that stage), below the start's
    o = Oracle(p, x0)
    y = inst.coords
    e, _ = o.energy_gradient(y)
    assert abs(e - r.energy) <= (1e-9 if r.fp64_iters > 0 else 1e-5) * max(abs(e), 1e-3)
    assert e < o.energy(x)


@pytest.mark.parametrize("case", [_lj(512), _lj(513), _lj(512, 2.5), _lj(513, 2.5), _pf1(64, 64), _pf1(17, 241),
                                  _sheet(14), _sheet(15), _sheet(36), _sheet(37)], ids=range(10))
def test_evaluation_sides(case):
    """FP64 evaluations on both sides of the bounds, of the shapes and of the 4096
    degrees of freedom that live in page-locked memory; E and g of the resident
    coordinates too."""
    p, x0, x = case
    x = x0 if x is None else x
    inst, o = runtime.Instance(p, x0), Oracle(p, x0)
    eo, go = o.energy_gradient(x)
    inst.coords = x
    assert np.array_equal(inst.coords, x)
    for args in ((x,), ()):
        e, g = inst.energy_gradient(*args)
        assert abs(e - eo) <= 1e-11 * abs(eo) and np.max(np.abs(g - go)) <= 1e-10 * np.max(np.abs(go))
        assert abs(inst.energy(*args) - eo) <= 1e-11 * abs(eo)


@pytest.mark.parametrize("case", [_lj(300), _lj(300, 2.5), _pf1(40, 40), _wall(30, 31), _sheet(30)], ids=range(5))
def test_without_clusters(case, monkeypatch):
    """A device that cannot hold a cluster of eight runs small instances on the grid."""
    p, x0, x = case
    x = x0 if x is None else x
    inst, o = runtime.Instance(p, x0), Oracle(p, x0)
    monkeypatch.setenv("MINIM_GPU_CLUSTERS", "0")
    eo, go = o.energy_gradient(x)
    e, g = inst.energy_gradient(x)
    assert abs(e - eo) <= 1e-11 * abs(eo) and np.max(np.abs(g - go)) <= 1e-10 * np.max(np.abs(go))
    inst.coords = x
    before = runtime.launch_count()
    r = inst.minimise(abi.minimiser("lbfgs", tol=0.0, max_iter=100, precision="fp64"))
    assert r.iter >= 100 and runtime.launch_count() - before > 1
    assert abs(o.energy(inst.coords) - r.energy) <= 1e-9 * max(abs(r.energy), 1e-3)


def test_page_locked_coordinates():
    """Coordinates of many small instances share chunks of page-locked memory that
    are used again and given back: everyone's own stay as they were, also past
    the pool's 256 MB, where they live on the device."""
    p = abi.lj(ndim=2)
    rng = np.random.default_rng(5)
    base = np.stack(np.meshgrid(np.arange(64), np.arange(32), indexing="ij"), -1).reshape(-1, 2) * 1.1
    held = {}

    def make(k, n):
        x = (base[:n] + rng.uniform(-0.05, 0.05, (n, 2))).ravel()
        held[k] = (runtime.Instance(p, x), x)

    for k in range(300):
        make(k, int(rng.integers(1, 2049)))
    for k in list(held)[::2]:
        held.pop(k)[0].close()
    for k in range(300, 600):
        make(k, int(rng.integers(1, 2049)))
    for inst, x in held.values():
        assert np.array_equal(inst.coords, x)
    for k in list(held)[:-1]:
        held.pop(k)[0].close()
    (inst, x), = held.values()
    e0, g0 = inst.energy_gradient()
    many = [runtime.Instance(p, base.ravel() + 1e-3 * k) for k in range(8300)]
    for k, h in enumerate(many):
        assert np.array_equal(h.coords, base.ravel() + 1e-3 * k)
    r = [h.minimise(abi.minimiser("lbfgs", tol=0.0, max_iter=3, precision="fp64")) for h in (many[0], many[-1])]
    assert abs(r[0].energy - r[1].energy) <= 1e-9 * abs(r[0].energy)
    e, g = inst.energy_gradient()
    assert e == e0 and np.array_equal(g, g0)
    for h in many:
        h.close()
