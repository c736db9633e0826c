"""BarAndHinge at the ends of its ranges: FP32 forces of very unequal elements
at one vertex, hinge angles on both sides of their rule, a vertex of thousands
of elements, the memory instances and
requests hold, a free vertex that is nowhere.
"""
import time

import numpy as np
import pytest
import torch

from minim_gb300 import abi, runtime
from tests.workloads import Rng, sheet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", [abi.EVAL_FP32_GRID, abi.EVAL_FP32_CTA])
@pytest.mark.parametrize("big", [0, 1, 2])
def test_unequal_forces_at_a_vertex(path, big):
    """Three triangles with sides 3, 4 and 5 times a power of two around one
    vertex, two of them mirror images 2^25 times the third, at rest at half their
    size: a bar's length, strain and force, its own vector, are exact in FP32.
    The large forces cancel, and what is left is the small triangle's."""
    scale = [1.0, 1.0, 1.0]
    scale[(big + 1) % 3], scale[(big + 2) % 3] = 2.0 ** 25, -2.0 ** 25
    pts = [[0.0, 0.0, 0.0]]
    tris = []
    for k, s in enumerate(scale):
        pts += [[3 * s, 0, 0], [3 * s, 4 * s, 0]]
        tris.append([0, 1 + 2 * k, 2 + 2 * k])
    x = np.array(pts).ravel()
    p = abi.bar_and_hinge(triangulation=np.array(tris, np.int32), rigidity=(1, 1))
    _, g = runtime.Instance(p, 0.5 * x).eval_kernel(path, x)
    assert list(g[:3]) == [-6.0, -4.0, 0.0]


@pytest.mark.parametrize("path", [abi.EVAL_FP64S_GRID, abi.EVAL_FP64S_CTA])
@pytest.mark.parametrize("d0", [0.0, 0.002, -0.0312, 0.0313, -0.5, 1.5])
def test_hinge_angle_on_both_sides_of_its_rule(d0, path):
    """One hinge folded by phi either way, with a rest angle d0 from flat: energies
    k (d0 -+ phi)^2 / 2.  Double-float arithmetic and the coordinates' rounding
    are some 2^-44 of the angles: 1e-12 of the larger one squared."""
    for phi in (1e-5, 0.0003, 0.0155, 0.0157, 0.1, 1.0):
        es = []
        for s in (1, -1):
            x = np.array([0.5, 1, 0, 0, 0, 0, 1, 0, 0, 0.5, -np.cos(phi), s * np.sin(phi)])
            p = abi.bar_and_hinge(bonds=np.array([[0, 1]]), hinges=np.array([[0, 1, 2, 3]]),
                                  rigidity=(np.array([1e-30]), np.array([1.0])), length0=np.array([1.0]),
                                  theta0=np.array([np.pi - d0]))
            e, _ = runtime.Instance(p, x).eval_kernel(path, x)
            es.append(e)
        want = [0.5 * (d0 - phi) ** 2, 0.5 * (d0 + phi) ** 2]
        tol = 1e-12 * max(phi, abs(d0)) ** 2
        assert np.max(np.abs(np.sort(es) - np.sort(want))) <= tol, (phi, es, want)


def _fan(n):
    a = np.arange(n) * 2 * np.pi / n
    pts = np.concatenate([[[0, 0, 0.2]], np.stack([np.cos(a) * 3, np.sin(a) * 3, 0.1 * np.cos(5 * a)], 1)])
    return pts.ravel(), np.array([[0, 1 + i, 1 + (i + 1) % n] for i in range(n)], np.int32)


def _exact(bars, bpar, hinges, hpar, x):
    """Energy and forces in 64 bits, the hinge's angle from pi by an arctangent
    (the reference's arccosine is good to 1e-8 only where triangles are nearly
    coplanar, as in a wide fan); its bar force carries a factor of two."""
    X = torch.from_numpy(x.reshape(-1, 3).copy()).requires_grad_(True)
    b, h = torch.from_numpy(bars.astype(np.int64)), torch.from_numpy(hinges.astype(np.int64))
    bp, hp = torch.from_numpy(bpar), torch.from_numpy(hpar)
    dl = (X[b[:, 0]] - X[b[:, 1]]).norm(dim=1) - bp[:, 1]
    q = [X[h[:, k]] for k in range(4)]
    b1, b2, b3 = q[1] - q[0], q[2] - q[1], q[3] - q[2]
    n1, n2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
    th = torch.atan2(-b2.norm(dim=1) * (n1 * b3).sum(1), -(n1 * n2).sum(1)) - (hp[:, 1] - np.pi)
    es, eb = 0.5 * (bp[:, 0] * dl * dl).sum(), 0.5 * (hp[:, 0] * th * th).sum()
    g, = torch.autograd.grad(2 * es + eb, X)
    return (es + eb).item(), g.numpy().ravel()


@pytest.mark.parametrize("n", [40, 90, 300, 3000])
def test_hub(n):
    """A vertex in n triangles has 2 n elements: its list is put in order without
    a quadratic pass (one thread would take a second at 3000), and the forces
    are 64-bit arithmetic's to 1e-12, times the triangles' aspect where they are thin."""
    x, tris = _fan(n)
    y = x + 0.05 * min(1.0, 40 / n) * (Rng(1).uniform(x.size) - 0.5)
    b, bp, h, hp = runtime.bah_elements(abi.bar_and_hinge(triangulation=tris, rigidity=(1, 0.1)), x)
    p = abi.bar_and_hinge(bonds=b, hinges=h, rigidity=(1, 0.1))
    runtime.Instance(p, x)
    t = time.perf_counter()
    inst = runtime.Instance(p, x)
    assert time.perf_counter() - t < 0.2
    eo, go = _exact(b, bp, h, hp, y)
    e, g = inst.energy_gradient(y)
    tol = 1e-12 * max(1.0, n / 40)
    assert abs(e - eo) <= tol * abs(eo) and np.max(np.abs(g - go)) <= tol * np.max(np.abs(go))


def test_set_fixed_gives_memory_back():
    """Fixing other coordinates builds the element lists anew; the old ones go."""
    flat, tris, _ = sheet(200, seed=3)
    inst = runtime.Instance(abi.bar_and_hinge(triangulation=tris, rigidity=(1, 0.01)), flat)
    inst.set_fixed([0, 1, 2])
    inst.energy()
    free = torch.cuda.mem_get_info()[0]
    for k in range(60):
        inst.set_fixed(list(range(3 * k, 3 * k + 9)))
    # a sheet of 40,000 vertices holds some 30 MB
    assert free - torch.cuda.mem_get_info()[0] < 256 << 20


@pytest.mark.parametrize("explicit", [False, True])
def test_server_budget_counts_the_elements(explicit):
    """The server's memory budget is for what a request keeps on the device: a
    sheet's element lists and force slots (over 600 bytes a vertex) are more
    than its minimiser's vectors."""
    flat, tris, pert = sheet(64, seed=5)
    p = abi.bar_and_hinge(triangulation=tris, rigidity=(1, 0.01))
    if explicit:
        b, _, h, _ = runtime.bah_elements(p, flat)
        p = abi.bar_and_hinge(bonds=b, hinges=h, rigidity=(1, 0.01))
    mp = abi.minimiser("lbfgs", m=5, tol=1e-6, max_iter=3)
    vectors = 3 * 64 * 64 * 4 * (2 * 1 + 2 * 2 + 2 + 2 * 6)
    for spare, status in ((500, abi.RES_REJECTED), (4000, abi.RES_MAXITER)):
        srv = runtime.Server(max_bytes=vectors + 20000 + spare * 64 * 64)
        srv.submit(p, pert if explicit else flat, mp)
        while srv.step() != (0, 0):
            pass
        (_, r), = srv.poll()
        assert (r.status == abi.RES_REJECTED) == (status == abi.RES_REJECTED)
        srv.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_free_vertex_at_no_height(bad):
    """A vertex in no triangle still carries the external force's element: without
    a force its energy is 0 z, no number where z is none."""
    flat, tris, pert = sheet(6, seed=2)
    x0 = np.concatenate([flat, [9.0, 9.0, 0.5]])
    x = np.concatenate([pert, [9.0, 9.0, 0.5]])
    inst = runtime.Instance(abi.bar_and_hinge(triangulation=tris, rigidity=(1, 0.01)), x0)
    assert np.isfinite(inst.energy(x))
    x[-1] = bad
    assert np.isnan(inst.energy(x))
    e, g = inst.energy_gradient(x)
    assert np.isnan(e) and np.all(np.isfinite(g))
    for path in (abi.EVAL_FP32_GRID, abi.EVAL_FP32_CTA, abi.EVAL_FP64S_GRID, abi.EVAL_FP64S_CTA):
        assert np.isnan(inst.eval_kernel(path, x)[0]), path
