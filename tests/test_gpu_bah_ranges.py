"""BarAndHinge at the ends of its ranges: FP32 forces of very unequal elements
at one vertex, hinge angles on both sides of their rule.
"""
import numpy as np
import pytest

from minim_gb300 import abi, runtime

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
