"""BarAndHinge at the ends of its ranges: FP32 forces of very unequal elements
at one vertex.
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
