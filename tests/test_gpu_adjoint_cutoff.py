"""The adjoint's pairs are the traversal's, also within a rounding of the cutoff.

Pairs across a periodic face, placed a few last places around the cutoff where x_i - (x_j - L) and (x_i + L) - x_j fall
on different sides of it. The unshifted potential's force does not vanish there, so a molecule has a gradient
exactly when it has a force.
"""
import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu

RC, L = 2.5, np.array([10.7, 43.0, 43.0])


def pairs(count):
    """x_i near the lower face, x_j near the upper one, the two forms on different sides of the cutoff."""
    rng = np.random.default_rng(2)
    out = []
    while len(out) < count:
        xi = rng.uniform(0.2, 2.3)
        xj = xi - RC + L[0]
        for k in range(-3, 4):
            x = xj + k * np.spacing(xj)
            image, shifted = xi - (x - L[0]), (xi + L[0]) - x
            if (image * image < RC * RC) != (shifted * shifted < RC * RC):
                out.append((xi, x))
                break
    return np.array(out[:count])


@pytest.mark.parametrize("precision", [M.FP64, M.MIXED])
def test_a_gradient_where_there_is_a_force(precision):
    x = pairs(49)
    y, z = np.meshgrid(3.0 + 5.5 * np.arange(7), 3.0 + 5.5 * np.arange(7))
    r = np.empty((98, 3))
    r[0::2] = np.stack([x[:, 0], y.ravel(), z.ravel()], axis=1)
    r[1::2] = np.stack([x[:, 1], y.ravel(), z.ravel()], axis=1)
    lc = M.LinkedCells(L, RC, [W.Component(1.0, 1.0, 1.0, False)], precision=precision)
    lc.addParticles(np.arange(1, 99, dtype=np.uint64), np.zeros(98, dtype=np.int32), r, np.zeros((98, 3)))
    lc.update()
    lc.traversePairs()
    F = lc.getParticles()["F"]
    gF = np.zeros((98, 3))
    gF[0::2, 0], gF[1::2, 0] = 1.0, -1.0
    g = lc.adjoint(gF, 0.0)[0]
    force, grad = np.any(F != 0.0, axis=1), np.any(g != 0.0, axis=1)
    assert 0 < np.count_nonzero(force) < 98
    np.testing.assert_array_equal(grad, force)
    lc.close()
