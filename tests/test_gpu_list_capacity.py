"""Skin runs of small boxes, whose cells (3 or 4 along an edge) put 2,000 to 6,000 molecules in a staged region.

The list kernels and the list build take three, two or one CTA per SM by that number. The runs follow the
per-step traversal up to summation order: forces are sums of about a hundred FP64 terms of relative error
1e-15 each and eight steps of 0.002 amplify that by less than 1e2, so 1e-11 of the rms force covers the FP64
form; the mixed form's pair forces are single precision, 1e-5 of the rms force as in its other tests.
"""
import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu

STEPS, DT = 8, 0.002


def run(system, precision, skin, prune):
    lc = M.LinkedCells.from_system(system, precision)
    lc.update()
    lc.traversePairs()
    if skin:
        lc.setSkin(skin)
        lc.setListPrune(prune)
    recs = lc.run(STEPS, DT)
    F = lc.getParticles()["F"]
    lc.close()
    return recs, F


# (molecules, cutoff, skin, prune): three CTAs per SM, two, one (evaluation), one (build as well), a grid of 27
# bricks, one of 4 cells per edge with pruned lists
@pytest.mark.parametrize("n,rc,skin,prune", [(1000, 2.5, 0.3, 0.0), (1500, 3.0, 0.4, 0.15), (3300, 2.5, 0.3, 0.15),
                                             (5000, 2.5, 0.3, 0.0), (5000, 3.0, 0.4, 0.15), (14000, 3.0, 0.4, 0.15)])
@pytest.mark.parametrize("species", [1, 2])
def test_large_regions_follow_the_traversal(n, rc, skin, prune, species):
    comps = W.two_species() if species == 2 else [W.Component(1.0, 1.0, 1.0, True)]
    s = W.lj_fcc_box(int(np.ceil((n / 4.0) ** (1.0 / 3.0))), 0.7, 1.0, n, rc, comps, n_atoms=n)
    rng = np.random.default_rng(n)
    s.r = (s.r + rng.uniform(-0.08, 0.08, s.r.shape)) % s.length
    s.r[s.r >= s.length] = 0.0
    ref, Fref = run(s, M.FP64, 0.0, 0.0)
    rms = np.sqrt(np.mean(np.sum(Fref ** 2, axis=1)))
    for precision, tol in ((M.FP64, 1e-11), (M.MIXED, 1e-5)):
        recs, F = run(s, precision, skin, prune)
        assert np.sqrt(np.mean(np.sum((F - Fref) ** 2, axis=1))) <= tol * rms
        if precision == M.FP64:
            assert np.array_equal(recs[:, 3], ref[:, 3])
