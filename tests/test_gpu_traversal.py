"""The traversal's lane split and filter blocks at their edges, against the independent gather kernel.

The molecules of a 2x2x2-cell brick share the CTA's 256 lanes, 1, 2, 4 or 8 lanes each as there are at
most 256, 128, 64 or 32 of them, and more than 256 take rounds; rows of cells are filtered in blocks of 16
slots. The boxes' 4x4x4 or odd-counted grids put a brick's molecules on both sides of these limits. The
gather kernel evaluates the same pairs in another order and with the reference's operations: the forces are
sums of about a hundred FP64 terms of relative error 1e-15 each, which 1e-12 of the rms force covers.
"""
import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu


def jittered(n, density, rc, seed, species):
    comps = W.two_species() if species == 2 else [W.Component(1.0, 1.0, 1.0, True)]
    s = W.lj_fcc_box(int(np.ceil((n / 4.0) ** (1.0 / 3.0))), density, 1.0, seed, rc, comps, n_atoms=n)
    rng = np.random.default_rng(seed)
    s.r = (s.r + rng.uniform(-0.08, 0.08, s.r.shape)) % s.length
    s.r[s.r >= s.length] = 0.0
    return s


# (molecules, density, rc): molecules per brick around 1, 32, 64, 128, 256 and beyond, rows of 1 to
# more than 64 slots, grids of 2, 3, 4, 5 and more cells per dimension
BOXES = [(8, 0.01, 2.5), (40, 0.02, 2.5), (250, 0.24, 2.5), (262, 0.25, 2.5), (500, 0.5, 2.5), (520, 0.52, 2.5),
         (1020, 0.95, 2.5), (1100, 1.0, 2.5), (640, 0.8, 2.5), (1500, 0.8, 3.0), (4100, 0.8, 2.5), (2900, 1.05, 3.4),
         (9001, 0.75, 3.0)]


@pytest.mark.parametrize("n,density,rc", BOXES)
@pytest.mark.parametrize("species", [1, 2])
def test_traversal_equals_the_gather_kernel(n, density, rc, species):
    s = jittered(n, density, rc, 100 + n, species)
    out = []
    for kind, precision in ((0, M.FP64), (1, M.FP64), (0, M.MIXED)):
        lc = M.LinkedCells.from_system(s, precision)
        lc.setPairKernel(kind)
        lc.update()
        sums = lc.traversePairs()
        out.append((np.array(sums), lc.getParticles()["F"]))
        lc.close()
    ref, frms = out[1], np.sqrt(np.mean(out[1][1] ** 2))
    for got in (out[0], out[2]):
        assert got[0][2] == ref[0][2]
        assert np.max(np.abs(got[0][:2] - ref[0][:2])) <= 1e-12 * np.max(np.abs(ref[0][:2]))
        assert np.max(np.abs(got[1] - ref[1])) <= 1e-12 * max(frms, 1.0)


@pytest.mark.parametrize("system", ["vapour", "dilute", "slab"])
@pytest.mark.parametrize("species", [1, 2])
def test_sparse_bricks(system, species):
    """Boxes of several rounds of bricks, most of them with a few molecules, which go one per warp: a vapour,
    a dilute fluid with bricks on both sides of the limits (128 staged, 32 own molecules), a liquid slab."""
    if system == "slab":
        s = W.config_c3(9, 41000)
        if species == 1:
            s.components, s.mix, s.cid = [W.Component(1.0, 1.0, 1.0, True)], np.ones((0, 2)), np.zeros_like(s.cid)
    else:
        n, density = (3100, 0.01) if system == "vapour" else (40001, 0.13)
        s = jittered(n, density, 2.5, 11, species)
    out = []
    for kind in (0, 1):
        lc = M.LinkedCells.from_system(s)
        lc.setPairKernel(kind)
        lc.update()
        sums = lc.traversePairs()
        again = lc.traversePairs()
        assert sums == again
        out.append((np.array(sums), lc.getParticles()["F"]))
        lc.close()
    assert out[0][0][2] == out[1][0][2]
    assert np.max(np.abs(out[0][0] - out[1][0])) <= 1e-12 * np.max(np.abs(out[1][0]))
    assert np.max(np.abs(out[0][1] - out[1][1])) <= 1e-12 * max(np.sqrt(np.mean(out[1][1] ** 2)), 1.0)


def test_lj_cutoff_below_the_cutoff():
    """rcLJ < rc: pairs between the two count as pairs and exert no force."""
    s = jittered(1372, 0.8, 2.8, 7, 1)
    s.lj_cutoff = 2.3
    out = []
    for kind in (0, 1):
        lc = M.LinkedCells.from_system(s)
        lc.setPairKernel(kind)
        lc.update()
        sums = lc.traversePairs()
        out.append((np.array(sums), lc.getParticles()["F"]))
        lc.close()
    assert out[0][0][2] == out[1][0][2]
    assert np.max(np.abs(out[0][0] - out[1][0])) <= 1e-12 * np.max(np.abs(out[1][0]))
    assert np.max(np.abs(out[0][1] - out[1][1])) <= 1e-12 * np.sqrt(np.mean(out[1][1] ** 2))
