"""The cell scan of large dilute boxes: up to 6,000 blocks of 1,024 cells add up the totals before them, beyond that the
totals are scanned first."""
import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu


def container(m, n=5000):
    """n molecules spread over m^3 cells; half of them in the last layer."""
    L = 2.5 * m + 0.1
    rng = np.random.default_rng(m)
    r = rng.uniform(0.0, L, (n, 3))
    r[::2, 2] = L - rng.uniform(0.1, 2.0, r[::2, 2].shape)
    lc = M.LinkedCells([L] * 3, 2.5, [W.Component(1.0, 1.0, 1.0, True)])
    lc.addParticles(rng.permutation(np.arange(1, n + 1)).astype(np.uint64), np.zeros(n, dtype=np.int32), r, np.zeros((n, 3)))
    return lc, r


# blocks below, at and above the limit, and above one round of the totals' scan's 4,096
@pytest.mark.parametrize("m", [64, 181, 182, 183, 250])
def test_cells_and_forces(m):
    lc, r = container(m)
    lc.update()
    geo = lc.geometry()
    c = np.floor((r - geo["halo_min"]) / geo["cell_length"]).astype(np.int64)
    cx, cy = geo["box_cells"][0] + 2, geo["box_cells"][1] + 2
    np.testing.assert_array_equal(lc.getCellIndexOfMolecule(), (c[:, 2] * cy + c[:, 1]) * cx + c[:, 0])
    np.testing.assert_array_equal(lc.getParticles()["r"], r)
    sums, F = lc.traversePairs(), lc.getParticles()["F"]
    lc.setPairKernel(1)
    lc.update()
    ref, Fref = lc.traversePairs(), lc.getParticles()["F"]
    assert sums[2] == ref[2]
    assert np.max(np.abs(F - Fref)) <= 1e-12 * max(np.sqrt(np.mean(Fref ** 2)), np.max(np.abs(Fref)))
    lc.close()


def test_the_work_grows_with_the_cells():
    """From 8 to 100 million cells, 12.5 times as many, the binning may take 15 times as long (without the scan of the
    totals 21)."""
    best = {}
    for m in (200, 464):
        lc, _ = container(m)
        lc.profileEnable(True)
        times = []
        for _ in range(6):
            lc.profileRead(True)
            lc.update()
            lc.synchronize()
            times.append(lc.profileRead(True)[0][0])
        best[m] = min(times)
        lc.close()
    assert best[464] <= 15.0 * best[200]
