"""Bricks whose staged region exceeds the shared-memory capacity: evaluated in halves, quarters or own cells, and
only beyond those gathered from global memory.

With two CTAs per SM 2,496 molecules fit (1,344 with three). A region is 64 cells, its halves 48, quarters 36, own
cells 27. The gather kernel evaluates the same pairs with the reference's operations in another order: sums of
some hundred FP64 terms of relative error 1e-15 each, which 1e-12 of the rms force covers.
"""
import time

import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu


def box(n, density, rc, species=1, seed=3):
    comps = W.two_species() if species == 2 else [W.Component(1.0, 1.0, 1.0, True)]
    s = W.lj_fcc_box(int(np.ceil((n / 4.0) ** (1.0 / 3.0))), density, 1.0, seed, rc, comps, n_atoms=n)
    s.r = (s.r + np.random.default_rng(seed).uniform(-0.05, 0.05, s.r.shape)) % s.length
    s.r[s.r >= s.length] = 0.0
    return s


def traversals(s, precision, r=None):
    out = []
    for kind in (0, 1):
        lc = M.LinkedCells.from_system(s, precision)
        lc.setPairKernel(kind)
        if r is not None:
            lc.setState(r, s.v)
        lc.update()
        sums = lc.traversePairs()
        assert lc.traversePairs() == sums
        out.append((np.array(sums), lc.getParticles()["F"]))
        lc.close()
    return out


def check(got, ref, rtol):
    frms = max(np.sqrt(np.mean(ref[1] ** 2)), 1.0)
    assert got[0][2] == ref[0][2]
    assert np.max(np.abs(got[0][:2] - ref[0][:2])) <= rtol * np.max(np.abs(ref[0][:2]))
    assert np.max(np.abs(got[1] - ref[1])) <= rtol * frms


# (molecules, density, rc): whole region, halves, quarters, own cells, beyond; grids of 3, 2, 5 (odd) and 4 cells
@pytest.mark.parametrize("n,density,rc", [(1030, 0.8, 3.0), (1200, 0.8, 3.0), (1600, 0.95, 3.0), (2300, 0.95, 4.4),
                                          (2700, 0.95, 4.4), (700, 0.95, 4.4), (8000, 0.85, 3.7), (3000, 0.9, 3.5)])
@pytest.mark.parametrize("species", [1, 2])
def test_parts_equal_the_gather_kernel(n, density, rc, species):
    got, ref = traversals(box(n, density, rc, species), M.FP64)
    check(got, ref, 1e-12)


@pytest.mark.parametrize("species", [1, 2])
def test_a_droplet_set_after_loading(species):
    """The staged capacity was chosen for the fluid that was loaded; bricks of the droplet exceed it."""
    s = box(30000, 0.1, 3.0, species)
    d = box(30000, 0.85, 3.0, species)
    r = np.ascontiguousarray(s.length / 2 + (d.r - d.length / 2) * 0.999)
    got, ref = traversals(s, M.FP64, r)
    check(got, ref, 1e-12)


@pytest.mark.parametrize("n,density,rc", [(1200, 0.8, 3.0), (1600, 0.95, 3.0), (700, 0.95, 4.4)])
def test_the_ensemble_evaluates_the_same_parts(n, density, rc):
    systems = [box(n, density, rc, seed=k) for k in range(3)]
    b = M.Batch.from_systems(systems, M.FP64)
    b.prepare()
    recs = b.run(2, 0.002)
    F = b.getParticles()["F"]
    b.close()
    for k, s in enumerate(systems):
        lc = M.LinkedCells.from_system(s, M.FP64)
        lc.update()
        lc.traversePairs()
        one = lc.run(2, 0.002)
        np.testing.assert_array_equal(one[:, 3], recs[:, k, 3])
        np.testing.assert_array_equal(lc.getParticles()["F"], F[k * n:(k + 1) * n])
        lc.close()


def test_no_cliff_at_the_capacity():
    """From a cutoff of 3.2 (staged whole) to 3.7 (in parts) the pairs grow 1.55-fold. A step of 200,000 molecules may
    take four times as long; where the regions above the capacity gathered, it took 6.4 times as long."""
    best = {}
    for rc in (3.2, 3.7):
        lc = M.LinkedCells.from_system(box(200000, 0.85, rc), M.MIXED)
        lc.update()
        lc.traversePairs()
        times = []
        for _ in range(4):
            t = time.perf_counter()
            lc.run(20, 0.001)
            times.append(time.perf_counter() - t)
        best[rc] = min(times)
        lc.close()
    assert best[3.7] <= 4.0 * best[3.2]
