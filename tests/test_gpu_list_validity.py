"""Lists are built again when what they were built for changes: their padding is the sentinel slot of the staged
capacity, which belongs to the precision form and to the CTAs per SM."""
import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu

DT = 0.002


def box(n, rc, seed, species=1):
    comps = W.two_species() if species == 2 else [W.Component(1.0, 1.0, 1.0, True)]
    s = W.lj_fcc_box(int(np.ceil((n / 4.0) ** (1.0 / 3.0))), 0.7, 1.0, seed, rc, comps, n_atoms=n)
    s.r = (s.r + np.random.default_rng(seed).uniform(-0.05, 0.05, s.r.shape)) % s.length
    s.r[s.r >= s.length] = 0.0
    return s


def rms(a):
    return np.sqrt(np.mean(np.sum(a ** 2, axis=1)))


# regions for three CTAs per SM in both forms, and for another number in one of them
@pytest.mark.parametrize("n,rc", [(1000, 2.5), (3300, 2.5), (5000, 2.5), (9000, 3.0)])
@pytest.mark.parametrize("prune", [0.0, 0.15])
@pytest.mark.parametrize("species", [1, 2])
def test_another_precision_builds_again(n, rc, prune, species):
    """The forces of a step after the change against the traversal of the same state; mixed forces are single
    precision pair by pair, 1e-5 of the rms force as in the other tests."""
    s = box(n, rc, n, species)
    lc = M.LinkedCells.from_system(s, M.FP64)
    lc.update()
    lc.traversePairs()
    lc.setSkin(0.3)
    lc.setListPrune(prune)
    for precision, tol in ((M.FP64, 1e-11), (M.MIXED, 1e-5), (M.FP64, 1e-11), (M.MIXED, 1e-5)):
        builds = lc.skinBuilds()
        lc.setPrecision(precision)
        lc.run(1, DT)
        assert lc.skinBuilds() == builds + 1
        st = lc.getParticles()
        ref = M.LinkedCells.from_system(s, M.FP64)
        ref.setState(st["r"], st["v"])
        ref.update()
        ref.traversePairs()
        F = ref.getParticles()["F"]
        ref.close()
        assert rms(st["F"] - F) <= tol * rms(F)
    lc.close()


@pytest.mark.parametrize("precision,tol", [(M.FP64, 1e-11), (M.MIXED, 1e-5)])
def test_other_tiles_build_again(precision, tol):
    systems = [box(n, 2.5, n) for n in (600, 1500, 3000)]
    b = M.Batch.from_systems(systems, precision)
    b.setSkin(0.3)
    b.prepare()
    for ctas in (1, 2, 1):
        b.setTiles(64, ctas, 1)
        b.run(1, DT)
        st = b.getParticles()
        at = 0
        for s in systems:
            ref = M.LinkedCells.from_system(s, M.FP64)
            k = slice(at, at + s.n)
            at += s.n
            ref.setState(np.ascontiguousarray(st["r"][k]), np.ascontiguousarray(st["v"][k]))
            ref.update()
            ref.traversePairs()
            F = ref.getParticles()["F"]
            ref.close()
            assert rms(st["F"][k] - F) <= tol * rms(F)
    b.close()


def test_a_wait_that_ran_out_builds_again():
    """The step that gave up may have sorted boxes without building their lists."""
    systems = [box(n, 2.5, n) for n in (600, 1500, 3000)]
    b = M.Batch.from_systems(systems, M.FP64)
    b.setSkin(0.3)
    b.prepare()
    builds = b.skinBuilds()
    b.setBarrierTimeout(0)
    with pytest.raises(M.MdgpuError) as ei:
        b.run(1, DT)
    assert ei.value.code == 9
    b.setBarrierTimeout(2_000_000_000)
    b.prepare()
    assert b.skinBuilds() == builds + len(systems)
    b.close()


@pytest.mark.parametrize("precision,tol", [(M.FP64, 1e-11), (M.MIXED, 1e-5)])
def test_positions_set_behind_pruned_lists(precision, tol):
    """Displacements below half the skin keep the lists, but not the inner lists within the cutoff + 0.15: two molecules
    may be 0.34 closer."""
    s = box(4000, 2.5, 8)
    lc = M.LinkedCells.from_system(s, precision)
    lc.update()
    lc.traversePairs()
    lc.setSkin(0.4)
    lc.setListPrune(0.15)
    rng = np.random.default_rng(9)
    lc.run(3, DT)
    for k in range(3):
        st = lc.getParticles()
        builds = lc.skinBuilds()
        r = st["r"] + rng.uniform(-0.1, 0.1, st["r"].shape) * (1.0 if k == 0 else 0.2)
        r = np.where((r >= 0.0) & (r < s.length), r, st["r"])
        lc.setState(r=r)
        lc.run(1, DT)
        st = lc.getParticles()
        ref = M.LinkedCells.from_system(s, M.FP64)
        ref.setState(st["r"], st["v"])
        ref.update()
        ref.traversePairs()
        F = ref.getParticles()["F"]
        ref.close()
        assert rms(st["F"] - F) <= tol * rms(F), (k, lc.skinBuilds() - builds)
    lc.close()
