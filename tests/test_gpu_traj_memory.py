"""The device memory of the trajectory adjoint: what a pass keeps, and a pass that gets none."""
import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu

DT = 0.002


def cluster(length, n=1000, species=2):
    """n molecules of a liquid in the middle of a box of the given edge."""
    s = W.lj_fcc_box(7, 0.7, 1.0, 5, 2.5, W.two_species() if species == 2 else [W.Component(1.0, 1.0, 1.0, True)], n_atoms=n)
    rng = np.random.default_rng(6)
    r = s.r + rng.uniform(-0.05, 0.05, s.r.shape) - s.length / 2
    lc = M.LinkedCells([length] * 3, 2.5, s.components, s.mix)
    lc.addParticles(s.ids, s.cid, np.ascontiguousarray(r + length / 2), s.v)
    return lc


def gradient(lc, steps, every):
    n = lc.n
    lc.trajForward(steps, every, DT)
    return lc.trajBackward(np.random.default_rng(7).standard_normal((n, 3)), 1.0)


def starve(lc):
    """A segment of tens of terabytes."""
    with pytest.raises(M.MdgpuError) as ei:
        lc.trajForward(2_000_000_000, 2_000_000_000, DT)
    assert ei.value.code == 2


def test_a_pass_without_memory_leaves_nothing_to_go_backward_on():
    lc = cluster(20.0)
    lc.trajForward(6, 3, DT)
    starve(lc)
    with pytest.raises(M.MdgpuError) as ei:
        lc.trajBackward(np.zeros((lc.n, 3)), 1.0)
    assert ei.value.code == 3
    lc.close()


def test_a_failed_call_is_reported_once():
    """The same pass afterwards, and another container, do not see the error of the call that failed."""
    lc = cluster(20.0)
    want = gradient(lc, 6, 3)
    lc.close()
    lc = cluster(20.0)
    starve(lc)
    for got in (gradient(lc, 6, 3), gradient(cluster(20.0), 6, 3)):
        for a, b in zip(got[:4], want[:4]):
            np.testing.assert_array_equal(a, b)
    lc.close()


@pytest.mark.parametrize("species", [1, 2])
def test_a_dilute_box_keeps_positions_only(species):
    """1,000 molecules in 64,000 cells: 200 steps of a segment take no more than their positions (24 bytes per molecule
    and step; 16 MB for the rest and the allocator's steps), not the cell starts of every step (51 MB more)."""
    import torch

    lc = cluster(100.0, species=species)
    lc.update()
    lc.traversePairs()
    lc.trajForward(1, 1, DT)
    free = torch.cuda.mem_get_info()[0]
    lc.trajForward(200, 200, DT)
    assert free - torch.cuda.mem_get_info()[0] <= 200 * 24 * lc.n + (16 << 20)
    lc.close()


@pytest.mark.parametrize("species", [1, 2])
@pytest.mark.parametrize("every", [2, 7])
def test_both_forms_give_the_same_gradient(species, every):
    """The molecules alone in the middle of a small box, which keeps binned states, and of a large one, which bins again:
    the same pairs with coordinates 40 larger, whose rounding (1e-14) the seven steps amplify by less than 1e2."""
    out = []
    for length in (20.0, 100.0):
        lc = cluster(length, species=species)
        assert (np.prod(lc.geometry()["box_cells"]) <= 2 * lc.n) == (length == 20.0)
        out.append(gradient(lc, 7, every))
        lc.close()
    for a, b in zip(out[0][:4], out[1][:4]):
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(a))
