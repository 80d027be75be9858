"""Calls that get no device memory: an error, and afterwards a container that says so instead of running without its
arrays, and that works once there is memory again."""
import numpy as np
import pytest
import torch

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu

DT = 0.002


def box(n, seed=3):
    return W.lj_fcc_box(int(np.ceil((n / 4.0) ** (1.0 / 3.0))), 0.7, 1.0, seed, 2.5, [W.Component(1.0, 1.0, 1.0, True)],
                        n_atoms=n)


class Full:
    """Leaves `left` bytes of device memory."""

    def __init__(self, left):
        torch.cuda.synchronize()
        self.hold = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        del self.hold
        torch.cuda.empty_cache()


def test_a_container_that_could_not_grow_holds_no_molecules():
    small, large = box(1000), box(2_000_000)     # 420 MB of particle arrays
    lc = M.LinkedCells(large.length, 2.5, large.components)
    r = small.r + 1.0
    lc.addParticles(small.ids, small.cid, r, small.v)
    with Full(256 << 20):
        with pytest.raises(M.MdgpuError) as ei:
            lc.addParticles(large.ids, large.cid, large.r, large.v)
        assert ei.value.code == 2
    for call in (lc.update, lambda: lc.run(1, DT), lc.traversePairs):
        with pytest.raises(M.MdgpuError) as ei:
            call()
        assert ei.value.code == 3
    lc.addParticles(large.ids, large.cid, large.r, large.v)
    lc.update()
    np.testing.assert_array_equal(lc.getParticles()["r"], large.r)
    lc.close()


def test_a_container_whose_copies_got_no_memory_holds_no_molecules():
    """The arrays fit (190 MB), the staging buffer (88 MB) does not: they hold nothing yet."""
    s = box(1_000_000)
    lc = M.LinkedCells(s.length, 2.5, s.components)
    with Full(240 << 20):
        with pytest.raises(M.MdgpuError) as ei:
            lc.addParticles(s.ids, s.cid, s.r, s.v)
        assert ei.value.code == 2
    for call in (lc.update, lambda: lc.run(1, DT), lc.traversePairs):
        with pytest.raises(M.MdgpuError) as ei:
            call()
        assert ei.value.code == 3
    lc.addParticles(s.ids, s.cid, s.r, s.v)
    lc.update()
    np.testing.assert_array_equal(lc.getParticles()["r"], s.r)
    lc.close()


def test_a_rigid_container_without_orientations_holds_no_molecules():
    s = W.rigid_fcc_box(16, 0.3, 2.0, 11, 3.0, [W.two_centre()])
    big = W.rigid_fcc_box(64, 0.3, 2.0, 11, 3.0, [W.two_centre()])      # 1,048,576 molecules: 230 and 500 MB
    lc = M.RigidLinkedCells(big.length, 3.0, big.components)
    lc.addParticles(s.ids, s.cid, s.r, s.v, s.q, s.D)
    with Full(480 << 20):
        with pytest.raises(M.MdgpuError) as ei:
            lc.addParticles(big.ids, big.cid, big.r, big.v, big.q, big.D)
        assert ei.value.code == 2
    with pytest.raises(M.MdgpuError) as ei:
        lc.run(1, DT)
    assert ei.value.code == 3
    lc.close()


def test_an_ensemble_without_lists_keeps_no_skin():
    systems = [box(16000, seed=k) for k in range(40)]     # lists of some 250 entries: 330 MB
    b = M.Batch.from_systems(systems, M.FP64)
    b.prepare()
    want = b.run(2, DT)
    b.setParticles(np.concatenate([s.ids for s in systems]), np.concatenate([s.cid for s in systems]),
                   np.concatenate([s.r for s in systems]), np.concatenate([s.v for s in systems]))
    with Full(128 << 20):
        with pytest.raises(M.MdgpuError) as ei:
            b.setSkin(0.3)
        assert ei.value.code == 2
    b.prepare()
    np.testing.assert_array_equal(b.run(2, DT), want)     # as without a skin
    b.setSkin(0.3)
    b.prepare()
    b.run(2, DT)
    b.close()
