"""States through the pinned-chunk copies: sizes around the chunk and thread limits (chunks of 512 KB, another
host thread from 3 MB on), arrays pinned by the caller, and two host threads with a container each. Copies
move bytes: everything comes back bit for bit."""
import threading

import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu


def container(n, seed, length=60.0):
    rng = np.random.default_rng(seed)
    s = W.System(length=np.full(3, length), components=[W.Component(1.0, 1.0, 1.0, True)], mix=np.ones((0, 2)),
                 ids=np.arange(1, n + 1, dtype=np.uint64), cid=np.zeros(n, dtype=np.int32),
                 r=rng.uniform(0.0, length, (n, 3)), v=rng.standard_normal((n, 3)))
    return s, M.LinkedCells.from_system(s)


def round_trips(n, seed, passes=2):
    s, lc = container(n, seed)
    rng = np.random.default_rng(seed + 1)
    st = lc.getParticles()
    np.testing.assert_array_equal(st["r"], s.r)
    np.testing.assert_array_equal(st["v"], s.v)
    np.testing.assert_array_equal(st["id"], s.ids)
    np.testing.assert_array_equal(st["cid"], s.cid)
    for _ in range(passes):
        r, v = rng.uniform(0.0, 60.0, (n, 3)), rng.standard_normal((n, 3))
        lc.setState(r, v)
        lc.update()                     # another order on the device
        st = lc.getParticles()
        np.testing.assert_array_equal(st["r"], r)
        np.testing.assert_array_equal(st["v"], v)
        np.testing.assert_array_equal(st["id"], s.ids)
        cells = lc.getCellIndexOfMolecule()
        assert cells.shape == (n,) and cells.min() >= 0
    lc.close()


# 24 bytes per molecule and array: 21,845 molecules end 8 bytes before a chunk, 21,846 begin the next
@pytest.mark.parametrize("n", [1, 2, 21845, 21846, 43691, 65536, 131072, 300001])
def test_states_come_back_bit_for_bit(n):
    round_trips(n, n)


def test_arrays_pinned_by_the_caller():
    import torch

    n = 50000
    s, lc = container(n, 5)
    pin = [torch.empty((n, 3), dtype=torch.float64, pin_memory=True).numpy() for _ in range(4)]
    rng = np.random.default_rng(6)
    pin[0][:] = rng.uniform(0.0, 60.0, (n, 3))
    pin[1][:] = rng.standard_normal((n, 3))
    lc.setState(pin[0], pin[1])
    lc.synchronize()
    assert lc.lib.mdgpu_get_particles(lc.h, n, None, None, pin[2].ctypes.data, pin[3].ctypes.data, None) == 0
    np.testing.assert_array_equal(pin[2], pin[0])
    np.testing.assert_array_equal(pin[3], pin[1])
    lc.close()


def test_two_threads():
    errors = []

    def work(seed):
        try:
            for k in range(3):
                round_trips(150000, seed + k, passes=1)
        except BaseException as e:   # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(seed,)) for seed in (10, 20)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
