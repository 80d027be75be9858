"""Host threads with a container each, of different sizes: the shared memory that one's launches ask for does not
limit the other's."""
import threading

import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu


def box(n, rc, seed):
    s = W.lj_fcc_box(int(np.ceil((n / 4.0) ** (1.0 / 3.0))), 0.7, 1.0, seed, rc, [W.Component(1.0, 1.0, 1.0, True)],
                     n_atoms=n)
    s.r = (s.r + np.random.default_rng(seed).uniform(-0.05, 0.05, s.r.shape)) % s.length
    s.r[s.r >= s.length] = 0.0
    return s


def run(s, precision, skin, calls, steps):
    lc = M.LinkedCells.from_system(s, precision)
    if skin:
        lc.setSkin(skin)
    out = []
    for _ in range(calls):
        lc.setState(s.r, s.v)
        lc.update()
        lc.traversePairs()
        out.append(lc.run(steps, 0.002))
    lc.close()
    return out


# binned: the one-launch binning of 4,096 molecules wants 57 KB, of 500 less than 10, the traversal of 1,400 at a cutoff
# of 3 twice that of 500; with a skin one, two or three CTAs per SM
@pytest.mark.parametrize("sizes,precision,skin", [(((500, 2.5), (4096, 2.5), (1200, 3.0)), M.FP64, 0.0),
                                                  (((1000, 2.5), (14000, 3.0), (5000, 2.5)), M.FP64, 0.3),
                                                  (((1000, 2.5), (14000, 3.0), (5000, 2.5)), M.MIXED, 0.3)])
def test_containers_of_different_sizes(sizes, precision, skin):
    errors = []
    start = threading.Barrier(len(sizes))

    def work(n, rc):
        try:
            s = box(n, rc, n)
            one = run(s, precision, skin, 1, 5)[0]
            start.wait(120)
            for recs in run(s, precision, skin, 150, 5):
                np.testing.assert_array_equal(recs, one)
        except BaseException as e:   # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
