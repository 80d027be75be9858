"""The FP64 list kernel with pruned lists runs three CTAs per SM where its regions fit. 702,464 molecules of the lattice
start, regions of 2,048, capacity 2,368: its step took 1.17 times the mixed form's with three and 1.39 times with two."""
import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_three_ctas_of_the_fp64_lists():
    s = W.lj_fcc_box(56, 0.75, 0.9, 1, 3.0, [W.Component(1.0, 1.0, 1.0, True)])
    best = {}
    for precision in (M.MIXED, M.FP64):
        lc = M.LinkedCells.from_system(s, precision)
        lc.update()
        lc.traversePairs()
        lc.setSkin(0.4)
        lc.setListPrune(0.15)
        lc.run(10, s.dt)
        lc.profileEnable(True)
        times = []
        for _ in range(4):
            lc.profileRead(True)
            lc.run(20, s.dt)
            times.append(lc.profileRead(True)[0][1])
        best[precision] = np.min(times)
        lc.close()
    assert best[M.FP64] <= 1.28 * best[M.MIXED]
