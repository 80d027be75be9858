"""Binning at the limits of its forms: up to 4096 molecules and 4096 cells one CTA does it all, beyond that one
thread per molecule over the device. Cells are the reference's formula on the wrapped position, bit for bit,
and the molecules of a cell are in id order whatever order they were given in."""
import numpy as np
import pytest

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu


# (molecules, box edge / cutoff): cells 2^3 to 16^3 = 4096 and one more per dimension
@pytest.mark.parametrize("n,edge", [(1, 2.0), (2, 3.5), (1023, 4.2), (1025, 5.0), (4095, 2.5), (4096, 16.0), (4096, 16.4),
                                    (4096, 17.0), (4097, 6.0), (6000, 2.0)])
@pytest.mark.parametrize("with_forces", [False, True])
def test_cells_and_state(n, edge, with_forces):
    rng = np.random.default_rng(n)
    L = np.array([edge * 1.5, edge * 1.5 + 0.1, edge * 1.5 + 0.2])
    r = rng.uniform(-0.05, 1.05, (n, 3)) * L       # some outside: wrapped by one box length
    ids = rng.permutation(np.arange(1, n + 1)).astype(np.uint64)
    v, F = rng.standard_normal((n, 3)), rng.standard_normal((n, 3))
    lc = M.LinkedCells(L, 1.5, [W.Component(1.0, 1.0, 1.0, True)])
    lc.addParticles(ids, np.zeros(n, dtype=np.int32), r, v, F if with_forces else None)
    lc.update()
    w = np.where(r < 0.0, r + L, np.where(r >= L, r - L, r))
    geo = lc.geometry()
    c = np.floor((w - geo["halo_min"]) / geo["cell_length"]).astype(np.int64)
    cx, cy = geo["box_cells"][0] + 2, geo["box_cells"][1] + 2
    np.testing.assert_array_equal(lc.getCellIndexOfMolecule(), (c[:, 2] * cy + c[:, 1]) * cx + c[:, 0])
    st = lc.getParticles()
    for key, want in (("r", w), ("v", v), ("F", F if with_forces else np.zeros((n, 3))), ("id", ids)):
        np.testing.assert_array_equal(st[key], want)
    lc.close()


def test_equal_starts_give_equal_bits():
    """The order within a cell is by id: two containers loaded in different orders sum the same forces."""
    s = W.lj_fcc_box(9, 0.7, 1.0, 3, 2.5, [W.Component(1.0, 1.0, 1.0, True)], n_atoms=2500)
    rng = np.random.default_rng(4)
    s.r = (s.r + rng.uniform(-0.05, 0.05, s.r.shape)) % s.length
    order = rng.permutation(s.n)
    out = []
    for o in (np.arange(s.n), order):
        lc = M.LinkedCells(s.length, s.cutoff, s.components)
        lc.addParticles(s.ids[o], s.cid[o], s.r[o], s.v[o])
        lc.update()
        lc.traversePairs()
        F = np.empty((s.n, 3))
        F[o] = lc.getParticles()["F"]
        out.append(F)
        lc.close()
    np.testing.assert_array_equal(out[0], out[1])
