"""Results do not depend on what an earlier kernel left in shared memory.

Lists end in padding, and a lane whose list is shorter than its warp's longest runs on without entries. Neither may
look at a slot that nothing was staged to: a NaN or an infinity there would reach the force, the energy and the
virial. Before the steps a kernel leaves all-ones words (a NaN as a double) or -inf in the shared memory of
every SM; the same run after zeros gives the same bits.
"""
import ctypes
import os
import struct
import subprocess

import numpy as np
import pytest

from madpac_b200 import build as B
from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu

PATTERNS = [0xFFFFFFFFFFFFFFFF, struct.unpack("<Q", struct.pack("<d", -np.inf))[0]]
STEPS, DT = 4, 0.002


@pytest.fixture(scope="module")
def fill(tmp_path_factory):
    src = os.path.join(os.path.dirname(__file__), "helpers", "fill_shared.cu")
    out = str(tmp_path_factory.mktemp("fill") / "fill.so")
    subprocess.run([B.nvcc()] + B.NVCC_FLAGS + ["-shared", "-cudart", "static", "-o", out, src], check=True)
    lib = ctypes.CDLL(out)
    lib.fill_shared.argtypes = [ctypes.c_ulonglong]

    def go(word):
        assert lib.fill_shared(word) == 0

    return go


def system(kind, species):
    comps = W.two_species() if species == 2 else [W.Component(1.0, 1.0, 1.0, True)]
    if kind == "slab":
        s = W.config_c3(9, 20000)
        if species == 1:
            s.components, s.mix, s.cid = comps, np.ones((0, 2)), np.zeros_like(s.cid)
        return s
    s = W.lj_fcc_box(9, 0.7, 1.0, 3, 2.5, comps, n_atoms=2800)
    s.r = (s.r + np.random.default_rng(5).uniform(-0.05, 0.05, s.r.shape)) % s.length
    s.r[s.r >= s.length] = 0.0
    return s


# dense bricks, the same with pruned lists, and a slab whose vapour goes one warp per brick
@pytest.mark.parametrize("kind,prune", [("box", 0.0), ("box", 0.15), ("slab", 0.15)])
@pytest.mark.parametrize("species", [1, 2])
@pytest.mark.parametrize("precision", [M.FP64, M.MIXED])
def test_skin_runs(fill, kind, prune, species, precision):
    s = system(kind, species)
    out = []
    for word in [0] + PATTERNS:
        lc = M.LinkedCells.from_system(s, precision)
        lc.update()
        lc.traversePairs()
        lc.setSkin(0.4)
        lc.setListPrune(prune)
        recs = []
        for _ in range(STEPS):
            fill(word)
            recs.append(lc.run(1, DT))
        out.append((np.concatenate(recs), lc.getParticles()["F"]))
        lc.close()
    for recs, F in out[1:]:
        np.testing.assert_array_equal(recs, out[0][0])
        np.testing.assert_array_equal(F, out[0][1])


@pytest.mark.parametrize("species", [1, 2])
def test_traversal(fill, species):
    for kind in ("box", "slab"):
        s = system(kind, species)
        out = []
        for word in [0] + PATTERNS:
            lc = M.LinkedCells.from_system(s, M.FP64)
            lc.update()
            fill(word)
            out.append((lc.traversePairs(), lc.getParticles()["F"]))
            lc.close()
        for sums, F in out[1:]:
            assert sums == out[0][0]
            np.testing.assert_array_equal(F, out[0][1])


@pytest.mark.parametrize("species", [1, 2])
@pytest.mark.parametrize("skin", [0.0, 0.3])
def test_ensemble(fill, species, skin):
    comps = W.two_species() if species == 2 else [W.Component(1.0, 1.0, 1.0, True)]
    systems = [W.lj_fcc_box(7, 0.7, 1.0, k, 2.5, comps, n_atoms=n) for k, n in enumerate((300, 700, 1300))]
    out = []
    for word in [0] + PATTERNS:
        b = M.Batch.from_systems(systems, M.FP64)
        if skin:
            b.setSkin(skin)
        fill(word)
        b.prepare()
        fill(word)
        recs = b.run(STEPS, DT)
        out.append((recs, b.getParticles()["F"]))
        b.close()
    for recs, F in out[1:]:
        np.testing.assert_array_equal(recs, out[0][0])
        np.testing.assert_array_equal(F, out[0][1])
