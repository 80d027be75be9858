"""States of more than 4.2 million molecules, whose fields pass through the staging buffer one by one: they come
back bit for bit, and the buffer takes 24 bytes per molecule, as before it held every field at once."""
import numpy as np
import pytest
import torch

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu

N = 4_200_000     # the fields go together up to 2^22 = 4,194,304


def state(n, length, seed=1):
    rng = np.random.default_rng(seed)
    return (rng.permutation(np.arange(1, n + 1)).astype(np.uint64), rng.uniform(0.0, length, (n, 3)),
            rng.standard_normal((n, 3)), rng.standard_normal((n, 3)))


def used(before):
    return before - torch.cuda.mem_get_info()[0]


def test_container():
    torch.cuda.synchronize()
    L = 174.0
    ids, r, v, F = state(N, L)
    lc = M.LinkedCells([L] * 3, 2.5, W.two_species(), np.ones((1, 2)))
    cid = (ids % 2).astype(np.int32)
    free = torch.cuda.mem_get_info()[0]
    lc.addParticles(ids, cid, r, v, F)
    # two sets of 88 bytes, the binning's 12, the staging's 24, per-block sums
    assert used(free) <= 225 * N + (64 << 20)
    st = lc.getParticles()
    assert used(free) <= 225 * N + (64 << 20)
    for key, want in (("id", ids), ("cid", cid), ("r", r), ("v", v), ("F", F)):
        np.testing.assert_array_equal(st[key], want)
    lc.close()


def test_ensemble():
    torch.cuda.synchronize()
    boxes, L = 420, 24.0
    n = N // boxes
    ids, r, v, _ = state(N, L)
    cid = (ids % 2).astype(np.int32)
    free = torch.cuda.mem_get_info()[0]
    b = M.Batch([[L] * 3] * boxes, [n] * boxes, 2.5, W.two_species(), np.ones((1, 2)))
    b.setParticles(ids, cid, r, v)
    assert used(free) <= 225 * N + (64 << 20)
    st = b.getParticles()
    for key, want in (("id", ids), ("cid", cid), ("r", r), ("v", v)):
        np.testing.assert_array_equal(st[key], want)
    b.close()


def test_rigid_container():
    L = 300.0
    ids, r, v, D = state(N, L)
    q = np.random.default_rng(2).standard_normal((N, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    lc = M.RigidLinkedCells([L] * 3, 3.0, [W.two_centre()])
    lc.addParticles(ids, np.zeros(N, dtype=np.int32), r, v, q, D)
    st = lc.getParticles()
    for key, want in (("id", ids), ("r", r), ("v", v), ("q", q), ("D", D)):
        np.testing.assert_array_equal(st[key], want)
    lc.close()
