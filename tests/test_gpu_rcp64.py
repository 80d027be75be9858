"""The FP64 reciprocal of the pair kernels against the correctly rounded 1/x.

The starting value y is the hardware's approximation, whose relative error e = 1 - x y is below 2^-19; the step
y + y (e + e^2) leaves e^3 < 2^-57, a sixteenth of a unit in the last place, and the rounding of the last
operation, half a unit: the nearest double or its neighbour.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from madpac_b200 import build as B
from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rcp64(tmp_path_factory):
    here = os.path.dirname(__file__)
    out = str(tmp_path_factory.mktemp("rcp64") / "rcp64.so")
    subprocess.run([B.nvcc()] + B.NVCC_FLAGS + ["-I", B.CSRC, "-I", os.path.join(B.ROOT, "include"), "-shared", "-cudart",
                    "static", "-o", out, os.path.join(here, "helpers", "rcp64_probe.cu")], check=True)
    lib = ctypes.CDLL(out)

    def go(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y = np.empty_like(x)
        assert lib.rcp64_of(x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), x.size) == 0
        return y

    return go


def numbers(kind):
    rng = np.random.default_rng(1)
    if kind == "squared distances":
        return rng.uniform(0.25, 400.0, 1 << 21)
    if kind == "exponents":
        return np.ldexp(rng.uniform(1.0, 2.0, 1 << 21), rng.integers(-1000, 1001, 1 << 21))
    # every exponent: the powers of two, their neighbours, and mantissas of few bits
    p = np.ldexp(1.0, np.arange(-1000, 1001))
    few = np.concatenate([p * (1.0 + k / 64.0) for k in range(64)])
    return np.concatenate([few, np.nextafter(few, np.inf), np.nextafter(few, 0.0)])


@pytest.mark.parametrize("kind", ["squared distances", "exponents", "powers of two"])
def test_within_one_unit_in_the_last_place(rcp64, kind):
    x = numbers(kind)
    y, want = rcp64(x), 1.0 / x
    assert np.all(np.abs(y - want) <= np.spacing(want))


@pytest.mark.parametrize("precision", [M.FP64, M.MIXED])
@pytest.mark.parametrize("component,h", [(W.two_centre(), 0.25), (W.charged_two_centre(charge_offset=0.375), 0.375)])
def test_coincident_sites_are_reported(precision, component, h):
    """Sites of two molecules in one place, their centres apart: the reciprocal of zero is a NaN where the division
    gave infinity, and the non-finite force is reported as before."""
    lc = M.RigidLinkedCells([12.0, 12.0, 12.0], 3.0, [component], precision=precision)
    r = np.array([[4.0, 4.0, 4.0], [4.0, 4.0, 4.0 + 2.0 * h]])
    lc.addParticles(np.array([1, 2], dtype=np.uint64), np.zeros(2, dtype=np.int32), r, np.zeros((2, 3)),
                    np.tile([1.0, 0.0, 0.0, 0.0], (2, 1)), np.zeros((2, 3)))
    lc.update()
    with pytest.raises(M.MdgpuError) as ei:
        lc.traversePairs()
    assert ei.value.code == 8
    lc.close()
