"""The copies between a caller's arrays and the device, against a stand-in for the CUDA runtime whose copies run only
when something waits for them and whose calls can be made to fail (no GPU)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "madpac_b200", "csrc")
HOST, DEVICE, MANAGED = 1, 2, 3     # memory types; 0: pageable
MB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("transfer") / "transfer.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-I", os.path.join(HERE, "helpers", "fake_cuda"),
                    "-I", CSRC, "-o", out, os.path.join(HERE, "helpers", "transfer_harness.cpp")], check=True)
    lib = ctypes.CDLL(out)
    lib.retain()
    return lib


def copy(lib, sizes, to_host, types=None):
    """Copies random bytes; (status, whether the target holds them)."""
    rng = np.random.default_rng(1)
    src = [rng.integers(0, 255, n, dtype=np.uint8) for n in sizes]
    dst = [np.zeros(n, dtype=np.uint8) for n in sizes]
    host, dev = (dst, src) if to_host else (src, dst)
    for a, t in zip(host, types or []):
        lib.fake_type(ctypes.c_void_p(a.ctypes.data), t)
    n = len(sizes)
    st = lib.copy_spans(n, (ctypes.c_void_p * n)(*[a.ctypes.data for a in host]),
                        (ctypes.c_void_p * n)(*[a.ctypes.data for a in dev]), (ctypes.c_size_t * n)(*sizes), int(to_host))
    in_flight = lib.fake_in_flight()
    same = [np.array_equal(a, b) for a, b in zip(src, dst)]
    lib.fake_finish()
    return st, in_flight, same, [np.array_equal(a, b) for a, b in zip(src, dst)]


@pytest.mark.parametrize("to_host", [False, True])
@pytest.mark.parametrize("sizes", [[1], [8, 0, 24], [MB // 2, MB // 2 + 1], [20 * MB, 3, 5 * MB + 7]])
def test_bytes(lib, sizes, to_host):
    lib.fake_reset(-1, -1)
    st, in_flight, same, after = copy(lib, sizes, to_host)
    assert st == 0 and in_flight == 0 and all(same) and lib.fake_plain() == 0


@pytest.mark.parametrize("to_host", [False, True])
def test_without_pinned_memory_the_driver_stages(lib, to_host):
    lib.release()       # give the idle chunks back
    lib.retain()
    assert lib.fake_chunks() == 0
    lib.fake_reset(0, -1)
    st, in_flight, same, after = copy(lib, [20 * MB, 3, 5 * MB + 7], to_host)
    assert st == 0 and all(after)
    if to_host:
        assert in_flight == 0 and all(same)
    lib.fake_reset(-1, -1)


@pytest.mark.parametrize("alloc_fails", [0, 1, 2, 5])
def test_a_copy_that_succeeds_leaves_no_error_behind(lib, alloc_fails):
    """Some pinned chunks are to be had, others not: the copy does with fewer, and the next call that looks for the
    errors of its own launches finds none."""
    lib.release()
    lib.retain()
    lib.fake_reset(alloc_fails, -1)
    st, in_flight, same, after = copy(lib, [20 * MB], True)
    assert st == 0 and all(same) and lib.fake_last_error() == 0
    lib.fake_reset(-1, -1)


@pytest.mark.parametrize("to_host", [False, True])
@pytest.mark.parametrize("fails_at", [1, 2, 3])
def test_an_error_leaves_no_copy_of_the_callers_memory_in_flight(lib, to_host, fails_at):
    """Two arrays that the caller pinned and a pageable one; the second, third or fourth copy fails."""
    lib.fake_reset(-1, fails_at)
    st, in_flight, same, after = copy(lib, [2 * MB, 2 * MB, MB], to_host, [HOST, HOST, 0])
    assert st == 1 and in_flight == 0


def test_managed_and_device_memory_go_to_the_driver(lib):
    for t in (MANAGED, DEVICE):
        lib.fake_reset(-1, -1)
        st, in_flight, same, after = copy(lib, [100, 3 * MB], True, [t, t])
        assert st == 0 and in_flight == 0 and all(same) and lib.fake_plain() == 2


def test_threads_follow_the_processors_the_process_may_use(lib):
    """A copy of 64 MB takes up to eight threads, but on one or two processors only the calling one."""
    allowed = os.sched_getaffinity(0)
    try:
        os.sched_setaffinity(0, sorted(allowed)[:2])
        lib.fake_reset(-1, -1)
        st, in_flight, same, after = copy(lib, [64 * MB], True)
        assert st == 0 and all(same) and lib.fake_threads() == 1
    finally:
        os.sched_setaffinity(0, allowed)
