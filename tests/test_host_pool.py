"""The copy threads and buffer sizes of host-array predictions, on the CPU."""
import ctypes as C
import os
import subprocess

import pytest

from tests.conftest import ROOT


@pytest.fixture(scope="module")
def pool(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pool") / "libpool_check.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", "-o", so,
                           os.path.join(ROOT, "tests", "native", "pool_check.cpp")])
    lib = C.CDLL(so)
    lib.pool_check_pinned_size.restype = C.c_size_t
    lib.pool_check_pinned_size.argtypes = [C.c_size_t]
    return lib


@pytest.mark.parametrize("threads", [1, 2, 5])
def test_every_item_of_every_job_is_done_once(pool, threads):
    """Callers that find the pool busy do their jobs alone; empty jobs, single items, many items."""
    assert pool.pool_check_jobs(threads, 2000, 200) == 0


def test_forked_child_does_its_jobs_alone(pool):
    assert pool.pool_check_fork(50) == 0


def test_pinned_sizes(pool):
    """At least what was asked for, at most a quarter more beyond a megabyte, and few different ones."""
    size = pool.pool_check_pinned_size
    for n in [1, 65_536, 65_537, 1 << 20, (1 << 20) + 1, 5 << 20, (5 << 20) + 1, (1 << 33) + 3]:
        assert size(n) >= n and size(size(n)) == size(n)
        assert size(n) <= (n * 5 // 4 + 1 if n > 1 << 20 else max(65_536, 2 * n))
    assert len({size(n) for n in range(1, 16 << 20, 4096)}) <= 5 + 16
