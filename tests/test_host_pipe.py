"""The pinned transfer ring's host logic, without a device.

host_pipe.cu is compiled against stand-ins for the CUDA calls it makes
(fake_cudart.cpp: copies in host memory, events that are complete), each test
in a process of its own:

* bytes arrive whole, both ways, for sizes around the piece and the ring;
* the ring is made once the contexts that are open have moved 192 MB, and
  given back with the last of them: contexts one after another, each with
  less, never make it;
* a transfer alone takes the ring only at sizes where it gains by it: 40 MB
  up, 3 MB down;
* beside kernels only the calling thread waits for the device: a worker that
  did would spin beside it for as long as the kernels before a copy take;
* a forked child, where the workers do not run, lets its contexts go and
  leaves its transfers to the driver.
"""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "peridigm_b200", "csrc")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    nvcc = os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")
    so = str(tmp_path_factory.mktemp("host_pipe") / "host_pipe.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-pthread", "-I", CSRC, "-I",
                    os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include"), "-x", "c++",
                    os.path.join(CSRC, "host_pipe.cu"), os.path.join(HERE, "fake_cudart.cpp"), "-o", so], check=True)
    return so


PRELUDE = """
import ctypes as C, os, sys, time
import numpy as np
L = C.CDLL(sys.argv[1])
MADE, FREED, WAITS, WORKER_WAITS = range(4)

def move(fn, dst, src, beside=1):
    return fn(C.c_void_p(dst.ctypes.data), C.c_void_p(src.ctypes.data), C.c_size_t(src.nbytes), beside)

def earn():
    a = np.zeros(32 << 20, np.uint8)
    b = np.zeros_like(a)
    for _ in range(6):
        move(L.up, b, a)
    assert L.count(MADE) == 1
"""


def run(library, body, seconds=60):
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(body), library], capture_output=True, text=True,
                       timeout=seconds)
    assert r.returncode == 0, r.stdout + r.stderr


def test_bytes_arrive_whole(library):
    run(library, """
        L.open_context()
        earn()
        rng = np.random.default_rng(0)
        for size in (1 << 20, (1 << 20) + 1, (8 << 20) - 3, 8 << 20, (8 << 20) + 5, 20_000_003):
            a = rng.integers(0, 256, size, dtype=np.uint8)
            for fn in (L.up, L.down):
                for beside in (1, 0):
                    b = np.zeros_like(a)
                    took = move(fn, b, a, beside)
                    assert took == (beside or (fn == L.down and size >= 3 << 20))
                    assert not took or np.array_equal(a, b)
        assert move(L.up, np.zeros(1000, np.uint8), np.zeros(1000, np.uint8)) == 0  # small: the driver's
        L.close_context()
        assert L.count(FREED) == 1
    """)


def test_contexts_one_after_another_do_not_make_the_ring(library):
    run(library, """
        a = np.zeros(15 << 20, np.uint8)
        b = np.zeros_like(a)
        for _ in range(30):  # 450 MB in all, 15 to a context
            L.open_context()
            assert move(L.up, b, a) == 0
            L.close_context()
        assert L.count(MADE) == 0
        L.open_context()  # 225 MB in one
        got = [move(L.down, b, a) for _ in range(15)]
        assert got == [0] * 12 + [1] * 3 and L.count(MADE) == 1
        L.close_context()
        assert L.count(FREED) == 1
    """)


def test_transfers_alone_that_the_driver_is_better_at_are_its(library):
    run(library, """
        L.open_context()
        a, b = np.zeros(48 << 20, np.uint8), np.zeros(48 << 20, np.uint8)
        for _ in range(30):  # nothing that counts towards the ring
            assert move(L.up, b[:24 << 20], a[:24 << 20], 0) == 0
            assert move(L.down, b[:2 << 20], a[:2 << 20], 0) == 0
        assert L.count(MADE) == 0
        earn()
        for fn, least in ((L.up, 40 << 20), (L.down, 3 << 20)):
            for size in (1 << 20, least - 1, least, 41 << 20):
                assert move(fn, b[:size], a[:size], 0) == (size >= least)
                assert move(fn, b[:size], a[:size], 1) == 1
        L.close_context()
    """)


def test_the_workers_do_not_wait_for_the_device(library):
    run(library, """
        L.open_context()
        earn()
        a = np.arange(40_000_001, dtype=np.uint8)
        for fn in (L.up, L.down):
            b = np.zeros_like(a)
            assert move(fn, b, a) == 1 and np.array_equal(a, b)
        assert L.count(WAITS) > 0 and L.count(WORKER_WAITS) == 0
        L.close_context()
    """)


def test_a_forked_child_does_without_the_workers(library):
    run(library, """
        L.open_context()
        earn()
        a, b = np.zeros(4 << 20, np.uint8), np.zeros(4 << 20, np.uint8)
        child = os.fork()
        if child == 0:
            ok = move(L.up, b, a) == 0 and move(L.down, b, a) == 0
            L.close_context()
            os._exit(0 if ok else 1)
        for _ in range(100):  # ten seconds
            pid, status = os.waitpid(child, os.WNOHANG)
            if pid:
                break
            time.sleep(0.1)
        else:
            os.kill(child, 9)
            os.waitpid(child, 0)
            sys.exit("the child did not come back")
        assert status == 0
        assert move(L.up, b, a) == 1  # the parent's ring is as it was
        L.close_context()
        assert L.count(FREED) == 1
    """)
