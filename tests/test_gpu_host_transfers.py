"""Large transfers between the device and pageable memory of the caller.

Coordinates and forces of a megabyte and more (beside the kernels) and states
and fields of 40 and 3 MB (alone) go through a pinned ring by worker threads,
once 192 MB of such have passed in the process (a context held open here sees
to that): what is read back is what was written, bit for bit, at sizes around
the thresholds, the pieces (512 KB) and the ring (8 MB, reused), for a force
evaluated from host buffers against the same from device pointers, and from
several threads at once, of which one at a time has the ring.
"""
import os
import threading

import numpy as np
import pytest

from peridigm_b200 import Context, workloads

pytestmark = pytest.mark.gpu


def _context(dims, precision="split"):
    x, vol = workloads.lattice(*dims, 1.0e-3, jitter=0.05, seed=1)
    ctx = Context(precision=precision)
    ctx.set_points(x, vol)
    ctx.set_horizons([1.6e-3])
    ctx.build_bonds()
    ctx.material(130.0e9, 78.0e9, 7800.0)
    ctx.critical_stretch(5.0e-4)
    return ctx, x


@pytest.fixture(scope="module", autouse=True)
def ring():
    ctx, x = _context((101, 103, 71))
    with ctx:
        before = len(os.listdir("/proc/self/task"))
        for _ in range(6):  # 35 MB each
            ctx.compute_force(x)
        assert len(os.listdir("/proc/self/task")) > before  # its workers
        yield


@pytest.mark.parametrize("dims", [(43, 127, 8), (43691, 1, 1), (65536, 1, 1), (61, 67, 83), (101, 103, 71), (131_072, 1, 1),
                                  (1_747_627, 1, 1)])
def test_state_round_trip(dims):
    ctx, x = _context(dims)
    rng = np.random.default_rng(0)
    with ctx:
        for _ in range(2):
            u, v = rng.normal(0, 1e-6, x.size), rng.normal(0, 1.0, x.size)
            ctx.set_state(u, v)
            assert np.array_equal(ctx.field("Displacement"), u) and np.array_equal(ctx.field("Velocity"), v)
            assert np.array_equal(ctx.field("Coordinates"), x + u)


@pytest.mark.parametrize("precision", ["split", "fp64"])
@pytest.mark.parametrize("dims", [(43, 127, 8), (101, 103, 71)])
def test_force_from_host_buffers_is_the_device_one(dims, precision):
    import torch

    ctx, x = _context(dims, precision)
    rng = np.random.default_rng(2)
    with ctx:
        for _ in range(3):
            y = x * (1.0 + 1.0e-4) + rng.normal(0, 1e-7, x.size)
            f = ctx.compute_force(y)
            yd = torch.from_numpy(y).cuda()
            fd = torch.empty_like(yd)
            torch.cuda.synchronize()
            ctx.compute_force_device(yd.data_ptr(), fd.data_ptr())
            assert np.array_equal(f, fd.cpu().numpy())
            pinned = torch.from_numpy(y).pin_memory()
            assert np.array_equal(ctx.compute_force(pinned.numpy()), f)


def test_threads_with_contexts_of_their_own():
    made = [_context((61, 67, 20 + k)) for k in range(4)]
    bad = []

    def work(ctx, x, seed):
        rng = np.random.default_rng(seed)
        for _ in range(6):
            u = rng.normal(0, 1e-6, x.size)
            ctx.set_state(u, u)
            if not (np.array_equal(ctx.field("Displacement"), u) and np.array_equal(ctx.field("Velocity"), u)):
                bad.append(seed)

    threads = [threading.Thread(target=work, args=(c, x, k)) for k, (c, x) in enumerate(made)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c, _ in made:
        c.close()
    assert not bad
