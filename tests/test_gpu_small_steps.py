"""Time steps of a small body in one cooperative launch against the general passes.

Recording kernel times (``kernel_timing``) keeps a context on the general
passes, two launches per step; the one-launch steps are the same arithmetic in
the same order, so every field agrees bit for bit: from a body of one block per
SM with a few lanes to the largest that fits the SMs' shared memory (and the
first that does not), with last blocks partly empty, with one critical stretch
and with one per point, with prescribed displacements, and in the stepping
form.
"""
import numpy as np
import pytest

from peridigm_b200 import Context, workloads

pytestmark = pytest.mark.gpu
FIELDS = ("Displacement", "Velocity", "Acceleration", "Force_Density", "Dilatation", "Damage", "Bond_Damage")


def _body(dims, hetero):
    if hetero:
        return workloads.large_plate(*dims, pull=3.0)
    return workloads.notched_plate(*dims, notch_cells=max(2, dims[0] // 4), pull=8.0)


def _run(w, precision, general, dt, stepping):
    with Context(precision=precision) as ctx:
        workloads.setup_context(ctx, w)
        if general:
            ctx.kernel_timing(True)
        if stepping:
            ctx.verlet_begin(dt)
            for k in (1, 7, 0, 31):
                ctx.verlet_step(k)
            st = ctx.verlet_finish()
        else:
            st = ctx.verlet_run(dt, 40)
        evaluations = ctx.kernel_times()["evaluations"]
        return st, evaluations, {k: ctx.field(k) for k in FIELDS}


@pytest.mark.parametrize("stepping", [False, True])
@pytest.mark.parametrize("precision,dims,hetero", [
    ("split", (9, 7, 3), False), ("split", (30, 13, 7), True), ("split", (41, 29, 11), False),
    ("split", (41, 29, 11), True), ("split", (60, 43, 10), True),
    ("fp64", (9, 7, 3), False), ("fp64", (30, 13, 7), True), ("fp64", (17, 16, 17), True)])
def test_one_launch_steps_match_the_passes(precision, dims, hetero, stepping):
    w = _body(dims, hetero)
    dt = 4.0e-8
    st, ev, one = _run(w, precision, False, dt, stepping)
    st2, ev2, two = _run(w, precision, True, dt, stepping)
    assert ev2 == 41 and ev == 0  # the general passes were timed, the others did not run timed
    assert st["broken_bonds"] == st2["broken_bonds"]
    for k in FIELDS:
        assert np.array_equal(one[k], two[k]), k


def test_bonds_break_in_the_one_launch_steps():
    w = _body((30, 13, 7), True)
    st, _, f = _run(w, "split", False, 4.0e-8, False)
    assert st["broken_bonds"] > 0 and f["Bond_Damage"].sum() == st["broken_bonds"]


def _kernels(ctx, steps):
    """Names of the bond kernels that verlet_step(steps) launches."""
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        ctx.verlet_step(steps)
    names = " ".join(e.name for e in prof.events())
    return {k for k in ("k_verlet_small", "k_dilatation") if k in names}


@pytest.mark.parametrize("precision,dims,least", [("split", (20, 20, 8), 2), ("split", (40, 32, 10), 5),
                                                  ("fp64", (10, 10, 10), 1)])
def test_few_steps_at_a_time_are_the_passes(precision, dims, least):
    """A launch that fills shared memory for a step or two is slower than the passes (a slab rank steps one by one)."""
    import torch

    torch.zeros(1, device="cuda")
    with Context(precision=precision) as ctx:
        workloads.setup_context(ctx, workloads.large_plate(*dims))
        ctx.verlet_begin(1.0e-9)
        _kernels(ctx, 3)  # (the profiler's own start)
        for k in range(1, 7):
            assert _kernels(ctx, k) == {"k_verlet_small" if k >= least else "k_dilatation"}, k


@pytest.mark.parametrize("precision", ["split", "fp64"])
@pytest.mark.parametrize("steps", [1025, 2050])
def test_more_steps_than_one_launch_takes(precision, steps):
    """1024 to a launch; of the rest of a run a single split step is the passes'."""
    w = _body((9, 7, 3), False)
    got = []
    for general in (False, True):
        with Context(precision=precision) as ctx:
            workloads.setup_context(ctx, w)
            ctx.kernel_timing(general)
            st = ctx.verlet_run(1.0e-8, steps)
            got.append((st["broken_bonds"], [ctx.field(k) for k in FIELDS]))
    assert got[0][0] == got[1][0]
    for k, a, b in zip(FIELDS, got[0][1], got[1][1]):
        assert np.array_equal(a, b), k


@pytest.mark.parametrize("precision", ["split", "fp64"])
def test_damage_of_one_half_and_a_point_without_bonds(precision):
    """Damage that the caller set on one half of a bond, and empty rows, take the same terms in both."""
    w = _body((30, 13, 7), True)
    x = np.concatenate([w["x"], [1.0, 1.0, 1.0], [2.0, 1.0, 1.0]])
    n = x.size // 3
    w = dict(w, x=x, vol=np.full(n, w["vol"][0]), K=np.resize(w["K"], n), mu=np.resize(w["mu"], n),
             s_c=np.resize(w["s_c"], n), v0=np.zeros_like(x))
    got = []
    for general in (False, True):
        with Context(precision=precision) as ctx:
            workloads.setup_context(ctx, w)
            ctx.kernel_timing(general)
            halves = np.zeros(ctx.num_bonds())
            halves[np.random.default_rng(1).permutation(halves.size)[: halves.size // 20]] = 1.0
            ctx.set_bond_damage(halves)
            ctx.verlet_run(4.0e-8, 40)
            got.append([ctx.field(k) for k in FIELDS])
            assert got[-1][-1].sum() > halves.sum()
    for k, a, b in zip(FIELDS, *got):
        assert np.array_equal(a, b, equal_nan=True), k
        if k in ("Displacement", "Velocity", "Force_Density"):
            assert np.isfinite(a).all()
