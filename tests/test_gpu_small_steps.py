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
