"""The bounded waits of the kernels that run a loop of a small body in one launch.

With the arrivals counted from a number that no target is reached from, the
first wait of the time steps and of the CG solve runs out (within a second):
the call says so, the blocks all leave, and nothing goes on with a state that is not of one step. After the
state is set again the context steps and solves as a new one does, bit for
bit.
"""
import ctypes as C

import _internals
import numpy as np
import pytest

from peridigm_b200 import Context, PDError, _lib, workloads

pytestmark = pytest.mark.gpu
FIELDS = ("Displacement", "Velocity", "Force_Density", "Dilatation", "Damage", "Bond_Damage")
DT = 4.0e-8


def _waits_run_out(ctx, on):
    _internals.load().set_waits_run_out(ctx.h, C.c_int(on))


def _fails(status, call, *args, **kw):
    with pytest.raises(PDError) as e:
        call(*args, **kw)
    assert e.value.code == status, str(e.value)


def _run(ctx):
    ctx.verlet_run(DT, 20)
    return [ctx.field(k) for k in FIELDS]


@pytest.mark.parametrize("stepping", [False, True])
@pytest.mark.parametrize("precision", ["split", "fp64"])
def test_time_steps_whose_wait_runs_out(precision, stepping):
    w = workloads.large_plate(30, 13, 7, pull=3.0)
    z = np.zeros_like(w["x"])
    with Context(precision=precision) as ctx:
        want = _run(workloads.setup_context(ctx, w))
        intact = np.zeros(ctx.num_bonds())
    assert want[-1].any()
    with Context(precision=precision) as ctx:
        workloads.setup_context(ctx, w)
        _waits_run_out(ctx, 1)
        if stepping:
            ctx.verlet_begin(DT)
            _fails(_lib.PD_ERR_TIMEOUT, ctx.verlet_step, 20)
            _fails(_lib.PD_ERR_STATE, ctx.verlet_step, 1)  # the run is over
            _fails(_lib.PD_ERR_STATE, ctx.verlet_finish)
        else:
            _fails(_lib.PD_ERR_TIMEOUT, ctx.verlet_run, DT, 20)
        _waits_run_out(ctx, 0)
        # (a second call is refused too: the error is not of one call)
        for _ in range(2):
            _fails(_lib.PD_ERR_STATE, ctx.verlet_run, DT, 20)
            _fails(_lib.PD_ERR_STATE, ctx.verlet_begin, DT)
            _fails(_lib.PD_ERR_STATE, ctx.qs_load_step, 0.0, 0.1, 1e-6)
            _fails(_lib.PD_ERR_STATE, ctx.implicit_run, 1e-7, 1)
            _fails(_lib.PD_ERR_STATE, ctx.set_state, z, None)
            _fails(_lib.PD_ERR_STATE, ctx.set_state, None, z)
        ctx.set_state(z, w["v0"])
        ctx.set_bond_damage(intact)
        for name, a, b in zip(FIELDS, _run(ctx), want):
            assert np.array_equal(a, b), name


def test_a_solve_whose_wait_runs_out():
    w = workloads.qs_cube(n=10, jitter=0.05, load_steps=4)
    z = np.zeros_like(w["x"])

    def step(ctx):
        ctx.qs_load_step(0.0, 0.25, newton_tolerance=-1e-9, use_predictor=False)
        return ctx.field("Displacement")

    with Context(precision="fp64") as ctx:
        want = step(workloads.setup_context(ctx, w))
    with Context(precision="fp64") as ctx:
        workloads.setup_context(ctx, w)
        _waits_run_out(ctx, 1)
        for _ in range(2):
            _fails(_lib.PD_ERR_TIMEOUT, step, ctx)
            assert np.array_equal(ctx.field("Displacement"), z)  # nothing of it was taken over
        _waits_run_out(ctx, 0)
        assert np.array_equal(step(ctx), want)
