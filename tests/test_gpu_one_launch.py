"""What can go wrong with the kernels that run a loop of a small body in one launch.

The bounded waits. With the arrivals counted from a number that no target is
reached from, the first wait of the time steps and of the CG solve runs out
(within a second): the call says so, the blocks all leave, and nothing goes on
with a state that is not of one step. After the state is set again the context
steps and solves as a new one does, bit for bit.

The launch itself. Where the driver refuses it, the general passes and the
general CG loop take the steps and the solve.
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


@pytest.mark.parametrize("stepping", [False, True])
@pytest.mark.parametrize("precision", ["split", "fp64"])
def test_time_steps_whose_launch_is_refused(precision, stepping):
    w = workloads.large_plate(30, 13, 7, pull=3.0)
    lib = _internals.load()
    got = []
    for refuse in (False, True):
        with Context(precision=precision) as ctx:
            workloads.setup_context(ctx, w)
            ctx.verlet_run(DT, 4)
            assert lib.small_step_threads(ctx.h) > 0
            if refuse:
                lib.ask_too_much(ctx.h)
            if stepping:
                ctx.verlet_begin(DT)
                ctx.verlet_step(9)
                ctx.verlet_step(10)
                ctx.verlet_finish()
            else:
                ctx.verlet_run(DT, 20)
            assert (lib.small_step_threads(ctx.h) == 0) == refuse
            got.append([ctx.field(k) for k in FIELDS])
    for name, a, b in zip(FIELDS, *got):
        assert np.array_equal(a, b), name


@pytest.mark.parametrize("precond", ["none", "block_jacobi"])
def test_a_solve_whose_launch_is_refused(precond):
    w = workloads.qs_cube(n=10, jitter=0.05, load_steps=4)
    lib = _internals.load()
    got = []
    for refuse in (False, True):
        with Context(precision="fp64") as ctx:
            workloads.setup_context(ctx, w)
            ctx.qs_load_step(0.0, 0.25, newton_tolerance=-1e-9, preconditioner=precond, use_predictor=False)
            if refuse:
                lib.ask_too_much(ctx.h)
            st = ctx.qs_load_step(0.25, 0.5, newton_tolerance=-1e-9, preconditioner=precond, use_predictor=False)
            got.append((st.cg_iterations, ctx.field("Displacement")))
    assert abs(got[0][0] - got[1][0]) <= 0.02 * got[0][0] + 1
    assert np.linalg.norm(got[0][1] - got[1][1]) <= 1e-7 * np.linalg.norm(got[0][1])
