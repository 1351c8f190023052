"""Trial evaluations that break no bond leave the damage buffers as they are.

An evaluation works on a copy of the committed damage; after one that broke
nothing the copy is still good and is neither made again nor its sliced mirror
refreshed. Every order of evaluations with and without breaks, commits, caller
set damage and time steps gives what a context gives that evaluates once on
the same committed damage, bit for bit.
"""
import numpy as np
import pytest

from peridigm_b200 import Context, workloads

pytestmark = pytest.mark.gpu


def _context(w, precision, material):
    ctx = Context(precision=precision)
    if material == "lps":
        return workloads.setup_context(ctx, w)
    ctx.set_points(w["x"], w["vol"])
    ctx.set_horizons([w["horizon"]])
    ctx.build_bonds([])
    ctx.material_bond_based(130.0e9, w["rho"])
    ctx.critical_stretch(4.0e-4)
    ctx.set_state(np.zeros_like(w["x"]), w["v0"])
    return ctx


def _once(w, precision, material, y, committed):
    """One evaluation on a given committed damage, in a context of its own."""
    with _context(w, precision, material) as ctx:
        ctx.set_bond_damage(committed)
        f = ctx.compute_force(y)
        return f, ctx.field("Bond_Damage"), ctx.field("Damage")


@pytest.mark.parametrize("precision,material", [("split", "lps"), ("fp64_sliced", "lps"), ("fp64", "lps"),
                                                ("split", "bond_based")])
def test_evaluations_with_and_without_breaks(precision, material):
    w = workloads.large_plate(19, 14, 9, pull=3.0)
    P = w["x"].reshape(-1, 3)
    calm, torn = P.copy(), P.copy()
    calm[:, 0] *= 1.0 + 1.0e-4
    torn[:, 0] *= 1.0 + 4.5e-4  # past the critical stretch of some points
    torn[:, 1] *= 1.0 - 1.0e-4
    calm, torn = calm.ravel(), torn.ravel()
    with _context(w, precision, material) as ctx:
        intact = np.zeros(ctx.num_bonds())
        ctx.set_bond_damage(intact)

        def check(y, committed):
            f = ctx.compute_force(y)
            ref = _once(w, precision, material, y, committed)
            bd = ctx.field("Bond_Damage")
            assert np.array_equal(f, ref[0]) and np.array_equal(bd, ref[1])
            assert np.array_equal(ctx.field("Damage"), ref[2])
            return bd

        assert not check(calm, intact).any()
        check(calm, intact)
        broken = check(torn, intact)
        assert 0 < broken.sum() < broken.size
        assert not check(calm, intact).any()  # the breaks were not committed
        check(calm, intact)
        ctx.update_state()  # commits an evaluation that broke nothing
        check(torn, intact)
        ctx.update_state()
        for _ in range(2):
            assert np.array_equal(check(calm, broken), broken)
            ctx.update_state()
        some = broken * (np.arange(broken.size) % 2)
        ctx.set_bond_damage(some)
        check(calm, some)
        ctx.set_bond_damage(intact)
        check(calm, intact)
        # time steps write the committed damage between evaluations
        ctx.set_state(torn - w["x"], np.zeros_like(torn))
        ctx.verlet_run(1.0e-9, 3)
        after = ctx.field("Bond_Damage")
        assert after.any()
        check(calm, after)
        check(calm, after)
