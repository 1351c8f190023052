"""The conjugate-gradient loop that keeps its scalars on the device.

* Tangent products of both lane counts (32 lanes per point up to 4096 points,
  8 above: 16^3 is the last of the one, 17x31x8 = 4216 is of the other) against
  the oracle's linearization: 1e-11 relative, the bound of the tangent tests.
* The iteration limit: CG stops at exactly max_cg iterations although the host
  runs ahead of the device, and the solution is the limited one, not a later
  iterate: a second solve with the same limit repeats it bit for bit.
* A converged load step leaves a force residual below the Newton tolerance.
* A point without bonds, and a page that cannot be had, change nothing.
"""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

from oracle import oracle as O
from peridigm_b200 import Context, PDError, _lib, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(7, 6, 5), (16, 16, 16), (17, 31, 8), (32, 32, 16), (33, 31, 17)])
def test_tangent_product_of_both_lane_counts(dims):
    x, vol = workloads.lattice(*dims, 1.0e-3, jitter=0.05, seed=2)
    h, K, mu = 3.015e-3, 130.0e9, 78.0e9
    rng = np.random.default_rng(5)
    u, w = rng.normal(0, 1e-6, x.size), rng.normal(0, 1.0, x.size)
    row, col = O.neighbor_search(x, h)
    ref = -np.repeat(vol, 3) * O.lps_jv(x, x + u, vol, row, col, K, mu, h, w)
    with Context(precision="fp64") as ctx:
        ctx.set_points(x, vol)
        ctx.set_horizons([h])
        ctx.build_bonds()
        ctx.material(K, mu, 7800.0)
        kw = ctx.jacobian_apply(u, w)
    assert np.linalg.norm(kw - ref) <= 1e-11 * np.linalg.norm(ref)


def _step(ctx, precond, max_cg, max_newton, tol):
    st = _lib.Stats()
    ctx.set_state(np.zeros(3 * ctx.n), np.zeros(3 * ctx.n))
    try:
        ctx.qs_load_step(0.0, 0.05, newton_tolerance=tol, cg_relative_tolerance=1e-12, max_newton=max_newton,
                         max_cg=max_cg, preconditioner=precond, use_predictor=False, stats=st)
    except PDError as e:
        assert "Newton" in str(e)
    return st, ctx.field("Displacement")


@pytest.mark.parametrize("precond,modes,n", [("none", 3, 13), ("block_jacobi", 3, 8), ("block_jacobi", 3, 13),
                                             ("block_jacobi", 3, 18), ("two_level", 3, 13), ("two_level", 6, 13)])
def test_iteration_limit_and_convergence(precond, modes, n):
    """13^3 points and fewer: one launch for the solve (without a coarse level); 18^3: the launch-by-launch loop."""
    w = workloads.qs_cube(n=n, jitter=0.05, load_steps=4)
    with Context(precision="fp64") as ctx:
        workloads.setup_context(ctx, w)
        ctx.coarse_modes(modes)
        for limit in (1, 2, 7):
            st, u = _step(ctx, precond, limit, 1, -1e-12)
            assert st.newton_iterations == 1 and st.cg_iterations == limit
            st, u2 = _step(ctx, precond, limit, 1, -1e-12)
            assert st.cg_iterations == limit and np.array_equal(u, u2)
        st, u = _step(ctx, precond, 4000, 20, -1e-9)
        f = ctx.field("Force_Density") * np.repeat(w["vol"], 3)
    free = np.ones(len(f), bool)
    for bc in w["bcs"]:
        free[3 * bc["points"] + bc["coordinate"]] = False
    row, col = O.neighbor_search(w["x"], w["horizon"])
    start = np.zeros(len(f))  # the prescribed increment alone: the scale of a relative tolerance
    for bc in w["bcs"]:
        start[3 * bc["points"] + bc["coordinate"]] = 0.05 * bc["a"]
    r0 = O.eval_model(w["x"], w["x"] + start, w["vol"], row, col, w["K"], w["mu"], w["horizon"])["force"]
    r0 = (r0 * np.repeat(w["vol"], 3))[free]
    metric = lambda r: np.linalg.norm(r) + 20.0 * np.abs(r).max()  # noqa: E731
    assert metric(f[free]) <= 1.01e-9 * metric(r0)


@pytest.mark.parametrize("n", [8, 18])
def test_a_point_without_bonds_does_not_reach_the_solve(n):
    """Nothing of its 0/0 owner constants enters a product: the load step is that
    of the body alone (8^3: one launch; 18^3: launch by launch)."""
    w = workloads.qs_cube(n=n, jitter=0.05, load_steps=4)
    alone = np.concatenate([w["x"], w["x"].max() + np.array([1.0, 1.0, 1.0])])
    got = []
    for x in (w["x"], alone):
        w2 = dict(w, x=x, vol=np.full(x.size // 3, w["vol"][0]), v0=np.zeros_like(x))
        with Context(precision="fp64") as ctx:
            workloads.setup_context(ctx, w2)
            st, u = _step(ctx, "none", 4000, 20, -1e-9)
            assert st.newton_iterations > 0
            got.append((st.cg_iterations, u[:w["x"].size]))
    assert np.isfinite(got[1][1]).all() and abs(got[0][0] - got[1][0]) <= 0.02 * got[0][0]
    assert np.linalg.norm(got[0][1] - got[1][1]) <= 1e-7 * np.linalg.norm(got[0][1])


def test_a_solve_without_a_page_to_report_through(tmp_path):
    """The page cannot be had (an allocation that fails, preloaded): the host reads the solve's record instead."""
    here = os.path.dirname(os.path.abspath(__file__))
    so = str(tmp_path / "no_page.so")
    subprocess.run(["gcc", "-O1", "-fPIC", "-shared", os.path.join(here, "no_page.c"), "-o", so], check=True)
    body = """
        import os
        import numpy as np
        from peridigm_b200 import Context, PDError, workloads

        w = workloads.qs_cube(n=18, jitter=0.05, load_steps=4)
        for precond in ("none", "two_level"):
            got = []
            for page in (True, False):
                os.environ.pop("PD_TEST_NO_PAGE", None)
                with Context(precision="fp64") as ctx:
                    workloads.setup_context(ctx, w)
                    if not page:
                        os.environ["PD_TEST_NO_PAGE"] = "1"
                    st = ctx.qs_load_step(0.0, 0.25, newton_tolerance=-1e-9, preconditioner=precond,
                                          use_predictor=False)
                    its, u = st.cg_iterations, ctx.field("Displacement")
                    try:  # a limit: exactly so many iterations
                        ctx.qs_load_step(0.25, 0.5, newton_tolerance=-1e-12, max_newton=1, max_cg=7,
                                         preconditioner=precond, use_predictor=False, stats=st)
                    except PDError as e:
                        assert "Newton" in str(e), e
                    assert st.cg_iterations == its + 7
                    got.append((its, u, ctx.field("Displacement")))
            assert got[0][0] == got[1][0]
            assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])
    """
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(body)], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(here), env=dict(os.environ, LD_PRELOAD=so))
    assert r.returncode == 0, r.stdout + r.stderr
