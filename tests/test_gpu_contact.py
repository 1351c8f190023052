"""GPU short-range contact against the reference's gold file and the oracle.

* Contact_2x1x1 gold (test/verification/Contact_2x1x1): displacement and
  velocity to 1e-13 absolute (Contact_2x1x1.comp), FP64 and split paths.
* contact search + force drop-in (pd_contact_force) vs the oracle on a
  deformed two-body configuration, with and without friction: pair lists
  identical, force relative error <= 1e-12 (FP64 arithmetic in both).
* plate + sphere explicit run with contact and damage vs the oracle explicit
  run (FP64: displacement relative error <= 1e-9, identical bond damage).
"""
import os

import numpy as np
import pytest

from oracle import oracle as O
from peridigm_b200 import Context, workloads

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")


@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_contact_2x1x1_gold(precision):
    z = np.load(os.path.join(G, "contact_2x1x1.npz"))
    rho, K, mu, h, rs, fq, rc, ks, dt, T = z["params"]
    with Context(precision=precision) as ctx:
        ctx.set_points(z["x"].ravel(), z["vol"])
        ctx.set_horizons([h])
        ctx.set_bonds(z["nl"])
        ctx.material(K, mu, rho)
        ctx.contact(rs, int(fq), rc, ks)
        ctx.set_state(np.zeros(6), z["v0"])
        for k in range(10):
            st = ctx.verlet_run(dt, 100, t0=k * 100 * dt)
            u, v = ctx.field("Displacement"), ctx.field("Velocity")
            tol = 1e-13 if precision == "fp64" else 1e-11  # split: y = x + u rounds differently
            assert np.abs(u[0::3] - z["disp_x"][k + 1]).max() < tol
            assert np.abs(v[0::3] - z["vel_x"][k + 1]).max() < tol
        assert st["contact_pairs"] == 2


@pytest.mark.parametrize("friction", [0.0, 0.3])
def test_contact_force_dropin_matches_oracle(friction):
    # bodies a horizon apart when bonded, then the sphere pushed 0.4h into the plate
    w = workloads.plate_sphere(nx=16, ny=16, nz=4, h=1.0e-3, radius_cells=3, gap_cells=3.5)
    n = len(w["vol"])
    rng = np.random.default_rng(2)
    y = w["x"] + rng.normal(0, 0.05e-3, size=w["x"].size)
    y[2::3][w["block"] == 1] -= 3.9e-3
    v = rng.normal(0, 1.0, size=w["x"].size)
    ct = w["contact"]
    with Context(precision="fp64") as ctx:
        ctx.set_points(w["x"], w["vol"], w["block"])
        ctx.set_horizons([w["horizon"]] * 2)
        ctx.build_bonds()
        ctx.material(w["K"], w["mu"], w["rho"], block=0)
        ctx.material(w["K"], w["mu"], w["rho"], block=1)
        ctx.contact(ct["r_search"], ct["freq"], ct["r_contact"], ct["k_spring"], friction)
        fc = ctx.contact_force(y, v)
        row, col = ctx.bonds_csr()
    crow, ccol = O.contact_search(y, ct["r_search"], row, col)
    assert len(ccol) > 0
    ref = O.contact_force(y, v, w["vol"], crow, ccol, ct["r_contact"], ct["k_spring"], w["horizon"], friction)
    assert np.abs(ref).max() > 0
    assert np.linalg.norm(fc - ref) <= 1e-12 * np.linalg.norm(ref)


def test_plate_sphere_explicit_matches_oracle():
    w = workloads.plate_sphere(nx=20, ny=20, nz=4, h=1.0e-3, radius_cells=4, s_c=1e-2, speed=150.0,
                               gap_cells=3.2, freq=5)
    nsteps = 300
    with Context(precision="fp64") as ctx:
        workloads.setup_context_blocks(ctx, w)
        dt = 0.7 * ctx.critical_time_step()
        row, col = ctx.bonds_csr()
        st = ctx.verlet_run(dt, nsteps)
        u, v, bd = ctx.field("Displacement"), ctx.field("Velocity"), ctx.field("Bond_Damage")
    assert st["contact_pairs"] > 0
    ref = O.explicit_run(workloads.oracle_problem_blocks(w, row, col, dt, nsteps), np.zeros_like(w["x"]), w["v0"])
    sphere = w["block"] == 1
    assert ref["v"][2::3][sphere].mean() > -140.0, "the sphere must have been slowed by contact"
    assert ref["bond_damage"].sum() < len(col)
    assert np.array_equal(bd, ref["bond_damage"])
    assert np.abs(u - ref["u"]).max() <= 1e-9 * np.abs(ref["u"]).max()
    assert np.abs(v - ref["v"]).max() <= 1e-9 * np.abs(ref["v"]).max()


@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_contact_force_of_points_that_left_the_list_is_zero(precision):
    """Only the points with a pair are visited: a call with other coordinates
    (two bodies far apart, an empty list) between steps leaves no force behind."""
    h = 1.0e-3
    xa, va = workloads.lattice(4, 4, 3, h)
    xb, vb = workloads.lattice(4, 4, 3, h, origin=(0.0, 0.0, 6.6 * h))
    x, vol = np.concatenate([xa, xb]), np.concatenate([va, vb])
    block = np.repeat([0, 1], len(va)).astype(np.int32)
    u = np.zeros_like(x)
    u[xa.size + 2::3] = -3.8 * h  # faces at 2.5 h and 7.1 h: 0.8 h apart
    with Context(precision=precision) as ctx:
        ctx.set_points(x, vol, block)
        ctx.set_horizons([3.015 * h] * 2)
        ctx.build_bonds()
        for b in (0, 1):
            ctx.material(130.0e9, 78.0e9, 7800.0, block=b)
        ctx.contact(1.5 * h, 1000, 0.9 * h, 130.0e9)
        ctx.set_state(u, np.zeros_like(x))
        ctx.verlet_begin(1.0e-9)
        ctx.verlet_step(2)
        fc = ctx.field("Contact_Force_Density").reshape(-1, 3)
        face = np.abs(fc[:, 2]) > 0
        assert face.sum() == 32 and np.allclose(fc[face][:, 2].sum(), 0.0, atol=1e-6 * np.abs(fc).max())
        assert not ctx.contact_force(x, np.zeros_like(x)).any()  # apart: no pair
        ctx.verlet_step(1)
        assert not ctx.field("Contact_Force_Density").any()


@pytest.mark.parametrize("precision", ["split", "fp64"])
@pytest.mark.parametrize("dims,search", [((9, 8, 7), 1.5), ((9, 8, 7), 3.4), ((31, 29, 26), 2.2), ((31, 29, 26), 3.4),
                                         ((36, 36, 36), 3.4)])
def test_every_point_in_many_pairs(dims, search, precision):
    """Points of one lattice bonded to their nearest neighbors alone: the pairs of either width of the search, few and
    many points, short and long runs of cells, and enough pairs that the coordinates are formed once. The steps'
    contact force is that of contact_force on the same coordinates, whose pairs a k-d tree counts."""
    from scipy.spatial import cKDTree

    h = 1.0e-3
    x, vol = workloads.lattice(*dims, h, jitter=0.03, seed=1)
    v = np.random.default_rng(2).normal(0.0, 1.0, x.size)
    with Context(precision=precision) as ctx:
        ctx.set_points(x, vol)
        ctx.set_horizons([1.3 * h])
        ctx.build_bonds()
        ctx.material(130.0e9, 78.0e9, 7800.0)
        ctx.contact(search * h, 0, search * h, 1.0, 0.2)
        fc = ctx.contact_force(x, v)
        ctx.set_state(np.zeros_like(x), v)
        st = ctx.verlet_run(1.0e-9, 0)
        pairs = 2 * len(cKDTree(x.reshape(-1, 3)).query_pairs(search * h))
        assert st["contact_pairs"] == pairs - ctx.num_bonds()
        assert np.linalg.norm(ctx.field("Contact_Force_Density") - fc) <= 1e-12 * np.linalg.norm(fc)
        assert np.count_nonzero(np.abs(fc.reshape(-1, 3)).max(1)) == vol.size
    # the sum of V f over all points vanishes: every pair's two halves are there
    total = (fc.reshape(-1, 3) * vol[:, None]).sum(0)
    assert np.abs(total).max() <= 1e-9 * (np.abs(fc.reshape(-1, 3)) * vol[:, None]).sum()
