"""The FP64 passes' branch-free roots and quotients against the CPU oracle.

A batch of bonds computes |X|, |Y| and the quotients in straight-line code and
goes back to the built-in functions when an operand is outside its range
(squares below 2^-900 or above 2^900): lengths of 1e-140 and 1e140 take that
branch, lengths of 1 do not. Rows of 0, 1 and up to 90 bonds leave every
remainder of a lane group's batches. Bounds of the FP64 paths: force 1e-11 and
dilatation 1e-12 relative L2 of the oracle, bond damage identical.
"""
import numpy as np
import pytest

from oracle import oracle as O
from peridigm_b200 import Context, workloads

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("scale", [1e-140, 1.0, 1e140])
@pytest.mark.parametrize("precision,influence", [("fp64", "One"), ("fp64", "Parabolic Decay"), ("fp64_sliced", "One")])
def test_fp64_passes_at_any_scale(precision, influence, scale):
    x, _ = workloads.lattice(6, 5, 7, 1.0, jitter=0.1, seed=3)
    # one pair apart from the body, and one point with no bonds
    x = np.concatenate([x, [40.0, 40.0, 40.0, 41.0, 40.0, 40.0, 60.0, 60.0, 60.0]])
    n = x.size // 3
    rng = np.random.default_rng(4)
    u = 1e-3 * x + rng.normal(0.0, 2e-3, x.size)
    x, y = scale * x, scale * (x + u)
    vol = rng.uniform(0.5, 1.5, n)
    h = 2.6 * scale
    row, col = O.neighbor_search(x, h)
    assert set(np.diff(row)) >= {0, 1}
    inf = {"One": 0, "Parabolic Decay": 1}[influence]
    ref = O.eval_model(x, y, vol, row, col, 1.0, 0.6, h, s_c=3e-3, influence=inf)
    assert 0 < ref["bond_damage"].sum() < len(col)
    with Context(precision=precision, influence=influence) as ctx:
        ctx.set_points(x, vol)
        ctx.set_horizons([h])
        ctx.build_bonds()
        ctx.material(1.0, 0.6, 1.0)
        ctx.critical_stretch(3e-3)
        f = ctx.compute_force(y)
        th, bd = ctx.field("Dilatation"), ctx.field("Bond_Damage")
    own = np.diff(row) > 0  # (the reference's loop leaves 0/0 terms of a point without bonds out)
    assert np.array_equal(bd, ref["bond_damage"])
    assert rel_l2(th[own], ref["theta"][own]) < 1e-12
    f, fr = f.reshape(-1, 3), ref["force"].reshape(-1, 3)
    assert rel_l2(f[own], fr[own]) < 1e-11
