"""The FP64 passes' branch-free roots and quotients against the CPU oracle.

A batch of bonds computes |X|, |Y| and the quotients in straight-line code and
goes back to the built-in functions when an operand is outside its range
(squares below 2^-900 or above 2^900): lengths of 1e-140 and 1e140 take that
branch, lengths of 1 do not. Rows of 0, 1 and up to 90 bonds leave every
remainder of a lane group's batches. Bounds of the FP64 paths: force 1e-11 and
dilatation 1e-12 relative L2 of the oracle, bond damage identical.

Within the ranges that the passes test, roots and quotients have the bits of
the correctly rounded built-in functions: random operands over and past the
ranges, operands whose root or quotient lies next to the middle of two
numbers, significands of ones alone, zeros, infinities and NaN. A term that
overflows keeps the sign and the infinity that the built-in division gives.
"""
import ctypes as C

import _internals
import numpy as np
import pytest

from oracle import oracle as O
from peridigm_b200 import Context, PDError, workloads

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


def _near_middle_quotients(rng, count):
    """(a, b), a/b within some 2^-53 of a unit of the middle of two doubles: Q odd of 54 bits, Q b = r mod 2^53."""
    a, b = [], []
    for k in range(count):
        d = (1 << 52) | int(rng.integers(0, 1 << 52)) | 1
        if k % 8 == 0:
            d = (1 << 53) - 1 - 2 * int(rng.integers(0, 8))
        r = int(rng.choice([-7, -5, -3, -1, 1, 3, 5, 7]))
        Q = pow(d, -1, 1 << 54) * r % (1 << 54)
        for e in (53, 54):
            p = Q * d - r
            if Q >> 53 == 1 and p % (1 << e) == 0 and (p >> e) >> 53 == 0:
                a.append(float(p >> e))
                b.append(float(d))
    return np.array(a), np.array(b)


def _near_middle_squares(count):
    """Numbers whose root lies next to the middle of two doubles: X odd of 54 bits, X^2 = r mod 2^54."""
    out = []
    for t in range(-count // 2, count // 2):
        r = 1 + 8 * t
        x = 1
        for k in range(3, 60):  # a root of r modulo 2^60, bit by bit
            if (x * x - r) % (1 << (k + 1)):
                x += 1 << (k - 1)
        for X in {s * x % (1 << 54) for s in (1, -1)} | {(s * x + (1 << 53)) % (1 << 54) for s in (1, -1)}:
            for e in (54, 55):
                p = X * X - r
                if X >> 53 == 1 and X & 1 and p % (1 << e) == 0 and (p >> e) >> 53 == 0:
                    out.append(float(p >> e) * 2.0 ** (e % 2))
    return np.array(out)


def test_roots_and_quotients_have_the_bits_of_the_built_in_functions():
    rng = np.random.default_rng(11)
    lib = _internals.load()

    def compare(a, c):
        a, c = np.ascontiguousarray(a), np.ascontiguousarray(c)
        n = np.zeros(5, np.uint64)
        p = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
        assert lib.compare_fp64(C.c_int64(a.size), p(a), p(c), p(n)) == 0
        roots, quotients, bad_root, bad_quotient, bad_by_m = (int(k) for k in n)
        assert bad_root == 0 and bad_quotient == 0 and bad_by_m == 0
        return roots, quotients

    def random(count, top):
        m = rng.integers(0, 1 << 52, count)
        few = rng.integers(0, 40, count)
        m = np.where(few == 0, (1 << 52) - 1 - few, np.where(few == 1, few * 3, m))
        return np.ldexp(1.0 + m * 2.0 ** -52, rng.integers(-top, top + 1, count))

    n = 4_000_000
    # ordinary magnitudes: none is left to the built-in functions, bar one in 2^32
    roots, quotients = compare(random(n, 200) * rng.choice([-1.0, 1.0], n), random(n, 400))
    assert roots == n and quotients > n * 0.95
    # magnitudes over the whole range of the type, and on both sides of the limits
    compare(random(n, 1020), random(n, 1020))
    edge = lambda e: np.ldexp(random(n // 4, 0), rng.choice([-e - 1, -e, e - 1, e], n // 4))  # noqa: E731
    for e in (450, 500, 900):
        compare(edge(500), edge(e))
    # significands of ones, as root and as divisor
    ones = np.ldexp(np.float64(2.0 - 2.0 ** -52), np.arange(-200, 200))
    powers = np.ldexp(1.0, rng.integers(-200, 200, ones.size))
    compare(powers, ones * ones)
    compare(powers, ones)
    # next to the middle
    a, b = _near_middle_quotients(rng, 60_000)
    assert a.size > 10_000
    compare(a, b)
    compare(a, b * b)
    hard = _near_middle_squares(20_000)
    assert hard.size > 10_000
    assert compare(np.ones_like(hard), hard)[0] == hard.size
    # zeros, the least numbers, infinities and NaN
    special = np.array([0.0, -0.0, 5e-324, -5e-324, 2.0 ** -1042, 2.0 ** -1022, 1e308, np.inf, -np.inf, np.nan])
    A, B = np.meshgrid(special, np.concatenate([special, [1.0, 3.0, 2.0 ** 449, 2.0 ** -449]]))
    compare(A.ravel(), B.ravel())
    assert compare(np.array([0.0]), np.array([3.0])) == (1, 1)  # a zero numerator stays on the fast path


@pytest.mark.parametrize("precision", ["fp64", "fp64_sliced"])
def test_terms_that_overflow_stay_infinite(precision):
    """|Y| is in range and the products with V and the moduli are not: the built-in division gives inf, not NaN."""
    x = np.array([0.0, 0.0, 0.0, 1.0, 0.0, 0.0])
    y = np.array([0.0, 0.0, 0.0, 1.0e60, 0.0, 0.0])
    with Context(precision=precision) as ctx:
        ctx.set_points(x, np.array([1.0e260, 1.0e260]))
        ctx.set_horizons([1.5])
        ctx.build_bonds()
        ctx.material(1.0, 0.1, 1.0)
        with pytest.raises(PDError, match="NaN returned by force evaluation"):
            ctx.compute_force(y)
        theta, f = ctx.field("Dilatation"), ctx.field("Force_Density").reshape(2, 3)
    assert np.array_equal(theta, [np.inf, np.inf])
    assert np.array_equal(f[:, 0], [np.inf, -np.inf])
