"""Performance cases: what a program that uses this framework has it do, at the
sizes, precisions and options it is used with.

Every case is a jittered lattice (spacing H, horizon 3.015 H) with the
materials, damage, notch, contact and boundary conditions of the benchmark
configurations, in a state met in mid-run: strained close to the critical
stretch, with smooth displacement and velocity waves. One pass is one of

* ``run``: ``verlet_run`` of some steps, then the output fields on the host,
  as a program does between two output times;
* ``steps``: ``verlet_step`` of some steps, then ``pack_state`` of the points
  into a device tensor, as a slab's rank or an in-situ reader does;
* ``force_device`` / ``force_host``: one model evaluation at given coordinates
  (``Material::computeForce`` of a host code), the host one with the state
  update that follows it;
* ``quasi_static``: two load steps from the unloaded state, then the
  displacement.

State advances from pass to pass in ``run`` and ``steps``, as it does in a
simulation; the other two kinds repeat the same work.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from peridigm_b200 import Context

H = 0.5e-3            # lattice spacing
HORIZON = 3.015 * H
JITTER = 0.05         # of the spacing, each coordinate
K0, RHO = 130.0e9, 7800.0
SC_LO, SC_HI = 3.0e-4, 6.0e-4   # critical stretch, uniform per point
SC = 5.0e-4                     # critical stretch of a body with one material
PULL = 0.25                     # m/s at the gripped layers
SPHERE_SPEED = 20.0
SEARCH_EVERY = 100
R_CONTACT, R_SEARCH = 0.9 * H, 1.5 * H
QS_SHEAR = 0.6
QS_TIMES = (0.0, 0.05, 0.1)
QS_PULL = 1.0e-4


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def _case(name, kind, precision, nx, ny, nz, **kw):
    c = dict(name=name, kind=kind, precision=precision, nx=nx, ny=ny, nz=nz, steps=1, material="lps",
             field=False, s_c=0.0, notch=False, sphere=0, preconditioner="")
    c.update(kw)
    return c


def listed():
    return [
        # a verification deck (some hundred to a few thousand points), FP64 in the reference's order:
        # launches and latency are all of it
        _case("deck_fp64", "run", "fp64", 27, 7, 6, steps=50),
        # the elastic wave in a bar, 100x10x10, at the library's default precision
        _case("bar_split", "run", "split", 100, 10, 10, steps=50),
        # the notched plate in tension, bonds breaking, output every 100 steps
        _case("notched_plate_split", "run", "split", 400, 200, 4, steps=100, s_c=SC, notch=True),
        # a heterogeneous plate of 4 million points, every bond with two critical stretches: the
        # production run, and the largest case
        _case("plate_split_large", "steps", "split", 250, 200, 80, steps=10, field=True, s_c=-1.0),
        # the same material in FP64 on the sliced bond stream
        _case("plate_fp64_sliced", "steps", "fp64_sliced", 160, 160, 40, steps=10, field=True, s_c=-1.0),
        # a ragged plate in the reference's FP64 operation order, damage on
        _case("plate_fp64", "run", "fp64", 131, 97, 21, steps=20, s_c=SC),
        # a plate hit by a sphere: contact search and forces beside the bond passes
        _case("plate_sphere_split", "run", "split", 200, 200, 20, steps=100, s_c=SC, sphere=15),
        # the bond-based material on a thin ragged plate
        _case("bond_based_split", "steps", "split", 257, 129, 9, steps=20, s_c=SC, material="bond_based"),
        # a host code on the GPU that asks for the force density at its coordinates
        _case("force_device_split", "force_device", "split", 101, 83, 37, field=True, s_c=-1.0),
        # the same through host buffers, with the damage committed: the drop-in call
        _case("force_host_split", "force_host", "split", 160, 160, 40, field=True, s_c=-1.0),
        # quasi-static load steps of the tensile cube, aggregate (rigid) two-level preconditioner
        _case("qs_cube_two_level", "quasi_static", "fp64", 60, 60, 60, preconditioner="two_level"),
        # the same of a small specimen with the reference's 3x3 block-Jacobi preconditioner
        _case("qs_bar_block_jacobi", "quasi_static", "fp64", 37, 11, 11, preconditioner="block_jacobi"),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "steps", "steps", "force_device", "force_host", "quasi_static"])
    precision = rng.choice(["split", "split", "fp64", "fp64_sliced"])
    top = {"split": 2.0e6, "fp64": 4.0e5, "fp64_sliced": 1.0e6}[precision]
    if kind == "quasi_static":
        precision, top = "fp64", 1.2e5
    points = math.exp(rng.uniform(math.log(1.0e3), math.log(top)))
    # aspect ratios from a bar to a plate to a cube, each at least 6 points thick
    # (a plate down to 4), odd sizes as they fall
    a, b = math.exp(rng.uniform(0.0, 1.6)), math.exp(rng.uniform(0.0, 1.0))
    side = (points / (a * b)) ** (1.0 / 3.0)
    nz = max(4 if kind != "quasi_static" else 8, int(round(side / 1.5)))
    ny = max(6 if kind != "quasi_static" else 8, int(round(math.sqrt(points * b / (a * nz)))))
    nx = max(12, int(round(points / (ny * nz))))
    if kind == "quasi_static":
        return _drawn(kind, precision, min(nx, 6 * ny), ny, nz, rng.choice(["two_level", "block_jacobi"]))
    nb = _bonds(nx, ny, nz)
    steps = max(5, min(50, int(2.0e9 / nb))) if kind in ("run", "steps") else 1
    s_c = rng.choice([0.0, SC, -1.0])
    material = "bond_based" if precision == "split" and rng.random() < 0.2 else "lps"
    return _drawn(kind, precision, nx, ny, nz, "", steps=steps, s_c=s_c, field=s_c < 0.0 and material == "lps",
                  material=material, notch=s_c > 0.0 and rng.random() < 0.5)


def _drawn(kind, precision, nx, ny, nz, preconditioner, **kw):
    c = _case("", kind, precision, nx, ny, nz, preconditioner=preconditioner, **kw)
    del c["name"]
    return c


# --------------------------------------------------------------------------
# the problem of a case: host arrays made from the seed alone
# --------------------------------------------------------------------------
def _lattice(nx, ny, nz, gen):
    x = torch.empty((nz, ny, nx, 3), dtype=torch.float64, device="cuda")  # x fastest
    at = lambda m: (torch.arange(m, dtype=torch.float64, device="cuda") + 0.5) * H  # noqa: E731
    x[..., 0], x[..., 1], x[..., 2] = at(nx), at(ny)[:, None], at(nz)[:, None, None]
    x += (2.0 * torch.rand(x.shape, dtype=torch.float64, device="cuda", generator=gen) - 1.0) * (JITTER * H)
    return x.view(-1, 3)


def _sphere(case):
    """Lattice points of the sphere over the middle of the plate, three and a half spacings above it."""
    r = case["sphere"]
    k = np.arange(-r, r + 1)
    g = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)[:, ::-1]
    g = g[(g * g).sum(1) <= r * r]
    centre = np.array([case["nx"] * H / 2, case["ny"] * H / 2, (case["nz"] - 0.5 + r + 3.5) * H])
    return g, g * H + centre


def _problem(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    quasi = case["kind"] == "quasi_static"
    x = _lattice(nx, ny, nz, gen)
    n0 = len(x)
    block = None
    if case["sphere"]:
        xs = torch.from_numpy(_sphere(case)[1]).cuda()
        block = np.concatenate([np.zeros(n0, np.int32), np.ones(len(xs), np.int32)])
        x = torch.cat([x, xs])
    n = len(x)
    p = dict(n=n, n0=n0, block=block, vol=np.full(n, H ** 3))
    K = K0 * math.exp(rng.uniform(-0.5, 0.5)) if quasi else K0
    if case["field"]:
        # lognormal, cut at 4.5 standard deviations
        z = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen).clamp_(-4.5, 4.5)
        K = (K * torch.exp(0.3 * z)).cpu().numpy()
    p["K"], p["mu"] = K, QS_SHEAR * K
    p["s_c"] = case["s_c"] if case["s_c"] > 0.0 else None
    if case["s_c"] < 0.0:
        r = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
        p["s_c"] = (SC_LO + (SC_HI - SC_LO) * r).cpu().numpy()
    # a time step below the stable one of the stiffest point
    stiff = K0 * (math.exp(0.3 * 4.5) if case["field"] else 1.0)
    p["dt"] = 0.6 * HORIZON * math.sqrt(RHO / (18.0 * stiff))
    col = np.arange(n0) % nx
    row = np.arange(n0) // nx % ny
    p["bcs"] = []
    u, v = torch.zeros_like(x), torch.zeros_like(x)
    if quasi:
        left, right = np.nonzero(col < 3)[0], np.nonzero(col >= nx - 3)[0]
        p["bcs"] = [(left, c, 0.0, 0.0) for c in range(3)] + [(right, 0, QS_PULL * nx / 60.0, 0.0)]
    else:
        axis = 1 if case["notch"] else 0
        # bonds break where the waves, the notch or the sphere add to it, not in the whole body at once
        strain = 0.72 * SC_LO if case["s_c"] < 0.0 else 0.55 * SC
        L = np.array([nx, ny, nz]) * H
        moving = case["kind"] in ("run", "steps")
        u[:n0, axis] = strain * (x[:n0, axis] - L[axis] / 2)
        for _ in range(3):  # smooth waves: strains of a few 1e-5, velocities below 1 m/s
            k = rng.integers(1, 4, 3) * np.pi / np.maximum(L, 24 * H)
            wave = torch.sin(x[:n0] @ torch.from_numpy(k).cuda() + rng.uniform(0.0, 2 * np.pi))
            for c in range(3):
                u[:n0, c] += wave * (rng.uniform(-1.0, 1.0) * 2.0e-5 / np.linalg.norm(k))
                v[:n0, c] += wave * rng.uniform(-0.2, 0.2)
        if case["sphere"]:  # the sphere has just reached the plate
            u[n0:, 2] = u[:n0, 2].max() - (3.5 - 0.88) * H
            v[n0:, 2] = -SPHERE_SPEED * rng.uniform(0.9, 1.0)
        elif case["s_c"] != 0.0 and moving:
            at, m = (row, ny) if axis == 1 else (col, nx)
            p["bcs"] = [(np.nonzero(at >= m - 3)[0], axis, PULL, 0.5 * strain * L[axis]),
                        (np.nonzero(at < 3)[0], axis, -PULL, -0.5 * strain * L[axis])]
            for pts, c, a, b in p["bcs"]:
                pts = torch.from_numpy(pts).cuda()
                u[pts, c], v[pts, c] = b, a
    p["x"], p["u"], p["v"] = x.cpu().numpy(), u.cpu().numpy(), v.cpu().numpy()
    return p


def _planes(case):
    if not case["notch"]:
        return []
    y = case["ny"] // 2 * H
    return [dict(normal=(0.0, 1.0, 0.0), lower_left=(-H, y, -H), bottom_unit=(1.0, 0.0, 0.0),
                 bottom_length=(case["nx"] // 8 + 1) * H, side_length=(case["nz"] + 2) * H)]


# --------------------------------------------------------------------------
# what a program has in hand, and one pass
# --------------------------------------------------------------------------
def prepare(case, seed):
    p = _problem(case, seed)
    device = torch.cuda.current_device()
    ctx = Context(device=device, precision=case["precision"])
    ctx.set_points(p["x"], p["vol"], p["block"])
    blocks = 1 if p["block"] is None else 2
    ctx.set_horizons([HORIZON] * blocks)
    ctx.build_bonds(_planes(case))
    for b in range(blocks):
        if case["material"] == "bond_based":
            ctx.material_bond_based(K0, RHO, block=b)
        elif np.ndim(p["K"]):
            ctx.material(K0, QS_SHEAR * K0, RHO, block=b)
        else:
            ctx.material(p["K"], p["mu"], RHO, block=b)
    if np.ndim(p["K"]):
        ctx.material_field(p["K"], p["mu"])
    if p["s_c"] is not None:
        if np.ndim(p["s_c"]):
            ctx.critical_stretch(0.0)
            ctx.critical_stretch_field(p["s_c"])
        else:
            ctx.critical_stretch(p["s_c"], block=0)  # the sphere, where there is one, does not break
    if case["sphere"]:
        ctx.contact(R_SEARCH, SEARCH_EVERY, R_CONTACT, K0)
    for pts, c, a, b in p["bcs"]:
        ctx.prescribed_displacement(pts, c, a, b)
    state = dict(case=case, ctx=ctx, dt=p["dt"], t=0.0)
    if case["kind"] == "quasi_static":
        state["zero"] = np.zeros(3 * p["n"])
        if case["preconditioner"] == "two_level":
            ctx.coarse_modes(6)
        return state
    if case["kind"] in ("force_device", "force_host"):
        y = np.ascontiguousarray((p["x"] + p["u"]).ravel())
        state["y"] = torch.from_numpy(y).cuda() if case["kind"] == "force_device" else y
        ctx.set_state(np.zeros(3 * p["n"]), np.zeros(3 * p["n"]))
        if case["kind"] == "force_device":
            state["f"] = torch.empty(3 * p["n"], dtype=torch.float64, device="cuda")
        return state
    ctx.set_state(p["u"], p["v"])
    if case["kind"] == "steps":
        state["idx"] = torch.arange(p["n"], dtype=torch.int32, device="cuda")
        state["out"] = torch.empty((p["n"], 6), dtype=torch.float64, device="cuda")
        ctx.verlet_begin(p["dt"], 0.0)
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "run":
        ctx.verlet_run(state["dt"], case["steps"], state["t"])
        state["t"] += case["steps"] * state["dt"]
        out = {"u": ctx.field("Displacement"), "v": ctx.field("Velocity")}
        if case["s_c"] != 0.0:
            out["damage"] = ctx.field("Damage")
        return out
    if kind == "steps":
        ctx.verlet_step(case["steps"])
        ctx.pack_state(state["idx"], state["out"])
        return {"u": state["out"][:, :3], "y": state["out"][:, 3:]}
    if kind == "force_device":
        ctx.compute_force_device(state["y"].data_ptr(), state["f"].data_ptr())
        return state["f"]
    if kind == "force_host":
        f = ctx.compute_force(state["y"])
        ctx.update_state()
        return f
    ctx.set_state(state["zero"], state["zero"])
    st = None
    for t0, t1 in zip(QS_TIMES, QS_TIMES[1:]):
        st = ctx.qs_load_step(t0, t1, newton_tolerance=-1e-8, cg_relative_tolerance=1e-8,
                              preconditioner=case["preconditioner"], stats=st)
    return ctx.field("Displacement")


def _bonds(nx, ny, nz):
    """Directed bonds of the lattice without its jitter."""
    o = _offsets(9)
    return int(sum(max(0, nx - abs(a)) * max(0, ny - abs(b)) * max(0, nz - abs(c)) for a, b, c in o))


def work(case):
    """Bytes and operations of one pass. A step (or evaluation) reads each bond's neighbor id (4 B), damage
    (1 B) and reference bond vector (three numbers of the bond arithmetic's type) once, and reads and writes
    each point's state once: coordinates, volume, material and critical stretch (72 B), displacement and
    velocity in and out (96 B), acceleration or force density out (24 B). Some 70 operations per bond and step
    (45 for the bond-based material). A quasi-static pass reads, per CG iteration, each bond's id and the
    reference bond vector in FP64 and some ten vectors of the points; the iterations of a load step grow with the
    length of the body under block Jacobi (about 2.5 per point of it) and not under the two-level
    preconditioner (about 40), over two Newton steps."""
    n = case["nx"] * case["ny"] * case["nz"]
    nb = _bonds(case["nx"], case["ny"], case["nz"])
    if case["sphere"]:
        m = len(_sphere(case)[0])
        n, nb = n + m, nb + 110 * m
    if case["kind"] == "quasi_static":
        its = (len(QS_TIMES) - 1) * (40 if case["preconditioner"] == "two_level" else int(2.5 * max(
            case["nx"], case["ny"], case["nz"])))
        return {"bytes": its * (28 * nb + 240 * n), "flops": its * (50 * nb + 60 * n)}
    real = 4 if case["precision"] == "split" else 8
    steps = case["steps"]
    return {"bytes": steps * ((5 + 3 * real) * nb + 192 * n),
            "flops": steps * ((45 if case["material"] == "bond_based" else 70) * nb + 30 * n)}


# --------------------------------------------------------------------------
# the same in plain torch, 64 bits
# --------------------------------------------------------------------------
def _offsets(r2):
    k = np.arange(-3, 4)
    g = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
    d = (g * g).sum(1)
    return [tuple(int(q) for q in o) for o in g[(d > 0) & (d <= r2)]]


class _Body:
    """Points, families and LPS or bond-based forces, padded rows of neighbors in chunks of points."""

    def __init__(self, case, p):
        dev = "cuda"
        self.case, self.p, self.n = case, p, p["n"]
        self.x = torch.from_numpy(p["x"]).to(dev)
        self.vol = torch.from_numpy(p["vol"]).to(dev)
        full = lambda v: torch.full((self.n,), float(v), dtype=torch.float64, device=dev)  # noqa: E731
        per = lambda v: torch.from_numpy(v).to(dev) if np.ndim(v) else full(v)  # noqa: E731
        self.K, self.mu = per(p["K"]), per(p["mu"])
        self.sc = None if p["s_c"] is None else per(p["s_c"]).clone()
        if self.sc is not None and case["sphere"]:
            self.sc[p["n0"]:] = math.inf
        self._families()
        width = self.idx.shape[1]
        self.chunks = [(a, min(self.n, a + max(1, (1 << 25) // width)))
                       for a in range(0, self.n, max(1, (1 << 25) // width))]
        self.own = torch.zeros(self.idx.shape, dtype=torch.bool, device=dev)   # broken: this row's half
        self.part = torch.zeros(self.idx.shape, dtype=torch.bool, device=dev)  # and the partner's
        self.m = torch.empty(self.n, dtype=torch.float64, device=dev)
        for a, b in self.chunks:
            j, live = self._row(a, b)
            X = self.x[j] - self.x[a:b, None]
            self.m[a:b] = ((X * X).sum(-1) * self.vol[j] * live).sum(1)

    def _grids(self):
        """(id of the point at each lattice site, -1 where there is none; site of each point) of each body."""
        case = self.case
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        q = torch.arange(nx * ny * nz, device="cuda")
        yield 0, q.view(nz, ny, nx), torch.stack([q % nx, q // nx % ny, q // (nx * ny)], 1)
        if case["sphere"]:
            r = case["sphere"]
            site = torch.from_numpy(np.ascontiguousarray(_sphere(case)[0] + r)).cuda()
            ids = torch.full((2 * r + 1,) * 3, -1, dtype=torch.int64, device="cuda")
            ids[site[:, 2], site[:, 1], site[:, 0]] = torch.arange(len(site), device="cuda") + self.p["n0"]
            yield self.p["n0"], ids, site

    def _families(self):
        offs = _offsets(10)
        idx = torch.full((self.n, len(offs)), -1, dtype=torch.int32, device="cuda")
        at = torch.zeros(self.n, dtype=torch.int64, device="cuda")
        planes = _planes(self.case)
        for first, ids, site in self._grids():
            dims = torch.tensor([ids.shape[2], ids.shape[1], ids.shape[0]], device="cuda")
            i = torch.arange(first, first + len(site), device="cuda")
            for o in offs:
                s = site + torch.tensor(o, device="cuda")
                inside = ((s >= 0) & (s < dims)).all(1)
                s = torch.where(inside[:, None], s, 0)
                j = torch.where(inside, ids[s[:, 2], s[:, 1], s[:, 0]], -1)
                ok = j >= 0
                xi, xj = self.x[i], self.x[j.clamp_min(0)]
                d = xj - xi
                ok &= d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2] <= HORIZON * HORIZON
                for pl in planes:
                    t = (pl["lower_left"][1] - xi[:, 1]) / torch.where(d[:, 1] == 0, 1e-300, d[:, 1])
                    w = xi[:, 0] + t * d[:, 0] - pl["lower_left"][0]
                    ok &= ~((t >= 0) & (t <= 1) & (w > 0) & (w < pl["bottom_length"]))
                rows = i[ok]
                idx[rows, at[rows]] = j[ok].to(torch.int32)
                at[rows] += 1
        self.count = at
        self.idx = idx[:, :int(at.max())].contiguous()

    def _row(self, a, b):
        j = self.idx[a:b].long()
        live = j >= 0
        return j.clamp_min(0), live

    def _bond(self, a, b, u):
        j, live = self._row(a, b)
        X = self.x[j] - self.x[a:b, None]
        d = u[j] - u[a:b, None]
        zeta = X.square().sum(-1).sqrt()
        # |Y| - |X| from the displacement difference, without cancellation
        num = 2.0 * (X * d).sum(-1) + d.square().sum(-1)
        Y = X.add_(d)
        lenY = Y.square().sum(-1).sqrt()
        e = num / (lenY + zeta)
        zeta = torch.where(live, zeta, 1.0)
        lenY = torch.where(live, lenY, 1.0)
        return j, live, Y, lenY, zeta, torch.where(live, e, 0.0)

    def _breaks(self, a, b, j, live, zeta, e, own, part):
        if self.sc is None:
            return
        s = e / zeta
        own[a:b] |= (s > self.sc[a:b, None]) & live
        part[a:b] |= (s > self.sc[j]) & live

    def force(self, u, commit=True):
        """Internal force density at displacement u [n, 3]; bonds past their critical stretch break first."""
        own, part = (self.own, self.part) if commit else (self.own.clone(), self.part.clone())
        f = torch.empty_like(u)
        if self.case["material"] == "bond_based":
            c = 18.0 * self.K / (math.pi * HORIZON ** 4)
            for a, b in self.chunks:
                j, live, Y, lenY, zeta, e = self._bond(a, b, u)
                self._breaks(a, b, j, live, zeta, e, own, part)
                t = 0.5 * (e / zeta) * (c[a:b, None] * ~own[a:b] + c[j] * ~part[a:b])
                f[a:b] = (Y * (t * self.vol[j] * live / lenY)[..., None]).sum(1)
            return f
        theta = torch.empty(self.n, dtype=torch.float64, device=u.device)
        for a, b in self.chunks:
            j, live, Y, lenY, zeta, e = self._bond(a, b, u)
            self._breaks(a, b, j, live, zeta, e, own, part)
            theta[a:b] = 3.0 / self.m[a:b] * (zeta * e * self.vol[j] * (live & ~own[a:b])).sum(1)
        B = 15.0 * self.mu / self.m
        A = theta * (3.0 * self.K / self.m - B / 3.0)
        for a, b in self.chunks:
            j, live, Y, lenY, zeta, e = self._bond(a, b, u)
            t = (A[a:b, None] * zeta + B[a:b, None] * e) * ~own[a:b] + (A[j] * zeta + B[j] * e) * ~part[a:b]
            f[a:b] = (Y * (t * self.vol[j] * live / lenY)[..., None]).sum(1)
        return f

    def contact(self, u):
        """Short-range force density between the plate and the sphere."""
        f = torch.zeros_like(u)
        n0, y = self.p["n0"], self.x + u
        low = n0 + torch.nonzero(y[n0:, 2] < y[:n0, 2].max() + R_CONTACT)[:, 0]
        if not len(low):
            return f
        lo, hi = y[low, :2].min(0).values - R_CONTACT, y[low, :2].max(0).values + R_CONTACT
        near = ((y[:n0, :2] >= lo) & (y[:n0, :2] <= hi)).all(1) & (y[:n0, 2] >= y[low, 2].min() - R_CONTACT)
        near = torch.nonzero(near)[:, 0]
        for k in range(0, len(near), 4096):
            i = near[k:k + 4096]
            d = y[low][None] - y[i][:, None]
            r = d.square().sum(-1).sqrt()
            s = torch.where(r < R_CONTACT, 2.0 * 9.0 * K0 / (math.pi * HORIZON ** 5) * (R_CONTACT - r) / r, 0.0)
            g = d * s[..., None]
            f[i] -= (g * self.vol[low][None, :, None]).sum(1)
            f[low] += (g * self.vol[i][:, None, None]).sum(0)
        return f

    def total(self, u, commit=True):
        f = self.force(u, commit)
        return f + self.contact(u) if self.case["sphere"] else f

    def node_damage(self):
        return self.own.sum(1).double() / self.count.clamp_min(1)


def _verlet(body, p, steps, last):
    """Velocity Verlet: the initial evaluation (whose damage is not kept), then `steps` steps; `last`: the run
    ends with the velocity completed, else with the state advanced once more."""
    u, v = (torch.from_numpy(p[k]).cuda().clone() for k in ("u", "v"))
    dt = p["dt"]

    def advance():
        for pts, c, a, _ in bcs:
            v[pts, c] = a
        u.add_(v, alpha=dt)

    bcs = [(torch.from_numpy(pts).cuda(), c, a, b) for pts, c, a, b in p["bcs"]]
    v += 0.5 * dt / RHO * body.total(u, commit=False)
    advance()
    for s in range(steps):
        acc = body.total(u) / RHO
        v += 0.5 * dt * acc
        if s + 1 < steps or not last:
            v += 0.5 * dt * acc
            advance()
    return u, v


def _equilibrium(body, p):
    """Displacement with zero force on the free degrees of freedom at the last load (Newton, CG)."""
    free = torch.ones((body.n, 3), dtype=torch.float64, device="cuda")
    u = torch.zeros_like(free)
    for pts, c, a, _ in p["bcs"]:
        pts = torch.from_numpy(pts).cuda()
        free[pts, c] = 0.0
        u[pts, c] = a * QS_TIMES[-1]
    B = 15.0 * body.mu / body.m
    q = 3.0 * body.K / body.m - B / 3.0
    for _ in range(4):
        r = body.force(u) * body.vol[:, None] * free
        # the tangent's bond terms at u
        geo, theta = [], torch.empty_like(body.m)
        for a, b in body.chunks:
            j, live, Y, lenY, zeta, e = body._bond(a, b, u)
            V = body.vol[j] * live
            theta[a:b] = 3.0 / body.m[a:b] * (zeta * e * V).sum(1)
            geo.append((a, b, j, Y / lenY[..., None], V, zeta, e, lenY))
        A = theta * q
        rows, block = [], torch.zeros((body.n, 3, 3), dtype=torch.float64, device="cuda")
        for a, b, j, yh, V, zeta, e, lenY in geo:
            c1 = V * zeta
            c2 = V * (zeta * (A[a:b, None] + A[j]) + (B[a:b, None] + B[j]) * e) / lenY
            c3 = V * (B[a:b, None] + B[j]) - c2
            block[a:b] = torch.einsum("nk,nki,nkj->nij", c3, yh, yh)
            block[a:b].diagonal(dim1=1, dim2=2).add_(c2.sum(1)[:, None])
            hv = (c1[..., None] * yh).sum(1)
            block[a:b] += (3.0 * q / body.m)[a:b, None, None] * hv[:, :, None] * hv[:, None, :]
            rows.append((a, b, j, yh, c1, c2, c3))
        del geo
        block *= body.vol[:, None, None]
        block = block * free[:, :, None] * free[:, None, :] + torch.diag_embed(1.0 - free)
        inv = torch.linalg.inv(block)

        def tangent(w):
            qd, out = torch.empty_like(body.m), torch.empty_like(w)
            for a, b, j, yh, c1, c2, c3 in rows:
                de = (yh * (w[j] - w[a:b, None])).sum(-1)
                qd[a:b] = (3.0 * q / body.m)[a:b] * (c1 * de).sum(1)
            for a, b, j, yh, c1, c2, c3 in rows:
                dw = w[j] - w[a:b, None]
                s = c1 * (qd[a:b, None] + qd[j]) + c3 * (yh * dw).sum(-1)
                out[a:b] = (yh * s[..., None] + dw.mul_(c2[..., None])).sum(1)
            return -out * body.vol[:, None] * free

        step, res = torch.zeros_like(u), r.clone()
        z = (inv @ res[..., None])[..., 0] * free
        d, rz, start = z.clone(), (res * z).sum(), res.norm()
        for it in range(4000):
            kd = tangent(d)
            alpha = rz / (d * kd).sum()
            step += alpha * d
            res -= alpha * kd
            if it % 16 == 0 and float(res.norm()) <= 1e-7 * float(start):
                break
            z = (inv @ res[..., None])[..., 0] * free
            new = (res * z).sum()
            d = z + (new / rz) * d
            rz = new
        u = u + step
        if float(step.norm()) <= 1e-11 * float(u.norm()):
            break
    return u


def exact(case, seed):
    p = _problem(case, seed)
    body = _Body(case, p)
    kind = case["kind"]
    if kind == "quasi_static":
        return _equilibrium(body, p).reshape(-1)
    if kind in ("force_device", "force_host"):
        u = torch.from_numpy((p["x"] + p["u"]) - p["x"]).cuda()
        return body.force(u).reshape(-1)
    if kind == "steps":
        u, _ = _verlet(body, p, case["steps"], last=False)
        return {"u": u, "y": body.x + u}
    u, v = _verlet(body, p, case["steps"], last=True)
    out = {"u": u.reshape(-1), "v": v.reshape(-1)}
    if case["s_c"] != 0.0:
        out["damage"] = body.node_damage()
    return out
