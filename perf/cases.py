"""Workloads for timing the framework through its public entry points.

Six kinds of work, over the sizes that the package's own configurations (workloads.py),
tests and benchmark use:

    point    one aperture simulation: upload a pre-load from pinned host memory with
             set_particles, then K timesteps with DigitalTwinSimulator.step, reading each
             step's result.  Every pass starts from the same particles, so a pass does the
             same work however often it is repeated.
    batch    several sweep points advanced together with SweepBatch.run, after the same
             upload.
    field    the Boltzmann-electron Picard field solve alone (recalc_poisson, 5 iterations,
             as every second timestep does) for a charge density that the caller deposited.
             Consecutive passes alternate between two densities, as consecutive solves of a
             run see a changed density.
    push     the module-level push_particles_boris on the caller's CUDA tensors, one push per
             pass; the sign of dt alternates from pass to pass, so that the cloud stays where
             it is.
    deposit  the module-level accumulate_rho: ions, then electrons, onto a cleared density.
    thermal  ten sweeps of the module-level thermal_conduction between two maps.
"""
import ctypes as C
import math

import numpy as np
import torch

from thruster_cx_code_b200 import _lib
from thruster_cx_code_b200 import physics_engine as PE
from thruster_cx_code_b200 import workloads as W
from thruster_cx_code_b200.serving import SweepBatch

Q = 1.602e-19
EPS0 = 8.854e-12
M_XE = 131.293 * 1.6605e-27

# the two grid stacks of the package's workloads: (V, thickness, gap, aperture radius), mm
STACKS = {
    "2grid": dict(grids=((1000.0, 0.38, 1.0, 0.95), (-200.0, 1.0, 1.0, 0.55)), pitch_mm=3.75),
    "3grid": dict(grids=((1000.0, 0.5, 0.5, 0.8), (-250.0, 0.5, 0.5, 0.5), (0.0, 0.5, 0.5, 0.7)), pitch_mm=4.0,
                  upstream_gap_mm=0.4),
}


def listed():
    return [
        # the reference's own CPU-runnable case: 65 x 284 nodes, 100k macro-particles, with
        # heating and conduction; latency of small launches and of the small field solve
        dict(name="point_small", kind="point", stack="2grid", dx=0.025, dt=1e-10, mass_ratio=100.0, ions=80_000,
             electrons=20_000, steps=20, mode="Both"),
        # an ordinary perveance-sweep point: 130 x 568 nodes, 1M macro-particles
        dict(name="point_sweep", kind="point", stack="2grid", dx=0.0125, dt=5e-11, mass_ratio=100.0, ions=750_000,
             electrons=250_000, steps=20, mode="Erosion"),
        # the 3-grid aperture at 257 x 1025 nodes, 8M macro-particles
        dict(name="point_large", kind="point", stack="3grid", dx=0.00625, dt=2.5e-11, mass_ratio=400.0,
             ions=6_000_000, electrons=2_000_000, steps=20, mode="Erosion"),
        # the largest configuration that the benchmark runs: 513 x 2049 nodes, 64M particles
        dict(name="point_long", kind="point", stack="3grid", dx=0.003125, dt=1.25e-11, mass_ratio=400.0,
             ions=48_000_000, electrons=16_000_000, steps=10, mode="Erosion"),
        # a batch of perveance-sweep points of mixed grids and particle counts
        dict(name="batch_sweep", kind="batch", points=8, grids="64x256,128x512", n_lo=200_000, n_hi=1_000_000,
             pick=3, steps=20),
        # the field solve alone on a sweep grid and on the 3-grid aperture
        dict(name="field_small", kind="field", stack="2grid", dx=0.025),
        dict(name="field_large", kind="field", stack="3grid", dx=0.00625),
        # a small electron set in a magnetic field (latency of one call)
        dict(name="push_small", kind="push", n=20_000, ny=65, nx=284, dx=0.025, dt=2e-12, species="electron", b=0.05),
        # as the reference's step calls it: all of a species at once, no magnetic field
        dict(name="push_large", kind="push", n=16_000_000, ny=513, nx=2049, dx=0.003125, dt=1.25e-11, species="ion",
             b=0.0),
        dict(name="deposit_small", kind="deposit", ions=80_000, electrons=20_000, ny=65, nx=284, dx=0.025),
        dict(name="deposit_large", kind="deposit", ions=6_000_000, electrons=2_000_000, ny=257, nx=1025, dx=0.00625),
        dict(name="thermal_large", kind="thermal", ny=513, nx=2049),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("point", "point", "point", "batch", "field", "field", "push", "push", "deposit", "thermal"))
    if kind in ("point", "field"):
        # spacings between those of the benchmark's largest grid and the smallest sweep grid
        dx = round(_log(rng, 0.0033, 0.03), 6)
        stack = rng.choice(("2grid", "3grid"))
        if kind == "field":
            return dict(kind=kind, stack=stack, dx=dx)
        n = int(_log(rng, 2e4, 1.6e7))
        ne = int(n * rng.uniform(0.15, 0.4))
        return dict(kind=kind, stack=stack, dx=dx, dt=1e-10 * dx / 0.025, mass_ratio=rng.choice((100.0, 400.0)),
                    ions=n - ne, electrons=ne, steps=rng.choice((4, 10, 20)), mode=rng.choice(("Both", "Erosion")))
    if kind == "batch":
        lo = int(_log(rng, 3e4, 3e5))
        return dict(kind=kind, points=rng.randint(2, 10), grids=rng.choice(("64x256", "128x512", "64x256,128x512")),
                    n_lo=lo, n_hi=4 * lo, pick=rng.randint(0, 10**6), steps=rng.choice((4, 10, 20)))
    ny = int(_log(rng, 48, 520))
    nx = int(ny * rng.uniform(2.0, 4.5))
    if kind == "thermal":
        return dict(kind=kind, ny=ny, nx=nx)
    dx = round(1.6 / (ny - 1), 6)
    n = int(_log(rng, 1e3, 2e7))
    if kind == "deposit":
        ne = int(n * rng.uniform(0.15, 0.4))
        return dict(kind=kind, ions=n - ne, electrons=ne, ny=ny, nx=nx, dx=dx)
    species = rng.choice(("ion", "electron"))
    dt = 1e-10 * dx / 0.025 * (1.0 if species == "ion" else 0.02)
    return dict(kind=kind, n=n, ny=ny, nx=nx, dx=dx, dt=dt, species=species, b=rng.choice((0.0, 0.05)))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _params(stack, mode="Erosion"):
    s = STACKS[stack]
    p = dict(grids=[dict(V=v, t=t, gap=gap, r=r, cham=0.0) for v, t, gap, r in s["grids"]], pitch_mm=s["pitch_mm"],
             Te_up=5.0, n0_plasma=1e17, Ti=0.1, Tn=300.0, n0=1e18, neutral_profile="uniform", sim_mode=mode,
             neut_rate=30, Te=5.0, Thresh=1e9)
    if "upstream_gap_mm" in s:
        p["upstream_gap_mm"] = s["upstream_gap_mm"]
    return p


def _simulator(dx, dt, mass_ratio, params, seed, table):
    sim = PE.DigitalTwinSimulator(seed=seed)
    sim.dx = sim.dy = dx
    sim.dt = dt
    sim.m_ion = M_XE
    sim.m_e = M_XE / mass_ratio
    # slow heating: the electrodes stay within the bow limit however often a pass is repeated
    sim.thermal_accel = 1e3
    if table:
        sim.user_cs = W.cx_store(W.cx_table_power_law())
    sim.build_domain(params)
    return sim


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _preload(sim, params, n_ions, n_e, seed):
    """Particles over the non-electrode cells in pinned host memory: ions at the Bohm speed
    up to the plume boundary, thermal electrons over the whole domain."""
    g = _gen(seed)
    free = torch.from_numpy(~np.asarray(sim.isBound)).cuda()

    def positions(n, x_hi):
        xs, ys, got = [], [], 0
        while got < n:
            m = int(1.4 * (n - got)) + 1024
            x = 1.5 * sim.dx + (x_hi - 1.5 * sim.dx) * torch.rand(m, generator=g, device="cuda")
            y = sim.Ly * torch.rand(m, generator=g, device="cuda")
            ix = (x / sim.dx).round().long().clamp_(0, sim.nx - 1)
            iy = (y / sim.dy).round().long().clamp_(0, sim.ny - 1)
            ok = free[iy, ix]
            xs.append(x[ok])
            ys.append(y[ok])
            got += xs[-1].numel()
        return torch.cat(xs)[:n], torch.cat(ys)[:n]

    v_b, v_ti, v_te = W.thermal_speeds(sim, params)
    plume = W.plume_boundary(sim, params)
    keep, out = [], []
    for n, x_hi, drift, spread in ((n_ions, min(sim.Lx - sim.dx, plume), v_b, 4 * v_ti), (n_e, sim.Lx - sim.dx, 0.0, v_te)):
        x, y = positions(n, x_hi)
        v = [spread * torch.randn(n, generator=g, device="cuda") for _ in range(3)]
        v[0] += drift
        arrays = [x, y, *v, torch.arange(n, dtype=torch.int32, device="cuda")]
        arrays = [_pinned(a) for a in arrays] + [_pinned(torch.zeros(n, dtype=torch.uint8, device="cuda"))]
        keep += arrays
        out.append([a.numpy() for a in arrays[:5]] + [arrays[5].numpy().view(np.uint32), arrays[6].numpy()])
    return keep, out


def _point(sim, params, n_ions, n_e, seed):
    keep, (ions, eles) = _preload(sim, params, n_ions, n_e, seed)
    return dict(sim=sim, params=params, ions=ions, eles=eles, keep=keep, store=_store(n_ions, n_e))


def _upload(p):
    i, e = p["ions"], p["eles"]
    p["sim"].set_particles("ions", *i[:5], is_cex=i[6], ids=i[5])
    p["sim"].set_particles("electrons", *e[:5], ids=e[5])


class _Memory:
    """Device memory of a simulator, for torch; it holds the simulator, which owns it."""

    def __init__(self, sim, ptr, shape, typestr):
        self.sim = sim
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


def _view(sim, ptr, shape, typestr):
    return torch.as_tensor(_Memory(sim, ptr.value, shape, typestr), device="cuda")


_FIELDS = {"V": (0, "<f8"), "Ex": (1, "<f4"), "Ey": (2, "<f4"), "rho": (3, "<f4"), "Tmap": (4, "<f4"), "damage": (5, "<f8")}
_COLUMNS = ("x", "y", "vx", "vy", "vz", "cex", "id")


def _field(sim, name):
    which, typestr = _FIELDS[name]
    ptr = C.c_void_p()
    _lib.check(sim._libh.pb_sim_field_ptr(sim._h, which, C.byref(ptr)), "field_ptr")
    return _view(sim, ptr, (sim.ny, sim.nx), typestr)


def _columns():
    return [(sp, tag, which, col) for sp, tag in ((0, "p"), (1, "e")) for which, col in enumerate(_COLUMNS)
            if not (sp == 1 and col == "cex")]


def _room(n):
    return n + n // 50 + 40_000  # injection and secondaries of a pass


def _store(n_ions, n_e):
    """The caller's arrays for the particles at the end of a pass."""
    kinds = {"cex": torch.uint8, "id": torch.int32}
    return {f"{tag}_{col}": torch.zeros(_room((n_ions, n_e)[sp]), dtype=kinds.get(col, torch.float32), device="cuda")
            for sp, tag, _, col in _columns()}


def _collect(sim, store):
    """The simulator's particles into the caller's arrays (zeros past the last one)."""
    for sp, tag, which, col in _columns():
        n = sim.num_p if sp == 0 else sim.num_e
        ptr = C.c_void_p()
        _lib.check(sim._libh.pb_sim_particle_ptr(sim._h, sp, which, C.byref(ptr)), "particle_ptr")
        dst = store[f"{tag}_{col}"]
        dst[:n].copy_(_view(sim, ptr, (n,), {"cex": "|u1", "id": "<i4"}.get(col, "<f4")))
        dst[n:].zero_()
    return dict(store, num_p=sim.num_p, num_e=sim.num_e)


def _diagnostics(results):
    """Per step: saddle potential, divergence, transparency, electrode temperatures, remesh."""
    return dict(min_pot=np.array([float(r[1]) for r in results]), divergence=np.array([float(r[2]) for r in results]),
                transparency=np.array([float(r[4]) for r in results]),
                temperature=np.array([[float(t) for t in r[3]] for r in results]),
                remeshed=np.array([bool(r[0]) for r in results]))


def _electric_field(ny, nx, dx, g):
    """A smooth potential of a kilovolt scale over the grid, plus noise, as (Ex, Ey)."""
    y, x = torch.meshgrid(torch.linspace(0, 1, ny, device="cuda", dtype=torch.float64),
                          torch.linspace(0, 1, nx, device="cuda", dtype=torch.float64), indexing="ij")
    V = 1000.0 * (1 - x) ** 2 + 300.0 * torch.sin(3 * math.pi * x) * torch.cos(math.pi * y)
    V += 0.05 * torch.randn(ny, nx, generator=g, device="cuda", dtype=torch.float64)
    h = dx * 1e-3
    ey, ex = (-d for d in torch.gradient(V, spacing=(h, h)))
    return ex.float().contiguous(), ey.float().contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "point":
        params = _params(case["stack"], case["mode"])
        sim = _simulator(case["dx"], case["dt"], case["mass_ratio"], params, seed, True)
        return dict(_point(sim, params, case["ions"], case["electrons"], seed), case=case)
    if kind == "batch":
        rng = np.random.default_rng(case["pick"])
        members = []
        for k in range(case["points"]):
            spec = W.sweep_point(rng, k, grids=tuple(case["grids"].split(",")), n_range=(case["n_lo"], case["n_hi"]))
            sim = _simulator(spec["dx"], spec["dt"], spec["m_e_ratio"], spec["params"], seed + k, False)
            members.append(_point(sim, spec["params"], spec["n_ions"], spec["n_e"], seed + k))
        return dict(case=case, members=members, batch=SweepBatch())
    if kind == "field":
        params = _params(case["stack"])
        sim = _simulator(case["dx"], 1e-10 * case["dx"] / 0.025, 100.0, params, seed, False)
        return dict(case=case, sim=sim, params=params, charge=_charges(sim.nx, sim.ny, sim.isBound, seed), at=0)
    g = _gen(seed)
    ny, nx = case["ny"], case["nx"]
    if kind == "thermal":
        T = 300.0 + 500.0 * torch.rand(ny, nx, generator=g, device="cuda")
        mask = torch.zeros(ny, nx, dtype=torch.int32, device="cuda")
        for lo, hi in ((0.1, 0.2), (0.3, 0.45), (0.55, 0.65)):
            mask[ny // 3:, int(lo * nx):int(hi * nx)] = 1
        return dict(case=case, T=T, a=torch.empty_like(T), b=torch.empty_like(T), mask=mask)
    dx = case["dx"]
    Lx, Ly = (nx - 1) * dx, (ny - 1) * dx

    def cloud(n):
        return (Lx * (0.02 + 0.96 * torch.rand(n, generator=g, device="cuda")),
                Ly * (0.02 + 0.96 * torch.rand(n, generator=g, device="cuda")))

    if kind == "deposit":
        return dict(case=case, ions=cloud(case["ions"]), eles=cloud(case["electrons"]),
                    rho=torch.zeros(ny, nx, device="cuda"), cd=Q * 1e17 / 80.0)
    n = case["n"]
    x, y = cloud(n)
    m = M_XE if case["species"] == "ion" else M_XE / 400.0
    v_th = math.sqrt(Q * (0.1 if case["species"] == "ion" else 5.0) / m)
    v = [v_th * torch.randn(n, generator=g, device="cuda") for _ in range(3)]
    if case["species"] == "ion":
        v[0] += math.sqrt(Q * 5.0 / m)
    B = [torch.zeros(ny, nx, device="cuda") for _ in range(3)]
    if case["b"]:
        B[0] += 0.2 * case["b"]
        B[2] += case["b"] * (0.5 + torch.rand(ny, nx, generator=g, device="cuda"))
    Ex, Ey = _electric_field(ny, nx, dx, g)
    return dict(case=case, cols=[x, y, *v], E=[Ex, Ey], B=B, qm=(Q if case["species"] == "ion" else -Q) / m, sign=1.0)


def _charges(nx, ny, bound, seed):
    """Two space-charge densities: 80 macro-particles a cell upstream, thinning downstream."""
    g = _gen(seed)
    x = torch.linspace(0, 1, nx, device="cuda")[None, :]
    mean = (80.0 * torch.exp(-4.0 * x)).expand(ny, nx).contiguous()
    free = torch.from_numpy(~np.asarray(bound)).cuda()
    return [(torch.poisson(mean, generator=g) * free * (Q * 1e17 / 80.0)).float() for _ in range(2)]


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "point":
        sim, params = state["sim"], state["params"]
        _upload(state)
        results = [sim.step(params) for _ in range(case["steps"])]
        return dict(_collect(sim, state["store"]), **{k: _field(sim, k) for k in _FIELDS}, **_diagnostics(results))
    if kind == "batch":
        members = state["members"]
        for m in members:
            _upload(m)
        steps = state["batch"].run([m["sim"] for m in members], [m["params"] for m in members], case["steps"])
        parts = [_collect(m["sim"], m["store"]) for m in members]
        out = {k: torch.cat([p[k] for p in parts]) for k in members[0]["store"]}
        out["counts"] = [(p["num_p"], p["num_e"]) for p in parts]
        out.update({k: torch.cat([_field(m["sim"], k).reshape(-1) for m in members]) for k in _FIELDS})
        out["steps"] = [_diagnostics([r for r, _ in s])["min_pot"] for s in steps]
        return out
    if kind == "field":
        sim = state["sim"]
        _field(sim, "rho").copy_(state["charge"][state["at"]])
        state["at"] ^= 1
        torch.cuda.current_stream().synchronize()  # the solver runs on the simulator's own stream
        sim.recalc_poisson(iterations=5, params=state["params"])
        return {k: _field(sim, k) for k in ("V", "Ex", "Ey")}
    if kind == "push":
        cols = state["cols"]
        PE.push_particles_boris(*cols, *state["E"], *state["B"], case["n"], case["dx"], case["dx"], case["nx"],
                                case["ny"], state["sign"] * case["dt"], state["qm"])
        state["sign"] = -state["sign"]
        return dict(zip(_COLUMNS, cols))
    if kind == "deposit":
        rho = state["rho"]
        rho.zero_()
        for (x, y), cd in ((state["ions"], state["cd"]), (state["eles"], -state["cd"])):
            PE.accumulate_rho(x, y, rho, x.numel(), case["dx"], case["dx"], case["nx"], case["ny"], cd)
        return rho
    src, dst = state["T"], state["a"]
    for _ in range(10):
        PE.thermal_conduction(src, dst, state["mask"], case["nx"], case["ny"], 0.2, 0.15)
        src, dst = dst, state["b"] if dst is state["a"] else state["a"]
    return src


# ------------------------------------------------------------------ work
def _nodes(case):
    s = STACKS[case["stack"]]
    lx = s.get("upstream_gap_mm", 0.75 * s["grids"][0][3]) + sum(t + gap for _, t, gap, _ in s["grids"]) + 3.0
    ly = 0.5 * s["grids"][0][3] + 0.3 * s["pitch_mm"]
    return (int(lx / case["dx"]) + 1) * (int(ly / case["dx"]) + 1)


def _step_work(nodes, particles, steps):
    """Per step every particle's state is read and written (41 B) and deposited (8 B); every
    second step solves five linear systems (9 B a node each); fields and maps are read and
    written once (40 B a node).  About 90 operations a particle push and 100 a node and
    linear solve.  The upload reads the pre-load once (25 B a particle)."""
    per = 49.0 * particles + 40.0 * nodes + 2.5 * 9.0 * nodes
    return dict(bytes=steps * per + 25.0 * particles, flops=steps * (90.0 * particles + 2.5 * 100.0 * nodes))


def work(case):
    kind = case["kind"]
    if kind == "point":
        return _step_work(_nodes(case), case["ions"] + case["electrons"], case["steps"])
    if kind == "batch":
        rng = np.random.default_rng(case["pick"])
        tot = dict(bytes=0.0, flops=0.0)
        for k in range(case["points"]):
            spec = W.sweep_point(rng, k, grids=tuple(case["grids"].split(",")), n_range=(case["n_lo"], case["n_hi"]))
            one = _step_work(_nodes(dict(stack="2grid", dx=spec["dx"])), spec["n_ions"] + spec["n_e"], case["steps"])
            tot = {k: tot[k] + one[k] for k in tot}
        return tot
    if kind == "field":
        n = _nodes(case)
        return dict(bytes=(5 * 9.0 + 24.0) * n, flops=5 * 100.0 * n)
    cells = case["ny"] * case["nx"]
    if kind == "push":
        return dict(bytes=40.0 * case["n"] + 20.0 * cells, flops=120.0 * case["n"])
    if kind == "deposit":
        return dict(bytes=8.0 * (case["ions"] + case["electrons"]) + 4.0 * cells,
                    flops=6.0 * (case["ions"] + case["electrons"]))
    return dict(bytes=10 * 12.0 * cells, flops=10 * 10.0 * cells)


# ------------------------------------------------------------------ 64-bit results
def exact(case, seed):
    if case["kind"] in ("point", "batch"):
        return None  # a whole run: its particles' random draws and thousands of solves have no short form
    if case["kind"] == "field":
        return _exact_field(case, seed)
    s = prepare(case, seed)
    ny, nx = case["ny"], case["nx"]
    if case["kind"] == "thermal":
        T, m = s["T"].double(), s["mask"] == 1
        for _ in range(10):
            c2 = 2.0 * T

            def nb(axis, step):
                t, k = torch.roll(T, -step, axis), torch.roll(m, -step, axis)
                k = k.clone()
                k.select(axis, -1 if step > 0 else 0).fill_(False)
                return torch.where(k, t, T)

            d = float(np.float32(0.2)) * (nb(1, 1) + nb(1, -1) - c2) + float(np.float32(0.15)) * (nb(0, 1) + nb(0, -1) - c2)
            T = torch.where(m, (T + d).clamp(min=300.0), T)
        return T
    dx = float(np.float32(case["dx"]))
    if case["kind"] == "deposit":
        rho = torch.zeros(ny * nx, dtype=torch.float64, device="cuda")
        for (x, y), cd in ((s["ions"], s["cd"]), (s["eles"], -s["cd"])):
            # the cell is defined by the single-precision quotient (by a tensor: a scalar
            # divisor would become a multiplication by its reciprocal)
            d = torch.full_like(x, dx)
            ix = (x / d).round().long().clamp_(1, nx - 2)
            iy = (y / d).round().long().clamp_(1, ny - 2)
            rho += cd * torch.bincount(iy * nx + ix, minlength=ny * nx).double()
        return rho.reshape(ny, nx)
    x, y, vx, vy, vz = (c.double() for c in s["cols"])
    qx, qy = x / dx, y / dx
    ix, iy = qx.floor().long().clamp_(0, nx - 2), qy.floor().long().clamp_(0, ny - 2)
    fx, fy = qx - ix, qy - iy

    def gather(F):
        F = F.double().reshape(-1)
        i = iy * nx + ix
        return (F[i] * (1 - fx) * (1 - fy) + F[i + 1] * fx * (1 - fy) + F[i + nx] * (1 - fx) * fy + F[i + nx + 1] * fx * fy)

    h = 0.5 * s["qm"] * case["dt"]
    ex, ey = (h * gather(F) for F in s["E"])
    t = torch.stack([h * gather(F) for F in s["B"]])
    v = torch.stack([vx + ex, vy + ey, vz])
    vp = v + torch.linalg.cross(v, t, dim=0)
    v = v + torch.linalg.cross(vp, 2.0 * t / (1.0 + (t * t).sum(0)), dim=0)
    vx, vy, vz = v[0] + ex, v[1] + ey, v[2]
    return dict(zip(_COLUMNS, (x + vx * case["dt"] * 1000.0, y + vy * case["dt"] * 1000.0, vx, vy, vz)))


def _exact_field(case, seed):
    """The build's 30 damped Picard iterations without space charge, then 5 with the first
    density, each linear system solved directly (block elimination by grid columns)."""
    p = _params(case["stack"])
    grids = p["grids"]
    gap = p.get("upstream_gap_mm", 0.75 * grids[0]["r"])
    Lx = gap + sum(g["t"] + g["gap"] for g in grids) + 3.0
    Ly = 0.5 * grids[0]["r"] + 0.30 * p["pitch_mm"]
    nx, ny = int(Lx / case["dx"]) + 1, int(Ly / case["dx"]) + 1
    if nx * ny > 600_000:
        return None  # the direct solve takes too long
    dx, dy = Lx / (nx - 1), Ly / (ny - 1)
    X, Y = np.meshgrid(np.linspace(0, Lx, nx), np.linspace(0, Ly, ny))
    bound, fixed = np.zeros((ny, nx), bool), np.zeros((ny, nx))
    at = gap
    for g in grids:
        m = (X >= at) & (X <= at + g["t"]) & ~(np.abs(Y) <= g["r"])
        bound |= m
        fixed[m] = g["V"]
        at = at + g["t"] + g["gap"]
    Vp = grids[0]["V"] + 20.0
    bound[:, 0], fixed[:, 0] = True, Vp
    right = ~bound & (np.arange(nx)[None, :] == nx - 1)
    top = ~bound & ~right & (np.arange(ny)[:, None] == ny - 1)
    bottom = ~bound & ~right & (np.arange(ny)[:, None] == 0)
    inner = ~(bound | right | top | bottom)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    inner_t, bound_t, fixed_t = t(inner), t(bound), t(fixed)
    # rows: 4 V - neighbours inside, V - (inward neighbour) on copy rows, V on electrodes
    west = t(-(inner | right).astype(np.float64))
    east = t(-inner.astype(np.float64))
    diag = t(np.where(inner, 4.0, 1.0))
    south, north = t(-(inner | top).astype(np.float64)), t(-(inner | bottom).astype(np.float64))
    inv = []
    for j in range(nx):
        A = torch.diag(diag[:, j]) + torch.diag(south[1:, j], -1) + torch.diag(north[:-1, j], 1)
        if j:
            A -= west[:, j, None] * inv[-1] * east[None, :, j - 1]
        inv.append(torch.linalg.inv(A))

    def solve(b):
        y = []
        for j in range(nx):
            y.append(b[:, j] - west[:, j] * (inv[j - 1] @ y[-1]) if j else b[:, 0])
        v = [inv[-1] @ y[-1]]
        for j in range(nx - 2, -1, -1):
            v.append(inv[j] @ (y[j] - east[:, j] * v[-1]))
        return torch.stack(v[::-1], 1)

    rho = _charges(nx, ny, bound, seed)[0].double()
    V = torch.zeros(ny, nx, dtype=torch.float64, device="cuda")
    coeff = (dx * 1e-3) ** 2 / EPS0
    for it in range(35):
        r = (rho if it >= 30 else 0.0) - Q * 1e17 * torch.exp((V.clamp(max=Vp) - Vp) / 5.0)
        b = torch.where(inner_t, coeff * r, torch.where(bound_t, fixed_t, torch.zeros_like(V)))
        V = 0.8 * V + 0.2 * solve(b)
    ey, ex = torch.gradient(V, spacing=(dy * 1e-3, dx * 1e-3))
    return dict(V=V, Ex=-ex, Ey=-ey)
