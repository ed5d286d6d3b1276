"""The solver's workloads as timed cases: what a program that drives the library does with it.

A pass takes the initial state of every block from pinned host memory through `set_states`, advances a number of time
steps (reading the residuals back every `report` steps, as the reference's residual table does, or once at the end) and
brings the whole state back through `get_states`. Tilings are the engine's own choice: a program that does not run the
autotuner gets those. The served case submits its requests to the library's server together, waits and fetches.

`exact` advances the same initial states with a plain torch restatement of the schemes in 64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fvm-3d-f90_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from fvm3d import abi, cases as fvm_cases, serving  # noqa: E402
from fvm3d.solver import Solver  # noqa: E402

GAMMA = 1.4
PREC = {"exact": abi.PREC_FP64_EXACT, "fp64": abi.PREC_FP64, "fp32": abi.PREC_FP32_FLUX}
RECON = {"simple": abi.RECON_SIMPLE, "muscl": abi.RECON_MUSCL, "weno": abi.RECON_WENO}
FLUX = {"roe": abi.FLUX_ROE, "vanleer": abi.FLUX_VANLEER, "ausm": abi.FLUX_AUSM}
LIMITER = {"none": abi.LIMITER_NONE, "minmod": abi.LIMITER_MINMOD, "vanleer": abi.LIMITER_VANLEER,
           "vanalbada": abi.LIMITER_VANALBADA}


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # The reference's own case file (21 x 21 nodes, two k planes, fixed time step) in the precision form that
        # configurations default to, with the residual table printed every step: the smallest call, all latency.
        dict(name="riemann_21_exact", family="riemann2d", n=21, nk=2, prec="exact", recon="muscl", limiter="minmod",
             flux="roe", fix=0.2, rk=3, dt="fixed", compat="reference", steps=25, report=1),
        # The four-quadrant 2D Riemann problem at the size its configuration names: few cells, many steps.
        dict(name="riemann_256_fp64", family="riemann2d", n=256, nk=1, prec="fp64", recon="muscl", limiter="minmod",
             flux="roe", fix=0.2, rk=3, dt="cfl", compat="reference", steps=200, report=200),
        # A finer 2D grid with an odd edge, the other flux and limiter, FP32 flux arithmetic.
        dict(name="riemann_701_fp32", family="riemann2d", n=701, nk=1, prec="fp32", recon="muscl", limiter="vanleer",
             flux="vanleer", fix=0.05, rk=3, dt="cfl", compat="reference", steps=100, report=100),
        # The headline: isentropic vortex in 8 uneven periodic blocks, WENO5 + AUSM, classic RK4.
        dict(name="vortex_128_fp64", family="vortex", N=128, layout="blocks8", prec="fp64", rk=4, dt="cfl",
             compat="reference", steps=40, report=40),
        # The same with FP32 reconstruction and flux.
        dict(name="vortex_128_fp32", family="vortex", N=128, layout="blocks8", prec="fp32", rk=4, dt="cfl",
             compat="reference", steps=40, report=40),
        # The exact form (the default precision, bit-identical to the reference's arithmetic) on an eighth of the cells.
        dict(name="vortex_64_exact", family="vortex", N=64, layout="blocks8", prec="exact", rk=4, dt="cfl",
             compat="reference", steps=40, report=10),
        # Navier-Stokes: the Taylor-Green vortex, MUSCL / Van Albada + Roe + central viscous fluxes.
        dict(name="tgv_128_fp64", family="tgv", N=128, prec="fp64", rk=3, dt="cfl", compat="reference", steps=40,
             report=40),
        # The same flow on an odd grid in the FP32 form.
        dict(name="tgv_75_fp32", family="tgv", N=75, prec="fp32", rk=3, dt="cfl", compat="reference", steps=60,
             report=20),
        # A spherical blast on a ragged box with open boundaries, the published WENO5 with its positivity fallback.
        dict(name="blast_ragged_fp64", family="blast", nx=61, ny=83, nz=47, prec="fp64", recon="weno", limiter="none",
             flux="roe", fix=0.05, rk=3, dt="cfl", compat="textbook", steps=60, report=60),
        # Many independent cases of uneven size and mixed schemes advanced together.
        dict(name="batch_24_fp32", family="batch", count=24, lo=32, hi=96, prec="fp32", rk=3, compat="textbook",
             steps=30, report=30),
        # Requests of the three solver families served by the library's continuous batching.
        dict(name="serve_6_fp32", family="serve", count=6, lo=32, hi=64, prec="fp32", steps=40, report=40),
        # The largest: one periodic block of 160^3 cells, published WENO5 + AUSM, classic RK4.
        dict(name="vortex_160_textbook", family="vortex", N=160, layout="single", prec="fp64", rk=4, dt="cfl",
             compat="textbook", steps=25, report=25),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _steps(rng, cells, stages, prec):
    """As many steps as a share of the largest listed case's time pays for (the exact form takes three times as long)."""
    most = (0.7e8 if prec == "exact" else 2.2e8) / (cells * stages)
    return max(4, min(rng.randint(40, 160), int(rng.uniform(0.3, 1.0) * most)))


def draw(rng):
    fam = rng.choice(["riemann2d", "riemann2d", "vortex", "vortex", "tgv", "blast", "tube", "batch"])
    prec = rng.choice(["fp64", "fp64", "fp32", "fp32", "exact"])
    if fam == "riemann2d":
        n, nk = _log(rng, 16, 700), rng.choice([1, 1, 2])
        steps = max(8, min(rng.randint(40, 300), int(rng.uniform(0.3, 1.0) * 3.0e7 / (n * n * nk))))
        return dict(family=fam, n=n, nk=nk, prec=prec, recon=rng.choice(["muscl", "muscl", "simple"]),
                    limiter=rng.choice(["minmod", "vanleer", "vanalbada"]), flux=rng.choice(["roe", "vanleer", "ausm"]),
                    fix=0.2, rk=rng.choice([3, 3, 4]), dt="cfl", compat="reference", steps=steps,
                    report=rng.choice([1, steps]))
    if fam == "vortex":
        N, rk = _log(rng, 32, 128), rng.choice([3, 4, 4])
        steps = _steps(rng, N ** 3, rk, prec)
        return dict(family=fam, N=N, layout=rng.choice(["blocks8", "blocks8", "single"]), prec=prec, rk=rk, dt="cfl",
                    compat=rng.choice(["reference", "textbook"]), steps=steps, report=rng.choice([1, steps]))
    if fam == "tgv":
        N = _log(rng, 24, 128)
        steps = _steps(rng, N ** 3, 3, prec)
        return dict(family=fam, N=N, prec=prec, rk=3, dt="cfl", compat="reference", steps=steps,
                    report=rng.choice([10, steps]))
    if fam in ("blast", "tube"):
        nx, ny, nz = (_log(rng, 24, 112) for _ in range(3))
        steps = _steps(rng, nx * ny * nz, 3, prec)
        return dict(family=fam, nx=nx, ny=ny, nz=nz, prec=prec, recon=rng.choice(["muscl", "weno"]),
                    limiter=rng.choice(["minmod", "vanleer", "vanalbada"]), flux=rng.choice(["roe", "ausm", "vanleer"]),
                    fix=0.05, rk=3, dt=rng.choice(["cfl", "cfl", "local"]), compat="textbook", steps=steps, report=steps)
    return dict(family=fam, count=rng.randint(6, 24), lo=24, hi=rng.randint(48, 96), prec=rng.choice(["fp64", "fp32"]),
                rk=3, compat="textbook", steps=rng.randint(10, 30), report=30)


# ---------------------------------------------------------------- seeded initial states (conservative, on the device)
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cons(rho, u, v, w, p):
    e = p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v + w * w)
    return torch.stack([rho, rho * u, rho * v, rho * w, e])


def _centres(n, h, origin):
    ax = [origin[a] + (torch.arange(n[a], dtype=torch.float64, device=_device()) + 0.5) * h[a] for a in range(3)]
    Z, Y, X = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return X, Y, Z


def _riemann(case, seed):
    """Four seeded quadrant states on n x n nodes of the unit square."""
    r = np.random.default_rng(seed)
    n, nk = case["n"], case["nk"]
    h = 1.0 / (n - 1)
    q = torch.empty((5, nk, n, n), dtype=torch.float64, device=_device())
    m = n // 2
    for js, ix in ((slice(m, n), slice(m, n)), (slice(m, n), slice(0, m)), (slice(0, m), slice(0, m)),
                   (slice(0, m), slice(m, n))):
        rho, p = r.uniform(0.5, 1.5), r.uniform(0.3, 1.5)
        u, v = r.uniform(-0.5, 0.5, 2)
        s = _cons(*(torch.tensor(x, dtype=torch.float64) for x in (rho, u, v, 0.0, p))).to(q.device)
        q[:, :, js, ix] = s[:, None, None, None]
    cfg = dict(idimension=2, reconstruct=RECON[case["recon"]], limiter=LIMITER[case["limiter"]], kappa=1.0 / 3.0,
               flux_split=FLUX[case["flux"]], entropy_fix=case["fix"])
    return q, (h, h, 1.0), cfg


def _vortex(case, seed):
    """Isentropic vortex of seeded strength and centre in the periodic box [-5,5]^3."""
    r = np.random.default_rng(seed)
    N = case["N"]
    beta, x0, y0 = r.uniform(4.0, 5.0), r.uniform(-2.0, 2.0), r.uniform(-2.0, 2.0)
    h = 10.0 / N
    X, Y, Z = _centres((N, N, N), (h, h, h), (-5.0, -5.0, -5.0))
    X, Y = torch.remainder(X - x0 + 5.0, 10.0) - 5.0, torch.remainder(Y - y0 + 5.0, 10.0) - 5.0
    e = torch.exp(0.5 * (1.0 - X * X - Y * Y))
    T = 1.0 - (GAMMA - 1.0) * beta * beta / (8.0 * GAMMA * math.pi ** 2) * e * e
    rho = T ** (1.0 / (GAMMA - 1.0))
    q = _cons(rho, 1.0 - beta / (2 * math.pi) * e * Y, 1.0 + beta / (2 * math.pi) * e * X, torch.ones_like(X), rho * T)
    return q, (h, h, h), dict(idimension=3, reconstruct=abi.RECON_WENO, flux_split=abi.FLUX_AUSM)


def _tgv(case, seed):
    """Taylor-Green vortex on [0,2 pi)^3, Ma 0.1, Re 1600, with a seeded phase per axis."""
    r = np.random.default_rng(seed)
    N = case["N"]
    h = 2 * math.pi / N
    X, Y, Z = _centres((N, N, N), (h, h, h), r.uniform(0.0, 2 * math.pi, 3))
    u, v = torch.sin(X) * torch.cos(Y) * torch.cos(Z), -torch.cos(X) * torch.sin(Y) * torch.cos(Z)
    p = 1.0 / (GAMMA * 0.01) + (1.0 / 16.0) * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0)
    q = _cons(torch.ones_like(X), u, v, torch.zeros_like(X), p)
    cfg = dict(idimension=3, equation=abi.EQ_NAVIER_STOKES, mu=1.0 / 1600.0, prandtl=0.71, reconstruct=abi.RECON_MUSCL,
               limiter=abi.LIMITER_VANALBADA, kappa=1.0 / 3.0, flux_split=abi.FLUX_ROE, entropy_fix=0.05)
    return q, (h, h, h), cfg


def _shock(case, seed):
    """A spherical blast or an oblique shock tube in the unit box, seeded states and geometry."""
    r = np.random.default_rng(seed)
    n = (case["nx"], case["ny"], case["nz"])
    h = tuple(1.0 / m for m in n)
    X, Y, Z = _centres(n, h, (0.0, 0.0, 0.0))
    (ra, rb), (pa, pb) = r.uniform(0.2, 2.0, 2), r.uniform(0.1, 5.0, 2)
    if case["family"] == "blast":
        a = (X - 0.5) ** 2 + (Y - 0.5) ** 2 + (Z - 0.5) ** 2 <= r.uniform(0.1, 0.3) ** 2
    else:
        d = r.normal(size=3)
        a = (X - 0.5) * d[0] + (Y - 0.5) * d[1] + (Z - 0.5) * d[2] < 0.0
    z = torch.zeros_like(X)
    q = _cons(torch.where(a, z + ra, z + rb), z, z, z, torch.where(a, z + pa, z + pb))
    cfg = dict(idimension=3, reconstruct=RECON[case["recon"]], limiter=LIMITER[case["limiter"]], kappa=1.0 / 3.0,
               flux_split=FLUX[case["flux"]], entropy_fix=case["fix"], cfl=0.4)
    return q, h, cfg


_FAMILY = {"riemann2d": _riemann, "vortex": _vortex, "tgv": _tgv, "blast": _shock, "tube": _shock}


def _members(case, seed):
    """The single cases of a batched or served one, seeded: sizes log-uniform in [lo, hi], mixed schemes."""
    r = np.random.default_rng(1000003 * seed + 17)
    sizes = np.random.default_rng(case["count"] * 1000 + case["hi"])  # the sizes and schemes are the case's, not the seed's
    out = []
    for i in range(case["count"]):
        edge = [int(round(case["lo"] * (case["hi"] / case["lo"]) ** x)) for x in sizes.uniform(size=3)]
        c = dict(prec=case["prec"], steps=case["steps"], report=case["report"], seed=int(r.integers(1 << 30)))
        if case["family"] == "batch":
            c.update(family=["blast", "tube"][int(sizes.integers(2))], nx=edge[0], ny=edge[1], nz=edge[2],
                     recon=["muscl", "weno"][int(sizes.integers(2))], flux=["roe", "ausm"][int(sizes.integers(2))],
                     limiter="minmod", fix=0.05, rk=case["rk"], dt="cfl", compat=case["compat"])
        else:
            c.update(dt="cfl", compat="reference", steps=case["steps"] + 5 * i)
            fam = i % 3
            if fam == 0:
                c.update(family="riemann2d", n=int(round(edge[0] ** 1.5)), nk=1, recon="muscl", limiter="minmod",
                         flux="roe", fix=0.2, rk=3)
            elif fam == 1:
                c.update(family="vortex", N=edge[0], layout="blocks8", rk=4)
            else:
                c.update(family="tgv", N=edge[0], rk=3)
        out.append(c)
    return out


def _config(case, cfg):
    d = dict(precision=PREC[case["prec"]], rk_stages=case["rk"], cfl=0.5)
    d["compat"] = abi.COMPAT_TEXTBOOK if case["compat"] == "textbook" else abi.COMPAT_REFERENCE
    d["timestep_set"] = {"fixed": abi.DT_FIXED, "cfl": abi.DT_CFL, "local": abi.DT_CFL_LOCAL}[case["dt"]]
    if case["dt"] == "fixed":
        d["dt"] = 2.0e-4
    d.update(cfg)
    return d


def _boxes(case, shape):
    """The blocks of a case: global cell ranges (lo, hi), hi exclusive."""
    if case.get("layout") == "blocks8":
        return fvm_cases.vortex_blocks(case["N"])
    return [((0, 0, 0), (shape[3], shape[2], shape[1]))]


def _cut(q, box):
    lo, hi = box
    return q[:, lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]]


def _describe(case, seed):
    """The framework's description of one case (blocks, boundaries, connections) and its block states on the device."""
    q, dr, cfg = _FAMILY[case["family"]](case, seed)
    boxes = _boxes(case, q.shape)
    c = fvm_cases.Case(name=case["family"], cfg=_config(case, cfg))
    for lo, hi in boxes:
        c.blocks.append((tuple(hi[a] - lo[a] for a in range(3)), dr))
        c.origins.append(lo)
    if case["family"] == "vortex" and len(boxes) > 1:
        c.conns, c.bcs = fvm_cases.periodic_box_connections((case["N"],) * 3, boxes)
    elif case["family"] in ("vortex", "tgv"):
        c.bcs = [(0, region, abi.BC_PERIODIC) for region in range(1, 7)]
    return c, [_cut(q, b) for b in boxes]


def _host(t):
    """A contiguous copy in pinned host memory."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    h.copy_(t)
    return h


# ---------------------------------------------------------------- preparing and running
def prepare(case, seed):
    if case["family"] == "serve":
        reqs, cells = [], 0
        for m in _members(case, seed):
            c, qs = _describe(m, m["seed"])
            c.states = [q.cpu().numpy().copy() for q in qs]
            reqs.append((c, m["steps"]))
            cells += sum(abi.block_cells(c.cfg["idimension"], n) for n, _ in c.blocks)
        return {"server": serving.Server(budget_cells=cells, max_active_cells=None), "requests": reqs}
    st = {"steps": case["steps"], "report": case["report"], "in": [], "out": [], "cases": []}
    if case["family"] == "batch":
        members = _members(case, seed)
        s = None
        for m in members:
            c, qs = _describe(m, m["seed"])
            if s is None:
                s = Solver(c.config())
                c.apply(s, states=False)
                st["cases"].append(0)
            else:
                cid = s.add_case(c.config())
                c.apply(s, states=False, case_id=cid)
                st["cases"].append(cid)
            st["in"] += [_host(q) for q in qs]
    else:
        c, qs = _describe(case, seed)
        s = Solver(c.config())
        c.apply(s, states=False)
        st["in"] = [_host(q) for q in qs]
    st["out"] = [_host(torch.zeros_like(q)) for q in st["in"]]
    st["blocks"] = list(range(len(st["in"])))
    st["in_ptr"] = [q.data_ptr() for q in st["in"]]
    st["out_ptr"] = [q.data_ptr() for q in st["out"]]
    st["solver"] = s
    return st


def run(state):
    if "server" in state:
        srv, out = state["server"], []
        ids = [srv.submit(c, steps) for c, steps in state["requests"]]
        for rid, (c, _) in zip(ids, state["requests"]):
            srv.wait(rid)
            out.append(srv.fetch(rid, c))
            srv.release(rid)
        return {"q": out}
    s = state["solver"]
    s.set_states_ptr(state["blocks"], state["in_ptr"])
    left, res = state["steps"], None
    while left > 0:
        k = min(left, state["report"])
        _, res, _ = s.step(k)
        left -= k
    if state["cases"]:
        res = np.stack([s.case_state(c)["res_abs"] for c in state["cases"]])
    s.get_states_ptr(state["blocks"], state["out_ptr"])
    return {"q": state["out"], "residual": res}


# ---------------------------------------------------------------- what a pass cannot do without
def _cells(case):
    f = case["family"]
    if f == "riemann2d":
        return case["n"] * case["n"] * case["nk"]
    if f in ("vortex", "tgv"):
        return case["N"] ** 3
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Bytes: the state up and down once (40 B a cell each way) and, per step, the state arrays that the Runge-Kutta
    stages read and write (8 of 40 B for three stages, 16 for four). Flops: what reconstruction, flux and update of a
    cell take per stage, each node and face once."""
    if case["family"] in ("batch", "serve"):
        parts = [work(m) for m in _members(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    cells, dim = _cells(case), 2 if case["family"] == "riemann2d" else 3
    recon = case.get("recon", "weno" if case["family"] == "vortex" else "muscl")
    node = {"weno": 260.0 * (1.8 if case["compat"] == "textbook" else 1.0), "muscl": 90.0, "simple": 0.0}[recon]
    per = dim * (node + 80.0) + 40.0 + (200.0 if case["family"] == "tgv" else 0.0)
    step = 320.0 if case["rk"] == 3 else 640.0
    return {"bytes": cells * (80.0 + step * case["steps"]), "flops": cells * per * case["rk"] * case["steps"]}


# ---------------------------------------------------------------- the schemes in plain torch, 64 bits
def _prim(q):
    u, v, w = q[1] / q[0], q[2] / q[0], q[3] / q[0]
    return torch.stack([q[0], u, v, w, (GAMMA - 1.0) * (q[4] - 0.5 * q[0] * (u * u + v * v + w * w))])


def _extend(a, axis, width, periodic):
    """`width` ghost layers on both sides of the last-but-`axis` dimension (axis 0 is x): wrapped or the edge cell."""
    d = a.dim() - 1 - axis
    n = a.shape[d]
    i = torch.arange(-width, n + width, device=a.device)
    return a.index_select(d, i % n if periodic else i.clamp(0, n - 1))


def _at(a, axis, lo, n):
    return a.narrow(a.dim() - 1 - axis, lo, n)


def _weno(u, textbook):
    u0, u1, u2, u3, u4 = u
    q = [u0 / 3 - 7 * u1 / 6 + 11 * u2 / 6, -u1 / 6 + 5 * u2 / 6 + u3 / 3, u2 / 3 + 5 * u3 / 6 - u4 / 6]
    b1 = (u1 - u3) if textbook else (u1 + u3)
    s = [13 / 12 * (u0 - 2 * u1 + u2) ** 2 + 0.25 * (u0 - 4 * u1 + 3 * u2) ** 2,
         13 / 12 * (u1 - 2 * u2 + u3) ** 2 + 0.25 * b1 ** 2,
         13 / 12 * (u2 - 2 * u3 + u4) ** 2 + 0.25 * (3 * u2 - 4 * u3 + u4) ** 2]
    a = [c / (x + 1e-6) ** 2 for c, x in zip((0.1, 0.6, 0.3), s)]
    return (a[0] * q[0] + a[1] * q[1] + a[2] * q[2]) / (a[0] + a[1] + a[2])


def _sign(x):
    return torch.copysign(torch.ones_like(x), x)


def _slopes(dm, dp, limiter):
    if limiter == abi.LIMITER_MINMOD:
        s = 0.5 * (_sign(dm) + _sign(dp)) * torch.minimum(dm.abs(), dp.abs())
    elif limiter == abi.LIMITER_VANLEER:
        s = (_sign(dm) + _sign(dp)) * dm * dp / (dm.abs() + dp.abs() + 1e-6)
    elif limiter == abi.LIMITER_VANALBADA:
        s = (dm * (dp * dp + 1e-6) + dp * (dm * dm + 1e-6)) / (dm * dm + dp * dp + 1e-6)
    else:
        return dm, dp
    return s, s


def _face_states(q, axis, cfg, periodic):
    """Primitive states on the left and right of the n + 1 faces along `axis`."""
    n = q.shape[q.dim() - 1 - axis]
    g = _extend(q, axis, 3, periodic)
    textbook = cfg["compat"] == abi.COMPAT_TEXTBOOK
    p = _prim(g)
    cl, cr = _at(p, axis, 2, n + 1), _at(p, axis, 3, n + 1)  # the cells on either side of each face
    if cfg["reconstruct"] == abi.RECON_SIMPLE:
        return cl, cr
    if cfg["reconstruct"] == abi.RECON_MUSCL:
        m, c, z = _at(p, axis, 1, n + 2), _at(p, axis, 2, n + 2), _at(p, axis, 3, n + 2)  # cells -1 .. n
        bm, bp = _slopes(c - m, z - c, cfg["limiter"])
        k = cfg["kappa"]
        right = c + 0.25 * ((1 - k) * bm + (1 + k) * bp)  # at the cell's right face
        left = c - 0.25 * ((1 - k) * bp + (1 + k) * bm)
        L, R = _at(right, axis, 0, n + 1), _at(left, axis, 1, n + 1)
    else:
        L = _prim(_weno([_at(g, axis, s, n + 1) for s in range(5)], textbook))
        if textbook:
            R = _prim(_weno([_at(g, axis, 5 - s, n + 1) for s in range(5)], True))
        else:  # the reference takes the left-biased formula one cell over
            R = _prim(_weno([_at(g, axis, 1 + s, n + 1) for s in range(5)], False))
    if textbook:
        L = torch.where((L[0] > 0) & (L[4] > 0), L, cl)
        R = torch.where((R[0] > 0) & (R[4] > 0), R, cr)
    return L, R


def _euler(s, vn, axis):
    H = GAMMA / (GAMMA - 1) * s[4] / s[0] + 0.5 * (s[1] ** 2 + s[2] ** 2 + s[3] ** 2)
    f = s[0] * vn * torch.stack([torch.ones_like(vn), s[1], s[2], s[3], H])
    f[1 + axis] += s[4]
    return f, H


def _roe(L, R, axis, fix):
    vl, vr = L[1 + axis], R[1 + axis]
    fl, Hl = _euler(L, vl, axis)
    fr, Hr = _euler(R, vr, axis)
    rb = torch.sqrt(L[0] * R[0])
    avg = lambda a, b: (L[0] * a + rb * b) / (L[0] + rb)  # noqa: E731
    ub, Hb = [avg(L[m], R[m]) for m in (1, 2, 3)], avg(Hl, Hr)
    vb, q2 = ub[axis], ub[0] ** 2 + ub[1] ** 2 + ub[2] ** 2
    c = torch.sqrt((GAMMA - 1) * (Hb - 0.5 * q2))
    delta = fix * (vb + c).abs()
    lam = lambda x: torch.where(x > delta, x, 0.5 * (x * x + delta * delta) / delta)  # noqa: E731
    l1, l2, l5 = lam((vb - c).abs()), lam(vb.abs()), lam((vb + c).abs())
    d, dv, dp = R - L, vr - vl, R[4] - L[4]
    a1, a2, a5 = l1 * (dp - rb * c * dv) / (2 * c * c), l2 * (d[0] - dp / (c * c)), l5 * (dp + rb * c * dv) / (2 * c * c)
    out = [a1 + a2 + a5]
    for m in range(3):
        on = m == axis
        out.append(a1 * (ub[m] - c if on else ub[m]) + a5 * (ub[m] + c if on else ub[m]) + a2 * ub[m]
                   + l2 * rb * (d[1 + m] - (dv if on else 0.0)))
    out.append(a1 * (Hb - c * vb) + a5 * (Hb + c * vb) + 0.5 * a2 * q2
               + l2 * rb * (ub[0] * d[1] + ub[1] * d[2] + ub[2] * d[3] - vb * dv))
    return 0.5 * (fl + fr - torch.stack(out))


def _van_leer(L, R, axis, textbook):
    total = 0.0
    for s, side in ((L, 1.0), (R, -1.0)):
        v, q2 = s[1 + axis], s[1] ** 2 + s[2] ** 2 + s[3] ** 2
        c = torch.sqrt(GAMMA * s[4] / s[0])
        M = v / c
        up, off = side * M >= 1, side * M <= -1
        Ms = torch.where(up, M, torch.where(off, torch.zeros_like(M), side * 0.25 * (M + side) ** 2))
        f0 = s[0] * c * Ms
        f = torch.stack([f0, f0 * s[1], f0 * s[2], f0 * s[3],
                         f0 * (((GAMMA - 1) * v + side * 2 * c) ** 2 / (2 * (GAMMA ** 2 - 1)) + (q2 - v * v) / 2)])
        f[1 + axis] += f0 * (-v + side * 2 * c) / GAMMA
        if textbook:
            f = torch.where(up, _euler(s, v, axis)[0], torch.where(off, torch.zeros_like(f), f))
        total = total + f
    return total


def _ausm(L, R, axis):
    side = []
    for s, w in ((L, 1.0), (R, -1.0)):
        v = s[1 + axis]
        c = torch.sqrt(GAMMA * s[4] / s[0])
        M = v / c
        sup = M.abs() >= 1
        Ms = torch.where(sup, 0.5 * (M + w * M.abs()), w * 0.25 * (M + w) ** 2)
        ps = torch.where(sup, 0.5 * (1 + w * _sign(M)), 0.25 * (M + w) ** 2 * (2 - w * M)) * s[4]
        H = GAMMA / (GAMMA - 1) * s[4] / s[0] + 0.5 * (s[1] ** 2 + s[2] ** 2 + s[3] ** 2)
        side.append((Ms, ps, s[0] * c * torch.stack([torch.ones_like(v), s[1], s[2], s[3], H])))
    M = side[0][0] + side[1][0]
    a = torch.where(M.abs() > 0.1, M.abs(), 0.5 * (M * M + 0.01) / 0.1)
    f = 0.5 * (M + a) * side[0][2] + 0.5 * (M - a) * side[1][2]
    f[1 + axis] += side[0][1] + side[1][1]
    return f


def _viscous(q, dr, cfg):
    """Central viscous flux differences of a periodic box."""
    p = _prim(q)
    t = torch.stack([p[1], p[2], p[3], p[4] / p[0]])
    kq = cfg["mu"] * GAMMA / (cfg["prandtl"] * (GAMMA - 1))
    sh = lambda a, axis, k: torch.roll(a, -k, dims=a.dim() - 1 - axis)  # noqa: E731  a at i + k
    out = torch.zeros_like(q)
    for axis in range(3):
        nxt = sh(t, axis, 1)  # the face above cell i
        grad = [None] * 3
        for d in range(3):
            if d == axis:
                grad[d] = (nxt - t) / dr[d]
            else:
                c = sh(t, d, 1) - sh(t, d, -1)
                grad[d] = (c + sh(c, axis, 1)) / (4 * dr[d])
        div = grad[0][0] + grad[1][1] + grad[2][2]
        tau = [cfg["mu"] * (grad[axis][m] + grad[m][axis]) for m in range(3)]
        tau[axis] = tau[axis] - 2.0 / 3.0 * cfg["mu"] * div
        uf = 0.5 * (t + nxt)
        g = torch.stack([torch.zeros_like(div), *tau, uf[0] * tau[0] + uf[1] * tau[1] + uf[2] * tau[2] + kq * grad[axis][3]])
        out += (g - sh(g, axis, -1)) / dr[axis]
    return out


def _rhs(q, dr, cfg, periodic):
    out = torch.zeros_like(q)
    for axis in range(cfg["idimension"]):
        L, R = _face_states(q, axis, cfg, periodic)
        if cfg["flux_split"] == abi.FLUX_ROE:
            f = _roe(L, R, axis, cfg["entropy_fix"])
        elif cfg["flux_split"] == abi.FLUX_VANLEER:
            f = _van_leer(L, R, axis, cfg["compat"] == abi.COMPAT_TEXTBOOK)
        else:
            f = _ausm(L, R, axis)
        n = q.shape[q.dim() - 1 - axis]
        out -= (_at(f, axis, 1, n) - _at(f, axis, 0, n)) / dr[axis]
    if cfg.get("equation", abi.EQ_EULER) == abi.EQ_NAVIER_STOKES:
        out += _viscous(q, dr, cfg)
    return out


def _advance(q, dr, cfg, periodic, steps):
    """The state after `steps` steps and the last step's rhs."""
    for _ in range(steps):
        if cfg["timestep_set"] == abi.DT_FIXED:
            h = cfg["dt"]
        else:
            p = _prim(q)
            c = torch.sqrt(GAMMA * p[4] / p[0])
            s = sum((p[1 + a].abs() + c) / dr[a] for a in range(cfg["idimension"]))
            h = cfg["cfl"] / (s if cfg["timestep_set"] == abi.DT_CFL_LOCAL else s.max())
        q0, f = q, lambda x: _rhs(x, dr, cfg, periodic)
        r = f(q0)
        if cfg["rk_stages"] == 3:
            q = q0 + h * r
            r = f(q)
            q = 0.75 * q0 + 0.25 * q + 0.25 * h * r
            r = f(q)
            q = q0 / 3 + 2.0 / 3.0 * q + 2.0 / 3.0 * h * r
        else:
            acc = q0 + h / 6 * r
            r = f(q0 + 0.5 * h * r)
            acc = acc + h / 3 * r
            r = f(q0 + 0.5 * h * r)
            acc = acc + h / 3 * r
            r = f(q0 + h * r)
            q = acc + h / 6 * r
    return q, r


def _exact_one(case, seed):
    q, dr, cfg = _FAMILY[case["family"]](case, seed)
    q, r = _advance(q, dr, _config(case, cfg), case["family"] in ("vortex", "tgv"), case["steps"])
    boxes = _boxes(case, q.shape)
    res2 = sum(_cut(r, b).square().mean(dim=(1, 2, 3)) for b in boxes)  # the norms accumulate over the blocks
    res = torch.sqrt(torch.cat([res2, res2.mean().reshape(1)]))
    return [_cut(q, b).contiguous().cpu() for b in boxes], res.cpu().numpy()


def exact(case, seed):
    if case["family"] in ("batch", "serve"):
        parts = [_exact_one(m, m["seed"]) for m in _members(case, seed)]
        if case["family"] == "serve":
            return {"q": [[b.numpy() for b in q] for q, _ in parts]}
        return {"q": [b for q, _ in parts for b in q], "residual": np.stack([r for _, r in parts])}
    q, res = _exact_one(case, seed)
    return {"q": q, "residual": res}
