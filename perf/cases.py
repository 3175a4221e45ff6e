"""Performance cases of the immersed-boundary time step, through the Python binding and the C ABI.

A case is one kind of work at one size:

* ``cylinder``   a rigid body in a free stream, the direct solve (num_stat), `steps` time steps
* ``plate``      a hinged plate, GMRES on the assembled Schur operator, `steps` time steps
* ``subdomain``  the same plate through the sub-domain precomputed-Schur method
* ``beam``       a clamped Euler-Bernoulli beam
* ``batch``      several independent plates of uneven grids advanced together
* ``adjoint``    a pitching airfoil: `steps` forward steps and the reverse sweep
* ``pressure``   the pressure recovery of the current state on every level
* ``vort2flux``  the streamfunction and fluxes of a given vorticity on every level
* ``poisson``    one Poisson solve on one level
* ``viscous``    one Crank-Nicolson viscous solve (the predictor's, on given right-hand sides)
* ``schur``      one matrix-free product with the Schur operator

A stepping pass is what a host's time loop does between two writes of its output: `steps` times the
step and its force coefficients (and hinge angle), then the vorticity of every level and the body
forces.  Operator passes take and return device arrays, which the C ABI uses in place.
"""
import math
import os

os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")   # before CUDA starts: what batches ask of a program

import numpy as np
import torch

from ib_parallel_gb300 import geometry as GEO
from ib_parallel_gb300 import ibgpu as G


def listed():
    return [
        # the impulsively started cylinder at the size of a first try: launches and host waits dominate
        dict(name="cylinder_64x32x3", kind="cylinder", m=64, n=32, levels=3, npts=25, re=100.0, dt=0.01, steps=10),
        # flow past a stationary cylinder, the everyday rigid-body run
        dict(name="cylinder_400x200x3", kind="cylinder", m=400, n=200, levels=3, npts=157, re=100.0, dt=0.004, steps=10),
        # strongly coupled fluid-structure interaction at the size the framework is quoted on
        dict(name="plate_800x400x5", kind="plate", m=800, n=400, levels=5, npts=51, re=500.0, dt=1e-3, steps=10),
        # the largest grid in use: a well resolved plate at Re 1000
        dict(name="plate_1536x1024x5", kind="plate", m=1536, n=1024, levels=5, npts=97, re=1000.0, dt=5e-4, steps=4),
        # the same physics through the precomputed sub-domain, the reference's default method
        dict(name="subdomain_512x256x4", kind="subdomain", m=512, n=256, levels=4, npts=33, re=300.0, dt=2e-3, steps=10),
        # a flexible plate on a grid that is no power of two
        dict(name="beam_600x300x4", kind="beam", m=600, n=300, levels=4, npts=39, re=500.0, dt=1e-3, steps=6),
        # a parameter sweep: independent simulations of uneven grids side by side
        dict(name="batch_12", kind="batch", sims=12, m=256, n=128, levels=3, dt=2e-3, steps=4),
        # gradients of the forces with respect to the motion of a pitching airfoil
        dict(name="adjoint_600x300x4", kind="adjoint", m=600, n=300, levels=4, re=200.0, dt=2e-3, steps=10, keep=5),
        # the pressure written with each output
        dict(name="pressure_800x400x5", kind="pressure", m=800, n=400, levels=5, npts=51, re=500.0, dt=1e-3),
        # the flux recovery as an operator, on a ragged grid
        dict(name="vort2flux_1000x540x4", kind="vort2flux", m=1000, n=540, levels=4),
        # one Poisson solve on a large single level, as a host program's own solver
        dict(name="poisson_1600x800", kind="poisson", m=1600, n=800, levels=1),
        # the matrix-free Schur product: set-up of direct solves, and bodies near the domain's edge
        dict(name="schur_800x400x5", kind="schur", m=800, n=400, levels=5, npts=51, re=500.0, dt=1e-3),
    ]


def _smooth(limit):
    """Numbers divisible by 4 whose only prime factors are 2, 3 and 5."""
    out = []
    for v in range(8, limit + 1, 4):
        q = v
        for f in (2, 3, 5):
            while q % f == 0:
                q //= f
        if q == 1:
            out.append(v)
    return out


def draw(rng):
    kind = rng.choice(["cylinder", "plate", "plate", "subdomain", "beam", "batch", "adjoint", "pressure", "vort2flux",
                       "poisson", "viscous", "schur"])
    sizes = _smooth(2000)

    def near(v):
        return min(sizes, key=lambda s: abs(math.log(s / v)))

    def log_between(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    levels = rng.randint(2, 5)
    if kind in ("poisson", "viscous"):
        return dict(kind=kind, m=near(log_between(48, 1600)), n=near(log_between(32, 800)), levels=1)
    lo, hi = dict(cylinder=(64, 800), plate=(200, 1200), subdomain=(240, 640), beam=(240, 800), adjoint=(320, 600),
                  batch=(160, 320)).get(kind, (128, 1000))
    m = near(log_between(lo, hi))
    n = near(m * rng.uniform(0.42, 0.7))
    if kind == "vort2flux":
        return dict(kind=kind, m=m, n=n, levels=levels)
    case = dict(kind=kind, m=m, n=n, levels=levels, re=round(log_between(50, 500), 1), dt=round(0.8 / m, 7))
    if kind == "batch":
        case.pop("re")
        return dict(case, sims=rng.randint(3, 12), steps=rng.randint(2, 4))
    if kind == "adjoint":
        keep = rng.randint(2, 5)
        return dict(case, steps=keep * 2, keep=keep)
    if kind == "cylinder":
        return dict(case, npts=max(8, round(math.pi * m / 8.0 / rng.uniform(1.0, 2.0))), steps=rng.randint(4, 10))
    # a plate's points are about two grid spacings apart, as the reference's inputs have them
    npts = max(9, round(m / 8.0 / rng.uniform(2.0, 2.4)) + 1)
    if kind in ("pressure", "schur"):
        return dict(case, npts=npts)
    return dict(case, npts=npts, steps=rng.randint(2, 8))


# ---------------------------------------------------------------------------------------------
def _params(case, rng, **over):
    m, n = case["m"], case["n"]
    height = 8.0 * n / m
    a = rng.uniform(-0.02, 0.02)   # the stream's direction
    kw = dict(m=m, n=n, mgridlev=case["levels"], dt=case.get("dt", 1e-3), Re=case.get("re", 100.0), len=8.0, offsetx=1.0,
              offsety=0.5 * height, fsi_tol=1e-10, atol=1e-10, rtol=1e-10, autotune=False,
              motion=(-math.cos(a), -math.sin(a), 0.0, 0.0, 0.0))
    kw.update(over)
    return G.Params(**kw)


def _plate(case, rng):
    return GEO.torsional_plate(case["npts"], 1.0, -10.0 + math.degrees(math.asin(0.01 * max(-2.0, min(2.0, rng.standard_normal())))),
                               itheta=0.5 / 3.0, ktheta=1e-3)


def _vorticity(m, n, levels, seed, device="cuda"):
    """Vorticity fields as a shed wake leaves them: Gaussian vortices of both signs, on every level."""
    gen = torch.Generator().manual_seed(int(seed))
    k = 24
    cx, cy = torch.rand(k, generator=gen, dtype=torch.float64) * 6 - 0.5, torch.rand(k, generator=gen, dtype=torch.float64) * 2 - 1
    r, s = 0.05 + 0.25 * torch.rand(k, generator=gen, dtype=torch.float64), torch.randn(k, generator=gen, dtype=torch.float64)
    out = torch.zeros((levels, n - 1, m - 1), dtype=torch.float64, device=device)
    d = 8.0 / m
    for l in range(levels):
        h = d * 2 ** l
        x = ((torch.arange(1, m, dtype=torch.float64, device=device) - m // 2) * h + (m // 2) * d - 1.0)[None, :]
        y = ((torch.arange(1, n, dtype=torch.float64, device=device) - n // 2) * h)[:, None]
        for a, b, c, g in zip(cx.tolist(), cy.tolist(), r.tolist(), s.tolist()):
            out[l] += (g * h * h) * torch.exp(-((x - a) ** 2 + (y - b) ** 2) / (2 * c * c))
    return out


def _run_in(sim, steps=3):
    """The first steps of a run: the influence band, the factorised matrix and the step's graphs are made."""
    for _ in range(steps):
        sim.advance()


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(int(seed))
    m, n, L = case["m"], case["n"], case["levels"]
    st = dict(kind=kind, case=case)
    if kind == "vort2flux":
        st["sim"] = G.Simulation(_params(case, rng))
        st["w"] = _vorticity(m, n, L, seed)
        st["s"] = torch.zeros_like(st["w"])
        st["qx"] = torch.zeros((L, n, m + 1), dtype=torch.float64, device="cuda")
        st["qy"] = torch.zeros((L, n + 1, m), dtype=torch.float64, device="cuda")
        return st
    if kind in ("poisson", "viscous"):
        st["sim"] = G.Simulation(_params(case, rng))
        st["w"] = _vorticity(m, n, 1, seed)[0]
        st["s"] = torch.zeros_like(st["w"])
        if kind == "viscous":
            st["rhs"], st["old"] = _vorticity(m, n, 1, seed + 1)[0], _vorticity(m, n, 1, seed + 2)[0]
            st["bc"] = torch.zeros_like(st["w"])
        return st
    if kind == "batch":
        runs = []
        for i in range(case["sims"]):
            mi, ni = ((m, n), (near_grid(m, 3, 2), near_grid(n, 3, 2)), (2 * m, 2 * n))[i % 3]
            length = (0.75, 1.0, 1.25)[(i // 3) % 3]
            mass = math.exp(rng.uniform(math.log(0.1), math.log(2.0)))
            c = dict(case, m=mi, n=ni, re=rng.uniform(100.0, 500.0))
            body = GEO.torsional_plate(int(round(length * mi / 16.0)) + 1, length, -rng.uniform(0.0, 20.0),
                                       itheta=mass * length ** 3 / 3.0, ktheta=math.exp(rng.uniform(math.log(1e-4), math.log(1e-2))))
            runs.append((_params(c, rng), [body]))
        b = G.Batch(runs)
        for _ in range(3):
            b.advance()
        st["batch"] = b
        st["omega"] = torch.zeros(sum(s.ns for s in b.sims), dtype=torch.float64, device="cuda")
        return st
    if kind == "adjoint":
        p = _params(case, rng, len=6.0, offsetx=1.5, offsety=3.0 * n / m, num_stat=True, motion=(-1.0, 0.0, 0.0, 0.25, 0.0))
        x, y = GEO.naca00(12.0, ds=2.0 * p.len / p.m)
        sim = G.Simulation(p, [G.Body(x=x, y=y, fam=1)])
        N = case["steps"]
        t = p.dt * np.arange(1, N + 1)
        arg = 2.0 * math.pi * 0.2 * t + rng.uniform(-0.2, 0.2)
        al, ald = math.radians(10.0) * np.sin(arg), math.radians(10.0) * 2.0 * math.pi * 0.2 * np.cos(arg)
        st.update(sim=sim, frames=np.stack([-np.cos(al), -np.sin(al), -ald], axis=1), dforces=rng.uniform(-1.0, 1.0, (N, 1, 2)) / N)
        _run_in(sim)
        return st
    if kind == "cylinder":
        sim = G.Simulation(_params(case, rng, num_stat=True, offsetx=2.0), [GEO.cylinder(case["npts"])])
    elif kind == "beam":
        p = _params(case, rng)
        sim = G.Simulation(p, [GEO.beam_plate(case["npts"], 1.0, 10.0 + rng.uniform(-1.0, 1.0), 0.5, 1e-3)])
    else:
        # the sizes that the framework is quoted on and larger ones are run long enough to tune their launch shapes
        sim = G.Simulation(_params(case, rng, autotune=(kind == "plate" and m >= 800)), [_plate(case, rng)])
    if kind == "subdomain":
        d = 8.0 / m
        sim.subdomain_setup(-6 * d, 1.0 + 6 * d, -0.3, 0.3, d)   # the region the plate sweeps
    if kind == "schur":
        st["x"] = torch.from_numpy(rng.standard_normal(sim.nf)).cuda()
        st["y"] = torch.zeros_like(st["x"])
    else:
        _run_in(sim)
    if kind == "pressure":
        st["p"] = torch.zeros((L, n, m), dtype=torch.float64, device="cuda")
    elif kind != "schur":
        st["omega"] = torch.zeros((L, n - 1, m - 1), dtype=torch.float64, device="cuda")
    st["sim"] = sim
    return st


def near_grid(v, num, den):
    return min(_smooth(2000), key=lambda s: abs(s - v * num / den))


def _call(name, *args):
    G._check(getattr(G.load(), name)(*args), name)


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        for _ in range(state["case"]["steps"]):
            b.advance()
        at = 0
        for s in b.sims:
            _call("ib_get_field", s.h, G.FIELDS["omega"], 0, G._ptr(state["omega"][at:at + s.ns]))
            at += s.ns
        return {"omega": state["omega"], "f": np.concatenate([s.get_vector("f") for s in b.sims]),
                "theta": np.concatenate([s.body_state()[0] for s in b.sims])}
    sim = state["sim"]
    if kind == "vort2flux":
        _call("ib_vort2flux", sim.h, *(G._ptr(state[k]) for k in ("w", "s", "qx", "qy")))
        return {k: state[k] for k in ("w", "s", "qx", "qy")}
    if kind == "poisson":
        _call("ib_ctci", sim.h, G._ptr(state["w"]), G._ptr(state["s"]))
        return state["s"]
    if kind == "viscous":
        state["s"].copy_(state["w"])
        torch.cuda.current_stream().synchronize()   # the library runs on its own stream
        _call("ib_fluid_predictor", sim.h, 0, *(G._ptr(state[k]) for k in ("s", "rhs", "old", "bc")))
        return state["s"]
    if kind == "schur":
        _call("ib_schur_apply", sim.h, G._ptr(state["x"]), G._ptr(state["y"]))
        return state["y"]
    if kind == "pressure":
        _call("ib_calculate_pressure", sim.h, G._ptr(state["p"]))
        return state["p"]
    if kind == "adjoint":
        forces = sim.adjoint_forward(state["frames"], state["case"]["keep"])
        return {"forces": forces, "dframes": sim.adjoint_backward(state["dforces"])}
    force, theta = [], []
    for _ in range(state["case"]["steps"]):
        sim.advance()
        force.append(sim.forces())
        if sim.ntors:
            theta.append(sim.body_state()[0])
        elif sim.beam_dofs:
            theta.append(sim.beam_state()[0])
    for l in range(state["case"]["levels"]):
        _call("ib_get_field", sim.h, G.FIELDS["omega"], l, G._ptr(state["omega"][l]))
    return {"force": np.array(force), "state": np.array(theta), "omega": state["omega"], "f": sim.get_vector("f")}


def work(case):
    """Bytes: every field of the state read once and written once by each step (or operand by an
    operator call).  Operations: two transforms along x and a solve along y for each spectral solve,
    and the stencils."""
    kind, m, n, L = case["kind"], case["m"], case["n"], case["levels"]
    ns, nu, nv = (m - 1) * (n - 1), n * (m + 1), (n + 1) * m
    solve = ns * (2 * 2.5 * math.log2(m) + 5.0)   # operations of one spectral solve of one level
    if kind in ("poisson", "viscous"):
        return dict(bytes=8.0 * ns * (2 if kind == "poisson" else 5), flops=solve)
    if kind == "vort2flux":
        return dict(bytes=8.0 * L * (2 * ns + nu + nv), flops=L * solve)
    if kind == "schur":
        return dict(bytes=8.0 * 2 * case["npts"] * 2, flops=(L + 1) * solve)
    if kind == "pressure":
        return dict(bytes=8.0 * L * (ns + 2 * nu + 2 * nv + m * n), flops=L * (solve + 20.0 * m * n))
    step_bytes = 8.0 * L * (2 * (3 * ns + nu + nv) + nu + nv)
    step_flops = L * (3 * solve + 40.0 * ns) + solve
    if kind == "adjoint":   # a forward, its recomputation, and the reverse of twice a step's work
        return dict(bytes=4.0 * case["steps"] * step_bytes, flops=4.0 * case["steps"] * step_flops)
    if kind == "batch":
        per = sum((1.0, 2.25, 4.0)[i % 3] for i in range(case["sims"]))
        return dict(bytes=per * case["steps"] * step_bytes, flops=per * case["steps"] * step_flops)
    return dict(bytes=case["steps"] * step_bytes, flops=case["steps"] * step_flops)


# ---------------------------------------------------------------------------------------------
def _sines(M):
    """The (M-1) x (M-1) matrix 2 sin(pi j k / M), its angles reduced before the sine."""
    j = np.arange(1, M, dtype=np.int64)
    return 2.0 * np.sin(np.pi * ((j[:, None] * j[None, :]) % (2 * M)) / M)


def _laplace(m, n):
    i, j = np.arange(1, m)[None, :], np.arange(1, n)[:, None]
    return 4.0 * np.sin(0.5 * np.pi * i / m) ** 2 + 4.0 * np.sin(0.5 * np.pi * j / n) ** 2


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("vort2flux", "poisson", "viscous"):
        return None   # whole steps and solves: nothing short stands for them
    m, n, L = case["m"], case["n"], case["levels"]
    sx, sy, lam, norm = _sines(m), _sines(n), _laplace(m, n), 4.0 * m * n

    def dst(a):
        return sy @ a @ sx

    if kind == "poisson":
        w = _vorticity(m, n, 1, seed)[0].cpu().numpy()
        return dst(dst(w) / lam / norm)
    if kind == "viscous":
        w, r, o = (_vorticity(m, n, 1, seed + k)[0].cpu().numpy() for k in range(3))
        dt, re, d2 = case.get("dt", 1e-3), case.get("re", 100.0), (8.0 / m) ** 2
        c = 0.5 * dt * lam / d2 / re
        inner = dst((1.5 * r - 0.5 * o) * (dt / d2 / norm))
        return dst((inner + (1.0 - c) / norm * dst(w)) / (1.0 + c))
    w = _vorticity(m, n, L, seed).cpu().numpy()
    for k in range(1, L):   # full weighting of the finer level onto the centre of the coarser one
        f = w[k - 1]
        g = f[1:-1, :][::2] + 0.5 * (f[:-2, :][::2] + f[2:, :][::2])
        w[k, n // 4:3 * n // 4 - 1, m // 4:3 * m // 4 - 1] = g[:, 1:-1][:, ::2] + 0.5 * (g[:, :-2][:, ::2] + g[:, 2:][:, ::2])
    s, qx, qy = np.zeros_like(w), np.zeros((L, n, m + 1)), np.zeros((L, n + 1, m))
    edge = None   # the coarser level's streamfunction on this level's (n+1) x (m+1) boundary vertices
    for k in range(L - 1, -1, -1):
        full = np.zeros((n + 1, m + 1))
        if edge is not None:
            full[:, 0], full[:, m], full[0, :], full[n, :] = edge
        rhs = w[k].copy()
        rhs[:, 0] += full[1:n, 0]
        rhs[:, -1] += full[1:n, m]
        rhs[0, :] += full[0, 1:m]
        rhs[-1, :] += full[n, 1:m]
        s[k] = dst(dst(rhs) / lam / norm)
        full[1:n, 1:m] = s[k]
        qx[k] = full[1:] - full[:-1]
        qy[k] = full[:, :-1] - full[:, 1:]

        def spread(line):
            out = np.empty(2 * len(line) - 1)
            out[::2] = line
            out[1::2] = 0.5 * (line[:-1] + line[1:])
            return out

        edge = (spread(full[n // 4:3 * n // 4 + 1, m // 4]), spread(full[n // 4:3 * n // 4 + 1, 3 * m // 4]),
                spread(full[n // 4, m // 4:3 * m // 4 + 1]), spread(full[3 * n // 4, m // 4:3 * m // 4 + 1]))
    return {"w": w, "s": s, "qx": qx, "qy": qy}
