"""The work a user of this framework has it do, as timed cases.

Kinds of case:

``steps``     integrate() through the drop-in C ABI on the caller's own (pageable) host arrays, one call a time step
              as the reference's main loop makes them: every call reads the state from the host and writes it back.
``run``       a simulation segment on the GPU: the state of a host case is loaded, stepped in the device-resident
              mode and brought back, as a program does between two outputs or restarts.
``ensemble``  a batch of independent bubbles on three grids, stepped together.
``potential`` fluid_compute_potential(), the Poisson solve, called by itself on host arrays.
``curvature`` interface_compute_curvature_tensor(), the interface geometry, called by itself on host arrays.
``train``     epochs of Adam on the learned curvature closure (rows in GPU memory).

Grids, bubble counts and physics are those of the package's own workloads (ic.py) and of its tests' odd sizes: the
64 x 64 static drop, the 256 x 128 bubble, swarms up to 2048 x 1024, the three ensemble grids; ny is a power of two
(a limit of the solver), nx is free.  States start from the exact-area bubbles of the package's generator with a
smooth divergence-free velocity on top, so that no field is uniformly zero.
"""
from __future__ import annotations

import math

import numpy as np

from simplebubblyflowsolver_gb300 import SYNC_NONE, SYNC_STATE, ic, load_library, state_from_fields
from simplebubblyflowsolver_gb300 import learned_curvature as closure
from simplebubblyflowsolver_gb300._abi import SolverState

STATE = ("ux", "uy", "p", "psi0", "vof")
PHYSICS = {
    "drop": dict(Re=math.sqrt(12000.0), We=1.0, Fr=math.inf, denr=1e-3, visr=1e-3),
    "bubble": dict(Re=35.0, We=10.0, Fr=1.0, denr=0.1, visr=0.1),
    "swarm": dict(Re=100.0, We=5.0, Fr=1.0, denr=1e-3, visr=1e-2),
}
# fused minimum of one step: 30 doubles read or written per cell and substage; FP64 operations per cell and step
STEP_BYTES, STEP_FLOPS = 720.0, 540.0


def listed():
    return [
        # the smallest calls: the static-drop grid, integrate() by integrate(); latency and launches count
        dict(name="steps_drop_64x64", kind="steps", flow="drop", nx=64, ny=64, steps=20),
        # the reference's single-bubble case through the drop-in call
        dict(name="steps_bubble_256x128", kind="steps", flow="bubble", nx=256, ny=128, steps=20),
        # the same case as a segment on the GPU, tuned and with the log's quantities at its end
        dict(name="run_bubble_256x128", kind="run", flow="bubble", nx=256, ny=128, steps=100, tune=True, monitor=True),
        # an ordinary swarm on a ragged grid (nx odd), default launch shapes
        dict(name="run_swarm_509x256", kind="run", flow="swarm", nx=509, ny=256, steps=40, tune=False, monitor=True),
        # the learned curvature closure in the step
        dict(name="run_learned_1000x512", kind="run", flow="swarm", nx=1000, ny=512, steps=20, tune=False,
             learned=True),
        # the benchmarked swarm, as bench.py runs it
        dict(name="run_swarm_2048x1024", kind="run", flow="swarm", nx=2048, ny=1024, steps=20, tune=True),
        # the same grid through the drop-in call, the state in host memory at every step
        dict(name="steps_swarm_2048x1024", kind="steps", flow="swarm", nx=2048, ny=1024, steps=8),
        # the largest: a swarm at twice that resolution
        dict(name="run_swarm_4096x2048", kind="run", flow="swarm", nx=4096, ny=2048, steps=6, tune=False),
        # a parameter study: independent bubbles on the three ensemble grids, batched
        dict(name="ensemble_32", kind="ensemble", cases=32, steps=20),
        # operators called one by one (a host program that keeps its own step)
        dict(name="potential_1000x512", kind="potential", nx=1000, ny=512),
        dict(name="curvature_300x256", kind="curvature", nx=300, ny=256),
        # training the closure: one epoch of 1024-row batches
        dict(name="train_65536", kind="train", rows=65536, batch=1024, epochs=1),
    ]


def _grid(rng, most):
    """a grid of at most `most` cells: ny a power of two, nx anything"""
    while True:
        ny = 1 << rng.randint(5, 11)
        nx = int(round(math.exp(rng.uniform(math.log(24), math.log(4096)))))
        if nx * ny <= most and ny / 6 <= nx <= 6 * ny:
            return nx, ny


def draw(rng):
    kind = rng.choice(("run", "run", "run", "steps", "steps", "ensemble", "potential", "curvature", "train"))
    if kind == "run":
        nx, ny = _grid(rng, 4096 * 2048)
        steps = max(2, min(rng.randint(8, 48), int(5e7 / (nx * ny))))
        return dict(kind=kind, flow=rng.choice(("swarm", "swarm", "bubble")), nx=nx, ny=ny, steps=steps,
                    tune=rng.random() < 0.3, monitor=rng.random() < 0.5, learned=rng.random() < 0.2)
    if kind == "steps":
        nx, ny = _grid(rng, 2048 * 1024)
        return dict(kind=kind, flow=rng.choice(("swarm", "bubble")), nx=nx, ny=ny,
                    steps=2 * rng.randint(4, 8))
    if kind == "ensemble":
        return dict(kind=kind, cases=rng.randint(3, 32), steps=rng.randint(5, 20))
    if kind in ("potential", "curvature"):
        nx, ny = _grid(rng, 2048 * 1024)
        return dict(kind=kind, nx=nx, ny=ny)
    return dict(kind=kind, rows=rng.randint(8192, 131072), batch=rng.choice((256, 512, 1000, 1024, 1024, 2048)),
                epochs=1)


# ------------------------------------------------------------------ inputs
def _lengths(nx, ny):
    """square cells; lx at most 4 (on longer domains the rounding of the x faces passes the solver's uniform-grid
    test no more)"""
    ly = min(2.0, 4.0 * ny / nx)
    return ly * nx / ny, ly


def _discs(rng, flow, nx, ny, lx, ly):
    h = ly / ny
    if flow in ("drop", "bubble"):
        r = 0.25 * min(lx, ly) * rng.uniform(0.9, 1.0)
        return [(0.5 * min(lx, ly) + 0.02 * rng.uniform(-1, 1), 0.5 * ly + 0.05 * rng.uniform(-1, 1), r)]
    rlo, rhi = max(0.05, 5 * h), max(0.10, 8 * h)
    want = max(1, int(round(64 * (lx * ly / 8.0) * (0.075 / (0.5 * (rlo + rhi))) ** 2)))
    out = []
    for _ in range(200 * want):
        r = rng.uniform(rlo, rhi)
        if lx < 2 * r + 4 * h or ly < 2 * r + 4 * h:
            r = 0.2 * min(lx, ly)
        cx, cy = rng.uniform(r + 2 * h, lx - r - 2 * h), rng.uniform(0.0, ly)
        if all(math.hypot(cx - ox, min(abs(cy - oy), ly - abs(cy - oy))) >= r + ro + 2 * h for ox, oy, ro in out):
            out.append((cx, cy, r))
            if len(out) == want:
                break
    return out


def _fields(rng, flow, nx, ny, lx=None, ly=None):
    """an initial condition in the package's .npy schema: exact-area bubbles, the velocity of a smooth stream
    function that vanishes with its slope at the walls (discretely divergence-free), zero pressure"""
    if lx is None:
        lx, ly = _lengths(nx, ny)
    wl = ic.Workload(flow, nx, ny, lx, ly, _discs(rng, flow, nx, ny, lx, ly), **PHYSICS[flow])
    f = wl.fields()
    amp = 0.02 if flow == "drop" else 0.2
    xs = np.linspace(0.0, 1.0, nx + 1)
    ys = np.arange(ny + 1) / ny
    sx = np.sin(math.pi * xs) ** 2
    sy = sum(rng.uniform(0.3, 1.0) / k * np.cos(2 * math.pi * (k * ys + rng.uniform())) for k in (1, 2, 3))
    sy[-1] = sy[0]
    scale = amp * ly / (2 * math.pi)
    hx, hy = lx / nx, ly / ny
    f["ux"][:] = scale / hy * (sy[1:] - sy[:-1])[:, None] * sx[None, :]
    f["uy"][:, 1:-1] = -scale / hx * sy[:-1, None] * (sx[1:] - sx[:-1])[None, :]
    return f


def _state(lib, fields, phys):
    st = state_from_fields(fields, **phys)
    lib.apply_initial_boundaries(st)
    return st


def _weights():
    """parameters of the closure; the same for every input, as a program trains them once"""
    return closure.init_params(0)


# the ensemble's cases and their physics: one batch a program sets up once (the library keeps a batch by its cases)
_batches = {}


def _batch(lib, n):
    if n not in _batches:
        _batches[n] = [_state(lib, wl.fields(), dict(Re=wl.Re, We=wl.We, Fr=wl.Fr, denr=wl.denr, visr=wl.visr))
                       for wl in ic.ensemble(n, seed=0)]
    return _batches[n]


def _point(to, at):
    """the structs of `to` take the arrays of `at` (a dict of array addresses)"""
    for s in STATE + ("psi1",):
        to._array_t(s).data = at[s]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    lib = load_library()
    if kind in ("steps", "run"):
        phys = PHYSICS[case["flow"]]
        st = _state(lib, _fields(rng, case["flow"], case["nx"], case["ny"]), phys)
        s = dict(case=case, lib=lib, st=st)
        if kind == "run":
            s["out"] = SolverState(st.nx, st.ny, st.lx, st.ly, xf=st.xf, xc=st.xc, **phys)
            if case.get("learned"):
                lib.mlp_set_params(_weights())
        elif case["nx"] * case["ny"] <= 1 << 18:
            s["start"] = st.snapshot(STATE)
        return s
    if kind == "ensemble":
        own = []
        for st in _batch(lib, case["cases"]):
            ph = dict(Re=st.fluid.Re, We=st.interface.We, Fr=st.fluid.Fr, denr=st.fluid.denr, visr=st.fluid.visr)
            new = _state(lib, _fields(rng, "bubble", st.nx, st.ny, st.lx, st.ly), ph)
            own.append(new)
        return dict(case=case, lib=lib, own=own, at=[{s: o._array_t(s).data for s in STATE + ("psi1",)} for o in own])
    if kind in ("potential", "curvature"):
        phys = PHYSICS["swarm"]
        f = _fields(rng, "swarm", case["nx"], case["ny"])
        st = _state(lib, f, phys)
        if kind == "potential":
            # a predicted velocity (not divergence-free), the density of the bubbles and the last potential
            _potential_inputs(rng, st, phys)
        return dict(case=case, lib=lib, st=st, dt=(1.3e-4, 2.1e-4))
    import torch
    x, y = closure.dataset(case["rows"] // 8 + 200, seed=seed)
    x, y = x[:case["rows"]], y[:case["rows"]]
    perm = rng.permutation(x.shape[0]).astype(np.int32)
    dev = "cuda:0"
    return dict(case=case, lib=lib, p0=closure.init_params(seed), n=x.shape[0],
                X=torch.from_numpy(x).to(dev).to(torch.bfloat16), Y=torch.from_numpy(y).to(dev),
                perm=torch.from_numpy(perm).to(dev))


def _smooth(rng, ny, nx):
    y, x = np.arange(ny) / ny, (np.arange(nx) + 0.5) / nx
    out = np.zeros((ny, nx))
    for k in (1, 2, 5):
        out += np.outer(np.cos(2 * math.pi * (k * y + rng.uniform())), np.cos(math.pi * k * x)) / k
    return out


def _potential_inputs(rng, st, phys):
    ny, nx = st.ny, st.nx
    st.interior_rows("ux")[:, 1:-1] += 0.05 * _smooth(rng, ny, nx)[:, 1:] + 0.01 * rng.standard_normal((ny, nx - 1))
    st.interior_rows("uy")[:, 1:-1] += 0.05 * _smooth(rng, ny, nx) + 0.01 * rng.standard_normal((ny, nx))
    den = 1.0 + (phys["denr"] - 1.0) * st.interior_rows("vof")
    psi = np.zeros((ny, nx + 2))
    psi[:, 1:-1] = 1e-4 * _smooth(rng, ny, nx)
    psi[:, 0], psi[:, -1] = psi[:, 1], psi[:, -2]
    for slot, rows in (("den1", den), ("psi0", psi), ("ux", st.interior_rows("ux").copy()),
                       ("uy", st.interior_rows("uy").copy())):
        a = st.field(slot)
        a[1:-1] = rows
        a[0], a[-1] = rows[-1], rows[0]


# --------------------------------------------------------------------- run
def _settings(lib, case, sync):
    lib.set_sync_mode(sync)
    lib.set_dt_coefs(0.4, 0.5, 0.95)
    lib.set_autotune(bool(case.get("tune")))
    lib.set_curvature_model(1 if case.get("learned") else 0)


def run(state):
    case, lib = state["case"], state["lib"]
    kind = case["kind"]
    if kind == "steps":
        st = state["st"]
        _settings(lib, case, SYNC_STATE)
        # a small case starts over (thousands of passes are made of it); a large one goes on from where it stands
        for s, a in state.get("start", {}).items():
            st.field(s)[...] = a
        dt = [lib.integrate(st) for _ in range(case["steps"])]
        return dict({s: st.interior_rows(s) for s in STATE}, dt=np.array(dt))
    if kind == "run":
        st, out = state["st"], state["out"]
        _settings(lib, case, SYNC_NONE)
        lib.invalidate_device()
        _, dt = lib.run_steps_timed(st, case["steps"])
        got = {}
        if case.get("monitor"):
            d = lib.diagnostics(st)
            got["log"] = np.array([d[k] for k in ("vof_max", "vof_integral", "volume", "interface_area", "energy_x",
                                                  "energy_y", "umax", "vmax")])
        lib.sync_to_host(out)
        lib.set_curvature_model(0)
        return dict({s: out.interior_rows(s) for s in STATE}, dt=dt, **got)
    if kind == "ensemble":
        batch, at = _batch(lib, case["cases"]), state["at"]
        _settings(lib, case, SYNC_STATE)
        for st, a in zip(batch, at):
            _point(st, a)
        dts = lib.integrate_batch(batch)  # the first step takes the state from the host arrays
        lib.set_sync_mode(SYNC_NONE)
        lib.run_batch_steps_timed(case["steps"] - 1)
        lib.batch_sync_to_host(batch)
        for st, o, a in zip(batch, state["own"], at):
            for s in STATE + ("psi1",):
                a[s] = o._array_t(s).data = st._array_t(s).data
        return {"dts": dts, **{s: np.concatenate([o.interior_rows(s).ravel() for o in state["own"]]) for s in STATE}}
    if kind == "potential":
        st = state["st"]
        lib.compute_potential(st, *state["dt"])
        return st.interior_rows("psi1")[:, 1:-1]
    if kind == "curvature":
        st = state["st"]
        lib.compute_curvature_tensor(st)
        return dict(dvof=st.interior_rows("dvof"), normal=st.interior_rows("normal"),
                    curv=st.interior_rows("curv")[:, 1:-1])
    lib.mlp_set_params(state["p0"])
    loss = [lib.mlp_train_epoch(state["X"].data_ptr(), state["Y"].data_ptr(), state["perm"].data_ptr(), state["n"],
                                case["batch"], 2e-3) for _ in range(case["epochs"])]
    return dict(params=lib.mlp_get_params(), loss=np.array(loss, dtype=np.float32))


# -------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(w.cells for w in ic.ensemble(case["cases"], seed=0))
        return {"bytes": cells * (STEP_BYTES * case["steps"] + 11 * 8.0), "flops": cells * STEP_FLOPS * case["steps"]}
    if kind == "train":
        n = case["rows"] * case["epochs"]
        # 16-64-64-1: forward, and backward twice that; rows read once, the index with them
        return {"bytes": n * (2 * 16 + 4 + 4.0), "flops": n * 6.0 * (16 * 64 + 64 * 64 + 64)}
    cells = case["nx"] * case["ny"]
    if kind == "steps":  # five fields in and six out at every step
        return {"bytes": cells * case["steps"] * (STEP_BYTES + 11 * 8.0), "flops": cells * STEP_FLOPS * case["steps"]}
    if kind == "run":
        return {"bytes": cells * (STEP_BYTES * case["steps"] + 11 * 8.0), "flops": cells * STEP_FLOPS * case["steps"]}
    if kind == "potential":
        return {"bytes": cells * 8.0 * 5, "flops": cells * (5.0 * math.log2(case["ny"]) + 30)}
    return {"bytes": cells * 8.0 * 7, "flops": cells * 20.0}


# ------------------------------------------------------- values in 64 bits
def exact(case, seed):
    if case["kind"] == "potential":
        return _exact_potential(prepare(case, seed))
    if case["kind"] == "curvature":
        return _exact_curvature(prepare(case, seed)["st"])
    return None  # whole steps and training have no closed form short of a second solver


def _exact_potential(s):
    """rho_ref / dt_new div u - dt_old / dt_new div((rho_ref / rho - 1) grad psi_old) as the right-hand side, the
    five-point operator (walls in x, periodic in y) inverted by a transform in y and elimination in x; zero mean"""
    st, (dt_old, dt_new) = s["st"], s["dt"]
    nx, ny, hx, hy = st.nx, st.ny, st.lx / st.nx, st.hy
    ref = st.fluid.refden
    ux, uy = st.interior_rows("ux"), st.interior_rows("uy")[:, 1:-1]
    den, psi = st.interior_rows("den1"), st.interior_rows("psi0")
    div = (ux[:, 1:] - ux[:, :-1]) / hx + (np.roll(uy, -1, 0) - uy) / hy
    ex = (ref / (0.5 * (den[:, 1:] + den[:, :-1])) - 1.0) * (psi[:, 1:] - psi[:, :-1]) / hx
    dc, pc = den[:, 1:-1], psi[:, 1:-1]
    ey = (ref / (0.5 * (dc + np.roll(dc, 1, 0))) - 1.0) * (pc - np.roll(pc, 1, 0)) / hy
    rhs = ref / dt_new * div - dt_old / dt_new * ((ex[:, 1:] - ex[:, :-1]) / hx + (np.roll(ey, -1, 0) - ey) / hy)
    q = np.fft.rfft(rhs, axis=0)
    lam = -(2.0 / hy * np.sin(np.pi * np.arange(ny // 2 + 1) / ny)) ** 2
    out = np.empty_like(q)
    # the mean mode: two sums
    d = np.cumsum(q[0].real) * hx * hx
    z = np.concatenate(([0.0], np.cumsum(d[:-1])))
    out[0] = z - z.mean()
    # the others: elimination along x, all wavenumbers at once
    off = 1.0 / (hx * hx)
    c, r = np.empty((nx, ny // 2)), np.empty((nx, ny // 2), dtype=complex)
    for i in range(nx):
        diag = lam[1:] - (off if i in (0, nx - 1) else 2.0 * off)
        piv = diag - (off * c[i - 1] if i else 0.0)
        c[i] = off / piv
        r[i] = (q[1:, i] - (off * r[i - 1] if i else 0.0)) / piv
    for i in range(nx - 2, -1, -1):
        r[i] -= c[i] * r[i + 1]
    out[1:] = r.T
    return np.fft.irfft(out, n=ny, axis=0)


def _exact_curvature(st):
    """unit corner gradients of vof (summed in the reference's order), the cell normal and intercept of interface
    cells (0 elsewhere: the arrays start at zero) and kappa = -div n"""
    hx, hy, eps = st.lx / st.nx, st.hy, np.finfo(np.float64).eps
    v = st.interior_rows("vof")
    a, b = np.roll(v, 1, 0)[:, :-1], np.roll(v, 1, 0)[:, 1:]
    c, d = v[:, :-1], v[:, 1:]
    gx = (((-a + b) - c) + d) / st.hxxf[None, :]
    gy = (((-a - b) + c) + d) / hy
    inv = 1.0 / np.maximum(np.sqrt(gx * gx + gy * gy), eps)
    dv = np.stack((gx * inv, gy * inv), axis=-1)
    up = np.roll(dv, -1, 0)
    d00, d10, d01, d11 = dv[:, :-1], dv[:, 1:], up[:, :-1], up[:, 1:]
    curv = -(0.5 / hx * ((d10[..., 0] + d11[..., 0]) - (d00[..., 0] + d01[..., 0]))
             + 0.5 / hy * ((d01[..., 1] + d11[..., 1]) - (d00[..., 1] + d10[..., 1])))
    phi = v[:, 1:-1]
    m = (((d00 + d10) + d01) + d11) / np.array([hx, hy])
    inv = 1.0 / np.maximum(np.sqrt((m ** 2).sum(-1)), eps)
    itf = (phi >= 1e-8) & (phi <= 1 - 1e-8)
    p = np.where(itf, phi, 0.5)
    normal = np.concatenate((m * inv[..., None], (-0.5 * np.log(1.0 / p - 1.0))[..., None]), axis=-1)
    return dict(dvof=dv, normal=np.where(itf[..., None], normal, 0.0), curv=curv)
