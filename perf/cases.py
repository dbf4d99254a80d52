"""Performance cases of the framework: what a user's program has it do, through the
public classes (Solver2D, CompressedSolver, Ensemble, CalibrationLoss), from a single
call on a few thousand cells to output intervals on tens of millions.

A pass advances a simulation by one output interval: `steps` CFL steps from where the
last pass left it (the calibration case restarts, as an optimiser's evaluation does).
Inputs are made on the GPU from a seed: fractal terrain with ponds, a wet film on the
lower slopes and dry ground above, a dam on a flat bed, or a tidal basin. `exact`
restates the same scheme in plain torch, binary64.
"""
from __future__ import annotations

import math
import warnings

import numpy as np
import torch

from geoswe_b200 import Config, Mesh2D, RainfallForcing, Solver2D, StageBoundary
from geoswe_b200.adjoint import CalibrationLoss, FlatAdjoint, Inlet
from geoswe_b200.compressed import CompressedSolver
from geoswe_b200.ensemble import Ensemble

G = 9.81
NGH = 2
FAR = 1.0e12                      # an end time no pass reaches: the step count ends it
MANNING = np.array([0.025, 0.04, 0.06, 0.1])
RAIN_MM_H = 50.0

DENSE = dict(kind="dense", scene="terrain", dtype="float32", arith="exact", bc="open", friction="table",
             rain="uniform", stage=False, inlet=False, masked=False)
FLAT = dict(kind="flat", scene="terrain", arith="exact", frac=0.6, rain="uniform", ring=False, inlet=False,
            forcings=False)


def listed():
    return [
        # a program that steps by itself and looks at the state after each step (a coupled
        # model, a callback): one call of step() on a small grid
        dict(DENSE, name="one step 96x80", kind="step", nx=96, ny=80, steps=1),
        # the classic verification run, small enough that launches and latency count
        dict(DENSE, name="dam break 512x512", scene="dam", nx=512, ny=512, steps=100, bc="wall", friction="none",
             rain="none"),
        # a street-block or small-catchment flood model, odd sizes
        dict(DENSE, name="rain 1000x777", nx=1000, ny=777, steps=50),
        # the pluvial flood map of a city, the configuration the throughput is quoted on
        dict(DENSE, name="rain 8192x8192", nx=8192, ny=8192, steps=8),
        # a screening run with the opt-in fast arithmetic
        dict(DENSE, name="fast rain 3000x4096", nx=3000, ny=4096, steps=16, arith="fast"),
        # a binary64 run, periodic in both directions, roughness as a field
        dict(DENSE, name="binary64 733x1021", nx=733, ny=1021, steps=24, dtype="float64", bc="periodic",
             friction="field", rain="none"),
        # an estuary: masked domain, tidal stage cells, a river inlet, radar rain, roughness field
        dict(DENSE, name="estuary 900x650", nx=900, ny=650, steps=40, bc="extrapolate", friction="field",
             rain="gridded", stage=True, inlet=True, masked=True),
        # a catchment on the compressed mesh: only the cells that can flood are stored
        dict(FLAT, name="catchment 2048x2048", nx=2048, ny=2048, steps=20),
        # a tidal basin, wet everywhere, on the compressed mesh
        dict(FLAT, name="tidal basin 5000x6000", scene="tidal", nx=5000, ny=6000, steps=6, frac=1.0, rain="none",
             ring=True),
        # compound flooding: infiltration, Green-Ampt and drain, sponge, clamp, a river inlet
        dict(FLAT, name="compound flood 1024x900", nx=1024, ny=900, steps=30, inlet=True, forcings=True),
        # an uncertainty ensemble of uneven members
        dict(kind="ensemble", name="ensemble of 8", members=8, lo=128, hi=1024, steps=48),
        # one loss and gradient evaluation of a calibration
        dict(kind="adjoint", name="calibration 512x512", nx=512, ny=512, steps=48, window=16, snapshots=12),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "dense", "dense", "dense", "flat", "flat", "ensemble", "adjoint"])
    if kind == "step":
        return dict(DENSE, kind="step", nx=size(24, 700), ny=size(24, 700), steps=1,
                    rain=rng.choice(["none", "uniform"]), friction=rng.choice(["none", "table"]))
    if kind == "dense":
        dtype = rng.choice(["float32", "float32", "float64"])
        arith = "fast" if dtype == "float32" and rng.random() < 0.3 else "exact"
        masked = rng.random() < 0.3
        c = dict(DENSE, nx=size(64, 4096), ny=size(64, 4096), steps=rng.randint(8, 48), dtype=dtype, arith=arith,
                 bc=rng.choice(["open", "wall", "periodic", "extrapolate"]),
                 friction=rng.choice(["table", "table", "field"]),
                 rain=rng.choice(["none", "uniform", "uniform", "gridded"]), masked=masked,
                 stage=masked and rng.random() < 0.5)
        if rng.random() < 0.2:
            c.update(scene="dam", friction="none", rain="none", masked=False, stage=False)
        return c
    if kind == "flat":
        if rng.random() < 0.3:
            return dict(FLAT, scene="tidal", nx=size(200, 3000), ny=size(200, 3000), steps=rng.randint(6, 30),
                        frac=1.0, rain="none", ring=True, arith=rng.choice(["exact", "fast"]))
        forced = rng.random() < 0.3
        return dict(FLAT, nx=size(128, 3000), ny=size(128, 3000), steps=rng.randint(6, 30),
                    frac=round(rng.uniform(0.3, 0.9), 2), rain=rng.choice(["none", "uniform", "gridded"]),
                    forcings=forced, inlet=forced or rng.random() < 0.3,
                    arith="exact" if forced else rng.choice(["exact", "exact", "fast"]))
    if kind == "ensemble":
        return dict(kind="ensemble", members=rng.randint(2, 12), lo=96, hi=rng.choice([384, 768, 1200]),
                    steps=rng.randint(8, 48))
    n = rng.randint(16, 48)
    return dict(kind="adjoint", nx=size(96, 640), ny=size(96, 640), steps=n, window=rng.randint(4, n),
                snapshots=rng.randint(4, 16))


# ------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(shape, gen):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)


def _quantile(x, p):
    """Quantile of a field from a regular sample of it (torch.quantile is limited in size)."""
    v = x.reshape(-1)
    return torch.quantile(v[:: max(1, v.numel() // 500_000)], p)


def _terrain(nx, ny, dx, gen):
    """Fractal bed (spectrum k^-3) with a slope along x; relief grows with the extent."""
    f = torch.fft.rfft2(_randn((nx, ny), gen))
    kx = torch.fft.fftfreq(nx, device="cuda")[:, None]
    ky = torch.fft.rfftfreq(ny, device="cuda")[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    f *= k ** -1.5
    f[0, 0] = 0.0
    z = torch.fft.irfft2(f, s=(nx, ny))
    del f, k
    z -= z.min()
    z *= 40.0 * math.sqrt(min(nx, ny) / 8192.0) / float(z.max())
    z += 0.002 * dx * (torch.arange(nx, device="cuda", dtype=torch.float32)[:, None] + 0.5)
    return z


def _scene(c, gen, dx):
    """(bed, state (3, nx, ny)) in binary32. A compressed mesh is a place: its terrain, and
    so its stored cells, belong to the case; the water on it to the seed."""
    nx, ny = c["nx"], c["ny"]
    q = torch.zeros((3, nx, ny), device="cuda")
    if c["scene"] == "dam":
        i = torch.arange(nx, device="cuda")[:, None] - (nx - 1) / 2.0
        j = torch.arange(ny, device="cuda")[None, :] - (ny - 1) / 2.0
        h = torch.where(torch.hypot(i, j) < min(nx, ny) / 8.0, 2.0, 0.5).to(torch.float32)
        q[0] = h * (1.0 + 0.002 * _randn((nx, ny), gen))
        return torch.zeros((nx, ny), device="cuda"), q
    if c["scene"] == "tidal":
        x = (torch.arange(nx, device="cuda", dtype=torch.float64) + 0.5) * dx
        y = (torch.arange(ny, device="cuda", dtype=torch.float64) + 0.5) * dx
        z = (0.5 * torch.sin(2 * math.pi * x / 2000.0)[:, None] * torch.cos(2 * math.pi * y / 1500.0)[None, :]).float()
        q[0] = (1.5 + 0.01 * _randn((nx, ny), gen) - z).clamp_min(0.0)
        return z, q
    z = _terrain(nx, ny, dx, _gen(4099 * nx + ny) if c["kind"] == "flat" else gen)
    film = c.get("film", 0.03) * (1.0 + 0.2 * _randn((nx, ny), gen)).clamp_min(0.1)
    q[0] = torch.where(z < _quantile(z, 0.75), film, torch.zeros_like(film))
    q[0] = torch.maximum(q[0], _quantile(z, 0.35) - z)      # ponds in the lower third
    speed = torch.minimum(q[0], torch.full_like(film, 0.5))  # m/s, slower in the film
    a, b = torch.rand(2, generator=gen, device="cuda") * 6.0
    i = torch.arange(nx, device="cuda", dtype=torch.float32)[:, None] * 0.02
    j = torch.arange(ny, device="cuda", dtype=torch.float32)[None, :] * 0.02
    q[1] = q[0] * speed * torch.sin(i + j + a)
    q[2] = q[0] * speed * torch.cos(i - j + b)
    return z, q


def _blocks(nx, ny, n, gen):
    """Land-cover classes on 24 x 24 patches, padded with the ghost layers (uint8)."""
    m = torch.randint(0, n, (nx // 24 + 2, ny // 24 + 2), generator=gen, device="cuda", dtype=torch.uint8)
    return m.repeat_interleave(24, 0)[: nx + 2 * NGH].repeat_interleave(24, 1)[:, : ny + 2 * NGH].contiguous()


def _case_inputs(c, seed):
    """Every input array of a dense or compressed case, on the GPU, from the seed alone."""
    gen = _gen(seed)
    dx = 1.0 if c["scene"] in ("dam", "tidal") else 3.0
    nx, ny = c["nx"], c["ny"]
    d = dict(dx=dx, nx=nx, ny=ny)
    d["z"], d["q"] = _scene(c, gen, dx)
    fr = c.get("friction", "table")
    if c["scene"] == "tidal":
        fr = "scalar"
    if fr == "table":
        d["cls"] = _blocks(nx, ny, len(MANNING), gen)
    elif fr == "field":
        pad = (nx + 2 * NGH, ny + 2 * NGH)
        d["nfield"] = (0.025 + 0.05 * torch.rand(pad, generator=gen, device="cuda")).to(torch.float32)
    d["friction"] = fr
    if c["rain"] == "gridded":
        w = torch.rand((2, nx // 64 + 1, ny // 64 + 1), generator=gen, device="cuda") * 2.0 * RAIN_MM_H
        w = w.repeat_interleave(64, 1)[:, :nx].repeat_interleave(64, 2)[:, :, :ny]
        d["rain"] = w.cpu().numpy().astype(np.float64)
    if c["kind"] == "flat":
        frac = c["frac"]
        d["mask"] = (d["z"] < _quantile(d["z"], frac)) if frac < 1.0 else None
        if d["mask"] is not None:
            d["mask"][:3] = d["mask"][-3:] = False
            d["mask"][:, :3] = d["mask"][:, -3:] = False
            d["q"] *= d["mask"]
    elif c.get("masked"):
        d["mask"] = d["z"] < _quantile(d["z"], 0.9)
    return d


def _rain_forcing(c, d):
    if c["rain"] == "uniform":
        return RainfallForcing(time_s=[0.0, 1.0e9], rate_mm_h=[RAIN_MM_H, RAIN_MM_H])
    if c["rain"] == "gridded":
        return RainfallForcing(time_s=[0.0, 3600.0], rate_mm_h=d["rain"])
    return None


def _config(c, d, **kw):
    bc = {"open": dict(bc_x="wall", bc_y="wall", bc={"x+": "fall"}), "wall": dict(bc_x="wall", bc_y="wall"),
          "periodic": dict(bc_x="periodic", bc_y="periodic"),
          "extrapolate": dict(bc_x="extrapolate", bc_y="extrapolate"),
          "fall": dict(bc_x="fall", bc_y="fall")}[c.get("bc", "fall")]
    fr = d["friction"]
    if fr == "scalar":
        kw["manning_n"] = 0.03
    if fr == "field":
        kw["manning_field"] = d["nfield"]
    return Config(friction=None if fr == "none" else "manning", dtype=c.get("dtype", "float32"), arith=c["arith"],
                  **bc, **kw)


def _stage_cells(c, d):
    """The lowest interior cells of the last twelve rows: an open sea edge."""
    z = d["z"]
    cells = torch.zeros_like(z, dtype=torch.bool)
    cells[-12:] = z[-12:] < _quantile(z[-12:], 0.5)
    return cells


STAGE_T = np.append(np.linspace(0.0, 43200.0, 73), 1.0e13)


def _stage_series(d, cells):
    base = float(d["z"][cells].max())
    return base + 0.2 + 0.5 * np.sin(2 * np.pi * STAGE_T / 44712.0)


INLET_T = np.array([0.0, 1.0e4, 1.0e9])
INLET_Q = np.array([12.0, 40.0, 5.0])


def _dense_inlet(d):
    """A third of the x- edge, as padded (row, columns), with a wet first row."""
    ny = d["ny"]
    return NGH, np.arange(NGH + ny // 3, NGH + ny // 3 + max(2, ny // 8))


def _dense(c, seed):
    d = _case_inputs(c, seed)
    kw = {}
    rf = _rain_forcing(c, d)
    if rf is not None:
        kw["rainfall_forcing"] = rf
    mesh = Mesh2D(nx=c["nx"], ny=c["ny"], dx=d["dx"], dy=d["dx"], ngh=NGH)
    if c["inlet"]:
        d["q"][0, 0] += 0.3
    if c["stage"]:
        cells = _stage_cells(c, d)
        kw["stage_boundary"] = StageBoundary.from_mask(cells.cpu().numpy(), mesh, d["z"].cpu().numpy(),
                                                       STAGE_T, _stage_series(d, cells))
    if d["friction"] == "field":
        kw["manning_n"] = 0.03
    s = Solver2D(mesh, _config(c, d, **kw), d["q"], d["z"])
    if "cls" in d:
        s.set_manning_table(d["cls"], MANNING)
    if "mask" in d:
        s.set_inside_mask(d["mask"])
    if c["inlet"]:
        i, jj = _dense_inlet(d)
        s.add_inflow(np.full(jj.size, i), jj, (1.0, 0.0), d["dx"], INLET_T, INLET_Q)
    return s


# The infiltration, drain and clamp parameters of the compound-flood case, per class.
INFIL = np.array([1.0e-7, 5.0e-7, 1.0e-6, 2.0e-6], np.float32)
KS, PSI, DTH = (np.array(v, np.float32) for v in ([0.0, 1e-6, 3e-6, 6e-6], [0.05, 0.1, 0.2, 0.3], [0.1, 0.2, 0.3, 0.4]))
TAU = 3600.0
CLAMP_H = 1.2


def _pad(x, value=0.0):
    return torch.nn.functional.pad(x, (NGH, NGH, NGH, NGH), value=value)


def _compound(d):
    """Sponge on the last 20 rows, soil classes, drained cells and clamped cells (padded)."""
    pad = (d["nx"] + 2 * NGH, d["ny"] + 2 * NGH)
    keep = torch.ones(pad, device="cuda")
    keep[-22:] = 0.98
    inv_tau = torch.zeros(pad, device="cuda")
    inv_tau[pad[0] // 4: pad[0] // 2] = 1.0 / TAU
    clamp = torch.zeros(pad, dtype=torch.bool, device="cuda")
    clamp[NGH + 4:NGH + 40, NGH + 4:-NGH - 4] = True
    return dict(keep=keep, inv_tau=inv_tau, clamp=clamp)


def _flat_inlet(cs):
    """A run of ring cells whose first active neighbours are the wettest, one normal."""
    g, a = cs.ghost_boundary_pairs()
    ij = cs.ij_active
    n = ij[a] - ij[g]
    east = np.nonzero((n[:, 0] == 1) & (n[:, 1] == 0))[0]
    h = cs.flat(0).cpu().numpy()[a[east]]
    pick = np.sort(east[np.argsort(-h, kind="stable")[:24]])
    return g[pick], a[pick]


def _flat(c, seed):
    d = _case_inputs(c, seed)
    mesh = Mesh2D(nx=c["nx"], ny=c["ny"], dx=d["dx"], dy=d["dx"], ngh=NGH)
    cfg = _config(dict(c, bc="wall" if c["ring"] else "fall"), d)
    s = Solver2D(mesh, cfg, d["q"], d["z"], track_max_depth=False)
    if "cls" in d:
        s.set_manning_table(d["cls"], MANNING)
    if d["mask"] is not None:
        s.set_inside_mask(d["mask"])
    s.apply_bc()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")          # the wall edges are the ring's business here
        cs = CompressedSolver.from_dense(s, track_max_depth=not c["ring"])
    rf = _rain_forcing(c, d)
    if rf is not None:
        cs.set_rain(rf)
    if c["ring"]:
        r = _ring(c, d)
        cs.set_ring(dict(i=r["i"], j=r["j"], bed=r["bed"], wg=np.ones((r["i"].size, 1), np.float32), NG=1,
                         n=r["i"].size, t_common=r["t"], stage_all=r["stage"][None, :].astype(np.float32)))
    if c["inlet"]:
        ghost, nbr = _flat_inlet(cs)
        if ghost.size:
            cs.add_inflow(ghost, nbr, (1.0, 0.0), d["dx"], INLET_T, INLET_Q)
    if c["forcings"]:
        k = _compound(d)
        cs.set_infil({"tab": INFIL})
        cs.set_sponge({"keep": k["keep"].cpu().numpy(), "amb": np.zeros(tuple(k["keep"].shape), np.float32)})
        cs.set_ga_drain(dict(cls_pad=d["cls"].cpu().numpy(), Ks_t=KS, psi_t=PSI, dth_t=DTH,
                             F_pad=np.full(tuple(k["keep"].shape), 1e-3, np.float32),
                             inv_tau_pad=k["inv_tau"].cpu().numpy(), mode="fused"))
        rows, cols = np.nonzero(k["clamp"].cpu().numpy() & _pad(d["mask"]).cpu().numpy())
        cs.set_clamp(dict(rows=rows, cols=cols, hmax=np.full(rows.size, CLAMP_H, np.float32)))
    return cs


def _ring(c, d):
    """Tidal stage on the two x- ghost rows."""
    ny = d["ny"]
    i = np.repeat(np.arange(NGH), ny)
    j = np.tile(np.arange(ny) + NGH, NGH)
    t = np.append(np.arange(0.0, 3660.0, 60.0), 1.0e13)
    return dict(i=i, j=j, bed=d["z"][:1].cpu().numpy().repeat(NGH, 0).reshape(-1), t=t,
                stage=1.5 + 0.3 * np.sin(2 * np.pi * t / 44712.0) * (t < 1.0e12))


def _members(c, seed):
    rng = np.random.default_rng([c["members"], c["lo"], c["hi"]])
    out = []
    for k in range(c["members"]):
        nx, ny = (int(round(math.exp(v))) for v in rng.uniform(math.log(c["lo"]), math.log(c["hi"]), 2))
        out.append(dict(FLAT, nx=nx, ny=ny, frac=float(rng.uniform(0.3, 0.9)), steps=c["steps"],
                        seed=int(seed) + 1009 * k))
    return out


def _calibration(c, seed):
    """Mesh, gauges and an inlet for FlatAdjoint: (CompressedSolver, pieces)."""
    m = dict(FLAT, nx=c["nx"], ny=c["ny"], frac=0.7, rain="none", film=0.2)
    cs = _flat(m, seed)
    rng = np.random.default_rng(int(seed))
    ghost, nbr = _flat_inlet(cs)
    act = np.nonzero(cs.is_active != 0)[0]
    gauges = np.sort(rng.choice(act, 32, replace=False))
    knots = 8.0 + 4.0 * rng.random(16)
    target = 0.5 * rng.random((c["window"], 32))
    return m, cs, dict(ghost=ghost[:1], nbr=nbr[:1], gauges=gauges, knots=knots, target=target,
                       t_knots=np.linspace(0.0, 60.0, 16), rain=40.0 / 3.6e6)


# --------------------------------------------------------------------------- the passes
def prepare(case, seed):
    kind, steps = case["kind"], case.get("steps")
    if kind in ("step", "dense"):
        return kind, steps, _dense(case, seed)
    if kind == "flat":
        return kind, steps, _flat(case, seed)
    if kind == "ensemble":
        ms = [_flat(m, m["seed"]) for m in _members(case, seed)]
        return kind, steps, Ensemble(ms)
    _, cs, p = _calibration(case, seed)
    adj = FlatAdjoint(cs, gauges=p["gauges"], n_steps=steps, window=case["window"], snapshots=case["snapshots"],
                      rain_times=np.array([0.0]), rain_base=np.array([p["rain"]]),
                      inlet=Inlet(ghost=p["ghost"], nbr=p["nbr"], normal=(1.0, 0.0), ds=cs.dx, t_knots=p["t_knots"]))
    slots = torch.from_numpy(np.ascontiguousarray(cs.slot_of)).cuda()
    return kind, steps, (adj, p, torch.from_numpy(p["target"]).cuda(), slots)


def run(state):
    kind, steps, s = state
    if kind == "step":
        dt = s.step()
        return {"q": s.q_interior, "dt": float(dt)}
    if kind == "dense":
        n = s.run(FAR, max_steps=steps)
        return {"q": s.q_interior, "t": float(s.t), "steps": int(n)}
    if kind == "flat":
        n = s.run(FAR, max_steps=steps)
        return {"q": [s.flat(k) for k in range(3)], "t": float(s.t), "steps": int(n)}
    if kind == "ensemble":
        n = s.run(FAR, max_steps=steps)
        return {"q": [s.flat(k, f) for k in range(len(s.members)) for f in range(3)], "steps": sum(n),
                "t": [float(m.t) for m in s.members]}
    adj, p, target, slots = s
    n_tab = torch.tensor(MANNING, requires_grad=True)
    scale = torch.tensor(1.0, dtype=torch.float64, requires_grad=True)
    knots = torch.tensor(p["knots"], requires_grad=True)
    loss = CalibrationLoss.apply(n_tab, scale, knots, adj, target)
    loss.backward()
    return {"loss": loss.detach(), "n": n_tab.grad, "scale": scale.grad, "knots": knots.grad,
            "q0": [adj.adjoint_state(k)[slots] for k in range(3)]}


# Per cell and step: state, bed and class in, state and running maximum out; about 330
# additions, multiplications, divisions and roots of four half-shared faces and the update.
FLOPS = 330.0


def work(case):
    kind = case["kind"]
    if kind == "ensemble":      # the expected cells of a member: log-uniform sides
        side = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        cells = case["members"] * 0.6 * side * side
        return {"bytes": 38.0 * cells * case["steps"], "flops": FLOPS * cells * case["steps"]}
    cells = float(case["nx"] * case["ny"])
    n = case["steps"]
    if kind == "adjoint":       # the recording pass, and a reverse step that recomputes each face
        cells *= 0.7
        return {"bytes": (30.0 + 41.0) * cells * n, "flops": 4.0 * FLOPS * cells * n}
    if kind == "flat":
        cells *= case["frac"]
        per = 30.0 if case["ring"] else 38.0
        return {"bytes": per * cells * n, "flops": FLOPS * cells * n}
    per = 37.0 if case["dtype"] == "float32" else 72.0
    return {"bytes": per * cells * n, "flops": FLOPS * cells * n}


def tolerance(case):
    """The largest error that another correct evaluation at the same precision shows: about
    four times the distance of the present one from binary64. The state of a dense run
    comes as one array, which the depths dominate; the compressed solvers return each
    field, and the momentum of water near rest is a difference of large terms."""
    if case["kind"] in ("step", "dense"):
        return {"rel": 2.0e-4, "max": 5.0e-2} if case["dtype"] == "float32" else {"rel": 1.0e-11, "max": 1.0e-9}
    return {"rel": 4.0e-3 if case["kind"] == "adjoint" else 4.0e-4, "max": 5.0e-2}


# ------------------------------------------------------- the scheme in binary64, plain torch
def _w(c, a, b):
    return torch.where(c, a, b)


def _pos(x):
    return _w(x > 0, x, torch.zeros_like(x))


def _min(a, b):
    return _w(a <= b, a, b)


def _max(a, b):
    return _w(a >= b, a, b)


def _root(x):
    p = x > 0
    return _w(p, torch.sqrt(_w(p, x, torch.ones_like(x))), torch.zeros_like(x))


def _ratio(a, b, ok):
    return _w(ok, a / _w(ok, b, torch.ones_like(b)), torch.zeros_like(a))


def _hllc(hL, uL, tL, hR, uR, tR, h_min):
    aL, aR = _root(G * hL), _root(G * hR)
    us = 0.5 * (uL + uR) + aL - aR
    hr = 0.5 * (aL + aR) + 0.25 * (uL - uR)
    a_s = _root(G * (_pos(hr) * _pos(hr) / G))
    dryL, dryR = hL <= h_min, hR <= h_min
    both = dryL & dryR
    z = torch.zeros_like(hL)
    SL = _w(both, z, _w(dryL, uR - 2 * aR, _min(uL - aL, us - a_s)))
    SR = _w(both, z, _w(dryR, uL + 2 * aL, _max(uR + aR, us + a_s)))
    den = hR * (uR - SR) - hL * (uL - SL)
    big = den.abs() > 1e-14
    SM = _w(big, _ratio(SL * hR * (uR - SR) - SR * hL * (uL - SL), den, big), 0.5 * (uL + uR))
    left = SM >= 0
    useL = SL >= 0
    side = useL | left
    h, u, t = _w(side, hL, hR), _w(side, uL, uR), _w(side, tL, tR)
    S = _w(left, SL, SR)
    star = (~useL) & (left | (SR >= 0))
    hs = h * _ratio(S - u, S - SM + 1e-30, star)
    F0, F1, F2 = h * u, h * u * u + 0.5 * G * h * h, h * u * t
    return (_w(star, F0 + S * (hs - h), F0), _w(star, F1 + S * (hs * SM - h * u), F1),
            _w(star, F2 + S * (hs * t - h * t), F2))


def _face(L, R, half, inv, h_min, x):
    """Flux and both bed sources of the faces between cells L and R (h, u, v, eta, b, g)."""
    hL, uL, vL, eL, bL, gL = L
    hR, uR, vR, eR, bR, gR = R
    zf = torch.maximum(bL, bR)
    clip = (bR - half * gR) - (bL + half * gL)
    dz = bR - bL - clip
    h1 = _pos(eL + _pos(_min(dz, eR - eL)) - zf)
    h2 = _pos(eR + _pos(_min(-dz, eL - eR)) - zf)
    F = _hllc(h1, uL, vL, h2, uR, vR, h_min) if x else _hllc(h1, vL, uL, h2, vR, uR, h_min)
    dL = _w(hR < h_min, _pos(zf - eL), _pos(_min(clip, zf - eL)))
    dR = _w(hL < h_min, _pos(zf - eR), _pos(_min(-clip, zf - eR)))
    sL = 0.5 * G * (h1 + hL) * ((zf - dL) - bL)
    sR = 0.5 * G * (h2 + hR) * ((zf - dR) - bR)
    wet = ~((hL < h_min) & (hR < h_min))
    z = torch.zeros_like(hL)
    return [_w(wet, f * inv, z) for f in (*F, sL, sR)]


def _residual(q, b, dx, h_min):
    """Residual (rh, rhu, rhv) of rows and columns [2, n - 2) of the padded state."""
    inv, half = 1.0 / dx, 0.5 * dx
    h = q[0]
    wet = h > h_min
    u, v = _ratio(q[1], h, wet), _ratio(q[2], h, wet)
    eta = h + b
    c = slice(2, -2)
    gx = 0.5 * (b[2:] - b[:-2]) * inv                 # rows 1 .. n-2
    gy = 0.5 * (b[:, 2:] - b[:, :-2]) * inv           # columns 1 .. n-2
    lo = lambda f: f[1:-2, c]                         # noqa: E731
    hi = lambda f: f[2:-1, c]                         # noqa: E731
    X = _face([lo(f) for f in (h, u, v, eta, b)] + [gx[:-1, c]], [hi(f) for f in (h, u, v, eta, b)] + [gx[1:, c]],
              half, inv, h_min, True)
    rh = X[0][:-1] - X[0][1:]
    rhu = X[1][:-1] - X[1][1:] - X[3][1:] + X[4][:-1]
    rhv = X[2][:-1] - X[2][1:]
    del X
    lo = lambda f: f[c, 1:-2]                         # noqa: E731
    hi = lambda f: f[c, 2:-1]                         # noqa: E731
    Y = _face([lo(f) for f in (h, u, v, eta, b)] + [gy[c, :-1]], [hi(f) for f in (h, u, v, eta, b)] + [gy[c, 1:]],
              half, inv, h_min, False)
    rh = rh + Y[0][:, :-1] - Y[0][:, 1:]
    rhv = rhv + Y[1][:, :-1] - Y[1][:, 1:] - Y[3][:, 1:] + Y[4][:, :-1]
    rhu = rhu + Y[2][:, :-1] - Y[2][:, 1:]
    return rh, rhu, rhv


def _tail(h, hu, hv, n, dt, h_min):
    """Wet/dry floor and point-implicit Manning friction (n None: the floor alone)."""
    dry = h < h_min
    z = torch.zeros_like(h)
    if n is not None:
        hs = _w(dry, torch.full_like(h, h_min), h)
        m = _root((hu / hs) ** 2 + (hv / hs) ** 2)
        p = hs ** (-4.0 / 3.0)
        over = m > 15.0
        ncri = torch.sqrt(1.0 / _w(over, (1e-10 + dt) * G * p * (m + 1e-30), torch.ones_like(m)))
        ne = _w(over & (ncri > n), ncri, n)
        a = 2.0 / (torch.sqrt(1.0 + 4.0 * dt * (G * ne * ne * p) * m) + 1.0)
        hu, hv = hu * a, hv * a
    return _w(dry, _pos(h), h), _w(dry, z, hu), _w(dry, z, hv)


def _advance(q, b, P, dt, rate):
    """One step of the padded state: cells outside P["act"] (None: all of the interior, with
    P["inside"] limiting the residual) keep their values."""
    rh, rhu, rhv = _residual(q, b, P["dx"], P["h_min"])
    c = q[:, 2:-2, 2:-2]
    ins = P.get("inside")
    if ins is not None:
        z = torch.zeros_like(rh)
        rh, rhu, rhv = _w(ins, rh + rate, z), _w(ins, rhu, z), _w(ins, rhv, z)
    else:
        rh = rh + rate
    h, hu, hv = _tail(c[0] + dt * rh, c[1] + dt * rhu, c[2] + dt * rhv, P["n"], dt, P["h_min"])
    act = P.get("act")
    if act is not None:
        h, hu, hv = _w(act, h, c[0]), _w(act, hu, c[1]), _w(act, hv, c[2])
    if torch.is_grad_enabled():
        out = q.clone()
        out[:, 2:-2, 2:-2] = torch.stack([h, hu, hv])
        return out
    q[0, 2:-2, 2:-2], q[1, 2:-2, 2:-2], q[2, 2:-2, 2:-2] = h, hu, hv
    return q


def _bc(q, kinds, skip=()):
    """Ghost fill: x faces over all columns, then y faces over all rows."""
    for ax, (lo, hi) in ((1, kinds[:2]), (2, kinds[2:])):
        p = q.transpose(1, ax)
        n = p.shape[1]
        for side, kind in ((0, lo), (1, hi)):
            for k in range(NGH):
                g = k if side == 0 else n - NGH + k
                if kind == "fall":
                    p[:, g] = 0.0
                    continue
                m = {"extrapolate": (NGH, n - NGH - 1), "wall": (2 * NGH - 1 - k, n - NGH - 1 - k),
                     "periodic": (n - 2 * NGH + k, NGH + k)}[kind][side]
                p[:, g] = p[:, m]
                if kind == "wall":
                    p[ax, g] *= -1.0


def _pad_bed(z, kinds):
    b = torch.zeros((z.shape[0] + 2 * NGH, z.shape[1] + 2 * NGH), dtype=torch.float64, device=z.device)
    b[NGH:-NGH, NGH:-NGH] = z
    t = b[None].expand(3, -1, -1).clone()
    _bc(t, ["periodic" if k == "periodic" else "extrapolate" for k in kinds])
    return t[0]


def _speed(q, ok, h_cfl, linf, h_min):
    """The largest wave speed over the cells `ok`: max(|u|, |v|) (dense) or the L2 norm."""
    h = q[0]
    hs = h.clamp_min(h_cfl)
    u, v = q[1] / hs, q[2] / hs
    s = torch.maximum(u.abs(), v.abs()) if linf else torch.sqrt(u * u + v * v)
    lam = _w(h < (h_cfl if linf else h_min), torch.zeros_like(h), s + torch.sqrt(G * h.clamp_min(0.0)))
    return float((lam if ok is None else lam[ok]).max())


def _interp(t, ts, vs):
    return float(np.interp(t, ts, vs))


def _manning64(c, d, s=slice(NGH, -NGH)):
    if d["friction"] == "none":
        return None
    if d["friction"] == "scalar":
        return torch.full((d["nx"], d["ny"]), float(np.float32(0.03)), dtype=torch.float64, device="cuda")
    if d["friction"] == "field":
        return d["nfield"][s, s].double()
    return torch.from_numpy(MANNING.astype(np.float32)).double().cuda()[d["cls"][s, s].long()]


def _rate64(c, d, k=0):
    if c["rain"] == "uniform":
        return float(np.float32(RAIN_MM_H / 3.6e6)), RAIN_MM_H / 3.6e6
    if c["rain"] == "gridded":
        f = torch.from_numpy(d["rain"][k] / 3.6e6).cuda()
        return f, float(d["rain"].max() if c["kind"] == "flat" else d["rain"][k].max()) / 3.6e6
    return 0.0, 0.0


def _film_limit(dx, rmax):
    return (0.5 * dx) ** (2.0 / 3.0) / (G * rmax) ** (1.0 / 3.0) if rmax > 0.0 else math.inf


def _exact_dense(c, seed):
    d = _case_inputs(c, seed)
    dx = d["dx"]
    if c["inlet"]:
        d["q"][0, 0] += 0.3
    kinds = {"open": ["wall", "fall", "wall", "wall"], "wall": ["wall"] * 4, "periodic": ["periodic"] * 4,
             "extrapolate": ["extrapolate"] * 4}[c["bc"]]
    f32 = c["dtype"] == "float32"
    h_min = 1.0e-6 if f32 else 1.0e-10
    b = _pad_bed(d["z"], kinds)
    q = _pad(d["q"].double())
    P = dict(dx=dx, h_min=h_min, n=_manning64(c, d), inside=d.get("mask"))
    rate, rmax = _rate64(c, d)
    lim = _film_limit(dx, rmax)
    inner = lambda: q[:, NGH:-NGH, NGH:-NGH]          # noqa: E731
    if c["stage"]:
        cells = _stage_cells(c, d)
        series = _stage_series(d, cells)
    t = 0.0
    for _ in range(c["steps"]):
        lam = max(_speed(inner(), None, h_min, True, h_min), math.sqrt(G * h_min))
        dt = min(0.5 * dx / (lam + 1e-12), lim if c["kind"] == "dense" else math.inf)
        _bc(q, kinds)
        if c["inlet"]:
            i, jj = _dense_inlet(d)
            j = torch.from_numpy(jj).cuda()
            h = q[0, i, j]
            qn = _interp(t, INLET_T, INLET_Q) / dx * (h / h.sum())
            for g in range(NGH):
                q[0, g, j], q[1, g, j], q[2, g, j] = h, qn, torch.zeros_like(qn)
        q = _advance(q, b, P, dt, rate)
        t += dt
        if c["stage"]:
            eta = _interp(t, STAGE_T, series)
            v = inner()
            v[0] = _w(cells, (eta - d["z"].double()).clamp_min(0.0), v[0])
            v[1:][:, cells] = 0.0
    return q[:, NGH:-NGH, NGH:-NGH], t, dt


def _stored(inside):
    st = inside.clone()
    for _ in range(2):
        e = st.clone()
        e[1:] |= st[:-1]
        e[:-1] |= st[1:]
        e[:, 1:] |= st[:, :-1]
        e[:, :-1] |= st[:, 1:]
        st = e
    return st


def _flat_setup(c, seed):
    """Padded binary64 state and bed of a compressed case (zero outside the stored cells)."""
    d = _case_inputs(c, seed)
    kinds = ["wall"] * 4 if c["ring"] else ["fall"] * 4
    b = _pad_bed(d["z"], kinds)
    q = _pad(d["q"].double())
    _bc(q, kinds)
    act = torch.ones_like(d["z"], dtype=torch.bool) if d["mask"] is None else d["mask"]
    stored = _stored(_pad(act))
    b = b * stored
    q = q * stored
    P = dict(dx=d["dx"], h_min=1.0e-6, n=_manning64(c, d), act=act)
    return d, q, b, P, stored


def _pairs(stored, act, h):
    """The inlet's padded (ghost, neighbour) cells, as _flat_inlet picks them: ring cells
    whose first active neighbour in E, W, N, S order is the one below in x."""
    a = _pad(act)
    up = torch.zeros_like(a)
    up[:-1] = a[1:]
    g = (stored & ~a & up).nonzero()
    hn = h[g[:, 0] + 1, g[:, 1]].float()
    pick = torch.argsort(-hn, stable=True)[:24].sort().values
    return g[pick]


def _compound64(q, d, F, k, dt):
    c = q[:, NGH:-NGH, NGH:-NGH]
    cl = d["cls"][NGH:-NGH, NGH:-NGH].long()
    tab = lambda t: torch.from_numpy(t.astype(np.float64)).cuda()[cl]      # noqa: E731
    act = d["mask"]
    one = torch.ones_like(c[0])
    ok = act & (c[0] >= 1.0e-6)
    hn = (c[0] - tab(INFIL) * dt).clamp_min(0.0)
    r = _w(ok, hn / _w(ok, c[0], one), one)
    c[0] = _w(ok, hn, c[0])
    c[1:] *= r
    q *= k["keep"].double()
    h = c[0].clone()
    Ks = tab(KS)
    ok = act & (h > 0.0)
    A = F + Ks * dt
    dF = (0.5 * (A + torch.sqrt((A * A + 4.0 * Ks * dt * (tab(PSI) + h) * tab(DTH)).clamp_min(0.0))) - F).clamp_min(0.0)
    dF = _w(ok & (Ks > 0), torch.minimum(dF, h), torch.zeros_like(h))
    F += dF
    decay = torch.exp(-dt * k["inv_tau"][NGH:-NGH, NGH:-NGH].double())
    hn = _w(ok, (h - dF) * decay, h)
    c[1:] *= _w(ok, hn / _w(ok, h, one), one)
    c[0] = hn
    ok = k["clamp"][NGH:-NGH, NGH:-NGH] & act & (c[0] > CLAMP_H)
    c[1:] *= _w(ok, CLAMP_H / _w(ok, c[0], one), one)
    c[0] = _w(ok, torch.full_like(one, float(np.float32(CLAMP_H))), c[0])


def _exact_flat(c, seed):
    d, q, b, P, stored = _flat_setup(c, seed)
    dx, act = d["dx"], P["act"]
    rate, rmax = _rate64(c, d)
    lim = _film_limit(dx, rmax)
    if c["inlet"]:
        gh = _pairs(stored, act, q[0])
    if c["forcings"]:
        k = _compound(d)
        F = torch.full_like(q[0, NGH:-NGH, NGH:-NGH], float(np.float32(1e-3)))
    t = 0.0
    for _ in range(c["steps"]):
        lam = max(_speed(q[:, NGH:-NGH, NGH:-NGH], act, 1e-6, False, 1e-6), math.sqrt(G * 1e-6))
        dt = min(0.5 * dx / (lam + 1e-12), lim)
        if c["inlet"] and len(gh):
            i, j = gh[:, 0], gh[:, 1]
            h = q[0, i + 1, j]
            q[0, i, j], q[1, i, j], q[2, i, j] = h, _interp(t, INLET_T, INLET_Q) / dx * h / h.sum(), 0.0 * h
        q = _advance(q, b, P, dt, rate)
        if c["forcings"]:
            _compound64(q, d, F, k, dt)
            q *= stored
        if c["ring"]:
            r = _ring(c, d)
            h = (_interp(t, r["t"], r["stage"]) - torch.from_numpy(r["bed"]).double().cuda()).clamp_min(0.0)
            ri, rj = torch.from_numpy(r["i"]).cuda(), torch.from_numpy(r["j"]).cuda()
            q[0, ri, rj] = h
            q[1:, ri, rj] = 0.0
        t += dt
    return [q[f][stored] for f in range(3)], t


def _exact_adjoint(c, seed):
    m, cs, p = _calibration(c, seed)          # gauges and inlet as canonical cell numbers
    ij = torch.from_numpy(cs.ij_active.astype(np.int64)).cuda()
    del cs
    d, q, b, P, stored = _flat_setup(m, seed)
    dx, act = d["dx"], P["act"]
    cls = d["cls"][NGH:-NGH, NGH:-NGH].long()
    n_tab = torch.tensor(MANNING.astype(np.float32).astype(np.float64), device="cuda", requires_grad=True)
    scale = torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True)
    knots = torch.tensor(p["knots"], device="cuda", requires_grad=True)
    target = torch.from_numpy(p["target"]).cuda()
    gi = ij[torch.from_numpy(p["gauges"]).cuda()]
    g0, a0 = (ij[int(p[x][0])].tolist() for x in ("ghost", "nbr"))
    lim = _film_limit(dx, float(np.float32(p["rain"])))
    q0 = q.clone().requires_grad_(True)
    x = q0 * 1.0
    loss = torch.zeros((), dtype=torch.float64, device="cuda")
    t = 0.0
    N, first = c["steps"], c["steps"] - c["window"] + 1
    for k in range(N):
        lam = max(_speed(x.detach()[:, NGH:-NGH, NGH:-NGH], act, 1e-6, False, 1e-6), math.sqrt(G * 1e-6))
        dt = min(0.5 * dx / (lam + 1e-12), lim)
        i = min(int(np.searchsorted(p["t_knots"], t, "right")) - 1, 14)
        w = (t - p["t_knots"][i]) / (p["t_knots"][i + 1] - p["t_knots"][i])
        Q = knots[i] * (1 - w) + knots[i + 1] * w
        h = x[0, a0[0], a0[1]]
        x = x.clone()
        x[0, g0[0], g0[1]] = h
        x[1, g0[0], g0[1]] = Q / dx
        x[2, g0[0], g0[1]] = 0.0
        x = _advance(x, b, dict(P, n=n_tab[cls]), dt, scale * p["rain"])
        t += dt
        if k + 1 >= first:
            e = x[0, gi[:, 0], gi[:, 1]] - target[k + 1 - first]
            loss = loss + (e * e).sum()
    loss.backward()
    # level water sits on kinks in the depths (the free-surface jumps of the face states
    # are clipped at zero), where rounding picks the side: no value for the depths' adjoint
    return {"loss": loss.detach(), "n": n_tab.grad, "scale": scale.grad, "knots": knots.grad,
            "q0": [None, q0.grad[1][stored], q0.grad[2][stored]]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        if kind in ("step", "dense"):
            q, t, dt = _exact_dense(case, seed)
            return {"q": q, "dt": dt} if kind == "step" else {"q": q, "t": t, "steps": case["steps"]}
        if kind == "flat":
            q, t = _exact_flat(case, seed)
            return {"q": q, "t": t, "steps": case["steps"]}
        got = [_exact_flat(m, m["seed"]) for m in _members(case, seed)]
        return {"q": [f for q, _ in got for f in q], "t": [t for _, t in got],
                "steps": case["steps"] * len(got)}
