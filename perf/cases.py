"""Workloads of the FDTD engine, as a user's program calls them.

Each case is one pass through the package's public entry points: single 2D runs
(``run_tm`` / ``run_te``), a kept plan over a batch of ragged structures or of designs,
3D runs (``run_3d``, a kept ``Engine3D``), gradients (``run_tm`` with eps requiring grad,
``run_3d_adjoint``) and a training step of the surrogate network. ``exact`` restates each
of them in float64 torch.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

DX2 = 0.05             # 2D cell, resolution 20
DX3 = 1.0 / 16         # 3D cell, resolution 16
NPML3 = 12
# a dispersive metal-like pair: (frequency, damping, strength[, drive frequency])
POLES = ((1.1, 0.08, 0.7), (0.0, 0.15, 1.0, 0.9))


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest call: a short TM run on a tiny cell (a first look, a unit test)
        dict(name="tm_small", kind="run2d", pol="tm", nx=64, ny=48, steps=200, npml=8, nf=3,
             full=True, material="plain"),
        # the waveguide transmission spectrum: one flux line at 50 frequencies, long run
        dict(name="tm_guide", kind="run2d", pol="tm", nx=320, ny=160, steps=4000, npml=20,
             nf=50, full=False, material="plain"),
        # a single TE structure of odd sides with full-grid DFT fields
        dict(name="te_odd", kind="run2d", pol="te", nx=501, ny=389, steps=1500, npml=20, nf=3,
             full=True, material="plain"),
        # a dispersive, lossy TM structure (Lorentz and Drude poles under masks, conductivity)
        dict(name="tm_metal", kind="run2d", pol="tm", nx=400, ny=301, steps=800, npml=20, nf=5,
             full=False, material="metal"),
        # a batch of ragged TM / TE bends on one kept plan (many design variants at once)
        dict(name="bends", kind="batch", count=20, lo=256, hi=768, steps=960, npml=20),
        # data generation for the surrogate: new designs through one kept plan
        dict(name="designs", kind="designs", count=64, steps=800),
        # the large 3D run: a kept plan, six flux faces at 20 frequencies
        dict(name="cube", kind="run3d", nx=256, ny=256, nz=256, steps=200, nf=20, kept=True,
             material="plain"),
        # a small 3D box of odd sides, one call
        dict(name="box_odd", kind="run3d", nx=117, ny=90, nz=75, steps=240, nf=5, kept=False,
             material="plain"),
        # a 3D dispersive particle (poles), one call
        dict(name="box_metal", kind="run3d", nx=128, ny=112, nz=100, steps=120, nf=5,
             kept=False, material="metal"),
        # inverse design: the gradient of a transmitted flux by every eps pixel
        dict(name="grad_tm", kind="grad2d", pol="tm", nx=600, ny=400, steps=2000, npml=25,
             every=256),
        # the same in 3D
        dict(name="grad_3d", kind="grad3d", nx=96, ny=80, nz=72, steps=96, chunk=32),
        # one training step of the surrogate network
        dict(name="fno_train", kind="fno", batch=8, size=128, width=64, modes=24),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run2d", "run2d", "run2d", "batch", "designs", "run3d", "run3d",
                       "grad2d", "grad3d", "fno"])
    if kind == "run2d":
        nx, ny = _between(rng, 48, 640), _between(rng, 48, 640)
        steps = min(_between(rng, 200, 4000), int(3.0e8 / (nx * ny)))
        return dict(kind=kind, pol=rng.choice(["tm", "te"]), nx=nx, ny=ny, steps=steps,
                    npml=rng.choice([8, 10, 16, 20]), nf=rng.randint(1, 50),
                    full=nx * ny * steps < 5.0e7 and rng.random() < 0.5,
                    material=rng.choice(["plain", "plain", "metal"]))
    if kind == "batch":
        lo = rng.randint(192, 320)
        return dict(kind=kind, count=rng.randint(6, 20), lo=lo,
                    hi=rng.randint(lo + 64, 768), steps=rng.randint(240, 960), npml=20)
    if kind == "designs":
        return dict(kind=kind, count=rng.randint(8, 64), steps=rng.randint(200, 800))
    if kind == "run3d":
        nx, ny, nz = (_between(rng, 40, 200) for _ in range(3))
        metal = rng.random() < 0.4
        steps = max(20, min(rng.randint(40, 240), int((2.0e8 if metal else 8.0e8) /
                                                      (nx * ny * nz))))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=steps, nf=rng.randint(1, 20),
                    kept=rng.random() < 0.3, material="metal" if metal else "plain")
    if kind == "grad2d":
        nx, ny = rng.randint(160, 600), rng.randint(160, 400)
        return dict(kind=kind, pol=rng.choice(["tm", "tm", "te"]), nx=nx, ny=ny,
                    steps=rng.randint(400, 2000), npml=20,
                    every=rng.choice([32, 64, 100, 256]))
    if kind == "grad3d":
        return dict(kind=kind, nx=rng.randint(40, 96), ny=rng.randint(40, 80),
                    nz=rng.randint(40, 72), steps=rng.randint(40, 96),
                    chunk=rng.choice([16, 24, 32]))
    return dict(kind=kind, batch=rng.randint(1, 8), size=rng.choice([64, 96, 128]), width=64,
                modes=24)


# ------------------------------------------------------------------ inputs

def _dev():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _rng(seed, salt=0):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _bend_eps(nx, ny, rng):
    """Input guide along +x and output guide along +y meeting a block of random pixels."""
    eps = np.ones((nx, ny), dtype=np.float32)
    cx, cy = nx // 2, ny // 2
    half = max(2, min(10, ny // 8))
    blk = max(3, min(20, nx // 5, ny // 5))
    eps[:cx - blk, cy - half:cy + half] = 12.0
    eps[cx - half:cx + half, cy + blk:] = 12.0
    pix = rng.random((2 * blk, 2 * blk)) < 0.5
    eps[cx - blk:cx + blk, cy - blk:cy + blk] = np.where(pix, 12.0, 2.1)
    return eps, half, blk


def _pulse(dt, steps):
    """A Gaussian pulse (fcen 0.65, fwidth 0.4) centred well inside the run."""
    return dict(fcen=0.65, fwidth=0.4, cutoff=min(5.0, 0.35 * steps * dt * 0.4))


def _freqs(nf):
    return np.linspace(0.5, 0.8, nf).tolist() if nf > 1 else [0.65]


def _geom2d(case, seed, b=0):
    """One 2D structure's inputs as plain values: eps, masks, source line, monitor lines."""
    nx, ny, npml = case["nx"], case["ny"], case["npml"]
    rng = _rng(seed, 100 + b)
    eps, half, blk = _bend_eps(nx, ny, rng)
    cx, cy = nx // 2, ny // 2
    g = dict(nx=nx, ny=ny, npml=npml, pol=case["pol"], steps=case["steps"], eps=eps,
             src=(min(npml + 4, cx - blk - 1), cy - half, cy + half),
             x_line=(min(nx - npml - 4, cx + blk + 6), max(1, cy - 2 * half),
                     min(ny - 1, cy + 2 * half)),
             y_line=(max(npml + 2, cy - blk - 6), max(1, cx - 2 * half),
                     min(nx - 1, cx + 2 * half)),
             freqs=_freqs(case.get("nf", 3)), full=case.get("full", True))
    if case.get("material") == "metal":
        m = np.zeros((nx, ny), dtype=np.float32)
        m[cx - blk:cx + blk, cy - blk:cy + blk] = 1.0
        m2 = (rng.random((nx, ny)) < 0.2).astype(np.float32) * m
        sig = np.zeros((nx, ny), dtype=np.float32)
        sig[cx + blk:, :] = 0.05 * rng.random((nx - cx - blk, ny)).astype(np.float32)
        g.update(masks=[m, m2], sigma=sig)
    return g


def _item2d(g, dev, eps=None):
    """(state, coeffs, source, monitors) of one structure through the public builders."""
    from meep_torch_b200.core.coeffs import build_te_coeffs, build_tm_coeffs
    from meep_torch_b200.core.grid import Grid
    from meep_torch_b200.core.monitors import (DFTFieldsMonitor, FluxMonitorTE, FluxMonitorTEY,
                                               FluxMonitorTM)
    from meep_torch_b200.core.sources import GaussianPulse, LineSource, TESource
    from meep_torch_b200.core.stepper_te import init_te_state
    from meep_torch_b200.core.stepper_tm import init_tm_state
    grid = Grid(nx=g["nx"], ny=g["ny"], dx=DX2, device=dev)
    eps = torch.from_numpy(g["eps"]).to(dev) if eps is None else eps
    kw = {}
    if "masks" in g:
        kw = dict(poles=POLES, pole_masks=[torch.from_numpy(m).to(dev) for m in g["masks"]],
                  sigma_d=torch.from_numpy(g["sigma"]).to(dev))
    npol = len(POLES) if kw else 0
    i, j0, j1 = g["src"]
    src = LineSource(grid, ix=i, j0=j0, j1=j1, profile=GaussianPulse(**_pulse(grid.dt,
                                                                              g["steps"])))
    fr, (ix, a, b), (iy, c, d) = g["freqs"], g["x_line"], g["y_line"]
    if g["pol"] == "tm":
        m = build_tm_coeffs(grid, eps_inf=eps, npml=g["npml"], **kw)
        mons = [FluxMonitorTM(grid, fr, x_normal=True, idx=ix, lo=a, hi=b),
                FluxMonitorTM(grid, fr, x_normal=False, idx=iy, lo=c, hi=d)]
        if g["full"]:
            mons.append(DFTFieldsMonitor(grid, fr, "Ez"))
        return init_tm_state(grid, n_poles=npol), m, src, mons
    m = build_te_coeffs(grid, eps_inf=eps, npml=g["npml"], **kw)
    mons = [FluxMonitorTE(grid, fr, ix=ix, lo=a, hi=b), FluxMonitorTEY(grid, fr, iy=iy, lo=c, hi=d)]
    if g["full"]:
        mons.append(DFTFieldsMonitor(grid, fr, "Hz"))
    return init_te_state(grid, n_poles=npol), m, TESource(src), mons


def _batch_geoms(case, seed):
    # the sides come from the case, the pixels from the seed: every seed costs the same
    sides = _rng(case["count"] * 7919 + case["lo"], 1).integers(
        case["lo"], case["hi"] + 1, size=(case["count"], 2))
    return [_geom2d(dict(nx=int(nx), ny=int(ny), npml=case["npml"], steps=case["steps"],
                         pol="tm" if b % 2 == 0 else "te"), seed, b)
            for b, (nx, ny) in enumerate(sides)]


def _densities(case, seed):
    """Smooth random design densities in [0, 1]: filtered noise, half of them binary."""
    n = case["count"]
    r = _rng(seed, 3).random((n, 64, 64)).astype(np.float32)
    r = F.avg_pool2d(torch.from_numpy(r)[:, None], 7, 1, 3)[:, 0]
    r = torch.sigmoid((r - 0.5) * 40.0)
    r[: n // 2] = (r[: n // 2] > 0.5).float()
    return F.avg_pool2d(r[:, None], 3, 1, 1)[:, 0].contiguous()


def _geom3d(case, seed):
    """Random dielectric spheres around a central dipole, and six flux faces round it, near
    enough for the pulse to pass them within the run."""
    dims = (case["nx"], case["ny"], case["nz"])
    rng = _rng(seed, 4)
    eps = np.ones(dims, dtype=np.float32)
    mask = np.zeros(dims, dtype=np.float32)
    npml = min(NPML3, min(dims) // 5)
    half = [min(n // 2 - npml - 5, max(3, case["steps"] // 5)) for n in dims]
    box = {a: (n // 2 - h, n // 2 + h) for a, n, h in zip("xyz", dims, half)}
    for q in range(40):
        r = rng.uniform(2.0, 9.0)
        c = [rng.uniform(npml, n - npml) for n in dims]
        e = rng.uniform(2.0, 12.0)
        lo = [max(0, int(v - r) - 1) for v in c]
        hi = [min(n, int(v + r) + 2) for v, n in zip(c, dims)]
        ax = [np.arange(a, b) - v for a, b, v in zip(lo, hi, c)]
        ins = (ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 +
               ax[2][None, None, :] ** 2) <= r * r
        cut = tuple(slice(a, b) for a, b in zip(lo, hi))
        eps[cut][ins] = e
        if q % 4 == 0:
            mask[cut][ins] = 1.0
    return dict(dims=dims, npml=npml, eps=eps, mask=mask if case.get("material") == "metal" else
                None, freqs=_freqs(case.get("nf", 3)), src=tuple(n // 2 for n in dims),
                steps=case["steps"],
                faces=[(a, i) for a in "xyz" for i in box[a]],
                wins=[tuple(v for b in "xyz" if b != a for v in box[b])
                      for a in "xyz" for _ in range(2)])


def _item3d(g, dev, eps=None):
    from meep_torch_b200.core.monitors_3d import FluxMonitor3D, PointSource3D
    from meep_torch_b200.core.sources import GaussianPulse
    from meep_torch_b200.core.stepper_3d import build_3d_coeffs, init_3d_state
    eps = torch.from_numpy(g["eps"]).to(dev) if eps is None else eps
    kw, npol = {}, 0
    if g["mask"] is not None:
        kw = dict(poles=POLES[1:], pole_masks=[torch.from_numpy(g["mask"]).to(dev)])
        npol = 1
    c = build_3d_coeffs(*g["dims"], DX3, eps=eps, npml=g["npml"], device=dev, **kw)
    s = init_3d_state(*g["dims"], npml=g["npml"], n_poles=npol, device=dev)
    src = PointSource3D(c.dt, "Ez", *g["src"], GaussianPulse(**_pulse(c.dt, g["steps"])))
    mons = [FluxMonitor3D(c.dt, g["freqs"], normal=a, idx=i, win=w)
            for (a, i), w in zip(g["faces"], g["wins"])]
    return s, c, src, mons


def _fno_weights(case, seed):
    """The network's parameters by state_dict name, scaled as its own initialisation."""
    gen = torch.Generator().manual_seed(int(seed) & 0x7FFFFFFF)
    w, m = case["width"], case["modes"]
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    out = {"lift.weight": rnd(w, 3, 1, 1) * 0.4, "lift.bias": rnd(w) * 0.2,
           "proj1.weight": rnd(128, w, 1, 1) / w ** 0.5, "proj1.bias": rnd(128) * 0.1,
           "proj2.weight": rnd(6, 128, 1, 1) / 128 ** 0.5, "proj2.bias": rnd(6) * 0.1}
    for k in range(4):
        out[f"spec.{k}.w"] = torch.complex(rnd(2, w, w, m, m), rnd(2, w, w, m, m)) / w ** 1.5
        out[f"mix.{k}.weight"] = rnd(w, w, 1, 1) / w ** 0.5
        out[f"mix.{k}.bias"] = rnd(w) * 0.1
    n = case["size"]
    x = F.avg_pool2d(torch.rand(case["batch"], 1, n, n, generator=gen), 5, 1, 2)
    y = F.avg_pool2d(rnd(case["batch"], 6, n, n), 5, 1, 2)
    return out, x, y


def prepare(case, seed):
    dev = _dev()
    kind = case["kind"]
    if kind == "run2d":
        s, m, src, mons = _item2d(_geom2d(case, seed), dev)
        return dict(case=case, args=(s, m), source=src, monitors=mons)
    if kind == "batch":
        from meep_torch_b200.engine2d import Engine2D
        return dict(case=case, engine=Engine2D([_item2d(g, dev) for g in
                                                _batch_geoms(case, seed)]))
    if kind == "designs":
        from meep_torch_b200.surrogate import Cfg5Problem
        prob = Cfg5Problem(dev, steps=case["steps"])
        rho = _densities(case, seed).to(dev)
        prob.simulate(rho.flip(0), batch=case["count"])     # the plan of the first batch is kept
        return dict(case=case, problem=prob, rho=rho)
    if kind == "run3d":
        from meep_torch_b200.engine3d import Engine3D
        s, c, src, mons = _item3d(_geom3d(case, seed), dev)
        st = dict(case=case, args=(s, c), source=src, monitors=mons)
        if case["kept"]:
            st["engine"] = Engine3D(s, c, src, mons)
        return st
    if kind == "grad2d":
        g = _geom2d(dict(case, full=False), seed)
        return dict(case=case, geom=g, eps=torch.from_numpy(g["eps"]).to(dev))
    if kind == "grad3d":
        g = _geom3d(case, seed)
        return dict(case=case, item=_item3d(g, dev), eps=torch.from_numpy(g["eps"]).to(dev))
    from meep_torch_b200.surrogate import FNO2d
    w, x, y = _fno_weights(case, seed)
    model = FNO2d(case["width"], case["modes"])
    model.load_state_dict(w)
    return dict(case=case, model=model.to(dev), x=x.to(dev), y=y.to(dev))


# ------------------------------------------------------------------ one pass

def _named(st):
    return {k: v for k, v in st._asdict().items() if torch.is_tensor(v) and v.numel()}


def _relative_error(p, y):
    return ((p - y).flatten(1).norm(dim=1) / y.flatten(1).norm(dim=1)).mean()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run2d":
        from meep_torch_b200.core.run import run_te, run_tm
        step = run_tm if case["pol"] == "tm" else run_te
        st, accs = step(*state["args"], case["steps"], source=state["source"],
                        monitors=state["monitors"])
        return dict(_named(st), accs=accs)
    if kind == "batch":
        eng = state["engine"]
        eng.reset()
        eng.run(0, case["steps"])
        return [eng.accumulators(b) for b in range(case["count"])]
    if kind == "designs":
        return state["problem"].simulate(state["rho"], batch=case["count"])
    if kind == "run3d":
        if case["kept"]:
            eng = state["engine"]
            eng.reset()
            eng.run(0, case["steps"])
            f = eng.fields()
            return dict({k: f[k] for k in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")},
                        accs=list(eng.accs))
        from meep_torch_b200.core.monitors_3d import run_3d
        st, accs = run_3d(*state["args"], case["steps"], source=state["source"],
                          monitors=state["monitors"])
        return dict(_named(st), accs=accs)
    if kind == "grad2d":
        from meep_torch_b200.core.run import run_te, run_tm
        step = run_tm if case["pol"] == "tm" else run_te
        eps = state["eps"].detach().clone().requires_grad_(True)
        s, m, src, mons = _item2d(state["geom"], eps.device, eps)
        _, accs = step(s, m, case["steps"], source=src, monitors=mons,
                       checkpoint_every=case["every"])
        loss = mons[0].flux(accs[0], DX2).mean() + mons[1].flux(accs[1], DX2).mean()
        loss.backward()
        return dict(loss=loss.detach(), grad=eps.grad, accs=[a.detach() for a in accs])
    if kind == "grad3d":
        from meep_torch_b200.core.adjoint3d import run_3d_adjoint
        s, c, src, mons = state["item"]
        eps = state["eps"].detach().clone().requires_grad_(True)
        _, accs = run_3d_adjoint(
            c._replace(eps=eps), case["steps"], case["chunk"], src, mons,
            lambda accs: sum(m.flux(a, DX3).mean() for m, a in zip(mons, accs)), s)
        return dict(grad=eps.grad, accs=accs)
    model = state["model"]
    model.zero_grad(set_to_none=True)
    out = model(state["x"])
    loss = _relative_error(out, state["y"])
    loss.backward()
    return dict(out=out.detach(), loss=loss.detach(),
                grads={k: (torch.view_as_real(p.grad) if p.is_complex() else p.grad)
                       for k, p in model.named_parameters()})


# ------------------------------------------------------------------ work

def _work2d(nx, ny, te, steps, nf, full, lines, poles=0):
    """State (3 fields), eps and accumulators once; the update's arithmetic each step."""
    cells = nx * ny
    acc = 8.0 * nf * (cells if full else 0) + 16.0 * nf * lines
    by = 4.0 * cells * (7 + te + 6 * poles) + acc
    fl = steps * (cells * (18.0 + te + 6 * poles) + 4.0 * nf * ((cells if full else 0) +
                                                                3 * lines))
    return by, fl


def work(case):
    """Bytes that any implementation moves (each input read and each output written once)
    and the floating-point operations of the updates."""
    kind = case["kind"]
    if kind == "run2d":
        by, fl = _work2d(case["nx"], case["ny"], case["pol"] == "te", case["steps"], case["nf"],
                         case["full"], 60, 2 if case["material"] == "metal" else 0)
    elif kind == "batch":
        by = fl = 0.0
        sides = _rng(case["count"] * 7919 + case["lo"], 1).integers(
            case["lo"], case["hi"] + 1, size=(case["count"], 2))
        for b, (nx, ny) in enumerate(sides):
            d = _work2d(int(nx), int(ny), b % 2, case["steps"], 3, True, 60)
            by, fl = by + d[0], fl + d[1]
    elif kind == "designs":
        d = _work2d(256, 256, 0, case["steps"], 3, True, 0)
        by, fl = d[0] * case["count"], d[1] * case["count"]
    elif kind in ("run3d", "grad3d"):
        cells = case["nx"] * case["ny"] * case["nz"]
        pol = 1 if case.get("material") == "metal" else 0
        by, fl = 4.0 * cells * (13 + 9 * pol), case["steps"] * cells * (54.0 + 21 * pol)
        if kind == "grad3d":
            by, fl = 8.0 * cells, 3.5 * fl
    elif kind == "grad2d":
        # eps in, its gradient out; the run, its recomputation and the reverse sweep
        by, fl = _work2d(case["nx"], case["ny"], case["pol"] == "te", case["steps"], 3, False, 60)
        by, fl = 8.0 * case["nx"] * case["ny"], 3.5 * fl
    else:
        b, n, w, m = case["batch"], case["size"], case["width"], case["modes"]
        pix = b * n * n
        fft = 2.5 * n * n * math.log2(n * n) * b * w * 2
        fwd = 4 * (2.0 * pix * w * w + fft + 2 * 8.0 * b * w * w * m * m) + \
            2.0 * pix * (3 * w + w * 128 + 128 * 6)
        par = 4 * (2 * w * w * m * m * 8.0 + w * w * 4)
        by, fl = 4.0 * pix * (3 + 6 + 9 * w * 2) + 2 * par, 3.0 * fwd
    return dict(bytes=by, flops=fl)


# ------------------------------------------------------------------ float64 restatement

def _cpml(n, npml, off, dt, dx, dev):
    """CFS-CPML (b, a) at positions i + off: cubic grading, R0 = 1e-6, alpha_max 0.05."""
    p = np.arange(n) + off
    d_lo = np.clip((npml - p) / npml, 0, None)
    d_hi = np.clip((p - (n - 1 + 2 * off - npml)) / npml, 0, None)
    sig = 4 * math.log(1e6) / (2 * npml * dx) * (d_lo ** 3 + d_hi ** 3)
    dep = np.minimum(d_lo + d_hi, 1)
    al = np.where(dep > 0, 0.05 * (1 - dep), 0.0)
    b = np.exp(-(sig + al) * dt)
    a = np.where(sig > 0, sig * (b - 1) / np.where(sig > 0, sig + al, 1.0), 0.0)
    t = lambda v: torch.tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    return t(b), t(a)


def _amps(dt, steps):
    p = _pulse(dt, steps)
    w = 1.0 / p["fwidth"]
    t = (np.arange(steps) + 0.5) * dt - p["cutoff"] * w
    return np.cos(2 * math.pi * p["fcen"] * t) * np.exp(-t * t / (2 * w * w))


def _pole_consts(dt):
    out = []
    for p in POLES:
        fn, gam, s = p[:3]
        fc = p[3] if len(p) > 3 else fn
        w0, wc, g = (2 * math.pi * v for v in (fn, fc, gam))
        den = 1 + g * dt / 2
        out.append(((2 - w0 * w0 * dt * dt) / den, -(1 - g * dt / 2) / den,
                    s * wc * wc * dt * dt / den))
    return out


def _pad(x, x0, x1, y0, y1):
    return F.pad(x, (y0, y1, x0, x1))


class _Ref2D:
    """A 2D structure (or a stack of equal ones) in float64; state is a tuple."""

    def __init__(self, g, dev, eps=None):
        self.te = g["pol"] == "te"
        self.dt, self.dx = 0.5 * DX2, DX2
        nx, ny, npml = g["nx"], g["ny"], g["npml"]
        self.eps = (torch.from_numpy(g["eps"]).to(dev, torch.float64) if eps is None else eps)
        cp = lambda n, off: _cpml(n, npml, off, self.dt, self.dx, dev)  # noqa: E731
        self.hx = [v[:, None] for v in cp(nx - 1, 0.5)]
        self.hy = [v[None, :] for v in cp(ny - 1, 0.5)]
        self.ex = [v[1:-1, None] for v in cp(nx, 0.0)]
        self.ey = [v[None, 1:-1] for v in cp(ny, 0.0)]
        i, j0, j1 = g["src"]
        self.mask = torch.zeros(nx, ny, dtype=torch.float64, device=dev)
        self.mask[i, j0:j1] = 1.0 / self.dx if j1 - j0 > 1 else 1.0 / self.dx ** 2
        self.d1, self.d2, self.c = 1.0, self.dt, None
        av_x = lambda v: 0.5 * (v[..., :-1, :] + v[..., 1:, :])  # noqa: E731
        av_y = lambda v: 0.5 * (v[..., :-1] + v[..., 1:])  # noqa: E731
        if self.te:
            self.e = (av_x(self.eps), av_y(self.eps))
            self.mask = self.mask[:, :-1]
        if "masks" in g:
            sig = torch.from_numpy(g["sigma"]).to(dev, torch.float64)
            ms = [torch.from_numpy(m).to(dev, torch.float64) for m in g["masks"]]
            pair = lambda s: ((1 - s * self.dt / 2) / (1 + s * self.dt / 2),  # noqa: E731
                              self.dt / (1 + s * self.dt / 2))
            pc = _pole_consts(self.dt)
            stk = lambda f: [(c1, c2, c3 * f(m)) for (c1, c2, c3), m in zip(pc, ms)]  # noqa: E731
            if self.te:
                self.d1x, self.d2x = pair(av_x(sig))
                self.d1y, self.d2y = pair(av_y(sig))
                self.c = (stk(av_x), stk(av_y))
            else:
                self.d1, self.d2 = pair(sig)
                self.c = stk(lambda m: m)
        elif self.te:
            self.d1x = self.d1y = 1.0
            self.d2x = self.d2y = self.dt
        b = tuple(self.eps.shape[:-2])
        z = lambda *s: torch.zeros(*b, *s, dtype=torch.float64, device=dev)  # noqa: E731
        npol = len(POLES) if self.c is not None else 0
        zs = lambda *s: torch.zeros(npol, *s, dtype=torch.float64, device=dev)  # noqa: E731
        if self.te:
            self.names = ("Hz", "Ex", "Ey", "Dx", "Dy", "psi_Eyx", "psi_Exy", "psi_Hzy",
                          "psi_Hzx", "Px_cur", "Px_prev", "Py_cur", "Py_prev")
            self.s0 = (z(nx - 1, ny - 1), z(nx - 1, ny), z(nx, ny - 1), z(nx - 1, ny),
                       z(nx, ny - 1), z(nx - 1, ny - 1), z(nx - 1, ny - 1), z(nx - 1, ny - 2),
                       z(nx - 2, ny - 1), zs(nx - 1, ny), zs(nx - 1, ny), zs(nx, ny - 1),
                       zs(nx, ny - 1))
        else:
            self.names = ("Ez", "Hx", "Hy", "Dz", "psi_Ezy", "psi_Ezx", "psi_Hyx", "psi_Hxy",
                          "P_cur", "P_prev")
            self.s0 = (z(nx, ny), z(nx, ny - 1), z(nx - 1, ny), z(nx, ny), z(nx, ny - 1),
                       z(nx - 1, ny), z(nx - 2, ny - 2), z(nx - 2, ny - 2), zs(nx, ny),
                       zs(nx, ny))

    def step(self, s, amp):
        dx, dt = self.dx, self.dt
        dxf = lambda v: (v[..., 1:, :] - v[..., :-1, :]) / dx  # noqa: E731
        dyf = lambda v: (v[..., 1:] - v[..., :-1]) / dx  # noqa: E731
        pole = lambda c, pc, pp, e: torch.stack(  # noqa: E731
            [c1 * pc[k] + c2 * pp[k] + c3 * e for k, (c1, c2, c3) in enumerate(c)])
        if not self.te:
            ez, hx, hy, dz, p0, p1, p2, p3, pc, pp = s
            d = dyf(ez)
            p0 = self.hy[0] * p0 + self.hy[1] * d
            hx = hx - dt * (d + p0)
            d = dxf(ez)
            p1 = self.hx[0] * p1 + self.hx[1] * d
            hy = hy + dt * (d + p1)
            da, db = dxf(hy)[..., 1:-1], dyf(hx)[..., 1:-1, :]
            p2 = self.ex[0] * p2 + self.ex[1] * da
            p3 = self.ey[0] * p3 + self.ey[1] * db
            dz = self.d1 * dz + self.d2 * _pad(da + p2 - db - p3, 1, 1, 1, 1) - \
                self.d2 * amp * self.mask
            rhs = dz
            if self.c is not None:
                pc, pp = pole(self.c, pc, pp, ez), pc
                rhs = dz - pc.sum(0)
            return rhs / self.eps, hx, hy, dz, p0, p1, p2, p3, pc, pp
        hz, ex, ey, ddx, ddy, q2, q3, q0, q1, xc, xp, yc, yp = s
        d = dyf(hz)
        q0 = self.ey[0] * q0 + self.ey[1] * d
        ddx = self.d1x * ddx + self.d2x * _pad(d + q0, 0, 0, 1, 1)
        d = dxf(hz)
        q1 = self.ex[0] * q1 + self.ex[1] * d
        ddy = self.d1y * ddy - self.d2y * _pad(d + q1, 1, 1, 0, 0) - self.d2y * amp * self.mask
        rx, ry = ddx, ddy
        if self.c is not None:
            xc, xp = pole(self.c[0], xc, xp, ex), xc
            yc, yp = pole(self.c[1], yc, yp, ey), yc
            rx, ry = ddx - xc.sum(0), ddy - yc.sum(0)
        ex, ey = rx / self.e[0], ry / self.e[1]
        da, db = dxf(ey), dyf(ex)
        q2 = self.hx[0] * q2 + self.hx[1] * da
        q3 = self.hy[0] * q3 + self.hy[1] * db
        hz = hz - dt * (da + q2 - db - q3)
        return hz, ex, ey, ddx, ddy, q2, q3, q0, q1, xc, xp, yc, yp


def _phase(freqs, dt, steps, off, dev):
    """dt (cos wt, -sin wt), (steps, nf, 2); frequencies as the monitors keep them (32 bits)."""
    f = np.asarray(freqs, dtype=np.float32).astype(np.float64)
    wt = 2 * math.pi * f[None, :] * ((np.arange(steps) + off) * dt)[:, None]
    return torch.tensor(dt * np.stack([np.cos(wt), -np.sin(wt)], -1), device=dev)


def _lines2d(g, s, names):
    v = dict(zip(names, s))
    (ix, a, b), (iy, c, d) = g["x_line"], g["y_line"]
    if g["pol"] == "tm":
        hy, hx = v["Hy"], v["Hx"]
        return [(v["Ez"][ix, a:b], 0.5 * (hy[ix - 1, a:b] + hy[ix, a:b])),
                (v["Ez"][c:d, iy], 0.5 * (hx[c:d, iy - 1] + hx[c:d, iy]))]
    hz = v["Hz"]
    return [(v["Ey"][ix, a:b], 0.5 * (hz[ix - 1, a:b] + hz[ix, a:b])),
            (v["Ex"][c:d, iy], 0.5 * (hz[c:d, iy - 1] + hz[c:d, iy]))]


def _run_ref2d(ref, g, dev, segment=0):
    """(final state, flux accumulators, full DFT); with ``segment`` under checkpointing."""
    steps = g["steps"]
    amp = _amps(ref.dt, steps)
    p_full, p_half = (_phase(g["freqs"], ref.dt, steps, o, dev) for o in (1.0, 0.5))
    pe, ph = (p_half, p_full) if ref.te else (p_full, p_half)
    pd = p_half if ref.te else p_full          # DFT of Hz (half step) or of Ez (full step)
    full = None

    def part(s, t0, t1):
        rows = [[], [], [], []]
        for t in range(t0, t1):
            s = ref.step(s, float(amp[t]))
            for k, pair in enumerate(_lines2d(g, s, ref.names)):
                rows[2 * k].append(pair[0])
                rows[2 * k + 1].append(pair[1])
            if full is not None:
                full.add_(pd[t][:, :, None, None] * s[0])
        return (s, [torch.stack(r) for r in rows])

    if g["full"]:
        full = torch.zeros(len(g["freqs"]), 2, *ref.s0[0].shape, dtype=torch.float64, device=dev)
    s, chunks = ref.s0, []
    seg = segment or 256
    for t0 in range(0, steps, seg):
        t1 = min(steps, t0 + seg)
        if segment:
            s, rows = checkpoint(part, s, t0, t1, use_reentrant=False)
        else:
            s, rows = part(s, t0, t1)
        chunks.append(rows)
    accs = []
    for k in range(2):
        e, h = (torch.cat([c[2 * k + q] for c in chunks]) for q in range(2))
        accs.append(torch.cat([torch.einsum("tfc,tl->fcl", pe, e),
                               torch.einsum("tfc,tl->fcl", ph, h)], 1))
    return s, accs, full


def _flux2d(g, accs):
    sg = (0.5, -0.5) if g["pol"] == "te" else (-0.5, 0.5)
    return sum(q * ((a[:, 0] * a[:, 2] + a[:, 1] * a[:, 3]).sum(-1) * DX2).mean()
               for q, a in zip(sg, accs))


class _Ref3D:
    """A 3D structure in float64. Fields and CPML memory by name."""

    # component: ((curl axis, differenced field, sign), ...) of the H and E updates
    H = {"Hx": ((1, "Ez", 1), (2, "Ey", -1)), "Hy": ((2, "Ex", 1), (0, "Ez", -1)),
         "Hz": ((0, "Ey", 1), (1, "Ex", -1))}
    E = {"Ex": ((1, "Hz", 1), (2, "Hy", -1)), "Ey": ((2, "Hx", 1), (0, "Hz", -1)),
         "Ez": ((0, "Hy", 1), (1, "Hx", -1))}

    def __init__(self, g, dev, eps=None):
        self.g, self.dims = g, g["dims"]
        self.dx, self.dt = DX3, 0.5 * DX3 / math.sqrt(3.0)
        eps = torch.from_numpy(g["eps"]).to(dev, torch.float64) if eps is None else eps

        def shape(name):
            k = "xyz".index(name[1])
            return [n - ((a == k) == (name[0] == "E")) for a, n in enumerate(self.dims)]
        ax = lambda v, a: v.reshape([-1 if q == a else 1 for q in range(3)])  # noqa: E731
        self.hp, self.ep = [], []
        for a, n in enumerate(self.dims):
            self.hp.append([ax(v, a) for v in _cpml(n - 1, g["npml"], 0.5, self.dt, self.dx, dev)])
            self.ep.append([ax(v[1:-1], a) for v in _cpml(n, g["npml"], 0.0, self.dt, self.dx,
                                                           dev)])
        z = lambda s: torch.zeros(*s, dtype=torch.float64, device=dev)  # noqa: E731
        self.s0 = {k: z(shape(k)) for k in list(self.H) + list(self.E)}
        for name, terms in list(self.H.items()) + list(self.E.items()):
            for a, f, _ in terms:
                sh = shape(f)
                sh[a] -= 1
                self.s0[f"psi_{f}_{'xyz'[a]}"] = z(sh)
        avg = lambda v, a: 0.5 * (v.narrow(a, 0, v.shape[a] - 1) +  # noqa: E731
                                  v.narrow(a, 1, v.shape[a] - 1))
        self.eps = {"E" + k: avg(eps, a) for a, k in enumerate("xyz")}
        self.c3 = None
        if g["mask"] is not None:
            m = torch.from_numpy(g["mask"]).to(dev, torch.float64)
            c1, c2, c3 = _pole_consts(self.dt)[1]
            self.c1, self.c2 = c1, c2
            self.c3 = {"E" + k: c3 * avg(m, a) for a, k in enumerate("xyz")}
            for k in "xyz":
                for w in ("cur", "prev"):
                    self.s0[f"P{k}_{w}"] = z([1] + shape("E" + k))

    def step(self, s, amp):
        o = {}

        def term(f, a, prof, src):
            v = src[f]
            n = v.shape[a] - 1
            d = (v.narrow(a, 1, n) - v.narrow(a, 0, n)) / self.dx
            key = f"psi_{f}_{'xyz'[a]}"
            o[key] = prof[a][0] * s[key] + prof[a][1] * d
            return d + o[key]
        for name, terms in self.H.items():
            curl = sum(sg * term(f, a, self.hp, s) for a, f, sg in terms)
            o[name] = s[name] - self.dt * curl
        for name, terms in self.E.items():
            # each term lives on the interior of its own derivative axis; the curl on both
            axes = [t[0] for t in terms]
            parts = []
            for a, f, sg in terms:
                other = axes[0] if a == axes[1] else axes[1]
                v = term(f, a, self.ep, o)
                parts.append(sg * v.narrow(other, 1, v.shape[other] - 2))
            pad = [0] * 6
            for a in axes:
                pad[2 * (2 - a)] = pad[2 * (2 - a) + 1] = 1
            curl = F.pad(parts[0] + parts[1], pad)
            e = s[name]
            if self.c3 is None:
                o[name] = e + self.dt * curl / self.eps[name]
            else:
                k = name[1]
                pc, pp = s[f"P{k}_cur"], s[f"P{k}_prev"]
                pn = self.c1 * pc + self.c2 * pp + self.c3[name] * e
                o[f"P{k}_cur"], o[f"P{k}_prev"] = pn, pc
                o[name] = (e * self.eps[name] + pc[0] + self.dt * curl - pn[0]) / self.eps[name]
        i, j, k = self.g["src"]
        pt = torch.zeros_like(o["Ez"])
        pt[i, j, k] = self.dt * amp
        o["Ez"] = o["Ez"] + pt / self.eps["Ez"]
        return o

    def planes(self, s):
        """Ea, Ha, Eb, Hb on every face, H averaged across the plane."""
        out = []
        for (a, i), (l0, h0, l1, h1) in zip(self.g["faces"], self.g["wins"]):
            q = "xyz".index(a)
            pairs = {"z": ("Ex", "Hy", "Ey", "Hx"), "x": ("Ey", "Hz", "Ez", "Hy"),
                     "y": ("Ez", "Hx", "Ex", "Hz")}[a]
            for f in pairs:
                v = s[f]
                p = v.select(q, i) if f[0] == "E" else 0.5 * (v.select(q, i - 1) + v.select(q, i))
                out.append(p[l0:h0, l1:h1])
        return out


def _run_ref3d(ref, dev, segment=0):
    steps = ref.g["steps"]
    amp = _amps(ref.dt, steps)
    pe, ph = (_phase(ref.g["freqs"], ref.dt, steps, o, dev) for o in (1.0, 0.5))
    keys = list(ref.s0)

    def part(vals, accs, t0, t1):
        s = dict(zip(keys, vals))
        for t in range(t0, t1):
            s = ref.step(s, float(amp[t]))
            smp = ref.planes(s)
            accs = [a + (pe if k % 2 == 0 else ph)[t][:, :, None, None] * p
                    for k, (a, p) in enumerate(zip(accs, smp))]
        return [s[k] for k in keys], accs

    accs = [torch.zeros(len(ref.g["freqs"]), 2, *p.shape, dtype=torch.float64, device=dev)
            for p in ref.planes(ref.s0)]
    vals = [ref.s0[k] for k in keys]
    if segment:
        for t0 in range(0, steps, segment):
            vals, accs = checkpoint(part, vals, accs, t0, min(steps, t0 + segment),
                                    use_reentrant=False)
    else:
        vals, accs = part(vals, accs, 0, steps)
    faces = [torch.cat(accs[4 * k:4 * k + 4], 1) for k in range(len(accs) // 4)]
    return dict(zip(keys, vals)), faces


def _exact_fno(case, seed, dev):
    w, x, y = _fno_weights(case, seed)
    p = {k: v.to(dev, torch.complex128 if v.is_complex() else torch.float64).requires_grad_(True)
         for k, v in w.items()}
    x, y = x.to(dev, torch.float64), y.to(dev, torch.float64)
    b, n, m = case["batch"], case["size"], case["modes"]
    t = torch.linspace(0, 1, n, device=dev).double()
    v = torch.cat([x, t[:, None].expand(b, 1, n, n), t[None, :].expand(b, 1, n, n)], 1)
    mix = lambda v, q: torch.einsum("oi,bihw->bohw", p[q + ".weight"][:, :, 0, 0], v) + \
        p[q + ".bias"][None, :, None, None]  # noqa: E731
    v = mix(v, "lift")
    for k in range(4):
        f = torch.fft.rfft2(v)
        o = torch.zeros_like(f)
        o[:, :, :m, :m] = torch.einsum("bixy,ioxy->boxy", f[:, :, :m, :m], p[f"spec.{k}.w"][0])
        o[:, :, -m:, :m] = torch.einsum("bixy,ioxy->boxy", f[:, :, -m:, :m], p[f"spec.{k}.w"][1])
        v = torch.fft.irfft2(o, s=(n, n)) + mix(v, f"mix.{k}")
        if k < 3:
            v = F.gelu(v)
    out = mix(F.gelu(mix(v, "proj1")), "proj2")
    loss = _relative_error(out, y)
    loss.backward()
    # the order of the network's own parameters
    names = ["lift.weight", "lift.bias"] + [f"spec.{k}.w" for k in range(4)] + \
        [f"mix.{k}.{q}" for k in range(4) for q in ("weight", "bias")] + \
        [f"proj{k}.{q}" for k in (1, 2) for q in ("weight", "bias")]
    return dict(out=out.detach(), loss=loss.detach(),
                grads={k: (torch.view_as_real(p[k].grad) if p[k].is_complex() else p[k].grad)
                       for k in names})


_STATE_ORDER = {
    "tm": ("Ez", "Hx", "Hy", "Dz", "P_cur", "P_prev", "psi_Ezy", "psi_Ezx", "psi_Hyx", "psi_Hxy"),
    "te": ("Hz", "Ex", "Ey", "Dx", "Dy", "Px_cur", "Px_prev", "Py_cur", "Py_prev", "psi_Eyx",
           "psi_Exy", "psi_Hzy", "psi_Hzx"),
    "3d": ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz", "psi_Ez_y", "psi_Ey_z", "psi_Ex_z", "psi_Ez_x",
           "psi_Ey_x", "psi_Ex_y", "psi_Hz_y", "psi_Hy_z", "psi_Hx_z", "psi_Hz_x", "psi_Hy_x",
           "psi_Hx_y", "Px_cur", "Px_prev", "Py_cur", "Py_prev", "Pz_cur", "Pz_prev"),
}


def exact(case, seed):
    dev = _dev()
    kind = case["kind"]
    if kind == "run2d":
        g = _geom2d(case, seed)
        with torch.no_grad():
            ref = _Ref2D(g, dev)
            s, accs, full = _run_ref2d(ref, g, dev)
        v = dict(zip(ref.names, s))
        out = {k: v[k] for k in _STATE_ORDER[g["pol"]] if v[k].numel()}
        return dict(out, accs=accs + ([full] if full is not None else []))
    if kind == "batch":
        out = []
        with torch.no_grad():
            for g in _batch_geoms(case, seed):
                _, accs, full = _run_ref2d(_Ref2D(g, dev), g, dev)
                out.append(accs + [full])
        return out
    if kind == "designs":
        rho = _densities(case, seed).to(dev, torch.float64)
        n, d0, r0, steps = 256, 96, 64, case["steps"]
        eps = torch.ones(rho.shape[0], n, n, dtype=torch.float64, device=dev)
        eps[:, d0:d0 + 64, d0:d0 + 64] = 1.0 + 3.0 * rho
        g = dict(nx=n, ny=n, npml=20, pol="tm", src=(30, 20, n - 20))
        with torch.no_grad():
            ref = _Ref2D(g, dev, eps)
            w, t0 = 1.0 / 0.25, 5.0 / 0.25
            t = (np.arange(steps) + 0.5) * ref.dt - t0
            amp = np.cos(2 * math.pi * 0.65 * t) * np.exp(-t * t / (2 * w * w))
            ph = _phase((0.6, 0.65, 0.7), ref.dt, steps, 1.0, dev)
            acc = torch.zeros(rho.shape[0], 6, 128, 128, dtype=torch.float64, device=dev)
            s = ref.s0
            for k in range(steps):
                s = ref.step(s, float(amp[k]))
                acc += ph[k].reshape(1, 6, 1, 1) * s[0][:, None, r0:r0 + 128, r0:r0 + 128]
        return acc
    if kind == "run3d":
        with torch.no_grad():
            s, faces = _run_ref3d(_Ref3D(_geom3d(case, seed), dev), dev)
        keys = _STATE_ORDER["3d"][:6] if case["kept"] else _STATE_ORDER["3d"]
        return dict({k: s[k] for k in keys if k in s}, accs=faces)
    if kind == "grad2d":
        g = _geom2d(dict(case, full=False), seed)
        eps = torch.from_numpy(g["eps"]).to(dev, torch.float64).requires_grad_(True)
        _, accs, _ = _run_ref2d(_Ref2D(g, dev, eps), g, dev, segment=50)
        loss = _flux2d(g, accs)
        loss.backward()
        return dict(loss=loss.detach(), grad=eps.grad, accs=[a.detach() for a in accs])
    if kind == "grad3d":
        g = _geom3d(case, seed)
        eps = torch.from_numpy(g["eps"]).to(dev, torch.float64).requires_grad_(True)
        _, faces = _run_ref3d(_Ref3D(g, dev, eps), dev, segment=8)
        loss = 0.0
        for a in faces:
            sa = a[:, 0] * a[:, 2] + a[:, 1] * a[:, 3]
            sb = a[:, 4] * a[:, 6] + a[:, 5] * a[:, 7]
            loss = loss + (0.5 * (sa - sb).sum((1, 2)) * DX3 * DX3).mean()
        loss.backward()
        return dict(grad=eps.grad, accs=[a.detach() for a in faces])
    return _exact_fno(case, seed, dev)
