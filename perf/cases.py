"""The workloads whose speed this framework is judged by, each through its public calls.

A case is a dict of plain values.  Kinds:

* ``scene``   one resident grid (``Scene``): frames of a few updates, with an energy
  report and / or a colour-mapped frame after each, and the fields at the end.
* ``batch``   many uneven grids stepped together (``Batch``).
* ``serve``   requests run to their last frame by the serving loop (``Server``).
* ``dropin``  the reference's ``evolve_wave`` on its own row-pointer fields, with the
  fields kept on the GPU between calls (``resident``) or copied on every call (strict).

``exact`` restates the leapfrog update (mirror, periodic and absorbing edges, the
oscillating left edge, the point source) and the energy in 64-bit torch operations.
"""
import ctypes
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]


def _package():
    name = "youtube_simulations_gb300"
    if name not in sys.modules:
        d = ROOT / "youtube-simulations_gb300"
        spec = importlib.util.spec_from_file_location(name, d / "__init__.py", submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


_package()
from youtube_simulations_gb300 import params as P  # noqa: E402
from youtube_simulations_gb300 import wavegpu as W  # noqa: E402

BC = {"dirichlet": P.BC_DIRICHLET, "periodic": P.BC_PERIODIC, "absorbing": P.BC_ABSORBING}
D_ELLIPSE, D_STADIUM, D_CIRCLES = 1, 2, 20


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The headline run: a large two-medium grid with absorbing edges and a point source,
        # an energy report every 100 updates, in the precision long runs use.
        dict(name="scene_fp32_discs_3840x2160", kind="scene", nx=3840, ny=2160, prec=32, table=True, bc="absorbing",
             shape="discs", ndiscs=64, two=True, gamma=1e-4, source=True, osc=False, frames=5, per=100, energy=True, plot=-1),
        # The same grid with the values of the reference (64 bits).
        dict(name="scene_fp64_discs_3840x2160", kind="scene", nx=3840, ny=2160, prec=64, table=True, bc="absorbing",
             shape="discs", ndiscs=64, two=True, gamma=1e-4, source=True, osc=False, frames=1, per=100, energy=True, plot=-1),
        # A billiard film in 64 bits: ten updates a frame, the amplitude picture to the host.
        dict(name="film_fp64_ellipse_1280x720", kind="scene", nx=1280, ny=720, prec=64, table=False, bc="dirichlet",
             shape="ellipse", ndiscs=0, two=False, gamma=0.0, source=False, osc=False, frames=20, per=10, energy=False, plot=0),
        # A full-HD film coloured by the logarithm of the energy.
        dict(name="film_fp32_log_1920x1080", kind="scene", nx=1920, ny=1080, prec=32, table=True, bc="absorbing",
             shape="discs", ndiscs=24, two=True, gamma=0.0, source=False, osc=False, frames=10, per=10, energy=False, plot=4),
        # The smallest interactive call: one frame of a small billiard, where launches and
        # latency count.
        dict(name="frame_fp32_small_256x192", kind="scene", nx=256, ny=192, prec=32, table=False, bc="dirichlet",
             shape="ellipse", ndiscs=0, two=False, gamma=0.0, source=False, osc=False, frames=1, per=10, energy=False, plot=0),
        # An odd-sized stadium driven from its left edge.
        dict(name="scene_fp32_osc_1277x717", kind="scene", nx=1277, ny=717, prec=32, table=False, bc="dirichlet",
             shape="stadium", ndiscs=0, two=False, gamma=2e-4, source=False, osc=True, frames=4, per=50, energy=True, plot=-1),
        # Uneven billiards advanced together, mirror and periodic edges mixed.
        dict(name="batch_fp32_uneven_48", kind="batch", count=48, lo=256, hi=960, prec=32, sweep=False, frames=40, per=10),
        # The same mix in 64 bits.
        dict(name="batch_fp64_uneven_16", kind="batch", count=16, lo=256, hi=960, prec=64, sweep=False, frames=10, per=10),
        # A parameter sweep: many small absorbing rectangles with obstacles.
        dict(name="sweep_fp32_192", kind="batch", count=192, lo=128, hi=512, prec=32, sweep=True, frames=30, per=10),
        # A reference program that keeps its fields on the GPU between draws.
        dict(name="dropin_resident_1280x720", kind="dropin", nx=1280, ny=720, resident=True, bc="dirichlet",
             shape="ellipse", ndiscs=0, two=False, gamma=0.0, calls=100),
        # A reference program that reads its own arrays after every call.
        dict(name="dropin_strict_1280x720", kind="dropin", nx=1280, ny=720, resident=False, bc="absorbing",
             shape="discs", ndiscs=12, two=True, gamma=1e-4, calls=1),
        # A serving session: requests of several sizes, more than fit at once, frames to the host.
        dict(name="serve_fp32_8", kind="serve", count=8, slots=6, lo=256, hi=900, prec=32, frames=12, per=10),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["scene"] * 6 + ["batch"] * 2 + ["dropin"] * 2 + ["serve"])
    shape = rng.choice(["ellipse", "stadium", "discs"])
    two = shape == "discs" and rng.random() < 0.7
    common = dict(bc=rng.choice(sorted(BC)), shape=shape, ndiscs=rng.randint(1, 40) if shape == "discs" else 0, two=two,
                  gamma=rng.choice([0.0, 1e-4, round(rng.uniform(0, 1e-3), 6)]))
    if kind == "scene":
        prec = rng.choice([32, 32, 64])
        nx, ny = _log(rng, 96, 3840), _log(rng, 96, 2160)
        updates = rng.choice([10, 40, 100, 200])
        if prec == 64 and nx * ny > 2000000:
            updates = min(updates, 40)
        per = min(updates, rng.choice([1, 4, 10, 10, 50]))
        plot = rng.choice([-1, -1, 0, 0, 1, 4, 6, 8])
        frames = max(1, min(updates // per, 20 if plot >= 0 else 100))
        osc = rng.random() < 0.25 and common["bc"] == "dirichlet"
        return dict(kind="scene", nx=nx, ny=ny, prec=prec, table=rng.random() < 0.5, source=rng.random() < 0.25, osc=osc,
                    frames=frames, per=per, energy=rng.random() < 0.5, plot=plot, **common)
    if kind == "batch":
        prec, sweep = rng.choice([32, 32, 64]), rng.random() < 0.5
        lo = rng.randint(96, 256)
        return dict(kind="batch", count=rng.randint(2, 40 if sweep else 16), lo=lo, hi=rng.randint(lo + 32, 700), prec=prec,
                    sweep=sweep, frames=rng.randint(1, 12), per=rng.choice([1, 2, 5, 10, 10, 16]))
    if kind == "dropin":
        nx, ny, resident = _log(rng, 64, 1920), _log(rng, 64, 1080), rng.random() < 0.6
        return dict(kind="dropin", nx=nx, ny=ny, resident=resident, calls=rng.randint(5, 40) if resident else 1, **common)
    lo = rng.randint(96, 300)
    return dict(kind="serve", count=rng.randint(2, 8), slots=rng.randint(2, 6), lo=lo, hi=rng.randint(lo + 32, 800),
                prec=rng.choice([32, 32, 64]), frames=rng.randint(4, 12), per=rng.choice([5, 10, 10]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _rng(case, seed):
    return np.random.default_rng([int(seed), 20011])


def _grid(p):
    """Cell centres, in the reference's order of operations (on the host: a division by a
    number is a product with its reciprocal in torch on the GPU)."""
    x = p.xmin + np.arange(p.nx) * (p.xmax - p.xmin) / float(p.nx)
    y = p.ymin + np.arange(p.ny) * (p.ymax - p.ymin) / float(p.ny)
    return torch.from_numpy(x).cuda()[:, None], torch.from_numpy(y).cuda()[None, :]


def _mask(p, shape, lam, discs):
    x, y = _grid(p)
    if shape == "ellipse":
        return (x * x).cpu().div(lam * lam).cuda() + y * y < 1.0
    if shape == "stadium":
        m = (x > -0.5 * lam) & (x < 0.5 * lam) & (y > -1.0) & (y < 1.0)
        m = m | (torch.sqrt((x + 0.5 * lam) * (x + 0.5 * lam) + y * y) < 1.0)
        return m | (torch.sqrt((x - 0.5 * lam) * (x - 0.5 * lam) + y * y) < 1.0)
    m = torch.ones((p.nx, p.ny), dtype=torch.bool, device="cuda")
    for a, b, r in discs:
        m = m & ~((x - a) * (x - a) + (y - b) * (y - b) < r * r)
    return m


def _discs(rng, n, rmin, rmax, box=(-2.0, 2.0, -1.125, 1.125)):
    return [(float(rng.uniform(box[0], box[1])), float(rng.uniform(box[2], box[3])), float(rng.uniform(rmin, rmax)))
            for _ in range(n)]


def _waves(p, rng, mask, n):
    """n circular pulses (amplitude, width and wavelength drawn) on the cells that move."""
    x, y = _grid(p)
    f = torch.zeros((p.nx, p.ny), dtype=torch.float64, device="cuda")
    for _ in range(n):
        xc, yc = float(rng.uniform(-1.2, 1.2)), float(rng.uniform(-0.8, 0.8))
        var = math.exp(rng.uniform(math.log(0.02 ** 2), math.log(0.3)))
        r2 = (x - xc) ** 2 + (y - yc) ** 2
        f += float(rng.uniform(0.3, 1.0)) * torch.exp(-r2 / var) * torch.cos(torch.sqrt(r2) / float(rng.uniform(0.02, 0.06)))
    if not p.twospeeds:
        f = torch.where(mask, f, 0.0)
    return f


def _instance(sizes, rng, lo, hi, sweep):
    """One grid of a batch or a serving session: params, mask, initial field.  Sizes come
    from `sizes`, the same for every seed."""
    cells = math.exp(sizes.uniform(math.log(lo * lo), math.log(hi * hi)))
    if sweep:
        nx, ny = (int(round(math.exp(sizes.uniform(math.log(lo), math.log(hi))))) for _ in range(2))
        p = P.make_params(nx, ny, b_cond=P.BC_ABSORBING, courant=float(rng.uniform(0.05, 0.2)), gamma=float(rng.uniform(0.0, 1e-3)))
        m = _mask(p, "discs", 0.0, _discs(rng, int(rng.integers(1, 4)), 0.1, 0.3, (-1.6, 1.6, -0.8, 0.8)))
    else:
        nx = int(round(math.sqrt(cells * math.exp(sizes.uniform(0.0, math.log(16.0 / 9.0))))))
        ny = max(16, int(round(cells / nx)))
        p = P.make_params(nx, ny, b_cond=int(rng.choice([P.BC_DIRICHLET, P.BC_PERIODIC])), courant=float(rng.uniform(0.05, 0.15)))
        shape = ("ellipse", "stadium", "discs")[int(rng.integers(0, 3))]
        lam = float(rng.uniform(1.2, 1.9)) if shape == "ellipse" else float(rng.uniform(0.6, 1.6))
        r = float(rng.uniform(0.08, 0.18))
        m = _mask(p, shape, lam, [(a, b, r) for a in (-1.6, -0.8, 0.0, 0.8, 1.6) for b in (-0.8, 0.0, 0.8)])
    return p, m, _waves(p, rng, m, int(rng.integers(1, 4)))


def _instances(case, seed):
    rng, sizes = _rng(case, seed), np.random.default_rng([case["count"], case["lo"], case["hi"]])
    return [_instance(sizes, rng, case["lo"], case["hi"], case.get("sweep", False)) for _ in range(case["count"])]


def _single(case, seed):
    """Params, mask, initial field and the shape's parameters of a scene or drop-in case."""
    rng = _rng(case, seed)
    two = case["two"]
    p = P.make_params(case["nx"], case["ny"], b_cond=BC[case["bc"]], twospeeds=int(two), courant=0.1,
                      courantb=0.1 / 1.5 if two else 0.05, gamma=case["gamma"], gammab=case["gamma"])
    lam = {"ellipse": 1.8, "stadium": 1.2, "discs": 0.0}[case["shape"]]
    discs = _discs(rng, case["ndiscs"], 0.02, 0.1)
    m = _mask(p, case["shape"], lam, discs)
    if case.get("osc"):
        p.oscillate_left, p.omega, p.damping = 1, 0.02, 0.001
    if case.get("source"):
        p.src_on, p.src_amp, p.src_period = 1, 0.05, float(rng.uniform(20.0, 60.0))
        p.src_i, p.src_j = int(rng.integers(p.nx // 4, 3 * p.nx // 4)), int(rng.integers(p.ny // 4, 3 * p.ny // 4))
    return p, m, _waves(p, rng, m, int(rng.integers(2, 7))), lam, discs


def _lut():
    k = np.arange(256)
    return np.stack([k, 255 - k, (k * 7) % 256], axis=1).astype(np.uint8)


# ---------------------------------------------------------------------------
# What a program has in hand before the call
# ---------------------------------------------------------------------------
def _pinned(*shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def _prepare_scene(case, seed):
    p, m, f, lam, discs = _single(case, seed)
    prec = P.FP32 if case["prec"] == 32 else P.FP64
    dt = torch.float32 if case["prec"] == 32 else torch.float64
    s = W.Scene(p, prec, P.COEF_TABLE if case["table"] else P.COEF_MASK)
    domain = {"ellipse": D_ELLIPSE, "stadium": D_STADIUM, "discs": D_CIRCLES}[case["shape"]]
    s.build_domain(domain, lam=lam, circles=discs if discs else None)
    phi, psi = _pinned(p.nx, p.ny, dtype=dt), _pinned(p.nx, p.ny, dtype=dt)
    phi.copy_(f)
    s.upload_state(phi.numpy(), phi.numpy())
    rgb = None
    if case["plot"] >= 0:
        rgb = _pinned(case["frames"], p.ny // 2, p.nx // 2, 3, dtype=torch.uint8)
    scale = {0: 1.0, 1: 50.0, 4: 1.0, 6: 1.0, 8: 50.0}.get(case["plot"], 1.0)
    fp = P.WgFrameParams(2, 0, -0.2, 1.0, 1.0, 0.8, scale, 1.0, 0, max(case["plot"], 0), 0.75, 0.75, 250.0, 0.95, 0.0, 0, 0)
    return dict(case=case, s=s, prec=prec, phi=phi, psi=psi, rgb=rgb, fp=fp, lut=_lut())


def _prepare_batch(case, seed):
    b = W.Batch(P.FP32 if case["prec"] == 32 else P.FP64)
    slots, sizes = [], []
    for p, m, f in _instances(case, seed):
        h = f.cpu().numpy()
        slots.append(b.add(p, h, h, m.to(torch.int16).cpu().numpy()))
        sizes.append(p.nx * p.ny)
    phi, psi = _pinned(sum(sizes), dtype=torch.float64), _pinned(sum(sizes), dtype=torch.float64)
    return dict(case=case, b=b, slots=slots, sizes=sizes, phi=phi, psi=psi)


def _prepare_serve(case, seed):
    srv = W.Server(_lut(), precision=P.FP32 if case["prec"] == 32 else P.FP64, steps_per_frame=case["per"],
                   max_scenes=case["slots"], pipeline=True)
    reqs = [(p, f.cpu().numpy(), m.to(torch.int16).cpu().numpy()) for p, m, f in _instances(case, seed)]
    return dict(case=case, srv=srv, reqs=reqs)


def _prepare_dropin(case, seed):
    p, m, f, _, _ = _single(case, seed)
    h, xy = f.cpu().numpy(), m.to(torch.int16).cpu().numpy()
    tcc, tc, tg = (t.cpu().numpy() for t in _tables(p, m))
    W.configure(p)
    return dict(case=case, rf=W.RowFields(p, h, h, np.zeros_like(h), xy, tcc, tc, tg))


_PREPARE = {"scene": _prepare_scene, "batch": _prepare_batch, "serve": _prepare_serve, "dropin": _prepare_dropin}


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_scene(st):
    case, s, L = st["case"], st["s"], W.lib()
    energies = []
    for k in range(case["frames"]):
        s.step(case["per"])
        if case["energy"]:
            energies.append(s.total_energy())
        if st["rgb"] is not None:
            W.check(L.wg_scene_frame_rgb8(s.h, ctypes.byref(st["fp"]), st["lut"].ctypes.data, st["rgb"][k].data_ptr(), None))
    W.check(L.wg_scene_download(s.h, st["phi"].data_ptr(), st["psi"].data_ptr(), st["prec"]))
    return {"energy": np.array(energies), "frames": st["rgb"], "phi": st["phi"], "psi": st["psi"]}


def _run_batch(st):
    case, b, L = st["case"], st["b"], W.lib()
    for _ in range(case["frames"]):
        b.step(case["per"])
    phi, psi = st["phi"].data_ptr(), st["psi"].data_ptr()
    for slot, n in zip(st["slots"], st["sizes"]):
        W.check(L.wg_batch_download(b.h, slot, phi, psi))
        phi, psi = phi + 8 * n, psi + 8 * n
    return {"phi": st["phi"], "psi": st["psi"]}


def _run_serve(st):
    case, srv = st["case"], st["srv"]
    ids = [srv.submit(p, f, f, m, case["frames"] + k, keep=True) for k, (p, f, m) in enumerate(st["reqs"])]
    seen, last = dict.fromkeys(ids, 0), {}
    while True:
        srv.tick()
        alive = False
        for rid in ids:
            state, done = srv.state(rid)
            if done > seen[rid]:
                seen[rid], last[rid] = done, srv.frame(rid)[1]
            alive = alive or state in (P.REQ_QUEUED, P.REQ_RESIDENT)
        if not alive:
            break
    out = [srv.result(rid) for rid in ids]
    return {"frames": [last[rid] for rid in ids], "phi": [a for a, _ in out], "psi": [b for _, b in out]}


def _run_dropin(st):
    case, rf = st["case"], st["rf"]
    W.set_mode(case["resident"])
    for _ in range(case["calls"]):
        W.evolve_wave(rf)
    if not case["resident"]:
        return {"phi": rf.phi, "psi": rf.psi, "tmp": rf.tmp}
    columns = W.compute_energy_x(rf)
    W.sync()
    return {"columns": columns, "phi": rf.phi, "psi": rf.psi, "tmp": rf.tmp}


_RUN = {"scene": _run_scene, "batch": _run_batch, "serve": _run_serve, "dropin": _run_dropin}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the state (two levels), the mask and the table read once, the state, the
    frames and the returned fields written once.  Operations: 10 an update and cell."""
    kind = case["kind"]
    if kind in ("scene", "dropin"):
        cells = case["nx"] * case["ny"]
        if kind == "scene":
            s, updates = case["prec"] // 8, case["frames"] * case["per"]
            frames = case["frames"] * (cells // 4) * 3 if case["plot"] >= 0 else 0
            b = cells * (6 * s + 0.125 + (s if case["table"] else 0)) + frames
        else:
            updates, b = 3 * case["calls"], cells * 8 * (3 + 3 + 3) + cells * 2
        return {"bytes": b, "flops": 10.0 * cells * updates}
    lo, hi = case["lo"], case["hi"]
    if case.get("sweep"):
        cells = case["count"] * ((hi - lo) / math.log(hi / lo)) ** 2
    else:
        cells = case["count"] * (hi * hi - lo * lo) / math.log(hi * hi / (lo * lo))
    frames = case["frames"]
    b = cells * (4 * case["prec"] // 8 + 16 + 0.125)
    if kind == "serve":
        b += cells * 16 + cells / 4 * 3 * frames
    return {"bytes": b, "flops": 10.0 * cells * frames * case["per"]}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _tables(p, m):
    """tcc, tc, tgamma: the inside speed and damping where the mask is set, the outside
    ones elsewhere with two speeds, zero elsewhere without."""
    out = []
    for a, b in ((p.courant * p.courant, p.courantb * p.courantb), (p.courant, p.courantb), (p.gamma, p.gammab)):
        a, b = (torch.full_like(m, v, dtype=torch.float64) for v in (a, b if p.twospeeds else 0.0))
        out.append(torch.where(m, a, b))
    return out


def _update(p, x, y, t, m, tables):
    """phi(t+1) from x = phi(t) and y = phi(t-1)."""
    tcc, tc, tg = tables
    if p.b_cond == P.BC_PERIODIC:
        n, s, e, w = x.roll(-1, 0), x.roll(1, 0), x.roll(-1, 1), x.roll(1, 1)
    else:
        n, s = torch.cat([x[1:], x[-1:]]), torch.cat([x[:1], x[:-1]])
        e, w = torch.cat([x[:, 1:], x[:, -1:]], 1), torch.cat([x[:, :1], x[:, :-1]], 1)
    new = 2.0 * x - y + tcc * (n + s + e + w - 4.0 * x) - tg * (x - y)
    if p.b_cond == P.BC_ABSORBING:
        for a, b in ((0, 1), (-1, -2)):
            xa, xb, ya = x[a], x[b], y[a]
            new[a] = xa - tc[a] * (xa - xb) - p.kappa_sides * xa - p.gamma_sides * (xa - ya)
        for a, b in ((0, 1), (-1, -2)):
            xa, xb, ya = x[:, a], x[:, b], y[:, a]
            new[:, a] = xa - tc[:, a] * (xa - xb) - p.kappa_topbot * xa - p.gamma_topbot * (xa - ya)
    if not p.twospeeds:
        new = torch.where(m, new, y)
    if p.oscillate_left:
        a = p.amplitude * math.cos(t * p.omega) * math.exp(-t * p.omega * p.damping)
        new[0, :-1] = a
        if p.nx <= p.ny:
            new[0, p.nx - 1] = a
    if p.src_on:
        new[p.src_i, p.src_j] += p.src_amp * math.sin(2.0 * math.pi * t / p.src_period)
    return new


def _energy_cells(p, x, y, m):
    n, s = torch.cat([x[1:], x[-1:]]), torch.cat([x[:1], x[:-1]])
    e, w = torch.cat([x[:, 1:], x[:, -1:]], 1), torch.cat([x[:, :1], x[:, :-1]], 1)
    g = (n - x) ** 2 + (x - s) ** 2 + (e - x) ** 2 + (x - w) ** 2
    half = 0.5 * (_tables(p, m)[1] ** 2)
    cell = p.e_scale ** 2 * ((x - y) ** 2 + half * g)
    return cell if p.twospeeds else torch.where(m, cell, 0.0)


def _advance(p, m, f, updates):
    x, y, z, tables = f, f.clone(), torch.zeros_like(f), _tables(p, m)
    for t in range(1, updates + 1):
        x, y, z = _update(p, x, y, t, m, tables), x, y
    return x, y, z


def exact(case, seed):
    kind = case["kind"]
    if kind == "scene":
        p, m, f, _, _ = _single(case, seed)
        tables, x, y, t, energies = _tables(p, m), f, f.clone(), 0, []
        for _ in range(case["frames"]):
            for _ in range(case["per"]):
                t += 1
                x, y = _update(p, x, y, t, m, tables), x
            if case["energy"]:
                energies.append(float(_energy_cells(p, x, y, m).sum()))
        return {"energy": np.array(energies), "frames": None, "phi": x, "psi": y}
    if kind == "dropin":
        p, m, f, _, _ = _single(case, seed)
        x, y, z = _advance(p, m, f, 3 * case["calls"])
        out = {"phi": x, "psi": y, "tmp": z}
        if case["resident"]:
            out["columns"] = _energy_cells(p, x, y, m)[:, : p.ny // 2].sum(1)
        return out
    got = []
    for k, (p, m, f) in enumerate(_instances(case, seed)):
        frames = case["frames"] + (k if kind == "serve" else 0)
        got.append(_advance(p, m, f, frames * case["per"])[:2])
    if kind == "batch":
        return {"phi": torch.cat([a.reshape(-1) for a, _ in got]), "psi": torch.cat([b.reshape(-1) for _, b in got])}
    return {"frames": [None] * len(got), "phi": [a.reshape(-1) for a, _ in got], "psi": [b.reshape(-1) for _, b in got]}
