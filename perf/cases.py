"""The work a user of this framework has it do, as cases that can be timed.

A case is one pass through the public entry points: an inversion iteration
(forward, misfit, hand adjoint), a forward survey, or a run of the FEM data
generator, on the grids of the benchmark configurations (plate128, rot256,
shots1024, damage512, multi64, fields301, fem301), on the sizes between them
and on odd ones.  Long time axes are cut so that a pass stays below a second;
grids, shots and receivers are whole.

`exact` evaluates the same discrete scheme and its adjoint with plain torch
in 64 bits.
"""
import contextlib
import math

import numpy as np
import torch

import ernn_gb300 as E
from ernn_gb300 import fem as EF
from ernn_gb300 import harness
from ernn_gb300.propagate import Instances

H, DT, RHO = 1e-4, 5e-9, 1560.0            # the benchmark configurations' grid step, time step, density
GAUSS, AMP, F0 = 5e6, 1e10, 1e6            # point-load width, amplitude, burst frequency
BOX = 45                                   # cells beyond which the point load underflows to zero
C_ROT = (80.25e9, 21.25e9, 26.25e9, 37.23909236e9, 13.85640646e9, 25.75e9)  # orthotropic plate, rotated 30 degrees
C_ORTHO = (130e9, 12e9, 6e9, 0.0, 0.0, 5.5e9)
# the reference loops' plate: 0.4 m, 30 ns steps, Ricker source (their drop-in simulators)
LOOP = dict(L=0.4, dt=30e-9, f0=100e3, t0=10e-6, amplitude=1e10, rho=1610.0, gauss=5e6,
            C=(130.74e9, 11.50e9, 10.49e9, 30.67e9, 3.75e9, 14.77e9))
FEM = dict(L=0.4, dt=30e-9, rho=1610.0, gauss=5e6, f0=100e3, t0=10e-6, amplitude=1e10,
           C=(130.74e9, 11.50e9, 10.49e9, 30.67e9, 3.75e9, 14.77e9))
NAMES = ("C11", "C22", "C12", "C16", "C26", "C66")


def listed():
    return [
        # a quick look at a coupon: the smallest call, a hundred steps
        dict(name="coupon64", kind="traces", S=1, nx=64, ny=64, nt=120, R=16, stride=1, ckpt=0),
        # the orthotropic plate of the first benchmark configuration, whole, every state kept
        dict(name="plate128", kind="traces", S=1, nx=128, ny=128, nt=1000, R=32, stride=1, ckpt=0),
        # the headline inversion iteration as the harness replays it (one graph, Adam included)
        dict(name="rot256", kind="graph", S=1, nx=256, ny=256, nt=2000, R=64, stride=1, ckpt=100),
        # one shot on a grid between the plate and the survey sizes
        dict(name="line512", kind="traces", S=1, nx=512, ny=512, nt=800, R=128, stride=2, ckpt=0),
        # three shots on an odd grid (rows of no multiple of 16 bytes), checkpointed
        dict(name="odd501x389", kind="traces", S=3, nx=501, ny=389, nt=500, R=75, stride=1, ckpt=50),
        # the multi-shot survey: full grid, shots and receivers, checkpointed, the largest
        dict(name="shots1024", kind="traces", S=16, nx=1024, ny=1024, nt=400, R=256, stride=1, ckpt=80),
        # forward modelling only (synthetic observations for a survey design)
        dict(name="survey640x720", kind="survey", S=8, nx=640, ny=720, nt=400, R=128, stride=2, ckpt=0),
        # degradation imaging: per-cell map, gradient of every cell
        dict(name="damage512", kind="damage", S=8, nx=512, ny=512, nt=400, R=128, stride=1, ckpt=0),
        # many inversions of uneven sizes and step counts on one canvas
        dict(name="canvas8", kind="canvas", S=8, side_lo=128, side_hi=768, R=32, steps=5.2, ckpt=100),
        # the reference's parameter loop on its generator's grid: dense history, drop-in simulator
        dict(name="param301", kind="dense", nx=301, ny=301, nt=1001, stride=5, ts=1, ss=2),
        # the reference's damage loop on the same grid: six constant fields, TV term, drop-in simulator
        dict(name="fields301", kind="fields", nx=301, ny=301, nt=4001, stride=5, ts=2, ss=1),
        # the FEM data generator at its own size
        dict(name="fem301", kind="fem", nx=301, ny=301, nt=2001, stride=5, damaged=False),
    ]


LARGEST = 16 * 1024 * 1024 * 400  # cell steps of the largest listed pass with a gradient


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["traces", "traces", "traces", "survey", "damage", "canvas", "dense", "fields", "fem"])
    if kind in ("traces", "survey", "damage"):
        hi = 600 if kind == "damage" else 1024
        nx, ny = _log(rng, 48, hi), _log(rng, 48, hi)
        if rng.random() < 0.7:  # most grids have rows of whole 16-byte words
            ny -= ny % 4
        S = rng.randint(1, 16) if kind != "damage" else rng.randint(1, 8)
        top = LARGEST // 2 if kind != "damage" else 8 * 512 * 512 * 400
        nt = max(60, min(_log(rng, 100, 2000), top // (S * nx * ny)))
        return dict(kind=kind, S=S, nx=nx, ny=ny, nt=nt, R=rng.randint(4, min(128, nx - 4)),
                    stride=rng.choice([1, 1, 2, 3]), ckpt=0 if kind == "survey" else rng.choice([0, max(10, nt // 7)]))
    if kind == "canvas":
        return dict(kind=kind, S=rng.randint(2, 10), side_lo=64, side_hi=rng.choice([256, 384, 512]),
                    R=rng.randint(8, 48), steps=rng.choice([2.0, 3.5, 5.2]), ckpt=rng.choice([50, 100]))
    n = _log(rng, 61, 301)
    if kind == "dense":
        return dict(kind=kind, nx=n, ny=_log(rng, 61, 301), nt=_log(rng, 200, 1001), stride=rng.choice([1, 2, 5]),
                    ts=rng.choice([1, 2]), ss=rng.choice([1, 2, 3]))
    if kind == "fields":
        return dict(kind=kind, nx=n, ny=n, nt=_log(rng, 200, 2001), stride=rng.choice([2, 5]), ts=rng.choice([1, 2]), ss=1)
    return dict(kind=kind, nx=n, ny=_log(rng, 61, 301), nt=_log(rng, 200, 2001), stride=rng.choice([1, 5]),
                damaged=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed, salt=0):
    return torch.Generator(device=_dev()).manual_seed(1000003 * (salt + 1) + seed)


def _rand(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device=_dev(), dtype=torch.float64)


def _burst(nt):
    t = np.arange(nt) * DT
    T = 5 / F0
    return np.where(t <= T, 0.5 * (1 - np.cos(2 * np.pi * t / T)), 0.0) * np.sin(2 * np.pi * F0 * t) * AMP


def _point_load(nx, ny, i, j, bx, by):
    """Gaussian load around cell (i, j) in a box of (bx, by) cells: (map, origin)."""
    r0, c0 = max(0, min(i - bx // 2, nx - bx)), max(0, min(j - by // 2, ny - by))
    X, Y = np.meshgrid((np.arange(bx) + r0 - i) * H, (np.arange(by) + c0 - j) * H, indexing="ij")
    return (GAUSS / np.pi * np.exp(-GAUSS * (X * X + Y * Y))).astype(np.float32), (r0, c0)


def _spread(n, nx, margin):
    return [nx // 2] if n == 1 else [int(round(v)) for v in np.linspace(margin, nx - 1 - margin, n)]


def _sources(S, nx, ny, x0=0, y0=0):
    """Top-edge loads of S shots: maps (S, bx, by), origins (S, 2)."""
    bx, by = min(nx, 2 * BOX + 1), min(ny, 2 * BOX + 1)
    maps, orgs = zip(*(_point_load(nx, ny, i, ny - 1, bx, by) for i in _spread(S, nx, min(32, nx // 4))))
    return np.stack(maps), np.array([(r + x0, c + y0) for r, c in orgs], np.int32)


def _constants(base, g):
    """The guess in hand: the plate's constants, scaled and perturbed by a few per cent (stays positive-definite)."""
    return (torch.tensor(base, dtype=torch.float64, device=_dev()) * _rand(g, 1, 0.85, 1.05)
            * _rand(g, 6, 0.99, 1.01)).float()


def _observed_traces(g, S, frames, R, step):
    """Band-limited arrivals (tone-burst wave packets of random delay, phase and size) with 0.5 % noise: (S, frames, R)."""
    dev = _dev()
    t = (torch.arange(frames, device=dev, dtype=torch.float32) * (DT * step)).view(1, -1, 1)
    out = []
    for rms in (2e-3, 4e-3):
        o = torch.zeros((S, frames, R), device=dev)
        for _ in range(2):
            t0 = _rand(g, S * R, 0.1, 0.9).float().view(S, 1, R) * (frames * DT * step)
            ph = _rand(g, S * R, 0.0, 2 * math.pi).float().view(S, 1, R)
            a = _rand(g, S * R, 0.5, 2.0).float().view(S, 1, R) * rms
            o += a * torch.exp(-((t - t0) / 1.5e-6) ** 2) * torch.cos(2 * math.pi * F0 * (t - t0) + ph)
        out.append((o + 0.005 * rms * torch.randn(o.shape, generator=g, device=dev)).contiguous())
    return out


def _observed_frames(g, frames, nx, ny):
    """A wave packet spreading over the plate from its centre, frame by frame, with noise: (1, frames, nx, ny)."""
    dev = _dev()
    x = torch.linspace(-1, 1, nx, device=dev).view(1, -1, 1)
    y = torch.linspace(-1, 1, ny, device=dev).view(1, 1, -1)
    k = torch.arange(frames, device=dev, dtype=torch.float32).view(-1, 1, 1) / frames
    out = []
    for rms in (7e-3, 2e-2):
        c, w, s, ph = (float(v) for v in _rand(g, 4, 0.8, 1.2))
        r = torch.sqrt((x * s) ** 2 + y ** 2)
        o = 2 * rms * torch.exp(-((r - 1.5 * c * k) / (0.2 * w)) ** 2) * torch.cos(30 * (r - 1.5 * c * k) + 5 * ph)
        o += 0.01 * rms * torch.randn(o.shape, generator=g, device=dev)
        out.append(o.unsqueeze(0).contiguous())
    return out


def _receivers(nx, ny, R, both=False):
    if both:  # half on the top edge, half on the bottom edge
        a = R // 2
        return [(i, ny - 1) for i in _spread(R - a, nx, 2)] + [(i, 0) for i in _spread(a, nx, 2)]
    return [(i, ny - 1) for i in _spread(R, nx, 2)]


def _degradation(g, nx, ny, top):
    """A smooth map of a few soft spots in [0, top]."""
    x = torch.linspace(0, 1, nx, device=_dev(), dtype=torch.float64).view(-1, 1)
    y = torch.linspace(0, 1, ny, device=_dev(), dtype=torch.float64).view(1, -1)
    D = torch.zeros((nx, ny), device=_dev(), dtype=torch.float64)
    for _ in range(3):
        cx, cy, sx, sy, p = (float(v) for v in _rand(g, 5, 0.0, 1.0))
        D = torch.maximum(D, top * (0.4 + 0.6 * p) * torch.exp(
            -0.5 * (((x - 0.1 - 0.8 * cx) / (0.03 + 0.1 * sx)) ** 2 + ((y - 0.1 - 0.8 * cy) / (0.03 + 0.1 * sy)) ** 2)))
    return D.float()


def _gather_inputs(case, seed):
    """Inputs of the trace cases as plain tensors."""
    g, dev = _gen(seed), _dev()
    S, nx, ny, nt, R = (case[k] for k in ("S", "nx", "ny", "nt", "R"))
    maps, orgs = _sources(S, nx, ny)
    frames = -(-nt // case["stride"])
    damage = case["kind"] == "damage"
    rec = _receivers(nx, ny, R, both=damage)
    size = _rand(g, 1, 0.8, 1.2).cpu().numpy()  # the source's strength
    out = dict(sig=torch.tensor(np.repeat((_burst(nt) * size)[None], S, 0).astype(np.float32), device=dev),
               map=torch.tensor(maps, device=dev), org=torch.tensor(orgs, device=dev),
               rec=torch.tensor([[i * ny + j for i, j in rec]] * S, dtype=torch.int32, device=dev))
    out["C"] = torch.tensor(C_ORTHO, device=dev).float() if damage else _constants(C_ROT, g)
    if damage:
        out["D"] = _degradation(g, nx, ny, 0.3)
    out["obs"] = None if case["kind"] == "survey" else _observed_traces(g, S, frames, R, case["stride"])
    return out


def _sides(case, seed=0):
    """Grid sides of the instances: spread over the range, multiples of 64 (the same for every seed)."""
    n, lo, hi = case["S"], case["side_lo"] // 64, case["side_hi"] // 64
    return [64 * int(round(lo + (hi - lo) * k / max(1, n - 1))) for k in range(n)]


def _canvas_inputs(case, seed):
    g, dev = _gen(seed), _dev()
    sides, R = _sides(case), case["R"]
    nts = [int(round(case["steps"] * s)) for s in sides]
    ws = [harness.Workload(str(k), s, s, n, np.zeros(6), [(s // 2, s - 1)], _receivers(s, s, R))
          for k, (s, n) in enumerate(zip(sides, nts))]
    X, Y, x0, y0 = harness.canvas_layout(ws)
    S, T = len(ws), max(nts)
    sig = np.zeros((S, T), np.float32)
    maps, orgs = [], []
    B = min(min(sides), 2 * BOX + 1)
    for k, w in enumerate(ws):
        sig[k, :w.nt] = _burst(w.nt)
        m, o = _point_load(w.nx, w.ny, w.nx // 2, w.ny - 1, B, B)
        maps.append(m)
        orgs.append((o[0] + x0[k], o[1] + y0[k]))
    rec = [[(x0[k] + i) * Y + y0[k] + j for i, j in w.rec_cells] for k, w in enumerate(ws)]
    obs = _observed_traces(g, S, T, R, 1)
    for k in range(S):
        for o in obs:
            o[k, nts[k]:] = 0.0
    return dict(sides=sides, nts=nts, canvas=(X, Y), x0=x0, y0=y0, obs=obs,
                sig=torch.tensor(sig, device=dev), map=torch.tensor(np.stack(maps), device=dev),
                org=torch.tensor(orgs, dtype=torch.int32, device=dev),
                rec=torch.tensor(rec, dtype=torch.int32, device=dev),
                C=torch.stack([_constants(C_ROT, g) for _ in ws]))


def _log_fields(g, nx, ny):
    """Log-constants of an inversion under way: a uniform plate with smooth soft spots and a per-cell ripple, (6, nx, ny)."""
    D = _degradation(g, nx, ny, 0.3).double()
    out = []
    for c in LOOP["C"]:
        ripple = 0.01 * torch.rand((nx, ny), generator=g, device=_dev(), dtype=torch.float64)
        out.append((math.log(c) + torch.log1p(-D * float(_rand(g, 1, 0.5, 1.0))) - ripple).float())
    return out


def _loop_inputs(case, seed):
    """The reference loops' inputs: log-constants (scalars or fields) and the observed history."""
    g = _gen(seed)
    nx, ny = case["nx"], case["ny"]
    logs = _log_fields(g, nx, ny) if case["kind"] == "fields" else list(torch.log(_constants(LOOP["C"], g)))
    return dict(logs=logs, obs=_observed_frames(g, -(-case["nt"] // case["stride"]), nx, ny))


def _ricker(nt, dt, p):
    s = (np.pi * p["f0"] * (np.arange(nt) * dt - p["t0"])) ** 2
    return p["amplitude"] * (1 - 2 * s) * np.exp(-s)


def _fem_inputs(case, seed):
    g, dev = _gen(seed), _dev()
    nx, ny = case["nx"], case["ny"]
    dx, dy = FEM["L"] / (nx - 1), FEM["L"] / (ny - 1)
    cx, cy = (float(v) for v in _rand(g, 2, -0.05, 0.05))
    X, Y = np.meshgrid(np.linspace(-FEM["L"] / 2, FEM["L"] / 2, nx), np.linspace(-FEM["L"] / 2, FEM["L"] / 2, ny),
                       indexing="ij")
    load = FEM["gauss"] / np.pi * np.exp(-FEM["gauss"] * ((X - cx) ** 2 + (Y - cy) ** 2))
    cf = None
    if case["damaged"]:
        soft = torch.where(_degradation(g, nx, ny, 0.5) > 0.15, 0.5, 1.0)
        cf = (torch.tensor(FEM["C"], device=dev).view(6, 1, 1) * soft).float().contiguous()
    return dict(dx=dx, dy=dy, cf=cf, load=torch.tensor(load.astype(np.float32), device=dev),
                sig=torch.tensor(_ricker(case["nt"], FEM["dt"], FEM).astype(np.float32), device=dev))


# ------------------------------------------------------------------ one pass
def _geometry(case, i, nx, ny, nt, instances=None):
    return E.Geometry(nx=nx, ny=ny, nt=nt, h=H, dt=DT, src_signal=i["sig"], src_map=i["map"], src_origin=i["org"],
                      stride=case.get("stride", 1), src_comp=1, rec_idx=i["rec"], ckpt_k=case["ckpt"] or None,
                      instances=instances)


def prepare(case, seed):
    kind, dev = case["kind"], _dev()
    if kind in ("traces", "survey", "damage"):
        i = _gather_inputs(case, seed)
        geom = _geometry(case, i, case["nx"], case["ny"], case["nt"])
        st = dict(kind=kind, obs=i["obs"], rho=torch.tensor(RHO, device=dev), geom=geom)
        if kind == "damage":
            st["sim"] = E.DegradationSimulator(geom, i["C"].cpu().numpy(), RHO, i["D"]).to(dev)
        elif kind == "survey":
            st["sim"], st["C"] = E.ShotGatherSimulator(geom, RHO).to(dev), i["C"]
        else:
            st["C"] = i["C"].requires_grad_(True)
        return st
    if kind == "graph":
        i = _gather_inputs(case, seed)
        nx, ny = case["nx"], case["ny"]
        w = harness.Workload("plate", nx, ny, case["nt"], np.array(C_ROT), [(nx // 2, ny - 1)],
                             _receivers(nx, ny, case["R"]), ckpt_k=case["ckpt"] or None, stride=case["stride"])
        inv = harness.Inversion(w, dev, seed=seed)
        inv.geom.src_signal, inv.geom.src_map, inv.geom.src_origin = i["sig"], i["map"], i["org"]
        guess = i["C"] / inv.params.scale
        inv.capture()
        with torch.no_grad():
            inv.params.theta.copy_(guess)
        return dict(kind=kind, inv=inv, obs=i["obs"])
    if kind == "canvas":
        i = _canvas_inputs(case, seed)
        inst = Instances(i["x0"], i["y0"], i["sides"], i["sides"], i["nts"])
        geom = _geometry(case, i, *i["canvas"], max(i["nts"]), instances=inst)
        return dict(kind=kind, C=i["C"].requires_grad_(True), rho=torch.full((case["S"],), RHO, device=dev), geom=geom,
                    obs=i["obs"])
    if kind == "fem":
        i = _fem_inputs(case, seed)
        return dict(kind=kind, args=(case["nx"], case["ny"], case["nt"], i["dx"], i["dy"], FEM["dt"], FEM["rho"], FEM["C"],
                                     i["load"], i["sig"]),
                    kw=dict(stride=case["stride"], device=dev, C_fields=i["cf"]))
    i = _loop_inputs(case, seed)
    kw = dict(source_f0=LOOP["f0"], source_t0=LOOP["t0"], source_amplitude=LOOP["amplitude"], rho_known=LOOP["rho"],
              gaussian_param=LOOP["gauss"])
    cls = E.SpatiallyVaryingAnisotropicSimulator if kind == "fields" else E.CFRPWaveSimulatorRicker
    sim = cls((case["nx"], case["ny"]), LOOP["L"] / (case["nx"] - 1), LOOP["dt"], case["nt"], case["stride"], **kw).to(dev)
    with torch.no_grad():
        for n, v in zip(NAMES, i["logs"]):
            p = getattr(sim, "log_" + n)
            p.copy_(v.reshape(p.shape))
    return dict(kind=kind, sim=sim, obs=i["obs"], ts=case["ts"], ss=case["ss"])


def run(state):
    kind, obs = state["kind"], state.get("obs")
    if kind in ("traces", "canvas"):
        C = state["C"]
        C.grad = None
        ux, uy = E.propagate(C, state["rho"], state["geom"])
        E.series_misfit(ux, uy, obs[0], obs[1]).backward()
        return [ux.detach(), uy.detach(), C.grad]
    if kind == "damage":
        sim = state["sim"]
        sim.D.grad = None
        ux, uy = sim()
        E.series_misfit(ux, uy, obs[0], obs[1]).backward()
        return [ux.detach(), uy.detach(), sim.D.grad]
    if kind == "survey":
        with torch.no_grad():
            return list(state["sim"](state["C"]))
    if kind == "graph":
        inv = state["inv"]
        inv.step(obs)
        return [inv.gradient(), inv.params.theta.detach()]
    if kind == "fem":
        return list(EF.fem_frames(*state["args"], **state["kw"]))
    sim = state["sim"]
    for p in sim.parameters():
        p.grad = None
    ux, uy = sim()
    if kind == "fields":
        loss, _, _ = E.damage_loss(sim, ux, uy, obs[0], obs[1], state["ts"], 1e-21)
    else:
        loss = E.parameter_loss(ux, uy, obs[0], obs[1], state["ts"], state["ss"])
    loss.backward()
    return [ux.detach(), uy.detach()] + [getattr(sim, "log_" + n).grad for n in NAMES]


# ------------------------------------------------------------------ what a pass cannot do without
def _cell_steps(case):
    if case["kind"] == "canvas":
        return sum(s * s * int(round(case["steps"] * s)) for s in _sides(case))
    return case.get("S", 1) * case["nx"] * case["ny"] * case["nt"]


def work(case):
    """Bytes: inputs and outputs once.  Flops of a cell step: 18 for the stencil sums, 22 for the operator, 6 for the
    update; the same again for the adjoint and 20 for its imaging sums (6 more for each cell's own constants)."""
    kind, n = case["kind"], _cell_steps(case)
    frames = -(-case.get("nt", 1) // case.get("stride", 1))
    if kind == "fem":
        # about six triangles a node: strains 12, stresses 15, forces 8
        return {"bytes": 4.0 * case["nx"] * case["ny"] * (2 * frames + (7 if case["damaged"] else 1)),
                "flops": 6 * 35.0 * n}
    fwd, adj = 46.0, 66.0 + (6.0 if kind in ("damage", "fields") else 0.0)
    cells = case.get("nx", 0) * case.get("ny", 0)
    if kind in ("dense", "fields"):
        series = frames * cells
        extra = 12 * cells if kind == "fields" else 12
    elif kind == "canvas":
        series, extra = case["R"] * sum(int(round(case["steps"] * s)) for s in _sides(case)), 12 * case["S"]
    else:
        series, extra = case["S"] * frames * case["R"], 2 * cells if kind == "damage" else 12
    if kind == "survey":
        return {"bytes": 4.0 * (2 * series + 12), "flops": fwd * n}
    return {"bytes": 4.0 * (4 * series + extra), "flops": (fwd + adj) * n}


# ------------------------------------------------------------------ the scheme in 64 bits
def _sums(u):
    p = torch.nn.functional.pad(u, (1, 1, 1, 1))
    c2 = 2 * u
    xx = p[..., 2:, 1:-1] + p[..., :-2, 1:-1] - c2
    yy = p[..., 1:-1, 2:] + p[..., 1:-1, :-2] - c2
    xy = p[..., 2:, 2:] + p[..., :-2, :-2] - p[..., 2:, :-2] - p[..., :-2, 2:]
    return xx, yy, xy


class _Exact:
    """Forward loop and discrete adjoint of S shots: constants 0-dim or (nx, ny) in float64, load (S, nx, ny), signal (S, nt)."""

    def __init__(self, C, rho, h, dt, sig, load, src_comp=1):
        self.C, self.q, self.kappa = C, dt * dt / (rho * h * h), dt * dt / rho
        self.sig, self.load, self.comp = sig.double(), load.double(), src_comp

    def step(self, u):
        C11, C22, C12, C16, C26, C66 = self.C
        sx, sy = _sums(u[0]), _sums(u[1])
        m = 0.25 * (C12 + C66)
        lx = C11 * sx[0] + C66 * sx[1] + m * sy[2] + 0.5 * C16 * sx[2] + C16 * sy[0] + C26 * sy[1]
        ly = C66 * sy[0] + C22 * sy[1] + m * sx[2] + C16 * sx[0] + C26 * sx[1] + 0.5 * C26 * sy[2]
        return torch.stack([lx, ly]) * self.q

    def forward(self, nt, record, stride, keep):
        S, nx, ny = self.load.shape
        u = torch.zeros((2, S, nx, ny), dtype=torch.float64, device=self.load.device)
        prev, out = u, []
        self.states = []
        for i in range(nt):
            if keep:
                self.states.append(u)  # u^i
            new = 2 * u - prev + self.step(u)
            new[self.comp] += self.kappa * self.sig[:, i].view(-1, 1, 1) * self.load
            prev, u = u, new
            if i % stride == 0:
                out.append(record(u))
        return [torch.stack([o[c] for o in out], 1) for c in (0, 1)]

    def adjoint(self, nt, inject, per_cell):
        """dL/dC of the six constants ((S,) sums, or planes summed over shots), where inject(m, lam) adds dL/du^m."""
        C11, C22, C12, C16, C26, C66 = self.C
        m4 = 0.25 * (C12 + C66)
        l1 = torch.zeros_like(self.states[0])
        l2 = l1
        gr = [0.0] * 6
        for m in range(nt, 0, -1):
            lx, ly = l1[0], l1[1]
            ax = _sums(C11 * lx + C16 * ly)[0] + _sums(C66 * lx + C26 * ly)[1] + _sums(0.5 * C16 * lx + m4 * ly)[2]
            ay = _sums(C16 * lx + C66 * ly)[0] + _sums(C26 * lx + C22 * ly)[1] + _sums(m4 * lx + 0.5 * C26 * ly)[2]
            lam = 2 * l1 - l2 + self.q * torch.stack([ax, ay])
            inject(m, lam)
            l2, l1 = l1, lam
            u = self.states[m - 1]  # the imaging pair (lam^m, u^{m-1})
            sx, sy = _sums(u[0]), _sums(u[1])
            lx, ly = lam[0], lam[1]
            mixed = 0.25 * (lx * sy[2] + ly * sx[2])
            for k, v in enumerate((lx * sx[0], ly * sy[1], mixed, lx * (0.5 * sx[2] + sy[0]) + ly * sx[0],
                                   lx * sy[1] + ly * (sx[1] + 0.5 * sy[2]), lx * sx[1] + ly * sy[0] + mixed)):
                gr[k] = gr[k] + (v.sum(0) if per_cell else v.sum((1, 2)))
        return [self.q * v for v in gr]


def _dense_load(maps, orgs, nx, ny):
    out = torch.zeros((maps.shape[0], nx, ny), dtype=torch.float64, device=maps.device)
    for s, (r, c) in enumerate(orgs.tolist()):
        out[s, r:r + maps.shape[1], c:c + maps.shape[2]] = maps[s].double()
    return out


def _trace_solve(C, sig, maps, orgs, rec, obs, nx, ny, nt, stride, per_cell=False, count=None):
    """(traces x, traces y, gradients of the constants) of the MSE misfit."""
    S, R = rec.shape
    idx = rec.long()
    ex = _Exact(C, RHO, H, DT, sig, _dense_load(maps, orgs, nx, ny))
    pick = lambda u: torch.gather(u.reshape(2, S, -1), 2, idx.expand(2, S, R))  # noqa: E731
    out = ex.forward(nt, pick, stride, obs is not None)
    if obs is None:
        return out, None
    count = count or out[0].numel()
    res = [2 * (o - b.double()[:, :o.shape[1]]) / count for o, b in zip(out, obs)]

    def inject(m, lam):
        if (m - 1) % stride == 0:
            g = torch.stack([r[:, (m - 1) // stride] for r in res])
            lam.view(2, S, -1).scatter_add_(2, idx.expand(2, S, R), g)

    return out, ex.adjoint(nt, inject, per_cell)


def _exact_traces(case, seed):
    i = _gather_inputs(case, seed)
    nx, ny, nt, kind = case["nx"], case["ny"], case["nt"], case["kind"]
    if kind != "survey" and case["S"] * nx * ny * nt > 1.05 * LARGEST:
        return None
    C = [c for c in i["C"].double()]
    if kind == "graph":  # the constants are scale x theta, both held in float32
        sc = torch.tensor(np.array(C_ROT, np.float32), device=_dev())
        th = i["C"] / sc
        C = [c for c in sc.double() * th.double()]
    if kind == "damage":
        w = 1 - i["D"].double()
        C0, C = C, [w * c for c in C]
    out, gr = _trace_solve(C, i["sig"], i["map"], i["org"], i["rec"], i["obs"], nx, ny, nt, case["stride"], kind == "damage")
    if kind == "survey":
        return out
    if kind == "damage":
        return out + [-sum(c * g for c, g in zip(C0, gr))]
    g = torch.stack([v.sum() for v in gr])
    return [g * sc.double(), None] if kind == "graph" else out + [g]


def _exact_canvas(case, seed):
    i = _canvas_inputs(case, seed)
    S, R, T = case["S"], case["R"], max(i["nts"])
    out = [torch.zeros((S, T, R), dtype=torch.float64, device=_dev()) for _ in (0, 1)]
    grads = []
    Y = i["canvas"][1]
    for k, (s, n) in enumerate(zip(i["sides"], i["nts"])):
        org = i["org"][k:k + 1].cpu() - torch.tensor([[i["x0"][k], i["y0"][k]]])
        r = i["rec"][k:k + 1]
        rec = (r // Y - i["x0"][k]) * s + (r % Y - i["y0"][k])
        o, g = _trace_solve([c for c in i["C"][k].double()], i["sig"][k:k + 1, :n], i["map"][k:k + 1], org, rec,
                            [b[k:k + 1] for b in i["obs"]], s, s, n, 1, count=S * T * R)
        for c in (0, 1):
            out[c][k, :n] = o[c][0]
        grads.append(torch.stack([v.sum() for v in g]))
        torch.cuda.empty_cache()
    return out + [torch.stack(grads)]


def _exact_loop(case, seed):
    i = _loop_inputs(case, seed)
    nx, ny, nt, ts, ss, stride = (case[k] for k in ("nx", "ny", "nt", "ts", "ss", "stride"))
    fields = case["kind"] == "fields"
    h = LOOP["L"] / (nx - 1)
    x = torch.linspace(-h * (nx - 1) / 2, h * (nx - 1) / 2, nx, device=_dev())
    y = torch.linspace(-h * (ny - 1) / 2, h * (ny - 1) / 2, ny, device=_dev())
    X, Y = torch.meshgrid(x, y, indexing="ij")
    load = (LOOP["gauss"] / np.pi) * torch.exp(-LOOP["gauss"] * (X ** 2 + Y ** 2))
    sig = torch.tensor(_ricker(nt, LOOP["dt"], LOOP).astype(np.float32), device=_dev()).unsqueeze(0)
    bounds = [(50e9, 250e9), (5e9, 50e9), (5e9, 50e9), (0, 60e9), (0, 20e9), (5e9, 30e9)] if fields else [(1e9, 1e13)] * 6
    logs = [v.double().requires_grad_(True) for v in i["logs"]]
    C = [torch.clamp(torch.exp(v), *b) for v, b in zip(logs, bounds)]
    ex = _Exact([c.detach() for c in C], LOOP["rho"], h, LOOP["dt"], sig, load.t().unsqueeze(0) if fields else load.unsqueeze(0))
    out = ex.forward(nt, lambda u: u, stride, True)
    wx = 5.0 if fields else 1.0
    res = []
    for o, b, w in zip(out, i["obs"], (wx, 1.0)):
        d = o[:, ::ts, ::ss, ::ss] - b[:, ::ts, ::ss, ::ss].double()
        res.append(2 * w * d / d.numel())

    def inject(m, lam):
        if (m - 1) % stride == 0 and (m - 1) // stride % ts == 0:
            for c in (0, 1):
                lam[c][:, ::ss, ::ss] += res[c][:, (m - 1) // stride // ts]

    gr = ex.adjoint(nt, inject, fields)
    total = sum((c * (g if fields else g.sum())).sum() for c, g in zip(C, gr))
    if fields:
        tv = sum((c[1:] - c[:-1]).abs().sum() + (c[:, 1:] - c[:, :-1]).abs().sum() for c in C)
        total = total + 1e-21 * tv
    total.backward()
    return out + [v.grad.unsqueeze(0) if fields else v.grad for v in logs]


def _exact_fem(case, seed):
    i = _fem_inputs(case, seed)
    nx, ny, nt, dev = case["nx"], case["ny"], case["nt"], _dev()
    dx, dy = i["dx"], i["dy"]
    a, b = torch.meshgrid(torch.arange(nx - 1, device=dev), torch.arange(ny - 1, device=dev), indexing="ij")
    n0 = a * ny + b
    corner = [n0, n0 + ny, n0 + ny + 1, n0 + 1]  # (0, 0), (1, 0), (1, 1), (0, 1)
    at = [(0, 0), (1, 0), (1, 1), (0, 1)]
    even = (a + b) % 2 == 0
    cf = torch.tensor(FEM["C"], dtype=torch.float64, device=dev).view(6, 1).expand(6, nx * ny) if i["cf"] is None \
        else i["cf"].double().reshape(6, -1)
    parts, mass = [], torch.zeros(nx * ny, dtype=torch.float64, device=dev)
    for mask, tri, near in ((even, (0, 1, 2), 1), (even, (0, 2, 3), 3), (~even, (0, 1, 3), 0), (~even, (1, 2, 3), 2)):
        p = np.array([(at[t][0] * dx, at[t][1] * dy) for t in tri])
        J = np.array([p[1] - p[0], p[2] - p[0]])
        G = np.linalg.inv(J) @ np.array([[-1.0, 1, 0], [-1, 0, 1]])
        node = torch.stack([corner[t][mask] for t in tri])
        parts.append((torch.tensor(G, device=dev), node, cf[:, corner[near][mask]]))
        mass.index_add_(0, node.reshape(-1), torch.full((node.numel(),), FEM["rho"] * dx * dy / 6, dtype=torch.float64, device=dev))
    inside = torch.zeros((nx, ny), dtype=torch.float64, device=dev)
    inside[1:-1, 1:-1] = 1
    inside = inside.reshape(-1)
    load, sig = i["load"].double().reshape(-1) / FEM["rho"], i["sig"].double()
    u = torch.zeros((2, nx * ny), dtype=torch.float64, device=dev)
    prev = u
    out = {0: u, 1: u}
    for n in range(1, nt - 1):
        f = torch.zeros_like(u)
        for G, node, c in parts:
            ue = u[:, node]  # (2, 3, elements)
            exx, gy = torch.einsum("a,cae->ce", G[0], ue)
            gx, eyy = torch.einsum("a,cae->ce", G[1], ue)
            gxy = gx + gy
            sxx, syy = c[0] * exx + c[2] * eyy + c[3] * gxy, c[2] * exx + c[1] * eyy + c[4] * gxy
            sxy = c[3] * exx + c[4] * eyy + c[5] * gxy
            w = dx * dy / 2
            for v in range(3):
                f[0].index_add_(0, node[v], w * (G[0, v] * sxx + G[1, v] * sxy))
                f[1].index_add_(0, node[v], w * (G[1, v] * syy + G[0, v] * sxy))
        acc = -f / mass
        acc[1] += sig[n] * load
        new = inside * (2 * u - prev + FEM["dt"] ** 2 * acc)
        prev, u = u, new
        if (n + 1) % case["stride"] == 0:
            out[n + 1] = u
    frames = [out[k] for k in range(0, nt, case["stride"])]
    return [0.7 * torch.stack([f[c] for f in frames]).view(-1, nx, ny) for c in (0, 1)]


def exact(case, seed):
    solve = {"canvas": _exact_canvas, "dense": _exact_loop, "fields": _exact_loop, "fem": _exact_fem}
    grad = contextlib.nullcontext() if case["kind"] in ("dense", "fields") else torch.no_grad()
    with grad:
        return solve.get(case["kind"], _exact_traces)(case, seed)
