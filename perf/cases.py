"""Cases that stand for the work this library does for its users: the time step
of one domain (both precisions, both y boundaries, small to large), the step
taken as the reference's three subroutines, the batched form, the
differentiable form and the stateless counting sort.

A pass of a domain case advances the plasma by a few steps and takes a snapshot
of its state on the device (particle records in cell order, field planes) with
the energies on the host, as a program with in-situ diagnostics does. `exact`
states the same step in double precision with plain torch operations.
"""
import ctypes
import math

import numpy as np
import torch

from pbpic_b200 import _lib as L
from pbpic_b200 import configs
from pbpic_b200.autograd import DiffEngine, HarrisLoss
from pbpic_b200.batch import Batch
from pbpic_b200.sim import Simulation, counting_sort_keys

DEV = "cuda"


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest runs: a few thousand cells, a step is launches and latency
        dict(name="uniform_64x64_fp32", kind="step", plasma="uniform", mx=64, my=64, ppc=8, precision="fp32", steps=8),
        # the uniform periodic plasma of the named workloads, both precisions
        dict(name="uniform_128x128_fp32", kind="step", plasma="uniform", mx=128, my=128, ppc=32, precision="fp32",
             steps=4),
        dict(name="uniform_128x128_fp64", kind="step", plasma="uniform", mx=128, my=128, ppc=32, precision="fp64",
             steps=4),
        # a ragged domain: neither the rows nor the columns divide into tiles or warps, walls in y
        dict(name="harris_193x131_fp32", kind="step", plasma="harris", mx=193, my=131, ppc=37, precision="fp32",
             steps=2),
        # electron beams on immobile ions: few particles a cell
        dict(name="beams_256x192_fp32", kind="step", plasma="two_stream", mx=256, my=192, ppc=12, precision="fp32",
             steps=2),
        # the reference's loop through its three subroutines, particles tracked by
        # pid, the current read back
        dict(name="three_calls_256x128_fp64", kind="calls", plasma="uniform", mx=256, my=128, ppc=24, precision="fp64",
             steps=2, pid=True),
        # reconnection sheets: the benchmark's physics at 100 pairs a cell, both precisions
        dict(name="harris_512x256_fp32", kind="step", plasma="harris", mx=512, my=256, ppc=100, precision="fp32",
             steps=2),
        dict(name="harris_512x256_fp64", kind="step", plasma="harris", mx=512, my=256, ppc=100, precision="fp64",
             steps=2),
        # many small domains of uneven size advanced together
        dict(name="batch_12_domains", kind="batch", domains=12, side=128, ppc=48, steps=2),
        # a gradient of the sheet's loss: forward run and adjoint
        dict(name="gradient_magnetic_256x128", kind="gradient", loss="magnetic", mx=256, my=128, ppc=64,
             precision="fp32", steps=6, every=3),
        dict(name="gradient_jdote_96x80", kind="gradient", loss="jdote", mx=96, my=80, ppc=20, precision="fp64",
             steps=6, every=3),
        # the counting sort on a caller's own keys
        dict(name="sort_keys_5M", kind="sort", n=5_000_011, cells=131072),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "calls", "batch", "gradient", "sort"])
    if kind in ("step", "calls"):
        precision = rng.choice(["fp32", "fp64"])
        plasma = rng.choice(["uniform", "harris", "two_stream"])
        mx, my = _log_int(rng, 48, 512), _log_int(rng, 48, 256)
        ppc = min(_log_int(rng, 4, 128), 8_000_000 // (mx * my))
        # the smallest domains take the most steps a pass
        steps = 8 if mx * my * ppc < 100_000 else 4 if mx * my * ppc < 1_000_000 else 2
        return dict(kind=kind, plasma=plasma, mx=mx, my=my, ppc=max(ppc, 3), precision=precision,
                    steps=min(steps, 2) if kind == "calls" else steps, pid=kind == "calls")
    if kind == "batch":
        return dict(kind=kind, domains=rng.randint(4, 16), side=rng.choice([64, 96, 128]), ppc=_log_int(rng, 16, 64),
                    steps=2)
    if kind == "gradient":
        return dict(kind=kind, loss=rng.choice(["magnetic", "jdote"]), mx=_log_int(rng, 32, 256),
                    my=_log_int(rng, 32, 128), ppc=_log_int(rng, 8, 64), precision=rng.choice(["fp32", "fp64"]),
                    steps=6, every=rng.choice([2, 3, 6]))
    return dict(kind="sort", n=_log_int(rng, 50_000, 16_000_000) | 1, cells=_log_int(rng, 1_000, 1_000_000))


# ------------------------------------------------------------------- the inputs
def _workload(case):
    """Configuration and speeds of a domain case, from the repository's own configurations."""
    mx, my, ppc = case["mx"], case["my"], case["ppc"]
    if case["plasma"] == "uniform":
        return configs.uniform_c1(mx=mx, my=my, ppc=ppc)
    if case["plasma"] == "harris":
        return configs.harris(mx, my, ppc, seed=0)
    return configs.two_stream(mx, my, ppc, seed=0)


def _u(v):
    return v / math.sqrt(1.0 - v * v)


def _plasma(case, seed):
    """Seeded particles (position in cells, momentum, charge) and Yee planes, float64 on the device."""
    cfg, ld = _workload(case)
    mx, my = case["mx"], case["my"]
    n = case["ppc"] * mx * my
    g = torch.Generator(device=DEV).manual_seed(1_000_003 * int(seed) + 17)

    def uni(k):
        return torch.rand(k, generator=g, device=DEV, dtype=torch.float64)

    def normal(k):
        return torch.randn(k, 3, generator=g, device=DEV, dtype=torch.float64)

    x, y = uni(n) * mx, uni(n) * my
    fields = torch.zeros(6, mx, my + 1, dtype=torch.float64, device=DEV)
    ue, ui = normal(n) * _u(ld["vthe"]), None
    if case["plasma"] == "two_stream":
        # two counter-drifting beams, the ions a fixed background
        ue[:, 0] += torch.where(torch.arange(n, device=DEV) % 2 == 0, 1.0, -1.0) * _u(ld["vdrift_e"])
    else:
        ui = normal(n) * _u(ld["vthi"])
    if case["plasma"] == "uniform":
        fields[5] = ld["b0z"]
    if case["plasma"] == "harris":
        lam, dx, dy = ld["lambda_"], cfg["dx"], cfg["dy"]
        lx, ly = mx * dx, my * dy
        ns = int(n * 2 * lam / (2 * lam + ld["nb"] * ly))
        # sech^2 sheet in the middle, kept inside the walls
        edge = math.tanh(0.5 * ly / lam)
        y[:ns] = (0.5 * ly + lam * torch.atanh((2 * uni(ns) - 1) * edge)) / dy
        y.clamp_(0.0, my * (1 - 1e-9))
        ue[:ns, 2] += _u(ld["vdrift_e"])
        ui[:ns, 2] += _u(ld["vdrift_i"])
        xn = (torch.arange(mx, device=DEV, dtype=torch.float64) * dx)[:, None]
        yn = (torch.arange(my + 1, device=DEV, dtype=torch.float64) * dy - 0.5 * ly)[None, :]
        psi0, kx, ky = ld["psi0"], 2 * math.pi / lx, math.pi / ly
        fields[3] = torch.tanh(yn / lam) - psi0 * ky * torch.cos(kx * (xn + 0.5 * dx)) * torch.sin(ky * yn)
        fields[4] = psi0 * kx * torch.sin(kx * xn) * torch.cos(ky * (yn + 0.5 * dy))
        fields[4][:, my] = 0.0
    if cfg["ybc"] == L.BC_PERIODIC:
        fields[:, :, my] = 0.0  # the planes' last row belongs to walls only
    if ui is None:
        u, q = ue, torch.full((n,), -1, dtype=torch.int32, device=DEV)
    else:  # pairs at one point, ion and electron in turn
        x, y = x.repeat_interleave(2), y.repeat_interleave(2)
        u = torch.stack([ui, ue], 1).reshape(-1, 3)
        q = torch.tensor([1, -1], dtype=torch.int32, device=DEV).repeat(n)
    ix, iy = x.floor().clamp_(0, mx - 1), y.floor().clamp_(0, my - 1)
    real = torch.float32 if case["precision"] == "fp32" else torch.float64
    part = torch.stack([x - ix - 0.5, y - iy - 0.5, u[:, 0], u[:, 1], u[:, 2]], 1).to(real).clamp_(-0.999, 0.999)
    part[:, :2].clamp_(-0.4999999, 0.4999999)
    return cfg, part, (ix * my + iy).to(torch.int32), q, fields.to(real).to(torch.float64)


def _domain(case, seed):
    cfg, part, cell, q, fields = _plasma(case, seed)
    n = part.shape[0]
    rec = L.PARTICLE_F32 if case["precision"] == "fp32" else L.PARTICLE_F64
    host = np.zeros(n, dtype=rec)
    cols = part.cpu().numpy()
    for k, name in enumerate(("dx", "dy", "ux", "uy", "uz")):
        host[name] = cols[:, k]
    host["grid"] = cell.cpu().numpy() + 1
    host["q"] = q.cpu().numpy()
    host["pid"] = np.arange(n, dtype=np.int32)
    sim = Simulation.from_config(cfg, precision=case["precision"], capacity=n, track_pid=bool(case.get("pid")))
    sim.load_particles(host)
    sim.load_fields(fields.cpu().numpy())
    sim.countingsort()
    return sim, n, cfg["ybc"]


class _Snapshot:
    """Device buffers for a domain's state: its records in cell order and its field planes."""

    def __init__(self, sim, n, precision, pid=False):
        self.sim, self.n, self.pid = sim, n, pid
        self.f32 = precision == "fp32"
        self.words = 8 if self.f32 else 14
        self.rec = torch.zeros(n, self.words, dtype=torch.int32, device=DEV)
        rows = sim.my + (1 if sim.cfg.ybc == L.BC_CONDUCTING else 0)
        self.rows = rows
        self.planes = torch.zeros(6, sim.mx, rows, dtype=torch.float32 if self.f32 else torch.float64, device=DEV)

    def take(self):
        lib, sim, got = L.lib(), self.sim, ctypes.c_int64()
        L.check(lib.pbpic_band_extract(sim.handle, 0, sim.my, sim.my, 0, ctypes.c_void_p(self.rec.data_ptr()), self.n,
                                       ctypes.byref(got)))
        L.check(lib.pbpic_field_rows_get(sim.handle, 0, self.rows, ctypes.c_void_p(self.planes.data_ptr())))
        if self.f32:
            reals, at = self.rec.view(torch.float32)[:, :5], 5
        else:
            reals, at = self.rec.view(torch.float64)[:, :5], 10
        return {"particles": reals, "where": self.rec[:, at:at + (3 if self.pid else 2)], "fields": self.planes}


def _at_precision(energies, precision):
    """Energies come as doubles; those of the FP32 form are sums of FP32 terms."""
    return energies.astype(np.float32) if precision == "fp32" else energies


def _batch_domains(case, seed):
    out = []
    side, ppc = case["side"], case["ppc"]
    for i in range(case["domains"]):
        mx, my = side - 8 * (i % 4), side // (1 + i % 2) + 3 * (i % 3)
        p = max(4, ppc - 5 * (i % 5))
        make = configs.two_stream if i % 2 == 0 else configs.weibel
        out.append(make(mx, my, p, 7919 * int(seed) + i))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "calls"):
        sim, n, _ = _domain(case, seed)
        return dict(case=case, sim=sim, snap=_Snapshot(sim, n, case["precision"], bool(case.get("pid"))))
    if kind == "batch":
        b = Batch(_batch_domains(case, seed))
        sims = [b.domain(i) for i in range(b.n)]
        return dict(case=case, batch=b, snaps=[_Snapshot(s, s.num_particles(), "fp32") for s in sims])
    if kind == "gradient":
        rng = np.random.default_rng(seed)
        params = torch.tensor([0.1, 0.2, 5.0], dtype=torch.float64) * torch.from_numpy(1 + 0.05 * rng.uniform(-1, 1, 3))
        engine = DiffEngine(case["mx"], case["my"], case["ppc"], nsteps=case["steps"], checkpoint_every=case["every"],
                            precision=case["precision"], loss=case["loss"], seed=int(seed) + 1)
        return dict(case=case, engine=engine, params=params.requires_grad_(True))
    keys = _keys(case, seed)
    return dict(case=case, keys=keys, perm=torch.zeros_like(keys),
                counts=torch.zeros(case["cells"], dtype=torch.int32, device=DEV))


def _keys(case, seed):
    """Cells of particles that were in order a step ago: mostly runs, a few moved to a cell nearby, and a tenth anywhere."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 29)
    n, cells = case["n"], case["cells"]
    k = torch.randint(0, cells, (n,), generator=g, device=DEV).sort().values
    r = torch.rand(n, generator=g, device=DEV)
    k = torch.where(r < 0.1, (k + torch.randint(-2, 3, (n,), generator=g, device=DEV)) % cells, k)
    return torch.where(r > 0.9, torch.randint(0, cells, (n,), generator=g, device=DEV), k).to(torch.int32)


# --------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        state["sim"].step(case["steps"], 1)
        out = state["snap"].take()
        out["energies"] = _at_precision(state["sim"].energies(), case["precision"])
        return out
    if kind == "calls":
        sim = state["sim"]
        for _ in range(case["steps"]):
            sim.pusher()
            sim.fieldsolver()
            sim.countingsort()
        out = state["snap"].take()
        out["denjr"] = sim.denjr() if case["precision"] == "fp64" else sim.denjr().astype(np.float32)
        out["energies"] = _at_precision(sim.energies(), case["precision"])
        return out
    if kind == "batch":
        state["batch"].step(case["steps"])
        out = {"energies": _at_precision(state["batch"].energies(), "fp32")}
        for i, s in enumerate(state["snaps"]):
            out["domain%02d" % i] = s.take()
        return out
    if kind == "gradient":
        p = state["params"]
        p.grad = None
        loss = HarrisLoss.apply(p, state["engine"])
        loss.backward()
        real = torch.float32 if case["precision"] == "fp32" else torch.float64
        return {"loss": loss.detach().to(real), "grad": p.grad.to(real)}
    counting_sort_keys(state["keys"].data_ptr(), case["n"], case["cells"], state["perm"].data_ptr(),
                       state["counts"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return {"perm": state["perm"], "counts": state["counts"]}


def work(case):
    """Bytes that have to move and operations of one pass: a step reads and
    writes each particle (cell word, 5 reals) and the fields and current of each
    cell once; a snapshot writes the records and planes."""
    kind = case["kind"]

    def domain(n, cells, real, steps, record):
        step = n * 2 * (4 + 5 * real) + cells * (12 * real + 3 * real)
        return steps * step + n * (4 + 5 * real + record) + 12 * cells * real, steps * n * 200

    if kind in ("step", "calls"):
        cells = case["mx"] * case["my"]
        n = case["ppc"] * cells * (1 if case["plasma"] == "two_stream" else 2)
        real = 4 if case["precision"] == "fp32" else 8
        b, f = domain(n, cells, real, case["steps"], 32 if real == 4 else 56)
        if kind == "calls":
            b += 32 * cells
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0
        for cfg, ld in _batch_domains(case, 0):
            cells = cfg["mx"] * cfg["my"]
            db, df = domain(ld["ppc"] * cells * (1 if ld.get("immobile_ions") else 2), cells, 4, case["steps"], 32)
            b, f = b + db, f + df
        return {"bytes": b, "flops": f}
    if kind == "gradient":
        n = 2 * case["ppc"] * case["mx"] * case["my"]
        real = 4 if case["precision"] == "fp32" else 8
        # forward, recomputed forward and adjoint: the state read and written,
        # the adjoint state read and written beside the state
        state = 4 + 5 * real
        return {"bytes": case["steps"] * n * (2 * state + 2 * state + state + 10 * real),
                "flops": case["steps"] * n * 900}
    return {"bytes": 8 * case["n"] + 4 * case["cells"], "flops": 0}


# ------------------------------------------------ the same in double precision
def _images(comp, gx, gy, mx, my, walls):
    """Entry and sign of deposit node (gx, gy) of component comp (0 jx, 1 jy, 2 jz, 3 rho)."""
    sign = torch.ones_like(gx, dtype=torch.float64)
    gx = gx % mx
    if not walls:
        return gx * (my + 1) + gy % my, sign
    if comp in (0, 3):  # node rows mirror about the walls
        gy = gy.abs()
        return gx * (my + 1) + torch.where(gy > my, 2 * my - gy, gy), sign
    out = (gy < 0) | (gy > my - 1)
    if comp == 1:
        sign = torch.where(out, -1.0, 1.0).to(torch.float64)
    gy = torch.where(gy < 0, -1 - gy, gy)
    return gx * (my + 1) + torch.where(gy > my - 1, 2 * my - 1 - gy, gy), sign


def _half(f, my, walls, image):
    """Rows -1 .. my of a half-row component: wrapped, or imaged with the sign at walls."""
    f = f[:, :my]
    if walls:
        return torch.cat([image * f[:, :1], f, image * f[:, -1:]], 1)
    return torch.cat([f[:, -1:], f, f[:, :1]], 1)


def _node_rows(f, my, walls):
    """Rows 0 .. my of a node-row component."""
    return f[:, :my + 1] if walls else torch.cat([f[:, :my], f[:, :1]], 1)


def _nodes(f, my, walls):
    """Node averages (6, mx, my + 1); node column mx is column 0."""
    def back(a):
        return torch.roll(a, 1, 0)

    ex, bx = _node_rows(f[0], my, walls), _node_rows(f[3], my, walls)
    ey, by = _half(f[1], my, walls, 1.0), _half(f[4], my, walls, -1.0)
    ez, bz = _half(f[2], my, walls, -1.0), _half(f[5], my, walls, 1.0)

    def y2(a):
        return a[:, 1:] + a[:, :-1]

    return torch.stack([(ex + back(ex)) / 2, y2(ey) / 2, (y2(ez) + y2(back(ez))) / 4,
                        (bx + back(bx)) / 2, y2(by) / 2, (y2(bz) + y2(back(bz))) / 4])


def _b_half(f, h, idx, idy, my, walls):
    ez = _half(f[2], my, walls, -1.0)
    ex = _node_rows(f[0], my, walls)
    rows = my + 1 if walls else my
    f[3][:, :rows] -= h * ((ez[:, 1:] - ez[:, :-1]) * idy)[:, :rows]
    f[4][:, :my] += h * (f[2] - torch.roll(f[2], 1, 0))[:, :my] * idx
    f[5][:, :my] += h * ((ex[:, 1:] - ex[:, :-1]) * idy - (torch.roll(f[1], -1, 0) - f[1])[:, :my] * idx)


def _step(p, cell, q, f, cfg):
    """One step: particles p (n, 5) in cell order, planes f; returns the new state, the current and the energies."""
    mx, my, dt, cva, mime = cfg["mx"], cfg["my"], cfg["dt"], cfg["cva"], cfg["mime"]
    dx, dy, walls = cfg["dx"], cfg["dy"], cfg["ybc"] == L.BC_CONDUCTING
    ix, iy = cell // my, cell % my
    qd = q.double()
    mass = torch.where(q > 0, mime, 1.0).double()
    g = _nodes(f, my, walls)
    px, py, u = p[:, 0], p[:, 1], p[:, 2:5]
    eb = 0.0
    for a, b, w in ((0, 0, (0.5 - px) * (0.5 - py)), (1, 0, (0.5 + px) * (0.5 - py)),
                    (0, 1, (0.5 - px) * (0.5 + py)), (1, 1, (0.5 + px) * (0.5 + py))):
        eb = eb + w * g[:, (ix + a) % mx, iy + b]
    e, bf = eb[:3].T, eb[3:].T
    c0 = (qd * dt * mime / mass / 2)[:, None]
    um = u + c0 / cva * e
    t = c0 / torch.sqrt(1 + (um * um).sum(1, keepdim=True)) * bf
    s = 2 * t / (1 + (t * t).sum(1, keepdim=True))
    u = um + torch.linalg.cross(um + torch.linalg.cross(um, t), s) + c0 / cva * e
    gamma = torch.sqrt(1 + (u * u).sum(1))
    ke = (u * u).sum(1) / (gamma + 1) * mass
    x1 = px + dt * cva / gamma * u[:, 0] / dx
    y1 = py + dt * cva / gamma * u[:, 1] / dy
    cx = (x1 > 0.5).long() - (x1 < -0.5).long()
    cy = (y1 > 0.5).long() - (y1 < -0.5).long()
    # zig-zag: two segments that meet at the relay point, in cell units from the old cell's corner
    xs, xe, ys, ye = px + 0.5, x1 + 0.5, py + 0.5, y1 + 0.5
    xm, ym = (xs + xe) / 2, (ys + ye) / 2
    xr = torch.where(cx == 0, xm, (cx > 0).double())
    yr = torch.where(cy == 0, ym, (cy > 0).double())
    j = torch.zeros(4, mx * (my + 1), dtype=torch.float64, device=p.device)

    def add(comp, gx, gy, v):
        k, sign = _images(comp, gx, gy, mx, my, walls)
        j[comp] += torch.bincount(k, weights=v * sign, minlength=mx * (my + 1))

    for ox, oy, xa, xb, ya, yb in ((0, 0, xs, xr, ys, yr), (cx, cy, xr, xe, yr, ye)):
        wx, wy = (xa + xb) / 2 - ox, (ya + yb) / 2 - oy
        fx, fy = qd * dx / dt * (xb - xa), qd * dy / dt * (yb - ya)
        add(0, ix + ox, iy + oy, fx * (1 - wy))
        add(0, ix + ox, iy + oy + 1, fx * wy)
        add(1, ix + ox, iy + oy, fy * (1 - wx))
        add(1, ix + ox + 1, iy + oy, fy * wx)
    vz = qd * u[:, 2] * cva / gamma
    sx, sy = torch.where(xm >= 0.5, 1, -1), torch.where(ym >= 0.5, 1, -1)
    ax, ay = (xm - 0.5).abs(), (ym - 0.5).abs()
    for ox, wx in ((0, 1 - ax), (sx, ax)):
        for oy, wy in ((0, 1 - ay), (sy, ay)):
            add(2, ix + ox, iy + oy, vz * wx * wy)
    for a, wx in ((0, 1 - xs), (1, xs)):
        for b, wy in ((0, 1 - ys), (1, ys)):
            add(3, ix + a, iy + b, qd * wx * wy)
    j = j.reshape(4, mx, my + 1) * cfg["in0"]
    # fields: B half, E, B half
    idx, idy = 1 / dx, 1 / dy
    f = f.clone()
    _b_half(f, dt / 2, idx, idy, my, walls)
    bz, bx = _half(f[5], my, walls, 1.0), _node_rows(f[3], my, walls)
    rows = my + 1 if walls else my
    cdt = dt * cva ** 2
    f[0][:, :rows] += cdt * ((bz[:, 1:] - bz[:, :-1]) * idy - j[0])[:, :rows]
    if walls:
        f[0][:, 0] = f[0][:, my] = 0.0
    f[1][:, :my] -= cdt * ((f[5] - torch.roll(f[5], 1, 0)) * idx + j[1])[:, :my]
    f[2][:, :my] += cdt * ((torch.roll(f[4], -1, 0) - f[4])[:, :my] * idx - (bx[:, 1:] - bx[:, :-1]) * idy
                           - j[2][:, :my])
    _b_half(f, dt / 2, idx, idy, my, walls)
    g = _nodes(f, my, walls)
    if walls:
        wgt = torch.ones(my + 1, dtype=torch.float64, device=p.device)
        wgt[0] = wgt[my] = 0.5
    else:
        g, wgt = g[:, :, :my], torch.ones(my, dtype=torch.float64, device=p.device)
    fs = 0.5 * mime / (cva ** 2 * cfg["in0"])
    energies = torch.stack([ke[q < 0].sum(), ke[q > 0].sum(), fs / cva ** 2 * (g[:3] ** 2 * wgt).sum(),
                            fs * (g[3:] ** 2 * wgt).sum()])
    # the new cell: wrap, or reflect at a wall
    nx, ny = (ix + cx) % mx, iy + cy
    y2, u = y1 - cy, u.clone()
    if walls:
        out = (ny < 0) | (ny >= my)
        ny = ny.clamp(0, my - 1)
        y2 = torch.where(out, -y2, y2)
        u[:, 1] = torch.where(out, -u[:, 1], u[:, 1])
    else:
        ny = ny % my
    p = torch.cat([(x1 - cx)[:, None], y2[:, None], u], 1)
    return _ordered(p, nx * my + ny, q) + (f, j, energies)


def _ordered(p, cell, q):
    order = torch.sort(cell, stable=True).indices
    return p[order], cell[order], q[order]


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        keys = _keys(case, seed)
        return {"perm": torch.sort(keys, stable=True).indices.to(torch.int32),
                "counts": torch.bincount(keys, minlength=case["cells"]).to(torch.int32)}
    if kind not in ("step", "calls"):
        return None
    cfg, part, cell, q, f = _plasma(case, seed)
    p, cell, q = _ordered(part.double(), cell.long(), q)
    for _ in range(case["steps"]):
        p, cell, q, f, j, energies = _step(p, cell, q, f, cfg)
    rows = case["my"] + (1 if cfg["ybc"] == L.BC_CONDUCTING else 0)
    out = {"particles": p, "where": None, "fields": f[:, :, :rows], "energies": energies}
    if kind == "calls":
        out["denjr"] = j
    return out
