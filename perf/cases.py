"""Performance cases of the framework's own propagators: 2-D and 3-D acoustic
modelling, time-reversal imaging, pfwi modelling, FWI gradients and passive
source inversion, each through the entry point a user's program calls.

A case is a dict of plain values whose "kind" names the call:

  afd2d    pw.afd2d on host arrays: one shot, small to medium 2-D grids
  tri2d    pw.tri_image on host arrays: 2-D time-reversal image of receiver groups
  batch2d  pw.afd.afd2d_batch on host arrays: shots of uneven size and length
  afd3d    pw.afd3d on host arrays, or pw_afd on device arrays (C ABI)
  tri3d    pw_tri_image on device arrays (C ABI): the framework's headline path
  model    pw.pfwi(mode=1) on host arrays: 8th-order modelling of a shot set
  exact    fwi.fwi_misfit: FWI misfit and exact-adjoint gradient (torch autograd)
  refgrad  fwi.gradient(mode="reference") on host arrays: gradient_av's imaging
  exact3d  fwi3d.fwi3d_misfit: 3-D FWI misfit and gradient (torch autograd)
  lstri    lstri.lstri_invert_torch: conjugate-gradient source inversion

The host-array kinds take whole calls (copies in and out included) because
that is how the drop-in API is called; the device kinds keep velocity, data
and results on the GPU as an imaging or inversion program does.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import pywave_b200 as pw
from pywave_b200 import _lib as L
from pywave_b200 import fwi, fwi3d, lstri

DT, CT = 0.001, 0.01


def listed():
    return [
        # the reference's afd2d defaults (81 x 81 at 20 m, two sources, a snapshot every
        # 4 steps): the smallest call, bound by latency per step
        dict(name="afd2d_demo", kind="afd2d", nz=81, nx=81, dz=20.0, dx=20.0, nt=1501, ns=2, nbt=30, jsnap=4),
        # one shot of an ordinary odd-sized section, traces only (the grid no longer fits
        # one cluster's shared memory)
        dict(name="afd2d_section", kind="afd2d", nz=501, nx=1501, dz=10.0, dx=10.0, nt=1000, ns=1, nbt=30, jsnap=0),
        # 2-D time-reversal location of events, four receiver bands
        dict(name="tri2d_201", kind="tri2d", nz=201, nx=201, dz=10.0, dx=10.0, nt=1501, groups=4, nbt=30, jsnap=4),
        # a survey of shots of uneven size and length, modelled in lockstep
        dict(name="batch2d_12", kind="batch2d", shots=12, nz=800, nx=1700, dz=10.0, dx=10.0, nt=600, nbt=30),
        # the reference's afd3d default grid, traces only: fields stay in L2
        dict(name="afd3d_81", kind="afd3d", nz=81, nx=81, ny=81, dz=20.0, dx=20.0, dy=20.0, nt=501, ns=3, nbt=30, host=True),
        # 3-D modelling on the benchmark's grid, device arrays
        dict(name="afd3d_201", kind="afd3d", nz=201, nx=201, ny=201, dz=10.0, dx=10.0, dy=10.0, nt=400, ns=3, nbt=30, host=False),
        # the headline: 3-D time-reversal image of four receiver groups
        dict(name="tri3d_201", kind="tri3d", nz=201, nx=201, ny=201, dz=10.0, dx=10.0, dy=10.0, nt=420, groups=4, nbt=30, jsnap=4),
        # pfwi modelling of a small survey with the reference's wide sponge
        dict(name="model_8", kind="model", nz=151, nx=301, dz=0.01, dx=0.01, nt=1000, ns=8, nb=60),
        # one FWI iteration's gradient on the benchmark's section (exact adjoint)
        dict(name="exact_16", kind="exact", nz=300, nx=600, dz=0.01, dx=0.01, nt=400, ns=16, nb=60),
        # the gradient inside fwic on a small model: latency per step, forward and adjoint
        dict(name="refgrad_4", kind="refgrad", nz=60, nx=121, dz=0.01, dx=0.01, nt=800, ns=4, nb=40, interval=1),
        # 3-D FWI gradient, two shots
        dict(name="exact3d_2", kind="exact3d", nz=120, nx=200, ny=200, h=0.0125, nt=120, ns=2, nb=20),
        # source inversion on the passive demos' grid (two CG iterations)
        dict(name="lstri_130", kind="lstri", nz=130, nx=334, dz=0.008, dx=0.012, nt=900, ns=1, nb=60, niter=2),
    ]


def draw(rng):
    """One more case: sizes log-uniform over each kind's range, every parity, cut in
    length until it costs no more than the largest listed case."""
    def lg(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["afd2d", "tri2d", "batch2d", "afd3d", "tri3d", "model", "exact", "refgrad", "exact3d", "lstri"])
    h = rng.choice([10.0, 12.5, 20.0])
    km = rng.choice([0.01, 0.0125, 0.02])
    nbt = rng.choice([20, 30, 40])
    if kind == "afd2d":
        c = dict(nz=lg(41, 601), nx=lg(41, 1601), dz=h, dx=10.0, nt=lg(300, 1501), ns=rng.randint(1, 3), nbt=nbt, jsnap=rng.choice([0, 4, 10]))
        if c["jsnap"] and c["nz"] * c["nx"] * c["nt"] // c["jsnap"] > 8e6:
            c["jsnap"] = 0
    elif kind == "tri2d":
        c = dict(nz=lg(61, 301), nx=lg(81, 401), dz=10.0, dx=10.0, nt=lg(300, 1501), groups=rng.randint(2, 5), nbt=nbt, jsnap=rng.randint(2, 8))
        c["nt"] = max(c["nt"], 2 * c["nx"])  # long enough for the groups' fields to meet
    elif kind == "batch2d":
        c = dict(shots=rng.randint(3, 16), nz=lg(200, 900), nx=lg(300, 1900), dz=h, dx=10.0, nt=lg(250, 700), nbt=nbt)
    elif kind == "afd3d":
        c = dict(nz=lg(41, 221), nx=lg(41, 221), ny=lg(41, 221), dz=10.0, dx=h, dy=10.0, nt=lg(80, 400), ns=rng.randint(1, 3), nbt=nbt, host=rng.random() < 0.5)
    elif kind == "tri3d":
        c = dict(nz=lg(61, 201), nx=lg(61, 201), ny=lg(61, 201), dz=10.0, dx=10.0, dy=10.0, nt=lg(150, 420), groups=rng.randint(2, 4), nbt=nbt, jsnap=rng.randint(2, 8))
        c["nt"] = max(c["nt"], 2 * c["nx"])
    elif kind == "model":
        c = dict(nz=lg(50, 300), nx=lg(61, 600), dz=0.01, dx=km, nt=lg(300, 1200), ns=rng.randint(1, 12), nb=rng.choice([40, 60, 100]))
    elif kind == "exact":
        c = dict(nz=lg(60, 300), nx=lg(100, 600), dz=0.01, dx=km, nt=lg(200, 500), ns=rng.randint(1, 20), nb=rng.choice([40, 60]))
    elif kind == "refgrad":
        c = dict(nz=lg(50, 150), nx=lg(81, 300), dz=0.01, dx=km, nt=lg(300, 1000), ns=rng.randint(1, 6), nb=rng.choice([40, 60]), interval=rng.choice([1, 2, 5]))
    elif kind == "exact3d":
        c = dict(nz=lg(40, 160), nx=lg(50, 220), ny=lg(50, 220), h=0.0125, nt=lg(40, 130), ns=rng.randint(1, 3), nb=rng.choice([15, 20, 25]))
    else:
        c = dict(nz=lg(60, 150), nx=lg(100, 400), dz=0.008, dx=0.012, nt=lg(300, 900), ns=rng.randint(1, 2), nb=rng.choice([40, 60]), niter=rng.randint(1, 2))
    c["kind"] = kind
    most = max(work(k)["flops"] for k in listed())
    while work(c)["flops"] > most:
        c["nt"] = int(0.9 * c["nt"])
    return c


# ------------------------------------------------------------------- inputs --

def _rand(seed, *tag):
    return torch.Generator().manual_seed((seed * 1000003 + sum((i + 1) * int(t) for i, t in enumerate(tag))) % (1 << 62))


def _vel(shape, seed, unit=1.0):
    """Velocity 1500 -> 3500 (times unit) along z with a smooth 5% perturbation, axes
    (z, x[, y]), float32 on the GPU."""
    g = _rand(seed, *shape)
    coarse = torch.rand((1, 1) + tuple(max(2, n // 16) for n in shape), generator=g).cuda() - 0.5
    p = F.interpolate(coarse, size=shape, mode="bilinear" if len(shape) == 2 else "trilinear", align_corners=True)[0, 0]
    z = torch.linspace(0, 1, shape[0], device="cuda").reshape((-1,) + (1,) * (len(shape) - 1))
    return ((1500.0 + 2000.0 * z) * (1.0 + 0.1 * p) * unit).float()


def _pulse(t, f):
    a = (math.pi * f * t) ** 2
    return (1 - 2 * a) * torch.exp(-a)


def _arrivals(shape, h, nt, seed, speed, count=3, f=15.0):
    """Traces [shape.., nt] (float32, GPU) of `count` buried events: Ricker pulses along
    hyperbolic moveouts with 1/r amplitudes."""
    g = _rand(seed, nt, *shape)
    axes = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float32) * d for n, d in zip(shape, h)], indexing="ij")
    t = torch.arange(nt, device="cuda", dtype=torch.float32) * DT
    out = torch.zeros(tuple(shape) + (nt,), device="cuda")
    for _ in range(count):
        u = torch.rand(len(shape) + 2, generator=g).tolist()
        depth = (0.2 + 0.3 * u[0]) * max(n * d for n, d in zip(shape, h))
        r2 = depth ** 2 + sum((a - v * n * d) ** 2 for a, v, n, d in zip(axes, u[2:], shape, h))
        r = torch.sqrt(r2)
        t0 = (0.15 + 0.35 * u[1]) * nt * DT
        out += (depth / r)[..., None] * _pulse(t - t0 - ((r - depth) / speed)[..., None], f)
    return out


def _points(c, seed):
    """Seeded source rows [sx, (sy,) sz], f, t, A of an afd case as lists; shallow enough
    for the waves to reach the receivers well inside the record."""
    g = _rand(seed, c["nt"])
    dims = [c["nx"]] + ([c["ny"]] if "ny" in c else [])
    rows = [[int((0.2 + 0.6 * u) * n) for u in torch.rand(c["ns"], generator=g).tolist()] for n in dims]
    rows.append([int((0.03 + 0.12 * u) * min(c["nz"], 0.4 * c["nt"])) for u in torch.rand(c["ns"], generator=g).tolist()])
    f = [10.0 + 10.0 * u for u in torch.rand(c["ns"], generator=g).tolist()]
    t = [min(0.3, 0.4 * c["nt"] * DT) * (0.3 + 0.7 * u) for u in torch.rand(c["ns"], generator=g).tolist()]
    return rows, f, t, [1.0 + i for i in range(c["ns"])]


def _par(c):
    k = max(1, c["nx"] // c["ns"])
    return dict(nz=c["nz"], nx=c["nx"], dz=c["dz"], dx=c["dx"], oz=0.0, ox=0.0, nt=c["nt"], dt=DT, ot=0.0, ns=c["ns"],
                ds=k * c["dx"], os=(k // 2) * c["dx"], nb=c["nb"], coef=0.005, f0=10.0, acqui_type=1,
                interval=c.get("interval", 1), niter=c.get("niter", 1))


def _wavelet(nt, f=10.0):
    # 1e6: the demos' source scale, which puts pfwi's km-unit fields at order one
    return (1e6 * _pulse(torch.arange(nt, dtype=torch.float64) * DT - min(1.2 / f, 0.3 * nt * DT), f)).float()


def _sections(c):
    """batch2d's shots: sizes between 0.45 and 1 times the largest, uneven lengths."""
    for i in range(c["shots"]):
        u = (0.37 + 0.618034 * i) % 1.0
        v = (0.11 + 0.754878 * i) % 1.0
        yield dict(nz=int(c["nz"] * (0.45 + 0.55 * u)), nx=int(c["nx"] * (0.45 + 0.55 * v)),
                   nt=int(c["nt"] * (0.6 + 0.4 * ((u + v) % 1.0))), dz=c["dz"], dx=c["dx"], nbt=c["nbt"], ns=1)


def _geom(c):
    side = 40
    rx = sorted({int((i + 0.5) * c["nx"] / side) for i in range(side)})
    ry = sorted({int((j + 0.5) * c["ny"] / side) for j in range(side)})
    src = [(5, int((i + 0.5) * c["nx"] / c["ns"]), int((0.3 + 0.4 * (i % 2)) * c["ny"])) for i in range(c["ns"])]
    return dict(nb=c["nb"], coef=0.015, dz=c["h"], dx=c["h"], dy=c["h"], nt=c["nt"], dt=DT, src=src, rz=1, rx=rx, ry=ry)


def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    c, kind = dict(case), case["kind"]
    s = dict(kind=kind, case=c)
    if kind == "afd2d":
        (sx, sz), f, t, a = _points(c, seed)
        s["vel"] = _host(_vel((c["nz"], c["nx"]), seed))
        s["kw"] = dict(nt=c["nt"], dt=DT, ax=[0, c["dx"], c["nx"]], az=[0, c["dz"], c["nz"]], ns=c["ns"], sx=sx, sz=sz, f=f,
                       t=t, A=a, nbt=c["nbt"], ct=CT, jsnap=c["jsnap"])
    elif kind == "tri2d":
        s["vel"] = _host(_vel((c["nz"], c["nx"]), seed))
        d = _arrivals((c["nx"],), (c["dx"],), c["nt"], seed, 2500.0)
        s["dat"] = _host(d).T  # (nt, nx), time fastest, as afd2d returns traces
        s["kw"] = dict(dt=DT, d=(c["dz"], c["dx"]), ngroups=c["groups"], nbt=c["nbt"], ct=CT, jsnap=c["jsnap"])
    elif kind == "batch2d":
        s["shots"] = []
        for i, b in enumerate(_sections(c)):
            (sx, _), f, t, a = _points(b, seed + i)
            s["shots"].append(dict(vel=_host(_vel((b["nz"], b["nx"]), seed + i)), nt=b["nt"], dt=DT, ax=[0, b["dx"], b["nx"]],
                                   az=[0, b["dz"], b["nz"]], ns=1, sx=sx, sz=[5], f=f, t=t, A=a, nbt=b["nbt"], ct=CT, gz=5))
    elif kind == "afd3d":
        (sx, sy, sz), f, t, a = _points(c, seed)
        v = _vel((c["nz"], c["nx"], c["ny"]), seed)
        if c["host"]:
            s["vel"] = np.asfortranarray(_host(v))
            s["kw"] = dict(nt=c["nt"], dt=DT, ax=[0, c["dx"], c["nx"]], ay=[0, c["dy"], c["ny"]], az=[0, c["dz"], c["nz"]],
                           ns=c["ns"], sx=sx, sy=sy, sz=sz, f=f, t=t, A=a, nbt=c["nbt"], ct=CT, jsnap=0)
        else:
            s["vel"] = v.permute(2, 1, 0).contiguous()  # [ny][nx][nz]
            s["src"] = torch.tensor(sx + sy + sz + f + t + a, dtype=torch.float32, device="cuda")
            s["dat"] = torch.empty(c["ny"], c["nx"], c["nt"], device="cuda")
            s["args"] = _afd_args(c, 0)
    elif kind == "tri3d":
        s["vel"] = _vel((c["nz"], c["nx"], c["ny"]), seed).permute(2, 1, 0).contiguous()
        s["dat"] = _arrivals((c["ny"], c["nx"]), (c["dy"], c["dx"]), c["nt"], seed, 2500.0)
        s["img"] = torch.empty_like(s["vel"])
        s["args"] = _afd_args(c, 1)
    elif kind in ("model", "exact", "refgrad"):
        v = _vel((c["nz"], c["nx"]), seed, 0.001)
        w = _wavelet(c["nt"])
        s["par"] = _par(c)
        if kind != "model":
            d = torch.stack([2.0 * _arrivals((c["nx"],), (c["dx"],), c["nt"], seed + i, 2.5) for i in range(c["ns"])])
        if kind == "exact":
            s["vel"], s["wav"], s["dobs"] = v.requires_grad_(True), w.cuda(), d  # d [ns][nr][nt]
        else:
            s["vel"], s["wav"] = _host(v), w.numpy()
            s["q"] = np.full_like(s["vel"], 100.0)
            if kind == "refgrad":
                s["dobs"] = np.asfortranarray(_host(d).transpose(2, 1, 0))  # (nt, nr, ns)
    elif kind == "exact3d":
        s["geom"] = _geom(c)
        s["vel"] = _vel((c["nz"], c["nx"], c["ny"]), seed, 0.001).requires_grad_(True)
        s["wav"] = _wavelet(c["nt"], 12.0).cuda()
        rx, ry = len(s["geom"]["rx"]), len(s["geom"]["ry"])
        d = [_arrivals((ry, rx), (c["h"] * c["ny"] / ry, c["h"] * c["nx"] / rx), c["nt"], seed + i, 2.5) for i in range(c["ns"])]
        s["dobs"] = 0.1 * torch.stack(d).reshape(c["ns"], rx * ry, c["nt"])
    else:
        s["par"] = _par(c)
        s["vel"] = _vel((c["nz"], c["nx"]), seed, 0.001).t().contiguous()  # [nx][nz]
        s["data"] = torch.stack([1e3 * _arrivals((c["nx"],), (c["dx"],), c["nt"], seed + i, 2.5) for i in range(c["ns"])])
        s["src"] = torch.empty(c["ns"], c["nt"], c["nx"], c["nz"], device="cuda")
    return s


def _afd_args(c, tri):
    return L.AfdArgs(dim=3, nz=c["nz"], nx=c["nx"], ny=c["ny"], nt=c["nt"], nbt=c["nbt"], ct=CT, dt=DT, dz=c["dz"], dx=c["dx"],
                     dy=c["dy"], ns=0 if tri else c["ns"], tri=tri, jsnap=c.get("jsnap", 0), gz=0, flags=0)


def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "afd2d":
        return pw.afd2d(s["vel"], **s["kw"])
    if kind == "tri2d":
        return pw.tri_image(s["vel"], s["dat"], **s["kw"])
    if kind == "batch2d":
        return pw.afd.afd2d_batch(s["shots"], stream=torch.cuda.current_stream().cuda_stream)
    if kind == "afd3d":
        if c["host"]:
            return pw.afd3d(s["vel"], **s["kw"])
        L.check(L.lib().pw_afd(s["args"], s["vel"].data_ptr(), s["src"].data_ptr(), None, s["dat"].data_ptr(), None,
                               torch.cuda.current_stream().cuda_stream))
        return s["dat"]
    if kind == "tri3d":
        L.check(L.lib().pw_tri_image(s["args"], c["groups"], None, s["vel"].data_ptr(), s["dat"].data_ptr(),
                                     s["img"].data_ptr(), 1, torch.cuda.current_stream().cuda_stream))
        return s["img"]
    if kind == "model":
        return pw.pfwi(s["vel"], s["q"], s["wav"], None, mode=1, par=s["par"])[0]
    if kind == "exact":
        j = fwi.fwi_misfit(s["vel"], s["wav"], s["dobs"], s["par"])
        return j.detach(), torch.autograd.grad(j, s["vel"])[0]
    if kind == "refgrad":
        g, j = fwi.gradient(s["vel"], s["wav"], s["dobs"], s["par"], mode="reference")
        return j, g
    if kind == "exact3d":
        j = fwi3d.fwi3d_misfit(s["vel"], s["wav"], s["dobs"], s["geom"])
        return j.detach(), torch.autograd.grad(j, s["vel"])[0]
    lstri.lstri_invert_torch(s["vel"], s["data"], s["src"], s["par"])
    return s["src"]


def work(case):
    """Bytes: inputs and outputs once.  Flops: the scheme's operations per padded cell and
    step (stencil sums, update, taper; image products, gradient sums)."""
    c, kind = case, case["kind"]
    vel = c.get("nz", 1) * c.get("nx", 1) * c.get("ny", 1) * 4
    if kind in ("afd2d", "tri2d", "batch2d", "afd3d", "tri3d"):
        fl = by = 0
        for b in _sections(c) if kind == "batch2d" else [c]:
            n = 2 * b["nbt"]
            cells = (b["nz"] + n) * (b["nx"] + n) * ((b["ny"] + n) if "ny" in b else 1)
            axes = 3 if "ny" in b else 2
            fl += b.get("groups", 1) * cells * b["nt"] * (8 * axes + 3 + 4 + 2 * axes)
            v = b["nz"] * b["nx"] * b.get("ny", 1) * 4
            by += v + b["nx"] * b.get("ny", 1) * b["nt"] * 4
            if kind in ("tri2d", "tri3d"):
                by += v
                fl += 2 * (b["groups"] + 1) * (v // 4) * (b["nt"] // b["jsnap"])
            elif b.get("jsnap"):
                by += v * ((b["nt"] - 1) // b["jsnap"] + 1)
        return {"bytes": by, "flops": fl}
    n = 2 * c["nb"]
    cells = (c["nz"] + n) * (c["nx"] + n) * ((c["ny"] + n) if "ny" in c else 1)
    axes = 3 if "ny" in c else 2
    step = axes * 14 + 5 + 2 * axes + 4
    if kind == "lstri":
        apps = 2 * c["niter"] * c["ns"]
        return {"bytes": vel + c["ns"] * c["nt"] * (vel + 4 * c["nx"]), "flops": apps * c["nt"] * cells * step}
    nr = len(_geom(c)["rx"]) * len(_geom(c)["ry"]) if kind == "exact3d" else c["nx"]
    traces = c["ns"] * nr * c["nt"] * 4
    if kind == "model":
        return {"bytes": vel + traces, "flops": c["ns"] * c["nt"] * cells * step}
    return {"bytes": 2 * vel + traces, "flops": c["ns"] * c["nt"] * cells * (2 * step + 2)}


# ------------------------------------------------ the schemes in 64 bits --

C4 = [-30.0 / 12, 16.0 / 12, -1.0 / 12]
C8 = [-205.0 / 72, 8.0 / 5, -1.0 / 5, 8.0 / 315, -1.0 / 560]


def _fast(n):
    """Smallest size >= n with no prime factor above 5."""
    while True:
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _f64(x):
    return torch.as_tensor(np.asarray(x) if not isinstance(x, torch.Tensor) else x.detach()).to("cuda", torch.float64)


def _outer(tables):
    out = tables[0]
    for t in tables[1:]:
        out = out[..., None] * t
    return out


def _pad(v, nb):
    """Edge replication by nb cells on every axis with nb > 0."""
    for ax, b in enumerate(nb):
        i = torch.arange(-b, v.shape[ax] + b, device=v.device).clamp(0, v.shape[ax] - 1)
        v = v.index_select(ax, i)
    return v


class _Wave:
    """Leapfrog a' = S(2 a - S b + V term), term = mask Lap(a) + injection, of `batch`
    fields on one grid; axes slowest first, z last."""

    def __init__(self, batch, V, S, mask, coef, inv_h2):
        self.h, self.coef, self.inv = len(coef) - 1, coef, inv_h2
        self.V, self.S, self.mask = V, S, mask
        shape = (batch,) + tuple(V.shape)
        full = (batch,) + tuple(n + 2 * self.h for n in V.shape)
        self.a = torch.zeros(full, dtype=torch.float64, device="cuda")
        self.b = torch.zeros_like(self.a)
        self.term = torch.empty(shape, dtype=torch.float64, device="cuda")
        self.tmp = torch.empty_like(self.term)

    def core(self, f, ax=None, d=0):
        h = self.h
        return f[(slice(None),) + tuple(slice(h + (d if i == ax else 0), f.shape[i + 1] - h + (d if i == ax else 0))
                                        for i in range(len(self.inv)))]

    def step(self, inject=None, weight=None):
        src = self.a
        if weight is not None:  # Laplacian of weight * a, not multiplied by V
            src = torch.zeros_like(self.a)
            self.core(src).copy_(self.core(self.a) * weight)
        torch.mul(self.core(src), self.coef[0] * sum(self.inv), out=self.term)
        for ax, w in enumerate(self.inv):
            for d in range(1, self.h + 1):
                torch.add(self.core(src, ax, d), self.core(src, ax, -d), out=self.tmp)
                self.term.add_(self.tmp, alpha=self.coef[d] * w)
        self.term.mul_(self.mask)
        if inject is not None:
            inject(self.term)
        b, a = self.core(self.b), self.core(self.a)
        b.mul_(self.S).neg_().add_(a, alpha=2.0)
        if weight is None:
            b.addcmul_(self.term, self.V)
        else:
            b.add_(self.term)
        b.mul_(self.S)
        self.a, self.b = self.b, self.a


def _span(n, lo, hi):
    m = torch.zeros(n, dtype=torch.float64, device="cuda")
    m[lo:hi] = 1.0
    return m


def _afd_wave(c, vel, batch):
    """vel in model axes (z, x[, y]); fields in axes ([y,] x, z)."""
    nb = c["nbt"]
    v = _f64(vel)
    v = v.permute(*reversed(range(v.dim()))).contiguous()
    V = _pad(v, [nb] * v.dim()) ** 2 * DT * DT
    w = torch.exp(-(CT * (nb - 1 - torch.arange(nb, dtype=torch.float64, device="cuda"))) ** 2)
    tables, masks = [], []
    for i, n in enumerate(V.shape):
        n2 = 2 * _fast((n + 1) // 2) if i == V.dim() - 1 else _fast(n)
        f = torch.ones(max(n, n2), dtype=torch.float64, device="cuda")
        f[:nb] = w
        f[n2 - nb:n2] = w.flip(0)
        tables.append(f[:n])
        masks.append(_span(n, 2, min(n, n2 - 2)))
    spacing = ([c["dy"]] if "ny" in c else []) + [c["dx"], c["dz"]]
    return _Wave(batch, V, _outer(tables), _outer(masks), C4, [1.0 / d ** 2 for d in spacing])


def _ricker(nt, f, t0, amp):
    n = 2 * _fast((nt + 1) // 2)
    x = np.zeros(n)
    x[int(np.float32(t0) / np.float32(DT))] = amp
    w = (np.arange(n // 2 + 1) / (n * f * DT)) ** 2
    return np.fft.irfft(np.fft.rfft(x) * w * np.exp(1 - w), n)[:nt]


def _afd_forward(c, vel, pts, f, t, a, gz=0, jsnap=0):
    """Traces [(y,) x, nt] and snapshots (n, [y,] x, z) of one shot."""
    wv, nb = _afd_wave(c, vel, 1), c["nbt"]
    nd = wv.V.dim()
    q = torch.stack([_f64(_ricker(c["nt"], *r)) for r in zip(f, t, a)])
    spread = torch.tensor([abs(i) for i in (-1, 0, 1)], device="cuda", dtype=torch.float64)
    den = spread
    for _ in range(nd - 1):
        den = den[..., None] + spread
    den = 1.0 / (den + 1.0)
    cells = [tuple(slice(p + nb - 1, p + nb + 2) for p in reversed(pt)) for pt in pts]  # pt = (z, x[, y])
    inner = tuple(slice(nb, n - nb) for n in wv.V.shape)
    rec = torch.empty((c["nt"],) + tuple(n - 2 * nb for n in wv.V.shape[:-1]), dtype=torch.float64, device="cuda")
    snaps = []
    for it in range(c["nt"]):
        def inject(term):
            for i, cell in enumerate(cells):
                term[0][cell] += den * q[i, it]
        wv.step(inject)
        now = wv.core(wv.a)[0][inner]
        rec[it] = now[..., gz]
        if jsnap and it % jsnap == 0:
            snaps.append(now.clone())
    return rec.movedim(0, -1), torch.stack(snaps) if snaps else None


def _tri(c, vel, dat):
    """Normalised image in axes ([y,] x, z); dat [(y,) x, nt]."""
    nb, G = c["nbt"], c["groups"]
    wv = _afd_wave(c, vel, G)
    d = _f64(dat)
    band = torch.arange(c["nx"], device="cuda") // (c["nx"] // G)
    sel = torch.stack([(band == g).double() for g in range(G)])  # [G, x]
    sel = sel[:, None, :] if "ny" in c else sel
    rows = (slice(None),) + tuple(slice(nb, n - nb) for n in wv.V.shape[:-1]) + (nb,)
    inner = (slice(None),) + tuple(slice(nb, n - nb) for n in wv.V.shape)
    img = 0.0
    for it in range(c["nt"] - 1, -1, -1):
        wv.step(lambda term: term[rows].add_(sel * d[..., it]))
        if it % c["jsnap"] == 0:
            img = img + wv.core(wv.a)[inner].square().prod(0)
    return img / img.max()


def _sponge(n, nb, coef):
    i = torch.arange(nb, dtype=torch.float64, device="cuda")
    f = torch.ones(n, dtype=torch.float64, device="cuda")
    f[:nb] = torch.exp(-(coef * (nb - i)) ** 2)
    f[n - nb:] = f[:nb].flip(0)
    return f


def _pf_wave(v, nb, coef, spacing, batch):
    """pfwi's scheme; v in axes ([y,] x, z)."""
    V = _pad(v, [nb] * v.dim()) ** 2 * DT * DT
    S = _outer([_sponge(n, nb, coef) for n in V.shape])
    M = _outer([_span(n, 4, n - 4) for n in V.shape])
    return _Wave(batch, V, S, M, C8, [1.0 / d ** 2 for d in spacing])


def _hat(pts, nb):
    """Per shot the cells of its smoothed point source, pts in axes ([y,] x, z)."""
    return [(i,) + tuple(slice(p + nb - 1, p + nb + 2) for p in pt) for i, pt in enumerate(pts)]


def _weights(nr, nt):
    w = torch.ones(nr, nt, dtype=torch.float64, device="cuda")
    s = torch.sin(0.5 * math.pi * torch.arange(1, 11, dtype=torch.float64, device="cuda") / 11)
    w[:10] *= s[:, None]
    w[-10:] *= s.flip(0)[:, None]
    w[:, :10] *= s
    w[:, -10:] *= s.flip(0)
    return w


def _pf_forward(wv, pts, wav, nb, rec_at, keep=None):
    """Traces [shot, receivers.., nt] recorded before each step; keep(it, wave) sees each
    step's field, and the list it may return collects the terms."""
    k = torch.tensor([0.25, 0.5, 0.25], dtype=torch.float64, device="cuda")
    hat = _outer([k] * wv.V.dim())
    cells = _hat(pts, nb)
    rec = []
    for it in range(len(wav)):
        rec.append(wv.core(wv.a)[rec_at].clone())

        def inject(term):
            for cell in cells:
                term[cell] += hat * wav[it]
        before = wv.core(wv.a)
        if keep is not None:
            keep(it, before, None)
        wv.step(inject)
        if keep is not None:
            keep(it, None, wv.term)
    return torch.stack(rec, -1)


def _fold(g, v, nb):
    """Adjoint of the edge replication, times 2 / v."""
    for ax in range(g.dim()):
        n = g.shape[ax] - 2 * nb
        i = torch.arange(-nb, n + nb, device="cuda").clamp(0, n - 1)
        shape = list(g.shape)
        shape[ax] = n
        g = torch.zeros(shape, dtype=torch.float64, device="cuda").index_add_(ax, i, g)
    return 2.0 * g / v


def _exact_gradient(v, nb, coef, spacing, pts, wav, dobs, weight, rec_at):
    """Misfit and exact-adjoint gradient; v in axes ([y,] x, z), dobs [shot, receivers.., nt]."""
    nt = len(wav)
    J, total = 0.0, 0.0
    for i in range(len(pts)):
        wv = _pf_wave(v, nb, coef, spacing, 1)
        terms = []
        d = _pf_forward(wv, [pts[i]], wav, nb, rec_at, lambda it, a, t: terms.append(t.clone()) if t is not None else None)
        r = d - dobs[i:i + 1]
        J = J + 0.5 * float((weight * r * r).sum())
        r = weight * r
        back = _pf_wave(v, nb, coef, spacing, 1)
        g = torch.zeros_like(terms[0])
        for it in range(nt - 1, -1, -1):
            g.addcmul_(back.core(back.a), terms[it])

            def inject(term):
                term[rec_at] = term[rec_at] + r[..., it]
            back.step(inject)
            terms[it] = None
        total = total + g[0]
    return J, _fold(total, v, nb)


def _reference_gradient(c, v, pts, wav, dobs):
    nb, nt, step = c["nb"], c["nt"], c["interval"]
    nx, nz = v.shape
    at = (slice(None), slice(nb, nb + nx), 1 + nb)
    inner = (slice(None), slice(nb, nb + nx), slice(nb, nb + nz))
    snaps = []
    wv = _pf_wave(v, nb, 0.005, [c["dx"], c["dz"]], len(pts))
    d = _pf_forward(wv, pts, wav, nb, at, lambda it, a, t: snaps.append(a[inner].clone()) if a is not None and it % step == 0 else None)
    r = dobs - d
    J = 0.5 * float((r * r).sum())
    r = r * _weights(nx, nt)
    back = _pf_wave(v, nb, 0.005, [c["dx"], c["dz"]], len(pts))
    g = torch.zeros_like(v)
    for it in range(nt - 1, -1, -1):
        w = it // step
        if it % step == 0 and 0 < w < len(snaps) - 1:
            utt = (snaps[w + 1] - 2 * snaps[w] + snaps[w - 1]) / (DT * step) ** 2
            g += (utt * back.core(back.a)[inner]).sum(0) * (-2.0 / v ** 3)
        back.step(lambda term: term[at].add_(r[..., it]))
    return J, g


class _TimeReversal:
    """lstric's modelling operator and its adjoint for one velocity."""

    def __init__(self, c, v):
        self.c, nb = c, c["nb"]
        self.V = _pad(v, [nb, nb]) ** 2 * DT * DT
        i = torch.arange(nb, dtype=torch.float64, device="cuda")
        f = []
        for n in self.V.shape:
            t = torch.ones(n, dtype=torch.float64, device="cuda")
            t[:nb] = torch.exp(-(0.005 * (nb - 1 - i)) ** 2)
            t[n - nb:] = t[:nb].flip(0)
            f.append(t)
        self.S = _outer(f)
        self.M = _outer([_span(n, 4, n - 4) for n in self.V.shape])
        self.inner = (0, slice(nb, nb + c["nx"]), slice(nb, nb + c["nz"]))
        self.row = (0, slice(nb, nb + c["nx"]), 1 + nb)

    def wave(self):
        return _Wave(1, self.V, self.S, self.M, C8, [1.0 / self.c["dx"] ** 2, 1.0 / self.c["dz"] ** 2])

    def forward(self, mod):
        wv, dat = self.wave(), []
        for it in range(self.c["nt"]):
            dat.append(wv.core(wv.a)[self.row].clone())
            wv.step(lambda term: term[self.inner].add_(mod[it]))
        return torch.stack(dat, -1)

    def adjoint(self, dat):
        wv, mod = self.wave(), torch.empty(self.c["nt"], self.c["nx"], self.c["nz"], dtype=torch.float64, device="cuda")
        for it in range(self.c["nt"] - 1, -1, -1):
            mod[it] = (wv.core(wv.a)[0] * self.V)[self.inner[1:]]
            wv.step(lambda term: term[self.row].add_(dat[:, it]), weight=self.V)
        return mod


def _lstri(c, v, data):
    op, out = _TimeReversal(c, v), []
    S = Ss = None
    for d in data:
        x, rr = 0.0, -d
        for _ in range(c["niter"]):
            g = op.adjoint(rr)
            gg = op.forward(g)
            gdg, gdr = float((gg * gg).sum()), -float((gg * rr).sum())
            if S is None:
                alfa, beta = gdr / gdg, 0.0
                S, Ss = torch.zeros_like(g), torch.zeros_like(gg)
            else:
                sds, gds, sdr = float((Ss * Ss).sum()), float((gg * Ss).sum()), -float((Ss * rr).sum())
                det = max(1.0 - (gds / gdg) * (gds / sds), 1e-12) * gdg * sds
                alfa, beta = (sds * gdr - gds * sdr) / det, (-gds * gdr + gdg * sdr) / det
            S, Ss = beta * S + alfa * g, beta * Ss + alfa * gg
            x, rr = x + S, rr + Ss
        out.append(x)
    return torch.stack(out)


def exact(case, seed):
    c, kind = case, case["kind"]
    s = prepare(case, seed)
    if kind == "afd2d":
        k = s["kw"]
        rec, snaps = _afd_forward(c, s["vel"], list(zip(k["sz"], k["sx"])), k["f"], k["t"], k["A"], jsnap=c["jsnap"])
        return (rec.t(), snaps.permute(2, 1, 0)) if c["jsnap"] else rec.reshape(-1)  # as afd2d: flat without snapshots
    if kind == "tri2d":
        return _tri(c, s["vel"], s["dat"].T).t()
    if kind == "batch2d":
        return [_afd_forward(b, q["vel"], list(zip(q["sz"], q["sx"])), q["f"], q["t"], q["A"], gz=5)[0].t()
                for b, q in zip(_sections(c), s["shots"])]
    if kind == "afd3d":
        (sx, sy, sz), f, t, a = _points(c, seed)
        v = _vel((c["nz"], c["nx"], c["ny"]), seed)
        rec = _afd_forward(c, v, list(zip(sz, sx, sy)), f, t, a)[0]  # [y, x, nt]
        return rec.reshape(-1) if c["host"] else rec
    if kind == "tri3d":
        return _tri(c, s["vel"].permute(2, 1, 0), s["dat"])
    if kind == "exact3d":
        geo, nb = s["geom"], c["nb"]
        v = _f64(s["vel"]).permute(2, 1, 0).contiguous()
        iy, ix = torch.tensor(geo["ry"], device="cuda") + nb, torch.tensor(geo["rx"], device="cuda") + nb
        at = (slice(None), iy[:, None], ix[None, :], geo["rz"] + nb)
        d = _f64(s["dobs"]).reshape(c["ns"], len(geo["ry"]), len(geo["rx"]), c["nt"])
        j, g = _exact_gradient(v, nb, geo["coef"], [c["h"]] * 3, [(y, x, z) for z, x, y in geo["src"]], _f64(s["wav"]).tolist(),
                               d, 1.0, at)
        return j, g.permute(2, 1, 0)
    if kind == "lstri":
        return _lstri(c, _f64(s["vel"]), _f64(s["data"]))
    v = _f64(s["vel"]).t().contiguous()
    k = max(1, c["nx"] // c["ns"])
    pts = [(k // 2 + i * k, 5) for i in range(c["ns"])]
    wav, nb = _f64(s["wav"]).tolist(), c["nb"]
    at = (slice(None), slice(nb, nb + c["nx"]), 1 + nb)
    if kind == "model":
        d = _pf_forward(_pf_wave(v, nb, 0.005, [c["dx"], c["dz"]], c["ns"]), pts, wav, nb, at)
        return d.permute(2, 1, 0)  # (nt, nr, ns)
    if kind == "exact":
        j, g = _exact_gradient(v, nb, 0.005, [c["dx"], c["dz"]], pts, wav, _f64(s["dobs"]), _weights(c["nx"], c["nt"]), at)
    else:
        j, g = _reference_gradient(c, v, pts, wav, _f64(s["dobs"]).permute(2, 1, 0))
    return j, g.t()
