"""The pfwi steps' division by dx^2 and dz^2 outside the range of the
constant-divisor method: the FP64 form for tiny and huge numerators, and
squares of the spacing that leave float's range."""
import ctypes
import ctypes.util
import re

import numpy as np
import pytest

f32 = np.float32

# spacings of the tests and benchmarks, and squares near the ends of float's range
SPACINGS = [0.01, 10.0, 0.012, 0.008, 0.03, 0.005, 0.025, 25.0, 1.5e19, 2e-19, 2e-20]


# x / d through FP64 as the kernel has it (q = RN(x RN(1/d)), its exact remainder added once,
# rounded to float) against IEEE float32 division: numerators around subnormal and
# overflowing quotients and over all bit patterns, both signs
@pytest.mark.parametrize("h", SPACINGS)
def test_fp64_division_is_correctly_rounded(h):
    fma = ctypes.CDLL(ctypes.util.find_library("m")).fma
    fma.restype, fma.argtypes = ctypes.c_double, [ctypes.c_double] * 3
    d = f32(f32(h) * f32(h))
    assert 0 < d < np.inf
    rd = 1.0 / float(d)
    rng = np.random.default_rng(int(np.float64(d).view(np.uint64) % 1000))
    tiny = f32(min(float(np.finfo(f32).tiny) * 2 * float(d), float(np.finfo(f32).max)))
    bits = [np.arange(1, 3000), rng.integers(1, max(int(tiny.view(np.uint32)), 2), 12000),
            rng.integers(1, 0x7f800000, 12000)]
    # ties of the subnormal grid and their neighbours: x near (k + 1/2) 2^-149 d
    k = rng.integers(0, 1 << 23, 2000) + 0.5
    with np.errstate(all="ignore"):
        near = (k * 2.0 ** -149 * float(d)).astype(f32).view(np.uint32).astype(np.int64)
        bits += [near, near + 1, np.maximum(near - 1, 1)]
        x = np.concatenate(bits).astype(np.uint32).view(f32)
        x = x[(x > 0) & np.isfinite(x)]
        x = np.concatenate([x, -x])
        ref = x / d
        q = np.empty(x.size)
        for i, v in enumerate(x.tolist()):
            y = v * rd
            q[i] = fma(fma(-y, float(d), v), rd, y)
        got = q.astype(f32)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


# the library compares its FP64 form with the IEEE quotient for every divisor that it meets,
# once per process, and says so
@pytest.mark.gpu
@pytest.mark.parametrize("h", [0.0117, 13.7, 1.5e19, 2e-19, 2e-20])
def test_fp64_division_is_checked_on_the_gpu(cuda_lib, monkeypatch, capfd, h):
    import pywave_b200 as pw
    n, nt = 16, 3
    dt = 1e-3 * h if h < 1e18 else 1e-3
    v = np.full((n, n), 100.0 if h < 1e18 else 2.0, f32)
    par = dict(nz=n, nx=n, dz=h, dx=h, oz=0.0, ox=0.0, nt=nt, dt=dt, ot=0.0, ns=1, ds=h,
               os=4 * h, nb=6, coef=0.01, f0=10.0, acqui_type=1, interval=1, niter=1)
    monkeypatch.setenv("PW_PFWI_VERBOSE", "1")
    pw.pfwi(v, np.full(v.shape, 1e4, f32), np.ones(nt, f32), None, mode=1, par=par)
    err = capfd.readouterr().err
    d = f32(h) * f32(h)
    said = {f32(a): b for a, b in re.findall(r"pfwi: division by (\S+):.* FP64 (\d)", err)}
    assert said == {d: "1"}, err


# dx^2 or dz^2 is infinite (that axis then has no coupling: x / inf = 0), or both
# are zero (0 / 0 = NaN in every cell of the stencil)
@pytest.mark.gpu
@pytest.mark.parametrize("dz,dx", [(0.01, 1e20), (1e20, 0.01), (1e20, 1e20), (1e-24, 1e-24)])
def test_spacing_whose_square_leaves_the_float_range(oracle, cuda_lib, dz, dx):
    import pywave_b200 as pw
    from pywave_b200 import fwi
    nz, nx, nb, nt, ns = 24, 22, 6, 50, 2
    h = min(dz, dx)
    dt = 1e-3 if h >= 0.01 else 1e-25
    rng = np.random.default_rng(7)
    v0 = 0.25 * min(h, 0.01) / dt
    vel = (v0 * (0.6 + 0.4 * rng.random((nz, nx)))).astype(f32)
    wav = rng.standard_normal(nt).astype(f32)
    ds = (nx // 2) * dx
    par = dict(nz=nz, nx=nx, dz=dz, dx=dx, oz=0.0, ox=0.0, nt=nt, dt=dt, ot=0.0, ns=ns, ds=ds,
               os=ds / 2, nb=nb, coef=0.01, f0=40.0, acqui_type=1, interval=1, niter=1)
    geo = oracle.pfwi_geometry(nz, nx, dz, dx, 0, 0, ns, ds, ds / 2, nb)
    kw = dict(nb=nb, coef=0.01, dz=dz, dx=dx, dt=dt, geo=geo, ns=ns)
    d = pw.pfwi(vel, np.full(vel.shape, 1e4, f32), wav, None, mode=1, par=par)[0]
    ref = oracle.pfwi_forward(vel, wav, **kw)
    if dz == 0.01:  # the column of the source reaches its receiver
        assert np.abs(ref).max() > 0 and np.isfinite(ref).all()
    assert np.array_equal(np.isnan(d), np.isnan(ref))
    assert np.array_equal(d[~np.isnan(d)].view(np.uint32), ref[~np.isnan(d)].view(np.uint32))
    dobs = rng.standard_normal(ref.shape).astype(f32)
    w = np.ones((nx, nt), f32)
    g, _ = fwi.gradient(vel, wav, dobs, par, mode="reference", per_shot=True, weight=w)
    go, _ = oracle.pfwi_gradient_ref(vel, wav, dobs, weight=w, **kw)
    assert np.array_equal(np.isnan(g), np.isnan(go))
    assert np.array_equal(g[~np.isnan(g)].view(np.uint32), go[~np.isnan(g)].view(np.uint32))
