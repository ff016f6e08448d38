"""The pfwi steps' division by dx^2 and dz^2 outside the range of the
constant-divisor method: squares of the spacing that leave float's range."""
import numpy as np
import pytest

f32 = np.float32


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
