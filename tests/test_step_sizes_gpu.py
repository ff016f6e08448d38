"""Step kernels at the sizes where their lane maps can go wrong (remainders of
float4, warp and block tiles, the smallest grids), against the oracle in the
reference's float order: identical bits.  GPU only."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _pulse(nt, dt, f):
    t = np.arange(nt) * dt - 1.2 / f
    a = (np.pi * f * t) ** 2
    return (1 - 2 * a) * np.exp(-a)


# padded depths of 4k, 4k + 1 .. 4k + 3 cells; 31, 32, 33 and 65 float4 per column;
# widths around multiples of the 4 planes of a CTA
@pytest.mark.parametrize("nz,nx,nb", [(9, 9, 4), (12, 14, 5), (40, 37, 7), (107, 21, 8),
                                      (111, 30, 8), (110, 23, 9), (113, 19, 8), (241, 18, 9)])
# unit, tiny (numerators below the constant-divisor range, subnormal quotients) and large fields
@pytest.mark.parametrize("scale,h", [(1e6, 0.01), (1e-32, 0.01), (1e-36, 10.0), (1e24, 0.01)])
def test_pfwi_step_sizes_bit_exact(oracle, cuda_lib, nz, nx, nb, scale, h):
    import pywave_b200 as pw
    from pywave_b200 import fwi
    nt, ns, dt = 90, 2, 0.001
    rng = np.random.default_rng(nz * 1000 + nx)
    vel = (250.0 * h * (0.6 + 0.4 * rng.random((nz, nx)))).astype(np.float32)
    wav = (scale * _pulse(nt, dt, 40.0)).astype(np.float32)
    ds = (nx // 2) * h
    par = dict(nz=nz, nx=nx, dz=h, dx=h, oz=0.0, ox=0.0, nt=nt, dt=dt, ot=0.0, ns=ns, ds=ds,
               os=ds / 2, nb=nb, coef=0.01, f0=40.0, acqui_type=1, interval=1, niter=1)
    geo = oracle.pfwi_geometry(nz, nx, h, h, 0, 0, ns, ds, ds / 2, nb)
    kw = dict(nb=nb, coef=0.01, dz=h, dx=h, dt=dt, geo=geo, ns=ns)
    d = pw.pfwi(vel, np.full(vel.shape, 1e4, np.float32), wav, None, mode=1, par=par)[0]
    ref = oracle.pfwi_forward(vel, wav, **kw)
    assert np.abs(ref).max() > 0
    assert np.array_equal(d.view(np.uint32), ref.view(np.uint32))
    if scale != 1e6:
        return
    dobs = (0.5 * ref).astype(np.float32)
    w = np.ones((nx, nt), np.float32)
    g, _ = fwi.gradient(vel, wav, dobs, par, mode="reference", per_shot=True, weight=w)
    go, _ = oracle.pfwi_gradient_ref(vel, wav, dobs, weight=w, **kw)
    assert np.array_equal(g.view(np.uint32), go.view(np.uint32))
    # 2 x 90 steps of float32 (6e-8 each) against FP64, the residual half the data
    ge, J = fwi.gradient(vel, wav, dobs, par, mode="exact", weight=w)
    gx, Jx = oracle.pfwi_gradient_exact(vel, wav, dobs, weight=w.astype(np.float64), **kw)
    assert rel_l2(ge, gx) < 1e-4 and abs(J - Jx) < 1e-4 * Jx
