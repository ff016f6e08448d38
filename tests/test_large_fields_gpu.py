"""Step kernels where their block maps change with the size: fields beyond half
of L2 (60 MB), whose odd steps run the blocks backwards, and planes beyond the
65535 rows of one launch dimension.  Against the oracle.  GPU only."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _pulse(nt, dt, f):
    t = np.arange(nt) * dt - 1.2 / f
    a = (np.pi * f * t) ** 2
    return (1 - 2 * a) * np.exp(-a)


# 2-D 5.3 M cells, 3-D 5 M cells, and 65 602 planes (3-D, small ones)
@pytest.mark.parametrize("shape,nbt", [((2300, 2300), 6), ((150, 170, 160), 6), ((3, 2, 65600), 1)])
def test_afd_large_grids_bit_exact(oracle, cuda_lib, shape, nbt):
    import pywave_b200 as pw
    nt, dim = 7, len(shape)
    rng = np.random.default_rng(shape[1])
    vel = (1500 + 1500 * rng.random(shape)).astype(np.float32)
    kw = dict(nt=nt, dt=0.001, ax=[0, 10, shape[1]], az=[0, 10, shape[0]], nbt=nbt, ct=0.02, jsnap=3)
    # sources at both ends of the slowest axis
    src = dict(sx=[1, shape[1] - 1], sz=[0, 1], f=[30.0, 25.0], t=[0.003, 0.004], A=[2.0, 1.0])
    if dim == 3:
        kw["ay"] = [0, 10, shape[2]]
        src["sy"] = [1, shape[2] - 1]
    run = pw.afd2d if dim == 2 else pw.afd3d
    d, w = run(vel, ns=2, **src, **kw)
    do, wo = oracle.afd(vel, nt, 0.001, (10.0,) * dim, nbt=nbt, ct=0.02, src=src, jsnap=3)
    assert np.abs(do[..., 0]).max() > 0 and np.abs(do[..., -1]).max() > 0
    assert np.array_equal(d, do) and np.array_equal(w, wo)
    tr = rng.standard_normal((nt,) + shape[1:]).astype(np.float32)
    _, w = run(vel, dat=tr, tri=True, **kw)
    _, wo = oracle.afd(vel, nt, 0.001, (10.0,) * dim, nbt=nbt, ct=0.02, tri=True, dat=tr, jsnap=3)
    assert np.abs(wo).max() > 0 and np.array_equal(w, wo)


def test_batch_of_large_shots_bit_exact(cuda_lib, oracle):
    from pywave_b200.afd import afd2d_batch
    rng = np.random.default_rng(9)
    shots = []
    for nz, nx, nt in [(1500, 1700, 9), (1100, 1310, 6), (1037, 1203, 8)]:
        shots.append(dict(vel=(1500 + 900 * rng.random((nz, nx))).astype(np.float32), nt=nt,
                          dt=0.001, ax=[0, 10.0, nx], az=[0, 10.0, nz], ns=1, sx=[nx // 2],
                          sz=[1], f=[30.0], t=[0.003], A=[1.0], nbt=5, ct=0.02, gz=0))
    got = afd2d_batch(shots)
    for sh, g in zip(shots, got):
        ref, _ = oracle.afd(sh["vel"], sh["nt"], 0.001, (10.0, 10.0), nbt=5, ct=0.02, jsnap=0,
                            src={k: sh[k] for k in ("sx", "sz", "f", "t", "A")})
        assert np.abs(ref).max() > 0 and np.array_equal(g, ref)


# 32 shots of 300 x 600 (420 x 720 padded): 85 MB of wavefields
def test_pfwi_many_shots(oracle, cuda_lib):
    import pywave_b200 as pw
    from pywave_b200 import fwi
    nz, nx, nb, ns, nt, h, dt = 300, 600, 60, 32, 24, 0.01, 0.001
    rng = np.random.default_rng(4)
    vel = (2.0 + 2.0 * rng.random((nz, nx))).astype(np.float32)
    wav = (1e6 * _pulse(nt, dt, 60.0)).astype(np.float32)
    ds = 18 * h
    par = dict(nz=nz, nx=nx, dz=h, dx=h, oz=0.0, ox=0.0, nt=nt, dt=dt, ot=0.0, ns=ns, ds=ds,
               os=ds / 2, nb=nb, coef=0.005, f0=60.0, acqui_type=1, interval=1, niter=1)
    geo = oracle.pfwi_geometry(nz, nx, h, h, 0, 0, ns, ds, ds / 2, nb)
    kw = dict(nb=nb, coef=0.005, dz=h, dx=h, dt=dt, geo=geo, ns=ns)
    d = pw.pfwi(vel, np.full(vel.shape, 1e4, np.float32), wav, None, mode=1, par=par)[0]
    ref = oracle.pfwi_forward(vel, wav, **kw)
    assert np.abs(ref).max(axis=(0, 1)).min() > 0
    assert np.array_equal(d.view(np.uint32), ref.view(np.uint32))
    # shots of unlike sign and size, so that none can stand in for another
    dobs = (ref * (1.0 + rng.standard_normal(ns))).astype(np.float32)
    w = np.ones((nx, nt), np.float32)
    # sums over 32 shots in another order (32 x 6e-8), and 2 x 24 float32 steps
    g, _ = fwi.gradient(vel, wav, dobs, par, mode="reference", weight=w)
    go, _ = oracle.pfwi_gradient_ref(vel, wav, dobs, weight=w, **kw)
    assert rel_l2(g, go) < 1e-5
    ge, J = fwi.gradient(vel, wav, dobs, par, mode="exact", weight=w)
    gx, Jx = oracle.pfwi_gradient_exact(vel, wav, dobs, weight=w.astype(np.float64), **kw)
    assert rel_l2(ge, gx) < 1e-4 and abs(J - Jx) < 1e-4 * Jx


# 2 shots of 110 x 150 x 130 (126 x 166 x 146 padded): 86 MB of wavefields
def test_pfwi3d_large_grid(oracle, cuda_lib):
    from pywave_b200 import fwi3d
    nz, nx, ny, nb, nt = 110, 150, 130, 8, 9
    rng = np.random.default_rng(6)
    vt = (1.8 + 0.8 * rng.random((nz, nx, ny))).astype(np.float32)
    wav = (1e6 * _pulse(nt, 0.001, 120.0)).astype(np.float32)
    geom = dict(nb=nb, coef=0.02, dz=0.01, dx=0.012, dy=0.011, nt=nt, dt=0.001,
                src=[(3, 2, 1), (nz // 2, nx - 3, ny - 2)], rz=4, rx=list(range(0, nx, 2)),
                ry=list(range(ny)))
    d = fwi3d.forward3d(vt, wav, geom)
    d32 = oracle.pf3_forward(vt, wav, geom, "f32")
    assert np.abs(d32).max() > 0 and np.array_equal(d.view(np.uint32), d32.view(np.uint32))
    dobs = (0.5 * d32).astype(np.float32)
    # 2 x 9 steps of float32 (6e-8 each) against FP64
    g, J = fwi3d.gradient3d(vt, wav, dobs, geom)
    go, Jo = oracle.pf3_gradient_exact(vt, wav, dobs, geom)
    assert rel_l2(g, go) < 1e-4 and abs(J - Jo) < 1e-4 * Jo
