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


# 2-D step per launch (the resident kernel switched off): depths around 1, 2, 31 .. 33 float4,
# widths around the 4 columns of a CTA
@pytest.mark.parametrize("nz,nx,nbt", [(3, 2, 0), (5, 9, 1), (60, 37, 4), (100, 13, 14),
                                       (101, 18, 14), (103, 31, 15)])
def test_afd2d_step_sizes_bit_exact(oracle, cuda_lib, monkeypatch, nz, nx, nbt):
    import pywave_b200 as pw
    monkeypatch.setenv("PW_AFD_RESIDENT", "0")
    nt = 60
    rng = np.random.default_rng(nz * 100 + nx)
    vel = (1500 + 1500 * rng.random((nz, nx))).astype(np.float32)
    kw = dict(nt=nt, dt=0.001, ax=[0, 10, nx], az=[0, 10, nz], nbt=nbt, ct=0.02, jsnap=7)
    s1 = dict(sx=[nx // 2], sz=[nz // 2], f=[30.0], t=[0.01], A=[2.0])
    if nbt >= 1:
        d, w = pw.afd2d(vel, ns=1, **s1, **kw)
        do, wo = oracle.afd(vel, nt, 0.001, (10.0, 10.0), nbt=nbt, ct=0.02, src=s1, jsnap=7)
        assert np.array_equal(d, do) and np.array_equal(w, wo)
    tr = rng.standard_normal((nt, nx)).astype(np.float32)
    _, w = pw.afd2d(vel, dat=tr, tri=True, **kw)
    _, wo = oracle.afd(vel, nt, 0.001, (10.0, 10.0), nbt=nbt, ct=0.02, tri=True, dat=tr, jsnap=7)
    assert np.abs(wo).max() > 0 and np.array_equal(w, wo)


@pytest.mark.parametrize("nz,nx,ny,nbt", [(3, 2, 3, 0), (7, 5, 6, 2), (58, 11, 9, 3),
                                          (100, 6, 5, 14), (103, 9, 4, 13)])
def test_afd3d_step_sizes_bit_exact(oracle, cuda_lib, nz, nx, ny, nbt):
    import pywave_b200 as pw
    nt = 40
    rng = np.random.default_rng(nz * 100 + nx)
    vel = (1500 + 1500 * rng.random((nz, nx, ny))).astype(np.float32)
    kw = dict(nt=nt, dt=0.001, ax=[0, 10, nx], ay=[0, 10, ny], az=[0, 10, nz], nbt=nbt, ct=0.02,
              jsnap=9)
    s2 = dict(sx=[nx // 2, nx - 1], sy=[ny // 2, 0], sz=[nz // 2, 1], f=[30.0, 25.0],
              t=[0.01, 0.004], A=[2.0, 1.0])
    if nbt >= 1:
        d, w = pw.afd3d(vel, ns=2, **s2, **kw)
        do, wo = oracle.afd(vel, nt, 0.001, (10.0,) * 3, nbt=nbt, ct=0.02, src=s2, jsnap=9)
        assert np.array_equal(d, do) and np.array_equal(w, wo)
    tr = rng.standard_normal((nt, nx, ny)).astype(np.float32)
    _, w = pw.afd3d(vel, dat=tr, tri=True, **kw)
    _, wo = oracle.afd(vel, nt, 0.001, (10.0,) * 3, nbt=nbt, ct=0.02, tri=True, dat=tr, jsnap=9)
    assert np.abs(wo).max() > 0 and np.array_equal(w, wo)


@pytest.mark.parametrize("dim", [2, 3])
def test_tri_image_groups_equal_single_runs(cuda_lib, monkeypatch, dim):
    """The image formed inside the step (3 groups in lockstep) against the
    product of three time reversals' snapshots, in group order."""
    import pywave_b200 as pw
    monkeypatch.setenv("PW_AFD_RESIDENT", "0")
    rng = np.random.default_rng(dim)
    nt, js, G = 90, 5, 3
    shape = (33, 30) if dim == 2 else (33, 18, 7)
    vel = (1500 + 1500 * rng.random(shape)).astype(np.float32)
    tr = rng.standard_normal((nt,) + shape[1:]).astype(np.float32)
    grp = rng.integers(-1, G, shape[:0:-1]).astype(np.int32).reshape(-1, shape[1])  # [ny, nx]
    kw = dict(dt=0.001, nbt=6, ct=0.02, jsnap=js)
    img = pw.tri_image(vel, tr, d=(10.0,) * dim, ngroups=G, groups=grp, normalize=False, **kw)
    prod = None
    ax = dict(ax=[0, 10, shape[1]], az=[0, 10, shape[0]])
    if dim == 3:
        ax["ay"] = [0, 10, shape[2]]
    for g in range(G):
        m = (grp == g).T if dim == 3 else (grp[0] == g)
        _, w = (pw.afd2d if dim == 2 else pw.afd3d)(vel, nt=nt, dat=(tr * m).astype(np.float32),
                                                    tri=True, **ax, **kw)
        prod = w * w if prod is None else prod * w * w
    ref = np.zeros(shape, np.float32)
    for k in range(prod.shape[-1] - 1, -1, -1):  # time reversal: the last snapshot comes first
        ref += prod[..., k]
    assert np.abs(ref).max() > 0 and np.array_equal(img, ref)


def test_batch_of_more_shots_than_the_constant_table(cuda_lib):
    import pywave_b200 as pw
    from pywave_b200.afd import afd2d_batch
    rng = np.random.default_rng(5)
    shots = []
    for k in range(101):
        nz, nx, nt = 12 + k % 7, 10 + k % 5, 20 + k % 9
        shots.append(dict(vel=(1500 + 900 * rng.random((nz, nx))).astype(np.float32), nt=nt,
                          dt=0.001, ax=[0, 10.0, nx], az=[0, 10.0, nz], ns=1, sx=[nx // 2],
                          sz=[nz // 2], f=[30.0], t=[0.005], A=[1.0], nbt=5, ct=0.02, gz=0))
    got = afd2d_batch(shots)
    for k, sh in enumerate(shots):
        kw = {n: sh[n] for n in ("nt", "dt", "ax", "az", "ns", "sx", "sz", "f", "t", "A", "nbt", "ct")}
        ref = pw.afd2d(sh["vel"], jsnap=0, **kw).reshape(sh["nt"], sh["ax"][2], order="F")
        assert np.abs(ref).max() > 0 and np.array_equal(got[k], ref), k


# padded depths of 15, 20, 128 (32 float4), 130 and 131 cells; widths off the 4 columns of a CTA
@pytest.mark.parametrize("nz,nx,ny,nb,ns", [(5, 6, 5, 5, 1), (8, 9, 7, 6, 3), (112, 7, 6, 8, 1),
                                            (114, 6, 7, 8, 2), (115, 9, 5, 8, 1)])
def test_pfwi3d_step_sizes(oracle, cuda_lib, nz, nx, ny, nb, ns):
    from pywave_b200 import fwi3d
    nt = 70
    rng = np.random.default_rng(nz * 10 + nx)
    vt = (1.8 + 0.8 * rng.random((nz, nx, ny))).astype(np.float32)
    wav = (1e6 * _pulse(nt, 0.001, 40.0)).astype(np.float32)
    geom = dict(nb=nb, coef=0.02, dz=0.01, dx=0.012, dy=0.011, nt=nt, dt=0.001,
                src=[(nz // 2, (i * 2) % nx, i % ny) for i in range(ns)], rz=nz // 2,
                rx=list(range(0, nx, 2)), ry=list(range(ny)))
    d = fwi3d.forward3d(vt, wav, geom)
    d32 = oracle.pf3_forward(vt, wav, geom, "f32")
    assert np.abs(d32).max() > 0 and np.array_equal(d.view(np.uint32), d32.view(np.uint32))
    dobs = (0.5 * d32).astype(np.float32)
    # 2 x 70 steps of float32 (6e-8 each) against FP64, the residual half the data; edges and
    # corners fold (nb + 1)^2 and (nb + 1)^3 padded cells
    g, J = fwi3d.gradient3d(vt, wav, dobs, geom)
    go, Jo = oracle.pf3_gradient_exact(vt, wav, dobs, geom)
    assert rel_l2(g, go) < 1e-4 and abs(J - Jo) < 1e-4 * Jo


# both sides of the rule that picks the lstri plan (small and large grids, one wave of shots
# and more), odd depths, and a velocity whose square overflows: the cluster-resident kernel, a
# launch per step and the default give identical bits (NaN where the others do)
@pytest.mark.parametrize("nz,nx,nb,ns,vmax", [(30, 37, 9, 1, 3.0), (85, 90, 40, 1, 3.0),
                                              (131, 150, 40, 1, 3.0), (131, 150, 40, 2, 3.0),
                                              (33, 34, 6, 24, 3.0), (70, 83, 20, 24, 3.0),
                                              (42, 45, 8, 1, 1e25)])
def test_lstri_plans_agree(cuda_lib, monkeypatch, nz, nx, nb, ns, vmax):
    from pywave_b200 import lstri
    nt = 40
    rng = np.random.default_rng(nz)
    vel = (1.5 + 1.5 * rng.random((nz, nx))).astype(np.float32)
    if vmax > 3.0:
        vel[5, 7] = vel[-1, 3] = vmax
    par = dict(nz=nz, nx=nx, dz=0.01, dx=0.012, oz=0, ox=0, nt=nt, dt=0.001, ot=0, ns=ns, ds=0.1,
               os=0.0, nb=nb, coef=0.01, f0=10, acqui_type=1, interval=1, niter=2, rz=2)
    src = rng.standard_normal((nz, nx, nt, ns)).astype(np.float32)
    dat = rng.standard_normal((nt, nx)).astype(np.float32)
    got = []
    for r in (None, "1", "0"):
        if r is None:
            monkeypatch.delenv("PW_LSTRI_RESIDENT", raising=False)
        else:
            monkeypatch.setenv("PW_LSTRI_RESIDENT", r)
        got.append([lstri.lstri_forward(vel, src, par),
                    lstri.timerev(False, vel, dict(par, ns=1), mod=src[..., 0]),
                    lstri.timerev(True, vel, dict(par, ns=1), dat=dat)])
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert np.array_equal(x, y, equal_nan=True)
    assert all(np.abs(x[np.isfinite(x)]).max() > 0 for x in got[0])


# launches below and above the size up to which a step's fixed operands are read before the
# previous step has ended (160 000 threads): 2-D and 3-D, forward and time reversal
@pytest.mark.parametrize("shape", [(391, 800), (415, 1650), (60, 40, 31), (92, 70, 61)])
def test_afd_fixed_operands_read_ahead(oracle, cuda_lib, monkeypatch, shape):
    import pywave_b200 as pw
    monkeypatch.setenv("PW_AFD_RESIDENT", "0")
    nt, dim, nbt = 9, len(shape), 6
    rng = np.random.default_rng(shape[1])
    vel = (1500 + 1500 * rng.random(shape)).astype(np.float32)
    kw = dict(nt=nt, dt=0.001, ax=[0, 10, shape[1]], az=[0, 10, shape[0]], nbt=nbt, ct=0.02, jsnap=4)
    src = dict(sx=[shape[1] // 2], sz=[0], f=[30.0], t=[0.003], A=[2.0])
    if dim == 3:
        kw["ay"] = [0, 10, shape[2]]
        src["sy"] = [shape[2] // 2]
    run = pw.afd2d if dim == 2 else pw.afd3d
    d, w = run(vel, ns=1, **src, **kw)
    do, wo = oracle.afd(vel, nt, 0.001, (10.0,) * dim, nbt=nbt, ct=0.02, src=src, jsnap=4)
    assert np.abs(do).max() > 0 and np.array_equal(d, do) and np.array_equal(w, wo)
    tr = rng.standard_normal((nt,) + shape[1:]).astype(np.float32)
    _, w = run(vel, dat=tr, tri=True, **kw)
    _, wo = oracle.afd(vel, nt, 0.001, (10.0,) * dim, nbt=nbt, ct=0.02, tri=True, dat=tr, jsnap=4)
    assert np.abs(wo).max() > 0 and np.array_equal(w, wo)
