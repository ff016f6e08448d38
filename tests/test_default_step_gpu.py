"""The 3-D kernel that runs when nothing is selected, against digests of the
reference's own outputs.  GPU only."""
import os
import sys

import numpy as np
import pytest

from conftest import ROOT

sys.path.insert(0, os.path.join(ROOT, "tests", "golden"))
import models as M  # noqa: E402

pytestmark = pytest.mark.gpu

SWITCHES = ["PW_AFD_TMA", "PW_AFD_NC", "PW_AFD_SPLIT", "PW_AFD_TILE_G1"]


def _plan(capfd):
    err = capfd.readouterr().err
    return "afd quad plan" in err, "afd tile plan" in err


def _environment(monkeypatch, env):
    for name in SWITCHES:
        monkeypatch.delenv(name, raising=False)
    for name, value in env.items():
        monkeypatch.setenv(name, value)
    monkeypatch.setenv("PW_AFD_VERBOSE", "1")


# nothing set; the TMA ring declined, which selects nothing either
@pytest.mark.parametrize("env", [{}, {"PW_AFD_TMA": "0"}])
def test_default_3d_step_bit_exact_vs_reference(golden, cuda_lib, monkeypatch, capfd, env):
    """80 x 72 x 64 interior, nbt 10, nt 60: the traces and snapshots of 2
    sources, and the snapshots of the time reversal of one x-band's traces,
    identical to the reference's."""
    import pywave_b200 as pw
    g = golden("afd3d_big")
    vel = M.big3d_velocity()
    assert M.digest(vel) == str(g["vel_digest"])
    kw = dict(M.BIG3D)
    _environment(monkeypatch, env)
    d, w = pw.afd3d(vel, wavelet=g["rick"], **kw)
    assert _plan(capfd) == (True, False)
    assert np.array_equal(d[::3, ::4, ::4], g["traces_dec"])
    assert M.digest(d) == str(g["traces_digest"])
    assert tuple(w.shape) == tuple(g["snaps_shape"])
    assert np.array_equal(w[::4, ::4, ::4, -1], g["snaps_last_dec"])
    assert M.digest(w) == str(g["snaps_digest"])
    dg = np.zeros_like(d)
    b0, b1 = M.BIG3D_BAND
    dg[:, b0:b1, :] = d[:, b0:b1, :]
    _, wt = pw.afd3d(vel, nt=kw["nt"], dt=0.001, ax=kw["ax"], ay=kw["ay"], az=kw["az"],
                     jsnap=M.BIG3D_TRI_JSNAP, dat=dg, tri=True, nbt=10, ct=0.02)
    assert _plan(capfd) == (True, False)
    assert tuple(wt.shape) == tuple(g["tri_shape"])
    assert np.array_equal(wt[::4, ::4, ::4, 0], g["tri_last_dec"])
    assert M.digest(wt) == str(g["tri_snaps_digest"])


# what the verbose switches print is what is launched: 100 x 92 x 84 expanded cells are 25 float4
# x 23 groups of 4 columns in 18 blocks per plane, 420 x 720 padded ones 105 float4 x 180 groups
# of 4 planes in 591 blocks per shot
def test_printed_plans_name_the_launch(cuda_lib, monkeypatch, capfd):
    import re

    import pywave_b200 as pw
    _environment(monkeypatch, {})
    kw = dict(M.BIG3D, nt=30)
    pw.afd3d(M.big3d_velocity(), **kw)
    err = capfd.readouterr().err
    assert "afd quad plan: G=1 nq=25 threads=128 grid=18x84x1" in err, err
    counts = re.search(r"afd quad warps per step: plain=(\d+) y_taper=(\d+) zx_taper=(\d+) other=(\d+)", err)
    assert sum(int(c) for c in counts.groups()) == 18 * 4 * 84  # every warp is counted once
    monkeypatch.setenv("PW_PFWI_VERBOSE", "1")
    nz, nx, nt = 300, 600, 4
    par = dict(nz=nz, nx=nx, dz=0.01, dx=0.01, oz=0.0, ox=0.0, nt=nt, dt=0.001, ot=0.0, ns=2, ds=3.0,
               os=1.5, nb=60, coef=0.005, f0=10.0, acqui_type=1, interval=1, niter=1)
    v = np.full((nz, nx), 2.0, np.float32)
    pw.pfwi(v, np.full(v.shape, 1e4, np.float32), np.ones(nt, np.float32), None, mode=1, par=par)
    err = capfd.readouterr().err
    assert "pfwi step: mode=0 nz4=105 shots=2 grid=591x2 threads=128 zig=0" in err, err
