"""3-D time reversal by the number of receiver groups: one to four have a kernel
each, more share one.  Against the oracle's runs of each group.  GPU only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 5 x 9 x 6 and 28 x 18 x 21 padded cells (fixed operands read ahead of the previous step), and
# 97 x 92 x 90 (more threads than that is done for); an image every step and every 3rd
@pytest.mark.parametrize("shape,nbt,jsnap", [((3, 7, 4), 1, 1), ((20, 10, 13), 4, 3),
                                             ((89, 84, 82), 4, 3)])
@pytest.mark.parametrize("ng", [1, 2, 3, 4, 5])
def test_image_of_each_group_count(oracle, cuda_lib, shape, nbt, jsnap, ng):
    import pywave_b200 as pw
    nt = 40 if shape[0] < 50 else 10
    rng = np.random.default_rng(shape[0] + ng)
    vel = (1500 + 1500 * rng.random(shape)).astype(np.float32)
    d = rng.standard_normal((nt,) + shape[1:]).astype(np.float32)
    grp = rng.integers(-1, ng, shape[:0:-1]).astype(np.int32)  # [ny, nx], some receivers unused
    grp.reshape(-1)[:ng] = np.arange(ng)  # none empty
    img = pw.tri_image(vel, d, dt=0.001, d=(10.0,) * 3, ngroups=ng, groups=grp, nbt=nbt, ct=0.02,
                       jsnap=jsnap, normalize=False)
    snaps = []
    for g in range(ng):
        dg = np.where(grp.T == g, d, np.float32(0))
        snaps.append(oracle.afd(vel, nt, 0.001, (10.0,) * 3, nbt=nbt, ct=0.02, tri=True, dat=dg,
                                jsnap=jsnap)[1])
    # product of the squares in group order, summed over the steps as they run (last first)
    ref = np.zeros(shape, np.float32)
    for it in range(snaps[0].shape[-1] - 1, -1, -1):
        p = np.ones(shape, np.float32)
        for w in snaps:
            p = p * w[..., it] * w[..., it]
        ref = ref + p
    assert all(np.abs(w).max() > 0 for w in snaps)
    if nbt > 1:  # on 5 x 9 x 6 cells the edge receivers' fields do not meet
        assert np.abs(ref).max() > 0
    assert np.array_equal(img, ref)
