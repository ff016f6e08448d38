"""pw_afd_noalloc at the exact size of its fixed scratch array.  GPU only."""
import numpy as np
import pytest

from test_zz_no_alloc import _case, _run

pytestmark = pytest.mark.gpu


# 149 x 256, 10 taper cells (169 x 276 expanded): 32135 steps of traces fill the 32 MiB to the
# byte (depth 4k + 1: a z table padded to 4k cells would take 256 bytes more); one more step does
# not fit
def test_noalloc_takes_a_call_that_fills_its_scratch(cuda_lib):
    from pywave_b200 import _lib as L
    a, dev, shapes = _case(2, (149, 256), 32135, 10, 1, 0, seed=3)
    dat, _ = _run(cuda_lib.pw_afd_noalloc, a, dev, shapes)
    ref, _ = _run(cuda_lib.pw_afd, a, dev, shapes)
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0 and np.array_equal(dat, ref)
    a, dev, shapes = _case(2, (149, 256), 32136, 10, 1, 0, seed=3)
    with pytest.raises(L.ShapeError, match="scratch"):
        _run(cuda_lib.pw_afd_noalloc, a, dev, shapes)
