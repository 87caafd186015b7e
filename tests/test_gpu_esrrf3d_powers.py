"""eSRRF-3D's RGC to integer and half-integer sensitivities: a one-frame map against
the float64 power of the map at sensitivity 1, whose values are the bases bit for
bit.  The products' and the root's errors are carried along, so what is left is the
last rounding: 0.51 ulp.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [2, 3, 4, 7, 16, 1.5, 2.5, 7.5])
@pytest.mark.parametrize("mags", [(1, 1), (2, 2)])
def test_powers(mags, s):
    x = np.random.default_rng(3).poisson(100, (1, 7, 21, 45)).astype(np.float32)
    kw = dict(magnification_xy=mags[0], magnification_z=mags[1], radius=1.5, mode="average",
              doIntensityWeighting=False)
    op = nx.eSRRF3D_ST(verbose=False)
    ref = op.run(x, sensitivity=1, **kw).astype(np.float64) ** s
    got = op.run(x, sensitivity=s, **kw)
    keep = ref > 1e-36  # normal results
    assert keep.mean() > 0.2
    ulp = np.spacing(ref[keep].astype(np.float32)).astype(np.float64)
    assert (np.abs(got[keep] - ref[keep]) / ulp).max() <= 0.51
