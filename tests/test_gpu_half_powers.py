"""RGC values to a half-integer sensitivity, correctly rounded but for 1 in 50: a
per-frame map at sensitivity n + 1/2 against the float64 power of the map at
sensitivity 1, whose values are the bases bit for bit, and the mean of one frame
through a sweep's and the accumulator's kernels.

The products' and the root's errors are carried along (terms of 2^-48, 15 at most),
so what is left is the last rounding: 0.51 ulp.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


def _ulps(got, base, s):
    ref = base.astype(np.float64) ** s
    keep = ref > 1e-36  # normal results
    assert keep.mean() > 0.5
    got, ref = got[keep], ref[keep]
    return float((np.abs(got - ref) / np.spacing(ref.astype(np.float32)).astype(np.float64)).max())


@pytest.mark.parametrize("s", [1.5, 2.5, 3.5, 4.5, 7.5, 15.5])
@pytest.mark.parametrize("m", [2, 4, 5, 7])
def test_half_integer_powers(m, s):
    x = torch.from_numpy(np.random.default_rng(m).poisson(100, (1, 40, 70)).astype(np.float32))
    x = x.cuda()
    kw = dict(magnification=m, radius=1.5, doIntensityWeighting=False)
    op = nx.eSRRF_ST(verbose=False)
    base = op.run(x, sensitivity=1, **kw).cpu().numpy()
    assert _ulps(op.run(x, sensitivity=s, **kw).cpu().numpy(), base, s) <= 0.51
    mean = nx.eSRRF(x, sensitivity=s, temporal_correlation="AVG", macro_pixel_correction=False,
                    **kw).cpu().numpy()
    assert _ulps(mean.reshape(base.shape), base, s) <= 0.51
