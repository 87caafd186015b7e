"""SRRF does not depend on the units of a stack: radiality is a ratio of gradients,
so frames scaled by a power of two give the radiality of the frames themselves.

Scaling by 2^-k is exact, so nothing differs until a squared gradient comes near
the smallest floats.  At k = 64 one of interpolated gradient 2^-2 is 2^-132, with
2^-18 of relative rounding, and moves its one of twelve ring terms by half of that;
the noise of these frames leaves hardly any below: the parity bar of 1e-4 holds.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("power", [30, -50, -60, -64])
def test_scale_of_the_frames(m, power):
    x = torch.from_numpy(np.random.default_rng(m).poisson(100, (3, 17, 37)).astype(np.float32))
    x = x.cuda()
    kw = dict(magnification=m, macro_pixel_correction=False, doIntensityWeighting=False)
    ref = nx.SRRF(x, **kw)
    got = nx.SRRF(torch.ldexp(x, torch.tensor(power)), **kw)
    assert float((got - ref).abs().max()) <= 1e-4 * float(ref.max() - ref.min())
