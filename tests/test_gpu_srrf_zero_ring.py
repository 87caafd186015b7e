"""SRRF with a ring of radius 0: every ring point is the output's centre, where no
gradient points outwards, so all twelve terms count 1 wherever there is a gradient
and the radiality is exactly 1 inside the image's frame of one pixel and 0 in it.
At an odd magnification the middle output of a pixel takes that pixel's gradient
alone: 0 where it is 0.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("positivity", [True, False])
def test_every_term_counts(m, positivity):
    x = np.random.default_rng(m).poisson(100, (3, 17, 37)).astype(np.float32)
    got = nx.SRRF(torch.from_numpy(x).cuda(), magnification=m, ringRadius=0.0,
                  radialityPositivityConstraint=positivity, doIntensityWeighting=False,
                  macro_pixel_correction=False).cpu().numpy()
    ref = np.zeros_like(got)
    ref[:, m:-m, m:-m] = 1.0
    if m % 2:
        for t in range(3):
            gx, gy = O.gradient_radiality(x[t])
            ref[t, m // 2::m, m // 2::m][(gx == 0) & (gy == 0)] = 0.0
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 8])
def test_rings_below_the_coordinates_resolution(m):
    """A ring too small to move a centre: every term is 1 with the sign of its outward
    component, whatever the radius."""
    x = torch.from_numpy(np.random.default_rng(m).poisson(100, (2, 17, 37)).astype(np.float32))
    kw = dict(magnification=m, radialityPositivityConstraint=False, doIntensityWeighting=False,
              macro_pixel_correction=False)
    ref = nx.SRRF(x.cuda(), ringRadius=1e-12, **kw)
    assert torch.isfinite(ref).all() and ref.abs().max() <= 1.0
    for ring in (1e-20, 1e-30):
        assert torch.equal(nx.SRRF(x.cuda(), ringRadius=ring, **kw), ref)
