"""SRRF one frame at a time (a stack of one frame, or images too small to fill the GPU)
against the frame pairs of larger stacks: the same operations per frame, so the same
bits, with the intensity formed in the kernel or given, a ring that moves no centre, and
frames in units whose squared gradients are denormal.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


def _frames(T, h, w, seed):
    return torch.from_numpy(np.random.default_rng(seed).poisson(100, (T, h, w)).astype(np.float32)).cuda()


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("T", [2, 3])
@pytest.mark.parametrize("ring,power", [(0.5, 0), (2.0, 0), (0.0, 0), (0.5, -62)])
def test_frames_of_a_pair(m, T, ring, power):
    x = torch.ldexp(_frames(T, 150, 210, m), torch.tensor(power))
    kw = dict(magnification=m, ringRadius=ring, radialityPositivityConstraint=False,
              doIntensityWeighting=power == 0, macro_pixel_correction=False)
    got = nx.SRRF(x, **kw)
    for t in range(T):
        assert torch.equal(got[t], nx.SRRF(x[t:t + 1], **kw)[0])


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 8])
def test_given_intensity(m):
    x, z = _frames(3, 150, 210, m), _frames(3, 150 * m, 210 * m, 1)
    op = nx.Radiality(verbose=False)
    got = op.run(x, z, magnification=m)
    for t in range(3):
        assert torch.equal(got[t], op.run(x[t:t + 1], z[t:t + 1], magnification=m)[0])


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("h,w", [(3, 3), (5, 33), (9, 31), (21, 70)])
def test_small_images(m, h, w):
    """Frames of a launch that leaves SMs idle against the same frames 60 times over."""
    x = _frames(2, h, w, m)
    kw = dict(magnification=m, macro_pixel_correction=False)
    many = nx.SRRF(x.repeat(160, 1, 1), **kw)
    assert torch.equal(nx.SRRF(x, **kw), many[-2:])
