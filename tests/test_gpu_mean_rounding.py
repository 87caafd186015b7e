"""The rounding of the temporal mean, as the 2-norm of its error over that of the image,
against the float64 mean of the same per-frame maps.

A running mean of n frames rounds by 0.4 x 2^-24 sqrt(n / 3): 8.7e-8 for chunks of 40
frames, the longest the 200-frame sweep may take here, with an eighth of it for the
merging of the chunks: 1.0e-7 (chunks of 100: 1.4e-7).
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


def _frames(T, H, W, seed):
    x = np.random.default_rng(seed).poisson(100, (T, H, W)).astype(np.float32)
    return torch.from_numpy(x).cuda()


def _error(mean, maps):
    ref = maps.double().mean(0)
    return float((mean.reshape(ref.shape).double() - ref).norm() / ref.norm())


def test_sweep_of_many_frames():
    x = _frames(200, 256, 256, 1)
    grid = nx.esrrf_parameter_sweep(x, magnification=4, sensitivities=[1, 2], radii=[1.5, 2.0])
    op = nx.eSRRF_ST(verbose=False)
    for i, s in enumerate((1, 2)):
        maps = op.run(x, magnification=4, radius=1.5, sensitivity=s)
        assert _error(torch.as_tensor(grid[i, 0]).cuda(), maps) <= 1.0e-7
