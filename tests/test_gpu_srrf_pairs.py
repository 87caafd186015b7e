"""The fused SRRF kernel's frame pairs: odd frame counts, chunks that end inside
a pair, tiles of every magnification with a remainder in both axes, and regions
without any gradient.  A frame's arithmetic does not depend on its partner, so
every frame of a stack equals the same frame run alone, bit for bit (the runs
alone are held against the float64 oracle by the parity tests).
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


def _frames(T, H, W, seed):
    rng = np.random.default_rng(seed)
    x = rng.poisson(100, (T, H, W)).astype(np.float32)
    x[:, : H // 3, : W // 3] = 100.0  # no gradient at all
    return x


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("T", [2, 3, 11])
def test_frames_do_not_mix(m, T):
    x = torch.from_numpy(_frames(T, 17, 37, seed=m)).cuda()
    whole = nx.SRRF(x, magnification=m, macro_pixel_correction=False)
    for t in range(T):
        one = nx.SRRF(x[t:t + 1], magnification=m, macro_pixel_correction=False)
        assert torch.equal(whole[t], one[0])


def test_nan_and_inf_stay():
    x = _frames(2, 16, 40, seed=5)
    x[0, 8, 20] = np.nan
    x[1, 8, 20] = np.inf
    got = nx.SRRF(torch.from_numpy(x).cuda(), macro_pixel_correction=False).cpu().numpy()
    assert np.isnan(got[0, 8 * 5:9 * 5, 20 * 5:21 * 5]).all()
    assert not np.isfinite(got[1, 8 * 5:9 * 5, 20 * 5:21 * 5]).any()
    assert np.isfinite(got[:, :4 * 5]).all() and np.isfinite(got[..., :14 * 5]).all()
