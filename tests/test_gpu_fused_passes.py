"""The fused eSRRF kernel where its passes, tiles and walks end: frame counts
that leave a pass with one to four frames, frames smaller than a tile, one past
a tile, with and without 16-byte rows, windows that reach past the clamped last
half-grid position, and every magnification's thread layout.

Integer-valued frames make the gradients and their half-grid interpolation
exact in float32, so what is left is the normalisation (2^-22), the weights
(2^-24), the mean of up to 169 terms, the power (x 2) and the intensity
coordinate fl(i / m) (~1e-6 of the range): 1e-5 of the range bounds the sum.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx
from conftest import rel_err
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _frames(T, H, W, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:H, 0:W]
    spots = sum(60.0 * np.exp(-((y - rng.uniform(0, H)) ** 2 + (x - rng.uniform(0, W)) ** 2) / 4)
                for _ in range(4))
    return rng.poisson(100 + spots, (T, H, W)).astype(np.float32)


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 7])
@pytest.mark.parametrize("shape", [(5, 7), (33, 36)])
def test_frames_left_in_the_last_pass(T, shape):
    x = _frames(T, *shape, seed=T)
    got = nx.eSRRF_ST(verbose=False).run(x, magnification=5, radius=1.5, sensitivity=2)
    assert rel_err(got, O.esrrf_st(x, 5, 1.5, 2)) <= TOL
    got = nx.eSRRF(torch.from_numpy(x).cuda(), 5, 1.5, 2, temporal_correlation=("AVG", "VAR"),
                   macro_pixel_correction=False)
    maps = O.esrrf_st(x, 5, 1.5, 2)
    assert rel_err(got[0].cpu().numpy(), maps.mean(0)) <= TOL
    if T > 1:
        assert rel_err(got[1].cpu().numpy(), maps.var(0)) <= 4 * TOL


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("radius", [0.5, 1.0, 2.0, 3.0])
def test_thread_layouts_and_window_reach(m, radius):
    # 9 rows end inside a tile of every height; 37 columns are one tile and
    # five columns, with rows that are not a multiple of 16 bytes
    x = _frames(5, 9, 37, seed=m)
    got = nx.eSRRF_ST(verbose=False).run(x, magnification=m, radius=radius, sensitivity=1)
    ref = O.esrrf_st(x, m, radius, 1)
    if ref.max() > ref.min():
        assert rel_err(got, ref) <= TOL
    else:
        assert np.array_equal(got, ref.astype(np.float32))
