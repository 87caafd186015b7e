"""eSRRF-3D where its frame pairs, tiles and shared slices end: odd frame counts,
volumes that leave a remainder in every axis, z magnifications whose voxels
share (or, at the first and last slices, do not share) their samples, and no
magnification at all.

Integer-valued frames make the gradients exact; the interpolation weights
(2^-24 of values up to ~150 against gradients of order 1), the normalisation
(2^-22) and the weighted mean of up to 44 samples leave 2e-5 of the range.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx
from conftest import rel_err
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu
TOL = 2e-5


def _frames(T, S, H, W, seed):
    return np.random.default_rng(seed).poisson(100, (T, S, H, W)).astype(np.float32)


@pytest.mark.parametrize("T", [1, 2, 3])
@pytest.mark.parametrize("mags", [(1, 1), (1, 2), (2, 1), (2, 3), (3, 2)])
@pytest.mark.parametrize("mode", ["average", "std"])
def test_pairs_tiles_and_slices(T, mags, mode):
    if T == 1 and mode == "std":
        pytest.skip("the deviation of one frame is 0 everywhere")
    x = _frames(T, 7, 21, 45, seed=T)
    got = nx.eSRRF3D_ST(verbose=False).run(x, magnification_xy=mags[0], magnification_z=mags[1],
                                           radius=1.5, sensitivity=1, mode=mode)
    ref = O.esrrf3d_st(x, mags[0], mags[1], 1.5, 2.8, 4.0, 1, mode, True)
    assert rel_err(got, ref) <= TOL
