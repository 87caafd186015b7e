"""eSRRF-3D at the ends of the gradients' range: stacks in units in which the squared
gradients leave float32, and infinite and missing pixels.

Scaling the frames by a power of two changes no direction: the normalisation is good
to 2^-22 either way, and so is the weighted mean of the samples: 2e-6.  An infinite
or NaN gradient counts nothing in the reference, so the map without intensity
weighting stays finite; 2e-5 as for ordinary frames.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx
from conftest import rel_err
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu


def _run(x, mags):
    return nx.eSRRF3D_ST(verbose=False).run(x, magnification_xy=mags[0], magnification_z=mags[1],
                                            radius=1.5, sensitivity=1, mode="average",
                                            doIntensityWeighting=False)


@pytest.mark.parametrize("mags", [(1, 1), (2, 2)])
@pytest.mark.parametrize("power", [-70, -100, 60, 90])
def test_scale_of_the_frames(mags, power):
    x = np.random.default_rng(2).poisson(100, (2, 7, 21, 45)).astype(np.float32)
    assert rel_err(_run(x * np.float32(2.0 ** power), mags), _run(x, mags)) <= 2e-6


@pytest.mark.parametrize("mags", [(1, 1), (1, 2)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_infinite_and_missing_pixels(mags, value):
    x = np.random.default_rng(5).poisson(100, (1, 7, 21, 45)).astype(np.float32)
    x[0, 3, 10, 20] = value
    with np.errstate(invalid="ignore"):
        ref = O.esrrf3d_st(x, mags[0], mags[1], 1.5, 2.8, 4.0, 1, "average", False)
    assert np.isfinite(ref).all()
    assert rel_err(_run(x, mags), ref) <= 2e-5
