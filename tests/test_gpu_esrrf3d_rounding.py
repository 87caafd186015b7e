"""How much rounding eSRRF-3D's weighted mean adds, as the 2-norm of the error over that
of the map (no magnification, one frame, no intensity: nothing else rounds).

A chain of n sums rounds by 0.4 x 2^-24 sqrt(n / 3) of its result.  Summed row by row
the longest chain is that over the rows with samples, about 30 at radius 2 and 56 at
radius 3: 7.5e-8 and 1.03e-7.  With as much as 2^-24 for the sum of the weights, a
constant of the map, and 3e-8 for a sample's own roundings, the division and the
weights, that is 1.0e-7 and 1.23e-7; the bounds leave a quarter.  One chain over all
83 and 300 samples gives 1.4e-7 and 2.5e-7.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,bound", [(2.0, 1.25e-7), (3.0, 1.55e-7)])
def test_weighted_mean(radius, bound):
    x = np.random.default_rng(8).poisson(100, (1, 14, 40, 70)).astype(np.float32)
    got = nx.eSRRF3D_ST(verbose=False).run(x, magnification_xy=1, magnification_z=1,
                                           radius=radius, sensitivity=1, mode="average",
                                           doIntensityWeighting=False)
    ref = O.esrrf3d_st(x, 1, 1, radius, 2.8, 4.0, 1, "average", False)
    assert np.linalg.norm(got - ref) <= bound * np.linalg.norm(ref)
