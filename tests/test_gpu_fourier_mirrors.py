"""The Fourier interpolation with the mirror images folded into its operators:
tiles taller than wide and wider than tall (either order of the products), one
pixel a side, odd and even numbers of images, sides at and next to multiples of
16, and frames above one tile whose last tiles are narrow.

The products are float32 sums over the tile's rows and columns (up to 256 terms,
~ 16 x 2^-24 of the amplitude) and the rescale adds a few roundings: 1e-5 of the
range.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx
from conftest import rel_err
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("shape,m", [((1, 1, 9), 2), ((1, 9, 1), 3), ((2, 16, 17), 2),
                                     ((9, 33, 129), 2), ((2, 129, 33), 3), ((2, 200, 70), 2),
                                     ((2, 70, 200), 2), ((1, 100, 100), 4), ((9, 20, 300), 2),
                                     ((1, 300, 20), 2)])
def test_folded_mirrors(shape, m):
    x = np.random.default_rng(m).poisson(50, shape).astype(np.float32)
    assert rel_err(nx.fht_space_interpolation(x, m), O.fht_space_interpolation(x, m)) <= TOL


@pytest.mark.parametrize("shape,m", [((8, 256, 250), 4), ((8, 128, 120), 2), ((3, 200, 256), 3)])
def test_product_tiles_by_size(shape, m):
    """Products of enough blocks for each of the tile sizes, and partly filled ones."""
    x = np.random.default_rng(m).poisson(50, shape).astype(np.float32)
    assert rel_err(nx.fht_space_interpolation(x, m), O.fht_space_interpolation(x, m)) <= TOL


@pytest.mark.parametrize("shape", [(2, 224, 257), (1, 225, 481), (2, 449, 30), (1, 500, 260)])
def test_tiles_overlap(shape):
    """Frames whose last tiles lie inside, at the edge of and beyond the one before."""
    x = np.random.default_rng(shape[1]).poisson(50, shape).astype(np.float32)
    assert rel_err(nx.fht_space_interpolation(x, 2), O.fht_space_interpolation(x, 2)) <= TOL
