"""The rounding of merged chunks, as the 2-norm of a mean's error over that of the image,
against the float64 mean of the same per-frame maps; small images, which split most.

A merge rounds the mean by 0.4 x 2^-24, diluted by the frames that follow: a chain of K
equal parts by that times sqrt(sum over k = 2 .. K of (k / K)^2).  32 frames in 16 chunks
of 2: one chain 5.8e-8; in two groups of 8, 3.9e-8 and less with their rounding carried along.  100 frames in pushes of 16 (8 chunks
each): one chain of all chunks 9.9e-8; of the pushes, each merged first, 4.3e-8.  The
bounds leave a quarter.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


def _stack(T, m):
    x = torch.from_numpy(np.random.default_rng(T).poisson(100, (T, 26, 64)).astype(np.float32))
    maps = nx.eSRRF_ST(verbose=False).run(x.cuda(), magnification=m, radius=1.0, sensitivity=2)
    return x.cuda(), maps.double().mean(0)


def _error(got, ref):
    return float((got.reshape(ref.shape).double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("m", [1, 2])
def test_chunks_of_one_call(m):
    x, ref = _stack(32, m)
    got = nx.eSRRF(x, magnification=m, radius=1.0, sensitivity=2, macro_pixel_correction=False)
    assert _error(got, ref) <= 4.8e-8


@pytest.mark.parametrize("m", [1, 2, 5])
def test_chunks_of_pushes(m):
    x, ref = _stack(100, m)
    acc = nx.ESRRFAccumulator(26, 64, magnification=m, radius=1.0, sensitivity=2)
    for a in range(0, 100, 16):
        acc.push(x[a:a + 16])
    assert _error(acc.finalize_device(("AVG",), False)[0], ref) <= 5.5e-8
