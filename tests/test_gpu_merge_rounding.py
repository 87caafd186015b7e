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


@pytest.mark.parametrize("m", [1, 2])
def test_sweep_maps_are_one_chain(m):
    """The maps that sweeps score at m <= 2 are one chain of chunk means whatever the
    chunks: 174 frames of 103 x 78 in more than 8, against the same chain in float32."""
    x = torch.from_numpy(np.random.default_rng(3).poisson(100, (174, 103, 78)).astype(np.float32))
    x = x.cuda()
    got = nx.esrrf_parameter_sweep(x, magnification=m, sensitivities=[1], radii=[1.0])[0, 0]
    maps = nx.eSRRF_ST(verbose=False).run(x, magnification=m, radius=1.0, sensitivity=1)

    def chain(chunks):
        mean, have = None, 0
        for c in range(chunks):
            a, b = c * 174 // chunks, (c + 1) * 174 // chunks
            part = maps[a]
            for k in range(1, b - a):  # one rounding per frame, as a fused multiply-add
                inv = np.float32(1) / np.float32(k + 1)
                part = ((maps[a + k] - part).double() * float(inv) + part.double()).float()
            if mean is None:
                mean = part
            else:
                q = np.float32(b - a) / (np.float32(have) + np.float32(b - a))
                mean = ((part - mean).double() * float(q) + mean.double()).float()
            have = b
        return mean

    # the kernel's reciprocal is good to an ulp, so a frame's step may round the other way:
    # most pixels agree with the chain of the right number of chunks and no other way
    same = max(float((chain(c) == got).float().mean()) for c in range(2, 44))
    assert same >= 0.9
