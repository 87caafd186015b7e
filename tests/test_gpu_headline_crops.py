"""The benchmarked configurations against the FP64 oracle, at full size on the GPU and
on crops of the frames in the oracle (every output depends on input pixels at most 6
away, so crops agree up to 8 pixels from a side that is not the image's own).

* Large single eSRRF: 108 frames x 512 x 512 from the 400-emitter blinking generator,
  magnification 5, radius 1.5, sensitivity 2, VAR and TAC2, 100 frames per timepoint
  (one full timepoint and a short 8-frame tail); the macro-pixel correction against the
  oracle's of the whole uncorrected image.
* Parameter sweep: 16 frames x 256 x 256 at 150 emitters, magnification 4, radius
  {1, 1.5, 2, 2.5} x sensitivity {1, 2, 3, 4}, AVG.

Bar: max |got - ref| / (max(ref) - min(ref)) <= 1e-4, per crop and image.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx
from conftest import rel_err
from nanopyx_gb300.synthetic import blinking_stack
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu
TOL = 1e-4
SIDE, EDGE = 44, 8


def _crops(x, m):
    """(input crop, slices of the output image, slices of the crop's output): two corners
    and one place inside."""
    H, W = x.shape[1:]
    for r, c in ((0, 0), (H - SIDE, W - SIDE), (H // 2 - 5, W // 3)):
        lo = [EDGE if a else 0 for a in (r, c)]
        hi = [SIDE if a + SIDE == n else SIDE - EDGE for a, n in ((r, H), (c, W))]
        out = tuple(slice((a + l) * m, (a + h) * m) for a, l, h in zip((r, c), lo, hi))
        sub = tuple(slice(l * m, h * m) for l, h in zip(lo, hi))
        yield np.ascontiguousarray(x[:, r:r + SIDE, c:c + SIDE]), out, sub


def test_large_single_esrrf():
    T, H, W, m, r, s, fpt = 108, 512, 512, 5, 1.5, 2.0, 100
    x = blinking_stack(T, H, W, 400, seed=1)
    kw = dict(magnification=m, radius=r, sensitivity=s, frames_per_timepoint=fpt,
              temporal_correlation=("VAR", "TAC2"))
    plain = nx.eSRRF(x, macro_pixel_correction=False, **kw)
    for crop, out, sub in _crops(x, m):
        st = O.esrrf_st(crop, m, r, s)
        for name, got in zip(("VAR", "TAC2"), plain):
            for tp in range(2):
                ref = O.temporal_correlation(st[tp * fpt:(tp + 1) * fpt], name)
                assert rel_err(got[tp][out], ref[sub]) <= TOL, (name, tp, out)
    for got, raw in zip(nx.eSRRF(x, macro_pixel_correction=True, **kw), plain):
        assert rel_err(got, O.macro_pixel_correct(raw, m)) <= TOL


def test_parameter_sweep_grid():
    x = blinking_stack(16, 256, 256, 150, seed=2)
    sens, radii, m = [1, 2, 3, 4], [1.0, 1.5, 2.0, 2.5], 4
    grid = nx.esrrf_parameter_sweep(x, magnification=m, sensitivities=sens, radii=radii)
    assert grid.shape == (4, 4, 1024, 1024)
    for k, (crop, out, sub) in enumerate(_crops(x, m)):  # each crop a third of the grid
        for j, r in enumerate(radii):
            for i, s in enumerate(sens):
                if (i + j) % 3 != k:
                    continue
                ref = O.temporal_correlation(O.esrrf_st(crop, m, r, s), "AVG")
                assert rel_err(grid[i, j][out], ref[sub]) <= TOL, (s, r, out)
