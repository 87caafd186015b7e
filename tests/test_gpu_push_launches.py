"""A push's cost does not depend on the chunks its block is split into: the fused kernel
and one merge, however many records the block leaves (small frames split most).  The
records are merged in order, so the state of one push gives the bits of the same frames
in one call.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu
NAMES = ("AVG", "VAR", "TAC2")


def _block(T):
    x = np.random.default_rng(T).poisson(100, (T, 48, 60)).astype(np.float32)
    return torch.from_numpy(x).cuda()


def _nodes(fn):
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    n = C.c_size_t()
    rc = C.CDLL("libcuda.so.1").cuGraphGetNodes(C.c_void_p(g.raw_cuda_graph()), None, C.byref(n))
    assert rc == 0
    return n.value


@pytest.mark.parametrize("m", [2, 5])
@pytest.mark.parametrize("T", [1, 8, 16, 40])
def test_two_launches(m, T):
    x = _block(T)
    acc = nx.ESRRFAccumulator(48, 60, magnification=m, sensitivity=2)
    acc.push(x)
    assert _nodes(lambda: acc.push(x)) <= 2
    acc.frames = 0
    assert _nodes(lambda: acc.push(x)) <= 2


@pytest.mark.parametrize("m", [2, 5])
@pytest.mark.parametrize("T", [1, 8, 16, 40])
def test_one_push_is_one_call(m, T):
    x = _block(T)
    acc = nx.ESRRFAccumulator(48, 60, magnification=m, sensitivity=2)
    acc.push(x)
    got = acc.finalize(NAMES)
    ref = nx.eSRRF(x, magnification=m, sensitivity=2, temporal_correlation=NAMES)
    for g, r in zip(got, ref):
        assert np.array_equal(g, r.cpu().numpy(), equal_nan=True)
