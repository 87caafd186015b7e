"""The error maps' device memory: the blur-width search's buffers are given back before
the final blur and its maps are made, so the peak is the larger of the two and not their
sum (64 KB for the allocator's rounding and the small results).
"""
import pytest
import torch

from nanopyx_gb300 import _native as N, scoring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 5])
def test_peak(B):
    H = W = 256
    g = torch.Generator().manual_seed(B)
    ref = (torch.rand((128, 128), generator=g) * 100 + 50).cuda()
    srs = (torch.rand((B, H, W), generator=g) * 100 + 50).cuda()
    ref_int = scoring._reference_interp(ref, 2)
    L = N.lib()
    maps = B * H * W * 4
    search = L.nx_blur_moments_workspace_bytes(H, W, B)
    final = maps + max(L.nx_gaussian_blur_batch_workspace_bytes(H, W, B),
                       L.nx_moment_sums_workspace_bytes(B), maps + maps)
    scoring.error_maps(ref, srs, ref_int=ref_int)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    scoring.error_maps(ref, srs, ref_int=ref_int)
    assert torch.cuda.max_memory_allocated() - before <= max(search, final) + 65536
