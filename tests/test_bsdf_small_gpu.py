"""BSDF query batches on both sides of the small-batch line (one launch up to 2^18 queries, three above): a
query's result depends on its global index and inputs alone, so a large batch and the small batches it is cut
into agree bit for bit, wherever the border between the distributions falls."""
import numpy as np
import pytest

from open_rendering_framework_b200 import _native as nat

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = (1 << 18) + 1


def batch(wo, alpha, first, n_ggx_below):
    n = alpha.numel()
    wi, rest = torch.full((3, n), 7.0, device="cuda"), torch.full((3, n), 7.0, device="cuda")
    nat.call("pt_bsdf_queries", wo.data_ptr(), alpha.data_ptr(), n, first, n_ggx_below, 1.0 / 1.5, wi.data_ptr(), rest[0].data_ptr(),
             rest[1].data_ptr(), rest[2].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return torch.cat([wi, rest])


@pytest.mark.parametrize("border", [0, 1, 63, 64, 65, 1000, N - 1, N])
def test_small_batches_match_a_large_one(border):
    g = torch.Generator("cuda").manual_seed(border)
    z = 0.01 + 0.99 * torch.rand(N, generator=g, device="cuda")
    p = 6.2831853 * torch.rand(N, generator=g, device="cuda")
    r = torch.sqrt(1.0 - z * z)
    wo = torch.stack([r * torch.cos(p), r * torch.sin(p), z]).contiguous()
    alpha = 0.05 + 0.95 * torch.rand(N, generator=g, device="cuda")
    whole = batch(wo, alpha, 5, 5 + border).cpu().numpy().view(np.uint32)
    for lo, hi in ((0, 1), (0, 64), (1, 130), (900, 1100), (0, 1 << 18), (N - 66, N)):
        part = batch(wo[:, lo:hi].contiguous(), alpha[lo:hi].contiguous(), 5 + lo, 5 + border).cpu().numpy().view(np.uint32)
        assert np.array_equal(part, whole[:, lo:hi]), (lo, hi)
