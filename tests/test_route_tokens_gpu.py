"""The router's kernel of several tokens a CTA against the one of a token a CTA, bit for bit: counts of tokens that fill the last CTA and that do not, on both
sides of where it takes over, up to eight experts, rows that end inside a round of the threads."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (rows of less than 2,048 channels go so from two tokens an SM on; below that another kernel adds in another order)
@pytest.mark.parametrize("T,E,W", [(T, E, W) for T in (149, 150, 297, 299, 300, 301) for E, W in ((8, 2048), (3, 2056), (1, 4096), (8, 4104), (5, 512))
                                   if W >= 2048 or T > 296])
def test_tokens_of_a_cta(T, E, W):
    from forge_b200 import kernels
    g = torch.Generator().manual_seed(T + W)
    x, w = torch.randn(T, W, generator=g).to(torch.bfloat16).cuda(), (torch.randn(E, W, generator=g) * W ** -0.5).cuda()
    corr = torch.randn(E, generator=g).cuda()
    for opts in ({}, {"softmax": True, "renorm": True}, {"correction": corr, "factor": 2.5}):
        idx, wts = kernels.moe_route(x, w, min(2, E), **opts)
        for lo in range(0, T, 100):
            i, v = kernels.moe_route(x[lo:lo + 100].contiguous(), w, min(2, E), **opts)
            assert torch.equal(idx[lo:lo + 100], i) and torch.equal(wts[lo:lo + 100], v)
