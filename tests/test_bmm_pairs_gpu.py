"""Batched products on CTA pairs where the result is narrower than a pair's 256 columns, which the planner takes as well as any width:
partial tiles both ways, one and several k-blocks, both storage orders of B, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,m", [(2, 1), (3, 129), (40, 256), (41, 300)])
@pytest.mark.parametrize("n", [64, 72, 80, 136, 200, 255, 264])
@pytest.mark.parametrize("k", [32, 72, 200])
@pytest.mark.parametrize("dtype,tol", [(torch.float16, 5e-4), (torch.bfloat16, 4e-3)])  # one rounding of the result: 2^-11, 2^-8 at most
def test_narrow_pairs(b, m, n, k, dtype, tol):
    from aitemplate_b200 import kernels

    g = torch.Generator(device="cuda").manual_seed(b * 1000 + n)
    x = torch.rand((b, m, k), device="cuda", generator=g).sub_(0.5).to(dtype)
    w = torch.rand((b, n, k), device="cuda", generator=g).sub_(0.5).to(dtype)
    want = x.double() @ w.double().transpose(1, 2)
    results = [kernels.bmm_rcr(x, w, tile_n=512), kernels.bmm_rcr(x, w)]
    if n % 8 == 0:
        wt = w.transpose(1, 2).contiguous()
        results += [kernels.bmm_rrr(x, wt, tile_n=512), kernels.bmm_rrr(x, wt)]
    for y in results:
        assert y.shape == want.shape and float((y.double() - want).norm() / want.norm()) < tol
    assert kernels.device_status() == 0
