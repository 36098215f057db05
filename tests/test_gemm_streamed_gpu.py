"""Batched products whose result is streamed to DRAM behind one k-block per tile: they run on 128-wide tiles with a shortened
operand ring. Ragged row and column tiles, K below and at the block, the batch just above the size from which the rule holds."""
import pytest
import torch

from aitemplate_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("m, n, k", [(512, 512, 64), (300, 344, 64), (129, 136, 64), (512, 256, 32), (321, 520, 8)])
def test_streamed_bmm(m, n, k, dtype):
    batch = (96 << 20) // (2 * m * n) + 2
    gen = torch.Generator(device="cuda").manual_seed(3)
    a = (torch.rand(batch, m, k, generator=gen, device="cuda") * 2 - 1).to(dtype)
    b = (torch.rand(batch, n, k, generator=gen, device="cuda") * 2 - 1).to(dtype)
    got = kernels.bmm_rcr(a, b)
    assert kernels.device_status() == 0
    eps = torch.finfo(dtype).eps
    for i in sorted({0, 1, batch // 2, batch - 2, batch - 1}):
        want = a[i].double() @ b[i].double().t()
        # fp32 sums of k products of values below one, then one rounding to the output type
        bound = eps / 2 * want.abs() + k * k * 2.0 ** -24 + 1e-7
        assert bool(((got[i].double() - want).abs() <= bound).all()), i
    if k == 64:  # and bit for bit what the other tile widths give
        assert torch.equal(got, kernels.bmm_rcr(a, b, tile_n=256))
