"""The reference maximum of an attention row: taken from the first key block, raised when a block outgrows it. Scores that rise by little
(no raise), by just about the limit, by far more than an exponent holds, at every position of a block, and rows that start at
minus infinity. Bound: P and O are rounded to the storage type, everything else is fp32."""
import math

import pytest
import torch

from aitemplate_b200 import kernels

pytestmark = pytest.mark.gpu


def _check(q, k, v, causal=False):
    got = kernels.mem_eff_attention(q, k, v, causal=causal).double()
    assert kernels.device_status() == 0
    s = q.double() @ k.double().transpose(2, 3) / math.sqrt(q.shape[3])
    if causal:
        s = s.masked_fill(torch.ones(s.shape[2:], dtype=torch.bool, device="cuda").triu(1), -math.inf)
    want = (torch.softmax(s, -1) @ v.double()).transpose(1, 2)
    eps = torch.finfo(q.dtype).eps
    bound = 2 * eps * v.abs().max().double() + 2e-4 * v.abs().max().double()  # P and O rounded; exponentials to 7.5e-5
    assert bool(((got - want).abs() <= bound).all()), float((got - want).abs().max())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("d", [40, 64, 128])
@pytest.mark.parametrize("rise", [3.0, 9.0, 10.4, 11.0, 30.0, 90.0, 260.0])
def test_one_key_stands_out(rise, d, dtype):
    """Key 64 + i of head i scores `rise` above the rest (nats): every position of the second block, and of the third below it."""
    heads, sq, skv = 64, 40, 224
    gen = torch.Generator(device="cuda").manual_seed(int(rise * 10) + d)
    q = torch.randn(1, heads, sq, d, generator=gen, device="cuda") * 0.1
    k = torch.randn(1, heads, skv, d, generator=gen, device="cuda") * 0.1
    v = torch.randn(1, heads, skv, d, generator=gen, device="cuda")
    q[..., 0] = 4.0
    k[..., 0] = 0.0
    for i in range(heads):
        k[0, i, 64 + i, 0] = rise * math.sqrt(d) / 4
        k[0, i, 128 + (i * 7) % 64, 0] = 2 * rise * math.sqrt(d) / 4  # and raised once more
    _check(q.to(dtype), k.to(dtype), v.to(dtype))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("skv", [1, 26, 63, 65, 100, 190])
@pytest.mark.parametrize("rise", [3.0, 5.5, 5.6, 30.0, 260.0])
def test_last_block_has_a_mask(rise, skv, d, dtype):
    """The last block of keys is cut; its last key scores `rise` (nats; 2^8 is 5.55) above the rest in half of the heads."""
    heads, sq = 12, 300
    gen = torch.Generator(device="cuda").manual_seed(int(rise * 10) + d + skv)
    q = torch.randn(2, heads, sq, d, generator=gen, device="cuda") * 0.1
    k = torch.randn(2, heads, skv, d, generator=gen, device="cuda") * 0.1
    v = torch.randn(2, heads, skv, d, generator=gen, device="cuda")
    q[..., 0] = 4.0
    k[..., 0] = 0.0
    k[:, ::2, skv - 1, 0] = rise * math.sqrt(d) / 4
    _check(q.to(dtype), k.to(dtype), v.to(dtype))


@pytest.mark.parametrize("d", [64, 96])
def test_rising_blocks_causal(d):
    gen = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn(2, 3, 400, d, generator=gen, device="cuda") for _ in range(3))
    k = k * (1 + torch.arange(400, device="cuda")[:, None] / 40)  # later keys score ever higher
    _check(q.half(), k.half(), v.half(), causal=True)


@pytest.mark.parametrize("d", [64, 128])
def test_rows_that_start_at_minus_infinity(d):
    """The first block scores -inf everywhere, the next ones far below zero: what comes first must not be the reference."""
    gen = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn(1, 2, 130, d, generator=gen, device="cuda").half() for _ in range(3))
    q[..., 0] = 60000.0
    k[..., 0] = -0.02
    k[:, :, :64, 0] = -math.inf
    got = kernels.mem_eff_attention(q, k, v, scale=1.0).double()
    s = q.double() @ k.double().transpose(2, 3)
    want = (torch.softmax(s, -1) @ v.double()).transpose(1, 2)
    assert bool(((got - want).abs() <= 2e-2).all()), float((got - want).abs().max())


@pytest.mark.parametrize("d", [64, 128])
def test_not_a_number_stays_one(d):
    gen = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn(1, 1, 200, d, generator=gen, device="cuda").half() for _ in range(3))
    q[0, 0, 7] = math.nan
    got = kernels.mem_eff_attention(q, k, v)
    assert bool(got[0, 7].isnan().all()) and not bool(got[0, :7].isnan().any()) and not bool(got[0, 8:].isnan().any())
