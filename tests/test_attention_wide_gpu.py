"""Heads of 65 to 128 channels on the tensor-core attention kernel: two CTAs per SM, K and V in two stages each, one Q
buffer and one O accumulator. What can go wrong there is the hand-over between a CTA's work items, so every case has
more items than the 296 CTAs of a full grid, or items of a single key block.
Bound: P is rounded to 11 significant bits and the output to fp16 (4e-3 absolute at unit-variance inputs)."""
import pytest
import torch

from oracle import reference_ops as oracle

pytestmark = pytest.mark.gpu


def _rand(shape, seed, dtype):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize(
    "b,h,sq,skv,d,causal,lengths",
    [
        (4, 40, 130, 64, 128, False, False),   # one key block per item, no masks
        (4, 40, 130, 33, 96, False, False),    # one ragged key block
        (3, 40, 300, 128, 72, False, False),   # two key blocks
        (3, 40, 300, 193, 128, False, False),  # an odd number of key blocks, ragged
        (3, 40, 300, 300, 128, True, False),
        (4, 40, 300, 200, 128, False, True),   # items of no, one and several key blocks
    ],
)
def test_items_follow_one_another(b, h, sq, skv, d, causal, lengths, dtype):
    from aitemplate_b200 import kernels

    q, k, v = (_rand((b, h, s, d), i, dtype) for i, s in enumerate((sq, skv, skv)))
    lens = torch.tensor([skv, 1, 0, 65][:b], dtype=torch.int32) if lengths else None
    got = kernels.mem_eff_attention(q.cuda(), k.cuda(), v.cuda(), causal=causal,
                                    lengths_kv=None if lens is None else lens.cuda()).float().cpu()
    want = oracle.mem_eff_attention(q, k, v, causal=causal, lengths_kv=lens)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    err = (got - want).nan_to_num(0.0).abs()
    bound = 4e-3 if dtype == torch.float16 else 3.2e-2  # three bits fewer in bfloat16
    assert float(err.max()) < bound, float(err.max())


@pytest.mark.parametrize("causal", [False, True])
def test_packed_sequences(causal):
    from aitemplate_b200 import kernels

    lens, h, d = [1, 64, 129, 640, 0, 200, 383], 24, 128
    starts = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    qkv = _rand((sum(lens), 3, h, d), 7, torch.float16)
    got = kernels.flash_attention(qkv.cuda(), starts.cuda(), max(lens), causal=causal).float().cpu()
    for lo, hi in zip(starts[:-1].tolist(), starts[1:].tolist()):
        if hi > lo:
            q, k, v = (t.permute(1, 0, 2)[None] for t in qkv[lo:hi].unbind(1))
            want = oracle.mem_eff_attention(q, k, v, causal=causal)[0]
            assert float((got[lo:hi] - want).abs().max()) < 4e-3


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize(
    "b,h,sq,skv,d,causal,lengths",
    [
        (1, 1, 1, 40, 128, False, False),     # one row, one ragged key block
        (2, 8, 1, 1000, 72, False, False),    # a decode step: the ring of four stages goes round several times
        (4, 37, 1, 320, 96, False, False),    # an item for every SM (148), no masks, five key blocks
        (1, 9, 129, 576, 128, True, False),
        (4, 5, 200, 700, 128, False, True),   # items of no, one and several key blocks
    ],
)
def test_an_item_per_sm(b, h, sq, skv, d, causal, lengths, dtype):
    """At most one work item per SM: the form with four K / V stages and one CTA per SM."""
    test_items_follow_one_another(b, h, sq, skv, d, causal, lengths, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [72, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,h", [(3, 40), (1, 9)])  # more items than CTAs; an item per SM
def test_row_maxima_that_outgrow_their_reference(b, h, causal, d, dtype):
    """Keys four times as large from block to block: the scores' spread is 1, 4, 16, 64, 256, so nearly every row's maximum
    outgrows its reference by more than 2^8 at every block, and O, the only accumulator, is rescaled in TMEM beside a ring of
    two stages. Bound: outputs reach |v| = 4.5; P and the output are each rounded once (2^-12 and 2^-9 relative), and a score
    of 256 carries fp32 sums' 1e-6 of its terms, 3e-4, in both the kernel and the oracle: 4.5 (2^-11 + 6e-4) and 4.5 (2^-8 +
    6e-4), doubled for the row sum's rounded terms."""
    from aitemplate_b200 import kernels

    s = 300
    q, k, v = (_rand((b, h, s, d), i, dtype) for i in range(3))
    k = (k.float() * 4.0 ** (torch.arange(s) // 64)[:, None]).to(dtype)
    got = kernels.mem_eff_attention(q.cuda(), k.cuda(), v.cuda(), causal=causal).float().cpu()
    err = (got - oracle.mem_eff_attention(q, k, v, causal=causal)).abs().max()
    assert float(err) < (1e-2 if dtype == torch.float16 else 4e-2), float(err)
