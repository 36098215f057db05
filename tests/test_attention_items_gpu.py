"""Attention over more work items than a grid of two CTAs per SM holds (296), in the forms in which the items reach the
CTAs: fixed shares, and a CTA per item, where a tile past the end of its sequence ends its CTA at once.
Bound: P is rounded to 11 significant bits (8 in bfloat16) and the output to the storage type, at unit-variance inputs."""
import pytest
import torch

from oracle import reference_ops as oracle

pytestmark = pytest.mark.gpu

_BOUND = {torch.float16: 4e-3, torch.bfloat16: 3.2e-2}


def _rand(shape, seed, dtype):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


def _check_packed(got, qkv, lens, causal):
    """One sequence and head at a time: a whole score matrix of the longest ones does not fit the host's caches."""
    row = 0
    for n in lens:
        for h in range(qkv.shape[2] if n else 0):
            q, k, v = (t[None, None, :, h] for t in qkv[row:row + n].unbind(1))
            err = (got[row:row + n, h] - oracle.mem_eff_attention(q, k, v, causal=causal)[0, :, 0]).abs().max()
            assert float(err) < _BOUND[qkv.dtype], (n, h, float(err))
        row += n


@pytest.mark.parametrize("dtype,d", [(torch.float16, 40), (torch.float16, 64), (torch.bfloat16, 128)])
@pytest.mark.parametrize("causal,lens,heads", [(True, [4096, 0, 3900, 1300, 2500], 3), (False, [4700, 1, 3000, 4608, 3200], 2)])
def test_packed_sequences_with_a_cta_per_item(causal, lens, heads, dtype, d):
    """Empty sequences and tiles among them; a bound that is too high changes the schedule and no bit of the result."""
    from aitemplate_b200 import kernels

    starts = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    qkv = _rand((sum(lens), 3, heads, d), 7, dtype)
    x = qkv.cuda()
    got = kernels.flash_attention(x, starts, max(lens), causal=causal)
    assert torch.equal(got, kernels.flash_attention(x, starts, 20000, causal=causal))
    _check_packed(got.float().cpu(), qkv, lens, causal)


@pytest.mark.parametrize("dtype,d", [(torch.float16, 64), (torch.bfloat16, 128), (torch.float16, 72)])
@pytest.mark.parametrize("heads,s", [(16, 2560), (16, 2497), (32, 2048)])  # a CTA per item; fixed shares
def test_causal_sequences_of_one_length(heads, s, dtype, d):
    from aitemplate_b200 import kernels

    q, k, v = (_rand((1, heads, s, d), i, dtype) for i in range(3))
    got = kernels.mem_eff_attention(q.cuda(), k.cuda(), v.cuda(), causal=True).float().cpu()
    for h in range(heads):
        want = oracle.mem_eff_attention(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1], causal=True)
        assert float((got[:, :, h:h + 1] - want).abs().max()) < _BOUND[dtype]


@pytest.mark.parametrize("dtype,d", [(torch.float16, 64), (torch.float16, 128), (torch.bfloat16, 96)])
@pytest.mark.parametrize("causal", [False, True])
def test_padded_lengths(causal, dtype, d):
    """Lengths on the device, 384 items of 4096 keys: whole, short and empty ones."""
    from aitemplate_b200 import kernels

    b, heads, s = 4, 3, 4096
    q, k, v = (_rand((b, heads, s, d), i, dtype) for i in range(3))
    kv, rows = torch.tensor([4096, 0, 70, 2000], dtype=torch.int32), torch.tensor([1000, 4096, 0, 3333], dtype=torch.int32)
    out = torch.full((b, s, heads, d), 7.0, dtype=dtype, device="cuda")
    kernels.mem_eff_attention(q.cuda(), k.cuda(), v.cuda(), causal=causal, lengths_kv=kv.cuda(), lengths_q=rows.cuda(), out=out)
    got = out.float().cpu()
    for i in range(b):
        n = int(rows[i])
        assert bool((got[i, n:] == 7).all())  # rows past lengths_q are not written
        if int(kv[i]) == 0:
            assert bool(torch.isnan(got[i, :n]).all())
            continue
        for h in range(heads):
            one = [t[i:i + 1, h:h + 1] for t in (q, k, v)]
            want = oracle.mem_eff_attention(*one, causal=causal, lengths_kv=kv[i:i + 1])[0, :n]
            assert n == 0 or float((got[i, :n, h:h + 1] - want).abs().max()) < _BOUND[dtype]


@pytest.mark.parametrize("s", [3100, 4096])
def test_equal_items_of_narrow_heads(s):
    """Rows of 80 bytes, a CTA per item: 384 and 375 items, with and without a last block to mask."""
    from aitemplate_b200 import kernels

    heads, d = (12, 40) if s == 4096 else (15, 40)
    q, k, v = (_rand((1, heads, s, d), i, torch.float16) for i in range(3))
    got = kernels.mem_eff_attention(q.cuda(), k.cuda(), v.cuda()).float().cpu()
    for h in range(heads):
        want = oracle.mem_eff_attention(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1])
        assert float((got[:, :, h:h + 1] - want).abs().max()) < _BOUND[torch.float16]
