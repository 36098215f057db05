"""Outputs that TMA cannot describe, which the tile kernels write row by row from the staging boxes: N or a row stride
that is not a multiple of 8 (odd ones among them, where every second row starts off a 4-byte boundary), residuals of
such rows, and permuted outputs whose runs are not whole boxes.
Bound: one rounding of the fp32 result to the storage type, and fp32 sums in another order."""
import pytest
import torch

from oracle import reference_ops as oracle

pytestmark = pytest.mark.gpu


def _rand(shape, seed, dtype, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


def _close(got, want, dtype):
    got = got.float().cpu()
    assert got.shape == want.shape
    step = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert bool(((got - want).abs() <= 2e-3 + 2 * step * want.abs()).all()), float((got - want).abs().max())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tile_n", [0, 64, 128, 256, 512])
@pytest.mark.parametrize("m,n", [(1, 9), (31, 63), (290, 33), (290, 43), (129, 49), (129, 65), (300, 127), (257, 129), (260, 191), (300, 257), (513, 516), (640, 1022)])
def test_odd_columns(m, n, tile_n, dtype):
    from aitemplate_b200 import kernels

    x, w, b = _rand((m, 328), 1, dtype), _rand((n, 328), 2, dtype, 0.05), _rand((n,), 3, dtype)
    d0, d1 = _rand((m, n), 4, dtype), _rand((m, n), 5, dtype)
    c = [t.cuda() for t in (x, w, b, d0, d1)]
    for epilogue, extra in (("", 0), ("relu", 0), ("add", 1), ("mul_add", 2)):
        want = oracle.gemm_rcr(x, w, b, *(d0, d1)[:extra], epilogue=epilogue)
        _close(kernels.gemm_rcr(*c[:3 + extra], epilogue=epilogue, tile_n=tile_n, split_k=1), want, dtype)


@pytest.mark.parametrize("tile_n", [64, 128, 256, 512])
@pytest.mark.parametrize("offset,pitch", [(0, 301), (1, 301), (3, 302), (8, 304)])
def test_column_block_of_a_wider_buffer(offset, pitch, tile_n):
    """Only the block is written, whatever its alignment; what lies beside it stays."""
    from aitemplate_b200 import kernels

    m, n, dtype = 290, 264, torch.float16
    x, w = _rand((m, 320), 1, dtype), _rand((n, 320), 2, dtype, 0.05)
    wide = torch.full((m, pitch), 7.0, dtype=dtype, device="cuda")
    kernels.gemm_rcr(x.cuda(), w.cuda(), tile_n=tile_n, split_k=1, out=wide[:, offset:offset + n])
    _close(wide[:, offset:offset + n], oracle.gemm_rcr(x, w), dtype)
    assert bool((wide[:, :offset] == 7).all()) and bool((wide[:, offset + n:] == 7).all())


@pytest.mark.parametrize("tile_n", [0, 64, 128, 256, 512])
@pytest.mark.parametrize("batch,seq,heads,d", [(3, 211, 3, 64), (5, 33, 2, 40), (2, 130, 4, 12), (1, 7, 5, 8)])
def test_ragged_permutes(batch, seq, heads, d, tile_n):
    from aitemplate_b200 import kernels

    dtype, n = torch.float16, 3 * heads * d
    x, w, b = _rand((batch * seq, 256), 1, dtype), _rand((n, 256), 2, dtype, 0.05), _rand((n,), 3, dtype)
    got = kernels.gemm_rcr(x.cuda(), w.cuda(), b.cuda(), permute_shape=(seq, 3, heads), tile_n=tile_n, split_k=1)
    _close(got, oracle.gemm_rcr_bias_permute(x, w, b, (seq, 3, heads), "20314"), dtype)


@pytest.mark.parametrize("batch,m,n,k", [(3, 130, 77, 64), (5, 65, 132, 40), (2, 200, 515, 128)])
def test_batches(batch, m, n, k):
    from aitemplate_b200 import kernels

    dtype = torch.bfloat16
    a, b = _rand((batch, m, k), 1, dtype, 0.3), _rand((batch, n, k), 2, dtype, 0.3)
    _close(kernels.bmm_rcr(a.cuda(), b.cuda()), oracle.bmm_rcr(a, b), dtype)


@pytest.mark.parametrize("tile_n", [64, 128, 256, 512])
def test_several_tiles_per_cta(tile_n):
    """102 pair tiles on 74 pairs, 204 and more on 148 CTAs: the staging box and both accumulators serve a second tile."""
    from aitemplate_b200 import kernels

    dtype, m, n, k = torch.float16, 6500, 1021, 328
    x, w, b, d0 = _rand((m, k), 1, dtype), _rand((n, k), 2, dtype, 0.05), _rand((n,), 3, dtype), _rand((m, n), 4, dtype)
    c = [t.cuda() for t in (x, w, b, d0)]
    for epilogue, extra in (("relu", 0), ("add", 1)):
        want = oracle.gemm_rcr(x, w, b, *(d0,)[:extra], epilogue=epilogue)
        _close(kernels.gemm_rcr(*c[:3 + extra], epilogue=epilogue, tile_n=tile_n, split_k=1), want, dtype)
