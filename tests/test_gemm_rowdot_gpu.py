"""One to four rows of X against 256 to 1023 channels: the short form of the row-by-row kernel, over its three widths of a
lane's share (K = 256, up to 512, up to 1023), partly filled last vectors, row counts that leave warps and blocks without
rows, and every epilogue. Bound: one rounding of the fp32 result, fp32 sums in another order."""
import pytest
import torch

from oracle import reference_ops as oracle

pytestmark = pytest.mark.gpu


def _rand(shape, seed, dtype, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


def _check(m, n, k, dtype, epilogue=""):
    from aitemplate_b200 import kernels

    x, w, b = _rand((m, k), 1, dtype), _rand((n, k), 2, dtype, 0.05), _rand((n,), 3, dtype)
    extra = [_rand((m, n), 4 + i, dtype) for i in range(sum(e is not None for e in oracle.EPILOGUES[epilogue][1:3]))]
    got = kernels.gemm_rcr(*(t.cuda() for t in (x, w, b, *extra)), epilogue=epilogue).float().cpu()
    want = oracle.gemm_rcr(x, w, b, *extra, epilogue=epilogue)
    step = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert bool(((got - want).abs() <= 2e-3 + 2 * step * want.abs()).all()), float((got - want).abs().max())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("k", [256, 264, 512, 520, 1016])
@pytest.mark.parametrize("n", [64, 65, 593, 2377, 19001])
def test_sizes(m, n, k, dtype):
    _check(m, n, k, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", [(2, 56008, 320), (2, 56000, 256), (3, 28008, 264), (4, 28008, 520), (3, 10008, 448), (4, 28001, 640)])
def test_where_the_tile_kernels_take_over(m, n, k, dtype):
    _check(m, n, k, dtype, "add")


@pytest.mark.parametrize("epilogue", sorted(oracle.EPILOGUES))
def test_epilogues(epilogue):
    _check(3, 777, 328, torch.float16, epilogue)


def test_permuted_output():
    from aitemplate_b200 import kernels

    dtype, heads, d = torch.float16, 4, 24
    x, w, b = _rand((4, 256), 1, dtype), _rand((3 * heads * d, 256), 2, dtype, 0.05), _rand((3 * heads * d,), 3, dtype)
    got = kernels.gemm_rcr(x.cuda(), w.cuda(), b.cuda(), permute_shape=(2, 3, heads)).float().cpu()
    assert float((got - oracle.gemm_rcr_bias_permute(x, w, b, (2, 3, heads))).abs().max()) < 4e-3
