"""Kernels that become resident before the one ahead of them has ended read what it wrote, whatever the pair: every operator
follows every other in one chain, which has to give the same bits as the chain with a synchronisation after each step."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(x, w, wide, narrow, step):
    """Every intermediate of a chain over [m, n]; buffers that are freed on the way are taken again by later steps."""
    from aitemplate_b200 import kernels as k

    m, n = x.shape
    ones, zeros = torch.ones(n, dtype=x.dtype, device="cuda"), torch.zeros(n, dtype=x.dtype, device="cuda")
    heads = n // 64

    def gemm(t):
        return k.gemm_rcr(t, w, None, t, epilogue="add")

    def mlp(t):
        return k.gemm_rcr(k.gemm_rcr(t, wide, None, None, epilogue="fast_gelu"), narrow, None, None)

    def layernorm(t):
        return k.layernorm(t, ones, zeros)

    def softmax(t):
        return k.softmax(t, 1)

    def transpose(t):
        return k.permute(k.permute(t, (1, 0)), (1, 0))

    def heads_first(t):
        return k.permute(k.permute(t.view(m, heads, 64), (1, 0, 2)), (1, 0, 2)).view(m, n)

    def concat(t):
        return k.concatenate(k.split(t, [n // 2, n - n // 2], 1), 1)

    def attention(t):
        q = t.view(1, m, heads, 64).transpose(1, 2).contiguous()
        return k.mem_eff_attention(q, q, q, False, 0.125).reshape(m, n)

    def product(t):
        a = t.view(m, heads, 64).transpose(0, 1).contiguous()
        return k.bmm_rcr(a, w.view(-1)[: heads * 64 * 64].view(heads, 64, 64)).transpose(0, 1).reshape(m, n)

    ops = [gemm, mlp, layernorm, softmax, transpose, heads_first, concat, attention, product]
    for i in range(len(ops)):
        for j in range(len(ops)):
            for op in (ops[i], ops[j]):
                x = op(x)
                step()
        x = layernorm(x)
        step()
    return x


@pytest.mark.parametrize("m", [1, 7, 64, 130, 1055, 5000])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_chain_equals_synchronised_chain(m, dtype):
    from aitemplate_b200 import kernels

    n = 768 if m < 5000 else 320
    g = torch.Generator().manual_seed(m)
    x, w, wide, narrow = ((torch.randn(s, generator=g) * c).to(dtype).cuda() for s, c in (((m, n), 1.0), ((n, n), 0.02), ((4 * n, n), 0.02), ((n, 4 * n), 0.02)))
    want = _chain(x, w, wide, narrow, torch.cuda.synchronize)
    assert torch.isfinite(want.float()).all()
    for _ in range(3):
        assert torch.equal(_chain(x, w, wide, narrow, lambda: None), want)
    # on two streams at once, and captured
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = []
    for s in streams:
        with torch.cuda.stream(s):
            got.append(_chain(x, w, wide, narrow, lambda: None))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want) for y in got)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = _chain(x, w, wide, narrow, lambda: None)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    assert kernels.device_status() == 0
