"""b200ait_gemm_rcr_scratch_bytes against the launches themselves: offered more scratch than it can use, a gemm_rcr runs as two
kernels (partial sums, then their sum) exactly where the query says that it takes scratch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 4, 5, 63, 64, 130, 2048, 2049, 4300])
def test_scratch_is_reported_where_a_launch_splits(m):
    from aitemplate_b200 import _lib, kernels

    lib, seen = _lib.load(), set()
    room = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    for n in (24, 63, 64, 96, 127, 128, 136, 256, 1000):
        for k in (64, 2040, 2048, 2050, 8192, 24576):
            x = torch.rand((m, k), device="cuda").sub_(0.5).half()
            w = torch.rand((n, k), device="cuda").sub_(0.5).mul_(0.1).half()
            y = torch.empty((m, n), dtype=torch.float16, device="cuda")
            for tile_n, split_k in ((0, 0), (64, 0), (0, 1), (0, 3), (128, 2)):
                before = _lib.kernel_launch_count()
                code = lib.b200ait_gemm_rcr(x.data_ptr(), w.data_ptr(), None, None, None, y.data_ptr(), 1, m, n, k, k, k, n, n, 0, 0, 0, 0,
                                            0, 1, 1.0, 0, 1, 1, 1, tile_n, room.data_ptr(), room.numel(), split_k, kernels._stream())
                assert code == 0, _lib.last_error()
                need = kernels._scratch_bytes(0, m, n, k, tile_n, split_k)
                assert need <= room.numel()
                assert (_lib.kernel_launch_count() - before == 2) == (need > 0), (n, k, tile_n, split_k, need)
                seen.add((tile_n, split_k, need > 0))
            want = x.double() @ w.double().T  # of the last of them, in K / 64 blocks of fp32 sums
            assert float((y.double() - want).norm() / want.norm()) < 5e-4, (n, k)
    assert {(0, 3, True), (0, 1, False)} <= seen
    torch.cuda.synchronize()
    assert kernels.device_status() == 0
