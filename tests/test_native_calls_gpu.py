"""The native host path of the eager calls against the Python code behind it: the same results bit for bit, and whatever is not plain
(or is refused) takes the Python code, which answers as if there were no native path."""
import pytest
import torch

from aitemplate_b200 import _lib
from aitemplate_b200 import kernels as K

pytestmark = pytest.mark.gpu


class _Absent:
    """Answers None to every call, as the native module does to a call that is not plain."""

    def __getattr__(self, name):
        return lambda *args: None


class _Recorder:
    """The native module, noting of every call whether it was served."""

    def __init__(self):
        self.module, self.served = _lib.load_calls(), []

    def __getattr__(self, name):
        function = getattr(self.module, name)

        def call(*args):
            y = function(*args)
            self.served.append(y is not None)
            return y

        return call


def _both(monkeypatch, call, served=None):
    """call() as it is and without the native module; `served`: whether the native module has to have served it."""
    def run():
        try:
            y = call()
        except Exception as e:  # noqa: BLE001
            return type(e), str(e)
        return y

    with monkeypatch.context() as m:
        recorder = _Recorder()
        m.setattr(K, "_calls", recorder)
        native = run()
        assert recorder.served == ([served] if served is not None else recorder.served)
    with monkeypatch.context() as m:
        m.setattr(K, "_calls", _Absent())
        python = run()
    torch.cuda.synchronize()
    return native, python


def _same(a, b):
    if torch.is_tensor(a):
        return torch.is_tensor(b) and a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)
    if isinstance(a, list):
        return isinstance(b, list) and len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    return a == b


def _t(*shape, dtype=torch.float16, seed=0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(dtype)


PLAIN = {
    "gemm": lambda: K.gemm_rcr(_t(33, 72), _t(40, 72, seed=1), _t(40, seed=2)),
    "gemm_3d_bf16": lambda: K.gemm_rcr(_t(2, 3, 264, dtype=torch.bfloat16), _t(136, 264, dtype=torch.bfloat16, seed=1), epilogue="gelu"),
    "gemm_one_row": lambda: K.gemm_rcr(_t(1, 2048), _t(513, 2048, seed=1), _t(513, seed=2), _t(1, 513, seed=3), epilogue="add"),
    "gemm_two_residuals": lambda: K.gemm_rcr(_t(70, 128), _t(64, 128, seed=1), _t(64, seed=2), _t(70, 64, seed=3), _t(70, 64, seed=4),
                                             epilogue="mul_add", alpha=0.5, tile_n=64, split_k=1),
    "gemm_split_k": lambda: K.gemm_rcr(_t(100, 4096), _t(64, 4096, seed=1), split_k=4),
    "gemm_narrow_deep": lambda: K.gemm_rcr(_t(100, 4096), _t(64, 4096, seed=1)),
    "gemm_odd_k": lambda: K.gemm_rcr(_t(20, 33), _t(9, 33, seed=1)),
    "gemm_unaligned": lambda: K.gemm_rcr(_t(1 + 64 * 64)[1:].view(64, 64), _t(128, 64, seed=1)),
    "gemm_parameter": lambda: K.gemm_rcr(_t(8, 64), torch.nn.Parameter(_t(16, 64, seed=1)), torch.nn.Parameter(_t(16, seed=2))),
    "gemm_no_rows": lambda: K.gemm_rcr(_t(0, 64), _t(16, 64, seed=1)),
    "bmm_rcr": lambda: K.bmm_rcr(_t(3, 17, 40), _t(3, 24, 40, seed=1), alpha=2),
    "bmm_rcr_broadcast": lambda: K.bmm_rcr(_t(17, 40), _t(3, 24, 40, seed=1)),
    "bmm_rrr": lambda: K.bmm_rrr(_t(3, 17, 40), _t(1, 40, 24, seed=1)),
    "attention": lambda: K.mem_eff_attention(_t(2, 3, 33, 40), _t(2, 3, 70, 40, seed=1), _t(2, 3, 70, 64, seed=2), causal=True, scale=0.3),
    "attention_lengths": lambda: K.mem_eff_attention(_t(2, 3, 33, 40), _t(2, 3, 70, 40, seed=1), _t(2, 3, 70, 40, seed=2),
                                                     lengths_kv=torch.tensor([70, 5], dtype=torch.int32, device="cuda")),
    "flash": lambda: K.flash_attention(_t(50, 3, 2, 64), torch.tensor([0, 20, 50], dtype=torch.int32, device="cuda"), 30, causal=True),
    "layernorm": lambda: K.layernorm(_t(4, 5, 96), _t(96, seed=1), None, eps=1e-3),
    "layernorm_two_dims": lambda: K.layernorm(_t(4, 5, 16), _t(80, seed=1), _t(80, seed=2), normalized_ndim=2),
    "softmax": lambda: K.softmax(_t(4, 5, 77)),
    "softmax_inner": lambda: K.softmax(_t(4, 5, 77), dim=-2),
    "concatenate": lambda: K.concatenate([_t(2, 3, 4), _t(2, 1, 4, seed=1)], dim=-2),
    "split": lambda: K.split(_t(2, 7, 4), 3, dim=1),
    "split_sections": lambda: K.split(_t(2, 7, 4), [2, 5], dim=1),
    "permute": lambda: K.permute(_t(2, 3, 4), (0, -1, 1)),
    "on_a_side_stream": lambda: _on_side_stream(lambda: K.softmax(_t(64, 64))),
}
# plain, but left to the Python code: scratch for split K, sections, no rows
LONG_WAY = {"gemm_split_k", "gemm_narrow_deep", "gemm_no_rows", "split_sections"}
REFUSED = {
    "strided": lambda: K.gemm_rcr(_t(72, 33).t(), _t(40, 72)),
    "host": lambda: K.softmax(torch.zeros(3, 4)),
    "k_differs": lambda: K.gemm_rcr(_t(8, 64), _t(16, 72)),
    "dtype": lambda: K.layernorm(_t(4, 64, dtype=torch.float32), None, None),
    "epilogue": lambda: K.gemm_rcr(_t(8, 64), _t(16, 64), epilogue="none_such"),
    "tile_n": lambda: K.gemm_rcr(_t(8, 64), _t(16, 64), tile_n=96),
    "bmm_batches": lambda: K.bmm_rcr(_t(2, 8, 64), _t(3, 8, 64)),
    "lengths_dtype": lambda: K.mem_eff_attention(_t(1, 1, 8, 64), _t(1, 1, 8, 64), _t(1, 1, 8, 64), lengths_kv=torch.zeros(1, device="cuda")),
    "head_size": lambda: K.flash_attention(_t(8, 3, 2, 60), torch.tensor([0, 8], dtype=torch.int32, device="cuda"), 8),
    "concatenate_shapes": lambda: K.concatenate([_t(2, 3), _t(3, 3)], dim=1),
    "permute_dims": lambda: K.permute(_t(2, 3), (0, 0)),
}


def _on_side_stream(call):
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        y = call()
    torch.cuda.current_stream().wait_stream(s)
    return y


@pytest.mark.parametrize("name", PLAIN)
def test_plain_calls(name, monkeypatch):
    native, python = _both(monkeypatch, PLAIN[name], served=name not in LONG_WAY)
    assert _same(native, python), (native, python)


@pytest.mark.parametrize("name", REFUSED)
def test_refused_calls(name, monkeypatch):
    native, python = _both(monkeypatch, REFUSED[name])
    assert isinstance(native, tuple) and native == python


def test_concatenate_of_a_list_that_changes_during_the_call():
    """Allocating the output may run Python code (a dispatch mode), and other threads run while the kernel is launched: the tensors
    of the call are the ones it was given."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Clears(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            parts.clear()
            return func(*args, **(kwargs or {}))

    want = torch.cat([_t(5, 3, 16), _t(5, 4, 16, seed=1)], dim=1)
    parts = [_t(5, 3, 16), _t(5, 4, 16, seed=1)]
    with Clears():
        y = K.concatenate(parts, dim=1)
    assert not parts and torch.equal(y, want)


def test_run_with_tensors(tmp_path, monkeypatch):
    from aitemplate_b200.compiler import compile_model
    from aitemplate_b200.testing import detect_target, workloads

    x, params = workloads.bert_layer_inputs(2, 40)
    _, y = workloads.build_bert_layer(2, 40)
    model = compile_model(y, detect_target(), str(tmp_path), "native_calls")
    model.set_many_constants_with_tensors({n: params[k].cuda() for n, k in workloads.BERT_PARAM_NAMES.items()})
    x = x.cuda()
    outs = [torch.empty((2, 40, 768), dtype=torch.float16, device="cuda") for _ in range(3)]
    recorder = _Recorder()
    monkeypatch.setattr(_lib, "_calls", recorder)
    a = model.run_with_tensors({"hidden_states": x}, {"output_0": outs[0]})
    b = model.run_with_tensors([x], [outs[1]], graph_mode=True)  # lists take the Python code
    wider = torch.empty((2, 41, 768), dtype=torch.float16, device="cuda")  # more room than the run needs
    c = model.run_with_tensors({"hidden_states": x}, {"output_0": wider}, sync=False, stream_ptr=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert recorder.served == [True, False, True]
    assert list(a) == list(b) == list(c) == ["output_0"]
    assert a["output_0"].data_ptr() == outs[0].data_ptr() and c["output_0"].shape == (2, 40, 768)
    assert torch.equal(a["output_0"], b["output_0"]) and torch.equal(a["output_0"], c["output_0"])
    with pytest.raises(ValueError, match="Got unexpected input"):
        model.run_with_tensors({"other": x}, {"output_0": outs[0]})
    with pytest.raises(ValueError, match="contiguous and on GPU"):
        model.run_with_tensors({"hidden_states": x.cpu()}, {"output_0": outs[0]})
    with pytest.raises(RuntimeError, match="Error in function: AITemplateModelContainerRun"):
        model.run_with_tensors({"hidden_states": x.float()}, {"output_0": outs[0]})
    model.close()
    with pytest.raises(RuntimeError, match="closed"):
        model.run_with_tensors({"hidden_states": x}, {"output_0": outs[0]})


def test_run_with_tensors_returns_the_outputs_in_the_order_they_were_given(tmp_path):
    from aitemplate_b200.compiler import compile_model, ops
    from aitemplate_b200.frontend import Tensor
    from aitemplate_b200.testing import detect_target

    x = Tensor([4, 64], name="x", is_input=True)
    outputs = []
    for name, dim in (("first", 0), ("second", 1), ("third", 1)):
        y = ops.softmax()(x, 1) if name == "first" else ops.concatenate()([x, x], dim)
        y._attrs["name"], y._attrs["is_output"] = name, True
        outputs.append(y)
    model = compile_model(outputs, detect_target(), str(tmp_path), "ordered")
    given = _t(4, 64)
    shapes = {"first": (4, 64), "second": (4, 128), "third": (4, 128)}
    for order in (["third", "first", "second"], ["second", "third", "first"], ["first", "second", "third"]):
        outs = {name: torch.empty(shapes[name], dtype=torch.float16, device="cuda") for name in order}
        got = model.run_with_tensors({"x": given}, outs)
        assert list(got) == order
        assert all(got[name].data_ptr() == outs[name].data_ptr() for name in order)
        assert torch.equal(got["first"], K.softmax(given)) and torch.equal(got["third"], torch.cat([given, given], 1))
    model.close()
