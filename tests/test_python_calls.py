"""The shim's short-cut calls into the operator library: what sees or refuses a call through torch.ops sees and refuses it here."""
import sys
from pathlib import Path

import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

PKG_DIR = Path(__file__).resolve().parent.parent / "ascend-python_b200"


@pytest.fixture(scope="module")
def npu():
    sys.path.insert(0, str(PKG_DIR))
    try:
        import torch_npu
    finally:
        sys.path.pop(0)
    return torch_npu


def _calls(npu, dev):
    """(name, short-cut call, the same through torch.ops) for every operator that has one."""
    ops = torch.ops.npu
    x, g = torch.randn((4, 256), device=dev).bfloat16(), torch.rand(256, device=dev).bfloat16()
    q = torch.randint(-127, 128, (4, 256), dtype=torch.int8, device=dev)
    w = torch.randint(-127, 128, (256, 64), dtype=torch.int8, device=dev)
    scale, pt, bias = torch.rand(64, device=dev), torch.rand(4, device=dev), torch.rand(64, device=dev).bfloat16()
    w4 = torch.randint(-2**31, 2**31 - 1, (256, 8), device=dev).int()
    s4 = (torch.rand((2, 64), device=dev) * 0.01).bfloat16()
    bf = torch.bfloat16
    return [("npu_dynamic_quant", lambda: npu.npu_dynamic_quant(x), lambda: ops.npu_dynamic_quant(x)),
            ("npu_rms_norm", lambda: npu.npu_rms_norm(x, g, 1e-5), lambda: ops.npu_rms_norm(x, g, 1e-5)),
            ("npu_rms_norm_dynamic_quant", lambda: npu.npu_rms_norm_dynamic_quant(x, g), lambda: ops.npu_rms_norm_dynamic_quant(x, g)),
            ("npu_quant_matmul", lambda: npu.npu_quant_matmul(q, w, scale, pertoken_scale=pt, bias=bias, output_dtype=bf),
             lambda: ops.npu_quant_matmul(q, w, scale, pertoken_scale=pt, bias=bias, output_dtype=bf)),
            ("npu_quant_matmul", lambda: npu.npu_quant_matmul(q, w, scale, offset=scale), lambda: ops.npu_quant_matmul(q, w, scale, offset=scale)),
            ("npu_weight_quant_batchmatmul", lambda: npu.npu_weight_quant_batchmatmul(x, w4, s4, s4, antiquant_group_size=128),
             lambda: ops.npu_weight_quant_batchmatmul(x, w4, s4, s4, antiquant_group_size=128))]


def _error(f):
    with pytest.raises(Exception) as e:
        f()
    return type(e.value), str(e.value).splitlines()[0]


def test_errors_are_those_of_torch_ops(npu):
    for name, short, through_ops in _calls(npu, "cpu"):  # CPU tensors: no kernel registered
        assert _error(short) == _error(through_ops) and _error(short)[0] is NotImplementedError
    for bad in (3, None, "x", [torch.ones(2)]):
        assert _error(lambda: npu.npu_dynamic_quant(bad))[0] is _error(lambda: torch.ops.npu.npu_dynamic_quant(bad))[0]
    x = torch.ones((2, 8))
    assert _error(lambda: npu.npu_rms_norm(x, x[0], "eps"))[0] is _error(lambda: torch.ops.npu.npu_rms_norm(x, x[0], "eps"))[0]


def test_function_modes_subclasses_and_tracing_see_the_call(npu):
    seen = []

    class Sub(torch.Tensor):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return "sub"

    class Mode(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return "mode"

    x = torch.ones((2, 8))
    assert npu.npu_dynamic_quant(x.as_subclass(Sub)) == "sub"
    assert npu.npu_rms_norm(x, x[0].as_subclass(Sub)) == "sub"
    with Mode():
        assert npu.npu_dynamic_quant(x) == "mode"
    assert len(seen) == 3 and all("npu_" in s for s in seen)
    graph = torch.fx.symbolic_trace(lambda a, b: npu.npu_rms_norm(a, b, 1e-5)[0]).graph
    assert any("npu_rms_norm" in str(n.target) for n in graph.nodes)


def test_dispatch_modes_see_the_operator(npu):
    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if func.namespace != "npu":
                return func(*args, **(kwargs or {}))
            names.append(func.name().split("::")[1])
            return tuple(torch.zeros(1) for _ in func._schema.returns) if len(func._schema.returns) > 1 else torch.zeros(1)

    for name, short, _ in _calls(npu, "cpu"):
        names = []
        with Record():
            short()
        assert names == [name]


@pytest.mark.gpu
def test_results_are_those_of_torch_ops(npu, dev):
    for name, short, through_ops in _calls(npu, dev):
        a, b = short(), through_ops()
        for u, v in zip(a if isinstance(a, tuple) else (a,), b if isinstance(b, tuple) else (b,), strict=True):
            assert u.dtype == v.dtype and u.shape == v.shape and u.stride() == v.stride() and torch.equal(u, v), name
