"""Kernels whose set-up overlaps the end of the kernel before them (programmatic dependent launch): what it must not cost."""
import re
import sys
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent
PKG_DIR = ROOT / "ascend-python_b200"


@pytest.fixture(scope="module")
def npu():
    sys.path.insert(0, str(PKG_DIR))
    try:
        import torch_npu
    finally:
        sys.path.pop(0)
    return torch_npu


def _us(calls, n=40):
    """Device time of one round of `calls`, best of five measurements of n rounds queued behind a spinning kernel."""
    for f in calls:
        f()
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(4_000_000)
        a.record()
        for _ in range(n):
            for f in calls:
                f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / n)
    return best


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["quant", "rms", "rms_quant", "matmul"])
def test_odd_columns_back_to_back(npu, dev, op):
    """Kernels of a few long-running CTAs for every SM (rows and outputs of odd widths), repeated calls: no slower than with
    a kernel of one element in between, which keeps the launches from overlapping."""
    x = torch.randn((300, 16383), device=dev, dtype=torch.bfloat16)
    gamma = torch.rand(16383, device=dev).to(torch.bfloat16)
    a = torch.ones((600, 4096), dtype=torch.int8, device=dev)
    w = torch.ones((4096, 1001), dtype=torch.int8, device=dev)
    scale = torch.rand(1001, device=dev)
    one = torch.zeros(1, device=dev)
    call = {"quant": lambda: npu.npu_dynamic_quant(x), "rms": lambda: npu.npu_rms_norm(x, gamma),
            "rms_quant": lambda: npu.npu_rms_norm_dynamic_quant(x, gamma),
            "matmul": lambda: npu.npu_quant_matmul(a, w, scale, output_dtype=torch.bfloat16)}[op]
    together, apart = _us([call]), _us([call, lambda: one.add_(1)])
    assert together < apart, f"{together:.1f} us back to back, {apart:.1f} us apart"


def test_released_behind_the_tensor_memory_allocation():
    """A kernel that allocates tensor memory releases its successor behind that, in the allocating warp: released earlier,
    a CTA of another kernel could hold the columns and wait for this one.  Read from the sources."""
    checked = 0
    for f in sorted((PKG_DIR / "csrc").glob("*.[ci]*")):
        for body in re.split(r"\b__global__\b", re.sub(r"//[^\n]*", "", f.read_text()))[1:]:
            if "tmem_alloc" in body and "pdl_launch_dependents" in body:
                block = re.search(r"if \(warp == \w+\) \{\s*tmem_alloc[^{}]*\}", body)
                assert block and block.group(0).count("pdl_launch_dependents") == 1, f.name
                assert body.count("pdl_launch_dependents") == 1, f.name
                checked += 1
    assert checked >= 4
