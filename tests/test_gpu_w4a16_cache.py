"""The operator's prepacked weights, when calls come from several streams and from graph captures: a weight is packed by the first
call that needs it, and every other call must find it packed."""
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu

MS = (1, 16, 200)  # the three kernels over the packed stream


@pytest.fixture(scope="module")
def npu():
    sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "ascend-python_b200"))
    try:
        import torch_npu
    finally:
        sys.path.pop(0)
    return torch_npu


def _case(npu, oracle, dev, M, seed, K=2048, N=2048):
    """A call with a weight of its own, and its result: from copies of the weight, so that nothing of it is packed yet."""
    args = [t.to(dev) for t in oracle.make_w4a16_inputs(M, K, N, seed=seed, group=128)]
    x, w, s, o = args
    call = lambda: npu.npu_weight_quant_batchmatmul(x, w, s, o, antiquant_group_size=128)  # noqa: E731
    want = npu.npu_weight_quant_batchmatmul(x, w.clone(), s.clone(), o.clone(), antiquant_group_size=128)
    torch.cuda.synchronize()
    return call, want


@pytest.mark.parametrize("M", MS)
def test_another_stream_waits_for_the_packing(npu, oracle, dev, M):
    call, want = _case(npu, oracle, dev, M, seed=100 + M)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        torch.cuda._sleep(50_000_000)  # some 25 ms before the packing
        a = call()
    with torch.cuda.stream(second):
        b = call()
    torch.cuda.synchronize()
    assert torch.equal(a, want) and torch.equal(b, want)


@pytest.mark.parametrize("M", MS)
def test_a_capture_waits_for_the_packing(npu, oracle, dev, M):
    """Packed on a stream outside the capture a moment ago: the graph may run at once, and on any stream."""
    call, want = _case(npu, oracle, dev, M, seed=200 + M)
    first, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        with torch.cuda.stream(first):  # not part of the capture
            torch.cuda._sleep(50_000_000)
            a = call()
        b = call()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(a, want) and torch.equal(b, want)


@pytest.mark.parametrize("M", MS)
def test_what_a_capture_packs_serves_that_capture(npu, oracle, dev, M):
    """Nothing is packed before the graph runs: an eager call packs for itself, two calls of the graph share what it packs."""
    call, want = _case(npu, oracle, dev, M, seed=400 + M)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph):
        a = call()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            b = call()
        torch.cuda.current_stream().wait_stream(side)
    eager = call()
    torch.cuda.synchronize()
    assert torch.equal(eager, want)
    for _ in range(2):
        a.zero_(), b.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(a, want) and torch.equal(b, want)
        assert torch.equal(call(), want)


def test_few_rows_without_memory_for_the_packing(npu, oracle, dev):
    """Three to eight rows pack the weight for the call; where there is no memory for that, the call needs none of it."""
    M, K, N = 5, 28672, 768
    x, w, s, o = oracle.make_w4a16_inputs(M, K, N, seed=11, group=K)
    y_ref = oracle.weight_quant_batchmatmul(x, w, s, o, antiquant_group_size=K)
    rms = ((y_ref ** 2).mean(axis=1, keepdims=True)) ** 0.5
    xd, wd, sd, od = (t.to(dev) for t in (x, w, s, o))
    odd = torch.empty(M * K + 1, dtype=x.dtype, device=dev)[1:].view(M, K)
    odd.copy_(xd)
    npu.npu_weight_quant_batchmatmul(odd, wd, sd, od, antiquant_group_size=K)  # the scratch of the stock layout's kernels
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(dev).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved(dev) + (6 << 20)) / total, dev)
        held = []
        with pytest.raises(torch.OutOfMemoryError):  # what is left, of the allocator's blocks as well
            while True:
                held.append(torch.empty(K * N // 2, dtype=torch.uint8, device=dev))
        y = npu.npu_weight_quant_batchmatmul(xd, wd, sd, od, antiquant_group_size=K).double().cpu().numpy()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, dev)
    assert (abs(y - y_ref) <= 2.0 ** -8 * abs(y_ref) + 2.0 ** -7 * rms).all()
