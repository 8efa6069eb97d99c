"""Split tiles of GEMMs that run at once: each stream, and each graph, exchanges its partial sums through memory of its own."""
import ctypes
import gc
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _count():
    from state_space_models_neuron_b200.ops import native
    out = (ctypes.c_int * 3)()
    native.lib().ssm_gemm_scratch_count(out)
    return list(out)


def _problems(n, M=256, N=512, K=8192):
    from state_space_models_neuron_b200.utils import debug
    assert debug.gemm_plan(M, N, K)["split"] > 1
    gen = torch.Generator(device="cuda").manual_seed(3)
    return [tuple(torch.randn(r, K, device="cuda", generator=gen).bfloat16() for r in (M, N)) for _ in range(n)]


def test_streams_at_once():
    from state_space_models_neuron_b200.ops import cuda_ops
    given = _problems(3)
    want = [cuda_ops.gemm(a, b).clone() for a, b in given]
    streams = [torch.cuda.Stream() for _ in given]
    before = _count()[0]
    out = [[] for _ in given]
    torch.cuda.synchronize()
    for _ in range(40):
        for s, (a, b), o in zip(streams, given, out):
            with torch.cuda.stream(s):
                o.append(cuda_ops.gemm(a, b))
    torch.cuda.synchronize()
    cuda_ops.check_status()
    assert all(torch.equal(y, w) for o, w in zip(out, want) for y in o)
    assert before < _count()[0] <= 16


def test_more_streams_than_are_kept():
    from state_space_models_neuron_b200.ops import cuda_ops
    (a, b), = _problems(1)
    want = cuda_ops.gemm(a, b).clone()
    for _ in range(2):
        for s in [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(10)]:
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                y = cuda_ops.gemm(a, b)
            s.synchronize()
            assert torch.equal(y, want)
    assert _count()[0] == 16


def test_graphs_at_once_give_theirs_back():
    from state_space_models_neuron_b200.ops import cuda_ops
    given = _problems(3)
    want = [cuda_ops.gemm(a, b).clone() for a, b in given]
    start = _count()
    graphs, out = [], []
    for a, b in given:                                     # all of them captured on the same stream
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            out.append([cuda_ops.gemm(a, b) for _ in range(4)])
    assert _count()[1] == start[1] + 3
    streams = [torch.cuda.Stream() for _ in given]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, g, o in zip(streams, graphs, out):
            with torch.cuda.stream(s):
                for y in o:
                    y.zero_()
                g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for o, w in zip(out, want) for y in o)
    cuda_ops.check_status()
    del graphs, g
    gc.collect()
    torch.cuda.synchronize()
    limit = time.time() + 5
    while _count()[1] > start[1] and time.time() < limit:
        time.sleep(0.01)
    assert _count()[1] == start[1]
    y = cuda_ops.gemm(*given[0])
    torch.cuda.synchronize()
    assert torch.equal(y, want[0])
