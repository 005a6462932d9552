"""Who owns the matmuls' scratch: a captured graph its own, large calls theirs, decode-sized calls one per stream."""

import threading

import pytest
import torch

from mlx_batch_invariant_b200 import _lib

pytestmark = pytest.mark.gpu


def _fp32(m, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(m, k, device="cuda", generator=g), torch.randn(n, k, device="cuda", generator=g) / k ** 0.5


def test_a_graph_keeps_its_scratch_when_a_larger_call_follows(bi):
    """Capture on an explicit stream that has been used before, then a larger call on that stream, then tensors that would
    land in freed scratch: a replay gives the captured call's bits and leaves those tensors alone."""
    s = torch.cuda.Stream()
    x, w = _fp32(8, 4096, 4096, 1)
    big_x, big_w = _fp32(30, 4096, 14336, 2)
    want = bi.batch_invariant_matmul(x, w.T, path="fused")
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        bi.batch_invariant_matmul(x, w.T)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            out = bi.batch_invariant_matmul(x, w.T)
        bi.batch_invariant_matmul(big_x, big_w.T)
        others = [torch.full((1 << 20,), 7, dtype=torch.uint8, device="cuda") for _ in range(64)]
        out.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert all(bool((t == 7).all()) for t in others)


def test_large_scratch_is_not_kept(bi):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        x, w = _fp32(300, 8192, 4096, 3)                            # 157 MB of partials
        got = bi.batch_invariant_matmul(x, w.T)
        assert torch.equal(got, bi.batch_invariant_matmul(x, w.T, path="fused"))
    torch.cuda.synchronize()
    assert max((ws.numel() for ws in _lib._workspaces.values()), default=0) <= _lib.KEPT_BYTES


def test_the_fold_inside_a_capture_finds_its_counters_zero(bi):
    x = torch.randn(16, 4096, device="cuda").to(torch.bfloat16)
    w = (torch.randn(4096, 4096, device="cuda") / 64).to(torch.bfloat16)
    want = bi.batch_invariant_matmul(x, w.T, path="split")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = bi.batch_invariant_matmul(x, w.T, path="fold")
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    bi.check_device_status()


def test_threads_on_one_stream_do_not_share_scratch(bi):
    """A split call is two launches; another thread's may lie between them on the same stream."""
    kept = {}

    def call(name):
        kept[name], zeroed = _lib.matmul_workspace(torch.device("cuda", 0), 1 << 21)
        assert zeroed and _lib.matmul_workspace(torch.device("cuda", 0), 1 << 20)[0] is kept[name]

    threads = [threading.Thread(target=call, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
        t.join()
    call("here")
    assert len({ws.data_ptr() for ws in kept.values()}) == 4


def test_a_wait_that_ran_out_drops_the_scratch_of_every_thread(bi):
    before = _lib.matmul_workspace(torch.device("cuda", 0), 1 << 20)[0]
    word = _lib.status_word(torch.device("cuda", 0))
    word.fill_(0x10000)

    def check():
        with pytest.raises(_lib.KernelError):
            bi.check_device_status()

    t = threading.Thread(target=check)
    t.start()
    t.join()
    assert _lib.matmul_workspace(torch.device("cuda", 0), 1 << 20)[0] is not before
    bi.check_device_status()


def test_the_calls_of_a_capture_share_scratch_and_captures_do_not(bi):
    x, w = _fp32(8, 2048, 4096, 4)
    want = bi.batch_invariant_matmul(x, w.T, path="fused")
    torch.cuda.synchronize()
    graphs, outs, used = [torch.cuda.CUDAGraph() for _ in range(2)], [], []
    s = torch.cuda.Stream()
    for graph in graphs:
        with torch.cuda.graph(graph, stream=s):
            outs += [bi.batch_invariant_matmul(x, w.T), bi.batch_invariant_matmul(x, w.T)]
            used += [_lib.matmul_workspace(x.device, 1 << 20)[0].data_ptr() for _ in range(2)]
    assert used[0] == used[1] and used[2] == used[3] and used[0] != used[2]
    bi.batch_invariant_matmul(x, w.T)
    assert not _lib._workspaces.captured                               # an eager call lets the captures' scratch go
    for graph in graphs:
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
