"""Matmuls that start on a weight at rest while the kernels in front of them still run: the bits of plain launches, eagerly and
from a graph, for every kernel and ring (rings deeper than K, several tiles a CTA, K that ends inside a step)."""

import pytest
import torch

import mlx_batch_invariant_b200 as bi
from mlx_batch_invariant_b200 import _lib
from mlx_batch_invariant_b200.runner.decoder import quantize_rows

pytestmark = pytest.mark.gpu


def weights(dims, packed):
    g = torch.Generator(device="cuda").manual_seed(sum(dims))
    ws = [(torch.randn(n, k, device="cuda", generator=g) * k ** -0.5).bfloat16() for k, n in zip(dims, dims[1:])]
    return [quantize_rows(w, 64, packed) for w in ws] if packed else ws


def chain(x, ws, packed, path, static):
    """Linear, norm, linear, norm, ...: every matmul follows a kernel that writes its activation."""
    for w in ws:
        h = bi.batch_invariant_rms_norm(x, None, 1e-5)
        if packed:
            x = bi.batch_invariant_quantized_matmul(h, *w, group_size=64, bits=packed, path=path, static_weight=static)
        else:
            x = bi.batch_invariant_matmul(h, w.T, path=path, static_weight=static)
    return x


@pytest.mark.parametrize("M,path", [(1, "auto"), (1, "fused"), (16, "auto"), (64, "split"), (64, "fused"), (70, "pair"), (300, "auto")])
@pytest.mark.parametrize("dims,packed", [((256, 4096, 320, 22000, 512), 0), ((1000, 136, 2056, 1000), 0), ((256, 4096, 320, 22016, 512), 4), ((512, 2048, 512), 8)])
def test_bits_of_plain_launches(M, path, dims, packed, monkeypatch):
    ws = weights(dims, packed)
    x = torch.randn(M, dims[0], device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).bfloat16()
    monkeypatch.setenv("BI_PDL", "0")
    want = chain(x, ws, packed, path, False)
    monkeypatch.delenv("BI_PDL")
    for _ in range(3):
        assert torch.equal(chain(x, ws, packed, path, True), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(x, ws, packed, path, True)
    for _ in range(3):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)
    _lib.check_device_status()


@pytest.mark.parametrize("captured", [False, True])
def test_behind_copies_memsets_and_joined_streams(captured):
    """What stands in front of an overlapped launch need not be a kernel, nor on its stream."""
    w = weights((512, 4096, 512), 0)
    src = torch.randn(16, 512, device="cuda").bfloat16()
    want = bi.batch_invariant_matmul(bi.batch_invariant_matmul(src, w[0].T), w[1].T)
    x, side = torch.empty_like(src), torch.cuda.Stream()

    def work():
        outs = []
        x.copy_(src)                                                       # a copy
        outs.append(bi.batch_invariant_matmul(bi.batch_invariant_matmul(x, w[0].T, static_weight=True), w[1].T))
        x.zero_()                                                          # a memset
        outs.append(bi.batch_invariant_matmul(x, w[0].T))
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):                                      # a kernel of the library and a copy on another stream
            y = bi.batch_invariant_matmul(src, w[0].T)
            x.copy_(src)
        z = bi.batch_invariant_rms_norm(src, None, 1e-5)
        torch.cuda.current_stream().wait_stream(side)
        outs += [bi.batch_invariant_matmul(y, w[1].T, static_weight=True), bi.batch_invariant_matmul(bi.batch_invariant_matmul(x, w[0].T), w[1].T), z]
        return outs

    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = work()
        for o in outs:
            o.fill_(7.0)
        graph.replay()
    else:
        outs = work()
    torch.cuda.synchronize()
    a, zero, b, c, z = outs
    assert torch.equal(a, want) and torch.equal(b, want) and torch.equal(c, want) and not zero.any()
    assert torch.equal(z, bi.batch_invariant_rms_norm(src, None, 1e-5))


@pytest.mark.parametrize("M,path,packed", [(16, "split", 0), (16, "fused", 4), (48, "pair", 0)])
def test_time_of_the_kernels_in_front_is_no_timeout(M, path, packed):
    """The norm in front lets the matmul in and then waits out its limit for a flag that nothing raises (2 s): the matmul's own
    limits begin when that is over."""
    from mlx_batch_invariant_b200.runner.decoder import KernelBackend
    (w,), ones = weights((512, 4096), packed), torch.ones(512, device="cuda").bfloat16()
    x = torch.randn(M, 512, device="cuda").bfloat16()
    flags, epoch = torch.zeros(8, dtype=torch.int32, device="cuda"), torch.tensor([3], dtype=torch.int32, device="cuda")

    def work(static, **kw):
        h = KernelBackend().add_rms_norm(x, x, ones, 1e-5, **kw)[1]
        if packed:
            return bi.batch_invariant_quantized_matmul(h, *w, group_size=64, bits=packed, path=path, static_weight=static)
        return bi.batch_invariant_matmul(h, w.T, path=path, static_weight=static)

    want = work(False)
    _lib.check_device_status()
    got = work(True, awaiting=(flags.data_ptr(), epoch.data_ptr(), 0, 2))
    torch.cuda.synchronize()
    with pytest.raises(_lib.KernelError, match="0x20103"):                # the norm's: 0x20000 | peer 1 << 8 | epoch 3
        _lib.check_device_status()
    assert torch.equal(got, want)
