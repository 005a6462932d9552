"""Launches that hold an SM's other places by shared memory, or that leave the overlap, give the bits of plain ones: a CTA, an SM's worth, one
more, and a wave of them, behind a kernel that may let them in."""

import pytest
import torch

import mlx_batch_invariant_b200 as bi
from mlx_batch_invariant_b200 import _lib
from mlx_batch_invariant_b200.runner.decoder import quantize_rows

pytestmark = pytest.mark.gpu
SMS = 148


def _rand(*shape, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


def _check(call, monkeypatch):
    """`call` behind a norm, plainly and overlapped, eagerly and from a graph."""
    x = _rand(4, 4096, dtype=torch.bfloat16)
    monkeypatch.setenv("BI_PDL", "0")
    want = call()
    monkeypatch.delenv("BI_PDL")
    bi.batch_invariant_rms_norm(x, None, 1e-5)
    assert torch.equal(call(), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(2):
            bi.batch_invariant_rms_norm(x, None, 1e-5)
            got = call()
    got.zero_()
    graph.replay()
    assert torch.equal(got, want)
    _lib.check_device_status()


# columns: 128 a CTA; 600 of K are three groups, which few columns split
@pytest.mark.parametrize("N,K", [(100, 256), (128 * SMS, 256), (128 * SMS + 1, 256), (128 * 49, 600), (128 * 9 * SMS, 64)])
@pytest.mark.parametrize("M", [1, 8, 9, 40, 128])
def test_fp32_linear(M, N, K, monkeypatch):
    a, w = _rand(M, K), _rand(N, K)
    _check(lambda: bi.batch_invariant_matmul(a, w.T), monkeypatch)


@pytest.mark.parametrize("M", [1, 16, 64])
def test_element_wise_and_packed_linear(M, monkeypatch):
    a, w = _rand(M, 512), _rand(1000, 512)
    packed = quantize_rows(w, 64, 4)
    _check(lambda: bi.batch_invariant_quantized_matmul(a, *packed, group_size=64, bits=4), monkeypatch)
    _check(lambda: bi.batch_invariant_matmul(a.bfloat16(), w.bfloat16().T.contiguous()), monkeypatch)


@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 64), (torch.float16, 128), (torch.float32, 256), (torch.bfloat16, 32)])
@pytest.mark.parametrize("B", [1, SMS, SMS + 1, 5 * SMS])
def test_prefill(B, dtype, D, monkeypatch):
    q, k, v = (_rand(B, 1, 5, D, dtype=dtype) for _ in range(3))
    _check(lambda: bi.batch_invariant_attention(q, k, v, scale=D ** -0.5, mask="causal"), monkeypatch)


@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 64), (torch.float32, 128), (torch.float32, 32)])
@pytest.mark.parametrize("B", [1, 4 * SMS, 4 * SMS + 1, 9 * SMS, 23 * SMS, 25 * SMS])      # four streams a CTA, or all on as few CTAs as fit
def test_decode_streams(B, dtype, D, monkeypatch):
    q, k, v = (_rand(B, 1, n, D, dtype=dtype) for n in (1, 40, 40))
    _check(lambda: bi.batch_invariant_decode_attention(q, k, v, scale=D ** -0.5), monkeypatch)
