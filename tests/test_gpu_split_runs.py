"""Split matmuls whose first CTA a tile folds its own run of K groups give the bits of the fused shape."""

import pytest
import torch

import mlx_batch_invariant_b200 as bi
from mlx_batch_invariant_b200 import _lib
from mlx_batch_invariant_b200.runner.decoder import quantize_rows

pytestmark = pytest.mark.gpu


# (N, K): one tile and many SMs (runs too short), groups that do not divide among the CTAs of a tile, a last group that
# is short, the most tiles that still get two CTAs, one tile more (no runs)
@pytest.mark.parametrize("N,K", [(128, 1024), (4096, 14336), (6144, 6400), (4160, 40 * 256 + 192), (9472, 4096), (9500, 4096)])
@pytest.mark.parametrize("M", [32, 33, 63, 64, 130])
def test_bits_of_the_fused_shape(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    ref = bi.batch_invariant_matmul(x, w.T, path="fused")
    assert torch.equal(bi.batch_invariant_matmul(x, w.T, path="split"), ref)
    assert torch.equal(bi.batch_invariant_matmul(x, w.T, path="split", bias=bias), ref + bias)
    assert torch.equal(bi.batch_invariant_matmul(x, w.T), ref)
    if M > 64:
        assert torch.equal(bi.batch_invariant_matmul(x, w.T, path="split", batch_tile=64), ref)      # a last tile of two rows
    if K % 64 == 0 and N * K < 1 << 25:
        q = quantize_rows(w, 64, 4)
        kw = dict(group_size=64, bits=4)
        assert torch.equal(bi.batch_invariant_quantized_matmul(x, *q, path="split", **kw), bi.batch_invariant_quantized_matmul(x, *q, path="fused", **kw))
    _lib.check_device_status()
