"""The SM-pair matmul (256 weight rows x up to 256 batch rows on two SMs) gives the bits of the one-SM shapes."""

import pytest
import torch

import mlx_batch_invariant_b200 as bi
from mlx_batch_invariant_b200 import _lib
from mlx_batch_invariant_b200.runner.decoder import quantize_rows

pytestmark = pytest.mark.gpu

# (M, N, K, batch tile): whole tiles; rows that leave the second half of a tile (or its second CTA) empty; weight rows
# that end inside the first and inside the second CTA; K that ends inside a K = 16 step, a 64 step, a slot of two steps
# and a group; one group; more units than pairs of SMs (ring and accumulator phases wrap between units)
SHAPES = [(256, 256, 256, 256), (257, 512, 1024, 256), (300, 384, 896, 96), (33, 100, 264, 32), (65, 896, 200, 64),
          (70, 640, 320, 64), (129, 130, 1152, 128), (1000, 2300, 512, 32), (700, 4096, 2048, 224)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,bm", SHAPES)
def test_pair_gives_the_one_sm_bits(M, N, K, bm, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    ref = bi.batch_invariant_matmul(x, w.T, path="fused")
    assert torch.equal(bi.batch_invariant_matmul(x, w.T, path="pair", batch_tile=bm), ref)
    assert torch.equal(bi.batch_invariant_matmul(x, w.T, path="pair", batch_tile=bm, bias=bias), ref + bias)
    assert torch.equal(bi.batch_invariant_matmul(x, w.T), ref)
    assert torch.equal(bi.batch_invariant_matmul(x[M - 1:], w.T), ref[M - 1:])          # a batch of one
    _lib.check_device_status()


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("gs", [32, 64, 128])
@pytest.mark.parametrize("M,N,K,bm", [(300, 384, 1024, 96), (33, 100, 384, 32), (700, 2300, 640, 256)])
def test_pair_on_packed_weights_gives_the_one_sm_bits(M, N, K, bm, gs, bits):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    for dtype in (torch.bfloat16, torch.float16):
        x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
        q = quantize_rows((torch.randn(N, K, device="cuda", generator=g) * 0.02).to(dtype), gs, bits)
        ref = bi.batch_invariant_quantized_matmul(x, *q, group_size=gs, bits=bits, path="fused")
        assert torch.equal(bi.batch_invariant_quantized_matmul(x, *q, group_size=gs, bits=bits, path="pair", batch_tile=bm), ref)
        assert torch.equal(bi.batch_invariant_quantized_matmul(x, *q, group_size=gs, bits=bits), ref)
    _lib.check_device_status()


def test_pair_reads_strided_rows_and_refuses_bad_tiles():
    x = torch.randn(300, 1032, device="cuda").to(torch.bfloat16)[:, :1024]
    w = torch.randn(512, 1040, device="cuda").to(torch.bfloat16)[:, :1024]
    assert torch.equal(bi.batch_invariant_matmul(x, w.T, path="pair", batch_tile=160), bi.batch_invariant_matmul(x, w.T, path="fused"))
    for bad in (16, 48, 288):
        with pytest.raises(_lib.KernelError):
            bi.batch_invariant_matmul(x, w.T, path="pair", batch_tile=bad)
