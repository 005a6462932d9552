"""CUDA-core matmul at the edges of its tiles: the weight-streaming kernel (up to 8 fp32 rows), the 16-, 32- and 64-row
tiles with their remainders in M, N (128 columns) and K (16- and 32-wide stages, 256-wide groups), vector and element-wise
fetches. Bit for bit against the oracle's order."""

import pytest
import torch

from oracle import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 4, 7, 8, 9, 16, 17, 32, 33, 49, 64, 65, 97])
@pytest.mark.parametrize("N,K", [(127, 260), (129, 12), (130, 1028), (33, 301)])
def test_fp32_tiles_bit_exact(bi, M, N, K):
    g = torch.Generator().manual_seed(M * 7 + N + K)
    x, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g) / K ** 0.5
    want = R.bits_of(R.matmul_f32order(x, w.T.contiguous()))
    for path in ("auto", "split", "fused"):
        assert R.bits_of(bi.batch_invariant_matmul(x.cuda(), w.cuda().T, path=path)) == want, path


@pytest.mark.parametrize("M", [5, 40, 70])
def test_element_wise_fetches_bit_exact(bi, M):
    """16-bit weights TMA cannot address, a row-major [K, N] operand, and a misaligned fp32 activation."""
    g = torch.Generator().manual_seed(M)
    for dt in (torch.bfloat16, torch.float16):
        x, w = torch.randn(M, 275, generator=g).to(dt), torch.randn(140, 275, generator=g).to(dt)
        assert R.bits_of(bi.batch_invariant_matmul(x.cuda(), w.cuda().T)) == R.bits_of(R.matmul_f32order(x, w.T.contiguous()))
    x, b = torch.randn(M, 300, generator=g), torch.randn(300, 140, generator=g)
    want = R.bits_of(R.matmul_f32order(x, b))
    assert R.bits_of(bi.batch_invariant_matmul(x.cuda(), b.cuda())) == want
    pad = torch.zeros(M, 303)
    pad[:, 1:301] = x
    assert R.bits_of(bi.batch_invariant_matmul(pad.cuda()[:, 1:301], b.cuda())) == want


@pytest.mark.parametrize("dt,K,gs", [(torch.float32, 288, 32), (torch.float32, 640, 128), (torch.bfloat16, 288, 32), (torch.float16, 544, 32)])
@pytest.mark.parametrize("bits", [4, 8])
def test_packed_pieces_bit_exact(bi, dt, K, gs, bits):
    """Packed weights the tensor-core path does not take (fp32, or K no multiple of 64): the four codes of a piece, its scale
    and bias, at the edges of the tiles and of the K groups."""
    g = torch.Generator().manual_seed(K + bits)
    N = 131
    p, s, b = R.quantize_affine(torch.randn(N, K, generator=g) * 0.02, group_size=gs, bits=bits, dtype=dt)
    wd = R.dequant(p, s, b, group_size=gs, bits=bits, dtype=dt)
    for M in (1, 9, 17, 33, 70):
        x = torch.randn(M, K, generator=g).to(dt)
        want = R.bits_of(R.matmul_f32order(x, wd.T.contiguous()))
        for path in ("auto", "split", "fused"):
            got = bi.batch_invariant_quantized_matmul(x.cuda(), p.cuda(), s.cuda(), b.cuda(), group_size=gs, bits=bits, path=path)
            assert R.bits_of(got) == want, (M, path)
