"""CUDA-core matmul at the ends of its range: more K groups than a grid has blocks in z."""

import pytest
import torch

from oracle import reference as R

pytestmark = pytest.mark.gpu

K_LONG = 65536 * 256 + 4          # 65537 groups


@pytest.mark.parametrize("K", [K_LONG, K_LONG + 1])               # rows of float4, and rows that are not
def test_more_groups_than_grid_blocks_fold_in_place(bi, K):
    g = torch.Generator().manual_seed(1)
    x, w = torch.randn(1, K, generator=g), torch.randn(1, K, generator=g) / K ** 0.5
    want = R.bits_of(R.matmul_f32order(x, w.T.contiguous()))
    xc, wc = x.cuda(), w.cuda()
    assert R.bits_of(bi.batch_invariant_matmul(xc, wc.T, path="fused")) == want
    for M in (1, 33):                                              # 33 equal rows: one row, stride 0
        got = bi.batch_invariant_matmul(xc.expand(M, K), wc.T)
        assert R.bits_of(got[:1]) == want and R.bits_of(got[M - 1:]) == want


def test_auto_ignores_a_misaligned_optional_workspace(bi):
    """Beyond 32 rows the workspace is optional: one that is not 16-byte aligned is not used. Up to 32 rows it is promised
    scratch, and a misaligned one is refused."""
    from mlx_batch_invariant_b200 import _lib
    M, N, K = 40, 64, 1024
    g = torch.Generator().manual_seed(2)
    x, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g) / 32
    want = R.bits_of(R.matmul_f32order(x, w.T.contiguous()))
    xc, wc, out = x.cuda(), w.cuda(), torch.empty(M, N, device="cuda")
    ws = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    call = lambda m, p: _lib.load().bi_matmul(xc.data_ptr(), wc.data_ptr(), out.data_ptr(), p, ws.numel() - 16, m, N, K, K, 1, 1, K,
                                              _lib.BI_F32, _lib.PATH_AUTO, None, _lib.stream_ptr(xc.device))
    for off in (0, 4, 8):
        out.zero_()
        _lib.check(call(M, ws.data_ptr() + off))
        assert R.bits_of(out) == want, off
    assert call(32, ws.data_ptr() + 4) == _lib.BI_ERR_MISALIGNED
