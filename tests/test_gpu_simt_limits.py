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
