"""Prefill attention at the edges of its tiling: row blocks (TQ * 1024 / D rows of one kv head, rows running over the
heads of the group), 32- or 64-key blocks inside the splits, and every rows-per-thread variant the launch rule picks."""

import pytest
import torch

from oracle import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,Hq,Hkv,Tq,L,D,split", [
    (1, 6, 2, 11, 43, 128, 256),       # 33 rows: one past a block of 32, straddling heads
    (1, 4, 4, 33, 289, 128, 256),      # key count one past a block, into the second split
    (2, 8, 2, 7, 64, 256, 32),         # widest head, splits as short as a block
    (1, 3, 1, 43, 43, 32, 20),         # split shorter than a block
    (3, 14, 2, 65, 300, 64, 256),
    (16, 32, 8, 40, 70, 128, 256),     # enough row blocks for four rows per thread
    (20, 16, 8, 70, 70, 64, 256),
    (1, 1, 1, 2, 2, 128, 256),         # smallest
])
def test_prefill_block_edges(bi, dt, B, Hq, Hkv, Tq, L, D, split):
    g = torch.Generator().manual_seed(B * 1000 + Tq + L)
    q, k, v = (torch.randn(B, h, n, D, generator=g).to(dt) for h, n in ((Hq, Tq), (Hkv, L), (Hkv, L)))
    for causal in (True, False):
        got = bi.batch_invariant_prefill_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5, causal=causal, split_size=split)
        assert R.bits_of(got) == R.bits_of(R.attn_prefill(q, k, v, scale=D ** -0.5, causal=causal, split_size=split))


def test_prefill_rows_not_16_byte_aligned(bi):
    """The C entry point takes K/V whose rows are aligned to a lane's chunk only (8 bytes here)."""
    from mlx_batch_invariant_b200 import _lib
    B, H, T, D = 1, 2, 37, 128
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(B, H, T, D, generator=g).to(torch.bfloat16) for _ in range(3))
    pad = [torch.zeros(B, H, T, D + 4, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    for p, x in zip(pad, (k, v)):
        p[..., 4:] = x.cuda()
    kc, vc = (p[..., 4:] for p in pad)
    qc, out = q.cuda(), torch.empty(B, H, T, D, dtype=torch.bfloat16, device="cuda")
    _lib.check(_lib.load().bi_attn_prefill(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), out.data_ptr(), B, H, H, T, T, D, kc.stride(0),
                                           kc.stride(1), kc.stride(2), D ** -0.5, 1, 256, _lib.BI_BF16, _lib.stream_ptr(qc.device)))
    assert R.bits_of(out) == R.bits_of(R.attn_prefill(q, k, v, scale=D ** -0.5, causal=True))
