"""Prefill attention at the edges of its tiling: row blocks (TQ * 1024 / D rows of one kv head, rows running over the
heads of the group), 32- or 64-key blocks inside the splits, every rows-per-thread variant the launch rule picks, and
values that are not finite behind the causal mask."""

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


# Launches of B sequences x 8 query / 4 kv heads x 45 queries that take 1, 2 and 4 rows per thread (a block is
# rows * 1024 / head_dim query rows; four rows from two blocks per SM on, two from one per two SMs on, 148 SMs).
ROWS_PER_THREAD = [(32, 1, 1), (32, 2, 10), (32, 4, 74), (64, 1, 1), (64, 2, 7), (64, 4, 37),
                   (128, 1, 1), (128, 2, 4), (128, 4, 25), (256, 1, 1), (256, 2, 2), (256, 4, 13)]


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("D,rows,B", ROWS_PER_THREAD)
def test_every_number_of_rows_per_thread(bi, dt, D, rows, B):
    """(fp32 with 256 dims has no room for four rows and stays at two.)"""
    g = torch.Generator().manual_seed(D * 10 + rows)
    q, k, v = (torch.randn(B, h, n, D, generator=g).to(dt) for h, n in ((8, 45), (4, 77), (4, 77)))
    for causal in (True, False):
        got = bi.batch_invariant_prefill_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5, causal=causal, split_size=32)
        assert R.bits_of(got) == R.bits_of(R.attn_prefill(q, k, v, scale=D ** -0.5, causal=causal, split_size=32))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("D,rows,B", ROWS_PER_THREAD)
def test_later_tokens_never_reach_a_row(bi, dt, D, rows, B):
    """Infinities and NaN in a later token's key and value: a row that does not see the token keeps the bits it has
    without them and those of the prefix run alone, in every row block and at every number of rows per thread."""
    L, T, split = 77, 45, 32
    g = torch.Generator().manual_seed(D + rows)
    q, k, v = (torch.randn(B, h, n, D, generator=g).to(dt).cuda() for h, n in ((8, T), (4, L), (4, L)))
    run = lambda q, k, v: bi.batch_invariant_prefill_attention(q, k, v, scale=D ** -0.5, causal=True, split_size=split)
    clean = run(q, k, v)
    for t in (1, 17, 30, 44):                                     # rows 0 .. t - 1 do not see keys from L - T + t on
        key = L - T + t
        kp, vp = k.clone(), v.clone()
        vp[:, :, key:, 0::2], vp[:, :, key:, 1::2] = float("inf"), float("nan")
        kp[:, :, key] = float("nan")
        kp[:, :, key + 1:] = float("-inf")
        got = run(q, kp, vp)[:, :, :t]
        assert R.bits_of(got) == R.bits_of(clean[:, :, :t]), t
        assert R.bits_of(got) == R.bits_of(run(q[:, :, :t], k[:, :, :key], v[:, :, :key])), t
