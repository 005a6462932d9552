"""The wide and the plain forms of the decoder's small kernels: the same bits on both sides of their rules."""

import pytest
import torch

from mlx_batch_invariant_b200 import _lib
from mlx_batch_invariant_b200.runner.decoder import KernelBackend
from oracle import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,F", [(11, 14336), (150, 1028), (600, 260), (150, 1030), (2, 80000)])      # widths of whole and broken quads
def test_swiglu_of_many_rows_has_the_bits_of_one(M, F, dtype):
    gu = (4 * torch.randn(M, 2 * F, device="cuda", generator=torch.Generator(device="cuda").manual_seed(F))).to(dtype)
    got = KernelBackend().swiglu(gu)
    for r in (0, M // 2, M - 1):
        assert torch.equal(KernelBackend().swiglu(gu[r:r + 1]), got[r:r + 1])
    shifted = torch.empty(gu.numel() + 1, device="cuda", dtype=dtype)[1:].view(M, 2 * F).copy_(gu)      # not aligned for the quads
    assert torch.equal(KernelBackend().swiglu(shifted), got)


# one head: the accumulators start 8 bytes past a 16-byte line (a dim a thread); 1, 4, 5 and 9 splits; lengths that differ
@pytest.mark.parametrize("B,Hq,D,L", [(1, 1, 64, 200), (1, 2, 128, 1024), (3, 4, 32, 1100), (2, 2, 256, 2304)])
def test_split_merge(B, Hq, D, L):
    g = torch.Generator().manual_seed(L)
    q, k, v = torch.randn(B, Hq, 1, D, generator=g), torch.randn(B, Hq, L, D, generator=g), torch.randn(B, Hq, L, D, generator=g)
    lens = torch.tensor([L, 1, 257][:B], dtype=torch.int32)
    ref = torch.cat([R.attn_decode(q[b:b + 1], k[b:b + 1, :, :lens[b]].contiguous(), v[b:b + 1, :, :lens[b]].contiguous(), scale=D ** -0.5) for b in range(B)])
    qc, kc, vc, lc = q.cuda(), k.cuda(), v.cuda(), lens.cuda()
    lib = _lib.load()
    nbytes = lib.bi_attn_decode_workspace_bytes(B, Hq, L, D, 256)
    ws = torch.empty(max(nbytes, 16), dtype=torch.uint8, device="cuda")
    for shift in (0, D // 32):                    # elements: for 32 and 64 dims an output that is not aligned for four
        out = torch.empty(shift + q.numel(), device="cuda")[shift:]
        _lib.check(lib.bi_attn_decode(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), out.data_ptr(), lc.data_ptr(), ws.data_ptr(), nbytes, B, Hq, Hq, L, D,
                                      Hq * L * D, L * D, D, D ** -0.5, 256, _lib.BI_F32, _lib.stream_ptr(qc.device)))
        assert R.bits_of(out.view_as(qc)) == R.bits_of(ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,hq,hkv,D", [(1, 1, 2, 1, 16), (2, 37, 14, 2, 64), (1, 300, 32, 8, 128), (3, 5, 3, 1, 96)])      # a head a thread ... blocks that a token does not fill
def test_rope_by_quads_of_pieces_has_the_bits_of_elements(B, T, hq, hkv, D, dtype):
    g = torch.Generator(device="cuda").manual_seed(T)
    cap, pos0 = T + 3, torch.tensor([2], dtype=torch.long, device="cuda")
    qkv = torch.randn(B * T, (hq + 2 * hkv) * D, device="cuda", generator=g).to(dtype)
    cos, sin = (torch.randn(cap, D, device="cuda", generator=g) for _ in range(2))
    shifted = torch.empty(qkv.numel() + 1, device="cuda", dtype=dtype)[1:].view_as(qkv).copy_(qkv)        # not aligned: an element a thread
    got = []
    for x in (qkv, shifted):
        kc, vc = (torch.full((B + 1, hkv, cap, D), 7.0, device="cuda", dtype=dtype) for _ in range(2))
        got.append((KernelBackend().rope_append(x, cos, sin, pos0, B, T, hq, hkv, D, kc, vc), kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*got))
    _lib.check_device_status()
