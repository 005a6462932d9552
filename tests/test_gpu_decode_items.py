"""Decode attention over sequences of different lengths: which warp takes which split is found from the lengths on the
device. Every row of the batch has the bits of its sequence decoded alone, whatever the others' lengths are."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bi():
    import mlx_batch_invariant_b200 as m
    return m


# (sequences, capacity, heads, kv heads): one and several groups of 32 sequences, a capacity below, at and above one split
# and two; few items (a warp per head) and more than a round of them; the last batch that is looked up and the first that is
# dealt over the capacity; equal lengths on seven of eight warps
CASES = [(1, 300, 8, 2), (5, 33, 8, 8), (31, 256, 8, 2), (32, 257, 4, 1), (33, 511, 8, 2), (64, 512, 32, 8), (65, 700, 8, 2),
         (130, 640, 14, 2), (9, 4096, 32, 8), (1024, 257, 2, 1), (1025, 257, 2, 1), (8, 8192, 32, 8)]


@pytest.mark.parametrize("B,L,Hq,Hkv", CASES)
@pytest.mark.parametrize("kind", ["random", "edges", "equal"])
def test_mixed_lengths_have_the_bits_of_each_sequence_alone(bi, B, L, Hq, Hkv, kind):
    g = torch.Generator(device="cuda").manual_seed(B * L + Hq)
    q = torch.randn(B, Hq, 1, 128, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, Hkv, L, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    if kind == "random":
        lens = torch.randint(1, L + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    elif kind == "edges":      # around the ends of a split, no keys at all, more than the cache holds
        edge = torch.tensor([1, 255, 256, 257, 31, 32, 33, 512, 0, L, L + 5, 511, 513], dtype=torch.int32, device="cuda")
        lens = edge[torch.arange(B, device="cuda") % len(edge)]
    else:
        lens = torch.full((B,), L, dtype=torch.int32, device="cuda")
    got = bi.batch_invariant_decode_attention(q, k, v, scale=128 ** -0.5, kv_lens=lens)
    for b, n in enumerate(lens.clamp(max=L).tolist()):
        if n:
            alone = bi.batch_invariant_decode_attention(q[b:b + 1], k[b:b + 1, :, :n], v[b:b + 1, :, :n], scale=128 ** -0.5)
            assert torch.equal(got[b:b + 1], alone), (b, n)
