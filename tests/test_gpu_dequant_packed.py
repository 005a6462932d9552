"""Dequantization by packed 16-bit arithmetic gives the bits of fp32-fma-then-round for every scale and bias: ordinary groups,
groups whose bias is so far from the scale that the fp32 fma is inexact, zeros, subnormal, huge, infinite and NaN entries."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bi():
    import mlx_batch_invariant_b200 as m
    return m


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("bits,group", [(4, 32), (4, 64), (4, 128), (8, 32), (8, 64)])
def test_streamed_weight_has_the_canonical_bits(bi, dtype, bits, group):
    """x = identity rows: the product is the dequantized weight, one column of it per row (a single nonzero term)."""
    N, K, per = 256, 256, 32 // bits
    g = torch.Generator(device="cuda").manual_seed(bits * 1000 + group)
    codes = torch.randint(0, 1 << bits, (N, K), generator=g, device="cuda")
    words = (codes.reshape(N, K // per, per).to(torch.int64) << (torch.arange(per, device="cuda") * bits)).sum(-1)
    words = torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)
    # every exponent of the scale against every distance of the bias, signs and mantissas at random
    lim = 120 if dtype == torch.bfloat16 else 14
    es = torch.randint(-lim, lim // 2, (N, K // group), generator=g, device="cuda").double()
    eb = (es + torch.randint(-26, 27, es.shape, generator=g, device="cuda")).clamp(-lim, lim // 2)
    def value(e):
        m = 1 + torch.rand(e.shape, generator=g, device="cuda", dtype=torch.float64)
        return (m * torch.exp2(e) * (1 - 2 * torch.randint(0, 2, e.shape, generator=g, device="cuda"))).to(dtype)
    scales, biases = value(es), value(eb)
    biases[0], scales[1], biases[2] = 0.0, 0.0, -0.0
    scales[3] = torch.finfo(dtype).smallest_normal / 4
    w = torch.addcmul(biases.float().repeat_interleave(group, 1).double(), codes.double(), scales.float().repeat_interleave(group, 1).double())
    w = w.float().to(dtype)                       # one fp32 rounding (the fp64 sum is exact: at most 26 + 24 places), one to T
    rows = torch.arange(0, K, 5, device="cuda")
    for r in rows.split(16):
        x = torch.zeros(len(r), K, dtype=dtype, device="cuda")
        x[torch.arange(len(r), device="cuda"), r] = 1.0
        for path in ("split", "fused"):
            got = bi.batch_invariant_quantized_matmul(x, words, scales, biases, group_size=group, bits=bits, path=path)
            assert torch.equal(got, bi.batch_invariant_matmul(x, w.T, path=path)), path


def test_infinite_and_nan_entries_stay_what_they_are(bi):
    K = N = 256
    x = torch.zeros(1, K, dtype=torch.bfloat16, device="cuda"); x[0, 0] = 1.0
    words = torch.full((N, K // 8), 0x11111111, dtype=torch.int32, device="cuda")
    scales, biases = (torch.ones(N, K // 64, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    scales[5], biases[6], scales[7] = float("inf"), float("-inf"), float("nan")
    got = bi.batch_invariant_quantized_matmul(x, words, scales, biases, group_size=64, bits=4)[0].float()
    assert not got[5].isfinite() and not got[6].isfinite() and got[7].isnan() and got[8] == 2.0
