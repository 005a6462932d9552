"""Dequantization by packed 16-bit arithmetic gives the bits of fp32-fma-then-round for every scale and bias. A warp takes it for
32 consecutive weight rows and 64 codes when all their scales and biases allow it, so scale and bias exponents are drawn per
block of 32 rows: blocks inside the bound, at each end of it, one beyond, and blocks that one row keeps out."""

import pytest
import torch

from oracle import reference as R

MANT = {torch.bfloat16: 7, torch.float16: 10}
FIELD = {torch.bfloat16: 255, torch.float16: 31}              # the exponent field of infinities and NaN
SCALES = {torch.bfloat16: (1, 240), torch.float16: (1, 20)}   # exponent fields of a scale that can be shifted
N, K, WARP, STEP = 1024, 512, 32, 64


def allowed(es, eb, zero_scale, zero_bias, dtype, bits):
    """The fp32 fma is exact for every code, by the places its operands can take (the rule the kernel votes on)."""
    lo, hi = SCALES[dtype]
    near = (es - eb <= 24 - MANT[dtype] - bits - 2) & (eb - es <= 24 - MANT[dtype] - 2)
    return zero_scale | (es >= lo) & (es <= hi) & (zero_bias | near)


def kinds(dtype, bits):
    """(scale's exponent field, bias's; None: the value is zero). Field 0 is a subnormal."""
    lo, hi = SCALES[dtype]
    below, above = 24 - MANT[dtype] - bits - 2, 24 - MANT[dtype] - 2
    top = FIELD[dtype] - 3                                    # no weight overflows
    out = [(None, None), (None, 0), (None, 7), (0, 0), (0, 3)]
    for es in (lo, lo + 1, (lo + hi) // 2, hi, hi + 1):
        out += [(es, None), (es, 0)] + [(es, es - d) for d in (0, 1, -1, below, below + 1, -above, -above - 1) if 1 <= es - d <= top]
    return out


def word(field, shape, dtype, g):
    """Values of one exponent field, signs and mantissas at random, as 16-bit words; a field of -1 is zero, of either sign."""
    mant = torch.randint(0, 1 << MANT[dtype], shape, generator=g)
    mant[(field == 0) & (mant == 0)] = 1
    sign = torch.randint(0, 2, shape, generator=g) << 15
    return sign | torch.where(field < 0, 0, (field.clamp(min=0) << MANT[dtype]) | mant)


def as_values(words, dtype):
    return torch.where(words >= 1 << 15, words - (1 << 16), words).to(torch.int16).view(dtype)


def pack(codes, bits):
    per = 32 // bits
    words = (codes.reshape(codes.shape[0], -1, per).to(torch.int64) << (torch.arange(per) * bits)).sum(-1)
    return torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)


def draw(dtype, bits, group):
    """Codes, scales, biases, and the share of (warp, step) pairs that may take the packed form."""
    g = torch.Generator().manual_seed(bits * 1000 + group)
    ks = kinds(dtype, bits)
    es, eb = torch.empty(N, K // group, dtype=torch.int64), torch.empty(N, K // group, dtype=torch.int64)
    unit = max(group, STEP)
    i = 0
    for b in range(N // WARP):
        rows = slice(b * WARP, (b + 1) * WARP)
        for u in range(K // unit):
            for e in range(unit // group):                    # two entries of a step: alike, or every third time not
                s, o = ks[(i + (e if i % 3 == 2 else 0)) % len(ks)]
                es[rows, u * (unit // group) + e] = -1 if s is None else s
                eb[rows, u * (unit // group) + e] = -1 if o is None else o
            if i % 5 == 4:                                    # one row, in one entry, that keeps the warp out
                es[b * WARP + i % WARP, u * (unit // group) + i % (unit // group)] = SCALES[dtype][1] + 1
            i += 1
    ok = allowed(es.clamp(min=0), eb.clamp(min=0), es < 0, eb < 0, dtype, bits)
    ok = ok.repeat_interleave(group, 1).reshape(N // WARP, WARP, K // STEP, STEP).all(3).all(1)      # per warp and step
    by_kind = {}
    for b in range(N // WARP):
        for st in range(K // STEP):
            r, c = b * WARP + (1 if (b * (K // unit) + st * STEP // unit) % WARP == 0 else 0), st * STEP // group
            by_kind.setdefault((int(es[r, c]), int(eb[r, c])), []).append(bool(ok[b, st]))
    for s, o in ks:
        s, o = -1 if s is None else s, -1 if o is None else o
        mine = bool(allowed(torch.tensor(max(s, 0)), torch.tensor(max(o, 0)), torch.tensor(s < 0), torch.tensor(o < 0), dtype, bits))
        assert any(by_kind[(s, o)]) == mine, (s, o)           # what is allowed is met by a whole warp, and the rest never
    codes = (torch.arange(N)[:, None] * group + torch.arange(K)) % (1 << bits)           # all codes in every block
    return codes, as_values(word(es, es.shape, dtype, g), dtype), as_values(word(eb, eb.shape, dtype, g), dtype), ok.float().mean().item()


CASES = [(dt, bits, group) for dt in (torch.bfloat16, torch.float16) for bits, group in ((4, 32), (4, 64), (4, 128), (8, 32), (8, 64))]


@pytest.mark.parametrize("dtype,bits,group", CASES, ids=str)
def test_the_drawn_weights_reach_both_forms(dtype, bits, group):
    assert 0.2 < draw(dtype, bits, group)[3] < 0.8


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,bits,group", CASES, ids=str)
def test_streamed_weight_has_the_canonical_bits(bi, dtype, bits, group):
    """x = identity rows: the product is the dequantized weight, one column of it per row (a single nonzero term)."""
    codes, scales, biases, _ = draw(dtype, bits, group)
    words = pack(codes, bits)
    w = R.dequant(words, scales, biases, group_size=group, bits=bits, dtype=dtype).cuda()
    assert w.isfinite().all()
    words, scales, biases = words.cuda(), scales.cuda(), biases.cuda()
    for x in torch.eye(K, dtype=dtype, device="cuda").split(64):
        for path in ("split", "fused"):
            got = bi.batch_invariant_quantized_matmul(x, words, scales, biases, group_size=group, bits=bits, path=path)
            assert torch.equal(got, bi.batch_invariant_matmul(x, w.T, path=path)), path


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
def test_infinite_and_nan_entries_stay_what_they_are(bi, dtype):
    """Rows 0-127: one odd entry a block of 32 rows, ordinary ones beside it. Rows 128-255: scales at the upper end, where an
    infinite or NaN bias is within the bound and whole blocks take the packed form. Every row has what fp32 gives."""
    g = torch.Generator().manual_seed(5)
    n, k, group, hi = 256, 256, 64, SCALES[dtype][1]
    codes = torch.randint(1, 16, (n, k), generator=g)         # no zero times infinity
    field = torch.full((n, k // group), FIELD[dtype] // 2 - 4)
    scales, biases = as_values(word(field, field.shape, dtype, g), dtype), as_values(word(field + 2, field.shape, dtype, g), dtype)
    inf, nan = float("inf"), float("nan")
    scales[5, 0], biases[37, 0], scales[70, 0], biases[101, 0] = inf, -inf, nan, nan
    big = as_values(word(torch.full((128,), hi), (128,), dtype, g), dtype)
    odd = torch.tensor([inf, -inf, nan], dtype=dtype)[torch.arange(128) % 3]
    scales[128:, 0], biases[128:, 0] = big, odd
    es, eb = torch.full((128,), hi), torch.full((128,), FIELD[dtype])
    assert allowed(es, eb, es < 0, eb < 0, dtype, 4).all()
    words = pack(codes, 4)
    w = R.dequant(words, scales, biases, group_size=group, bits=4, dtype=dtype)
    x = torch.zeros(1, k, dtype=dtype, device="cuda")
    x[0, :group] = 1.0                                        # the odd entries' group; the others are finite
    want = bi.batch_invariant_matmul(x, w.cuda().T)[0].cpu()
    got = bi.batch_invariant_quantized_matmul(x, words.cuda(), scales.cuda(), biases.cuda(), group_size=group, bits=4)[0].cpu()
    torch.testing.assert_close(got, want, rtol=0, atol=0, equal_nan=True)
    assert want[8].isfinite() and want[5].abs() == want[37].abs() == inf and want[70].isnan() and want[101].isnan()
    assert torch.equal(want[128:].isnan(), odd.isnan()) and torch.equal(want[128:][~odd.isnan()], odd[~odd.isnan()])
