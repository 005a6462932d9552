"""RMSNorm of many 16-bit rows (a warp per row, the row staged in two halves) against the same rows in calls of a few (a CTA
per row), bit for bit: the shortest and longest rows staged, halves of unequal length, an odd last row."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,D", [(512, 8192), (513, 8184), (512, 8200), (511, 8192), (600, 8), (601, 248), (700, 256), (701, 264), (512, 512),
                                    (640, 768), (1001, 520), (515, 5000), (2999, 4096)])
def test_staged_rows_give_the_bits_of_few(bi, dt, rows, D):
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    x = (3 * torch.randn(rows, D, device="cuda", generator=g)).to(dt)
    w = (1 + 0.1 * torch.randn(D, device="cuda", generator=g)).to(dt)
    for weight in (w, None):
        many = bi.batch_invariant_rms_norm(x, weight, 1e-5)
        assert torch.equal(many, torch.cat([bi.batch_invariant_rms_norm(c, weight, 1e-5) for c in x.split(200)]))
