"""RMSNorm of many rows (a warp per row) against the same rows in calls of a few (a CTA per row), bit for bit: ragged counts and
widths, and both sides of the limits of fp32 (1024 rows, 1024 elements)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,D", [(2048, 4096), (2047, 4096), (1027, 896), (1024, 1024), (1500, 8), (1501, 264), (2050, 4088), (2050, 4104), (2048, 3072), (2047, 3072), (2369, 4096), (3801, 4096), (3749, 4088), (1023, 896), (1023, 1024), (1024, 1032)])
def test_many_rows_give_the_bits_of_few(bi, dt, rows, D):
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    x = (3 * torch.randn(rows, D, device="cuda", generator=g)).to(dt)
    w = (1 + 0.1 * torch.randn(D, device="cuda", generator=g)).to(dt)
    for weight in (w, None):
        many = bi.batch_invariant_rms_norm(x, weight, 1e-5)
        few = torch.cat([bi.batch_invariant_rms_norm(c, weight, 1e-5) for c in x.split(200)])
        assert torch.equal(many, few)
