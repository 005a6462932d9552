"""The SM-pair matmul on an activation that is still arriving from other ranks: with the flags raised it gives the bits of the
plain call, dense and packed; with a flag that nothing raises it gives up after its time limit, says so, and leaves the
context usable."""

import time

import pytest
import torch

from mlx_batch_invariant_b200 import _lib
from mlx_batch_invariant_b200.runner.decoder import quantize_rows
from oracle import reference as R

pytestmark = pytest.mark.gpu


def _xw(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    return torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16), (torch.randn(N, K, device="cuda", generator=g) / 32).to(torch.bfloat16)


@pytest.mark.parametrize("M,N,K", [(300, 512, 1024), (129, 300, 264), (700, 4096, 4096)])
def test_raised_flags_give_the_plain_bits(bi, M, N, K):
    x, w = _xw(M, N, K)
    flags = torch.tensor([0, 5, 9, 0, 0, 0, 0, 0], dtype=torch.int32, device="cuda")      # this rank is 0 of 3
    epoch = torch.tensor([5], dtype=torch.int32, device="cuda")
    aw = (flags.data_ptr(), epoch.data_ptr(), 0, 3)
    want = R.bits_of(bi.batch_invariant_matmul(x, w.T, path="fused"))
    for path in ("pair", "auto"):
        assert R.bits_of(bi.batch_invariant_matmul(x, w.T, path=path, awaiting=aw)) == want
    if K % 64 == 0:
        q = quantize_rows(w, 64, 4)
        run = lambda **kw: R.bits_of(bi.batch_invariant_quantized_matmul(x, *q, group_size=64, bits=4, **kw))
        want = run(path="fused")
        assert run(path="pair", awaiting=aw) == want and run(awaiting=aw) == want
    bi.check_device_status()


def test_a_flag_that_nothing_raises_ends_the_pair_kernel(bi):
    x, w = _xw(300, 4096, 1024)
    flags = torch.zeros(8, dtype=torch.int32, device="cuda")
    epoch = torch.tensor([3], dtype=torch.int32, device="cuda")
    bi.check_device_status()
    t0 = time.perf_counter()
    bi.batch_invariant_matmul(x, w.T, path="pair", awaiting=(flags.data_ptr(), epoch.data_ptr(), 0, 2))
    torch.cuda.synchronize()
    waited = time.perf_counter() - t0
    assert 1.5 < waited < 30, waited
    with pytest.raises(_lib.KernelError, match="0x20103"):                # 0x20000 | peer 1 << 8 | epoch 3
        bi.check_device_status()
    assert R.bits_of(bi.batch_invariant_matmul(x, w.T, path="pair")) == R.bits_of(bi.batch_invariant_matmul(x, w.T, path="fused"))
    bi.check_device_status()
