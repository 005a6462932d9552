"""Which packed batches are unpacked for pairs of SMs, as the scratch query tells: no GPU needed (148 SMs are assumed)."""

import pytest

from mlx_batch_invariant_b200 import _lib


@pytest.mark.parametrize("M,N,K,pair", [
    (200, 4096, 14336, False), (220, 4096, 14336, False),          # a long K: one SM per tile is as fast or faster
    (300, 4096, 14336, True), (300, 4096, 4096, True), (128, 4864, 896, True), (2048, 896, 896, True), (128, 6144, 4096, True),
    (200, 4096, 4096, False), (65, 14336, 4096, False),
])
def test_packed_batches_on_pairs_of_sms(M, N, K, pair):
    need = _lib.load().bi_qmm_scratch_bytes(M, N, K, _lib.BI_BF16)
    assert need == (_lib.COUNTER_BYTES + 2 * N * K if pair else 0)
