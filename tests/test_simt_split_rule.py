"""Which fp32 batches beyond 32 rows are split over their K groups, as the scratch query tells: no GPU needed (148 SMs)."""

import pytest

from mlx_batch_invariant_b200 import _lib


@pytest.mark.parametrize("M,N,K,split", [
    (100, 4096, 4096, True), (256, 14336, 4096, True), (100, 896, 512, True), (600, 4096, 512, True), (1000, 4096, 1024, True),
    (256, 4096, 300, False), (1000, 896, 300, False),                  # K below two whole groups
    (2000, 4096, 512, False), (2000, 4096, 2048, False),               # more than three waves of fused tiles
    (100, 14336, 512, False), (2000, 896, 512, False),                 # two groups, half a wave to a whole one
    (100, 4096, 256, False),                                           # one group
])
def test_fp32_batches_that_split(M, N, K, split):
    G = (K + 255) // 256
    need = _lib.load().bi_matmul_scratch_bytes(M, N, K, _lib.BI_F32)
    assert need == (_lib.COUNTER_BYTES + G * M * N * 4 if split else 0)
