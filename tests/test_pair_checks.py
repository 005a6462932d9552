"""What the pair shape of the matmuls refuses, before any CUDA call: no GPU needed."""

import ctypes

import pytest
import torch

from mlx_batch_invariant_b200 import _lib
from mlx_batch_invariant_b200.kernels.matmul import _launch_shape

P = 4096                                     # a pointer that is aligned and never followed
PAIR = _lib.PATH_PAIR


@pytest.mark.parametrize("dtype,b_sk,b_sn,K", [(_lib.BI_F32, 1, 512, 512), (_lib.BI_BF16, 64, 1, 512), (_lib.BI_BF16, 1, 515, 515)])
def test_dense_weights_off_the_tensor_core_path(dtype, b_sk, b_sn, K):
    for ws_bytes in (0, 1 << 30):
        rc = _lib.load().bi_matmul(P, P, P, P, ws_bytes, 100, 64, K, K, 1, b_sk, b_sn, dtype, PAIR, None, None)
        assert rc == _lib.BI_ERR_UNSUPPORTED and "pair" in _lib.last_error()


@pytest.mark.parametrize("dtype,K", [(_lib.BI_F32, 512), (_lib.BI_BF16, 544)])
def test_packed_weights_off_the_tensor_core_path(dtype, K):
    for ws_bytes in (0, 1 << 30):
        rc = _lib.load().bi_qmm(P, P, P, P, P, P, ws_bytes, 100, 64, K, K, 32, 4, dtype, PAIR, None, None)
        assert rc == _lib.BI_ERR_UNSUPPORTED and "pair" in _lib.last_error()


def test_pushing_and_rotating_calls():
    L, two = _lib.load(), (ctypes.c_void_p * 2)(P, P)
    path = PAIR | _lib.batch_tile(48)
    rope = (P, P, P, P, P, P, 4, 1, 2, 1, 128, 512, 512, 128, 4)
    calls = [L.bi_matmul_push(P, P, P, 1 << 30, 4, 512, 512, 512, 1, 1, 512, _lib.BI_BF16, path, None, None, None, None, two, two, P, 0, 2, 0),
             L.bi_qmm_push(P, P, P, P, P, 1 << 30, 4, 512, 512, 512, 64, 4, _lib.BI_BF16, path, None, None, None, None, two, two, P, 0, 2, 0),
             L.bi_matmul_rope(P, P, P, 1 << 30, 4, 512, 512, 512, 1, 1, 512, _lib.BI_BF16, path, None, None, *rope),
             L.bi_qmm_rope(P, P, P, P, P, 1 << 30, 4, 512, 512, 512, 64, 4, _lib.BI_BF16, path, None, None, *rope)]
    assert calls == [_lib.BI_ERR_BAD_ARG] * 4


@pytest.mark.parametrize("tile", [1, 16, 31, 33, 48, 257, 288, 544])
def test_batch_tiles_that_are_no_multiple_of_32_up_to_256(tile):
    with pytest.raises(_lib.KernelError) as e:
        _launch_shape("pair", tile, 300, 512, 1024, 0, torch.device("cpu"))
    assert e.value.code == _lib.BI_ERR_BAD_ARG
