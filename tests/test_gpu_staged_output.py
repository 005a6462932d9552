"""Matmul outputs that leave by TMA (rows of whole 16-byte units) have the bits of outputs the threads store, and nothing
beyond the output is written: ragged rows and columns, tiles of one CTA that follow one another, an output that is not aligned."""

import pytest
import torch

import mlx_batch_invariant_b200 as bi
from mlx_batch_invariant_b200 import _lib

pytestmark = pytest.mark.gpu
GUARD = 4096


def call(x, w, path, offset):
    """bi_matmul into a buffer of sentinels: (output, whether the sentinels around it are untouched)."""
    M, K, N = x.shape[0], x.shape[1], w.shape[0]
    buf = torch.full((GUARD + offset + M * N + GUARD,), 777.0, device="cuda", dtype=x.dtype)
    out = buf[GUARD + offset:GUARD + offset + M * N]
    G = (K + 255) // 256
    ws = torch.full((G * M * N + GUARD,), 777.0, device="cuda", dtype=torch.float32)
    _lib.check(_lib.load().bi_matmul(x.data_ptr(), w.data_ptr(), out.data_ptr(), ws.data_ptr(), G * M * N * 4, M, N, K, K, 1, 1, K,
                                     _lib.DTYPE_CODE[x.dtype], path, _lib.status_word(x.device).data_ptr(), _lib.stream_ptr(x.device)))
    clean = bool((buf[:GUARD + offset] == 777.0).all() and (buf[GUARD + offset + M * N:] == 777.0).all() and (ws[G * M * N:] == 777.0).all())
    return out.view(M, N), clean


# (M, N, K, batch tile): rows and columns that end inside a piece, a half, a tile, a second CTA; several units a pair
@pytest.mark.parametrize("M,N,K,bm", [(257, 520, 512, 256), (33, 136, 256, 32), (1000, 2304, 320, 32), (2000, 4616, 512, 256), (511, 264, 768, 160)])
def test_pairs_of_sms(M, N, K, bm):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = torch.randn(M, K, device="cuda", generator=g).bfloat16(), torch.randn(N, K, device="cuda", generator=g).bfloat16()
    ref = torch.cat([bi.batch_invariant_matmul(x[i:i + 1], w.T) for i in range(0, M, 97)])
    for offset in (0, 8, 1):                       # elements: the last leaves the output misaligned
        out, clean = call(x, w, _lib.PATH_PAIR | _lib.batch_tile(bm // 2), offset)
        assert clean and torch.equal(out[::97], ref)
    _lib.check_device_status()
