"""Chains of calls in a captured graph take no longer with overlapped launches than with plain ones: a kernel that is let in
beside a running one may find its CTAs packed on the SMs that came free first."""

import pytest
import torch

import mlx_batch_invariant_b200 as bi

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype=torch.float32):
    return torch.randn(*shape, device="cuda").to(dtype) * shape[-1] ** -0.5


def _linear(M, K, N, dtype=torch.float32, row_major=False):
    x, w = _rand(M, K, dtype=dtype), _rand(K, N, dtype=dtype) if row_major else _rand(N, K, dtype=dtype).T
    return lambda: bi.batch_invariant_matmul(x, w)


def _norm_linears(M, dtype=torch.float32, row_major=False):
    """A norm, and one or two linears on what it wrote."""
    x, up, down = _rand(M, 896, dtype=dtype), _rand(4864, 896, dtype=dtype).T, _rand(896, 4864, dtype=dtype).T
    if row_major:
        up = up.contiguous()
        return lambda: bi.batch_invariant_matmul(bi.batch_invariant_rms_norm(x, None, 1e-5), up)
    return lambda: bi.batch_invariant_matmul(bi.batch_invariant_matmul(bi.batch_invariant_rms_norm(x, None, 1e-5), up), down)


def _behind_another_linear(M, K, N):
    other, call = _linear(64, 896, 896, torch.bfloat16), _linear(M, K, N)
    return lambda: (other(), call())


def _decode(B, L, dtype, heads=14, kv_heads=2, dim=64):
    q, k, v = _rand(B, heads, 1, dim, dtype=dtype), *(_rand(B, kv_heads, L, dim, dtype=dtype) for _ in range(2))
    return lambda: bi.batch_invariant_decode_attention(q, k, v, scale=dim ** -0.5)


def _decode_behind_a_linear():
    x, w, attend = _rand(64, 896, dtype=torch.bfloat16), _rand(896, 896, dtype=torch.bfloat16).T, _decode(64, 561, torch.bfloat16)
    return lambda: (bi.batch_invariant_matmul(bi.batch_invariant_rms_norm(x, None, 1e-5), w), attend())


def _prefill_behind_a_linear(T):
    x, w = _rand(T, 896, dtype=torch.bfloat16), _rand(896, 896, dtype=torch.bfloat16).T
    q, k, v = _rand(1, 14, T, 64, dtype=torch.bfloat16), *(_rand(1, 2, T, 64, dtype=torch.bfloat16) for _ in range(2))
    return lambda: (bi.batch_invariant_matmul(x, w), bi.batch_invariant_attention(q, k, v, scale=0.125, mask="causal"))


def _norm(rows, dim, dtype, op=bi.batch_invariant_rms_norm):
    x, w = _rand(rows, dim, dtype=dtype), torch.ones(dim, device="cuda", dtype=dtype)
    return (lambda: op(x, w, w, 1e-5)) if op is bi.batch_invariant_layer_norm else (lambda: op(x, w, 1e-5))


CHAINS = {
    "fp32 few rows": lambda: _linear(2, 2048, 2048),
    "fp32 9 x 4096 -> 4096": lambda: _linear(9, 4096, 4096),
    "fp32 128 x 2048 -> 2048": lambda: _linear(128, 2048, 2048),
    "fp32 in element-wise fetches": lambda: _linear(128, 897, 1001),
    "fp32 norm and linears": lambda: _norm_linears(32),
    "fp32 behind a 16-bit linear": lambda: _behind_another_linear(64, 2048, 2048),
    "bf16 in element-wise fetches": lambda: _linear(16, 4092, 4096, torch.bfloat16),
    "bf16 norm and row-major linear": lambda: _norm_linears(16, torch.bfloat16, True),
    "bf16 decode attention": lambda: _decode(64, 561, torch.bfloat16),
    "fp32 decode attention": lambda: _decode(64, 561, torch.float32),
    "bf16 decode attention behind a linear": _decode_behind_a_linear,
    "bf16 norm of 1200 rows": lambda: _norm(1200, 4096, torch.bfloat16),
    "fp32 norm of 1200 rows": lambda: _norm(1200, 896, torch.float32),
    "bf16 LayerNorm of 300 rows": lambda: _norm(300, 4096, torch.bfloat16, bi.batch_invariant_layer_norm),
    "bf16 prefill attention behind a linear": lambda: _prefill_behind_a_linear(512),
    "short bf16 prefill attention behind a linear": lambda: _prefill_behind_a_linear(100),
    "fp32 16 x 2048 -> 2048": lambda: _linear(16, 2048, 2048),
}


def _times(make, monkeypatch):
    """Shortest replay of 16 calls, overlapped and plain, taken in turn."""
    call, graphs = make(), []
    for switch in (None, "0"):
        monkeypatch.delenv("BI_PDL", raising=False) if switch is None else monkeypatch.setenv("BI_PDL", switch)
        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(16):
                call()
        graphs.append(graph)
    best = [float("inf")] * 2
    begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    for _ in range(20):
        for i, graph in enumerate(graphs):
            begin.record()
            graph.replay()
            end.record()
            end.synchronize()
            best[i] = min(best[i], begin.elapsed_time(end))
    return best


@pytest.mark.parametrize("name", CHAINS)
def test_overlap_costs_no_chain_its_time(name, monkeypatch):
    overlapped, plain = _times(CHAINS[name], monkeypatch)
    assert overlapped < 1.1 * plain, (overlapped, plain)      # packed on some SMs: 1.1 (few rows) to 1.8 times
