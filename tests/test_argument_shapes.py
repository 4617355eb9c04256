"""Shapes that the one-call operators refuse before anything reaches the device (no GPU: the checks come first)."""
import pytest
import torch

import triteia_b200.ops as ops

T, K, N, D, M, R = 3, 256, 384, 2, 4, 16


def _inputs():
    q = torch.zeros(D, K // 32, 2 * N, dtype=torch.int32)
    meta = torch.zeros(D, N, K // 16, dtype=torch.int16)
    s = torch.zeros(D, K // 128, N, dtype=torch.float16)
    x, idx = torch.zeros(T, K, dtype=torch.float16), torch.zeros(T, dtype=torch.int32)
    return x, idx, q, meta, s


@pytest.mark.parametrize("base", [(N - 128, K), (N + 128, K), (N, K - 64), (N, K + 64)])
def test_sbmm_refuses_a_base_weight_that_does_not_fit_the_deltas(base):
    x, idx, q, meta, s = _inputs()
    with pytest.raises(RuntimeError, match="the deltas and inputs need"):
        ops.sbmm_4bit_2_4_native(q, x, meta, s, idx, base_weight=torch.zeros(base, dtype=torch.float16))


@pytest.mark.parametrize("base,a,b", [
    ((N - 128, K), (M, K, R), (M, R, N)),
    ((N, K - 64), (M, K, R), (M, R, N)),
    ((N, K), (M, K - 64, R), (M, R, N)),
    ((N, K), (M, K, R), (M - 1, R, N)),
    ((N, K), (M, K, R), (M, R - 8, N)),
    ((N, K), (M, K, R), (M, R, N - 8)),
])
def test_ldmm_refuses_weights_that_do_not_fit_the_deltas(base, a, b):
    x, idx, q, meta, s = _inputs()
    half = dict(dtype=torch.float16)
    with pytest.raises(RuntimeError, match="the deltas and inputs need"):
        ops.ldmm(idx, x, torch.zeros(a, **half), torch.zeros(b, **half), q, meta, s, base_weight=torch.zeros(base, **half))
