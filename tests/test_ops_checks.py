"""Calls the tensor-level entry points refuse, by checks that come before any device is touched."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from racetrack_b200 import _lib, moe, ops


def _experts(hidden=128, inter=64, count=4):
    u8 = lambda *s: torch.zeros(*s, dtype=torch.uint8)
    return SimpleNamespace(
        w13_codes=u8(count * 2 * inter, hidden // 2), w13_sf=u8(count * 2 * inter * hidden // 16), w13_gs=torch.ones(count),
        w2_codes=u8(count * hidden, inter // 2), w2_sf=u8(count * hidden * inter // 16), w2_gs=torch.ones(count),
        count=count, inter=inter)


def _routing(tokens, topk=2):
    return torch.ones(tokens, topk), torch.zeros(tokens, topk, dtype=torch.int64)


X = torch.zeros(16, 128, dtype=torch.bfloat16)
CODES, SF, GS = torch.zeros(16, 64, dtype=torch.uint8), torch.zeros(16, 8, dtype=torch.uint8), torch.ones(1)


@pytest.mark.parametrize("x,x_quant,rows,says", [
    (X.view(1, 16, 128), None, 16, "x must be"),                          # a batch dimension
    (X[0], None, 1, "x must be"),
    (None, (CODES.view(1, 16, 64), SF, GS), 16, "x must be"),
    (None, None, 16, "is required"),
    (None, (CODES, None, GS), 16, "is required"),
    (X, None, 17, "disagree"),                                            # more routed rows than x has
])
def test_expert_mlp_refuses_what_it_cannot_index(x, x_quant, rows, says):
    weights, indices = _routing(rows)
    with pytest.raises(RuntimeError, match=says):
        moe.fused_moe_experts(x, weights, indices, _experts(), n_experts=4, x_quant=x_quant)


def test_expert_mlp_refuses_weights_of_other_tokens():
    weights, indices = _routing(16)
    for bad in (_routing(17)[0], _routing(16, 3)[0], weights.view(-1)):
        with pytest.raises(RuntimeError, match="disagree"):
            moe.fused_moe_experts(X, bad, indices, _experts(), n_experts=4)


@pytest.mark.parametrize("call", [
    lambda: ops.fused_rope_half(torch.zeros(2, 3, 64), None),
    lambda: ops.fused_rope(torch.zeros(2, 3, 64), None),
    lambda: ops.fused_norm_rope(X, X[0], X, X[0], X, None, eps=1e-6, rope_base=1e4),
    lambda: ops.fused_norm_rope_interleaved(X, X[0], X, X[0], X, None, eps=1e-6),
    lambda: ops.fused_act_quant(X, out=(X, None)),
    lambda: ops.fused_act_quant(X, out=(None, X)),
    lambda: ops.fused_nvfp4_quant(X, out=(X, None)),
    lambda: ops.fused_moe_route(torch.zeros(2, 8), None, n_groups=1, topk_groups=1, topk=2, route_scale=1.0,
                                out=(torch.zeros(2, 2), None)),
])
def test_a_missing_tensor_is_refused(call):
    """A None where a tensor belongs raises; it is not dereferenced."""
    with pytest.raises(RuntimeError, match="is missing|must be a pair"):
        call()


@pytest.mark.parametrize("offset", [None, 3, 3.0, torch.tensor(3.0)])
def test_numbers_of_any_kind_are_taken(offset):
    """A causal offset that int() takes gets past the conversion (to the check for CUDA tensors)."""
    z = torch.zeros
    with pytest.raises(RuntimeError, match="need CUDA"):
        ops.fp8_index(z(1, 2, 4, 128), z(1, 2, 4), z(1, 5, 128), z(1, 5), causal_offset=offset)


@pytest.mark.parametrize("n,k", [(256, 7168), (2112, 7168), (7168, 16384), (1024, 2048)])
def test_no_product_of_more_than_128_rows_is_cut_along_k(n, k):
    """What the bit-identity of token-sharded layers rests on: a rank's rows and all rows are summed alike."""
    lib = _lib.load()
    for m in (129, 256, 512, 777, 8192):
        assert lib.rt_gemm_bf16_splitk_splits(m, n, k) == 1
        assert lib.rt_gemm_fp8_workspace_bytes(m, n, k) == 0
