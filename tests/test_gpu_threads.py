"""Calls from several Python threads."""
from __future__ import annotations

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_call_lets_other_python_threads_run():
    """The interpreter lock is not held while the library is called (a launch may block on a full queue).
    PyGILState_Check takes the place of a few library functions: its 1 for "held" reads as an error."""
    from racetrack_b200 import _lib, ops
    native, lib = _lib.native(), _lib.load()
    names = ("rt_rms_norm", "rt_swiglu", "rt_absmax", "rt_gemm_bf16", "rt_moe_route", "rt_moe_plan")
    addresses = {n: ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in native.table()}
    held = ctypes.cast(ctypes.pythonapi.PyGILState_Check, ctypes.c_void_p).value
    x = torch.zeros(4, 128, device="cuda", dtype=torch.bfloat16)
    bias = torch.zeros(8, device="cuda")
    try:
        native.bind({**addresses, **dict.fromkeys(names, held)})
        ops.fused_rms_norm(x, x[0], eps=1e-6)
        ops.fused_swiglu(x, x)
        ops.tensor_absmax(x)
        ops.linear_bf16(x[:, :8].contiguous(), x[:, :8].contiguous())
        ops.fused_moe_route(torch.zeros(4, 8, device="cuda"), bias, n_groups=1, topk_groups=1, topk=2, route_scale=1.0)
    finally:
        native.bind(addresses)
    ops.fused_rms_norm(x, x[0], eps=1e-6)
    torch.cuda.synchronize()
