"""v4 WKV op: drop-in for RWKV-v4neo's ``torch.ops.rwkv.wkv``.

Mirrors, name for name, the host interface of RWKV-infctx-trainer's v4 path:
  * ``WKVFunction`` / ``wkv``  -- RWKV-v4neo/cuda/wkv_op_bf16.cpp:13-92
  * op registration ``rwkv::wkv(Tensor w, Tensor u, Tensor k, Tensor v,
    Tensor last_state) -> Tensor[]`` -- wkv_op_bf16.cpp:98
  * ``wkv_op(time_decay, time_first, k, v, wkv_state)`` -- RWKV-v4neo/src/model.py:130-132
Beyond the project's kernel: u,k,v may be fp32 or fp16 as well as bf16, and T has
no compile-time limit.
"""
from __future__ import annotations

import torch

from . import _lib as L


class WKVFunction:
    """``apply(time_decay, time_first, k, v, last_state) -> (y, new_state)``, differentiable in all five."""

    @staticmethod
    def apply(raw_w, raw_u, raw_k, raw_v, raw_last_state):
        return tuple(L.native().wkv4(raw_w, raw_u, raw_k, raw_v, raw_last_state))


def wkv(w, u, k, v, last_state):
    """Same as the project's C++ ``wkv``: returns [y, new_state]."""
    return L.native().wkv4(w, u, k, v, last_state)


def wkv_op(time_decay, time_first, k, v, wkv_state):
    """RWKV-v4neo/src/model.py:130-132 (``torch.ops.rwkv.wkv``, without the dispatcher in between)."""
    return L.native().wkv4(time_decay, time_first, k, v, wkv_state)


def register_torch_op() -> None:
    """``rwkv::wkv`` with the schema of wkv_op_bf16.cpp:98 is registered when the native module is
    loaded: ``torch.ops.rwkv.wkv`` resolves to this implementation."""
    L.native()
    torch.ops.rwkv.wkv
