"""The elementwise neighbours of the WKV op in the time-mix block, each one fused CUDA pass.

``lnx_gate(y, g, weight, bias, eps, n_head)``
    ``ln_x(y.view(-1,C)).view(B,T,C) * g`` of RWKV-v6/src/module/TimeMix.py:296-298
    (``ln_x = nn.GroupNorm(n_head, C, eps=...)``), differentiable w.r.t. y, g, weight, bias.

``ddlerp(x, shift, maa, m=None)``
    the token-shift mixes of RWKV-v6/src/module/TimeMix.py:262-273:
    ``x + (x_prev - x) * (maa[i] + m[i])`` for every i, with ``x_prev`` the previous token
    (``shift`` [B,C] before a row's first token).  ``maa`` [n,C], ``m`` [n,B,T,C] or None,
    n = 1, 3, 4 or 5; returns [n,B,T,C].  Differentiable w.r.t. x, shift, maa, m.

bf16 tensors only (the dtype the trainer runs these in); parameters may have any float dtype.
"""
from __future__ import annotations

from . import _lib as L


def lnx_gate(y, g, weight, bias, eps, n_head):
    return L.native().lnx_gate(y, g, weight, bias, float(eps), n_head)


def ddlerp(x, shift, maa, m=None):
    return L.native().ddlerp(x, shift, maa, m)
