"""v5 WKV op (per-head 64x64 fp32 state, static per-channel decay).

Two interfaces over the same kernels:

``WKV5.apply(B,T,C,H,r,k,v,w,u,state_in) -> (y, state_out)``
    the full contract: differentiable w.r.t. r,k,v,w,u and state_in, accepts a
    gradient on state_out.  ``w`` is the raw ``time_decay`` (decay =
    exp(-exp(w))), state is fp32 ``[B,H,N,N]`` indexed [key,value] like
    rwkv_inner's kv_state (RWKV-v5/src/module/rwkv_inner.py:22).

``WKV5_CUDA`` / ``RUN_WKV5_CUDA`` / ``wkv5_cuda_kernel``
    name-for-name mirrors of RWKV-v5/src/module/TimeMix.py:20-154 and of the
    extension module bound in RWKV-v5/src/module/cuda/wkv5_op.cpp:124-142:
    same argument order, outputs pre-allocated by the caller, ``state`` mutated
    in place in the project kernels' [value,key] layout, no state gradient.
    Unlike the project's kernel the state is indexed per batch row.
"""
from __future__ import annotations

import torch

from . import _lib as L
from . import wkv56

N = wkv56.HEAD_SIZE


class WKV5:
    @staticmethod
    def apply(B, T, C, H, r, k, v, w, u, state_in, path=L.WKV_PATH_AUTO, saved=None):
        return wkv56.apply("wkv5", B, T, C, H, r, k, v, w, u, state_in, path, saved)


def wkv5(r, k, v, w, u, state_in, path=L.WKV_PATH_AUTO):
    """Convenience form of ``WKV5.apply`` taking the sizes from ``r`` and ``u``."""
    B, T, C = r.shape
    return WKV5.apply(B, T, C, C // N, r, k, v, w, u, state_in, path)


# ----------------------------------------------------------------------------
# literal drop-ins


class _Wkv5Kernel:
    """Stand-in for the project's ``wkv5`` extension module (wkv5_op.cpp:124-142)."""

    @staticmethod
    def _fwd(dt, B, T, C, H, state, r, k, v, eew, u, y):
        for t in (r, k, v, u, y):
            if t.dtype != dt:
                raise TypeError(f"expected {dt} tensors")
        if state.dtype != torch.float32 or eew.dtype != torch.float32:
            raise TypeError("state and w must be float32")
        ew = torch.log(eew.float()).contiguous()
        y_new, _ = wkv56.forward("wkv5", r, k, v, ew, u, state, w_kind=L.WKV_W_NEGEXP,
                                 layout=L.WKV_STATE_VK, state_out=state)
        y.copy_(y_new)

    @staticmethod
    def _bwd(dt, B, T, C, H, state, r, k, v, eew, ew, u, gy, gr, gk, gv, gw, gu):
        for t in (r, k, v, u, gy):
            if t.dtype != dt:
                raise TypeError(f"expected {dt} tensors")
        a, b, c, d, e, _ = wkv56.backward("wkv5", r, k, v, ew.float().contiguous(), u, state, gy,
                                          None, w_kind=L.WKV_W_NEGEXP, layout=L.WKV_STATE_VK,
                                          want_gstate=False)
        gr.copy_(a); gk.copy_(b); gv.copy_(c); gw.copy_(d.view_as(gw)); gu.copy_(e.view_as(gu))

    def forward_bf16(self, *a): self._fwd(torch.bfloat16, *a)
    def forward_fp16(self, *a): self._fwd(torch.float16, *a)
    def forward_fp32(self, *a): self._fwd(torch.float32, *a)
    def backward_bf16(self, *a): self._bwd(torch.bfloat16, *a)
    def backward_fp16(self, *a): self._bwd(torch.float16, *a)
    def backward_fp32(self, *a): self._bwd(torch.float32, *a)


wkv5_cuda_kernel = _Wkv5Kernel()


class WKV5_CUDA:
    """RWKV-v5/src/module/TimeMix.py:20-143: ``apply(B,T,C,H,state,r,k,v,w,u) -> y``;
    ``state`` (fp32, [B,H,value,key]) is updated in place; no gradient flows to it."""

    @staticmethod
    def apply(B, T, C, H, state, r, k, v, w, u):
        return wkv56.apply_dropin("wkv5", B, T, C, H, r, k, v, w, u, state)


def RUN_WKV5_CUDA(B, T, C, H, state, r, k, v, w, u):
    """RWKV-v5/src/module/TimeMix.py:145-154."""
    return WKV5_CUDA.apply(B, T, C, H, state, r, k, v, w, u)
