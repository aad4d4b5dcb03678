"""state_out may be the memory of state_in (the drop-in wrappers update the state in place): the same bits as with
buffers of their own, wherever the starting states of a chain's groups of chunks come from -- one group, groups folded by
their own CTAs, groups scanned by a kernel of its own, the token-serial kernels."""
import numpy as np
import pytest
import torch

import wkv_testlib as TL
import test_chunked_gpu as CG

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("variant", ["v5", "v6"])
@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("B,H,T,groups", [(1, 2, 65, 2), (3, 40, 1024, 16), (2, 64, 500, 4), (1, 2, 17 * 64, 17), (2, 3, 200, 1), (2, 3, 20, 0)])
def test_in_place_equals_separate_buffers(variant, layout, B, H, T, groups):
    W, wkv56 = CG._pkg()
    name = "wkv6" if variant == "v6" else "wkv5"
    g = torch.Generator(device="cuda").manual_seed(T + groups)
    C = H * 64
    normal = lambda *s: torch.randn(s, generator=g, device="cuda")
    r, k, v = (normal(B, T, C).to(BF) for _ in range(3))
    w = (normal(B, T, C) * 0.5 - 0.6).to(BF) if variant == "v6" else -1.0 - 5.0 * torch.rand((H, 64), generator=g, device="cuda")
    u, s0 = normal(H, 64).to(BF), normal(B, H, 64, 64)
    kw = dict(w_kind=W.WKV_W_RAW, layout=layout, time_groups=groups)
    y, s1 = wkv56.forward(name, r, k, v, w, u, s0, **kw)
    for _ in range(3):
        state = s0.clone()
        y2, s2 = wkv56.forward(name, r, k, v, w, u, state, state_out=state, **kw)
        assert s2.data_ptr() == state.data_ptr()
        assert torch.equal(y2, y) and torch.equal(state, s1)
    # against the same call with the caller's zero state left out
    y3, s3 = wkv56.forward(name, r, k, v, w, u, torch.zeros_like(s0), **kw)
    y4, s4 = wkv56.forward(name, r, k, v, w, u, None, **kw)
    assert torch.equal(y3, y4) and torch.equal(s3, s4)


@pytest.mark.parametrize("variant", ["v5", "v6"])
def test_dropin_wrapper_over_several_groups(variant):
    """the wrapper's in-place state on a segment the library cuts into groups by itself, against the oracle"""
    W, wkv56 = CG._pkg()
    B, T, H = 1, 1003, 2
    C = H * 64
    q = TL.case56(variant, B, T, H, BF, seed=61, gstate=False)
    want = CG.floored_oracle(variant, q)
    d = {n: TL.to_dev(q[n], BF).requires_grad_(True) for n in ("r", "k", "v", "u")}
    s = TL.to_dev(np.swapaxes(q["state_in"], -1, -2), torch.float32)
    w = TL.to_dev(q["x"], BF if variant == "v6" else torch.float32).requires_grad_(True)
    y = (W.RUN_WKV6STATE_CUDA(B, T, C, H, d["r"], d["k"], d["v"], w, d["u"], s) if variant == "v6"
         else W.RUN_WKV5_CUDA(B, T, C, H, s, d["r"], d["k"], d["v"], w, d["u"]))
    y.backward(TL.to_dev(q["gy"], BF))
    TL.assert_close("y", y, want["y"], 2e-2)
    TL.assert_close("state", np.swapaxes(TL.back(s), -1, -2), want["state_out"], 2e-2)
    for n in ("r", "k", "v"):
        TL.assert_close("g" + n, d[n].grad, want["g" + n], 2e-2)
