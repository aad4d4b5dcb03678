"""The token-serial kernels at the sizes where they can go wrong: tokens around the staged tile of 8 and the
ring of 4 tiles, both state layouts, head counts that select each of their three shapes, and bf16 forward
calls short enough to run on them (decays floored like the chunked kernels')."""
import numpy as np
import pytest
import torch

import wkv_testlib as TL
import test_chunked_gpu as CG
import test_wkv56_gpu as TW

pytestmark = pytest.mark.gpu


# up to 10 heads x rows: the one-warp shape both ways; 80 to 200: the two-column shape (forward from 12 tokens on, under that
# the four-column shape); 300: the four-column shape
@pytest.mark.parametrize("variant,B,T,H,layout", [
    ("v6", 1, 1, 1, 0), ("v6", 2, 7, 4, 1), ("v6", 1, 8, 8, 0), ("v5", 1, 9, 8, 1), ("v6", 1, 33, 2, 0), ("v5", 2, 41, 2, 0),
    ("v6", 4, 17, 20, 0), ("v6", 4, 9, 30, 1), ("v5", 4, 10, 20, 0), ("v6", 5, 19, 40, 1), ("v5", 5, 9, 40, 0),
    ("v6", 6, 11, 50, 0), ("v5", 6, 13, 50, 1), ("v6", 4, 12, 30, 0), ("v6", 1, 12, 11, 1)])
def test_serial_kernels_match_oracle(variant, B, T, H, layout):
    import rwkv_infctx_trainer_b200 as W
    q = TL.case56(variant, B, T, H, torch.float32, seed=700 + T)
    got = TW.run_abi(variant, q, torch.float32, (W.WKV_STATE_KV, W.WKV_STATE_VK)[layout], W.WKV_W_RAW, W.WKV_PATH_SCALAR)
    TW.compare(variant, got, TL.oracle56(variant, q), torch.float32)


@pytest.mark.parametrize("T", [1, 2, 8, 47, 48, 49])
def test_short_bf16_forward_matches_the_floored_oracle(T):
    """without a hand-over to leave, calls of up to 48 tokens run on the serial kernel; some decays hit the floor"""
    import rwkv_infctx_trainer_b200 as W
    from rwkv_infctx_trainer_b200 import wkv56
    BF = torch.bfloat16
    q = TL.case56("v6", 2, T, 3, BF, seed=720 + T, x_shift=1.5)
    d = {n: TL.to_dev(q[n], BF) for n in ("r", "k", "v", "u", "x")}
    y, s = wkv56.forward("wkv6", d["r"], d["k"], d["v"], d["x"], d["u"], TL.to_dev(q["state_in"], torch.float32), w_kind=W.WKV_W_RAW)
    want = CG.floored_oracle("v6", q)
    TL.assert_close("y", y, want["y"], 2e-2)
    TL.assert_close("state_out", s, want["state_out"], 2e-2 if T > 48 else 1e-3)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("variant", ["v5", "v6"])
def test_bonus_that_starts_on_an_odd_element(variant, dtype):
    """u is [H,64] wherever the caller keeps it: as a slice of a larger buffer it need not start on a pair of elements;
    same numbers, so the same bits"""
    import rwkv_infctx_trainer_b200 as W
    from rwkv_infctx_trainer_b200 import wkv56
    q = TL.case56(variant, 2, 11, 3, dtype, seed=730)
    d = {n: TL.to_dev(q[n], dtype) for n in ("r", "k", "v", "u", "gy")}
    w = TL.to_dev(q["x"], dtype if variant == "v6" else torch.float32)
    s, gs = TL.to_dev(q["state_in"], torch.float32), TL.to_dev(q["gstate_out"], torch.float32)
    buf = torch.zeros(d["u"].numel() + 8, dtype=dtype, device="cuda")
    odd = buf[1:1 + d["u"].numel()].view_as(d["u"])
    odd.copy_(d["u"])
    kw = dict(w_kind=W.WKV_W_RAW, path=W.WKV_PATH_SCALAR)
    name = "wkv6" if variant == "v6" else "wkv5"
    runs = []
    for u in (d["u"], odd):
        y, s1 = wkv56.forward(name, d["r"], d["k"], d["v"], w, u, s, **kw)
        runs.append((y, s1) + tuple(wkv56.backward(name, d["r"], d["k"], d["v"], w, u, s, d["gy"], gs, **kw)))
    for a, b in zip(*runs):
        assert torch.equal(a, b)
