"""The per-chunk backward kernel gives up in the middle of a walk: groups whose second chunk, mild or steep, never gets its
loads unwind after a first one that was done, and the next call works.  (A host-side decision and short waits, nothing that
hangs or faults.)"""
import ctypes

import pytest
import torch

import wkv_testlib as TL

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("steep", [False, True])
def test_unwinding_after_a_first_chunk(steep, monkeypatch):
    import rwkv_infctx_trainer_b200 as W
    from rwkv_infctx_trainer_b200 import _lib as L, wkv56
    monkeypatch.setattr(wkv56, "CHECK_STATUS", True)
    lib = L.load()
    # 448 chunks on 296 groups, 7 a head: a group's first and second chunk have different places in their heads
    B, T, H, skip = 1, 448, 64, 2
    g = torch.Generator(device="cuda").manual_seed(7)
    n = lambda *s, std=1.0, mean=0.0: torch.randn(s, generator=g, device="cuda") * std + mean
    d = {name: n(B, T, 64 * H).to(BF) for name in ("r", "k", "v", "gy")}
    x = n(B, T, 64 * H, std=0.5, mean=-0.6)
    if steep:
        x[:, 64 * skip:64 * (skip + 1)] = 1.3
    d["w"], u = x.to(BF), n(H, 64).to(BF)
    s_in, gso = n(B, H, 64, 64), n(B, H, 64, 64)
    b = wkv56.prepare_backward("wkv6", d["r"], d["k"], d["v"], d["w"], u, s_in, d["gy"], gso, w_kind=W.WKV_W_RAW,
                               path=W.WKV_PATH_CHUNKED)
    b.workspace.zero_()
    assert lib.wkv56_selftest_abort(ctypes.byref(b._a), 1, 1, 2, skip, 20000, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert int(b.workspace[:4].view(torch.int32).item()) & 4
    b.run()
    assert b.status() == 0
    want = wkv56.backward("wkv6", d["r"], d["k"], d["v"], d["w"], u, s_in, d["gy"], gso, w_kind=W.WKV_W_RAW,
                          layout=W.WKV_STATE_KV, path=W.WKV_PATH_SCALAR)
    for name, t in zip(("gr", "gk", "gv", "gw", "gu", "gstate_in"), want):
        TL.assert_close(name, getattr(b, name), TL.back(t), 2e-2)
