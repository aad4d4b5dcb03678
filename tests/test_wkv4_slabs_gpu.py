"""The time-parallel v4 kernels at the edges of what they cut the tokens and channels into: tiles of 8 tokens,
slabs of 64, 128 and 256, channel blocks of 16, rows that are and are not 16-byte aligned, with and without
the hand-over from forward to backward."""
import numpy as np
import pytest
import torch

import inputs
import wkv_testlib as TL
from oracle import wkv_oracle as O

pytestmark = pytest.mark.gpu


def spread(c, how):
    """keys, bonus and decay that leave the range one reference exponent per tile can hold, for some channels and tokens"""
    if how == "wild":
        c["k"][:, ::5, ::3] += 70.0
        c["k"][:, 3::7, 1::3] -= 90.0
        c["u"][2::4] *= 50.0
        c["td"][1::5] = 3.0
    return c


@pytest.mark.parametrize("how", ["plain", "wild"])
@pytest.mark.parametrize("B,T,C,dtype", [
    (1, 16, 16, torch.float32), (2, 17, 24, torch.bfloat16), (1, 63, 40, torch.float32), (2, 64, 20, torch.bfloat16),
    (1, 65, 7, torch.float32), (1, 129, 9, torch.float32), (1, 127, 16, torch.float32), (1, 128, 32, torch.bfloat16), (3, 257, 48, torch.float32),
    (1, 511, 16, torch.bfloat16), (2, 300, 1, torch.float32), (4, 200, 1264, torch.float32), (8, 136, 1200, torch.bfloat16),
    (8, 260, 960, torch.float32), (8, 256, 960, torch.bfloat16), (4, 130, 2384, torch.float32)])
def test_v4_matches_oracle(B, T, C, dtype, how):
    import rwkv_infctx_trainer_b200 as W
    from rwkv_infctx_trainer_b200 import _lib as L
    c = spread(inputs.wkv4_case(B, T, C, seed=800 + T), how)
    d = {n: TL.to_dev(c[n], dtype) for n in ("u", "k", "v", "gy")}
    td = TL.to_dev(c["td"], torch.float32)
    f64 = lambda t: t.detach().float().cpu().double().numpy()
    w64 = -np.exp(f64(td))
    s0 = np.stack([inputs.normal((B, C), 1, stream=40), inputs.uniform((B, C), 1, 0.5, 2.0, stream=41),
                   inputs.normal((B, C), 1, stream=42)], -1)
    gs = np.stack([inputs.normal((B, C), 1, stream=43), inputs.normal((B, C), 1, stream=44),
                   inputs.uniform((B, C), 1, -1.0, 0.0, stream=45)], -1)
    s0, gs = TL.to_dev(s0, torch.float32), TL.to_dev(gs, torch.float32)
    yo, so = O.wkv4_fwd(w64, f64(d["u"]), f64(d["k"]), f64(d["v"]), f64(s0))
    g = O.wkv4_bwd(w64, f64(d["u"]), f64(d["k"]), f64(d["v"]), f64(s0), f64(d["gy"]), f64(gs))
    tol = TL.TOL[dtype]
    state = lambda t: (f64(t)[..., :2] * np.exp(f64(t)[..., 2:])) if torch.is_tensor(t) else t[..., :2] * np.exp(t[..., 2:])

    leaves = [t.clone().requires_grad_(True) for t in (td, d["u"], d["k"], d["v"], s0)]
    y, s1 = W.wkv_op(*leaves)
    got = torch.autograd.grad((y, s1), leaves, (d["gy"], gs))
    TL.assert_close("y", y, yo, tol)
    TL.assert_close("state", state(s1), state(so), tol)
    for n, a, b in (("gw", got[0], g["gw"].sum(0)), ("gu", got[1], g["gu"].sum(0)), ("gk", got[2], g["gk"]), ("gv", got[3], g["gv"]),
                    ("gstate", state(got[4]), state(g["gstate_in"]))):
        TL.assert_close(n, a, b, tol)

    # without a hand-over, through the C ABI
    lib, st = L.load(), torch.cuda.current_stream().cuda_stream
    w = -torch.exp(td)
    o = {n: torch.empty_like(d["k"]) for n in ("gk", "gv")}
    gw, gu, gsi = torch.empty((B, C), device="cuda"), torch.empty((B, C), device="cuda"), torch.empty_like(s0)
    n = lib.wkv4_backward_workspace(B, T, C)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    L.check(lib.wkv4_backward(B, T, C, L.DTYPE_CODE[dtype], w.data_ptr(), d["u"].data_ptr(), d["k"].data_ptr(), d["v"].data_ptr(),
                              s0.data_ptr(), d["gy"].data_ptr(), gs.data_ptr(), gw.data_ptr(), gu.data_ptr(), o["gk"].data_ptr(),
                              o["gv"].data_ptr(), gsi.data_ptr(), ws.data_ptr(), n, st), "wkv4_backward")
    for n, a, b in (("gw", gw, g["gw"]), ("gu", gu, g["gu"]), ("gk", o["gk"], g["gk"]), ("gv", o["gv"], g["gv"]),
                    ("gstate", state(gsi), state(g["gstate_in"]))):
        TL.assert_close("no hand-over " + n, a, b, tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [20, 200])
def test_tensors_that_start_on_an_odd_element(dtype, T):
    """any one tensor of a call (the bonus, an input, an output, the hand-over) off its 16-byte boundary: the same result
    as with all of them on it, up to the order of fp32 operations"""
    from rwkv_infctx_trainer_b200 import _lib as L
    B, C = 2, 48
    lib, st, code = L.load(), torch.cuda.current_stream().cuda_stream, L.DTYPE_CODE[dtype]
    c = inputs.wkv4_case(B, T, C, seed=850 + T)
    src = {n: TL.to_dev(c[n], dtype) for n in ("u", "k", "v", "gy")}
    w = TL.to_dev(-np.exp(c["td"]), torch.float32)
    nck, nws = lib.wkv4_state_ckpt_bytes(B, T, C), lib.wkv4_backward_workspace(B, T, C)
    nfw = lib.wkv4_forward_workspace(B, T, C)

    def place(t, odd):
        buf = torch.empty(t.numel() + 8, device="cuda", dtype=t.dtype)
        out = buf[1:1 + t.numel()] if odd else buf[:t.numel()]
        out.copy_(t.flatten())
        return out

    def run(odd):
        t = {n: place(x, n == odd) for n, x in src.items()}
        o = {n: place(torch.zeros_like(src["k"]), n == odd) for n in ("y", "gk", "gv")}
        o.update({n: place(torch.zeros((B, C), device="cuda"), n == odd) for n in ("gw", "gu")})
        ck = place(torch.zeros(max(nck // 4, 1), device="cuda"), odd == "ckpt")
        ws = place(torch.zeros(max(nws, nfw) // 4, device="cuda"), odd == "ws")
        p = lambda x: x.data_ptr()
        hand = [(p(ck), nck)] if nck else []
        for args in hand + [(None, 0)]:          # with a hand-over, then without
            assert lib.wkv4_forward_ckpt(B, T, C, code, p(w), p(t["u"]), p(t["k"]), p(t["v"]), None, p(o["y"]), None, p(ws), ws.numel() * 4, *args, st) == 0
            assert lib.wkv4_backward_ckpt(B, T, C, code, p(w), p(t["u"]), p(t["k"]), p(t["v"]), None, p(t["gy"]), None, p(o["gw"]), p(o["gu"]), p(o["gk"]),
                                          p(o["gv"]), None, p(ws), ws.numel() * 4, *args, st) == 0
            yield {n: x.clone() for n, x in o.items()}

    # fp32 values: a chain of T steps of about four roundings of 2^-24 each; bf16: one rounding may fall the other way
    tol = {True: 4 * 200 * 2.0 ** -24, False: 2.0 ** -7}
    for odd in ("u", "k", "v", "gy", "y", "gk", "gv", "gw", "gu", "ckpt", "ws"):
        for a, b in zip(run(odd), run(None)):
            for n in a:
                TL.assert_close(f"{n} with {odd} moved", a[n], TL.back(b[n]), tol[dtype == torch.float32 or n in ("gw", "gu")])
