"""Infinite, small and large inputs of the chunked v5/v6 kernels.

The backward kernel reads w, r and k through a product with an identity matrix, in which an infinite element meets the
zeros of its 15 neighbours; states and gradients are scaled by powers of two taken from a mild chunk's decay."""
import numpy as np
import pytest
import torch

import wkv_testlib as TL
import test_chunked_gpu as CG

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
NAMES = ("gr", "gk", "gv", "gw", "gu", "gstate_in")
INF = float("inf")


def both_paths(variant, x, r, k, v, gy, u, s, gs, w_kind=None):
    """(y, state_out and gradients) on the chunked and on the token-serial kernels"""
    W, wkv56 = CG._pkg()
    w_kind = W.WKV_W_RAW if w_kind is None else w_kind
    name, out = "wkv6" if variant == "v6" else "wkv5", []
    for path in (W.WKV_PATH_CHUNKED, W.WKV_PATH_SCALAR):
        kw = dict(w_kind=w_kind, layout=W.WKV_STATE_KV, path=path)
        out.append(dict(zip(("y", "state_out"), wkv56.forward(name, r, k, v, x, u, s, **kw)))
                   | dict(zip(NAMES, wkv56.backward(name, r, k, v, x, u, s, gy, gs, **kw))))
    return out


def normal(g, *shape, std=1.0, mean=0.0, dtype=BF):
    return (torch.randn(shape, generator=g, device="cuda") * std + mean).to(dtype)


# (row, token, channel): the first and last token of a run of 16, of a chunk and of a row, one channel twice
PLACES = [(0, 0, 3), (0, 17, 3), (0, 31, 64), (0, 63, 5), (1, 64, 70), (1, 100, 70), (1, 108, 70), (1, 199, 127)]


@pytest.mark.parametrize("encoding", ["raw", "negexp"])
def test_infinite_decay_activations(encoding):
    """x = -inf is a decay of exactly 1, x = +inf the floor; neither has a gradient, and no other token notices"""
    W, wkv56 = CG._pkg()
    q = TL.case56("v6", 2, 200, 2, BF, seed=93)
    for i, at in enumerate(PLACES):
        q["x"][at] = INF if i % 2 else -INF
    with np.errstate(over="ignore", divide="ignore", invalid="ignore"):
        want = CG.floored_oracle("v6", q)
    d = {n: TL.to_dev(q[n], BF) for n in ("r", "k", "v", "gy", "u")}
    x = TL.to_dev(q["x"], BF)
    s, gs = TL.to_dev(q["state_in"], torch.float32), TL.to_dev(q["gstate_out"], torch.float32)
    if encoding == "negexp":
        x, kind = -torch.exp(x.float()), W.WKV_W_NEGEXP
    else:
        kind = W.WKV_W_RAW
    got = both_paths("v6", x, d["r"], d["k"], d["v"], d["gy"], d["u"], s, gs, kind)[0]
    for n in CG.EXTREME_CHECKED:
        if n != "gw" or encoding == "raw":      # (the literal call's gw is with respect to ew)
            TL.assert_close(f"v6.{n} {encoding}", got[n], want[n], 2e-2)
        assert torch.isfinite(got[n].float()).all(), n


def test_a_nan_decay_activation_is_the_floor():
    """as x = +inf is, in the forward and in the backward pass"""
    g = torch.Generator(device="cuda").manual_seed(97)
    r, k, v, gy = (normal(g, 1, 150, 64) for _ in range(4))
    x, u = normal(g, 1, 150, 64, std=0.5, mean=-0.6), normal(g, 1, 64)
    s, gs = normal(g, 1, 1, 64, 64, dtype=torch.float32), normal(g, 1, 1, 64, 64, dtype=torch.float32)
    runs = []
    for value in (float("nan"), INF):
        x[0, 70, 11] = x[0, 149, 63] = value
        runs.append(both_paths("v6", x, r, k, v, gy, u, s, gs)[0])
    for n in runs[0]:
        assert torch.isfinite(runs[0][n].float()).all() and torch.equal(runs[0][n], runs[1][n]), n


@pytest.mark.parametrize("variant", ["v6", "v5"])
@pytest.mark.parametrize("which", ["r", "k"])
def test_an_infinite_element_stays_with_its_own_token(which, variant):
    """gr does not depend on r nor gk on k; gv depends on r at later tokens and on k at its own"""
    T, t, g = 192, 83, torch.Generator(device="cuda").manual_seed(94)
    r, k, v, gy = (normal(g, 1, T, 64) for _ in range(4))
    x = normal(g, 1, T, 64, std=0.5, mean=-0.6) if variant == "v6" else normal(g, 1, 64, mean=-3, dtype=torch.float32)
    u, s, gs = normal(g, 1, 64), normal(g, 1, 1, 64, 64, dtype=torch.float32), normal(g, 1, 1, 64, 64, dtype=torch.float32)
    (r if which == "r" else k)[0, t, 9] = INF
    got, want = both_paths(variant, x, r, k, v, gy, u, s, gs)
    keep = torch.ones(T, dtype=torch.bool, device="cuda")
    keep[t] = False
    if which == "r":
        keep[:t] = False          # (those gradients are infinite: the token's output is)
    own = "gr" if which == "r" else "gk"
    for n, a, b in ((own, got[own], want[own]), ("gv", got["gv"][:, keep], want["gv"][:, keep])):
        if n == own:              # the bonus term of the other side's element
            a, b = a[:, keep], b[:, keep]
        assert torch.isfinite(b.float()).all(), n
        TL.assert_close(n, a, TL.back(b), 2e-2)


@pytest.mark.parametrize("bits", [2.1, 2.8, 3.7, 4.5])
def test_gradient_of_a_strong_static_decay(bits):
    """v5's decay gradient is what is left of a sum over all tokens in which large terms cancel; against the token-serial
    fp32 kernels, the worst of six draws at the bar of every bf16 output"""
    B, T, H, mean = 1, 330, 2, float(np.log(bits * np.log(2)))
    for seed in range(6):
        g = torch.Generator(device="cuda").manual_seed(seed)
        r, k, v, gy = (normal(g, B, T, 64 * H) for _ in range(4))
        x, u = normal(g, H, 64, std=0.02, mean=mean, dtype=torch.float32), normal(g, H, 64)
        s, gs = (normal(g, B, H, 64, 64, dtype=torch.float32) for _ in range(2))
        got, want = both_paths("v5", x, r, k, v, gy, u, s, gs)
        for n in got:
            TL.assert_close(f"v5.{n}", got[n], TL.back(want[n]), 2e-2, extra=f"(bits={bits}, seed={seed})")


@pytest.mark.parametrize("bits", [1.9, 2.1, 2.8, 3.4, 3.7])
@pytest.mark.parametrize("kv,gs", [(1, 1e-4), (1, 1e-6), (1, 1e-8), (1e-3, 1), (1e-3, 1e-3), (1e-3, 1e-6), (1e-6, 1), (1, 1e6)])
@pytest.mark.parametrize("variant", ["v6", "v5"])
def test_small_and_large_values_at_strong_decay(variant, bits, kv, gs):
    """`bits` of decay per token on average, k and v of size kv (states kv^2), gradients of size gs: each output against the
    token-serial fp32 kernels, relative to its own maximum"""
    B, T, H, g = 1, 330, 2, torch.Generator(device="cuda").manual_seed(95)
    r, k, v, gy = normal(g, B, T, 64 * H), normal(g, B, T, 64 * H, std=kv), normal(g, B, T, 64 * H, std=kv), normal(g, B, T, 64 * H, std=gs)
    mean = float(np.log(bits * np.log(2)))
    x = normal(g, B, T, 64 * H, std=0.02, mean=mean) if variant == "v6" else normal(g, H, 64, std=0.02, mean=mean, dtype=torch.float32)
    u = normal(g, H, 64)
    s = normal(g, B, H, 64, 64, std=kv * kv, dtype=torch.float32)
    gso = normal(g, B, H, 64, 64, std=gs, dtype=torch.float32)
    got, want = both_paths(variant, x, r, k, v, gy, u, s, gso)
    for n in got:
        TL.assert_close(f"{variant}.{n}", got[n], TL.back(want[n]), 2e-2, extra=f"(bits={bits}, kv={kv}, gs={gs})")
    # what a chunk's first token takes from the carried state
    first = torch.arange(64, T, 64, device="cuda")
    TL.assert_close("y at chunk starts", got["y"][:, first], TL.back(want["y"][:, first]), 2e-2)


@pytest.mark.parametrize("tokens,kv,gs", [(n, *s) for n in (8, 15, 16, 17) for s in ((1, 1), (1e-3, 1e-6))] + [(24, 1, 1)])
def test_bursts_of_strong_decay(tokens, kv, gs):
    """`tokens` of a chunk decay by 5.8 bits each in a few channels, the others by 0.5: on either side of what one
    reference point takes (128 bits a chunk), however the decay is spread"""
    B, T, H, g = 1, 320, 2, torch.Generator(device="cuda").manual_seed(96 + tokens)
    r, k, v, gy = normal(g, B, T, 64 * H), normal(g, B, T, 64 * H, std=kv), normal(g, B, T, 64 * H, std=kv), normal(g, B, T, 64 * H, std=gs)
    x = normal(g, B, T, 64 * H, std=0.1, mean=-1.1)
    for chunk, at in ((0, 0), (1, 20), (3, 64 - tokens), (4, 31)):
        x[:, 64 * chunk + at:64 * chunk + at + tokens, 5::40] = 1.39
    u, s = normal(g, H, 64), normal(g, B, H, 64, 64, std=kv * kv, dtype=torch.float32)
    got, want = both_paths("v6", x, r, k, v, gy, u, s, normal(g, B, H, 64, 64, std=gs, dtype=torch.float32))
    for n in got:
        TL.assert_close(n, got[n], TL.back(want[n]), 2e-2, extra=f"(tokens={tokens}, kv={kv}, gs={gs})")
