"""The parameter gradients gu and (v5) gw are folded over the batch and the chunks: by 16 groups of threads up to 16 rows, by
64 beyond.  Against the per-row sums that `wkv56.backward` leaves, which another kernel makes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["wkv6", "wkv5"])
@pytest.mark.parametrize("B,n", [(1, 1), (2, 1), (5, 3), (1, 16), (16, 1), (17, 1), (1, 17), (3, 21), (1, 64), (13, 5), (2, 70)])
def test_folded_parameter_gradients(variant, B, n):
    import rwkv_infctx_trainer_b200 as W
    from rwkv_infctx_trainer_b200 import wkv56
    T, H, g = 64 * n - 5, 3, torch.Generator(device="cuda").manual_seed(100 * B + n)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda")
    r, k, v, gy = (normal(B, T, 64 * H).bfloat16() for _ in range(4))
    w = (normal(B, T, 64 * H) * 0.5 - 0.6).bfloat16() if variant == "wkv6" else normal(H, 64) - 3
    u, s = normal(H, 64).bfloat16(), normal(B, H, 64, 64)
    for t in (w, u):
        t.requires_grad_(True)
    op = W.WKV6 if variant == "wkv6" else W.WKV5
    y, _ = op.apply(B, T, 64 * H, H, r, k, v, w, u, s, W.WKV_PATH_CHUNKED)
    gw, gu = torch.autograd.grad(y, (w, u), gy)
    part = wkv56.backward(variant, r, k, v, w.detach(), u.detach(), s, gy, None, w_kind=W.WKV_W_RAW, layout=W.WKV_STATE_KV,
                          path=W.WKV_PATH_CHUNKED)
    pairs = [(gu, part[4])] + ([(gw, part[3])] if variant == "wkv5" else [])
    for got, want in pairs:
        want = want.double().sum(0).view(H, 64)
        # fp32 sums of at most 140 rows in another order, then the parameter's own rounding (gu: 2^-9 of the element)
        bar = 2e-5 * want.abs().max() + (2 ** -8 * want.abs() if got.dtype == torch.bfloat16 else 0)
        assert bool(((got.double().view(H, 64) - want).abs() <= bar).all())
