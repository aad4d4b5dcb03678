"""How the per-chunk backward kernel deals chunks out to its groups of warps, two on every SM: fewer chunks than SMs, one
more, a few more than groups, several rounds; both kinds of chunk in one walk, of a per-token and of a static decay.
Compared chunk by chunk, so that a chunk of small gradients counts as well."""
import pytest
import torch

import wkv_testlib as TL

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
NAMES = ("gr", "gk", "gv", "gw", "gu", "gstate_in")


def worst(a, b, H):
    """the largest |a - b| of a chunk (or of a head's parameters) over 2 % of the chunk's largest |b| and 1 % of all of b's"""
    a, b = a.float(), b.float()
    if a.dim() == 3:                                  # [B, T, C]
        B, T, C = a.shape
        pad = (0, 0, 0, -T % 64)
        a, b = (torch.nn.functional.pad(t, pad).view(B, -1, 64, H, 64).transpose(2, 3).flatten(3) for t in (a, b))
    else:
        a, b = a.reshape(-1, 64), b.reshape(-1, 64)
    return float(((a - b).abs().amax(-1) / (2e-2 * b.abs().amax(-1) + 1e-2 * b.abs().max())).max())


@pytest.mark.parametrize("B,T,H,steep", [(1, 64, 147, 0.3), (1, 64, 148, 0.0), (1, 100, 75, 0.5), (1, 64, 297, 0.2), (3, 1000, 10, 0.4), (2, 2500, 12, 1.0)])
@pytest.mark.parametrize("variant", ["wkv6", "wkv5"])
def test_every_chunk_of_a_walk(variant, B, T, H, steep, monkeypatch):
    import rwkv_infctx_trainer_b200 as W
    from rwkv_infctx_trainer_b200 import wkv56
    monkeypatch.setattr(wkv56, "CHECK_STATUS", True)
    C, g = 64 * H, torch.Generator(device="cuda").manual_seed(T + H)
    n = lambda *s, std=1.0, mean=0.0: torch.randn(s, generator=g, device="cuda") * std + mean
    r, k, v, gy = (n(B, T, C).to(BF) for _ in range(4))
    # (steep: 3.5 to 5.8 bits a token, above the floor that only one of the two paths applies)
    if variant == "wkv6":
        chunk = torch.arange(T, device="cuda") // 64
        pick = torch.rand((B, int(chunk[-1]) + 1, H), generator=g, device="cuda") < steep
        x = torch.where(pick[:, chunk].repeat_interleave(64, 2), n(B, T, C, std=0.1, mean=1.2).clamp(max=1.4), n(B, T, C, std=0.5, mean=-0.6)).to(BF)
    else:
        pick = torch.rand((H, 1), generator=g, device="cuda") < steep
        x = torch.where(pick, n(H, 64, std=0.1, mean=1.2).clamp(max=1.4), n(H, 64, std=1.0, mean=-3.5).clamp(max=-0.5))
    u = (torch.rand((H, 64), generator=g, device="cuda") * 2 - 1).to(BF)
    s, gs = n(B, H, 64, 64, std=0.5), n(B, H, 64, 64, std=0.5)
    got, want = (wkv56.backward(variant, r, k, v, x, u, s, gy, gs, w_kind=W.WKV_W_RAW, layout=W.WKV_STATE_KV, path=p)
                 for p in (W.WKV_PATH_CHUNKED, W.WKV_PATH_SCALAR))
    for name, a, b in zip(NAMES, got, want):
        assert worst(a, b, H) <= 1, name
