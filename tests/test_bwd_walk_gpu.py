"""The per-chunk backward kernel walks over a list of chunks per group of warps, mild ones first: more chunks than one
lookup of 32 covers, with steep ones scattered among them, alone, or none, and a last chunk that is not full."""
import pytest
import torch

import wkv_testlib as TL

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("B,T,H,steep", [(4, 4096, 40, 0.1), (4, 4090, 40, 0.0), (1, 8000, 3, 0.5), (2, 700, 2, 1.0), (1, 64, 1, 0.0)])
def test_gradients_of_many_chunks_match_the_token_serial_kernels(B, T, H, steep):
    """bf16 operands on the tensor cores against fp32 arithmetic token by token, max|a-b| / max|b| <= 2e-2; the decays
    (3.5 to 6 bits a token in a steep chunk) stay above the floor that only one of the two applies"""
    import rwkv_infctx_trainer_b200 as W
    from rwkv_infctx_trainer_b200 import wkv56
    wkv56.CHECK_STATUS = True
    C, g = 64 * H, torch.Generator(device="cuda").manual_seed(T + H)
    n = lambda *s, std=1.0, mean=0.0: torch.randn(s, generator=g, device="cuda") * std + mean
    r, k, v, gy = (n(B, T, C).to(BF) for _ in range(4))
    x = n(B, T, C, std=0.5, mean=-0.6)
    chunk = torch.arange(T, device="cuda") // 64
    pick = torch.rand((B, int(chunk[-1]) + 1, H), generator=g, device="cuda") < steep
    x = torch.where(pick[:, chunk].repeat_interleave(64, 2), n(B, T, C, std=0.1, mean=1.2).clamp(max=1.4), x).to(BF)
    u = (torch.rand((H, 64), generator=g, device="cuda") * 2 - 1).to(BF)
    s, gs = n(B, H, 64, 64, std=0.5), n(B, H, 64, 64, std=0.5)
    got, want = (wkv56.backward("wkv6", r, k, v, x, u, s, gy, gs, w_kind=W.WKV_W_RAW, layout=W.WKV_STATE_KV, path=p)
                 for p in (W.WKV_PATH_CHUNKED, W.WKV_PATH_SCALAR))
    for name, a, b in zip(("gr", "gk", "gv", "gw", "gu", "gstate_in"), got, want):
        e = float((a.float() - b.float()).abs().max() / b.float().abs().max())
        assert e <= 2e-2, (name, e)
