"""One token of a v5 / v6 block for a few rows runs on kernels of its own: against the same block over a longer
call (the library GEMMs), at row counts around their variants and widths around what a warp prefetches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _block(cls, C, H, dtype):
    import rwkv_infctx_trainer_b200 as W
    torch.manual_seed(C + H)
    blk = getattr(W, cls)(1, 4, C, H, 64, C).cuda()
    with torch.no_grad():
        for n, p in blk.named_parameters():
            if "w2" in n or "w1" in n:
                p.normal_(0, 0.1)
    return blk.to(dtype)


@pytest.mark.parametrize("cls", ["RWKV_TimeMix6_0", "RWKV_TimeMix"])
@pytest.mark.parametrize("B,H,dtype", [(1, 1, torch.bfloat16), (1, 41, torch.bfloat16), (2, 12, torch.float32), (3, 40, torch.bfloat16),
                                       (5, 3, torch.float32), (8, 48, torch.bfloat16), (9, 4, torch.bfloat16)])
def test_decode_steps_match_the_same_tokens_in_one_call(cls, B, H, dtype):
    C, T = 64 * H, 3
    blk = _block(cls, C, H, dtype)
    x = torch.randn((B, T, C), device="cuda").bfloat16()
    state = (torch.randn((B, C), device="cuda").bfloat16(), torch.randn((B, H, 64, 64), device="cuda"))
    with torch.no_grad():
        want, (ws, wk) = blk(x, state)
        outs = []
        for t in range(T):
            o, state = blk(x[:, t:t + 1], state)
            outs.append(o)
    got = torch.cat(outs, 1)
    rel = lambda a, b: float((a.float() - b.float()).norm() / b.float().norm())
    assert got.shape == want.shape and got.dtype == want.dtype
    assert rel(got, want) < 1e-2
    assert rel(state[1], wk) < 5e-3
    assert torch.equal(state[0], ws)
