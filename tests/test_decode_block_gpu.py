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


@pytest.mark.parametrize("cls", ["RWKV_TimeMix6_0", "RWKV_TimeMix"])
@pytest.mark.parametrize("B,H,own", [(1, 96, True), (1, 97, False), (2, 64, True), (2, 65, False), (4, 64, True), (4, 65, False), (5, 32, True),
                                     (5, 33, False), (8, 32, True), (8, 33, False), (9, 2, False)])
def test_rows_and_widths_on_both_sides_of_the_rule(cls, B, H, own):
    """which call runs on the decode kernels (no library product at all), and that both sides give what the same token gives
    as the first of two"""
    C = 64 * H
    blk = _block(cls, C, H, torch.bfloat16)
    x = torch.randn((B, 2, C), device="cuda").bfloat16()
    state = (torch.randn((B, C), device="cuda").bfloat16(), torch.randn((B, H, 64, 64), device="cuda"))
    rel = lambda a, b: float((a.float() - b.float()).norm() / b.float().norm())
    with torch.no_grad(), torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        got, _ = blk(x[:, :1], state)
    products = sum(e.count for e in prof.key_averages() if e.key in ("aten::mm", "aten::addmm", "aten::bmm"))
    assert (products == 0) == own
    with torch.no_grad():
        want, _ = blk(x, state)
    assert rel(got, want[:, :1]) < 1e-2
