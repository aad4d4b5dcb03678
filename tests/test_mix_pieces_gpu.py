"""Backward of the token-shift mixes where its cut of a row can go wrong: rows shorter than a CTA's tokens, a last piece
of one token, several waves of CTAs, channels that do not fill a column block -- against autograd in fp32."""
import pytest
import torch

import rwkv_infctx_trainer_b200 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmix,data", [(5, True), (4, False), (1, False)])
@pytest.mark.parametrize("B,T,C", [(1, 1, 64), (2, 17, 320), (3, 129, 768), (40, 33, 2048), (1, 2049, 192)])
def test_mix_backward_at_the_edges_of_its_pieces(nmix, data, B, T, C):
    g = torch.Generator(device="cuda").manual_seed(T + C)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()
    x, shift = rnd(B, T, C).requires_grad_(), rnd(B, C).requires_grad_()
    maa = torch.rand((nmix, C), generator=g, device="cuda").requires_grad_()
    m = (rnd(nmix, B * T, C) * 0.1).requires_grad_() if data else None
    gout = rnd(nmix, B, T, C)
    leaves = [x, shift, maa] + ([m] if data else [])
    out = W.ddlerp(x, shift, maa, m.view(nmix, B, T, C) if data else None)
    got = torch.autograd.grad(out, leaves, gout.view(out.shape))
    xf, sf = x.detach().float().requires_grad_(), shift.detach().float().requires_grad_()
    af, mf = maa.detach().clone().requires_grad_(), m.detach().float().requires_grad_() if data else None
    prev = torch.cat([sf[:, None], xf[:, :-1]], 1)
    a = af[:, None, None] + (mf.view(nmix, B, T, C) if data else 0)
    ref = torch.autograd.grad(xf + (prev - xf) * a, [xf, sf, af] + ([mf] if data else []), gout.float())
    for r, q in zip(ref, got):
        assert (q.float() - r).abs().max() <= 1e-2 * r.abs().max()
